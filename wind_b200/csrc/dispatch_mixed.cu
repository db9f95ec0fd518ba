// dispatch_mixed.cu -- the single persistent launch over mass-action groups.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <numeric>
#include <vector>

#include "api_internal.h"
#include "mixed_kernel.cuh"

namespace wind {

MixedFn mixed_fn_counted(int method, int ctrl, int solver);  // dispatch_mixed_counted.cu

static int nmax_of(int n) { return n <= 8 ? 8 : (n <= 16 ? 16 : 32); }
bool team_admitted(int n, int R, bool lin, bool lists, int teams, size_t budget);
bool warp_admitted(int n, int R, bool lin, int solver, int threads, size_t budget);

// Launch all mass-action groups `ps` (kernel parameters with their counters
// already set) in one kernel on `stream`.  `spare`, `taken`: as launch_batch.
wind_status launch_mixed(const wind_options& o, const std::vector<KParams>& ps, cudaStream_t stream, size_t spare,
                         size_t* taken) {
    if (ps.empty()) return WIND_OK;
    const int solver = (o.method == WIND_METHOD_RK2) ? WIND_SOLVER_LU_F64 : o.solver;
    int dev = 0, cap = 227 * 1024;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&cap, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cap -= 1024;
    size_t smem = 0, gslot = 0, gneed = 0;
    bool counted = false;
    for (const KParams& p : ps) {
        // the solver each group runs (AUTO: MIXED above 32 species, LU_F64 below)
        const int gs = resolve_solver(solver, p.kind, p.n_eq);
        counted = counted || mixed_counted(p.n_eq, p.n_react);
        if (p.n_eq > 32) {
            const CtaLayout lay(p.n_eq, p.n_react, p.linear != nullptr, gs, cap, false,
                                o.method == WIND_METHOD_SIE);
            smem = std::max(smem, (size_t)lay.bytes);
            gslot = std::max(gslot, lay.slot_doubles());
            gneed = std::max(gneed, lay.g_doubles);
        } else {
            const int nm = nmax_of(p.n_eq);
            const bool reg = o.method == WIND_METHOD_SIE && gs != WIND_SOLVER_GJE_F64;
            const bool plin = p.linear != nullptr;
            if (reg) {
                if (!warp_admitted(p.n_eq, p.n_react, plin, gs, MIXED_THREADS, (size_t)cap))
                    return WIND_ERR_UNSUPPORTED;
                size_t bytes = (size_t)(MIXED_THREADS / nm) * WarpLayout(nm, p.n_react, plin, gs).bytes;
                if (gs == WIND_SOLVER_LU_F64) {
                    const LuLayout lay(nm, p.n_eq, p.n_react, plin, true);
                    bytes = (size_t)mixed_teams(nm, lay.bytes, cap) * lay.bytes;
                }
                smem = std::max(smem, bytes);
            } else {
                if (!team_admitted(p.n_eq, p.n_react, plin, o.method == WIND_METHOD_RK2, MIXED_THREADS / nm,
                                   (size_t)cap))
                    return WIND_ERR_UNSUPPORTED;
                const TeamLayout lay(nm, p.n_react, plin, o.method == WIND_METHOD_SIE);
                smem = std::max(smem, (size_t)mixed_teams(nm, lay.bytes, cap) * lay.bytes);
            }
        }
    }
    if (smem > (size_t)cap) return WIND_ERR_UNSUPPORTED;
    // (the MIXED team kernel has lists of its own)
    counted = counted && !(o.method == WIND_METHOD_SIE && o.solver == WIND_SOLVER_MIXED);
    const MixedFn fn = counted ? mixed_fn_counted(o.method, o.controller, o.solver)
                               : mixed_fn<false>(o.method, o.controller, o.solver);
    if (allow_block_smem((const void*)fn) != cudaSuccess)
        return launch_status("k_mixed shared-memory attribute");
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, MIXED_THREADS, smem) != cudaSuccess || nb < 1)
        return WIND_ERR_UNSUPPORTED;
    const int grid = nb * device_sm_count();
    // largest N first, then the larger group
    std::vector<int> order(ps.size());
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        if (ps[a].n_eq != ps[b].n_eq) return ps[a].n_eq > ps[b].n_eq;
        return ps[a].nsys > ps[b].nsys;
    });
    const size_t pbytes = ps.size() * sizeof(KParams), obytes = order.size() * sizeof(int);
    unsigned char* dparams = nullptr;
    if (pool_alloc((void**)&dparams, pbytes + obytes + 16, stream) != cudaSuccess) return WIND_ERR_NOMEM;
    double* gscratch = nullptr;
    if ((gslot - gneed) * grid * sizeof(double) > spare) gslot = gneed;
    if (gslot && pool_alloc((void**)&gscratch, gslot * grid * sizeof(double), stream) != cudaSuccess) {
        (void)cudaGetLastError();
        gscratch = nullptr;
        gslot = gneed;
    }
    if (gslot && !gscratch &&
        pool_alloc((void**)&gscratch, gslot * grid * sizeof(double), stream) != cudaSuccess) {
        cudaFreeAsync(dparams, stream);
        return WIND_ERR_NOMEM;
    }
    // one pageable host-to-device copy: it returns once the source has been
    // staged, so the host blob may go out of scope right after
    std::vector<unsigned char> blob(pbytes + obytes);
    std::memcpy(blob.data(), ps.data(), pbytes);
    std::memcpy(blob.data() + pbytes, order.data(), obytes);
    wind_status st = WIND_OK;
    st = cuda_status(cudaMemcpyAsync(dparams, blob.data(), blob.size(), cudaMemcpyHostToDevice, stream),
                     "group table upload");
    if (st == WIND_OK) {
        fn<<<grid, MIXED_THREADS, smem, stream>>>(reinterpret_cast<const KParams*>(dparams),
                                                  reinterpret_cast<const int*>(dparams + pbytes),
                                                  (int)ps.size(), gscratch, gslot, cap);
        g_launches++;
        st = launch_status("k_mixed launch");
        if (taken) *taken = (gslot - gneed) * grid * sizeof(double);
    }
    cudaFreeAsync(dparams, stream);
    if (gscratch) cudaFreeAsync(gscratch, stream);
    return st;
}

}  // namespace wind
