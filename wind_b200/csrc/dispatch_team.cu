// dispatch_team.cu -- launch of the team-per-system kernels (mass action,
// N <= 32: the reference Gauss-Jordan and RK2).
#include <algorithm>
#include <mutex>
#include <vector>

#include "api_internal.h"
#include "team_kernel.cuh"

namespace wind {

using TeamFn = void (*)(KParams, int);
TeamFn team_fn_8(int method, int ctrl);
TeamFn team_fn_16(int method, int ctrl);
TeamFn team_fn_32(int method, int ctrl);

int team_nmax(int n) { return n <= 8 ? 8 : (n <= 16 ? 16 : 32); }

// Shared memory one team may ask for when `teams` of them share a block's
// `budget`: the sizes (N, R) the entry points accept are the ones whose
// matrices, vectors, rates and species (and, for RK2 in a mixed-size launch,
// incidence lists) fit a full block, whatever a launch then uses.
bool team_admitted(int n, int R, bool lin, bool lists, int teams, size_t budget) {
    const int nm = team_nmax(n);
    auto a16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    size_t b = a16((size_t)10 * nm * 8) + a16(lin ? (size_t)nm * nm * 4 : 0) + 2 * a16((size_t)R * 8);
    if (lists) b += a16((size_t)nm * (nm + 2) * 8) + a16((nm + 1) * 4) + a16((size_t)8 * R) + a16(nm * 4);
    else b += a16((size_t)nm * nm * 8) + a16((size_t)2 * (2 * nm + 4) * 8);
    return (size_t)teams * b <= budget;
}

static int team_blocks_per_sm(TeamFn fn, size_t smem) {
    static std::mutex mu;
    static std::vector<std::pair<std::pair<const void*, size_t>, int>> cache;
    std::lock_guard<std::mutex> g(mu);
    for (auto& e : cache)
        if (e.first.first == (const void*)fn && e.first.second == smem) return e.second;
    (void)allow_block_smem((const void*)fn);
    int nb = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, 32, smem) != cudaSuccess || nb < 1) {
        (void)cudaGetLastError();
        nb = 0;
    }
    cache.push_back({{(const void*)fn, smem}, nb});
    return nb;
}

wind_status launch_warp(const wind_options& o, const KParams& p, cudaStream_t stream);

// One warp per block, 1 to 32/NMAX teams per warp.  A team's time per substep
// is its own dependent chain as long as it has the warp to itself, and teams
// that share a warp wait for each other's divergent parts: a batch that fits
// the GPU with fewer teams per warp takes the fewest that hold it; a larger
// one takes the split with the most resident teams.
wind_status launch_team(const wind_options& o, const KParams& p, cudaStream_t stream) {
    // SIE with an LU or mixed solve: the register-resident kernel
    if (o.method == WIND_METHOD_SIE && o.solver != WIND_SOLVER_GJE_F64) return launch_warp(o, p, stream);
    const bool lin = p.linear != nullptr;
    const int nmax = team_nmax(p.n_eq);
    if (!team_admitted(p.n_eq, p.n_react, lin, false, 128 / nmax, 227 * 1024)) return WIND_ERR_UNSUPPORTED;
    TeamFn fn = nmax == 8 ? team_fn_8(o.method, o.controller)
              : nmax == 16 ? team_fn_16(o.method, o.controller)
                           : team_fn_32(o.method, o.controller);
    const TeamLayout lay(nmax, p.n_react, lin, o.method == WIND_METHOD_SIE);
    int tpw = 0;
    int64_t resident = 0;  // warps
    for (int t = 1; t <= 32 / nmax; t *= 2) {
        const size_t smem = (size_t)t * lay.bytes;
        if (smem > 227 * 1024) break;
        const int64_t r = (int64_t)team_blocks_per_sm(fn, smem) * device_sm_count();
        if (r * t >= resident * tpw && r > 0) {
            resident = r;
            tpw = t;
        }
        if (resident * tpw >= p.nsys) break;
    }
    if (tpw == 0) return WIND_ERR_UNSUPPORTED;
    const size_t smem = (size_t)tpw * lay.bytes;
    const int grid = (int)std::min<int64_t>((p.nsys + tpw - 1) / tpw, resident);
    if (allow_block_smem((const void*)fn) != cudaSuccess)
        return launch_status("k_team shared-memory attribute");
    fn<<<grid, 32, smem, stream>>>(p, tpw);
    g_launches++;
    return launch_status("k_team launch");
}

}  // namespace wind
