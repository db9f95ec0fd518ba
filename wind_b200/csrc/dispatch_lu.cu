// dispatch_lu.cu -- launch of the FP64 LU team kernels (mass action, N <= 32).
#include <algorithm>
#include <mutex>
#include <vector>

#include "api_internal.h"
#include "lu_kernel.cuh"

namespace wind {

using LuFn = void (*)(KParams, int, int);

// The kernel of a size: rows padded to a multiple of four columns, on a team of
// 8, 16 or 32 lanes.  (Two rows per lane -- half the shared-memory reads per
// update -- measured half as fast: 230 to 255 registers, and twice the updates
// in every step of the pivot chain.)
struct LuKernel {
    LuFn fn;
    int lanes, cols;
};
template <int L, int COLS>
static LuKernel lu_pick(int ctrl) {
    return {ctrl == WIND_CTRL_GOLD ? k_lu<L, COLS, WIND_CTRL_GOLD> : k_lu<L, COLS, WIND_CTRL_DEVICE>, L,
            COLS};
}
static LuKernel lu_kernel(int n, int ctrl) {
    switch ((n + 3) / 4) {
    case 1: return lu_pick<8, 4>(ctrl);
    case 2: return lu_pick<8, 8>(ctrl);
    case 3: return lu_pick<16, 12>(ctrl);
    case 4: return lu_pick<16, 16>(ctrl);
    case 5: return lu_pick<32, 20>(ctrl);
    case 6: return lu_pick<32, 24>(ctrl);
    case 7: return lu_pick<32, 28>(ctrl);
    default: return lu_pick<32, 32>(ctrl);
    }
}

static int lu_blocks_per_sm(LuFn fn, size_t smem) {
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

bool warp_admitted(int n, int R, bool lin, int solver, int threads, size_t budget);

// One warp per block.  As in launch_team: the fewest teams per warp that hold
// the batch, or the split with the most resident teams.
wind_status launch_lu(const wind_options& o, const KParams& p, cudaStream_t stream) {
    const bool lin = p.linear != nullptr;
    if (!warp_admitted(p.n_eq, p.n_react, lin, WIND_SOLVER_LU_F64, WARP_THREADS, 227 * 1024))
        return WIND_ERR_UNSUPPORTED;
    const LuKernel k = lu_kernel(p.n_eq, o.controller);
    const LuFn fn = k.fn;
    const int lanes = k.lanes;
    // The sorted Jacobian terms are half of what a reaction takes, and the faster
    // path while two teams fit an SM with them.  A batch that would get one (above
    // some 1,620 reactions) goes without, with three: 4,000 systems of 32 species
    // and 1,900 reactions, 40 attempts each, 48.0 ms with the terms, 28.9 without;
    // one attempt 4.7 and 2.0 ms.
    int tpw = 0, sorted = 1;
    int64_t resident = 0;  // warps
    size_t bytes = 0;      // of a team
    for (sorted = 1; sorted >= 0; sorted--) {
        bytes = (size_t)LuLayout(k.cols, p.n_eq, p.n_react, lin, sorted != 0).bytes;
        tpw = 0;
        resident = 0;
        for (int t = 1; t <= 32 / lanes; t *= 2) {
            const size_t smem = (size_t)t * bytes;
            if (smem > 227 * 1024) break;
            const int64_t r = (int64_t)lu_blocks_per_sm(fn, smem) * device_sm_count();
            if (r * t >= resident * tpw && r > 0) {
                resident = r;
                tpw = t;
            }
            if (resident * tpw >= p.nsys) break;
        }
        if (!sorted || resident * tpw >= p.nsys || resident * tpw > device_sm_count()) break;
    }
    if (tpw == 0) return WIND_ERR_UNSUPPORTED;
    const size_t smem = (size_t)tpw * bytes;
    const int grid = (int)std::min<int64_t>((p.nsys + tpw - 1) / tpw, resident);
    if (allow_block_smem((const void*)fn) != cudaSuccess)
        return launch_status("k_lu shared-memory attribute");
    fn<<<grid, 32, smem, stream>>>(p, tpw, sorted);
    g_launches++;
    return launch_status("k_lu launch");
}

}  // namespace wind
