// api.cu -- extern "C" entry points of libwind (include/wind.h).
//
// Host side of the integrators: argument checks, device workspace, the
// kernel dispatch table, launches and copies.  The reference's harness
// (cuda/common/harness.cu:5-106) did cudaMalloc / copy / launch / copy /
// cudaFree per call on the default stream and returned an int step count;
// here allocations are stream-ordered (from a pool of the library's own, so
// repeated calls do not hit the driver), the caller may
// pass device pointers to skip the copies, and every failure is a status.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "api_internal.h"
#include "float32.h"
#include "networks.cuh"

using namespace wind;

namespace wind {

std::atomic<int64_t> g_launches{0};

static thread_local char t_last_error[160] = "";

void record_cuda_error(cudaError_t e, const char* where) {
    std::snprintf(t_last_error, sizeof(t_last_error), "%s: %s", where, cudaGetErrorName(e));
}
const char* last_error_text() { return t_last_error; }

template <class Fn>
static Fn driver_entry(const char* name) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
        (void)cudaGetLastError();
        f = nullptr;
    }
    return reinterpret_cast<Fn>(f);
}

bool current_context(ContextKey* out) {
    static const auto get = driver_entry<CUresult (*)(CUcontext*)>("cuCtxGetCurrent");
    static const auto id = driver_entry<CUresult (*)(CUcontext, unsigned long long*)>("cuCtxGetId");
    *out = ContextKey{};
    CUcontext c = nullptr;
    if (!get || !id || get(&c) != CUDA_SUCCESS || !c || id(c, &out->id) != CUDA_SUCCESS) return false;
    out->handle = c;
    return true;
}

// The library's pool of the current device and context, or null (then the
// device's default pool serves).
static cudaMemPool_t library_pool() {
    struct Pool {
        int device;
        ContextKey ctx;
        cudaMemPool_t pool;
    };
    static std::mutex mu;
    static std::vector<Pool> pools;
    int dev = -1;
    ContextKey ctx;
    std::lock_guard<std::mutex> g(mu);
    if (cudaGetDevice(&dev) != cudaSuccess || !current_context(&ctx)) return nullptr;
    for (const Pool& e : pools)
        if (e.device == dev && e.ctx.id == ctx.id) return e.pool;
    // a context that took over a destroyed one's handle: its pool went with it
    for (size_t i = 0; i < pools.size();) {
        if (pools[i].device == dev && pools[i].ctx.handle == ctx.handle) pools.erase(pools.begin() + i);
        else i++;
    }
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t made = nullptr;
    uint64_t keep = POOL_KEEP;
    if (cudaMemPoolCreate(&made, &props) != cudaSuccess) return nullptr;
    if (cudaMemPoolSetAttribute(made, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
        cudaMemPoolDestroy(made);
        return nullptr;
    }
    pools.push_back({dev, ctx, made});
    return made;
}

cudaError_t pool_alloc(void** p, size_t bytes, cudaStream_t stream) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    // inside a capture the allocation is the graph's, not a pool's
    if (cudaStreamIsCapturing(stream, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
        cudaMemPool_t pool = library_pool();
        if (pool) {
            if (cudaMallocFromPoolAsync(p, bytes, pool, stream) == cudaSuccess) return cudaSuccess;
            // what the pool keeps unused goes back before the device's own pool is asked
            (void)cudaMemPoolTrimTo(pool, 0);
        }
    }
    (void)cudaGetLastError();
    return cudaMallocAsync(p, bytes, stream);
}

static int builtin_n(int kind) {
    switch (kind) {
    case WIND_NET_NR_TEST: return NetNR::N;
    case WIND_NET_KATZ96: return NetKatz96::N;
    case WIND_NET_STIFFTRIG: return NetTrig::N;
    default: return -1;
    }
}
static int builtin_nc(int kind) {
    switch (kind) {
    case WIND_NET_NR_TEST: return NetNR::NC;
    case WIND_NET_KATZ96: return NetKatz96::NC;
    case WIND_NET_STIFFTRIG: return NetTrig::NC;
    default: return -1;
    }
}

cudaError_t allow_block_smem(const void* fn) {
    static std::mutex mu;
    static std::vector<std::pair<const void*, int>> fixed;  // static shared memory of each kernel
    int dev = 0, most = 0, used = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> g(mu);
        for (const auto& f : fixed)
            if (f.first == fn) used = f.second;
        if (used < 0) {
            cudaFuncAttributes fa{};
            e = cudaFuncGetAttributes(&fa, fn);
            if (e != cudaSuccess) return e;
            used = (int)fa.sharedSizeBytes;
            fixed.push_back({fn, used});
        }
    }
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most - used);
}

int device_sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
    return n;
}

wind_status check_network(const wind_network* net, int64_t nsys) {
    if (!net) return WIND_ERR_ARGUMENT;
    if (net->kind == WIND_NET_MASS_ACTION) {
        if (net->n_eq < 1 || net->n_eq > WIND_MAX_EQ) return WIND_ERR_UNSUPPORTED;
        if (net->n_react > 65535) return WIND_ERR_UNSUPPORTED;
        if (net->n_react < 0) return WIND_ERR_ARGUMENT;
        if (nsys > 0 && net->n_react > 0 && (!net->rates || !net->species)) return WIND_ERR_ARGUMENT;
        return WIND_OK;
    }
    const int n = builtin_n(net->kind);
    if (n < 0) return WIND_ERR_ARGUMENT;
    // n_eq = Ntile x N: Ntile copies of the network (the Precompiler's
    // tiling, python/ode_systems/ode_base.py:86-88, 219-281)
    if (net->n_eq < n || net->n_eq % n != 0) return WIND_ERR_ARGUMENT;
    if (net->n_eq / n > WIND_MAX_TILES) return WIND_ERR_UNSUPPORTED;
    if (net->n_const < builtin_nc(net->kind)) return WIND_ERR_ARGUMENT;
    if (nsys > 0 && !net->constants) return WIND_ERR_ARGUMENT;
    return WIND_OK;
}

// Launch the right kernel family for one homogeneous batch already on the
// device.  `p.counters` must point at zeroed device counters.
wind_status launch_integrate(const wind_options& o_in, const KParams& p, cudaStream_t stream,
                             bool allow_alloc) {
    if (p.nsys == 0) return WIND_OK;
    if (o_in.method == WIND_METHOD_SIM) return launch_sim(o_in, p, stream);
    // the tensor-core variant exists for the CTA kernels' MIXED inverse only
    if (o_in.solver == WIND_SOLVER_MIXED_TC &&
        (p.kind != WIND_NET_MASS_ACTION || p.n_eq <= WIND_TEAM_MAX_EQ || o_in.method != WIND_METHOD_SIE))
        return WIND_ERR_UNSUPPORTED;
    wind_options o = o_in;
    o.solver = resolve_solver(o.solver, p.kind, p.n_eq);
    if (p.kind != WIND_NET_MASS_ACTION) {
        const int n = builtin_n(p.kind);
        return p.n_eq == n ? launch_lane(o, p, stream) : launch_tile(o, p, n, stream);
    }
    if (p.n_eq <= WIND_TEAM_MAX_EQ) return launch_team(o, p, stream);
    // CTA kernels: global scratch for the matrices that do not fit in shared
    // memory, taken from the stream-ordered pool and returned after the launch
    CtaPlan pl;
    const wind_status pst = plan_cta(o, p, allow_alloc, &pl);
    if (pst != WIND_OK) return pst;
    if (pl.gstride == 0) return launch_cta(pl, p, stream, nullptr);
    double* scratch = nullptr;
    if (pool_alloc((void**)&scratch, (size_t)pl.grid * pl.gstride * sizeof(double), stream) != cudaSuccess) {
        (void)cudaGetLastError();
        pl.gstride = pl.need;
        if (pl.need == 0) return launch_cta(pl, p, stream, nullptr);
        if (pool_alloc((void**)&scratch, (size_t)pl.grid * pl.gstride * sizeof(double), stream) != cudaSuccess)
            return WIND_ERR_NOMEM;
    }
    const wind_status st = launch_cta(pl, p, stream, scratch);
    cudaFreeAsync(scratch, stream);
    return st;
}

}  // namespace wind

// ===========================================================================
extern "C" {

void wind_default_options(wind_options* opt) {
    if (!opt) return;
    opt->method = WIND_METHOD_SIE;
    opt->solver = WIND_SOLVER_GJE_F64;
    opt->controller = WIND_CTRL_DEVICE;
    opt->spec_width = 0;
    opt->max_attempts = 0;
    opt->timeout_s = 0.0;
}

const char* wind_version(void) { return "wind_b200 0.1 (sm_100a)"; }

const char* wind_status_string(int s) {
    switch (s) {
    case WIND_OK: return "ok";
    case WIND_ERR_ARGUMENT: return "invalid argument";
    case WIND_ERR_UNSUPPORTED: return "unsupported configuration";
    case WIND_ERR_CUDA: return "CUDA runtime error";
    case WIND_ERR_NOMEM: return "out of device memory";
    case WIND_ERR_TIMEOUT: return "timed out";
    case WIND_ERR_BUSY: return "admission refused";
    case WIND_ERR_NOT_FOUND: return "unknown request";
    default: return "unknown status";
    }
}

int64_t wind_launch_count(void) { return g_launches.load(); }

const char* wind_last_error(void) { return wind::last_error_text(); }

int wind_integrate(const wind_options* opt_in, const wind_network* net, double tnow,
                   double tend, int32_t n_integration_steps, double* y, int64_t nsys,
                   double atol, double rtol, int32_t* sys_status, int64_t* sys_nsteps,
                   int64_t* total_nsteps, int32_t memory, void* stream_v) {
    wind_options o;
    if (opt_in) o = *opt_in; else wind_default_options(&o);
    (void)cudaGetLastError();  // an earlier, unrelated error is not this call's
    if (check_options(o, true) != WIND_OK) return WIND_ERR_ARGUMENT;
    if (nsys < 0 || n_integration_steps < 1) return WIND_ERR_ARGUMENT;
    if (memory != WIND_MEM_HOST && memory != WIND_MEM_DEVICE) return WIND_ERR_ARGUMENT;
    wind_status st = check_network(net, nsys);
    if (st != WIND_OK) return st;
    if (nsys > 0 && !y) return WIND_ERR_ARGUMENT;
    if (total_nsteps) *total_nsteps = 0;
    if (nsys == 0) return WIND_OK;
    cudaStream_t stream = (cudaStream_t)stream_v;

    IntegrateCall call;
    st = call.prepare(o, *net, tnow, tend, n_integration_steps, y, nsys, atol, rtol,
                      sys_status, sys_nsteps, memory, stream);
    if (st == WIND_OK) st = launch_integrate(o, call.params, stream);
    if (st == WIND_OK) st = call.finish(total_nsteps);
    call.release();
    return st;
}

}  // extern "C"

// ---- the drop-in libraries' call on float32 host arrays ---------------------
// Widened and narrowed on the device (the same values as on the host): half the
// bytes cross the bus and the host touches them once.  One allocation; up to
// F32_PACK floats go in one copy and come back, with the substep total, in one.
// Through host conversions and a copy per array 8,000 Katz96 cells spent 360 us
// of a 675 us call outside the integrator.
constexpr size_t F32_PACK = 8192;

__global__ void k_widen(const float* in, double* out, size_t n, unsigned long long* counters) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < CNT_SLOTS) counters[i] = 0ull;
    for (size_t k = i; k < n; k += (size_t)gridDim.x * blockDim.x) out[k] = (double)in[k];
}
// The total goes right behind the results, as two 4-byte halves.
__global__ void k_narrow(const double* in, float* out, size_t n, const unsigned long long* counters) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        const unsigned long long total = counters[CNT_STEPS];
        out[n] = __uint_as_float((unsigned)total);
        out[n + 1] = __uint_as_float((unsigned)(total >> 32));
    }
    for (size_t k = i; k < n; k += (size_t)gridDim.x * blockDim.x) out[k] = (float)in[k];
}

extern "C" int wind_integrate_f32(const wind_options* opt_in, int32_t kind, int32_t n_eq, int32_t n_const,
                                  double tnow, double tend, int32_t n_integration_steps,
                                  const float* constants, float* y, int64_t nsys, double atol, double rtol,
                                  int64_t* total_nsteps) {
    wind_options o;
    if (opt_in) o = *opt_in; else wind_default_options(&o);
    (void)cudaGetLastError();
    *total_nsteps = 0;
    if (check_options(o) != WIND_OK || nsys < 0 || n_integration_steps < 1) return WIND_ERR_ARGUMENT;
    if (nsys > 0 && (!y || !constants)) return WIND_ERR_ARGUMENT;
    static const double present = 0.0;  // (the double constants only exist on the device)
    wind_network net = {};
    net.kind = kind;
    net.n_eq = n_eq;
    net.n_const = n_const;
    net.constants = &present;
    wind_status st = check_network(&net, nsys);
    if (st != WIND_OK || nsys == 0) return st;
    const size_t ny = (size_t)nsys * n_eq, nc = (size_t)nsys * n_const, n = ny + nc;
    cudaStream_t stream = nullptr;
    // [counters][y, constants as doubles][y and the total, constants as floats]
    const size_t o_f64 = 64, o_f32 = o_f64 + n * sizeof(double);
    unsigned char* d = nullptr;
    if (pool_alloc((void**)&d, o_f32 + (n + 2) * sizeof(float), stream) != cudaSuccess) return WIND_ERR_NOMEM;
    unsigned long long* counters = reinterpret_cast<unsigned long long*>(d);
    double* f64 = reinterpret_cast<double*>(d + o_f64);
    float* f32 = reinterpret_cast<float*>(d + o_f32);
    const bool packed = n <= F32_PACK;
    float pack[F32_PACK + 2];
    cudaError_t e;
    if (packed) {
        std::memcpy(pack, y, ny * sizeof(float));
        std::memcpy(pack + ny, constants, nc * sizeof(float));
        e = cudaMemcpyAsync(f32, pack, n * sizeof(float), cudaMemcpyHostToDevice, stream);
    } else {
        e = cudaMemcpyAsync(f32, y, ny * sizeof(float), cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(f32 + ny, constants, nc * sizeof(float), cudaMemcpyHostToDevice, stream);
    }
    st = cuda_status(e, "float upload");
    const int blocks = (int)std::min<size_t>((n + 255) / 256, (size_t)device_sm_count() * 8);
    if (st == WIND_OK) {
        k_widen<<<blocks, 256, 0, stream>>>(f32, f64, n, counters);
        g_launches++;
        KParams p{};
        p.kind = kind;
        p.n_eq = n_eq;
        p.n_const = n_const;
        p.constants = f64 + ny;
        p.tnow = tnow;
        p.tend = tend;
        p.h0 = (tend - tnow) / n_integration_steps;
        p.n_steps = n_integration_steps;
        p.atol = atol;
        p.rtol = rtol;
        p.y = f64;
        p.nsys = nsys;
        p.counters = counters;
        p.max_attempts = o.max_attempts > 0 ? o.max_attempts : ((int64_t)1 << 40);
        p.timeout_ns = o.timeout_s > 0 ? (uint64_t)(o.timeout_s * 1e9) : 0;
        st = launch_integrate(o, p, stream);
    }
    if (st == WIND_OK) {
        // (the constants' floats behind y are read already)
        k_narrow<<<blocks, 256, 0, stream>>>(f64, f32, ny, counters);
        g_launches++;
        unsigned total[2] = {};
        if (packed) {
            e = cudaMemcpyAsync(pack, f32, (ny + 2) * sizeof(float), cudaMemcpyDeviceToHost, stream);
        } else {
            e = cudaMemcpyAsync(y, f32, ny * sizeof(float), cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(total, f32 + ny, sizeof(total), cudaMemcpyDeviceToHost, stream);
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        st = cuda_status(e, "float download");
        if (st == WIND_OK && packed) {
            std::memcpy(y, pack, ny * sizeof(float));
            std::memcpy(total, pack + ny, sizeof(total));
        }
        if (st == WIND_OK) *total_nsteps = (int64_t)((unsigned long long)total[1] << 32 | total[0]);
    }
    cudaFreeAsync(d, stream);
    return st;
}

// ---- device-resident output loop and multi-group batch ---------------------
extern "C" {

int wind_integrate_output_steps(const wind_options* opt_in, const wind_network* net, double tnow,
                                double tend, int32_t n_integration_steps, int32_t n_output_steps,
                                double* y, int64_t nsys, double atol, double rtol,
                                double* out_over_time, int64_t* steps_per_output, int32_t memory,
                                void* stream_v) {
    wind_options o;
    if (opt_in) o = *opt_in; else wind_default_options(&o);
    if (n_output_steps < 1 || n_integration_steps < 1 || nsys < 0) return WIND_ERR_ARGUMENT;
    (void)cudaGetLastError();
    if (check_options(o, true) != WIND_OK) return WIND_ERR_ARGUMENT;
    if (memory != WIND_MEM_HOST && memory != WIND_MEM_DEVICE) return WIND_ERR_ARGUMENT;
    wind_status st = check_network(net, nsys);
    if (st != WIND_OK) return st;
    if (nsys > 0 && (!y || !out_over_time)) return WIND_ERR_ARGUMENT;
    if (nsys == 0) return WIND_OK;
    cudaStream_t stream = (cudaStream_t)stream_v;
    const int N = net->n_eq;
    const size_t ybytes = (size_t)nsys * N * sizeof(double);

    IntegrateCall call;
    st = call.prepare(o, *net, tnow, tend, n_integration_steps, y, nsys, atol, rtol, nullptr,
                      nullptr, memory, stream);
    // per-interval counters and the trajectory buffer live on the device
    unsigned long long* cnt = nullptr;
    double* traj = nullptr;
    if (st == WIND_OK) {
        cnt = static_cast<unsigned long long*>(
            call.alloc((size_t)n_output_steps * CNT_SLOTS * sizeof(unsigned long long)));
        traj = (memory == WIND_MEM_DEVICE) ? out_over_time
                                           : static_cast<double*>(call.alloc(ybytes * (n_output_steps + 1)));
        if (call.failed) st = WIND_ERR_NOMEM;
    }
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaStream_t cap = nullptr;
    if (st == WIND_OK && cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking) != cudaSuccess)
        st = WIND_ERR_CUDA;
    // Order the capture stream after the uploads on `stream`.
    cudaEvent_t ready = nullptr;
    if (st == WIND_OK) {
        cudaEventCreateWithFlags(&ready, cudaEventDisableTiming);
        cudaEventRecord(ready, stream);
        cudaStreamWaitEvent(cap, ready, 0);
        cudaStreamSynchronize(cap);
    }
    // ode_base.py:338-378: intervals [tcur, tcur+dt], tcur += dt
    if (st == WIND_OK && cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
        const double dt = (tend - tnow) / n_output_steps;
        double tcur = tnow;
        cudaMemsetAsync(cnt, 0, (size_t)n_output_steps * CNT_SLOTS * sizeof(unsigned long long), cap);
        cudaMemcpyAsync(traj, call.params.y, ybytes, cudaMemcpyDeviceToDevice, cap);
        for (int k = 0; k < n_output_steps && st == WIND_OK; k++) {
            KParams p = call.params;
            p.tnow = tcur;
            p.tend = tcur + dt;
            p.h0 = (p.tend - p.tnow) / n_integration_steps;
            p.counters = cnt + (size_t)k * CNT_SLOTS;
            st = launch_integrate(o, p, cap);
            cudaMemcpyAsync(traj + (size_t)(k + 1) * nsys * N, call.params.y, ybytes,
                            cudaMemcpyDeviceToDevice, cap);
            tcur += dt;
        }
        if (cudaStreamEndCapture(cap, &graph) != cudaSuccess) st = WIND_ERR_CUDA;
        if (st == WIND_OK && cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) st = WIND_ERR_CUDA;
        if (st == WIND_OK && cudaGraphLaunch(exec, cap) != cudaSuccess) st = WIND_ERR_CUDA;
        g_launches++;  // the graph launch (its kernel nodes are counted above)
        if (st == WIND_OK) {
            cudaEventRecord(ready, cap);
            cudaStreamWaitEvent(stream, ready, 0);
        }
    } else if (st == WIND_OK) {
        st = WIND_ERR_CUDA;
    }
    if (st == WIND_OK) {
        std::vector<unsigned long long> hc((size_t)n_output_steps * CNT_SLOTS);
        cudaMemcpyAsync(hc.data(), cnt, hc.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                        stream);
        if (memory == WIND_MEM_HOST)
            cudaMemcpyAsync(out_over_time, traj, ybytes * (n_output_steps + 1), cudaMemcpyDeviceToHost,
                            stream);
        st = call.finish(nullptr);
        if (st == WIND_OK && cudaStreamSynchronize(stream) != cudaSuccess) st = WIND_ERR_CUDA;
        if (st == WIND_OK && steps_per_output) {
            if (memory == WIND_MEM_HOST) {
                for (int k = 0; k < n_output_steps; k++)
                    steps_per_output[k] = (int64_t)hc[(size_t)k * CNT_SLOTS + CNT_STEPS];
            } else {
                std::vector<int64_t> tmp(n_output_steps);
                for (int k = 0; k < n_output_steps; k++)
                    tmp[k] = (int64_t)hc[(size_t)k * CNT_SLOTS + CNT_STEPS];
                cudaMemcpy(steps_per_output, tmp.data(), tmp.size() * sizeof(int64_t), cudaMemcpyHostToDevice);
            }
        }
    }
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    if (cap) {
        cudaStreamSynchronize(cap);
        cudaStreamDestroy(cap);
    }
    if (ready) cudaEventDestroy(ready);
    call.release();
    return st;
}

}  // extern "C"

extern "C" int wind_integrate_batch(const wind_options* opt_in, const wind_group* groups,
                                    int32_t ngroups, void* stream_v) {
    wind_options o;
    if (opt_in) o = *opt_in; else wind_default_options(&o);
    if (ngroups < 0 || (ngroups > 0 && !groups)) return WIND_ERR_ARGUMENT;
    (void)cudaGetLastError();
    if (wind::check_options(o) != WIND_OK) return WIND_ERR_ARGUMENT;
    return wind::launch_batch(o, groups, ngroups, (cudaStream_t)stream_v);
}
