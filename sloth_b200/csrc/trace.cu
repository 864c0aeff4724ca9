// K2 (FP32 split) and K3 (FP64 port) tracer entry points: one trace of one
// ray set through one grid (the device code is in tracer.cuh).
#include "tracer.cuh"

namespace sloth {

// Which FP32 build traces n rays with Runge-Kutta-Nystrom steps: the one that
// fetches the next cell ahead while its 12 warps per SM hold all the rays at once,
// the 16-warp one above. With few warps a step waits for its cell (long scoreboard
// a third of it); with 16 the load and store pipe has no room for the ring's
// extra copies. Measured, time of the 16-warp build over the other's, turbulent and slab
// fields, along x, y and z (the two transverse strides differ: the cells that a ray along
// z crosses share lines):
//   rays               3e3        1e4        3e4        5e4        5.7e4 (12 warps)  7.2e4 (16-warp build)
//   512^3          1.0 .. 1.64 1.1 .. 1.60 1.1 .. 1.43 1.0 .. 1.26 1.0 .. 1.27      0.94 .. 1.31
//   256^3          1.1 .. 1.64 1.0 .. 1.60 1.1 .. 1.37 1.0 .. 1.26 1.0 .. 1.27      0.84 .. 1.09
//   192^3          1.0 .. 1.19 1.1 .. 1.32 1.1 .. 1.14 1.0 .. 1.12 1.0 .. 1.13      0.85 .. 0.94
//   128^3          1.0 .. 1.13 1.0 .. 1.13 1.0 .. 1.03 .97 .. 1.00 .94 .. 1.03      0.83 .. 1.04
//   64^3           1.0 .. 1.10 1.0 .. 1.03 .95 .. 1.02 .93 .. 1.01 .90 .. 1.02      0.81 .. 0.98
// A grid of up to 6 MB spreads over the SMs' L1s (40 KB each), where a cell comes
// soon enough once every scheduler has more than one warp: there four warps per SM end
// the build's range (64^3 turbulent, 3e4 and 5.7e4 rays 4 and 10 % faster so, the slab
// within 2 %; at 80^3 to 128^3 the turbulent field would gain 3 to 5 % and the slab lose as much).
// 512^3, 1e7 rays: 105 ms against 119.
constexpr int kAheadWarps = 12, kAheadWarpsL1 = 4;
constexpr long long kL1GridBytes = 6LL << 20;
static bool fetch_ahead(const TraceArgs& ta, int sms) {
    const long long bytes = 16LL * ta.geo.n[0] * ta.geo.n[1] * ta.geo.n[2];
    return ta.n <= (long long)sms * (bytes <= kL1GridBytes ? kAheadWarpsL1 : kAheadWarps) * 32;
}
// Rays of a warp's first take: 32, or as few as kSpreadMin as long as that gives
// each of an SM's four schedulers one warp (fewer rays, fewer cells that the warp waits
// for: FP64, 5e3 rays 597 -> 529 us; 1e4 rays, 128^3 107 -> 105). More, smaller warps
// share the schedulers and lose: 1e4 rays in warps of 8 (two per scheduler) 133 us.
constexpr int kSpreadWarps = 4, kSpreadMin = 8;

template <class P, int IB, int FAST, int INTEG, bool AHEAD>
__global__ void __launch_bounds__(trace_threads<P, AHEAD>(), trace_min_blocks<P, INTEG, AHEAD>())
trace_kernel(const __grid_constant__ TraceArgs a, int first_rays) {
    unsigned long long my_steps = 0;
    CellCacheFor<P, AHEAD> cc;
    reset_cache(cc);
    const unsigned n = (unsigned)a.n;
    constexpr unsigned kWarps = trace_threads<P, AHEAD>() / 32;
    const unsigned warp = blockIdx.x * kWarps + (threadIdx.x >> 5), warps = gridDim.x * kWarps;
    TraceQueue q{a.queue, warps * first_rays, min(warp * first_rays, n), min((warp + 1) * first_rays, n), n};
    trace_warp<P, IB, FAST, INTEG>(a, q, cc, my_steps);
    if constexpr (AHEAD) fetch_wait();
    warp_add(my_steps, a.total_steps);
}

template <class P, int IB, int FAST, int INTEG, bool AHEAD>
static int launch_trace_k(const TraceArgs& ta, int sms, cudaStream_t s) {
    constexpr int kCta = trace_threads<P, AHEAD>(), kWarps = kCta / 32;
    static int cached[64] = {0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_status(e);
    int per_sm = (dev >= 0 && dev < 64) ? cached[dev] : 0;
    if (per_sm <= 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, trace_kernel<P, IB, FAST, INTEG, AHEAD>, kCta, 0) != cudaSuccess || per_sm < 1)
            per_sm = 1;
        if (dev >= 0 && dev < 64) cached[dev] = per_sm;
    }
    long long blocks = (long long)sms * per_sm;
    int first = 32;
    const long long spread = (ta.n + (long long)sms * kSpreadWarps - 1) / ((long long)sms * kSpreadWarps);
    if (spread < first) first = spread > kSpreadMin ? (int)spread : kSpreadMin;
    const long long want = (ta.n + first * kWarps - 1) / (first * kWarps);
    if (blocks > want) blocks = want;
    trace_kernel<P, IB, FAST, INTEG, AHEAD><<<(int)blocks, kCta, 0, s>>>(ta, first);
    note_launch();
    return cuda_status(cudaGetLastError());
}

template <class P, int IB, int INTEG, bool AHEAD = false>
static int launch_trace_i(const TraceArgs& ta, int sms, cudaStream_t s, int fast) {
    return fast == 1 ? launch_trace_k<P, IB, 1, INTEG, AHEAD>(ta, sms, s)
         : fast == 2 ? launch_trace_k<P, IB, 2, INTEG, AHEAD>(ta, sms, s)
                     : launch_trace_k<P, IB, 0, INTEG, AHEAD>(ta, sms, s);
}

template <class P, int IB>
static int launch_trace(const TraceArgs& ta, int sms, cudaStream_t s, int fast, int integ) {
    if (integ == INTEG_RK4) return launch_trace_i<P, IB, INTEG_RK4>(ta, sms, s, fast);
    if constexpr (sizeof(typename P::R) == 4)
        if (fetch_ahead(ta, sms)) return launch_trace_i<P, IB, INTEG_RKN, true>(ta, sms, s, fast);
    return launch_trace_i<P, IB, INTEG_RKN>(ta, sms, s, fast);
}

template <class P>
static int trace_impl(const SlothGridDesc* g, const void* grid, const SlothTraceParams* p,
                      const void* rays, int64_t n, const SlothTraceOutputs* out, void* ws,
                      size_t ws_bytes, void* stream) {
    using R = typename P::R;
    int rc = check_trace_params(g, p, n);
    if (rc) return rc;
    if (!out) return SLOTH_ERR_NULL_POINTER;
    if (n == 0) {
        if (out->total_steps) {
            cudaError_t e = cudaMemsetAsync(out->total_steps, 0, sizeof(unsigned long long), (cudaStream_t)stream);
            return cuda_status(e);
        }
        return SLOTH_OK;
    }
    if (!grid || !rays || !out->jones || !ws) return SLOTH_ERR_NULL_POINTER;
    if (((uintptr_t)grid & 15u) != 0 || ((uintptr_t)ws & 255u) != 0) return SLOTH_ERR_MISALIGNED;
    if (((uintptr_t)rays & (sizeof(R) - 1)) != 0 || ((uintptr_t)out->jones & (sizeof(R) - 1)) != 0)
        return SLOTH_ERR_MISALIGNED;
    if (ws_bytes < workspace_bytes(n)) return SLOTH_ERR_WORKSPACE_TOO_SMALL;

    cudaStream_t s = (cudaStream_t)stream;
    char* base = reinterpret_cast<char*>(ws);
    unsigned* queue = reinterpret_cast<unsigned*>(base);
    unsigned* hist = reinterpret_cast<unsigned*>(base + kHeaderBytes);
    const size_t an = align256((size_t)n * 4u);
    unsigned* keys = reinterpret_cast<unsigned*>(base + kHeaderBytes + kHistBytes);
    unsigned* perm = reinterpret_cast<unsigned*>(base + kHeaderBytes + kHistBytes + an);
    unsigned* offs = reinterpret_cast<unsigned*>(base + kHeaderBytes + kHistBytes + 2 * an);

    const int bbits = bucket_bits_for(n);
    cudaError_t e;
    int sms = 148;
    rc = device_sm_count(&sms);
    if (rc) return rc;
    rc = launch_prepass<R>(g, p->probing_axis, reinterpret_cast<const R*>(rays), n, bbits, keys, hist, perm,
                           offs, out->total_steps, queue, sms, s);
    if (rc) return rc;

    TraceArgs ta;
    fill_trace_args(ta, g, grid, p, rays, n, out, perm);
    ta.queue = queue;
    const int ib = trace_mode(p);
    // interior runs with interior sampling, interior runs only, or neither
    const int fast = interior_bound_ok(g, p) ? 1 : (std::isfinite(interior_accel_bound(g, p)) ? 2 : 0);

    if (out->trace_event_begin) {
        e = cudaEventRecord((cudaEvent_t)out->trace_event_begin, s);
        if (e != cudaSuccess) return cuda_status(e);
    }
    const int integ = p->integrator;
    if (ib == IB_OFF)
        rc = launch_trace<P, IB_OFF>(ta, sms, s, fast, integ);
    else if (ib == IB_SUBCRITICAL)
        rc = launch_trace<P, IB_SUBCRITICAL>(ta, sms, s, fast, integ);
    else
        rc = launch_trace<P, IB_GENERAL>(ta, sms, s, fast, integ);
    if (rc) return rc;
    if (out->trace_event_end) {
        e = cudaEventRecord((cudaEvent_t)out->trace_event_end, s);
        if (e != cudaSuccess) return cuda_status(e);
    }
    return SLOTH_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of the FP32 tracer: its scratch (ray counter,
// bucket histogram, keys, permutation) lives in one file-scope device array
// sized for SLOTH_NOALLOC_MAX_RAYS rays, so the caller passes only inputs and
// outputs and nothing here allocates. Host code cannot use the array's name
// as a device address; every call looks the current device's address up with
// cudaGetSymbolAddress (the first call on a device also loads the library's
// device code there). A cached address would dangle after cudaDeviceReset,
// which reloads the device code at a new address. All calls share the array,
// which keeps the previous call's contents (the tracer zeroes the parts that
// must start at zero), so calls that overlap on the GPU race.
// ---------------------------------------------------------------------------
constexpr size_t kNoAllocScratchBytes = kHeaderBytes + kHistBytes + 3 * (size_t)4 * SLOTH_NOALLOC_MAX_RAYS;
static_assert(kNoAllocScratchBytes % 256 == 0, "scratch sections must stay 256-byte aligned");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

static int noalloc_scratch(void** out) {
    void* addr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&addr, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_status(e);
    if (addr == nullptr || ((uintptr_t)addr & 255u) != 0) return SLOTH_ERR_MISALIGNED;
    *out = addr;
    return SLOTH_OK;
}

}  // namespace sloth

extern "C" {

size_t sloth_trace_workspace_bytes(int64_t n_rays) { return sloth::workspace_bytes(n_rays); }

int sloth_trace_f32_noalloc(const SlothGridDesc* g, const void* grid, const SlothTraceParams* p,
                            const float* rays, int64_t n, const SlothTraceOutputs* out, void* stream) {
    if (n < 0) return SLOTH_ERR_INVALID_ARGUMENT;
    if (n > (int64_t)SLOTH_NOALLOC_MAX_RAYS) return SLOTH_ERR_TOO_LARGE;
    void* scratch = nullptr;
    const int rc = sloth::noalloc_scratch(&scratch);
    if (rc) return rc;
    return sloth::trace_impl<sloth::PolF32>(g, grid, p, rays, n, out, scratch, sloth::kNoAllocScratchBytes,
                                            stream);
}

int sloth_trace_f32(const SlothGridDesc* g, const void* grid, const SlothTraceParams* p, const float* rays,
                    int64_t n, const SlothTraceOutputs* out, void* workspace, size_t workspace_bytes,
                    void* stream) {
    return sloth::trace_impl<sloth::PolF32>(g, grid, p, rays, n, out, workspace, workspace_bytes, stream);
}

int sloth_trace_f64(const SlothGridDesc* g, const void* grid, const SlothTraceParams* p, const double* rays,
                    int64_t n, const SlothTraceOutputs* out, void* workspace, size_t workspace_bytes,
                    void* stream) {
    return sloth::trace_impl<sloth::PolF64>(g, grid, p, rays, n, out, workspace, workspace_bytes, stream);
}

}  // extern "C"
