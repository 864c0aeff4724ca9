// K1 grid pack and K0 trilinear sample.
//
// K1 follows precompute_gradients (src/core/propagator.py:72-93): the driving
// term is proportional to ne, and its gradient is taken with jnp.gradient
// semantics along each axis (second-order central differences inside,
// first-order one-sided differences on the two faces). Here the gradient is
// kept per grid cell and normalised to the critical density, q = ne/nc; the
// tracers fold the -c^2/2 and 1/h^2 factors into one per-axis constant.
// Channel 0 holds q itself (the value layout, read by the K0 sampler and the
// detector-image model) or, in the trace layout, the refractive index minus
// one, n - 1 = sqrt(1 - x) - 1 with x = (omega_pe/omega)^2 = ope_ratio2 * q,
// which the tracers interpolate for the optical phase as the legacy solver
// interpolates its n grid (src/legacy/full_solver.py:289, :292-296, :342-345).
// It is evaluated as -x / (1 + sqrt(1 - x)), free of cancellation, and is -x
// above the critical density (where the legacy n is not real).
// All arithmetic is FP64; the FP32 grid rounds the final values once. q = ne *
// scale is rounded on its own (__dmul_rn keeps the compiler from fusing it into
// the differences), so the result is a plain IEEE evaluation of the formula.
#include "common.cuh"

namespace sloth {

// n - 1 of x = ope2 * q, every operation rounded on its own (no fused
// multiply-add), so that it equals a plain IEEE evaluation of the formula.
__device__ __forceinline__ double n_minus_1_of(double q, double ope2) {
    const double x = __dmul_rn(ope2, q);
    const double om = fmax(__dsub_rn(1.0, x), 0.0);
    return -__ddiv_rn(x, __dadd_rn(1.0, __dsqrt_rn(om)));
}

// The same for the FP32 grid, whose result is rounded to FP32: m = 1 - sqrt(1 - x)
// is the root below 1 of m (2 - m) = x, found by two simplified Newton steps
// in FP64 (Newton's iteration with the derivative 2 sqrt(1 - x) held at its
// FP32 value) from an FP32 estimate. A step leaves delta (eps + delta / 2s) of
// an error delta, s = sqrt(1 - x) and eps <= 2^-19 the FP32 derivative's
// relative error; with s > 1/8 the estimate's 2^-21 becomes 2^-38 and then
// less than FP64's rounding of the terms (a few 2^-53), so the FP32 result is
// the formula's but for one value in about 2^27 that lies that close to a
// rounding boundary. 9 FP64 operations against about 45 of a division and a square
// root. xs = ope2 * scale in FP32 (0: not usable there). Close to or above the critical density,
// and for values that are not finite, the formula itself.
__device__ __forceinline__ float n_minus_1_f32(float nef, float xs, double q, double ope2) {
    const float xf = nef * xs;
    const float omf = 1.0f - xf;
    if (omf > 0.015625f && omf < 1e6f && xs > 0.0f) {
        float rs, r1;   // hardware estimates of 1 / s and 1 / (1 + s)
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rs) : "f"(omf));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(fmaf(omf, rs, 1.0f)));
        const double m0 = (double)(xf * r1), g = (double)(0.5f * rs);
        const double x = __dmul_rn(ope2, q);
        const double m1 = __fma_rn(__fma_rn(-m0, __dsub_rn(2.0, m0), x), g, m0);
        return (float)-__fma_rn(__fma_rn(-m1, __dsub_rn(2.0, m1), x), g, m1);
    }
    return (float)n_minus_1_of(q, ope2);
}

// Order-preserving 64-bit keys of doubles: larger value, larger key; a NaN is
// above everything. Zero is below every value's key.
__device__ __forceinline__ unsigned long long order_key(double v) {
    if (v != v) return ~0ull;
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// Asynchronous copy of one density to shared memory, and the wait for all but
// the newest N committed groups of this thread's copies.
template <class In>
__device__ __forceinline__ void copy_async(In* dst, const In* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"((int)sizeof(In)) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Running range of the densities of one thread, NaN kept.
__device__ __forceinline__ void range_add(float v, float& lo, float& hi) {
    asm("min.NaN.f32 %0, %0, %1;" : "+f"(lo) : "f"(v));
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(hi) : "f"(v));
}
__device__ __forceinline__ void range_add(double v, double& lo, double& hi) {
    lo = v < lo || v != v ? v : lo;
    hi = v > hi || v != v ? v : hi;
}

// Pack: a CTA takes a kTileJ x kTileK patch of the (j, k) plane and walks
// `planes` planes along i. Each density is loaded, converted and scaled once
// per patch (1.5 times with the patch's border): the i neighbours are the
// thread's own previous and next value, the j and k neighbours come from the
// plane's copy in shared memory (two buffers, one barrier per plane). The next
// kAhead planes' densities are on their way as asynchronous copies into slots
// that only the copying thread reads, so they hold no registers and need no
// barrier of their own. Indices are clamped into the grid and the half of a
// central difference becomes 1 on a face, which is the one-sided difference
// there (x * 1.0 is exact), so no access and no difference needs a test.
// 512^3, FP32 in and out, trace layout: 1.70 ms before, reading all seven
// densities per voxel through L1 with the formula's division and square root
// (FP64, conversion and address instructions), 0.65 ms now (4.1 TB/s), bound by the
// latency of a plane (load, conversion, barrier) at the 16 warps that fit an SM. With loads
// ahead in registers instead 0.76; 32-wide patches on 24 or 32 warps 0.70 and 0.82
// (spills); eight planes ahead are no faster.
// With `range`, the CTA's largest density and largest negated density go to
// range[0] and range[1] as order keys.
constexpr int kTileK = 64, kTileJ = 8;
constexpr int kAhead = 4;                              // planes on their way (cp.async groups)
constexpr int kCols = kTileK / 32;                     // columns (k) per thread, 32 apart
constexpr int kPackThreads = 32 * kTileJ;
constexpr int kPackBorder = 2 * kTileK + 2 * kTileJ;   // border densities of a patch (no corners)
static_assert(kPackBorder <= kPackThreads, "one border density per thread");

template <class In, bool F64OUT, bool NM1, bool RANGE>
__global__ void __launch_bounds__(kPackThreads, 2)
pack_kernel(const In* __restrict__ ne, void* __restrict__ out, GridGeo g, double scale, double ope2, float xs,
            int planes, unsigned tiles_k, unsigned tiles_j, unsigned long long* range) {
    __shared__ double s_q[2][kTileJ + 2][kTileK + 2];
    __shared__ In s_raw[kAhead][kCols + 1][kPackThreads];   // each thread reads only what it copied itself
    const int t = threadIdx.x, tk = t & 31, tj = t >> 5;
    const unsigned bk = blockIdx.x % tiles_k, bj = (blockIdx.x / tiles_k) % tiles_j, bi = blockIdx.x / (tiles_k * tiles_j);
    const int k0 = (int)bk * kTileK + tk, j = (int)bj * kTileJ + tj;
    const int i0 = (int)bi * planes, i1 = min(i0 + planes, g.n[0]);
    const int nj = g.n[1], nk = g.n[2], last = g.n[0] - 1;
    const double wj = j == 0 || j == nj - 1 ? 1.0 : 0.5;
    bool mine[kCols];
    double wk[kCols];
    unsigned col[kCols];                               // offset in a plane, clamped into it
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
        const int k = k0 + 32 * c;
        mine[c] = j < nj && k < nk;
        wk[c] = k == 0 || k == nk - 1 ? 1.0 : 0.5;
        col[c] = (unsigned)min(j, nj - 1) * nk + (unsigned)min(k, nk - 1);
    }
    // this thread's border density: rows j0 - 1 and j0 + kTileJ, then columns k0 - 1 and k0 + kTileK
    const bool border = t < kPackBorder;
    int pj, pk;
    if (t < 2 * kTileK) {
        pj = t < kTileK ? 0 : kTileJ + 1;
        pk = (t & (kTileK - 1)) + 1;
    } else {
        pj = (t & (kTileJ - 1)) + 1;
        pk = t < 2 * kTileK + kTileJ ? 0 : kTileK + 1;
    }
    const int gj = min(max((int)bj * kTileJ + pj - 1, 0), nj - 1), gk = min(max((int)bk * kTileK + pk - 1, 0), nk - 1);
    const unsigned bcol = (unsigned)gj * nk + (unsigned)gk;
    double* const sb = &s_q[0][pj][pk];
    double* const sm = &s_q[0][tj + 1][tk + 1];
    constexpr int kRow = kTileK + 2, kBuf = (kTileJ + 2) * kRow;

    auto scaled = [&](In v) { return __dmul_rn((double)v, scale); };
    const unsigned plane = g.sx;
    const int top = min(i1, last);                     // the last plane that this CTA reads
    const In* at = ne + (size_t)i0 * plane;            // the plane that is fetched next
    int ahead = i0;
    auto fetch = [&]() {                               // copies plane `ahead`; one group per plane
        In (*d)[kPackThreads] = s_raw[(ahead - i0) % kAhead];
        if (ahead <= top) {
#pragma unroll
            for (int c = 0; c < kCols; ++c) copy_async(&d[c][t], at + col[c]);
            if (border) copy_async(&d[kCols][t], at + bcol);
        }
        copy_commit();
        at += plane;
        ++ahead;
    };
    char* o = reinterpret_cast<char*>(out) + (size_t)i0 * plane * (F64OUT ? 32 : 16);
    for (int u = 0; u < kAhead; ++u) fetch();
    copy_wait<kAhead - 2>();                           // planes i0 and i0 + 1
    double q[kCols], prev[kCols];
    In raw[kCols], lo[kCols], hi[kCols];
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
        raw[c] = lo[c] = hi[c] = s_raw[0][c][t];
        q[c] = scaled(raw[c]);
        prev[c] = i0 > 0 ? scaled(__ldg(ne + (size_t)(i0 - 1) * plane + col[c])) : q[c];
    }
    for (int i = i0; i < i1; i += 2) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (i + u >= i1) break;                    // the same in every thread
            const int buf = u & 1 ? kBuf : 0;
            const int slot = (i + u - i0) % kAhead;
#pragma unroll
            for (int c = 0; c < kCols; ++c) sm[buf + 32 * c] = q[c];
            if (border) sb[buf] = scaled(s_raw[slot][kCols][t]);
            In next_raw[kCols];
#pragma unroll
            for (int c = 0; c < kCols; ++c)
                next_raw[c] = i + u < last ? s_raw[(slot + 1) % kAhead][c][t] : raw[c];
            fetch();                                   // into this plane's slot, just read
            copy_wait<kAhead - 2>();                   // the next two planes
            __syncthreads();
            const double wi = i + u == 0 || i + u == last ? 1.0 : 0.5;
#pragma unroll
            for (int c = 0; c < kCols; ++c) {
                const double next = scaled(next_raw[c]);
                if (mine[c]) {
                    if constexpr (RANGE) range_add(raw[c], lo[c], hi[c]);
                    const double* p = sm + buf + 32 * c;
                    const double d0 = wi * (next - prev[c]);
                    const double d1 = wj * (p[kRow] - p[-kRow]);
                    const double d2 = wk[c] * (p[1] - p[-1]);
                    if constexpr (F64OUT) {
                        double2* v = reinterpret_cast<double2*>(o + (size_t)col[c] * 32);
                        v[0] = make_double2(NM1 ? n_minus_1_of(q[c], ope2) : q[c], d0);
                        v[1] = make_double2(d1, d2);
                    } else {
                        const float c0 = NM1 ? n_minus_1_f32((float)raw[c], xs, q[c], ope2) : (float)q[c];
                        *reinterpret_cast<float4*>(o + (size_t)col[c] * 16) =
                            make_float4(c0, (float)d0, (float)d1, (float)d2);
                    }
                }
                prev[c] = q[c];
                q[c] = next;
                raw[c] = next_raw[c];
            }
            o += (size_t)plane * (F64OUT ? 32 : 16);
        }
    }
    if constexpr (RANGE) {
        unsigned long long a = 0ull, b = 0ull;
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
            const bool nan = lo[c] != lo[c] || hi[c] != hi[c];
            if (mine[c]) {
                a = max(a, nan ? ~0ull : order_key((double)hi[c]));
                b = max(b, nan ? ~0ull : order_key(-(double)lo[c]));
            }
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            a = max(a, __shfl_xor_sync(0xffffffffu, a, s));
            b = max(b, __shfl_xor_sync(0xffffffffu, b, s));
        }
        // few warps raise the running maxima: most see at once that they need not
        if ((t & 31) == 0) {
            if (a > *reinterpret_cast<volatile unsigned long long*>(range)) atomicMax(range, a);
            if (b > *reinterpret_cast<volatile unsigned long long*>(range + 1)) atomicMax(range + 1, b);
        }
    }
}

template <class P>
__global__ void __launch_bounds__(256) sample_kernel(const void* __restrict__ grid, GridGeo g,
                                                     double o0, double o1, double o2,
                                                     double ih0, double ih1, double ih2,
                                                     const double* __restrict__ pts, long long n,
                                                     typename P::R* __restrict__ out) {
    using R = typename P::R;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const R px = (R)((pts[i] - o0) * ih0);
        const R py = (R)((pts[n + i] - o1) * ih1);
        const R pz = (R)((pts[2 * n + i] - o2) * ih2);
        typename P::V v;
        sample<P>(grid, g, px, py, pz, v);
        out[i] = v.x;
        out[n + i] = v.y;
        out[2 * n + i] = v.z;
        out[3 * n + i] = v.w;
    }
}

static int grid_blocks(long long work, int per_sm) {
    int sms = 148;
    if (device_sm_count(&sms) != SLOTH_OK) sms = 148;
    long long b = (work + 255) / 256;
    long long cap = (long long)sms * per_sm;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

template <bool F64OUT, bool NM1>
static int pack_impl(const SlothGridDesc* g, const void* ne, int ne_is_f64, double ne_scale, double ope2,
                     void* grid_out, unsigned long long* range, void* stream) {
    int rc = check_grid(g);
    if (rc) return rc;
    if (!ne || !grid_out) return SLOTH_ERR_NULL_POINTER;
    if (!(ne_scale > 0.0) || !std::isfinite(ne_scale)) return SLOTH_ERR_INVALID_ARGUMENT;
    if (NM1 && (!(ope2 > 0.0) || !std::isfinite(ope2))) return SLOTH_ERR_INVALID_ARGUMENT;
    if (((uintptr_t)grid_out & 15u) != 0 || ((uintptr_t)range & 7u) != 0) return SLOTH_ERR_MISALIGNED;
    if (((uintptr_t)ne & (ne_is_f64 ? 7u : 3u)) != 0) return SLOTH_ERR_MISALIGNED;
    int sms = 148;
    if ((rc = device_sm_count(&sms)) != SLOTH_OK) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    if (range) {
        const cudaError_t e = cudaMemsetAsync(range, 0, 2 * sizeof(unsigned long long), s);
        if (e != cudaSuccess) return cuda_status(e);
    }
    const GridGeo geo = make_geo(g);
    const unsigned tk = (unsigned)((g->n[2] + kTileK - 1) / kTileK), tj = (unsigned)((g->n[1] + kTileJ - 1) / kTileJ);
    // Planes per CTA: long walks read less border along i (2 planes per walk), and
    // eight CTAs per SM want something to do: 64 for large grids, fewer for small.
    const long long patches = (long long)tk * tj;
    int planes = 64;
    while (planes > 4 && patches * ((g->n[0] + planes - 1) / planes) < 8LL * sms) planes /= 2;
    const unsigned blocks = (unsigned)(patches * ((g->n[0] + planes - 1) / planes));
    const double x = ne_scale * ope2;
    const float xs = NM1 && x > 1e-36 && x < 1e36 ? (float)x : 0.0f;
    auto launch = [&](auto kernel, auto* src) {
        kernel<<<blocks, kPackThreads, 0, s>>>(src, grid_out, geo, ne_scale, ope2, xs, planes, tk, tj, range);
    };
    const double* n64 = (const double*)ne;
    const float* n32 = (const float*)ne;
    if (range)
        ne_is_f64 ? launch(pack_kernel<double, F64OUT, NM1, true>, n64) : launch(pack_kernel<float, F64OUT, NM1, true>, n32);
    else
        ne_is_f64 ? launch(pack_kernel<double, F64OUT, NM1, false>, n64) : launch(pack_kernel<float, F64OUT, NM1, false>, n32);
    note_launch();
    return cuda_status(cudaGetLastError());
}

template <class P>
static int sample_impl(const SlothGridDesc* g, const void* grid, const double* points, int64_t n,
                       typename P::R* out, void* stream) {
    int rc = check_grid(g);
    if (rc) return rc;
    if (n < 0) return SLOTH_ERR_INVALID_ARGUMENT;
    if (n == 0) return SLOTH_OK;
    if (!grid || !points || !out) return SLOTH_ERR_NULL_POINTER;
    if (((uintptr_t)grid & 15u) != 0) return SLOTH_ERR_MISALIGNED;
    const GridGeo geo = make_geo(g);
    cudaStream_t s = (cudaStream_t)stream;
    sample_kernel<P><<<grid_blocks(n, 8), 256, 0, s>>>(
        grid, geo, g->origin[0], g->origin[1], g->origin[2], 1.0 / g->spacing[0], 1.0 / g->spacing[1],
        1.0 / g->spacing[2], points, (long long)n, out);
    note_launch();
    return cuda_status(cudaGetLastError());
}

}  // namespace sloth

extern "C" {

size_t sloth_grid_bytes(const SlothGridDesc* g, int real_bytes) {
    if (sloth::check_grid(g) != SLOTH_OK) return 0;
    if (real_bytes != 4 && real_bytes != 8) return 0;
    return (size_t)g->n[0] * (size_t)g->n[1] * (size_t)g->n[2] * 4u * (size_t)real_bytes;
}

int sloth_grid_pack_f32(const SlothGridDesc* g, const void* ne, int ne_is_f64, double ne_scale,
                        void* grid_out, void* stream) {
    return sloth::pack_impl<false, false>(g, ne, ne_is_f64, ne_scale, 0.0, grid_out, nullptr, stream);
}

int sloth_grid_pack_f64(const SlothGridDesc* g, const void* ne, int ne_is_f64, double ne_scale,
                        void* grid_out, void* stream) {
    return sloth::pack_impl<true, false>(g, ne, ne_is_f64, ne_scale, 0.0, grid_out, nullptr, stream);
}

int sloth_grid_pack_trace_f32(const SlothGridDesc* g, const void* ne, int ne_is_f64, double ne_scale,
                              double ope_ratio2, void* grid_out, void* stream) {
    return sloth::pack_impl<false, true>(g, ne, ne_is_f64, ne_scale, ope_ratio2, grid_out, nullptr, stream);
}

int sloth_grid_pack_trace_f64(const SlothGridDesc* g, const void* ne, int ne_is_f64, double ne_scale,
                              double ope_ratio2, void* grid_out, void* stream) {
    return sloth::pack_impl<true, true>(g, ne, ne_is_f64, ne_scale, ope_ratio2, grid_out, nullptr, stream);
}

int sloth_grid_pack_range(const SlothGridDesc* g, const void* ne, int ne_is_f64, int out_is_f64, double ne_scale,
                          double ope_ratio2, void* grid_out, unsigned long long* range, void* stream) {
    if (!range) return SLOTH_ERR_NULL_POINTER;
    const bool trace = ope_ratio2 != 0.0;
    if (out_is_f64)
        return trace ? sloth::pack_impl<true, true>(g, ne, ne_is_f64, ne_scale, ope_ratio2, grid_out, range, stream)
                     : sloth::pack_impl<true, false>(g, ne, ne_is_f64, ne_scale, 0.0, grid_out, range, stream);
    return trace ? sloth::pack_impl<false, true>(g, ne, ne_is_f64, ne_scale, ope_ratio2, grid_out, range, stream)
                 : sloth::pack_impl<false, false>(g, ne, ne_is_f64, ne_scale, 0.0, grid_out, range, stream);
}

int sloth_sample_f32(const SlothGridDesc* g, const void* grid, const double* points, int64_t n,
                     float* out, void* stream) {
    return sloth::sample_impl<sloth::PolF32>(g, grid, points, n, out, stream);
}

int sloth_sample_f64(const SlothGridDesc* g, const void* grid, const double* points, int64_t n,
                     double* out, void* stream) {
    return sloth::sample_impl<sloth::PolF64>(g, grid, points, n, out, stream);
}

}  // extern "C"
