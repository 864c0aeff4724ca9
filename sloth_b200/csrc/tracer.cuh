// Device code shared by the tracer entry points (trace.cu) and the request
// server (server.cu): kernel arguments, samplers, the integration step, per-ray
// bookkeeping, the per-tile tracing loop and the Morton pre-pass.
//
// What the reference does (src/core/propagator.py):
//   dsdt (:168-243): ds/dt = (v, grad(G)(r) [, kappa(r)]), G = -c^2/2 * ne/nc,
//                    grad(G) from precomputed grids through the trilinear
//                    interpolator (fill 0 outside the grid);
//   solve / trace_and_save_depths (:723-793, :1159-1198): vmap of a diffrax
//                    solve from t = 0 to the save times; output through
//                    ray_to_Jonesvector (src/shared/propagation.py:4-90).
// What runs here: the same ODE with a fixed-step fourth-order Runge-Kutta-
// Nystrom method in scaled units (grid cells, cells per step; see rkn_step),
// one thread per ray, plus the optical phase integral of omega*(n - 1) with
// n - 1 interpolated from the trace layout's channel 0, as the legacy solver
// interpolates its n grid (src/legacy/full_solver.py:289, :341-347), and the
// inverse-bremsstrahlung optical depth, both as Simpson quadratures of the
// stage values, and the Jones-vector projection at each save.
//
// Grid faces: the RHS jumps to the outside fill there. A step whose
// straight-line prediction p + w crosses a face is cut to end on it (a step
// of a fraction phi) and the ray then leaves on a straight line; a
// step whose prediction ends within kFaceMargin cells of a face, or is cut,
// samples its stage points clamped into the grid, i.e. it integrates the
// field's limit from inside, so that no stage sits on the discontinuity.
//
// Launch structure (all on the caller's stream):
//   1. keys_kernel   : Morton key of each ray's entry cell + bucket histogram
//   2. scan_kernel   : exclusive scan of the bucket counts
//   3. scatter_kernel: ray ids into bucket order
//   4. trace_kernel  : persistent CTAs of one or two warps; each warp traces 32
//                      neighbouring rays of the bucket order, one thread per
//                      ray, and refills finished lanes from the queue with one
//                      warp ballot + one atomic (see trace_warp).
#pragma once

#include <climits>
#include <cmath>
#include <type_traits>

#include "common.cuh"

namespace sloth {

constexpr int kThreads = 64;     // threads of the largest tracing CTA
constexpr int kWarpsPerSm = 16;  // FP32 tracing warps per SM, at 128 registers
constexpr int kRefill = 28;      // idle lanes that a warp refills together
constexpr double kFaceMargin = 0.02;     // cells

// Inverse-bremsstrahlung modes of the tracer.
enum { IB_OFF = 0, IB_SUBCRITICAL = 1, IB_GENERAL = 2 };

// Integration methods (SlothTraceParams::integrator): Nystrom's fourth-order
// Runge-Kutta-Nystrom step (3 field samples) or the classical RK4 step of
// the first-order system (4 samples).
enum { INTEG_RKN = SLOTH_INTEGRATOR_RKN, INTEG_RK4 = SLOTH_INTEGRATOR_RK4 };

// How a step samples its stage points: PLAIN tests each point against the
// grid (fill 0 outside); CLAMP moves it into the grid first (steps at a
// face); INTERIOR skips the test, for steps whose stage points are known to
// lie inside (see interior_bound_ok). Every mode clamps the cell index into
// the grid, so no mode can read outside the grid.
enum { SAMPLE_PLAIN = 0, SAMPLE_CLAMP = 1, SAMPLE_INTERIOR = 2 };

// Largest |acceleration| (cells per step^2) for which an interior step
// (ray inside, prediction p + w at least kFaceMargin inside on every axis)
// has every stage point inside: the stages sit at p + w/2 + A1/8 and
// p + w + A2/2, at least kFaceMargin/2 and kFaceMargin from the faces before
// the A terms, so |A| <= min(8 * kFaceMargin/2, 2 * kFaceMargin) = 0.04
// suffices; 0.03 keeps headroom for rounding.
constexpr double kInteriorAccel = 0.03;

// ---------------------------------------------------------------------------
// Kernel arguments.
// ---------------------------------------------------------------------------
struct TraceArgs {
    GridGeo geo;
    const void* grid;
    const void* rays;          // (6, N) of R
    long long n;
    const unsigned* perm;      // bucket-ordered ray ids
    unsigned* queue;           // rays handed out beyond each warp's first ones
    unsigned sa, s1, s2;       // voxel strides along the probing axis and the transverse axes t1, t2
    unsigned ahead_max;        // last voxel at which a fetched face may start
    double origin[3], spacing[3];
    double w_of_v[3];          // w = v * w_of_v   (cells per step per m/s)
    double v_of_w[3];          // v = w * v_of_w
    double S[3];               // -(dtau/h)^2 / 2
    double S4[3], S2[3], S6[3];     // S/4, S/2, S/6: the FP64 unit step's coefficients
    float Sf[3];               // S rounded to FP32 once here (the FP32 tracer reads these
                               // instead of converting the doubles inside its loop)
    float S4f[3], S2f[3], S6f[3];   // Sf/4, Sf/2 and fl(1/6)*Sf in FP32: the paired RKN step's
                                    // unit-step coefficients with S folded in
    float ope2f, cl_lof, cl_wf;
    float inv_ope2f;           // 1 / ope2 (q from x = ope2 * q)
    float accel_bound;         // bound on |acceleration| (cells per step^2), 0 when unknown
                               // (see interior_run and interior_sampling_ok)
    double phase_scale;        // (omega/c) * dtau / 6
    double tau_scale;          // kappa_q2 * dtau / 6
    double cl_w, cl_lo;        // Coulomb log below nc, and max(2, cl_w)
    double ope2;               // (omega_pe/omega)^2 per unit q
    double inv_ope2;
    double plane;
    int first_save, save_every, n_saves;
    int axis, t1, t2;
    int project;
    void* jones;
    void* state;
    double* phase;
    void* amp;
    uint8_t* status;
    int32_t* steps;
    unsigned long long* total_steps;
};

// Scalar parameters in the tracer's precision (FP32 copies made on the host).
template <class R> __device__ __forceinline__ R arg_ope2(const TraceArgs& a) {
    if constexpr (sizeof(R) == 4) return a.ope2f; else return a.ope2;
}
template <class R> __device__ __forceinline__ R arg_cl_lo(const TraceArgs& a) {
    if constexpr (sizeof(R) == 4) return a.cl_lof; else return a.cl_lo;
}
template <class R> __device__ __forceinline__ R arg_cl_w(const TraceArgs& a) {
    if constexpr (sizeof(R) == 4) return a.cl_wf; else return a.cl_w;
}
template <class R> __device__ __forceinline__ R arg_inv_ope2(const TraceArgs& a) {
    if constexpr (sizeof(R) == 4) return a.inv_ope2f; else return a.inv_ope2;
}

__device__ __forceinline__ double sel3(const double (&v)[3], int i) {
    return i == 0 ? v[0] : (i == 1 ? v[1] : v[2]);
}

template <class P>
struct Ray {
    typename P::Acc p[3];      // position (cells)
    typename P::Acc w[3];      // velocity (cells per step)
    typename P::Acc tau;       // sum of kappa stage combinations
    double ph;                 // sum of (n-1) stage combinations
    double lag;                // steps between the ray's time and `step` after an exit step
    int step, save_j, next_save;
    int run;                   // steps ahead that are certainly interior steps (fast path)
    unsigned id;
    bool exited;               // left the grid through a face-clipped step
};

// One field sample: n - 1 (the trace layout's channel 0), the three gradient
// channels and the inverse-bremsstrahlung rate per kappa_q2.
template <class P>
struct Sample {
    typename P::R n1, g0, g1, g2, k;
};

// The cell cache: the last cell as trilinear polynomials in the in-cell
// coordinates (fx, fy, fz), kept across stages and steps. Per channel T = a +
// bx fx + by fy + bz fz + cxy fx fy + cxz fx fz + cyz fy fz + cxyz fx fy fz,
// channels n - 1, dq/du, dq/dv, dq/dw in registers and the inverse-
// bremsstrahlung corner rate in shared memory (see kappa_store): seven
// multiply-adds per channel and sample. In FP64 the eight corners with the
// weights rebuilt at each sample (about 79 FP64 operations with the rate against 35)
// took 5.80 ms for 256^3 / 4e5 rays, the polynomials 4.53 ms.
struct CellPolyD {
    unsigned base;
    double t[4][8];
};

template <class R>
__device__ __forceinline__ void poly_coeffs(R (&t)[8], R v0, R v1, R v2, R v3, R v4, R v5, R v6, R v7) {
    // corner index = 4*dx + 2*dy + dz
    const R bz = v1 - v0, by = v2 - v0, bx = v4 - v0;
    const R dyz = v3 - v2, dxz = v5 - v4, dxy = v6 - v4;
    t[0] = v0;
    t[1] = bx;
    t[2] = by;
    t[3] = bz;
    t[4] = dxy - by;                       // cxy
    t[5] = dxz - bz;                       // cxz
    t[6] = dyz - bz;                       // cyz
    t[7] = ((v7 - v6) - dxz) - (dyz - bz); // cxyz
}

__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

template <class R>
__device__ __forceinline__ R poly_eval(const R (&t)[8], R fx, R fy, R fz) {
    // explicit fused multiply-adds: every kernel that inlines this rounds alike
    const R cz = fma_rn(fy, fma_rn(fx, t[7], t[6]), fma_rn(fx, t[5], t[3]));   // coefficient of fz
    const R cy = fma_rn(fx, t[4], t[2]);                                         // of fy (without fz)
    return fma_rn(fz, cz, fma_rn(fy, cy, fma_rn(fx, t[1], t[0])));
}

// FP32 cell cache on paired instructions. The packed voxel is a float4
// (q, dq/du, dq/dv, dq/dw), so (q, dq/du) and (dq/dv, dq/dw) arrive in
// register pairs; each pair of trilinear polynomials is built and evaluated
// with sm_100's two-wide FP32 instructions (__fadd2/__ffma2: one instruction
// for two channels, each component rounded exactly as the scalar operation).
// The inverse-bremsstrahlung channel stays scalar.
struct CellPolyF2 {
    unsigned base;
    float2 t[2][8];
};

// The same with the next cell along the probing axis fetched ahead (see
// cell_fill).
struct CellAheadF2 : CellPolyF2 {
    unsigned pred;      // the cell whose far face is on its way
    unsigned slot;      // byte offset of the cell's near face in s_face
};

// The cell's kappa polynomial stays in shared memory rather than registers:
// each thread owns one slot, [2][threads] float4 (FP64: [4][threads] double2) so
// that a warp's 16-byte loads do not conflict. This keeps 8 values out of the
// step's register budget; the coefficients are written once per cell and
// read once per stage, off the step's critical path.
static __shared__ float4 s_kappa_coef[2][kThreads];
static __shared__ double2 s_kappa_coefd[4][kThreads];

__device__ __forceinline__ void kappa_store(const float (&k)[8]) {
    s_kappa_coef[0][threadIdx.x] = make_float4(k[0], k[1], k[2], k[3]);
    s_kappa_coef[1][threadIdx.x] = make_float4(k[4], k[5], k[6], k[7]);
}

__device__ __forceinline__ void kappa_store(const double (&k)[8]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) s_kappa_coefd[i][threadIdx.x] = make_double2(k[2 * i], k[2 * i + 1]);
}

__device__ __forceinline__ float kappa_eval(float fx, float fy, float fz) {
    const float4 a = s_kappa_coef[0][threadIdx.x], b = s_kappa_coef[1][threadIdx.x];
    const float k[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    return poly_eval<float>(k, fx, fy, fz);
}

__device__ __forceinline__ double kappa_eval(double fx, double fy, double fz) {
    double k[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double2 v = s_kappa_coefd[i][threadIdx.x];
        k[2 * i] = v.x;
        k[2 * i + 1] = v.y;
    }
    return poly_eval<double>(k, fx, fy, fz);
}

__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);          // a - b, one rounding
}

__device__ __forceinline__ void poly_coeffs2(float2 (&t)[8], float2 v0, float2 v1, float2 v2, float2 v3, float2 v4,
                                             float2 v5, float2 v6, float2 v7) {
    const float2 bz = sub2(v1, v0), by = sub2(v2, v0), bx = sub2(v4, v0);
    const float2 dyz = sub2(v3, v2), dxz = sub2(v5, v4), dxy = sub2(v6, v4);
    t[0] = v0;
    t[1] = bx;
    t[2] = by;
    t[3] = bz;
    t[4] = sub2(dxy, by);
    t[5] = sub2(dxz, bz);
    t[6] = sub2(dyz, bz);
    t[7] = sub2(sub2(sub2(v7, v6), dxz), sub2(dyz, bz));
}

__device__ __forceinline__ float2 poly_eval2(const float2 (&t)[8], float2 fx, float2 fy, float2 fz) {
    const float2 cz = __ffma2_rn(fy, __ffma2_rn(fx, t[7], t[6]), __ffma2_rn(fx, t[5], t[3]));
    const float2 cy = __ffma2_rn(fx, t[4], t[2]);
    return __ffma2_rn(fz, cz, __ffma2_rn(fy, cy, __ffma2_rn(fx, t[1], t[0])));
}

// x = (omega_pe/omega)^2 of a grid point from its n - 1 (the trace layout):
// n - 1 = sqrt(1 - x) - 1 gives x = -(n - 1)(2 + (n - 1)) up to the critical
// density (n - 1 >= -1), and the layout stores -x above it.
template <class R>
__device__ __forceinline__ R x_of_n1(R n1) {
    if constexpr (sizeof(R) == 4)
        return n1 >= -1.0f ? -__fmul_rn(n1, __fadd_rn(2.0f, n1)) : -n1;
    else
        return n1 >= -1.0 ? -__dmul_rn(n1, __dadd_rn(2.0, n1)) : -n1;
}

// Inverse-bremsstrahlung rate of one grid point per kappa_q2: q^2 * CL(q),
// CL = max(2, cl_w - ln(max(omega_pe/omega, 1))) (src/core/propagator.py:155-162),
// with q rebuilt from the point's n - 1.
template <class P>
__device__ __forceinline__ typename P::R corner_kappa(const TraceArgs& a, typename P::R n1) {
    using R = typename P::R;
    const R x = x_of_n1<R>(n1);
    const R q = x * arg_inv_ope2<R>(a);
    const R cl = (x > R(1)) ? fmax(R(2), arg_cl_w<R>(a) - R(0.5) * P::log_(x)) : arg_cl_lo<R>(a);
    return q * q * cl;
}

// Below the critical density the rate is kappa_q2 * CL * q^2 with a constant
// CL, so the sub-critical corners carry x^2 = (ope2 * q)^2 and the optical
// depth's scale the constant factor cl_lo / ope2^2.
template <class R>
__device__ __forceinline__ R corner_x2(R n1) {
    const R x = x_of_n1<R>(n1);
    if constexpr (sizeof(R) == 4) return __fmul_rn(x, x); else return __dmul_rn(x, x);
}

// The paired cache's polynomials from a cell's corners (index 4*dx + 2*dy + dz),
// two channels per instruction.
template <int IB>
__device__ __forceinline__ void paired_coeffs(const TraceArgs& a, CellPolyF2& cc, float4 v0, float4 v1, float4 v2,
                                              float4 v3, float4 v4, float4 v5, float4 v6, float4 v7) {
#define SLOTH_LO(v) make_float2(v.x, v.y)
#define SLOTH_HI(v) make_float2(v.z, v.w)
    poly_coeffs2(cc.t[0], SLOTH_LO(v0), SLOTH_LO(v1), SLOTH_LO(v2), SLOTH_LO(v3), SLOTH_LO(v4), SLOTH_LO(v5),
                 SLOTH_LO(v6), SLOTH_LO(v7));
    poly_coeffs2(cc.t[1], SLOTH_HI(v0), SLOTH_HI(v1), SLOTH_HI(v2), SLOTH_HI(v3), SLOTH_HI(v4), SLOTH_HI(v5),
                 SLOTH_HI(v6), SLOTH_HI(v7));
#undef SLOTH_LO
#undef SLOTH_HI
    if constexpr (IB == IB_SUBCRITICAL) {
        float k[8];
        poly_coeffs<float>(k, corner_x2(v0.x), corner_x2(v1.x), corner_x2(v2.x), corner_x2(v3.x), corner_x2(v4.x),
                           corner_x2(v5.x), corner_x2(v6.x), corner_x2(v7.x));
        kappa_store(k);
    } else if constexpr (IB == IB_GENERAL) {
        float k[8];
        poly_coeffs<float>(k, corner_kappa<PolF32>(a, v0.x), corner_kappa<PolF32>(a, v1.x), corner_kappa<PolF32>(a, v2.x),
                           corner_kappa<PolF32>(a, v3.x), corner_kappa<PolF32>(a, v4.x), corner_kappa<PolF32>(a, v5.x),
                           corner_kappa<PolF32>(a, v6.x), corner_kappa<PolF32>(a, v7.x));
        kappa_store(k);
    }
}

// A corner of the packed grid. The 256-byte hint has L2 fetch the neighbouring
// 128 bytes (eight voxels further along z) from memory with a missing line: 512^3 / 1e7
// rays 105.0 -> 104.0 ms, 3e5 rays 4.53 -> 4.38 ms, 192^3 / 8e4 755 -> 741 us.
__device__ __forceinline__ float4 load_corner(const float4* p) {
    float4 v;
    asm("ld.global.nc.L2::256B.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// Loads cell b into the paired cache.
template <int IB>
__device__ __forceinline__ void cell_fill(const TraceArgs& a, unsigned b, CellPolyF2& cc) {
    const GridGeo& g = a.geo;
    const float4* gp = reinterpret_cast<const float4*>(a.grid) + b;
    cc.base = b;
    paired_coeffs<IB>(a, cc, load_corner(gp), load_corner(gp + 1u), load_corner(gp + g.sy), load_corner(gp + g.sy + 1u),
                      load_corner(gp + g.sx), load_corner(gp + g.sx + 1u), load_corner(gp + g.sx + g.sy),
                      load_corner(gp + g.sx + g.sy + 1u));
}

// Faces of cells across the probing axis in shared memory: a ring of three per
// thread, four corners each, [face][corner][lane] so that a warp's 16-byte accesses do not
// conflict. Corner 2*d1 + d2 sits d1, d2 points along the transverse axes.
constexpr unsigned kFaceRow = 32u * 16u, kFaceBytes = 4u * kFaceRow;
static __shared__ float4 s_face[3][4][32];

__device__ __forceinline__ unsigned face_after(unsigned f) { return f == 2u * kFaceBytes ? 0u : f + kFaceBytes; }

__device__ __forceinline__ void fetch_face(unsigned to, const float4* from, const TraceArgs& a) {
    auto copy = [](unsigned d, const float4* p) {
        asm volatile("cp.async.ca.shared.global.L2::256B [%0], [%1], 16;" ::"r"(d), "l"(p) : "memory");
    };
    copy(to, from);
    copy(to + kFaceRow, from + a.s2);
    copy(to + 2u * kFaceRow, from + a.s1);
    copy(to + 3u * kFaceRow, from + a.s1 + a.s2);
}

__device__ __forceinline__ float4 face_corner(unsigned at) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}

// Waits for this thread's copies; the last prefetched face may still be on its
// way when its warp runs out of rays.
__device__ __forceinline__ void fetch_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The fill of kernels whose warps wait for memory rather than for issue slots:
// a ray mostly moves on to the next cell along the probing axis, whose near face is
// this cell's far face, so each fill asks for the far face after that one and
// finds its own, asked for about two steps earlier, in shared memory. Any other
// cell's two faces are fetched now. The same corners, so bitwise the same rays.
template <int IB>
__device__ __forceinline__ void cell_fill(const TraceArgs& a, unsigned b, CellAheadF2& cc) {
    const float4* gp = reinterpret_cast<const float4*>(a.grid);
    const unsigned own = (unsigned)__cvta_generic_to_shared(&s_face[0][0][threadIdx.x & 31]);
    unsigned near = cc.slot;
    if (b == cc.pred) {
        near = face_after(near);
    } else {
        fetch_face(own + near, gp + b, a);
        fetch_face(own + face_after(near), gp + b + a.sa, a);
    }
    const unsigned far = face_after(near);
    fetch_wait();
    const unsigned along = far - near;       // modulo 2^32
    const unsigned dx = a.axis == 0 ? along : 2u * kFaceRow;
    const unsigned dy = a.axis == 1 ? along : (a.axis == 0 ? 2u * kFaceRow : kFaceRow);
    const unsigned dz = a.axis == 2 ? along : kFaceRow;
    const unsigned at = own + near;
    const float4 v0 = face_corner(at), v1 = face_corner(at + dz), v2 = face_corner(at + dy), v3 = face_corner(at + dy + dz);
    const float4 v4 = face_corner(at + dx), v5 = face_corner(at + dx + dz), v6 = face_corner(at + dx + dy),
                 v7 = face_corner(at + dx + dy + dz);
    // clamped into the grid: beyond it there is no cell that would use the face
    fetch_face(own + face_after(far), gp + min(b + 2u * a.sa, a.ahead_max), a);
    cc.base = b;
    cc.pred = b + a.sa;
    cc.slot = near;
    paired_coeffs<IB>(a, cc, v0, v1, v2, v3, v4, v5, v6, v7);
}

// FP64 trilinear sample of the packed grid (rules of src/core/interpolator.py:79-104:
// cell i = floor(p) clamped to [0, n-2], product weights, fill 0 outside)
// returning q, the three gradient channels and, when IB, the interpolated
// inverse-bremsstrahlung rate per kappa_q2. The reference interpolates a
// kappa grid computed at the grid points (src/core/propagator.py:239,
// :623-631); with uniform Te and Z that grid is q^2 * CL(q) per point, so its
// interpolant is the weighted sum of the corner values, formed here from the
// corners already loaded (CL is constant below the critical density).
//
// CLAMP moves the point into the grid first. (The stages of FP32 pass a running
// position and a small offset instead, see sample_f2.)
template <int IB, int MODE>
__device__ __forceinline__ void sample_d(const TraceArgs& a, const double (&at)[3], Sample<PolF64>& out, CellPolyD& cc) {
    using P = PolF64;
    using R = double;
    using V = typename P::V;
    const GridGeo& g = a.geo;
    double p[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        p[x] = at[x];
        if constexpr (MODE == SAMPLE_CLAMP) p[x] = fmin(fmax(p[x], 0.0), g.limd[x]);
    }
    int ix, iy, iz;
    if constexpr (MODE != SAMPLE_INTERIOR) {
        const bool in = (p[0] >= 0.0) & (p[0] <= g.limd[0]) & (p[1] >= 0.0) & (p[1] <= g.limd[1]) & (p[2] >= 0.0) &
                        (p[2] <= g.limd[2]);
        if (!in) {
            out.n1 = out.g0 = out.g1 = out.g2 = out.k = 0.0;
            return;
        }
        ix = min((int)p[0], g.n[0] - 2);
        iy = min((int)p[1], g.n[1] - 2);
        iz = min((int)p[2], g.n[2] - 2);
    } else {
        // one unsigned min clamps both ends (a negative index wraps to a large value)
        ix = (int)min((unsigned)(int)p[0], (unsigned)(g.n[0] - 2));
        iy = (int)min((unsigned)(int)p[1], (unsigned)(g.n[1] - 2));
        iz = (int)min((unsigned)(int)p[2], (unsigned)(g.n[2] - 2));
    }
    const double fx = p[0] - (double)ix, fy = p[1] - (double)iy, fz = p[2] - (double)iz;
    const unsigned b = (unsigned)ix * g.sx + (unsigned)iy * g.sy + (unsigned)iz;
    if (b != cc.base) {
        cc.base = b;
        const V v0 = P::load(a.grid, b), v1 = P::load(a.grid, b + 1u);
        const V v2 = P::load(a.grid, b + g.sy), v3 = P::load(a.grid, b + g.sy + 1u);
        const V v4 = P::load(a.grid, b + g.sx), v5 = P::load(a.grid, b + g.sx + 1u);
        const V v6 = P::load(a.grid, b + g.sx + g.sy), v7 = P::load(a.grid, b + g.sx + g.sy + 1u);
        poly_coeffs<R>(cc.t[0], v0.x, v1.x, v2.x, v3.x, v4.x, v5.x, v6.x, v7.x);
        poly_coeffs<R>(cc.t[1], v0.y, v1.y, v2.y, v3.y, v4.y, v5.y, v6.y, v7.y);
        poly_coeffs<R>(cc.t[2], v0.z, v1.z, v2.z, v3.z, v4.z, v5.z, v6.z, v7.z);
        poly_coeffs<R>(cc.t[3], v0.w, v1.w, v2.w, v3.w, v4.w, v5.w, v6.w, v7.w);
        if constexpr (IB == IB_SUBCRITICAL) {
            R k[8];
            poly_coeffs<R>(k, corner_x2(v0.x), corner_x2(v1.x), corner_x2(v2.x), corner_x2(v3.x), corner_x2(v4.x),
                           corner_x2(v5.x), corner_x2(v6.x), corner_x2(v7.x));
            kappa_store(k);
        } else if constexpr (IB == IB_GENERAL) {
            R k[8];
            poly_coeffs<R>(k, corner_kappa<P>(a, v0.x), corner_kappa<P>(a, v1.x), corner_kappa<P>(a, v2.x),
                           corner_kappa<P>(a, v3.x), corner_kappa<P>(a, v4.x), corner_kappa<P>(a, v5.x),
                           corner_kappa<P>(a, v6.x), corner_kappa<P>(a, v7.x));
            kappa_store(k);
        }
    }
    out.n1 = poly_eval<R>(cc.t[0], fx, fy, fz);
    out.g0 = poly_eval<R>(cc.t[1], fx, fy, fz);
    out.g1 = poly_eval<R>(cc.t[2], fx, fy, fz);
    out.g2 = poly_eval<R>(cc.t[3], fx, fy, fz);
    if constexpr (IB != IB_OFF) out.k = kappa_eval(fx, fy, fz);   // sub-critical: cl_lo / ope2^2 is in tau_scale
    else out.k = R(0);
}

// One step of length phi (in steps; phi = 1 except for a step cut at a grid
// face) in scaled units; see the file header. The ray equation is second
// order with a position-only force, p'' = A(p), and the phase and optical
// depth integrate functions of the position only, so the step is Nystrom's
// fourth-order Runge-Kutta-Nystrom method, three samples of the field instead
// of RK4's four:
//   stage points p, p + phi*w/2 + phi^2 A1/8, p + phi*w + phi^2 A2/2,
//   p' = p + phi*w + phi^2 (A1 + 2 A2)/6,  w' = w + phi (A1 + 4 A2 + A3)/6,
// and the phase and depth take Simpson's weights (1, 4, 1)/6 on the stages.
// The position and velocity are fourth order; the two integrals are third
// order in the step (their middle stage point is second order), an error
// many orders below the FP32 rounding here. Stage sums are accumulated as the
// stages are produced to keep few values live.
// The phase integrand n - 1 is interpolated from the trace layout's channel 0
// (the legacy solver's interpolated n, src/legacy/full_solver.py:289, :342-345).
// FP64: S multiplies the step's coefficients, not every stage's gradient; unit
// steps (UNIT, phi = 1) read them from the arguments. The position is one FP64
// number, so a stage samples at its point (the FP32 step's sum of a running position and
// a small offset buys nothing here). 256^3 / 4e5 rays: 4.54 -> 4.16 ms, RK4 6.68 -> 6.19.
template <int IB, int MODE, bool UNIT>
__device__ __forceinline__ void rkn_step_d(const TraceArgs& a, Ray<PolF64>& r, CellPolyD& cc, double phi) {
    if constexpr (UNIT) phi = 1.0;
    double k4[3], k2[3], k6[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        k4[x] = UNIT ? a.S4[x] : 0.25 * phi * a.S[x];
        k2[x] = UNIT ? a.S2[x] : 0.5 * phi * a.S[x];
        k6[x] = UNIT ? a.S6[x] : phi * (1.0 / 6.0) * a.S[x];
    }
    double p[3], w[3], gA[3], gW[3], st[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        p[x] = r.p[x].s;
        w[x] = r.w[x].s;
    }
    Sample<PolF64> s;
    sample_d<IB, MODE>(a, p, s, cc);
    double g = s.n1, kq = s.k;
    {
        const double G[3] = {s.g0, s.g1, s.g2};
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            gA[x] = gW[x] = G[x];
            st[x] = p[x] + 0.5 * phi * (w[x] + k4[x] * G[x]);     // p + phi*w/2 + phi^2 A1/8
        }
    }
    sample_d<IB, MODE>(a, st, s, cc);
    {
        const double G[3] = {s.g0, s.g1, s.g2};
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            gA[x] += 2.0 * G[x];
            gW[x] += 4.0 * G[x];
            st[x] = p[x] + phi * (w[x] + k2[x] * G[x]);             // p + phi*w + phi^2 A2/2
        }
    }
    g += 4.0 * s.n1;
    kq += 4.0 * s.k;
    sample_d<IB, MODE>(a, st, s, cc);
    gW[0] += s.g0; gW[1] += s.g1; gW[2] += s.g2;
    g += s.n1;
    kq += s.k;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        r.p[x].s = p[x] + phi * (w[x] + k6[x] * gA[x]);
        r.w[x].s = w[x] + k6[x] * gW[x];
    }
    r.ph += phi * g;
    if constexpr (IB != IB_OFF) r.tau.s += phi * kq;
}

// ---------------------------------------------------------------------------
// FP32 with the paired cell cache: the y and z components of every
// per-axis quantity of the step travel as one register pair and use sm_100's
// paired FP32 instructions (the cell polynomials already deliver dq/dv and
// dq/dw as a pair); x stays scalar. Each component is rounded exactly as the
// scalar step rounds it.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 bc2(float v) { return make_float2(v, v); }

// sample at (hx + lx, hyz + lyz)
template <int IB, int MODE, class Cache>
__device__ __forceinline__ void sample_f2(const TraceArgs& a, float hx, float lx, float2 hyz, float2 lyz,
                                          Sample<PolF32>& out, Cache& cc) {
    const GridGeo& g = a.geo;
    float px = hx + lx;
    float2 pyz = __fadd2_rn(hyz, lyz);
    if constexpr (MODE == SAMPLE_CLAMP) {
        const float cx = fminf(fmaxf(px, 0.0f), g.limf[0]);
        if (cx != px) { hx = cx; lx = 0.0f; px = cx; }
        const float cy = fminf(fmaxf(pyz.x, 0.0f), g.limf[1]);
        if (cy != pyz.x) { hyz.x = cy; lyz.x = 0.0f; pyz.x = cy; }
        const float cz = fminf(fmaxf(pyz.y, 0.0f), g.limf[2]);
        if (cz != pyz.y) { hyz.y = cz; lyz.y = 0.0f; pyz.y = cz; }
    }
    int ix, iy, iz;
    if constexpr (MODE != SAMPLE_INTERIOR) {
        const bool in = (px >= 0.0f) & (px <= g.limf[0]) & (pyz.x >= 0.0f) & (pyz.x <= g.limf[1]) &
                        (pyz.y >= 0.0f) & (pyz.y <= g.limf[2]);
        if (!in) {
            out.n1 = out.g0 = out.g1 = out.g2 = out.k = 0.0f;
            return;
        }
        ix = min((int)px, g.n[0] - 2);
        iy = min((int)pyz.x, g.n[1] - 2);
        iz = min((int)pyz.y, g.n[2] - 2);
    } else {
        ix = (int)min((unsigned)(int)px, (unsigned)(g.n[0] - 2));
        iy = (int)min((unsigned)(int)pyz.x, (unsigned)(g.n[1] - 2));
        iz = (int)min((unsigned)(int)pyz.y, (unsigned)(g.n[2] - 2));
    }
    const float fx = (hx - (float)ix) + lx;
    const float2 fyz = __fadd2_rn(__fadd2_rn(hyz, make_float2(-(float)iy, -(float)iz)), lyz);
    const unsigned b = (unsigned)ix * g.sx + (unsigned)iy * g.sy + (unsigned)iz;
    if (b != cc.base) cell_fill<IB>(a, b, cc);
    const float2 fx2 = bc2(fx), fy2 = bc2(fyz.x), fz2 = bc2(fyz.y);
    const float2 r0 = poly_eval2(cc.t[0], fx2, fy2, fz2);
    const float2 r1 = poly_eval2(cc.t[1], fx2, fy2, fz2);
    out.n1 = r0.x;
    out.g0 = r0.y;
    out.g1 = r1.x;
    out.g2 = r1.y;
    if constexpr (IB != IB_OFF) out.k = kappa_eval(fx, fyz.x, fyz.y);   // sub-critical: cl_lo / ope2^2 is in tau_scale
    else out.k = 0.0f;
}

// s + x with the compensation c (AccF::add on a pair)
__device__ __forceinline__ void kahan2(float2& s, float2& c, float2 x) {
    const float2 y = __fadd2_rn(x, c);
    const float2 t = __fadd2_rn(s, y);
    c = __fadd2_rn(y, __ffma2_rn(s, bc2(1.0f), make_float2(-t.x, -t.y)) );
    s = t;
}

// kahan2 of a * b, the product's rounding folded into the compensated add
__device__ __forceinline__ void kahan2_fma(float2& s, float2& c, float2 a, float2 b) {
    const float2 y = __ffma2_rn(a, b, c);
    const float2 t = __fadd2_rn(s, y);
    c = __fadd2_rn(y, __ffma2_rn(s, bc2(1.0f), make_float2(-t.x, -t.y)) );
    s = t;
}

// UNIT: phi is 1 (every step but a cut one); the multiplications by phi are
// left out, which gives bitwise the results of the general form at phi = 1
// (fma(1, a, b) rounds as a + b).
template <int IB, int MODE, bool UNIT, class Cache>
__device__ __forceinline__ void rkn_step_f2(const TraceArgs& a, Ray<PolF32>& r, Cache& cc, float phi) {
    if constexpr (UNIT) phi = 1.0f;
    auto mphi = [&](float x) { return UNIT ? x : __fmul_rn(phi, x); };
    auto mphi2 = [&](float2 x) { return UNIT ? x : __fmul2_rn(bc2(phi), x); };
    const float hphi = 0.5f * phi, phi6 = phi * (1.0f / 6.0f), phi2_6 = phi * phi6;
    const float phi2_2 = 0.5f * phi * phi;
    // The accelerations enter the step only through the stage points and the
    // two weighted sums, so S multiplies the step's coefficients rather than
    // every stage's gradient: k4 = phi S/4 and k2 = phi^2 S/2 (stage points,
    // p + (phi/2)(w + k4 G1) and p + phi w + k2 G2), k6 = phi^2 S/6 (position),
    // kw = phi S/6 (velocity). Unit steps read them from the arguments, formed
    // there exactly as here at phi = 1.
    float k4x, k2x, k6x, kwx;
    float2 k4yz, k2yz, k6yz, kwyz;
    if constexpr (UNIT) {
        k4x = a.S4f[0];
        k2x = a.S2f[0];
        k6x = kwx = a.S6f[0];
        k4yz = make_float2(a.S4f[1], a.S4f[2]);
        k2yz = make_float2(a.S2f[1], a.S2f[2]);
        k6yz = kwyz = make_float2(a.S6f[1], a.S6f[2]);
    } else {
        const float S0 = a.Sf[0];
        const float2 S12 = make_float2(a.Sf[1], a.Sf[2]);
        k4x = __fmul_rn(0.25f * phi, S0);
        k2x = __fmul_rn(phi2_2, S0);
        k6x = __fmul_rn(phi2_6, S0);
        kwx = __fmul_rn(phi6, S0);
        k4yz = __fmul2_rn(bc2(0.25f * phi), S12);
        k2yz = __fmul2_rn(bc2(phi2_2), S12);
        k6yz = __fmul2_rn(bc2(phi2_6), S12);
        kwyz = __fmul2_rn(bc2(phi6), S12);
    }
    const float2 hphi2 = bc2(hphi), phi22 = bc2(phi);
    // Every rounding is explicit (intrinsics), so that each kernel that
    // inlines this step (the tracer's and the server's) rounds alike.
    const float phx = r.p[0].s, plx = r.p[0].c, wex = r.w[0].s + r.w[0].c;
    const float2 phyz = make_float2(r.p[1].s, r.p[2].s), plyz = make_float2(r.p[1].c, r.p[2].c);
    const float2 weyz = __fadd2_rn(make_float2(r.w[1].s, r.w[2].s), make_float2(r.w[1].c, r.w[2].c));
    Sample<PolF32> s;
    // stage 1 at p; gA = g1 + 2 g2 and gW = g1 + 4 g2 + g3 are the gradient
    // sums (S applied in the coefficients)
    sample_f2<IB, MODE>(a, phx, plx, phyz, plyz, s, cc);
    float g = s.n1;
    float kq = s.k;
    float gAx = s.g0;
    float2 gAyz = make_float2(s.g1, s.g2);
    float gWx = gAx;
    float2 gWyz = gAyz;
    // stage 2 at p + phi*w/2 + phi^2 A1/8 = p + (phi/2)(w + k4 G1)
    float stx = __fmaf_rn(hphi, __fmaf_rn(k4x, gAx, wex), plx);
    float2 styz = __ffma2_rn(hphi2, __ffma2_rn(k4yz, gAyz, weyz), plyz);
    sample_f2<IB, MODE>(a, phx, stx, phyz, styz, s, cc);
    {
        const float Gx = s.g0;
        const float2 Gyz = make_float2(s.g1, s.g2);
        gAx = __fmaf_rn(2.0f, Gx, gAx);
        gAyz = __ffma2_rn(bc2(2.0f), Gyz, gAyz);
        gWx = __fmaf_rn(4.0f, Gx, gWx);
        gWyz = __ffma2_rn(bc2(4.0f), Gyz, gWyz);
        // stage 3 at p + phi*w + phi^2 A2/2
        stx = __fadd_rn(plx, __fmaf_rn(k2x, Gx, mphi(wex)));
        styz = __fadd2_rn(plyz, __ffma2_rn(k2yz, Gyz, mphi2(weyz)));
    }
    g = __fmaf_rn(4.0f, s.n1, g);
    kq = __fmaf_rn(4.0f, s.k, kq);
    sample_f2<IB, MODE>(a, phx, stx, phyz, styz, s, cc);
    gWx = __fadd_rn(gWx, s.g0);
    gWyz = __fadd2_rn(gWyz, make_float2(s.g1, s.g2));
    g = __fadd_rn(g, s.n1);
    kq = __fadd_rn(kq, s.k);
    // x: the scalar update
    if constexpr (UNIT)
        r.p[0].add(__fadd_rn(r.w[0].hi(), __fmaf_rn(k6x, gAx, r.w[0].lo())));
    else
        r.p[0].add(__fmaf_rn(phi, r.w[0].hi(), __fmaf_rn(k6x, gAx, __fmul_rn(phi, r.w[0].lo()))));
    r.w[0].add_fma(kwx, gWx);
    // y, z: the same update on pairs
    {
        const float2 whi = make_float2(r.w[1].s, r.w[2].s), wlo = make_float2(r.w[1].c, r.w[2].c);
        const float2 dp = UNIT ? __fadd2_rn(whi, __ffma2_rn(k6yz, gAyz, wlo))
                               : __ffma2_rn(phi22, whi, __ffma2_rn(k6yz, gAyz, __fmul2_rn(phi22, wlo)));
        float2 ps = phyz, pc = plyz;
        kahan2(ps, pc, dp);
        r.p[1].s = ps.x; r.p[2].s = ps.y; r.p[1].c = pc.x; r.p[2].c = pc.y;
        float2 ws = whi, wc = wlo;
        kahan2_fma(ws, wc, kwyz, gWyz);
        r.w[1].s = ws.x; r.w[2].s = ws.y; r.w[1].c = wc.x; r.w[2].c = wc.y;
    }
    r.ph += (double)mphi(g);
    if constexpr (IB != IB_OFF) r.tau.add(mphi(kq));
}

// One classical RK4 step of the first-order system (p, w)' = (w, A(p)) of
// length phi, four samples of the field (the integrator the workload
// descriptions name; INTEG_RK4):
//   stage points p, p + phi*w/2, p + phi*w2/2, p + phi*w3
//   with w2 = w + phi*A1/2, w3 = w + phi*A2/2;
//   p' = p + phi*w + phi^2 (A1 + A2 + A3)/6,  w' = w + phi (A1 + 2A2 + 2A3 + A4)/6,
// and the phase and depth take RK4's weights (1, 2, 2, 1)/6 on the stages.
// The stage points lie within phi^2 |A|/4 and phi^2 |A|/2 of the segment
// from p to p + phi*w, as the RKN step's do, so the interior-sampling bound
// kInteriorAccel and the interior-run envelope hold for both methods.
template <int IB, int MODE>
__device__ __forceinline__ void rk4_step_d(const TraceArgs& a, Ray<PolF64>& r, CellPolyD& cc, double phi) {
    const double hphi = 0.5 * phi;
    double p[3], w[3], gA[3], gW[3], w3[3], st[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        p[x] = r.p[x].s;
        w[x] = r.w[x].s;
    }
    Sample<PolF64> s;
    // stage 1 at p, stage 2 at p + phi*w/2
    sample_d<IB, MODE>(a, p, s, cc);
    double g = s.n1, kq = s.k;
    gA[0] = s.g0; gA[1] = s.g1; gA[2] = s.g2;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        gW[x] = gA[x];
        st[x] = p[x] + hphi * w[x];
    }
    sample_d<IB, MODE>(a, st, s, cc);
    {
        const double G[3] = {s.g0, s.g1, s.g2};
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            st[x] = p[x] + hphi * (w[x] + hphi * a.S[x] * gA[x]);    // p + phi*w2/2
            w3[x] = w[x] + hphi * a.S[x] * G[x];
            gA[x] += G[x];
            gW[x] += 2.0 * G[x];
        }
    }
    g += 2.0 * s.n1;
    kq += 2.0 * s.k;
    // stage 3 at p + phi*w2/2, stage 4 at p + phi*w3
    sample_d<IB, MODE>(a, st, s, cc);
    {
        const double G[3] = {s.g0, s.g1, s.g2};
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            gA[x] += G[x];
            gW[x] += 2.0 * G[x];
            st[x] = p[x] + phi * w3[x];
        }
    }
    g += 2.0 * s.n1;
    kq += 2.0 * s.k;
    sample_d<IB, MODE>(a, st, s, cc);
    gW[0] += s.g0; gW[1] += s.g1; gW[2] += s.g2;
    g += s.n1;
    kq += s.k;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const double k6 = phi * (1.0 / 6.0) * a.S[x];
        r.p[x].s = p[x] + phi * (w[x] + k6 * gA[x]);
        r.w[x].s = w[x] + k6 * gW[x];
    }
    r.ph += phi * g;
    if constexpr (IB != IB_OFF) r.tau.s += phi * kq;
}

// The RK4 step in the paired FP32 form (y and z components as register
// pairs), every rounding explicit.
template <int IB, int MODE, bool UNIT, class Cache>
__device__ __forceinline__ void rk4_step_f2(const TraceArgs& a, Ray<PolF32>& r, Cache& cc, float phi) {
    if constexpr (UNIT) phi = 1.0f;
    auto mphi = [&](float x) { return UNIT ? x : __fmul_rn(phi, x); };
    auto mphi2 = [&](float2 x) { return UNIT ? x : __fmul2_rn(bc2(phi), x); };
    const float hphi = 0.5f * phi, phi6 = phi * (1.0f / 6.0f), phi2_6 = phi * phi6;
    const float S0 = a.Sf[0];
    const float2 S12 = make_float2(a.Sf[1], a.Sf[2]);
    const float2 hphi2 = bc2(hphi), two2 = bc2(2.0f);
    const float phx = r.p[0].s, plx = r.p[0].c, wex = __fadd_rn(r.w[0].s, r.w[0].c);
    const float2 phyz = make_float2(r.p[1].s, r.p[2].s), plyz = make_float2(r.p[1].c, r.p[2].c);
    const float2 weyz = __fadd2_rn(make_float2(r.w[1].s, r.w[2].s), make_float2(r.w[1].c, r.w[2].c));
    Sample<PolF32> s;
    // stage 1 at p
    sample_f2<IB, MODE>(a, phx, plx, phyz, plyz, s, cc);
    float g = s.n1;
    float kq = s.k;
    float sAx = __fmul_rn(S0, s.g0);
    float2 sAyz = __fmul2_rn(S12, make_float2(s.g1, s.g2));
    float sWx = sAx;
    float2 sWyz = sAyz;
    // stage 2 at p + phi*w/2
    float stx = __fmaf_rn(hphi, wex, plx);
    float2 styz = __ffma2_rn(hphi2, weyz, plyz);
    sample_f2<IB, MODE>(a, phx, stx, phyz, styz, s, cc);
    stx = __fmaf_rn(hphi, __fmaf_rn(hphi, sAx, wex), plx);                 // p + phi*w2/2
    styz = __ffma2_rn(hphi2, __ffma2_rn(hphi2, sAyz, weyz), plyz);
    float w3x;
    float2 w3yz;
    {
        const float Ax = __fmul_rn(S0, s.g0);
        const float2 Ayz = __fmul2_rn(S12, make_float2(s.g1, s.g2));
        w3x = __fmaf_rn(hphi, Ax, wex);
        w3yz = __ffma2_rn(hphi2, Ayz, weyz);
        sAx = __fadd_rn(sAx, Ax);
        sAyz = __fadd2_rn(sAyz, Ayz);
        sWx = __fmaf_rn(2.0f, Ax, sWx);
        sWyz = __ffma2_rn(two2, Ayz, sWyz);
    }
    g = __fmaf_rn(2.0f, s.n1, g);
    kq = __fmaf_rn(2.0f, s.k, kq);
    // stage 3 at p + phi*w2/2
    sample_f2<IB, MODE>(a, phx, stx, phyz, styz, s, cc);
    {
        const float Ax = __fmul_rn(S0, s.g0);
        const float2 Ayz = __fmul2_rn(S12, make_float2(s.g1, s.g2));
        sAx = __fadd_rn(sAx, Ax);
        sAyz = __fadd2_rn(sAyz, Ayz);
        sWx = __fmaf_rn(2.0f, Ax, sWx);
        sWyz = __ffma2_rn(two2, Ayz, sWyz);
        stx = __fadd_rn(plx, mphi(w3x));
        styz = __fadd2_rn(plyz, mphi2(w3yz));
    }
    g = __fmaf_rn(2.0f, s.n1, g);
    kq = __fmaf_rn(2.0f, s.k, kq);
    // stage 4 at p + phi*w3
    sample_f2<IB, MODE>(a, phx, stx, phyz, styz, s, cc);
    sWx = __fmaf_rn(S0, s.g0, sWx);
    sWyz = __ffma2_rn(S12, make_float2(s.g1, s.g2), sWyz);
    g = __fadd_rn(g, s.n1);
    kq = __fadd_rn(kq, s.k);
    // x: the scalar update
    if constexpr (UNIT)
        r.p[0].add(__fadd_rn(r.w[0].hi(), __fadd_rn(r.w[0].lo(), __fmul_rn(phi2_6, sAx))));
    else
        r.p[0].add(__fmaf_rn(phi, r.w[0].hi(), __fmaf_rn(phi, r.w[0].lo(), __fmul_rn(phi2_6, sAx))));
    r.w[0].add(__fmul_rn(phi6, sWx));
    // y, z: the same update on pairs
    {
        const float2 phi2 = bc2(phi);
        const float2 whi = make_float2(r.w[1].s, r.w[2].s), wlo = make_float2(r.w[1].c, r.w[2].c);
        const float2 dp = UNIT ? __fadd2_rn(whi, __fadd2_rn(wlo, __fmul2_rn(bc2(phi2_6), sAyz)))
                               : __ffma2_rn(phi2, whi, __ffma2_rn(phi2, wlo, __fmul2_rn(bc2(phi2_6), sAyz)));
        float2 ps = phyz, pc = plyz;
        kahan2(ps, pc, dp);
        r.p[1].s = ps.x; r.p[2].s = ps.y; r.p[1].c = pc.x; r.p[2].c = pc.y;
        float2 ws = whi, wc = wlo;
        kahan2(ws, wc, __fmul2_rn(bc2(phi6), sWyz));
        r.w[1].s = ws.x; r.w[2].s = ws.y; r.w[1].c = wc.x; r.w[2].c = wc.y;
    }
    r.ph += (double)mphi(g);
    if constexpr (IB != IB_OFF) r.tau.add(mphi(kq));
}

// One step: the paired form in FP32, the plain one in FP64; RKN unless
// INTEG selects RK4.
template <class P, int IB, int MODE, bool UNIT = false, int INTEG = INTEG_RKN, class Cache>
__device__ __forceinline__ void step_any(const TraceArgs& a, Ray<P>& r, Cache& cc, typename P::R phi) {
    if constexpr (sizeof(typename P::R) == 4) {
        if constexpr (INTEG == INTEG_RK4) rk4_step_f2<IB, MODE, UNIT>(a, r, cc, phi);
        else rkn_step_f2<IB, MODE, UNIT>(a, r, cc, phi);
    } else {
        if constexpr (INTEG == INTEG_RK4) rk4_step_d<IB, MODE>(a, r, cc, phi);
        else rkn_step_d<IB, MODE, UNIT>(a, r, cc, phi);
    }
}

// Kind of the next step of a ray: 0 plain step of a ray inside the grid whose
// prediction stays more than kFaceMargin inside; 1 full step sampled with
// clamped stage points (its prediction ends within kFaceMargin of a face);
// 2 step cut at the face its prediction crosses, length phi, after which the
// ray leaves; 3 plain step of a ray outside the grid (zero RHS).
template <class P>
__device__ __forceinline__ int step_kind(const TraceArgs& a, const Ray<P>& r, typename P::R& phi) {
    using R = typename P::R;
    const R margin = R(kFaceMargin);
    R p[3], w[3];
    bool in = true;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        p[x] = r.p[x].val();
        w[x] = r.w[x].val();
        in = in & (p[x] >= R(0)) & (p[x] <= lim_of<R>(a.geo, x));
    }
    phi = R(1);
    if (!in) return 3;
    bool near = false;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const R pn = p[x] + w[x];
        const R lim = lim_of<R>(a.geo, x);
        if (pn > lim - margin) {
            near = true;
            // distance to the face from the compensated position
            if (pn > lim) phi = fmin(phi, ((lim - r.p[x].hi()) - r.p[x].lo()) / w[x]);
        }
        if (pn < margin) {
            near = true;
            if (pn < R(0)) phi = fmin(phi, (-r.p[x].hi() - r.p[x].lo()) / w[x]);
        }
    }
    phi = fmax(phi, R(0));
    return phi < R(1) ? 2 : (near ? 1 : 0);
}

// Number of steps after the current interior step (kind 0) that are certainly
// kind 0 too, for a trace whose accelerations are bounded by B =
// a.accel_bound: 127, 31, 7 or 0. From the state (p, w) now, after j steps
// |w_j - w| <= j B (each step adds a weighted mean of stage accelerations)
// and |p_j - p - j w| <= B j^2 / 2 (each step moves w_i + (A1 + A2 + A3) / 6),
// so the position p_j and the prediction p_j + w_j lie within
// B (j^2 / 2 + j) of the segment from p + w to p + (j + 1) w. If that segment,
// widened by the bound for j = m plus a rounding slack, keeps kFaceMargin from
// every face, the next m steps are interior steps, and step_kind need not run
// for them: the steps take the same path as with it, bit for bit.
template <class P>
__device__ __forceinline__ int interior_run(const TraceArgs& a, const Ray<P>& r) {
    using R = typename P::R;
    const R B = (R)a.accel_bound;
    const R margin = R(kFaceMargin) + R(0.25);       // face margin + rounding slack (cells)
    R p[3], w[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        p[x] = r.p[x].val();
        w[x] = r.w[x].val();
    }
    auto fits = [&](int m) {
        const R dev = margin + B * R(0.5 * m * m + m);
        bool ok = true;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            const R e1 = p[x] + w[x], e2 = p[x] + R(m + 1) * w[x];
            ok = ok & (fmin(e1, e2) >= dev) & (fmax(e1, e2) <= lim_of<R>(a.geo, x) - dev);
        }
        return ok;
    };
    if (fits(127)) return 127;
    if (fits(31)) return 31;
    if (fits(7)) return 7;
    return 0;
}

// Whether a trace's interior steps may sample without the grid test: its
// accelerations are bounded by kInteriorAccel (accel_bound carries 0.1% of
// headroom over the bound).
__host__ __device__ __forceinline__ bool interior_sampling_ok(const TraceArgs& a) {
    return a.accel_bound > 0.0f && a.accel_bound <= (float)(kInteriorAccel * 1.001);
}

template <class P>
__device__ __forceinline__ bool ray_in_grid(const TraceArgs& a, const Ray<P>& r) {
    using R = typename P::R;
    bool in = true;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const R p = r.p[x].val();
        in = in & (p >= R(0)) & (p <= lim_of<R>(a.geo, x));
    }
    return in;
}

// True once the ray is outside the grid on an axis and moving away from it
// on that axis: its path is then a straight line that never re-enters.
template <class P>
__device__ __forceinline__ bool ray_gone(const TraceArgs& a, const Ray<P>& r) {
    using R = typename P::R;
    bool gone = false;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const R p = r.p[x].val(), w = r.w[x].val();
        gone = gone | ((p < R(0)) & (w <= R(0))) | ((p > lim_of<R>(a.geo, x)) & (w >= R(0)));
    }
    return gone;
}

// Writes save j of ray `id` from its state (cells, cells per step, FP64)
// `drift` unit steps before the save time (drift > 0 only for rays that have
// left the grid for good, whose path is a straight line).
template <class R>
__device__ __forceinline__ void emit_save(const TraceArgs& a, unsigned id, int j, double drift,
                                       double p0, double p1, double p2, double w0, double w1,
                                       double w2, double ph, double tau) {
    double x[3], v[3];
    const double p[3] = {p0, p1, p2}, w[3] = {w0, w1, w2};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        x[k] = a.origin[k] + (p[k] + drift * w[k]) * a.spacing[k];
        v[k] = w[k] * a.v_of_w[k];
    }
    const double xa = sel3(x, a.axis), va = sel3(v, a.axis);
    const double x1 = sel3(x, a.t1), v1 = sel3(v, a.t1);
    const double x2 = sel3(x, a.t2), v2 = sel3(v, a.t2);
    double pos1 = x1, pos2 = x2;
    if (a.project) {
        const double tbp = (xa - a.plane) / va;
        pos1 = x1 - v1 * tbp;
        pos2 = x2 - v2 * tbp;
    }
    const size_t n = (size_t)a.n;
    R* jo = reinterpret_cast<R*>(a.jones) + (size_t)j * 4u * n;
    jo[id] = (R)pos1;
    jo[n + id] = (R)atan(v1 / va);
    jo[2 * n + id] = (R)pos2;
    jo[3 * n + id] = (R)atan(v2 / va);
    if (a.state) {
        R* so = reinterpret_cast<R*>(a.state) + (size_t)j * 6u * n;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            so[k * n + id] = (R)x[k];
            so[(3 + k) * n + id] = (R)v[k];
        }
    }
    if (a.phase) a.phase[(size_t)j * n + id] = ph * a.phase_scale;
    if (a.amp) reinterpret_cast<R*>(a.amp)[(size_t)j * n + id] = (R)exp(-tau * a.tau_scale);
}

template <class P>
__device__ __forceinline__ void emit(const TraceArgs& a, const Ray<P>& r, double drift) {
    emit_save<typename P::R>(a, r.id, r.save_j, drift, r.p[0].vald(), r.p[1].vald(), r.p[2].vald(),
                             r.w[0].vald(), r.w[1].vald(), r.w[2].vald(), r.ph, r.tau.vald());
}

template <class P>
__device__ __forceinline__ void finish_ray(const TraceArgs& a, const Ray<P>& r, uint8_t st,
                                           unsigned long long& my_steps) {
    bool finite = isfinite(r.ph);
#pragma unroll
    for (int k = 0; k < 3; ++k) finite = finite & isfinite(r.p[k].vald()) & isfinite(r.w[k].vald());
    if (!finite) st = SLOTH_RAY_NONFINITE;
    if (a.status) a.status[r.id] = st;
    if (a.steps) a.steps[r.id] = r.step;
    my_steps += (unsigned long long)r.step;
}

// Saves due at the current step, then the end / exit checks. Returns true
// while the ray still needs steps. `check_gone` is false after a plain step
// taken from inside the grid with its prediction more than kFaceMargin inside
// (the ray cannot have left); the outside test is skipped then.
//
// Most steps need nothing here, which the first test decides with integer
// compares. The rest goes through one loop with a single emit call site: a
// save due now is taken at the ray's time (lag), and a ray that has left
// the grid for good takes all its remaining saves by straight-line drift.
// (Two emit call sites with the same arguments let the compiler hoist their
// common part, the state's FP64 conversions and the Jones angles, into
// every step.)
template <class P>
__device__ __forceinline__ bool settle(const TraceArgs& a, Ray<P>& r, unsigned long long& my_steps,
                                      bool check_gone = true) {
    const bool leaving = r.exited || (check_gone && ray_gone<P>(a, r));
    if (r.next_save != r.step && !leaving) return true;
    while (r.save_j < a.n_saves) {
        const bool due = r.next_save == r.step;
        if (!due && !leaving) break;
        const double drift = due ? r.lag : (double)(r.next_save - r.step) + r.lag;
        emit<P>(a, r, drift);
        ++r.save_j;
        r.next_save += a.save_every;
    }
    if (r.save_j >= a.n_saves) {
        finish_ray<P>(a, r, (!r.exited && ray_in_grid<P>(a, r)) ? SLOTH_RAY_INSIDE_AT_END : SLOTH_RAY_EXITED,
                      my_steps);
        return false;
    }
    return true;
}

template <class P>
__device__ __forceinline__ bool start_ray(const TraceArgs& a, unsigned id, Ray<P>& r,
                                          unsigned long long& my_steps) {
    using R = typename P::R;
    const R* rays = reinterpret_cast<const R*>(a.rays);
    const size_t n = (size_t)a.n;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double x = (double)rays[k * n + id];
        const double v = (double)rays[(3 + k) * n + id];
        r.p[k].set((x - a.origin[k]) / a.spacing[k]);
        r.w[k].set(v * a.w_of_v[k]);
    }
    r.tau.set(0.0);
    r.ph = 0.0;
    r.lag = 0.0;
    r.exited = false;
    r.step = 0;
    r.save_j = 0;
    r.next_save = a.first_save;
    r.run = 0;
    r.id = id;
    return settle<P>(a, r, my_steps);
}

// Ray queue of a whole trace: each warp first takes rays of its own
// (`first` to `first_end`), then rays from the shared counter, which starts
// behind the first rays of all the warps.
struct TraceQueue {
    unsigned* counter;
    unsigned base0, first, first_end, n;
    __device__ __forceinline__ bool take(int k, int lane, unsigned& base, unsigned& end) {
        if (first < first_end) {
            base = first;
            end = first_end;
            first = first_end;
            return true;
        }
        unsigned b = 0;
        if (lane == 0) b = atomicAdd(counter, (unsigned)k);
        base = base0 + __shfl_sync(0xffffffffu, b, 0);
        end = min(base + (unsigned)k, n);
        return base + (unsigned)k < n;
    }
};

// A run of rays known in advance (a serving tile's share).
struct RangeQueue {
    unsigned head, n;
    __device__ __forceinline__ bool take(int k, int, unsigned& base, unsigned& end) {
        base = head;
        head += (unsigned)k;
        end = min(head, n);
        return head < n;
    }
};

// Traces the rays of a queue, one thread per ray of this warp. `q.take(k)`
// hands out up to k rays [base, end) of the bucket order and returns whether
// more may follow. Shared by the single-trace and serving kernels.
// Rays taken together start in neighbouring cells at the same place along the
// beam, so the warp's cell fills stay together and its lanes finish within a
// few steps of each other; a lane refilled in the middle would fill its cells
// alone (a fill costs about a fifth of two steps) for the rest of its life.
// So finished lanes wait until kRefill lanes are idle, which keeps one late
// ray from holding the whole warp. 512^3 / 1e7 rays with 3 mm beams and 256^3 /
// 1e6 rays with 6 mm beams (many side exits): 132.6 and - ms refilled one by one,
// 117.1 and 5.21 at 8 idle lanes, 107.1 and 5.13 at 16, 105.4 and 5.13 at 24,
// 104.7 and 5.20 at 30, 105.0 and 5.43 at 32. Nothing else synchronises: a CTA
// is one or two warps, and no warp waits for another one's rays. (Tiles of 1024 rays,
// sorted and traced by CTAs of eight warps that met at each tile's end, took
// 110.7 ms; and a small trace's tiles kept most SMs idle: 1e4 rays through
// 128^3 took 180 us in the kernel on 40 CTAs, 113 us on 313.)
// FAST: 0 every step runs the face test; 1 steps proven interior by the
// acceleration bound skip it and sample without the grid test (bound at most
// kInteriorAccel); 2 they skip the face test but sample with the grid test
// (any finite bound). Every mode takes the same steps.
template <class P, int IB, int FAST, int INTEG = INTEG_RKN, class Queue, class Cache>
__device__ __forceinline__ void trace_warp(const TraceArgs& a, Queue& q, Cache& cc, unsigned long long& my_steps) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    Ray<P> r;
    bool active = false, more = true;
    for (;;) {
        const unsigned idle = __ballot_sync(FULL, !active);
        if (more && __popc(idle) >= kRefill) {
            unsigned base, end;
            more = q.take(__popc(idle), lane, base, end);
            if (!active) {
                const unsigned k = base + __popc(idle & lt_mask);
                if (k < end) active = start_ray<P>(a, a.perm[k], r, my_steps);
            }
        }
        if (__ballot_sync(FULL, active) == 0u) {
            if (!more) break;
            continue;
        }
        typename P::R phi = typename P::R(1);
        int kind = -1;
        if (active) {
            if (FAST && r.run > 0) {
                --r.run;
                kind = 0;
            } else {
                kind = step_kind<P>(a, r, phi);
                if (FAST && kind == 0) r.run = interior_run<P>(a, r);
            }
        }
        // Fast path: when every live lane takes an interior step, the warp
        // takes `extra` more of them in a uniform loop, as many as every such
        // lane's run allows before its next save (so no save falls inside the
        // loop and no lane needs the face test, the refill or settle in
        // between). Idle lanes wait outside the minimum.
        int extra = 0;
        if (FAST) {
            const int mine = !active ? INT_MAX : (kind == 0 ? min(r.run, r.next_save - r.step - 1) : 0);
            extra = __reduce_min_sync(FULL, mine);
        }
        if (active) {
            if (FAST && kind == 0) {
#pragma unroll 1
                for (int e = 0;; ++e) {
                    step_any<P, IB, FAST == 1 ? SAMPLE_INTERIOR : SAMPLE_PLAIN, true, INTEG>(
                        a, r, cc, typename P::R(1));
                    if (e == extra) break;
                    ++r.step;
                }
                r.run -= extra;
            } else if (kind == 0 || kind == 3) {
                step_any<P, IB, SAMPLE_PLAIN, true, INTEG>(a, r, cc, typename P::R(1));
            } else {
                step_any<P, IB, SAMPLE_CLAMP, false, INTEG>(a, r, cc, phi);
                if (kind == 2) {
                    r.exited = true;
                    r.lag = 1.0 - (double)phi;
                }
            }
            ++r.step;
            active = settle<P>(a, r, my_steps, kind != 0);
        }
    }
}

// The cell cache of a precision; AHEAD: FP32 with the next cell fetched ahead.
template <class P, bool AHEAD = false>
using CellCacheFor = typename std::conditional<sizeof(typename P::R) != 4, CellPolyD,
                                               typename std::conditional<AHEAD, CellAheadF2, CellPolyF2>::type>::type;

__device__ __forceinline__ void reset_cache(CellPolyD& cc) { cc.base = 0xffffffffu; }
__device__ __forceinline__ void reset_cache(CellPolyF2& cc) { cc.base = 0xffffffffu; }
__device__ __forceinline__ void reset_cache(CellAheadF2& cc) {
    cc.base = cc.pred = 0xffffffffu;
    cc.slot = 0u;
}

// Threads per CTA of the single-trace kernels. No CTA synchronises; two warps that
// take neighbouring rays share their cells' lines in L1 (FP32, 256^3 trough / 1e6 rays:
// 4.40 ms in one-warp CTAs, 4.34 in two, 4.40 in eight; 192^3 / 2e5 1.194, 1.185, 1.230).
template <class P, bool AHEAD> constexpr int trace_threads() { return sizeof(typename P::R) == 4 && !AHEAD ? 64 : 32; }

// Warps per SM: FP32 16 at 128 registers (12 at 152 with the next cell fetched
// ahead); FP64 12 at 168, which holds the polynomials without spilling (256^3 /
// 4e5 rays: 4.53 ms, against 5.33 ms at 128 registers and 16 warps with 330 B of
// spill, 4.61 at 10 warps, 4.98 at 8).
template <class P, int INTEG, bool AHEAD> constexpr int trace_min_blocks() {
    const int warps = sizeof(typename P::R) == 4 ? (AHEAD ? 12 : kWarpsPerSm) : (INTEG == INTEG_RK4 ? 8 : 12);
    return warps * 32 / trace_threads<P, AHEAD>();
}

// Sum of `v` over the warp, added to *dst by one lane.
__device__ __forceinline__ void warp_add(unsigned long long v, unsigned long long* dst) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v && dst) atomicAdd(dst, v);
}

// ---------------------------------------------------------------------------
// Morton bucket pre-pass.
// ---------------------------------------------------------------------------
struct KeyArgs {
    const void* rays;
    long long n;
    double origin[3], inv_h[3];
    int cmax[3];      // n - 2 per axis
    int shift[3];     // right shift to fit 10 bits
    int axis, t1, t2;
    int bucket_shift; // key >> bucket_shift = bucket
    unsigned* keys;
    unsigned* hist;
};

// Morton key of ray i's entry cell.
template <class R>
__device__ __forceinline__ unsigned ray_key(const KeyArgs& k, long long i) {
    const R* rays = reinterpret_cast<const R*>(k.rays);
    unsigned c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        double u = floor(((double)rays[a * k.n + i] - k.origin[a]) * k.inv_h[a]);
        u = fmin(fmax(u, 0.0), (double)k.cmax[a]);   // NaN -> 0
        c[a] = ((unsigned)u) >> k.shift[a];
    }
    const unsigned c1 = k.t1 == 0 ? c[0] : c[1];
    const unsigned c2 = k.t2 == 1 ? c[1] : c[2];
    const unsigned ca = k.axis == 0 ? c[0] : (k.axis == 1 ? c[1] : c[2]);
    return morton_key(c1, c2, ca);
}

template <class R>
__global__ void __launch_bounds__(256) keys_kernel(const KeyArgs k) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < k.n; i += stride) {
        const unsigned key = ray_key<R>(k, i);
        k.keys[i] = key;
        atomicAdd(k.hist + (key >> k.bucket_shift), 1u);
    }
}

// The whole pre-pass of few rays in one CTA: keys, histogram, scan and scatter
// with the counts in shared memory and each ray's place in its bucket in a
// register. 3e3 rays: 7 us against 13 us for a memset and three kernels, most of that
// their launches (a 128^3 trace 104.5 -> 98.3 us); one SM has no more to give: 15
// us at 1e4 rays, so it ends at six rays per thread.
constexpr int kSmallThreads = 1024;
constexpr int kSmallPer = 6;
constexpr int kSmallRays = kSmallThreads * kSmallPer;
constexpr int kSmallBuckets = kSmallThreads;              // at least 2^bucket_bits_for(kSmallRays)

template <class R>
__global__ void __launch_bounds__(kSmallThreads) small_prepass_kernel(const KeyArgs k, unsigned* __restrict__ perm,
                                                                      unsigned long long* zero64, unsigned* zero32) {
    __shared__ unsigned s_count[kSmallBuckets];
    __shared__ unsigned s_warp[kSmallThreads / 32];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, n = (int)k.n;
    s_count[t] = 0u;
    if (t == 0) {
        if (zero64) *zero64 = 0ull;
        if (zero32) *zero32 = 0u;
    }
    __syncthreads();
    unsigned at[kSmallPer];                               // bucket << 16 | place in it
#pragma unroll
    for (int j = 0; j < kSmallPer; ++j) {
        const int i = t + j * kSmallThreads;
        if (i < n) {
            const unsigned b = ray_key<R>(k, i) >> k.bucket_shift;
            at[j] = b << 16 | atomicAdd(s_count + b, 1u);
        }
    }
    __syncthreads();
    const unsigned count = s_count[t];
    unsigned inc = count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) s_warp[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        unsigned w = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        s_warp[lane] = w;
    }
    __syncthreads();
    s_count[t] = inc - count + (wid > 0 ? s_warp[wid - 1] : 0u);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSmallPer; ++j) {
        const int i = t + j * kSmallThreads;
        if (i < n) perm[s_count[at[j] >> 16] + (at[j] & 0xffffu)] = (unsigned)i;
    }
}

// Exclusive scan of nb (<= 2^18) counts into offs, kScanSeg counts per CTA.
// Each CTA first sums every count before its segment, so that no CTA waits
// for another and one launch does it: at 2^18 counts the last of 64 CTAs
// reads 1 MB through L2 (one CTA alone: 56 us). hist and offs are 16-byte aligned and padded to a
// multiple of four counts; hist's padding is zero.
constexpr int kScanThreads = 256;
constexpr int kScanPer = 16;
constexpr int kScanSeg = kScanThreads * kScanPer;

__device__ __forceinline__ unsigned scan_block_sum(unsigned v, unsigned* s_warp) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    v = __reduce_add_sync(0xffffffffu, v);
    __syncthreads();
    if (lane == 0) s_warp[wid] = v;
    __syncthreads();
    unsigned t = 0;
#pragma unroll
    for (int k = 0; k < kScanThreads / 32; ++k) t += s_warp[k];
    return t;
}

static __global__ void __launch_bounds__(kScanThreads) scan_kernel(const unsigned* __restrict__ hist,
                                                                   unsigned* __restrict__ offs, int nb,
                                                                   unsigned long long* zero64, unsigned* zero32) {
    __shared__ unsigned s_warp[kScanThreads / 32];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const int seg = blockIdx.x * kScanSeg;
    if (blockIdx.x == 0 && t == 0) {
        if (zero64) *zero64 = 0ull;
        if (zero32) *zero32 = 0u;
    }
    const uint4* h4 = reinterpret_cast<const uint4*>(hist);
    unsigned before = 0;
#pragma unroll 8
    for (int i = t; i < seg / 4; i += kScanThreads) {
        const uint4 u = __ldg(h4 + i);
        before += (u.x + u.y) + (u.z + u.w);
    }
    const unsigned carry = scan_block_sum(before, s_warp);
    const int i0 = seg + t * kScanPer;
    unsigned v[kScanPer];
    unsigned sum = 0;
#pragma unroll
    for (int q = 0; q < kScanPer / 4; ++q) {
        uint4 u = make_uint4(0u, 0u, 0u, 0u);
        if (i0 + 4 * q < nb) u = __ldg(h4 + i0 / 4 + q);
        v[4 * q] = sum;
        v[4 * q + 1] = v[4 * q] + u.x;
        v[4 * q + 2] = v[4 * q + 1] + u.y;
        v[4 * q + 3] = v[4 * q + 2] + u.z;
        sum = v[4 * q + 3] + u.w;
    }
    unsigned inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    __syncthreads();
    if (lane == 31) s_warp[wid] = inc;
    __syncthreads();
    unsigned excl = carry + (inc - sum);
    for (int k = 0; k < wid; ++k) excl += s_warp[k];
#pragma unroll
    for (int q = 0; q < kScanPer / 4; ++q)
        if (i0 + 4 * q < nb)
            reinterpret_cast<uint4*>(offs)[i0 / 4 + q] =
                make_uint4(v[4 * q] + excl, v[4 * q + 1] + excl, v[4 * q + 2] + excl, v[4 * q + 3] + excl);
}

static __global__ void __launch_bounds__(256) scatter_kernel(const unsigned* __restrict__ keys, long long n,
                                                      int bucket_shift, unsigned* offs,
                                                      unsigned* __restrict__ perm) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        perm[atomicAdd(offs + (keys[i] >> bucket_shift), 1u)] = (unsigned)i;
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
inline size_t align256(size_t x) { return (x + 255u) & ~(size_t)255u; }

constexpr size_t kHeaderBytes = 256;
constexpr size_t kHistBytes = (size_t)4 << kMaxBucketBits;

inline size_t workspace_bytes(long long n) {
    const size_t a = align256((size_t)(n > 0 ? n : 1) * 4u);
    return kHeaderBytes + kHistBytes + 3 * a;
}

// Buckets of the pre-pass: about one per kBucketRays rays, at most 2^18. The
// histogram takes kHistBytes of the workspace and its scan the n words
// behind the permutation (2^bits < n / 4 for n > kBucketRays).
constexpr int kBucketRays = 8;
inline int bucket_bits_for(long long n) {
    int bits = 0;
    while (bits < kMaxBucketBits && ((long long)1 << bits) * kBucketRays < n) ++bits;
    return bits;
}

static_assert(kSmallBuckets * kBucketRays >= kSmallRays, "a small pre-pass has a count per bucket");

// Bytes of the histogram (the scan reads whole uint4).
inline size_t hist_bytes(int bbits) { return bbits < 2 ? 16 : (size_t)4 << bbits; }

// Morton pre-pass of n rays into bucket order: keys, histogram (2^bbits
// buckets, hist_bytes of them), exclusive scan, scatter into perm. `offs`
// holds max(4, 2^bbits) words; *zero64 and *zero32 (may be null) are set to 0 on the way.
// The buckets are the top bbits bits of those bits that the grid's keys use:
// with few rays per bucket a warp's 32 rays come from one or two neighbouring
// buckets, which needs no further sort, and the atomics spread over as many
// words. (The top bits of the whole 30-bit key, most of which a grid of 2^8
// cells leaves at zero, put 217k rays into 512 buckets: 40 us each for the
// histogram and the scatter against 4 us, and a sort per tile of 1024 rays in
// the tracer.)
template <class R>
inline int launch_prepass(const SlothGridDesc* g, int axis, const R* rays, long long n, int bbits,
                          unsigned* keys, unsigned* hist, unsigned* perm, unsigned* offs,
                          unsigned long long* zero64, unsigned* zero32, int sms, cudaStream_t s) {
    const int t1 = axis == 0 ? 1 : 0;
    const int t2 = axis == 2 ? 1 : 2;
    KeyArgs ka;
    ka.rays = rays;
    ka.n = n;
    for (int k = 0; k < 3; ++k) {
        ka.origin[k] = g->origin[k];
        ka.inv_h[k] = 1.0 / g->spacing[k];
        ka.cmax[k] = g->n[k] - 2;
        int sh = 0;
        while (((g->n[k] - 2) >> sh) > 1023) ++sh;
        ka.shift[k] = sh;
    }
    ka.axis = axis;
    ka.t1 = t1;
    ka.t2 = t2;
    int tb = 0;   // bits of the largest transverse cell coordinate
    for (int t : {t1, t2})
        while (((g->n[t] - 2) >> ka.shift[t]) >> tb) ++tb;
    const int used = 2 * tb + 10;
    ka.bucket_shift = used > bbits ? used - bbits : 0;
    ka.keys = keys;
    ka.hist = hist;
    if (n <= kSmallRays) {
        small_prepass_kernel<R><<<1, kSmallThreads, 0, s>>>(ka, perm, zero64, zero32);
        note_launch();
        return cuda_status(cudaGetLastError());
    }
    const cudaError_t e = cudaMemsetAsync(hist, 0, hist_bytes(bbits), s);
    if (e != cudaSuccess) return cuda_status(e);
    const long long nblk = (n + 255) / 256;
    const int kb = (int)(nblk < (long long)sms * 8 ? nblk : (long long)sms * 8);
    const int nb = 1 << bbits;
    keys_kernel<R><<<kb, 256, 0, s>>>(ka);
    note_launch();
    scan_kernel<<<(nb + kScanSeg - 1) / kScanSeg, kScanThreads, 0, s>>>(hist, offs, nb, zero64, zero32);
    note_launch();
    scatter_kernel<<<kb, 256, 0, s>>>(keys, n, ka.bucket_shift, offs, perm);
    note_launch();
    return cuda_status(cudaGetLastError());
}

// Inverse-bremsstrahlung path of a trace: off, sub-critical (the grid's
// density stays below nc, so the Coulomb log is a constant), or general.
inline int trace_mode(const SlothTraceParams* p) {
    const double xmax = p->q_max > 0.0 ? p->q_max * p->ope_ratio2 : 1e300;
    return !p->inv_brems ? IB_OFF : (xmax <= 1.0 ? IB_SUBCRITICAL : IB_GENERAL);
}

// Largest |acceleration| (cells per step^2) the grid's density range allows:
// max_k |S_k| * (q_max - min(q_min, 0)); infinite when the range is unknown.
inline double interior_accel_bound(const SlothGridDesc* g, const SlothTraceParams* p) {
    if (!(p->q_max > 0.0) || !std::isfinite(p->q_min) || !(p->q_min <= p->q_max)) return INFINITY;
    double smax = 0.0;
    for (int k = 0; k < 3; ++k) {
        const double r = p->dtau / g->spacing[k];
        smax = fmax(smax, 0.5 * r * r);
    }
    return smax * (p->q_max - fmin(p->q_min, 0.0));
}

// Kernel arguments of one trace from the public descriptors.
inline void fill_trace_args(TraceArgs& ta, const SlothGridDesc* g, const void* grid, const SlothTraceParams* p,
                            const void* rays, long long n, const SlothTraceOutputs* out, const unsigned* perm) {
    const int axis = p->probing_axis;
    ta.geo = make_geo(g);
    ta.grid = grid;
    ta.rays = rays;
    ta.n = n;
    ta.perm = perm;
    ta.queue = nullptr;
    const unsigned stride[3] = {ta.geo.sx, ta.geo.sy, 1u};
    ta.sa = stride[axis];
    ta.s1 = stride[axis == 0 ? 1 : 0];
    ta.s2 = stride[axis == 2 ? 1 : 2];
    ta.ahead_max = (unsigned)g->n[0] * (unsigned)g->n[1] * (unsigned)g->n[2] - 1u - ta.s1 - ta.s2;
    for (int k = 0; k < 3; ++k) {
        const double h = g->spacing[k];
        ta.origin[k] = g->origin[k];
        ta.spacing[k] = h;
        ta.w_of_v[k] = (p->dtau / h) / kC;
        ta.v_of_w[k] = kC * h / p->dtau;
        ta.S[k] = -0.5 * (p->dtau / h) * (p->dtau / h);
        ta.S4[k] = 0.25 * ta.S[k];
        ta.S2[k] = 0.5 * ta.S[k];
        ta.S6[k] = (1.0 / 6.0) * ta.S[k];
        ta.Sf[k] = (float)ta.S[k];
        // as the step forms them at phi = 1: exact scalings by 1/4 and 1/2, one
        // FP32 rounding of fl(1/6) * Sf
        ta.S4f[k] = 0.25f * ta.Sf[k];
        ta.S2f[k] = 0.5f * ta.Sf[k];
        ta.S6f[k] = (1.0f / 6.0f) * ta.Sf[k];
    }
    ta.phase_scale = (p->omega / kC) * p->dtau / 6.0;
    ta.tau_scale = p->kappa_q2 * p->dtau / 6.0;   // times cl_lo below for the sub-critical mode
    ta.cl_w = p->coulomb_log_w;
    ta.cl_lo = p->coulomb_log_w > 2.0 ? p->coulomb_log_w : 2.0;
    ta.ope2 = p->ope_ratio2;
    ta.ope2f = (float)ta.ope2;
    ta.inv_ope2 = 1.0 / p->ope_ratio2;
    ta.inv_ope2f = (float)ta.inv_ope2;
    ta.cl_lof = (float)ta.cl_lo;
    // Below the critical density the Coulomb log is the constant cl_lo and the
    // corners carry x^2 = (ope2 q)^2, so the optical depth's scale takes
    // cl_lo / ope2^2 once.
    if (trace_mode(p) == IB_SUBCRITICAL) ta.tau_scale *= ta.cl_lo * ta.inv_ope2 * ta.inv_ope2;
    ta.cl_wf = (float)ta.cl_w;
    {
        const double B = interior_accel_bound(g, p);
        ta.accel_bound = std::isfinite(B) ? (float)(B * 1.001) : 0.0f;
    }
    ta.plane = p->plane;
    ta.first_save = p->first_save;
    ta.save_every = p->n_saves > 1 ? p->save_every : 1;
    ta.n_saves = p->n_saves;
    ta.axis = axis;
    ta.t1 = axis == 0 ? 1 : 0;
    ta.t2 = axis == 2 ? 1 : 2;
    ta.project = p->project_to_plane ? 1 : 0;
    ta.jones = out->jones;
    ta.state = out->state;
    ta.phase = out->phase;
    ta.amp = out->amp;
    ta.status = out->status;
    ta.steps = out->steps;
    ta.total_steps = out->total_steps;
}

// Validation shared by the trace entry points (everything but buffers).
inline int check_trace_params(const SlothGridDesc* g, const SlothTraceParams* p, int64_t n) {
    int rc = check_grid(g);
    if (rc) return rc;
    if (!p) return SLOTH_ERR_NULL_POINTER;
    if (n < 0 || n > 2147483647LL) return n < 0 ? SLOTH_ERR_INVALID_ARGUMENT : SLOTH_ERR_TOO_LARGE;
    if (!(p->omega > 0.0) || !(p->dtau > 0.0) || !std::isfinite(p->dtau) || !std::isfinite(p->omega))
        return SLOTH_ERR_INVALID_ARGUMENT;
    if (p->n_saves < 1 || p->n_saves > SLOTH_MAX_SAVES || p->first_save < 0) return SLOTH_ERR_INVALID_ARGUMENT;
    if (p->n_saves > 1 && p->save_every < 1) return SLOTH_ERR_INVALID_ARGUMENT;
    if (p->probing_axis < 0 || p->probing_axis > 2) return SLOTH_ERR_INVALID_ARGUMENT;
    const long long last =
        (long long)p->first_save + (long long)(p->n_saves - 1) * (p->n_saves > 1 ? p->save_every : 0);
    if (last > 2000000000LL) return SLOTH_ERR_TOO_LARGE;
    if (p->inv_brems && !(p->kappa_q2 >= 0.0)) return SLOTH_ERR_INVALID_ARGUMENT;
    if (p->project_to_plane && !std::isfinite(p->plane)) return SLOTH_ERR_INVALID_ARGUMENT;
    if (!(p->ope_ratio2 > 0.0) || !std::isfinite(p->ope_ratio2)) return SLOTH_ERR_INVALID_ARGUMENT;
    if (!std::isfinite(p->q_max)) return SLOTH_ERR_INVALID_ARGUMENT;
    if (p->integrator != SLOTH_INTEGRATOR_RKN && p->integrator != SLOTH_INTEGRATOR_RK4)
        return SLOTH_ERR_INVALID_ARGUMENT;
    if (p->reserved != 0) return SLOTH_ERR_INVALID_ARGUMENT;
    return SLOTH_OK;
}

// True when interior steps may skip the per-stage grid test: the
// acceleration |S_k * dq/du_k| is at most max_k |S_k| * (q_max - min(q_min, 0))
// (a difference of q over at most one cell), and that is within
// kInteriorAccel. Needs q_max > 0 (known) and q_min <= q_max.
inline bool interior_bound_ok(const SlothGridDesc* g, const SlothTraceParams* p) {
    return interior_accel_bound(g, p) <= kInteriorAccel;
}


}  // namespace sloth
