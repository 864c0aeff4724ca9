// Detector-image forward model and its adjoint: the gradient of a loss on a
// synthetic detector image with respect to the density grid.
//
// No counterpart in the reference, which never differentiates. The model
// differentiates the reference's ray equations (src/core/propagator.py:
// 168-243, dr/dt = v, dv/dt = -(c^2/2) grad(ne/nc) from the precomputed
// gradient grid through the trilinear interpolator, src/core/interpolator.py:
// 79-104, fill 0 outside) through a detector image:
//
//   ne --pack (K1)--> (q, dq/du, dq/dv, dq/dw)
//      --fixed-step Runge-Kutta-Nystrom, at most n_steps steps--> final ray state
//      --straight line to the detector plane--> (X, Y)
//      --Gaussian splat--> image I
//
// The step is the tracer's (fourth-order Runge-Kutta-Nystrom, unit steps in
// grid cells) without face
// clipping: every stage samples the interpolant with fill 0 outside, so a
// ray's map is smooth except where a stage point crosses a grid face. A ray
// stops early once it is outside the grid on some axis and moving away from
// it along that axis: its remaining steps are straight lines, and the
// projection to the detector plane (src/shared/propagation.py:92-134) gives
// the same point from any point of that line.
//
// Splat: a ray at pixel coordinates (a, b) adds norm * g(i - a) * g(j - b)
// to pixel (i, j), with g(d) = exp(-d^2 / (2 s^2)) * taper(|d| / s), taper = 1
// up to 3 s and a C2 smoothstep from 1 to 0 between 3 s and 4 s, and norm =
// 1 / (2 pi s^2). The taper keeps the splat twice differentiable with a
// finite support of 4 s.
//
// Adjoint (backward): for each ray, d L / d(final state) from the image
// gradient through the splat and the projection; then, segment by segment
// from the last, the trajectory is recomputed from the segment's checkpoint
// (the forward stores one every ckpt_every steps) and the discrete adjoint of
// each step runs in reverse. Each stage's contribution to d L / d(grid
// gradient channels) is accumulated in registers for the 8 corners of the
// stage's cell and added to the grid-gradient buffer when the cell changes.
// pack_adjoint_kernel maps d L / d(packed grid) through the transposed
// difference stencil of K1 to d L / d ne.
#include <climits>
#include <cmath>

#include "tracer.cuh"

namespace sloth {

// One-warp CTAs for the forward and the backward: a finished warp's place is
// taken at once, and few rays spread over all SMs.
// The backward's recompute of a checkpoint segment records where each stage
// of each step sampled the field (its cell and in-cell coordinates), and the
// step adjoints linearise there. Five of a step's nine in-cell coordinates go to
// shared memory, [step][word][thread] so that a warp's accesses are
// consecutive; the three cells and the other coordinates stay in a per-thread
// array. A 20-step segment takes 12.8 KB of shared memory per warp in FP32, so 16
// warps share an SM (the kernel is latency-bound).
constexpr int kAdjThreads = 32;
constexpr int kAdjStateWords = 5;
// Two FP32 builds of the backward: 16 warps per SM (128 registers) when as
// many segment buffers fit an SM's shared memory (on B200, 228 KB per SM and
// 1 KB reserved per CTA: checkpoints at most every 21 steps), 12 otherwise
// (room for 168 registers a thread, of which it takes 148). FP64 runs 8. The FP32 forward runs 24 (80 registers).
template <class P> constexpr int adj_fwd_min_blocks() { return sizeof(typename P::R) == 4 ? 24 : 12; }
constexpr int kMaxCkptEvery = 32;
constexpr int kMaxTaps = 65;          // 2 * 4 * sigma + 1 pixels at sigma <= 8

struct ImageArgs {
    GridGeo geo;
    const void* grid;
    const void* rays;            // (6, n) of R, original order
    long long n;
    const unsigned* perm;        // slot -> ray id (bucket order)
    double origin[3], w_of_v[3], inv_h[3];
    double S[3];                 // -(dtau/h)^2 / 2
    float Sf[3];                 // S rounded to FP32 once on the host (the FP32 kernels' copy)
    float S4f[3], S2f[3], S6f[3];   // Sf/4, Sf/2 and fl(1/6)*Sf: the FP32 step's coefficients
    int n_steps, ckpt_every, n_seg;
    int axis, t1, t2;
    double plane;                // detector plane (cells along axis)
    double px0[2], px_per_cell[2];
    int npx[2];
    int taps;                    // pixels per axis in a splat window
    double sigma, radius, norm;  // pixels
    void* ckpt;                  // [n_seg + 1][12 floats | 6 doubles][n]
    int* nsteps;                 // steps taken, per slot
    void* image;                 // forward: the image; backward: d L / d image
    void* ggrad;                 // backward: d L / d(packed grid)
    unsigned long long* total_steps;   // forward: steps of all rays are added here (may be null)
    const unsigned* accel_bound;       // float bits of max |S_k dq/du_k| over the grid (workspace)
};

// S_k in the kernel's precision: FP32 kernels read the host-rounded copy, so
// no step converts it.
template <class R> __device__ __forceinline__ R img_S(const ImageArgs& a, int k);
template <> __device__ __forceinline__ float img_S<float>(const ImageArgs& a, int k) { return a.Sf[k]; }
template <> __device__ __forceinline__ double img_S<double>(const ImageArgs& a, int k) { return a.S[k]; }

// ---------------------------------------------------------------------------
// Ray state and checkpoints.
// ---------------------------------------------------------------------------
template <class P>
struct MState {
    typename P::Acc p[3], w[3];
};

// A checkpoint is 48 bytes per ray: FP32 stores the value and compensation of
// each of the six sums, FP64 the six values; component-major for coalescing.
template <class P>
__device__ __forceinline__ void store_state(const ImageArgs& a, int k, long long slot, const MState<P>& r) {
    if constexpr (sizeof(typename P::R) == 4) {
        float* c = reinterpret_cast<float*>(a.ckpt) + (size_t)k * 12 * a.n + slot;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            c[(2 * x) * a.n] = r.p[x].s;
            c[(2 * x + 1) * a.n] = r.p[x].c;
            c[(6 + 2 * x) * a.n] = r.w[x].s;
            c[(7 + 2 * x) * a.n] = r.w[x].c;
        }
    } else {
        double* c = reinterpret_cast<double*>(a.ckpt) + (size_t)k * 6 * a.n + slot;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            c[x * a.n] = r.p[x].s;
            c[(3 + x) * a.n] = r.w[x].s;
        }
    }
}

template <class P>
__device__ __forceinline__ void load_state(const ImageArgs& a, int k, long long slot, MState<P>& r) {
    if constexpr (sizeof(typename P::R) == 4) {
        const float* c = reinterpret_cast<const float*>(a.ckpt) + (size_t)k * 12 * a.n + slot;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            r.p[x].s = c[(2 * x) * a.n];
            r.p[x].c = c[(2 * x + 1) * a.n];
            r.w[x].s = c[(6 + 2 * x) * a.n];
            r.w[x].c = c[(7 + 2 * x) * a.n];
        }
    } else {
        const double* c = reinterpret_cast<const double*>(a.ckpt) + (size_t)k * 6 * a.n + slot;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            r.p[x].s = c[x * a.n];
            r.w[x].s = c[(3 + x) * a.n];
        }
    }
}

// Outside the grid on some axis and moving away from it along that axis (or
// not finite): every later step is a straight line.
template <class P>
__device__ __forceinline__ bool ray_gone_model(const ImageArgs& a, const MState<P>& r) {
    using R = typename P::R;
    bool gone = false;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const R p = r.p[x].val(), w = r.w[x].val();
        gone |= (p < R(0) && w <= R(0)) || (p > lim_of<R>(a.geo, x) && w >= R(0)) || !(p == p) || !(w == w);
    }
    return gone;
}

// ---------------------------------------------------------------------------
// The gradient channels of one cell as trilinear polynomials.
// ---------------------------------------------------------------------------
template <class P>
struct GradCell {
    unsigned base;
    typename P::R t[3][8];
};

// Cell and in-cell coordinates of the point hi + lo (the tracer's split: the
// cell from the rounded sum, the fractions from (hi - i) + lo). False when
// the point is outside the grid (fill 0).
template <class P>
__device__ __forceinline__ bool locate(const GridGeo& g, const typename P::R (&hi)[3],
                                       const typename P::R (&lo)[3], unsigned& base, typename P::R (&f)[3]) {
    using R = typename P::R;
    R p[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) p[x] = hi[x] + lo[x];
    const bool in = (p[0] >= R(0)) & (p[0] <= lim_of<R>(g, 0)) & (p[1] >= R(0)) & (p[1] <= lim_of<R>(g, 1)) &
                    (p[2] >= R(0)) & (p[2] <= lim_of<R>(g, 2));
    if (!in) return false;
    const int ix = min((int)p[0], g.n[0] - 2), iy = min((int)p[1], g.n[1] - 2), iz = min((int)p[2], g.n[2] - 2);
    f[0] = (hi[0] - (R)ix) + lo[0];
    f[1] = (hi[1] - (R)iy) + lo[1];
    f[2] = (hi[2] - (R)iz) + lo[2];
    base = (unsigned)ix * g.sx + (unsigned)iy * g.sy + (unsigned)iz;
    return true;
}

// FP32: the gradient channels as a scalar polynomial, dq/du, and a pair of
// them, (dq/dv, dq/dw), evaluated with sm_100's paired FP32 instructions. (As the
// pair (q, dq/du), q would be carried along on the FMA pipe.)
struct GradCellF2 {
    unsigned base;
    float t0[8];      // dq/du
    float2 t1[8];     // (dq/dv, dq/dw)
};

__device__ __forceinline__ void load_cell_f2(const ImageArgs& a, unsigned b, GradCellF2& cc) {
    if (b == cc.base) return;
    cc.base = b;
    const GridGeo& g = a.geo;
    const float4* gp = reinterpret_cast<const float4*>(a.grid);
    const float4 v0 = __ldg(gp + b), v1 = __ldg(gp + b + 1u);
    const float4 v2 = __ldg(gp + b + g.sy), v3 = __ldg(gp + b + g.sy + 1u);
    const float4 v4 = __ldg(gp + b + g.sx), v5 = __ldg(gp + b + g.sx + 1u);
    const float4 v6 = __ldg(gp + b + g.sx + g.sy), v7 = __ldg(gp + b + g.sx + g.sy + 1u);
#define SLOTH_HI(v) make_float2(v.z, v.w)
    poly_coeffs<float>(cc.t0, v0.y, v1.y, v2.y, v3.y, v4.y, v5.y, v6.y, v7.y);
    poly_coeffs2(cc.t1, SLOTH_HI(v0), SLOTH_HI(v1), SLOTH_HI(v2), SLOTH_HI(v3), SLOTH_HI(v4), SLOTH_HI(v5),
                 SLOTH_HI(v6), SLOTH_HI(v7));
#undef SLOTH_HI
}

template <class P>
__device__ __forceinline__ void load_cell(const ImageArgs& a, unsigned b, GradCell<P>& cc) {
    using R = typename P::R;
    if (b == cc.base) return;
    cc.base = b;
    const GridGeo& g = a.geo;
    const typename P::V v0 = P::load(a.grid, b), v1 = P::load(a.grid, b + 1u);
    const typename P::V v2 = P::load(a.grid, b + g.sy), v3 = P::load(a.grid, b + g.sy + 1u);
    const typename P::V v4 = P::load(a.grid, b + g.sx), v5 = P::load(a.grid, b + g.sx + 1u);
    const typename P::V v6 = P::load(a.grid, b + g.sx + g.sy), v7 = P::load(a.grid, b + g.sx + g.sy + 1u);
    poly_coeffs<R>(cc.t[0], v0.y, v1.y, v2.y, v3.y, v4.y, v5.y, v6.y, v7.y);
    poly_coeffs<R>(cc.t[1], v0.z, v1.z, v2.z, v3.z, v4.z, v5.z, v6.z, v7.z);
    poly_coeffs<R>(cc.t[2], v0.w, v1.w, v2.w, v3.w, v4.w, v5.w, v6.w, v7.w);
}

// Where one stage sampled the field: the cell (kNone when the point was
// outside the grid, fill 0) and the in-cell coordinates. The backward's
// recompute records the three stages of every step, and the step's adjoint
// linearises at exactly those points.
constexpr unsigned kNone = 0xffffffffu;

template <class P>
struct StageRec {
    unsigned b;
    typename P::R f[3];
};

// FP64: acceleration S * grad(q) at hi + lo (zero outside); with rec, where it
// sampled.
template <class P>
__device__ __forceinline__ void accel(const ImageArgs& a, const typename P::R (&hi)[3], const typename P::R (&lo)[3],
                                      typename P::R (&A)[3], GradCell<P>& cc, StageRec<P>* rec) {
    using R = typename P::R;
    unsigned b;
    R f[3];
    if (!locate<P>(a.geo, hi, lo, b, f)) {
        A[0] = A[1] = A[2] = R(0);
        if (rec) {
            rec->b = kNone;
            rec->f[0] = rec->f[1] = rec->f[2] = R(0);
        }
        return;
    }
    if (rec) {
        rec->b = b;
        rec->f[0] = f[0];
        rec->f[1] = f[1];
        rec->f[2] = f[2];
    }
    load_cell<P>(a, b, cc);
#pragma unroll
    for (int k = 0; k < 3; ++k) A[k] = a.S[k] * poly_eval<R>(cc.t[k], f[0], f[1], f[2]);
}

// FP32: the gradient at (hx + lx, hyz + lyz), y and z as a pair (zero outside);
// with rec, where it sampled.
template <bool INTERIOR>
__device__ __forceinline__ void gradient_f2(const ImageArgs& a, float hx, float lx, float2 hyz, float2 lyz, float& Gx,
                                            float2& Gyz, GradCellF2& cc, StageRec<PolF32>* rec) {
    const GridGeo& g = a.geo;
    const float px = hx + lx;
    const float2 pyz = __fadd2_rn(hyz, lyz);
    int ix, iy, iz;
    if constexpr (!INTERIOR) {
        const bool in = (px >= 0.0f) & (px <= g.limf[0]) & (pyz.x >= 0.0f) & (pyz.x <= g.limf[1]) &
                        (pyz.y >= 0.0f) & (pyz.y <= g.limf[2]);
        if (!in) {
            Gx = 0.0f;
            Gyz = make_float2(0.0f, 0.0f);
            if (rec) {
                rec->b = kNone;
                rec->f[0] = rec->f[1] = rec->f[2] = 0.0f;
            }
            return;
        }
        ix = min((int)px, g.n[0] - 2);
        iy = min((int)pyz.x, g.n[1] - 2);
        iz = min((int)pyz.y, g.n[2] - 2);
    } else {
        // a point of an interior step: inside by construction; one unsigned
        // min per axis keeps the index in the grid all the same
        ix = (int)min((unsigned)(int)px, (unsigned)(g.n[0] - 2));
        iy = (int)min((unsigned)(int)pyz.x, (unsigned)(g.n[1] - 2));
        iz = (int)min((unsigned)(int)pyz.y, (unsigned)(g.n[2] - 2));
    }
    const float fx = (hx - (float)ix) + lx;
    const float2 fyz = __fadd2_rn(__fadd2_rn(hyz, make_float2(-(float)iy, -(float)iz)), lyz);
    const unsigned b = (unsigned)ix * g.sx + (unsigned)iy * g.sy + (unsigned)iz;
    if (rec) {
        rec->b = b;
        rec->f[0] = fx;
        rec->f[1] = fyz.x;
        rec->f[2] = fyz.y;
    }
    load_cell_f2(a, b, cc);
    Gx = poly_eval<float>(cc.t0, fx, fyz.x, fyz.y);
    Gyz = poly_eval2(cc.t1, bc2(fx), bc2(fyz.x), bc2(fyz.y));
}

// One step (the tracer's Runge-Kutta-Nystrom step with phi = 1, without
// phase and depth):
//   p' = p + w + (A1 + 2 A2)/6,  w' = w + (A1 + 4 A2 + A3)/6,
//   stages at p, p + w/2 + A1/8, p + w + A2/2.
// INTERIOR (FP32): the step's points are known to lie inside the grid, bitwise
// the same step. The FP32 step is the tracer's paired one: S in the coefficients,
// y and z as register pairs, every rounding explicit, so that the forward's and the
// recompute's steps agree bit for bit.
template <bool INTERIOR>
__device__ __forceinline__ void model_step(const ImageArgs& a, MState<PolF32>& r, GradCellF2& cc,
                                           StageRec<PolF32>* rec = nullptr) {
    const float phx = r.p[0].s, plx = r.p[0].c, wex = __fadd_rn(r.w[0].s, r.w[0].c);
    const float2 phyz = make_float2(r.p[1].s, r.p[2].s), plyz = make_float2(r.p[1].c, r.p[2].c);
    const float2 whi = make_float2(r.w[1].s, r.w[2].s), wlo = make_float2(r.w[1].c, r.w[2].c);
    const float2 weyz = __fadd2_rn(whi, wlo);
    const float2 S6yz = make_float2(a.S6f[1], a.S6f[2]);
    float Gx;
    float2 Gyz;
    gradient_f2<INTERIOR>(a, phx, plx, phyz, plyz, Gx, Gyz, cc, rec);
    float gAx = Gx, gWx = Gx;                   // g1 + 2 g2 and g1 + 4 g2 + g3
    float2 gAyz = Gyz, gWyz = Gyz;
    float stx = __fmaf_rn(0.5f, __fmaf_rn(a.S4f[0], Gx, wex), plx);       // p + (w + S/4 G1)/2
    float2 styz = __ffma2_rn(bc2(0.5f), __ffma2_rn(make_float2(a.S4f[1], a.S4f[2]), Gyz, weyz), plyz);
    gradient_f2<INTERIOR>(a, phx, stx, phyz, styz, Gx, Gyz, cc, rec ? rec + 1 : nullptr);
    gAx = __fmaf_rn(2.0f, Gx, gAx);
    gAyz = __ffma2_rn(bc2(2.0f), Gyz, gAyz);
    gWx = __fmaf_rn(4.0f, Gx, gWx);
    gWyz = __ffma2_rn(bc2(4.0f), Gyz, gWyz);
    stx = __fadd_rn(plx, __fmaf_rn(a.S2f[0], Gx, wex));                   // p + w + S/2 G2
    styz = __fadd2_rn(plyz, __ffma2_rn(make_float2(a.S2f[1], a.S2f[2]), Gyz, weyz));
    gradient_f2<INTERIOR>(a, phx, stx, phyz, styz, Gx, Gyz, cc, rec ? rec + 2 : nullptr);
    gWx = __fadd_rn(gWx, Gx);
    gWyz = __fadd2_rn(gWyz, Gyz);
    r.p[0].add(__fadd_rn(r.w[0].hi(), __fmaf_rn(a.S6f[0], gAx, r.w[0].lo())));
    r.w[0].add_fma(a.S6f[0], gWx);
    float2 ps = phyz, pc = plyz, ws = whi, wc = wlo;
    kahan2(ps, pc, __fadd2_rn(whi, __ffma2_rn(S6yz, gAyz, wlo)));
    kahan2_fma(ws, wc, S6yz, gWyz);
    r.p[1].s = ps.x; r.p[2].s = ps.y; r.p[1].c = pc.x; r.p[2].c = pc.y;
    r.w[1].s = ws.x; r.w[2].s = ws.y; r.w[1].c = wc.x; r.w[2].c = wc.y;
}

template <bool INTERIOR, class P>
__device__ __forceinline__ void model_step(const ImageArgs& a, MState<P>& r, GradCell<P>& cc,
                                           StageRec<P>* rec = nullptr) {
    using R = typename P::R;
    R ph[3], pl[3], we[3], st[3], A1[3], A2[3], A3[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        ph[x] = r.p[x].hi();
        pl[x] = r.p[x].lo();
        we[x] = r.w[x].val();
    }
    accel<P>(a, ph, pl, A1, cc, rec);
#pragma unroll
    for (int x = 0; x < 3; ++x) st[x] = pl[x] + (R(0.5) * we[x] + R(0.125) * A1[x]);
    accel<P>(a, ph, st, A2, cc, rec ? rec + 1 : nullptr);
#pragma unroll
    for (int x = 0; x < 3; ++x) st[x] = pl[x] + (we[x] + R(0.5) * A2[x]);
    accel<P>(a, ph, st, A3, cc, rec ? rec + 2 : nullptr);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const R sA = A1[x] + R(2) * A2[x];
        const R sW = (A1[x] + R(4) * A2[x]) + A3[x];
        r.p[x].add(r.w[x].hi() + (r.w[x].lo() + sA * R(1.0 / 6.0)));
        r.w[x].add(sW * R(1.0 / 6.0));
    }
}

// ---------------------------------------------------------------------------
// Adjoint of one step.
// ---------------------------------------------------------------------------
template <class P>
struct CornerAcc {
    unsigned base;               // cell of the pending sums (kNone: none)
    typename P::R v[3][8];       // d L / d(channel k) at corner c
};

template <class P> struct AdjTypes { using Cell = GradCell<P>; using Acc = CornerAcc<P>; };
struct CornerAccF2;
template <> struct AdjTypes<PolF32> { using Cell = GradCellF2; using Acc = CornerAccF2; };

// Adds (x, y, z, w) to *p as one vector reduction that returns nothing
// (red.global.add.v4.f32, sm_90 and later). A float4 atomicAdd compiles to
// an atomic that sends each old value back through the crossbar; with about
// one flush of eight corners per three ray-steps that return traffic cost
// the backward 9% of its time.
__device__ __forceinline__ void red_add_v4(float4* p, float x, float y, float z, float w) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                 :: "l"(p), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

template <class P>
__device__ __forceinline__ void flush(const ImageArgs& a, CornerAcc<P>& acc) {
    using R = typename P::R;
    if (acc.base == kNone) return;
    const GridGeo& g = a.geo;
    const unsigned b = acc.base;
    const unsigned off[8] = {b, b + 1u, b + g.sy, b + g.sy + 1u, b + g.sx, b + g.sx + 1u, b + g.sx + g.sy,
                             b + g.sx + g.sy + 1u};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        if constexpr (sizeof(R) == 4) {
            red_add_v4(reinterpret_cast<float4*>(a.ggrad) + off[c], 0.0f, acc.v[0][c], acc.v[1][c], acc.v[2][c]);
        } else {
            double* d = reinterpret_cast<double*>(a.ggrad) + 4 * (size_t)off[c];
            atomicAdd(d + 1, acc.v[0][c]);
            atomicAdd(d + 2, acc.v[1][c]);
            atomicAdd(d + 3, acc.v[2][c]);
        }
    }
    acc.base = kNone;
}

// FP32 corner sums as pairs: v[k][i] holds channel k + 1 at corners 2i and
// 2i + 1, which differ in z only, so that a pair is one sm_100 paired FP32
// operation and one pair of adjacent voxels in the flush.
struct CornerAccF2 {
    unsigned base;
    float2 v[3][4];
};

// The lanes of a warp that flush the same cell together first combine their
// corner sums in groups of up to four, and one lane per group of four issues
// the eight reductions. Rays of a warp share their entry cell and cross cell
// faces at the same steps, so a flush typically has most of the warp in one
// cell; 26 lanes issuing eight reductions each to the same eight voxels
// serialise in L2 (about a third of the backward's time before this). The
// combination is a tree over the members' ranks (the lanes that flush the same
// cell, in lane order): at stride d, rank r (r a multiple of 2d) adds the
// partial sum of rank r + d, found by pointer jumping (the member d ranks up
// is the member d/2 ranks up of the member d/2 ranks up). Two rounds measured
// best: 11.2 ms for the bench's backward, against 12.1 ms for a tree over the
// whole group (its shuffles cost more than the reductions they save) and
// 13.1 ms without combining. Every lane of `active` (the lanes that reached
// this call together) runs the same rounds, so the shuffles are matched.
constexpr int kFlushCombine = 4;   // lanes combined per reduction, a power of two
__device__ __forceinline__ void flush(const ImageArgs& a, CornerAccF2& acc) {
    const unsigned active = __activemask();
    const unsigned grp = __match_any_sync(active, acc.base);
    const int lane = threadIdx.x & 31;
    const unsigned above = grp & ~((2u << lane) - 1u);       // members above this lane
    int up = above ? __ffs(above) - 1 : lane;                // the member one rank up
    int has = above != 0u;
    const int rank = __popc(grp & ((1u << lane) - 1u));
    const int rounds = __reduce_max_sync(active, __popc(grp));
    int span = 1;   // after the rounds, rank r (a multiple of span) holds ranks r .. r + span - 1
    for (int d = 1; d < rounds && d < kFlushCombine; d <<= 1) {
        span = 2 * d;
        const float take = (has && (rank & (2 * d - 1)) == 0) ? 1.0f : 0.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float tx = __shfl_sync(active, acc.v[k][i].x, up);
                const float ty = __shfl_sync(active, acc.v[k][i].y, up);
                acc.v[k][i].x = fmaf(take, tx, acc.v[k][i].x);
                acc.v[k][i].y = fmaf(take, ty, acc.v[k][i].y);
            }
        const int up2 = __shfl_sync(active, up, up);
        const int has2 = __shfl_sync(active, has, up);
        has = has && has2;
        up = has ? up2 : lane;   // no member that far up: read this lane's own sums (taken times 0)
    }
    if ((rank & (span - 1)) == 0 && acc.base != kNone) {
        const GridGeo& g = a.geo;
        const unsigned b = acc.base;
        const unsigned off[4] = {b, b + g.sy, b + g.sx, b + g.sx + g.sy};
        float4* gg = reinterpret_cast<float4*>(a.ggrad);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            red_add_v4(gg + off[i], 0.0f, acc.v[0][i].x, acc.v[1][i].x, acc.v[2][i].x);
            red_add_v4(gg + off[i] + 1u, 0.0f, acc.v[0][i].y, acc.v[1][i].y, acc.v[2][i].y);
        }
    }
    acc.base = kNone;
}

// Stage adjoint on the paired FP32 cache: channels 2 and 3 of the Jacobian
// transpose, the corner weights and the corner sums run as paired FP32
// operations (__ffma2_rn / __fmul2_rn), channel 1 scalar.
template <class P>
__device__ __forceinline__ void stage_adjoint(const ImageArgs& a, const StageRec<PolF32>& rec,
                                              const float (&Abar)[3], float (&q)[3], GradCellF2& cc,
                                              CornerAccF2& acc) {
    const unsigned b = rec.b;
    if (b == kNone) {
        q[0] = q[1] = q[2] = 0.0f;
        return;
    }
    const float f[3] = {rec.f[0], rec.f[1], rec.f[2]};
    load_cell_f2(a, b, cc);
    const float fx = f[0], fy = f[1], fz = f[2];
    const float2 fx2 = make_float2(fx, fx), fy2 = make_float2(fy, fy), fz2 = make_float2(fz, fz);
    float gb[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) gb[k] = img_S<float>(a, k) * Abar[k];
    // J^T gb. Channel 1 (dq/du) is t0, channels 2 and 3 are the pairs t1.
    const float* t0 = cc.t0;
    const float2* t1 = cc.t1;
    const float u76 = fmaf(fx, t0[7], t0[6]);
    const float d1x = fmaf(fz, fmaf(fy, t0[7], t0[5]), fmaf(fy, t0[4], t0[1]));
    const float d1y = fmaf(fz, u76, fmaf(fx, t0[4], t0[2]));
    const float d1z = fmaf(fy, u76, fmaf(fx, t0[5], t0[3]));
    const float2 v76 = __ffma2_rn(fx2, t1[7], t1[6]);
    const float2 d2x = __ffma2_rn(fz2, __ffma2_rn(fy2, t1[7], t1[5]), __ffma2_rn(fy2, t1[4], t1[1]));
    const float2 d2y = __ffma2_rn(fz2, v76, __ffma2_rn(fx2, t1[4], t1[2]));
    const float2 d2z = __ffma2_rn(fy2, v76, __ffma2_rn(fx2, t1[5], t1[3]));
    q[0] = fmaf(gb[2], d2x.y, fmaf(gb[1], d2x.x, gb[0] * d1x));
    q[1] = fmaf(gb[2], d2y.y, fmaf(gb[1], d2y.x, gb[0] * d1y));
    q[2] = fmaf(gb[2], d2z.y, fmaf(gb[1], d2z.x, gb[0] * d1z));
    if (b != acc.base) {
        flush(a, acc);
        acc.base = b;
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc.v[k][i] = make_float2(0.0f, 0.0f);
    }
    // corner weights: pair i = (corner 2i, 2i + 1) = X * Y * (1 - fz, fz) with
    // X = 1 - fx or fx (i >> 1), Y = 1 - fy or fy (i & 1)
    const float2 one = make_float2(1.0f, 1.0f), neg = make_float2(-1.0f, -1.0f);
    const float2 ex2 = __ffma2_rn(fx2, neg, one), ey2 = __ffma2_rn(fy2, neg, one);
    const float2 zz = __ffma2_rn(fz2, make_float2(-1.0f, 1.0f), make_float2(1.0f, 0.0f));
    const float2 xz0 = __fmul2_rn(ex2, zz), xz1 = __fmul2_rn(fx2, zz);
    const float2 w[4] = {__fmul2_rn(xz0, ey2), __fmul2_rn(xz0, fy2), __fmul2_rn(xz1, ey2), __fmul2_rn(xz1, fy2)};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float2 g2 = make_float2(gb[k], gb[k]);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc.v[k][i] = __ffma2_rn(g2, w[i], acc.v[k][i]);
    }
}

// Stage adjoint: with Abar = d L / d(stage acceleration), adds
// Abar_k * S_k * (corner weight) to the corners of the stage's cell and
// returns q = J^T (S * Abar), J = d grad(q) / d p at the stage point.
template <class P>
__device__ __forceinline__ void stage_adjoint(const ImageArgs& a, const StageRec<P>& rec,
                                              const typename P::R (&Abar)[3], typename P::R (&q)[3],
                                              GradCell<P>& cc, CornerAcc<P>& acc) {
    using R = typename P::R;
    const unsigned b = rec.b;
    if (b == kNone) {
        q[0] = q[1] = q[2] = R(0);
        return;
    }
    const R f[3] = {rec.f[0], rec.f[1], rec.f[2]};
    load_cell<P>(a, b, cc);
    const R fx = f[0], fy = f[1], fz = f[2];
    R gb[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) gb[k] = img_S<R>(a, k) * Abar[k];
    // J^T gb: derivatives of the three trilinear polynomials
    q[0] = q[1] = q[2] = R(0);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const R* t = cc.t[k];
        const R dx = (t[1] + fy * t[4]) + fz * (t[5] + fy * t[7]);
        const R dy = (t[2] + fx * t[4]) + fz * (t[6] + fx * t[7]);
        const R dz = (t[3] + fx * t[5]) + fy * (t[6] + fx * t[7]);
        q[0] += gb[k] * dx;
        q[1] += gb[k] * dy;
        q[2] += gb[k] * dz;
    }
    // corner weights, corner index 4*dx + 2*dy + dz
    if (b != acc.base) {
        flush<P>(a, acc);
        acc.base = b;
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int c = 0; c < 8; ++c) acc.v[k][c] = R(0);
    }
    const R ex = R(1) - fx, ey = R(1) - fy, ez = R(1) - fz;
    const R w00 = ex * ey, w01 = ex * fy, w10 = fx * ey, w11 = fx * fy;
    const R w[8] = {w00 * ez, w00 * fz, w01 * ez, w01 * fz, w10 * ez, w10 * fz, w11 * ez, w11 * fz};
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc.v[k][c] += gb[k] * w[c];
}

// Reverse of model_step from where its three stages sampled the field (the
// records of the recompute): (lp, lw) = adjoint of the output (p', w') on
// entry, of the input (p, w) on return. The step's stage points are
// p, p + w/2 + A1/8 and p + w + A2/2, so the chain through them needs only
// each stage's Jacobian transpose, not the step's p or w.
template <class P, class Cell, class Acc>
__device__ __forceinline__ void model_step_adjoint(const ImageArgs& a, const StageRec<P> (&rec)[3],
                                                   typename P::R (&lp)[3], typename P::R (&lw)[3], Cell& cc,
                                                   Acc& acc) {
    using R = typename P::R;
    // Direct terms of p' = p + w + (A1 + 2 A2)/6, w' = w + (A1 + 4 A2 + A3)/6:
    R a1[3], a2[3], a3[3], pb[3], wb[3], q[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        a1[x] = (lp[x] + lw[x]) * R(1.0 / 6.0);
        a2[x] = lp[x] * R(1.0 / 3.0) + lw[x] * R(2.0 / 3.0);
        a3[x] = lw[x] * R(1.0 / 6.0);
        pb[x] = lp[x];
        wb[x] = lp[x] + lw[x];
    }
    // stage 3 at p + w + A2/2
    stage_adjoint<P>(a, rec[2], a3, q, cc, acc);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        pb[x] += q[x];
        wb[x] += q[x];
        a2[x] += R(0.5) * q[x];
    }
    // stage 2 at p + w/2 + A1/8
    stage_adjoint<P>(a, rec[1], a2, q, cc, acc);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        pb[x] += q[x];
        wb[x] += R(0.5) * q[x];
        a1[x] += R(0.125) * q[x];
    }
    // stage 1 at p
    stage_adjoint<P>(a, rec[0], a1, q, cc, acc);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        lp[x] = pb[x] + q[x];
        lw[x] = wb[x];
    }
}

// ---------------------------------------------------------------------------
// Detector projection and splat.
// ---------------------------------------------------------------------------

// Splat profile g(d) and its derivative dg/dd (d and s in pixels).
template <class R>
__device__ __forceinline__ R splat_g(R d, R s, R& dg) {
    const R u = fabs(d) / s;
    if (u >= R(4)) {
        dg = R(0);
        return R(0);
    }
    R e;
    if constexpr (sizeof(R) == 4) e = expf(R(-0.5) * u * u);
    else e = exp(R(-0.5) * u * u);
    R t = R(1), dt = R(0);
    if (u > R(3)) {
        const R x = u - R(3);
        t = R(1) - x * x * x * (R(10) + x * (R(-15) + x * R(6)));
        dt = R(-30) * x * x * (R(1) - x) * (R(1) - x);
    }
    // d/dd [e(u) t(u)] with u = |d|/s
    const R sgn = d < R(0) ? R(-1) : R(1);
    dg = (e * (-u * t + dt)) * sgn / s;
    return e * t;
}

// Detector coordinates (pixels) of a final state; false if the ray never
// meets the plane or is not finite.
template <class P>
__device__ __forceinline__ bool detector_point(const ImageArgs& a, const MState<P>& r, double& pa, double& pb,
                                               double& t, double (&p)[3], double (&w)[3]) {
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        p[x] = r.p[x].vald();
        w[x] = r.w[x].vald();
    }
    const double wa = a.axis == 0 ? w[0] : (a.axis == 1 ? w[1] : w[2]);
    const double pax = a.axis == 0 ? p[0] : (a.axis == 1 ? p[1] : p[2]);
    if (!(wa != 0.0)) return false;
    t = (a.plane - pax) / wa;
    const double X = p[a.t1] + t * w[a.t1];
    const double Y = p[a.t2] + t * w[a.t2];
    pa = a.px0[0] + a.px_per_cell[0] * X;
    pb = a.px0[1] + a.px_per_cell[1] * Y;
    return isfinite(pa) && isfinite(pb) && fabs(pa) < 1e9 && fabs(pb) < 1e9;
}

// The splats of a block of rays, formed in shared memory and added to the
// image once per pixel and tile. Rays that are neighbours at entry overlap on the
// detector; adding each ray's taps to the image directly (17 x 17 reductions per
// ray at sigma = 2) serialises in L2: at 3e4 rays on 97 x 97 pixels that alone took
// 90 us. The block's first ray that is left sets a kSplatTile x kSplatTile tile with its
// window in the middle; the rays whose windows (clipped to the image) fit in it
// leave their separable weights g(i - a) * norm (rows) and g(j - b) (columns) over
// the tile in shared memory, splat_rays at a time, and pixel (r, c) = sum over rays
// of row_weight(r) * column_weight(c), a small matrix product: four groups of 64
// threads take a quarter of the rays each, a thread 4 x 4 pixels (two 16-byte
// loads per 16 multiply-adds), and the groups' sums meet in shared memory. The next ray
// left sets the next tile, kSplatRounds times at most; what is then left (rays
// far apart, or windows larger than a tile) is splatted by its warp, one ray after
// the other, its lanes on consecutive taps, so that a reduction covers whole rows of
// the window.
constexpr int kSplatRounds = 6;
// Rays that are worth a tile: its pixels are added once each, twice as many
// taps or more go into it.
__device__ __forceinline__ int splat_min(int taps) { return max(8, 2 * 32 * 32 / (taps * taps)); }
constexpr int kSplatThreads = 256;
constexpr int kSplatTile = 32;                // pixels per side of a block's tile
constexpr int kSplatPitch = kSplatTile + 4;   // 16-byte rows
template <class P> constexpr int splat_rays() { return sizeof(typename P::R) == 4 ? 64 : 32; }   // staged per round

template <class R> struct Quad { R v[4]; };
template <class R> __device__ __forceinline__ Quad<R> load_quad(const R* p) {
    Quad<R> q;
    if constexpr (sizeof(R) == 4) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        q.v[0] = x.x; q.v[1] = x.y; q.v[2] = x.z; q.v[3] = x.w;
    } else {
        const double2 x = reinterpret_cast<const double2*>(p)[0], y = reinterpret_cast<const double2*>(p)[1];
        q.v[0] = x.x; q.v[1] = x.y; q.v[2] = y.x; q.v[3] = y.y;
    }
    return q;
}

template <class P>
__global__ void __launch_bounds__(kSplatThreads) splat_kernel(const __grid_constant__ ImageArgs a) {
    using R = typename P::R;
    constexpr int kRays = splat_rays<P>(), kWarps = kSplatThreads / 32;
    __shared__ __align__(16) R s_row[kRays * kSplatPitch], s_col[kRays * kSplatPitch];
    __shared__ R s_tile[kSplatTile * kSplatTile];
    __shared__ double s_a[kSplatThreads], s_b[kSplatThreads];
    __shared__ int s_box[2], s_count[kWarps];
    static_assert(kWarps * 2 * kMaxTaps <= kRays * kSplatPitch, "the warps' tap weights share s_row");
    const int t = threadIdx.x, lane = t & 31;
    const long long slot = (long long)blockIdx.x * kSplatThreads + t;
    bool has = false;
    double pa = 0.0, pb = 0.0;
    if (slot < a.n) {
        MState<P> r;
        load_state<P>(a, a.n_seg, slot, r);
        double tt, p[3], w[3];
        has = detector_point<P>(a, r, pa, pb, tt, p, w);
    }
    int i0 = 0, j0 = 0, r0 = 0, r1 = -1, c0 = 0, c1 = -1;
    if (has) {
        i0 = (int)floor(pa - a.radius) + 1;
        j0 = (int)floor(pb - a.radius) + 1;
        r0 = max(i0, 0);
        r1 = min(i0 + a.taps - 1, a.npx[0] - 1);
        c0 = max(j0, 0);
        c1 = min(j0 + a.taps - 1, a.npx[1] - 1);
    }
    const R s = (R)a.sigma;
    R* img = reinterpret_cast<R*>(a.image);
    const int group = t >> 6, rb = 4 * ((t >> 3) & 7), cb = 4 * (t & 7), wid = t >> 5;
    bool left_over = r0 <= r1 && c0 <= c1, direct = false;
    for (int round = 0; round < kSplatRounds; ++round) {
        // the first ray that is left sets the tile
        const unsigned lmask = __ballot_sync(0xffffffffu, left_over);
        if (lane == 0) s_count[wid] = lmask ? (t + __ffs(lmask) - 1) : INT_MAX;
        __syncthreads();
        int lead = INT_MAX;
#pragma unroll
        for (int k = 0; k < kWarps; ++k) lead = min(lead, s_count[k]);
        if (lead == INT_MAX) break;        // the same in every thread
        if (t == lead) {
            s_box[0] = max((r0 + r1 + 1) / 2 - kSplatTile / 2, 0);
            s_box[1] = max((c0 + c1 + 1) / 2 - kSplatTile / 2, 0);
        }
        __syncthreads();
        const int br = s_box[0], bc = s_box[1];
        const bool tiled = left_over && r0 >= br && r1 < br + kSplatTile && c0 >= bc && c1 < bc + kSplatTile;
        // the tile's rays, compacted
        const unsigned tmask = __ballot_sync(0xffffffffu, tiled);
        if (lane == 0) s_count[wid] = __popc(tmask);
        __syncthreads();
        int before = 0, members = 0;
#pragma unroll
        for (int k = 0; k < kWarps; ++k) {
            before += k < wid ? s_count[k] : 0;
            members += s_count[k];
        }
        if (tiled) {
            const int at = before + __popc(tmask & ((1u << lane) - 1u));
            s_a[at] = pa;
            s_b[at] = pb;
        }
        __syncthreads();
        if (members < splat_min(a.taps)) {         // not worth a tile (none when the window is larger than it)
            direct = direct || tiled || t == lead;
            left_over = left_over && !direct;
            continue;
        }
        left_over = left_over && !tiled;
        R acc[4][4] = {};
        for (int base = 0; base < members; base += kRays) {
            // weights: this thread's share of 2 * kSplatTile per staged ray
            constexpr int kShare = kSplatThreads / kRays;
            const int u = t / kShare;
            const bool mine = base + u < members;
            const double qa = mine ? s_a[base + u] : 0.0, qb = mine ? s_b[base + u] : 0.0;
            for (int k = t % kShare; k < kSplatTile; k += kShare) {
                R dg;
                const int ii = br + k, jj = bc + k;
                const double di = (double)ii - qa, dj = (double)jj - qb;
                s_row[u * kSplatPitch + k] =
                    mine && fabs(di) < a.radius && ii < a.npx[0] ? splat_g<R>((R)di, s, dg) * (R)a.norm : R(0);
                s_col[u * kSplatPitch + k] = mine && fabs(dj) < a.radius && jj < a.npx[1] ? splat_g<R>((R)dj, s, dg) : R(0);
            }
            __syncthreads();
#pragma unroll 4
            for (int v = group * (kRays / 4); v < (group + 1) * (kRays / 4); ++v) {
                const Quad<R> x = load_quad(s_row + v * kSplatPitch + rb), y = load_quad(s_col + v * kSplatPitch + cb);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] += x.v[i] * y.v[j];
            }
            __syncthreads();
        }
        for (int g = 0; g < 4; ++g) {
            if (group == g) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        R& d = s_tile[(rb + i) * kSplatTile + cb + j];
                        d = g ? d + acc[i][j] : acc[i][j];
                    }
            }
            __syncthreads();
        }
        for (int k = t; k < kSplatTile * kSplatTile; k += kSplatThreads) {
            const int ii = br + k / kSplatTile, jj = bc + k % kSplatTile;
            const R v = s_tile[k];
            if (v != R(0) && ii < a.npx[0] && jj < a.npx[1]) atomicAdd(img + (size_t)ii * a.npx[1] + jj, v);
        }
    }
    __syncthreads();

    unsigned left = __ballot_sync(0xffffffffu, left_over || direct);
    if (left) {
        R* gx = s_row + (t >> 5) * 2 * kMaxTaps;
        R* gy = gx + kMaxTaps;
        const float inv = 1.0f / (float)a.taps;
        for (; left; left &= left - 1) {
            const int src = __ffs(left) - 1;
            const double qa = __shfl_sync(0xffffffffu, pa, src), qb = __shfl_sync(0xffffffffu, pb, src);
            const int qi = __shfl_sync(0xffffffffu, i0, src), qj = __shfl_sync(0xffffffffu, j0, src);
            __syncwarp();
            for (int k = lane; k < a.taps; k += 32) {
                R dg;
                gx[k] = splat_g<R>((R)((double)(qi + k) - qa), s, dg) * (R)a.norm;
                gy[k] = splat_g<R>((R)((double)(qj + k) - qb), s, dg);
            }
            __syncwarp();
            for (int k = lane; k < a.taps * a.taps; k += 32) {
                const int i = (int)(((float)k + 0.5f) * inv), j = k - i * a.taps;   // taps <= 65: exact
                const int ii = qi + i, jj = qj + j;
                if (ii >= 0 && ii < a.npx[0] && jj >= 0 && jj < a.npx[1]) {
                    const R v = gx[i] * gy[j];
                    if (v != R(0)) atomicAdd(img + (size_t)ii * a.npx[1] + jj, v);
                }
            }
        }
    }
}

// d L / d(pixel coordinates) from the image gradient.
template <class P>
__device__ __forceinline__ void splat_adjoint(const ImageArgs& a, double pa, double pb, double& ga, double& gb) {
    using R = typename P::R;
    const int i0 = (int)floor(pa - a.radius) + 1;
    const int j0 = (int)floor(pb - a.radius) + 1;
    const R s = (R)a.sigma;
    R gy[kMaxTaps], dgy[kMaxTaps];
    for (int j = 0; j < a.taps; ++j) gy[j] = splat_g<R>((R)((double)(j0 + j) - pb), s, dgy[j]);
    const R* gi = reinterpret_cast<const R*>(a.image);
    R sa = R(0), sb = R(0);
    for (int i = 0; i < a.taps; ++i) {
        const int ii = i0 + i;
        if (ii < 0 || ii >= a.npx[0]) continue;
        R dgx;
        const R gx = splat_g<R>((R)((double)ii - pa), s, dgx);
        if (gx == R(0) && dgx == R(0)) continue;
        R r0 = R(0), r1 = R(0);
        for (int j = 0; j < a.taps; ++j) {
            const int jj = j0 + j;
            if (jj < 0 || jj >= a.npx[1]) continue;
            const R v = gi[(size_t)ii * a.npx[1] + jj];
            r0 += v * gy[j];
            r1 += v * dgy[j];
        }
        // d/da g(i - a) = -g'(i - a)
        sa -= dgx * r0;
        sb -= gx * r1;
    }
    ga = (double)sa * a.norm;
    gb = (double)sb * a.norm;
}

// The tracer's interior-step test on the model state: inside the grid, and
// the prediction p + w at least kFaceMargin inside on every axis. With every
// stage acceleration below kInteriorAccel, all stage points of the step
// are then inside, and locate needs no grid test.
template <class P>
__device__ __forceinline__ bool model_interior(const ImageArgs& a, const MState<P>& r) {
    using R = typename P::R;
    const R margin = R(kFaceMargin);
    bool ok = true;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const R p = r.p[x].val(), pn = p + r.w[x].val(), lim = lim_of<R>(a.geo, x);
        ok = ok & (p >= R(0)) & (p <= lim) & (pn >= margin) & (pn <= lim - margin);
    }
    return ok;
}

// Steps after an interior step that are certainly interior too (31, 7 or 0),
// for accelerations bounded by B; the argument of the tracer's interior_run:
// j steps on, the position and the prediction lie within B (j^2 / 2 + j) of
// the segment from p + w to p + (j + 1) w.
template <class P>
__device__ __forceinline__ int model_interior_run(const ImageArgs& a, const MState<P>& r, float B) {
    using R = typename P::R;
    const R margin = R(kFaceMargin) + R(0.25);
    R p[3], w[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        p[x] = r.p[x].val();
        w[x] = r.w[x].val();
    }
    auto fits = [&](int m) {
        const R dev = margin + R(B) * R(0.5 * m * m + m);
        bool ok = true;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            const R e1 = p[x] + w[x], e2 = p[x] + R(m + 1) * w[x];
            ok = ok & (fmin(e1, e2) >= dev) & (fmax(e1, e2) <= lim_of<R>(a.geo, x) - dev);
        }
        return ok;
    };
    if (fits(31)) return 31;
    if (fits(7)) return 7;
    return 0;
}

// The acceleration bound of the fast path: infinity (no fast path) without one.
__device__ __forceinline__ float load_accel_bound(const ImageArgs& a) {
    if (!a.accel_bound) return INFINITY;
    const float b = __uint_as_float(*a.accel_bound);
    return b * 1.001f;
}

// Largest |S_k dq/du_k| over the packed grid's gradient channels. Trilinear
// interpolation stays within its corners' range, so this bounds every stage
// acceleration of the model. Non-negative floats order as their bit
// patterns, so the blocks combine with an unsigned atomicMax; a NaN channel
// gives infinity (no fast path).
template <class P>
__global__ void __launch_bounds__(256) accel_bound_kernel(const void* __restrict__ grid, size_t nvox,
                                                          double s0, double s1, double s2, unsigned* out) {
    __shared__ float s_max[8];
    float m = 0.0f;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvox; i += (size_t)gridDim.x * blockDim.x) {
        double g0, g1, g2;
        if constexpr (sizeof(typename P::R) == 4) {
            const float4 v = reinterpret_cast<const float4*>(grid)[i];
            g0 = v.y; g1 = v.z; g2 = v.w;
        } else {
            const double* d = reinterpret_cast<const double*>(grid) + 4 * i;
            g0 = d[1]; g1 = d[2]; g2 = d[3];
        }
        const double x = fmax(fabs(s0 * g0), fmax(fabs(s1 * g1), fabs(s2 * g2)));
        const bool nan = !(g0 == g0) || !(g1 == g1) || !(g2 == g2);
        const float xf = nan ? INFINITY : __double2float_ru(x);
        m = xf > m ? xf : m;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int wi = 1; wi < (int)(blockDim.x >> 5); ++wi) m = fmaxf(m, s_max[wi]);
        atomicMax(out, __float_as_uint(m));
    }
}

// ---------------------------------------------------------------------------
// Kernels.
// ---------------------------------------------------------------------------
// One warp per CTA, one thread per ray: steps to the end, a checkpoint every
// ckpt_every steps and the final state. The warp's rays run in step, so between
// checkpoints (and for as many steps as every live ray's run allows) the steps
// follow each other in a uniform loop. Bound by instruction issue (71 %, FMA pipe 64 %):
// 128^3, 1e6 rays, 400 steps in 2.92 ms (1.34e11 ray-steps/s), 183 instructions a
// ray-step; 3.26 ms and 235 before the paired step, the scalar dq/du polynomial and
// this loop.
template <class P>
__global__ void __launch_bounds__(kAdjThreads, adj_fwd_min_blocks<P>()) image_forward_kernel(const __grid_constant__ ImageArgs a) {
    using R = typename P::R;
    const long long slot = (long long)blockIdx.x * kAdjThreads + threadIdx.x;
    bool active = slot < a.n;
    MState<P> r;
    if (active) {
        const unsigned id = a.perm[slot];
        const R* rays = reinterpret_cast<const R*>(a.rays);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            r.p[x].set(((double)rays[x * a.n + id] - a.origin[x]) * a.inv_h[x]);
            r.w[x].set((double)rays[(3 + x) * a.n + id] * a.w_of_v[x]);
        }
    }
    typename AdjTypes<P>::Cell cc;
    cc.base = kNone;
    const float B = load_accel_bound(a);
    const bool fast = B <= (float)kInteriorAccel;
    int t = 0, run = 0, ck = 0, seg = 0;    // run: steps ahead that are proven interior; ck: steps to the next checkpoint
    while (__any_sync(0xffffffffu, active)) {
        bool interior = false;
        if (active) {
            if (run > 0) {                  // inside, so not gone either
                --run;
                interior = true;
            } else if (ray_gone_model<P>(a, r)) {
                active = false;
            } else if (fast && model_interior<P>(a, r)) {
                interior = true;
                run = model_interior_run<P>(a, r, B);
            }
        }
        if (active && ck == 0) {
            store_state<P>(a, seg++, slot, r);
            ck = a.ckpt_every;
        }
        const int mine = !active ? INT_MAX : (interior ? min(run, min(ck, a.n_steps - t) - 1) : 0);
        const int extra = __reduce_min_sync(0xffffffffu, mine);
        if (active) {
            if (interior) {
#pragma unroll 1
                for (int e = 0; e <= extra; ++e) model_step<true>(a, r, cc);
                run -= extra;
                ck -= extra + 1;
                t += extra + 1;
            } else {
                model_step<false>(a, r, cc);
                --ck;
                ++t;
            }
            if (t >= a.n_steps) active = false;
        }
    }
    if (slot < a.n) {
        store_state<P>(a, a.n_seg, slot, r);
        a.nsteps[slot] = t;
    }
    warp_add((unsigned long long)t, a.total_steps);
}

// In-cell coordinates of stage 1 and the first two of stage 2 of step j of
// the current segment into / out of the shared buffer (`buf` points at this
// thread's column).
template <class P>
__device__ __forceinline__ void put_step(typename P::R* buf, int j, const StageRec<P> (&rec)[3]) {
    typename P::R* b = buf + (size_t)j * kAdjStateWords * kAdjThreads;
#pragma unroll
    for (int x = 0; x < 3; ++x) b[x * kAdjThreads] = rec[0].f[x];
    b[3 * kAdjThreads] = rec[1].f[0];
    b[4 * kAdjThreads] = rec[1].f[1];
}

template <class P>
__device__ __forceinline__ void get_step(const typename P::R* buf, int j, StageRec<P> (&rec)[3]) {
    const typename P::R* b = buf + (size_t)j * kAdjStateWords * kAdjThreads;
#pragma unroll
    for (int x = 0; x < 3; ++x) rec[0].f[x] = b[x * kAdjThreads];
    rec[1].f[0] = b[3 * kAdjThreads];
    rec[1].f[1] = b[4 * kAdjThreads];
}

template <class P, int MINB>
__global__ void __launch_bounds__(kAdjThreads, MINB) image_backward_kernel(const __grid_constant__ ImageArgs a) {
    using R = typename P::R;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    R* s_seg = reinterpret_cast<R*>(s_dyn) + threadIdx.x;   // this thread's column of the segment buffer
    const long long slot = (long long)blockIdx.x * kAdjThreads + threadIdx.x;
    if (slot >= a.n) return;
    MState<P> r;
    load_state<P>(a, a.n_seg, slot, r);
    double pa, pb, t, p[3], w[3];
    if (!detector_point<P>(a, r, pa, pb, t, p, w)) return;
    double ga, gb;
    splat_adjoint<P>(a, pa, pb, ga, gb);
    // projection X = p1 + t w1, Y = p2 + t w2, t = (plane - pa) / wa
    const double Xb = ga * a.px_per_cell[0], Yb = gb * a.px_per_cell[1];
    const double wa = a.axis == 0 ? w[0] : (a.axis == 1 ? w[1] : w[2]);
    const double tb = Xb * w[a.t1] + Yb * w[a.t2];
    double lpd[3] = {0.0, 0.0, 0.0}, lwd[3] = {0.0, 0.0, 0.0};
    lpd[a.t1] = Xb;
    lwd[a.t1] = Xb * t;
    lpd[a.t2] = Yb;
    lwd[a.t2] = Yb * t;
    lpd[a.axis] = -tb / wa;
    lwd[a.axis] = -tb * t / wa;
    R lp[3], lw[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        lp[x] = (R)lpd[x];
        lw[x] = (R)lwd[x];
    }
    if (lp[0] == R(0) && lp[1] == R(0) && lp[2] == R(0) && lw[0] == R(0) && lw[1] == R(0) && lw[2] == R(0))
        return;
    const int T = a.nsteps[slot];
    typename AdjTypes<P>::Cell cc;
    cc.base = kNone;
    typename AdjTypes<P>::Acc acc;
    acc.base = kNone;
    // the three stage cells and the in-cell coordinates that the shared
    // buffer does not hold (stage 2's third, stage 3's) of each step
    unsigned segB[kMaxCkptEvery][3];
    R segF[kMaxCkptEvery][4];
    for (int s = (T + a.ckpt_every - 1) / a.ckpt_every - 1; s >= 0; --s) {
        load_state<P>(a, s, slot, r);
        const int m = min(a.ckpt_every, T - s * a.ckpt_every);
        // recompute the segment from its checkpoint (bitwise the forward's
        // steps), recording where each stage sampled. (A second loop without the
        // grid tests for segments proven interior took 1e6 rays, 128^3 from 10.3 to 10.2 ms
        // and 3e4 rays, 61^3 from 290 to 435 us: warps whose rays disagree run both.)
        StageRec<P> rec[3];
#pragma unroll 1
        for (int j = 0; j < m; ++j) {
            model_step<false>(a, r, cc, rec);
            put_step<P>(s_seg, j, rec);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                segB[j][k] = rec[k].b;
                segF[j][k] = rec[2].f[k];
            }
            segF[j][3] = rec[1].f[2];
        }
        // then its adjoint in reverse. segB / segF live in local memory, mostly
        // in L2: step j - 1's records are loaded while step j's adjoint runs
        unsigned Bn[3];
        R Fn[4];
#pragma unroll
        for (int k = 0; k < 3; ++k) Bn[k] = segB[m - 1][k];
#pragma unroll
        for (int k = 0; k < 4; ++k) Fn[k] = segF[m - 1][k];
        for (int j = m - 1; j >= 0; --j) {
            get_step<P>(s_seg, j, rec);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                rec[k].b = Bn[k];
                rec[2].f[k] = Fn[k];
            }
            rec[1].f[2] = Fn[3];
            const int jn = j > 0 ? j - 1 : 0;
#pragma unroll
            for (int k = 0; k < 3; ++k) Bn[k] = segB[jn][k];
#pragma unroll
            for (int k = 0; k < 4; ++k) Fn[k] = segF[jn][k];
            model_step_adjoint<P>(a, rec, lp, lw, cc, acc);
        }
    }
    flush(a, acc);
}

// d L / d ne from d L / d(packed grid): the transpose of K1's per-axis
// stencil (one-sided differences on the faces, central inside), times
// ne_scale. Gathers from the 6 neighbours; no atomics.
template <class P>
__device__ __forceinline__ void load_gg(const void* gg, size_t i, double (&v)[4]) {
    if constexpr (sizeof(typename P::R) == 4) {
        const float4 x = reinterpret_cast<const float4*>(gg)[i];
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
        const double* d = reinterpret_cast<const double*>(gg) + 4 * i;
        v[0] = d[0]; v[1] = d[1]; v[2] = d[2]; v[3] = d[3];
    }
}

// Transpose of one axis' stencil at index j of n: sum over the differences
// D[i] that use q[j] of d D[i] / d q[j] * Dbar[i], where Dbar[i] is channel
// `ch` of the neighbour at offset (i - j) * stride.
template <class P>
__device__ __forceinline__ double stencil_t(const void* gg, size_t v, int j, int n, size_t stride, int ch) {
    double r = 0.0, x[4];
    if (j >= 1) {          // D[j-1] holds +q[j] with weight 1 (face j-1 == 0) or 1/2
        load_gg<P>(gg, v - stride, x);
        r += (j - 1 == 0 ? 1.0 : 0.5) * x[ch];
    }
    if (j <= n - 2) {      // D[j+1] holds -q[j] with weight 1 (face j+1 == n-1) or 1/2
        load_gg<P>(gg, v + stride, x);
        r -= (j + 1 == n - 1 ? 1.0 : 0.5) * x[ch];
    }
    if (j == 0 || j == n - 1) {   // the one-sided differences on the faces use q[j] itself
        load_gg<P>(gg, v, x);
        r += (j == 0 ? -1.0 : 1.0) * x[ch];
    }
    return r;
}

template <class P, class Out>
__global__ void __launch_bounds__(256) pack_adjoint_kernel(const void* __restrict__ gg, Out* __restrict__ out,
                                                           GridGeo g, double scale) {
  // x over k (coalesced), y over j, z over i, as the pack kernel
  for (int i = blockIdx.z; i < g.n[0]; i += gridDim.z)
    for (int j = blockIdx.y; j < g.n[1]; j += gridDim.y)
      for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.n[2]; k += gridDim.x * blockDim.x) {
        const size_t vi = ((size_t)i * g.n[1] + j) * g.n[2] + k;
        double self[4];
        load_gg<P>(gg, vi, self);
        double r = self[0];
        r += stencil_t<P>(gg, vi, i, g.n[0], g.sx, 1);
        r += stencil_t<P>(gg, vi, j, g.n[1], g.sy, 2);
        r += stencil_t<P>(gg, vi, k, g.n[2], 1, 3);
        out[vi] = (Out)(r * scale);
      }
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
static int image_n_seg(const SlothImageParams* p) { return (p->n_steps + p->ckpt_every - 1) / p->ckpt_every; }

static size_t image_ws_bytes(const SlothImageParams* p, long long n) {
    const size_t nn = (size_t)(n > 0 ? n : 1);
    return workspace_bytes(n) + align256((size_t)(image_n_seg(p) + 1) * 48u * nn) + align256(4u * nn);
}

static int check_image_params(const SlothGridDesc* g, const SlothImageParams* p, int64_t n) {
    int rc = check_grid(g);
    if (rc) return rc;
    if (!p) return SLOTH_ERR_NULL_POINTER;
    if (n < 0) return SLOTH_ERR_INVALID_ARGUMENT;
    if (n > 2147483647LL) return SLOTH_ERR_TOO_LARGE;
    if (p->reserved != 0 || !(p->dtau > 0.0) || !std::isfinite(p->dtau)) return SLOTH_ERR_INVALID_ARGUMENT;
    if (p->n_steps < 1 || p->n_steps > 1000000) return SLOTH_ERR_INVALID_ARGUMENT;
    if (p->ckpt_every < 1 || p->ckpt_every > kMaxCkptEvery) return SLOTH_ERR_INVALID_ARGUMENT;
    if (p->probing_axis < 0 || p->probing_axis > 2) return SLOTH_ERR_INVALID_ARGUMENT;
    if (p->n_px[0] < 1 || p->n_px[1] < 1 || p->n_px[0] > 16384 || p->n_px[1] > 16384) return SLOTH_ERR_INVALID_ARGUMENT;
    if (!(p->sigma_px > 0.0) || !(p->sigma_px <= 8.0)) return SLOTH_ERR_INVALID_ARGUMENT;
    if (!std::isfinite(p->plane)) return SLOTH_ERR_INVALID_ARGUMENT;
    for (int k = 0; k < 4; ++k)
        if (!std::isfinite(p->window[k])) return SLOTH_ERR_INVALID_ARGUMENT;
    if (!(p->window[1] > p->window[0]) || !(p->window[3] > p->window[2])) return SLOTH_ERR_INVALID_ARGUMENT;
    return SLOTH_OK;
}

static void fill_image_args(ImageArgs& a, const SlothGridDesc* g, const void* grid, const SlothImageParams* p,
                            const void* rays, long long n, const unsigned* perm, void* ckpt, int* nsteps) {
    a.geo = make_geo(g);
    a.grid = grid;
    a.rays = rays;
    a.n = n;
    a.perm = perm;
    for (int k = 0; k < 3; ++k) {
        const double h = g->spacing[k];
        a.origin[k] = g->origin[k];
        a.inv_h[k] = 1.0 / h;
        a.w_of_v[k] = (p->dtau / h) / kC;
        a.S[k] = -0.5 * (p->dtau / h) * (p->dtau / h);
        a.Sf[k] = (float)a.S[k];
        a.S4f[k] = 0.25f * a.Sf[k];
        a.S2f[k] = 0.5f * a.Sf[k];
        a.S6f[k] = (1.0f / 6.0f) * a.Sf[k];
    }
    a.n_steps = p->n_steps;
    a.ckpt_every = p->ckpt_every;
    a.n_seg = image_n_seg(p);
    a.axis = p->probing_axis;
    a.t1 = a.axis == 0 ? 1 : 0;
    a.t2 = a.axis == 2 ? 1 : 2;
    a.plane = (p->plane - g->origin[a.axis]) / g->spacing[a.axis];
    const int tr[2] = {a.t1, a.t2};
    for (int d = 0; d < 2; ++d) {
        const double lo = p->window[2 * d], hi = p->window[2 * d + 1];
        const double pix = (hi - lo) / p->n_px[d];
        a.px_per_cell[d] = g->spacing[tr[d]] / pix;
        a.px0[d] = (g->origin[tr[d]] - lo) / pix - 0.5;
        a.npx[d] = p->n_px[d];
    }
    a.sigma = p->sigma_px;
    a.radius = 4.0 * p->sigma_px;
    a.taps = 2 * (int)ceil(a.radius) + 1;
    a.norm = 1.0 / (2.0 * 3.141592653589793 * p->sigma_px * p->sigma_px);
    a.ckpt = ckpt;
    a.nsteps = nsteps;
    a.image = nullptr;
    a.ggrad = nullptr;
    a.total_steps = nullptr;
    a.accel_bound = nullptr;
}

struct ImageWs {
    unsigned *hist, *keys, *perm, *offs;
    void* ckpt;
    int* nsteps;
    unsigned* bound;    // acceleration bound of the forward (float bits), in the header's second half
};

static ImageWs carve(void* ws, const SlothImageParams* p, long long n) {
    ImageWs w;
    char* base = reinterpret_cast<char*>(ws);
    const size_t a = align256((size_t)(n > 0 ? n : 1) * 4u);
    w.bound = reinterpret_cast<unsigned*>(base + kHeaderBytes / 2);
    w.hist = reinterpret_cast<unsigned*>(base + kHeaderBytes);
    w.keys = reinterpret_cast<unsigned*>(base + kHeaderBytes + kHistBytes);
    w.perm = reinterpret_cast<unsigned*>(base + kHeaderBytes + kHistBytes + a);
    w.offs = reinterpret_cast<unsigned*>(base + kHeaderBytes + kHistBytes + 2 * a);
    char* c = base + workspace_bytes(n);
    w.ckpt = c;
    w.nsteps = reinterpret_cast<int*>(c + align256((size_t)(image_n_seg(p) + 1) * 48u * (size_t)(n > 0 ? n : 1)));
    return w;
}

// The acceleration bound of the interior fast path into the workspace.
template <class P>
static int launch_accel_bound(const SlothGridDesc* g, const void* grid, const ImageArgs& a, unsigned* bound, int sms,
                              cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(bound, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return cuda_status(e);
    const size_t vox = (size_t)g->n[0] * g->n[1] * g->n[2];
    const size_t want = (vox + 255) / 256, cap = (size_t)sms * 8;
    accel_bound_kernel<P><<<(unsigned)(want < cap ? want : cap), 256, 0, s>>>(grid, vox, fabs(a.S[0]), fabs(a.S[1]),
                                                                               fabs(a.S[2]), bound);
    note_launch();
    return cuda_status(cudaGetLastError());
}

template <class P>
static int image_forward_impl(const SlothGridDesc* g, const void* grid, const SlothImageParams* p,
                              const typename P::R* rays, int64_t n, typename P::R* image,
                              unsigned long long* total_steps, void* ws, size_t ws_bytes, void* stream) {
    int rc = check_image_params(g, p, n);
    if (rc) return rc;
    if (!grid || !image || !ws || (n > 0 && !rays)) return SLOTH_ERR_NULL_POINTER;
    if (((uintptr_t)grid & 15u) || ((uintptr_t)ws & 255u) || ((uintptr_t)image & (sizeof(typename P::R) - 1)) ||
        ((uintptr_t)rays & (sizeof(typename P::R) - 1)))
        return SLOTH_ERR_MISALIGNED;
    if (ws_bytes < image_ws_bytes(p, n)) return SLOTH_ERR_WORKSPACE_TOO_SMALL;
    int sms = 148;
    if ((rc = device_sm_count(&sms)) != SLOTH_OK) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaMemsetAsync(image, 0, sizeof(typename P::R) * (size_t)p->n_px[0] * p->n_px[1], s);
    if (e != cudaSuccess) return cuda_status(e);
    if (n == 0) return SLOTH_OK;
    ImageWs w = carve(ws, p, n);
    // One thread per ray in bucket order: buckets of few rays keep a warp's
    // rays in few cells, so that its cell loads and gradient flushes share
    // addresses.
    const int bbits = bucket_bits_for(n);
    rc = launch_prepass<typename P::R>(g, p->probing_axis, rays, n, bbits, w.keys, w.hist, w.perm, w.offs, nullptr,
                                       nullptr, sms, s);
    if (rc) return rc;
    ImageArgs a;
    fill_image_args(a, g, grid, p, rays, n, w.perm, w.ckpt, w.nsteps);
    a.image = image;
    a.total_steps = total_steps;
    if ((rc = launch_accel_bound<P>(g, grid, a, w.bound, sms, s)) != SLOTH_OK) return rc;
    a.accel_bound = w.bound;
    image_forward_kernel<P><<<(unsigned)((n + kAdjThreads - 1) / kAdjThreads), kAdjThreads, 0, s>>>(a);
    note_launch();
    splat_kernel<P><<<(unsigned)((n + kSplatThreads - 1) / kSplatThreads), kSplatThreads, 0, s>>>(a);
    note_launch();
    return cuda_status(cudaGetLastError());
}

template <class P>
static int image_backward_impl(const SlothGridDesc* g, const void* grid, const SlothImageParams* p, int64_t n,
                               const typename P::R* image_grad, void* grid_grad, void* ws, size_t ws_bytes,
                               void* stream) {
    int rc = check_image_params(g, p, n);
    if (rc) return rc;
    if (!grid || !image_grad || !grid_grad || !ws) return SLOTH_ERR_NULL_POINTER;
    if (((uintptr_t)grid & 15u) || ((uintptr_t)grid_grad & 15u) || ((uintptr_t)ws & 255u) ||
        ((uintptr_t)image_grad & (sizeof(typename P::R) - 1)))
        return SLOTH_ERR_MISALIGNED;
    if (ws_bytes < image_ws_bytes(p, n)) return SLOTH_ERR_WORKSPACE_TOO_SMALL;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t vox = (size_t)g->n[0] * g->n[1] * g->n[2];
    cudaError_t e = cudaMemsetAsync(grid_grad, 0, vox * 4 * sizeof(typename P::R), s);
    if (e != cudaSuccess) return cuda_status(e);
    if (n == 0) return SLOTH_OK;
    ImageWs w = carve(ws, p, n);
    ImageArgs a;
    fill_image_args(a, g, grid, p, nullptr, n, w.perm, w.ckpt, w.nsteps);
    a.image = const_cast<typename P::R*>(image_grad);
    a.ggrad = grid_grad;
    const size_t smem = (size_t)p->ckpt_every * kAdjStateWords * sizeof(typename P::R) * kAdjThreads;
    const unsigned blocks = (unsigned)((n + kAdjThreads - 1) / kAdjThreads);
    auto launch = [&](auto kernel) {
        cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err == cudaSuccess) kernel<<<blocks, kAdjThreads, smem, s>>>(a);
        return err;
    };
    if constexpr (sizeof(typename P::R) == 4) {
        int dev = 0, per_sm = 0, reserved = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
            (e = cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess ||
            (e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev)) != cudaSuccess)
            return cuda_status(e);
        if (16 * (smem + (size_t)reserved) <= (size_t)per_sm)
            e = launch(image_backward_kernel<P, 16>);
        else
            e = launch(image_backward_kernel<P, 12>);
    } else {
        e = launch(image_backward_kernel<P, 8>);
    }
    if (e != cudaSuccess) return cuda_status(e);
    note_launch();
    return cuda_status(cudaGetLastError());
}

template <class P, class Out>
static int pack_adjoint_impl(const SlothGridDesc* g, const void* grid_grad, double ne_scale, Out* ne_grad,
                             void* stream) {
    int rc = check_grid(g);
    if (rc) return rc;
    if (!grid_grad || !ne_grad) return SLOTH_ERR_NULL_POINTER;
    if (!(ne_scale > 0.0) || !std::isfinite(ne_scale)) return SLOTH_ERR_INVALID_ARGUMENT;
    if (((uintptr_t)grid_grad & 15u) || ((uintptr_t)ne_grad & (sizeof(Out) - 1))) return SLOTH_ERR_MISALIGNED;
    int sms = 148;
    if ((rc = device_sm_count(&sms)) != SLOTH_OK) return rc;
    const dim3 grid((unsigned)((g->n[2] + 255) / 256), (unsigned)(g->n[1] < 65535 ? g->n[1] : 65535),
                    (unsigned)(g->n[0] < 65535 ? g->n[0] : 65535));
    pack_adjoint_kernel<P, Out><<<grid, 256, 0, (cudaStream_t)stream>>>(grid_grad, ne_grad, make_geo(g), ne_scale);
    note_launch();
    return cuda_status(cudaGetLastError());
}

}  // namespace sloth

extern "C" {

size_t sloth_image_workspace_bytes(const SlothImageParams* p, int64_t n) {
    if (!p || p->ckpt_every < 1 || p->n_steps < 1 || n < 0) return 0;
    return sloth::image_ws_bytes(p, n);
}

int sloth_image_forward_f32(const SlothGridDesc* g, const void* grid, const SlothImageParams* p, const float* rays,
                            int64_t n, float* image, unsigned long long* total_steps, void* ws, size_t ws_bytes,
                            void* stream) {
    return sloth::image_forward_impl<sloth::PolF32>(g, grid, p, rays, n, image, total_steps, ws, ws_bytes, stream);
}

int sloth_image_forward_f64(const SlothGridDesc* g, const void* grid, const SlothImageParams* p, const double* rays,
                            int64_t n, double* image, unsigned long long* total_steps, void* ws, size_t ws_bytes,
                            void* stream) {
    return sloth::image_forward_impl<sloth::PolF64>(g, grid, p, rays, n, image, total_steps, ws, ws_bytes, stream);
}

int sloth_image_backward_f32(const SlothGridDesc* g, const void* grid, const SlothImageParams* p, int64_t n,
                             const float* image_grad, void* grid_grad, void* ws, size_t ws_bytes, void* stream) {
    return sloth::image_backward_impl<sloth::PolF32>(g, grid, p, n, image_grad, grid_grad, ws, ws_bytes, stream);
}

int sloth_image_backward_f64(const SlothGridDesc* g, const void* grid, const SlothImageParams* p, int64_t n,
                             const double* image_grad, void* grid_grad, void* ws, size_t ws_bytes, void* stream) {
    return sloth::image_backward_impl<sloth::PolF64>(g, grid, p, n, image_grad, grid_grad, ws, ws_bytes, stream);
}

int sloth_grid_pack_adjoint_f32(const SlothGridDesc* g, const void* grid_grad, double ne_scale, float* ne_grad,
                                void* stream) {
    return sloth::pack_adjoint_impl<sloth::PolF32, float>(g, grid_grad, ne_scale, ne_grad, stream);
}

int sloth_grid_pack_adjoint_f64(const SlothGridDesc* g, const void* grid_grad, double ne_scale, double* ne_grad,
                                void* stream) {
    return sloth::pack_adjoint_impl<sloth::PolF64, double>(g, grid_grad, ne_scale, ne_grad, stream);
}

}  // extern "C"
