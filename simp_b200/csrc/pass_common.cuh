// Shared device code of the two pair passes of one right-hand-side evaluation (single_step.f90:5-109)
// and the predictor-corrector update fused into the second pass's epilogue.
//
// Kinematic pass (single_step.f90:50-84 + internal_stress.f90:20-42), per
// particle i: the exact criterion and the pair math over its candidates (a
// Verlet list, built first where the basin's are stale):
//        wdvx = (v_i - v_j) (x) grad W_ij            (kernel.f90:515-518)
//        div_i  -= m_j (wdvx1 + wdvx4)               (vector_divergence.f90:27)
//        grad_i -= m_j wdvx / rho_j                  (vector_gradient.f90:56-69)
//   then strain (single_step.f90:80-84), strength, bulk and shear viscosity,
//   replacement pressure and stress (bulk_viscosity.f90:65-76,
//   shear_viscosity.f90:57, eos.f90:141-147, stress_tensor.f90:31-39).
//   Writes tau = sigma / rho^2 and div.
//
// Stress pass (internal_stress.f90:103-137 stress_1, boundary_kernel.f90 +
// boundary_force.f90:74-84, wind_forcing.f90:35-51, water_drag.f90:35-53,
// single_step.f90:104-106) over the kinematic pass's pairs:
//   a_i = rho_i / (rho_ice h_i) sum_j m_j (tau_i + tau_j) . grad W_ij
//         - sum_walls F_b / rho_i + wind + water drag
//   followed by one of three epilogues: the rates (single_step), the
//   predictor half step (time_integration.f90:204-227) or the corrector and
//   final update (:343-388).
//
// Each pair is evaluated from both sides (gather form, no atomics on the
// accumulations); grad W is odd in dx so both sides see the same per-pair
// terms as the reference's scatter loop, summed in a different order.
//
// Where the neighbours' data comes from: tile.cuh.
#pragma once

#include <cmath>

#include "ctx.h"
#include "neighbors.cuh"

namespace simp {
namespace pass {

// Pair arithmetic type T: double for the plain form, float for the mixed
// form.  Positions and velocities stay FP64; their differences are formed in
// FP64 and rounded to T, after which the kernel gradient and the pair sums
// run in T (compensated when T is float).
__device__ __forceinline__ double rsq(double v) { return rsqrt(v); }
__device__ __forceinline__ float rsq(float v) { return rsqrtf(v); }

// Sum of pair terms a * b: plain FP64, or FP32 with Kahan compensation.
// Every multiply-add of the pair arithmetic is an explicit fma, so the
// rounding does not depend on which products a compiler chooses to fuse
// (both pass implementations then give the same bits).
template <class T>
struct Sum {
    double s = 0.0;
    __device__ __forceinline__ void madd(double a, double b) { s = fma(a, b, s); }
    __device__ __forceinline__ double get() const { return s; }
};
template <>
struct Sum<float> {
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void madd(float a, float b) {
        const float y = fmaf(a, b, -c);
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ double get() const { return (double)s - (double)c; }
};

// Per-pair geometry and kernel gradient: dw = gfac * (dx, dy).
// r = s * rsqrt(s) and 1/hsml_ij from the particle's own 1/hsml when the two
// smoothing lengths are equal (then hsml_ij = hsml_i exactly).
template <class T>
struct PairGeom {
    T dx, dy, gfac, w;
};

// dx, dy: x_i - x_j (differences of the FP64 positions, rounded to T);
// hi, inv_hi, hj: the smoothing lengths in T (the FP32 copies in the mixed
// form).
template <class T, bool WANT_W, int SKF = 0>
__device__ __forceinline__ PairGeom<T> pair_geom(const Phys &P, T dx, T dy, T hi, T inv_hi, T hj) {
    PairGeom<T> g;
    g.dx = dx;
    g.dy = dy;
    const T s = fma(g.dx, g.dx, g.dy * g.dy);
    const T rs = rsq(s);
    const T r = s * rs;
    const T inv_h = (hj == hi) ? inv_hi : T(2) / (hi + hj);
    const T sh = (T)P.scale_h;
    const T shh = sh * inv_h;
    const T q = r * shh;
    T gq, w = 0;
    kernel_wg<T, WANT_W, SKF>(P.skf, q, shh, inv_h, &w, &gq);
    if (WANT_W) g.w = w;
    g.gfac = gq * shh * rs;
    return g;
}

// sqrt(u) and 1 / (2 sqrt(u)).  FP64, from the hardware's approximate
// reciprocal root (relative error 2^-20): a round of Goldschmidt's coupled
// iteration (g -> sqrt(u), h -> 1 / (2 sqrt(u)), r = 1/2 - g h) to 2^-39, then
// one correction of both: with d = u - g^2, sqrt(u) = g + d h, and the deviation
// of 2 h sqrt(u) from 1 is 2 (d h^2 - r).  What is left is the last rounding
// (largest error over 3 million arguments: 1.00 of 2^-53; u * rsqrt(u)
// and rsqrt(u) have 1.49 and 1.00).  Unlike rsqrt() it has no branch for subnormal
// arguments, which a squared distance is not, so that two pairs' roots
// interleave.  u = 0 gives NaN, as rsqrt(0) * 0 does.
__device__ __forceinline__ void root_pair(double u, double &g, double &h) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(u));
    g = u * y;
    h = 0.5 * y;
    double r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    const double e = fma(-g, g, u) * h;
    r = fma(-e, h, fma(-g, h, 0.5));
    g += e;
    h = fma(h + h, r, h);
}
__device__ __forceinline__ void root_pair(float u, float &g, float &h) {
    const float y = rsqrtf(u);
    g = u * y;
    h = 0.5f * y;
}

// grad W_ij = g (x_i - x_j) of the compiled kernels, split so that a uniform
// hsml costs nothing per pair: g = scale * shape, where the shape depends on
// q^2 alone and the scale on hsml_ij.  With H = hsml_ij, R = sqrt(r^2 H^2) = r H
// and n = 1 / (2 R): q / scale_h = r / H = 2 r^2 n and 1 / H^2 = 4 r^2 n^2, so
// one root gives both without a division.
//   cubic (kernel.f90:324-340), q = 2 r / H: dW/dq / q is 1.5 q - 2 up to
//     q = 1 and -(2 - q)^2 / (2 q) beyond, scale 15/(7 pi) (2 / H)^4;
//   Wendland C6 (kernel.f90:499-508), q = r / H: -22 (1 - q)^7 (16 q^2 +
//     7 q + 1), scale 78/(7 pi) / H^4.
template <class T, int SKF>
struct Grad;
template <class T>
struct Grad<T, SIMP_SKF_CUBIC> {
    static constexpr double factor = 15.0 / (7.0 * kPi) * 16.0;
    static constexpr double qscale = 2.0;
    // h = 1 / (2 q)
    static __device__ __forceinline__ T shape(T q, T h) {
        const T u = T(2) - q;
        return q <= T(1) ? fma(T(1.5), q, T(-2)) : -(u * u) * h;
    }
};
template <class T>
struct Grad<T, SIMP_SKF_WENDLAND_C6> {
    static constexpr double factor = 78.0 / (7.0 * kPi);
    static constexpr double qscale = 1.0;
    static __device__ __forceinline__ T shape(T q, T) {
        const T om = T(1) - q, om2 = om * om;
        return (T(-22) * (om2 * om2) * (om2 * om)) * fma(fma(T(16), q, T(7)), q, T(1));
    }
};

// What a launch knows of its basins' hsml: one value in each of them; not so (a
// single basin, or one whose hsml evolves); or so in some of a batch's, each of
// which then gets the very operations of the first form, so that its sums do not
// depend on which basins it is batched with.  (The last form selects operand by
// operand: a branch would part the chains of a particle's two candidates.  As a
// form for single basins too it costs the reference's switches at 90,007
// particles 122 -> 127 us per step.)
enum Hsml : int { HSML_ONE, HSML_VARIED, HSML_EITHER };

// The pair's gradient factor without the constant part of a particle's sums,
// from s = r^2.
template <class T, int SKF, int HS>
struct PairGrad {
    T hi, k;   // hsml_i; where hsml is one value: (qscale / hsml)^2
    T inv_hi;  // (generic kernels)
    bool one;
    __device__ __forceinline__ void init(const Phys &P, const Inst &I, T h) {
        hi = h;
        one = HS == HSML_ONE || (HS == HSML_EITHER && I.hmin == I.hmax);
        if (SKF == 0) {
            inv_hi = T(1) / h;
        } else if (HS != HSML_VARIED) {
            k = (T)I.grad_k;
        }
    }
    // factor common to all pairs of the particle
    __device__ __forceinline__ double common(const Inst &I) const {
        if (SKF == 0) return 1.0;
        return HS == HSML_VARIED || !one ? Grad<T, SKF ? SKF : SIMP_SKF_CUBIC>::factor : I.grad_c;
    }
    __device__ __forceinline__ T operator()(const Phys &P, T s, T hj) const {
        if constexpr (SKF == 0) {
            const T rs = rsq(s), r = s * rs;
            const T inv_h = (HS == HSML_ONE || hj == hi) ? inv_hi : T(2) / (hi + hj);
            const T shh = (T)P.scale_h * inv_h;
            T w = 0, gq;
            kernel_wg<T, false, 0>(P.skf, r * shh, shh, inv_h, &w, &gq);
            return gq * shh * rs;
        } else if constexpr (HS == HSML_ONE) {
            T q, h;
            root_pair(s * k, q, h);
            return Grad<T, SKF>::shape(q, h);
        } else {
            constexpr T c = (T)Grad<T, SKF>::qscale;
            const T H = T(0.5) * (hi + hj), H2 = H * H;
            T R, n;
            const bool o = HS == HSML_EITHER && one;
            root_pair(s * (o ? k : H2), R, n);
            const T q = T(2) * s * n, ih2 = T(2) * q * n;   // r / H, 1 / H^2
            return (o ? T(1) : ih2 * ih2) * Grad<T, SKF>::shape(o ? R : c * q, (o ? T(1) : H2 / c) * n);
        }
    }
};

// Stress-pass records written by the kinematic pass: (tau11, tau12),
// (tau22, m), and what the mixed form's neighbours read, (tau11, tau12,
// tau22, m) in FP32.
struct TauRec {
    double2 *ta, *tb;
    float4 *tq;         // mixed form
};

// Kinematic-pass pair terms (kernel.f90:515-518, vector_divergence.f90:27,
// vector_gradient.f90:56-69): sums of -div and of the velocity gradient, whose
// off-diagonal parts are only needed added (the shear strain rate).
template <class T>
struct KinSums {
    Sum<T> dv, g1, g23, g4;
    // grad W_ij = (dwx, dwy); nothing is added where `in` is false
    __device__ __forceinline__ void add(bool in, T dwx, T dwy, T dvx, T dvy, T mj, T mrj) {
        const T w1 = dvx * dwx, w4 = dvy * dwy;
        const T w23 = fma(dvy, dwx, dvx * dwy);
        if (in) {
            dv.madd(mj, w1 + w4);
            g1.madd(mrj, w1);
            g23.madd(mrj, w23);
            g4.madd(mrj, w4);
        }
    }
};

// Stress-pass pair terms (internal_stress.f90:103-137): sum_j m_j grad W
// and sum_j m_j tau_j . grad W.
template <class T>
struct StressSums {
    Sum<T> sx, sy, tx, ty;
    int pairs = 0;
    // (nothing is added where `in` is false)
    __device__ __forceinline__ void add(bool in, T dwx, T dwy, T mj, T t11, T t12, T t22) {
        const T fx = fma(t11, dwx, t12 * dwy), fy = fma(t12, dwx, t22 * dwy);
        if (in) {
            sx.madd(mj, dwx);
            sy.madd(mj, dwy);
            tx.madd(mj, fx);
            ty.madd(mj, fy);
        }
    }
};

struct KinArgs {
    State s;
    const double2 *xyr;    // sort positions
    const int *cell_start, *bstart;
    const Inst *inst;
    const int *cell;
    Phys P;
    Scalars *sc;
    double *div;
    TauRec rec;            // the stress pass's records (written here)
    double *diag;
    PairList pl;
    int maxn;
    const Chunk *chunks;   // tile of each block
    unsigned char *halos;  // their halos (written here)
    unsigned char *halo_walls;
    int cap;               // halo particles that fit in shared memory
    int second;            // the step's second right-hand side
    int single;            // instance 0 owns every particle
    int prefetch;          // fetch the epilogue's values ahead
};

// Strain rates, rheology and stress of particle i from its velocity
// divergence dv and velocity gradient (g1, g23 / 2, g4) (single_step.f90:80-84,
// internal_stress.f90:20-42): writes tau = sigma / rho^2, div and the
// optional diagnostics.
__device__ __forceinline__ void kin_rheology(const KinArgs &a, int i, double dv, double g1, double g23, double g4) {
    const State &s = a.s;
    const Phys &P = a.P;
    // strain rates, single_step.f90:80-84
    const double e11 = g1, e22 = g4, e12 = 0.5 * g23;
    // rheology, internal_stress.f90:20-42
    const double hh = s.h[i], AA = s.A[i];
    const double rho = s.rho[i];
    const double em2 = P.em2;
    const double Pstr = P.P_star * hh * exp(-(P.c_eos * (1.0 - AA)));
    const double delta = sqrt(fma(fma(e11, e11, e22 * e22), 1.0 + em2,
                                  fma(4.0 * em2, e12 * e12, 2.0 * e11 * e22 * (1.0 - em2))));
    const double dcap = (fabs(delta) < P.delta_min) ? P.delta_min : delta;
    double zeta = 0.0, eta = 0.0, p = 0.0;
    if (P.viscosity) {
        p = Pstr;
        if (P.rheology == 2) {
            // Mohr-Coulomb, bulk_viscosity.f90:86-145 and shear_viscosity.f90:67-124
            const double root = sqrt(fma(e11 - e22, e11 - e22, 4.0 * (e12 * e12)));
            const double eps1 = 0.5 * ((e11 + e22) + root), eps2 = 0.5 * ((e11 + e22) - root);
            const double zero = 1.0e-18;
            double epsI = fabs(eps1 + eps2);
            if (epsI < zero) epsI = zero;
            zeta = 0.5 * p * (1.0 + P.k_t) / epsI;
            if (zeta > P.zeta_max * p) zeta = P.zeta_max * p;
            double epsII = eps1 - eps2;
            if (fabs(epsII) < zero) epsII = zero;
            eta = P.mu * (0.5 * p * (1.0 + P.k_t) - zeta * (eps1 + eps2)) / epsII;
            if (eta > P.eta_max * p) eta = P.eta_max * p;
        } else {
            // elliptical, bulk_viscosity.f90:65-76 and shear_viscosity.f90:57
            zeta = 0.5 * Pstr * (1.0 + P.k_t) / dcap;
            eta = zeta * em2;
        }
    }
    if (P.pressure_force) {   // eos.f90:20-31
        if (P.eos_alg == 3) {
            p = zeta * 2.0 * delta * P.inv_1kt;               // Kreyscher :141-147
        } else if (P.eos_alg == 2) {
            // Gutfraind :96-104 (rho_0 = rho_ice, rho_max = 934)
            const double gamma = 1.9e5 * hh * exp(-20.0 * (1.0 - AA));
            p = gamma * (rho - P.rho_ice) / (934.0 - rho);
            if (p < 0.0) p = 0.0;
        } else {
            p = Pstr;                                         // Hibler :59
        }
    }
    const double ph = p * (1.0 - P.k_t) / 2.0;
    const double s11 = fma(zeta + eta, e11, fma(zeta - eta, e22, -ph));
    const double s12 = 2.0 * eta * e12;
    const double s22 = fma(zeta + eta, e22, fma(zeta - eta, e11, -ph));
    // stress_1 pairs sigma / rho^2 with m; stress_2 pairs sigma with m / rho
    // (internal_stress.f90:103-137, 146-219)
    const double ir2 = (P.pa_sph == 2) ? 1.0 : 1.0 / (rho * rho);
    const double2 mm = s.mm[i];
    const double mw = (P.pa_sph == 2) ? mm.y : mm.x;
    const double t11 = s11 * ir2, t12 = s12 * ir2, t22 = s22 * ir2;
    a.rec.ta[i] = make_double2(t11, t12);
    a.rec.tb[i] = make_double2(t22, mw);
    if (a.rec.tq) a.rec.tq[i] = make_float4((float)t11, (float)t12, (float)t22, (float)mw);
    a.div[i] = dv;
    if (a.diag) {
        const size_t M = (size_t)a.maxn;
        a.diag[i] = e11;
        a.diag[M + i] = e12;
        a.diag[2 * M + i] = e22;
        a.diag[3 * M + i] = zeta;
        a.diag[4 * M + i] = eta;
        a.diag[5 * M + i] = p;
        a.diag[6 * M + i] = s11;
        a.diag[7 * M + i] = s12;
        a.diag[8 * M + i] = s22;
    }
}

struct StressArgs {
    State rhs;     // state the right-hand side is evaluated at
    State base;    // step-start state (own values for the integrator)
    State out;     // state written by the epilogue
    const int *cell_start;
    Inst *inst;
    const int *cell;
    const double *bx, *by, *bm;
    const double *bnx, *bny;   // wall normals (bfa = 2)
    const int *bstart;
    int nb;
    Phys P;
    Scalars *sc;
    const double *div;
    TauRec rec;
    PairList pl;
    double *rates;
    // regularisation terms of this right-hand side (k_regularize), 4 maxn:
    // the artificial-viscosity acceleration (x, y) and the XSPH sum (x, y),
    // which a rates epilogue replaces by dx/dt; null when both are off
    double *reg;
    double *hs_next;
    int maxn, mode, single, prefetch;
    const Chunk *chunks;
    const unsigned char *halos, *halo_walls;
    int cap;
};

// The two passes' kernels, compiled by kernel function and precision
// (pass_kernels.cuh), for an hsml form (Hsml) and resident blocks per SM.
struct PassForm {
    void (*kin)(KinArgs);
    void (*stress)(StressArgs);
};
PassForm passes_cubic_fp64(int hs, int blocks);
PassForm passes_cubic_mixed(int hs, int blocks);
PassForm passes_wendland_fp64(int hs, int blocks);
PassForm passes_wendland_mixed(int hs, int blocks);
PassForm passes_generic_fp64(int hs, int blocks);
PassForm passes_generic_mixed(int hs, int blocks);

// Max / min of 64-bit values over a warp, word by word.
__device__ __forceinline__ unsigned long long warp_top(unsigned long long v) {
    const unsigned hi = (unsigned)(v >> 32), H = __reduce_max_sync(0xffffffffu, hi);
    const unsigned L = __reduce_max_sync(0xffffffffu, hi == H ? (unsigned)v : 0u);
    return ((unsigned long long)H << 32) | L;
}
__device__ __forceinline__ unsigned long long warp_least(unsigned long long v) { return ~warp_top(~v); }

// Block-wide max folded into one device atomic per block (the
// same-address atomics of every warp would serialise in L2).  Called by all
// threads of the block at the same point.
__device__ __forceinline__ void block_max_u64(unsigned long long *dst, unsigned long long v) {
    __shared__ unsigned long long part[32];
    v = warp_top(v);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) v = part[w] > v ? part[w] : v;
        atomicMax(dst, v);
    }
    __syncthreads();
}
__device__ __forceinline__ void block_max_i32(int *dst, int v) {
    __shared__ int part[32];
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) v = max(v, part[w]);
        atomicMax(dst, v);
    }
    __syncthreads();
}

// The per-step bounds of the stress pass in one block-wide reduction (two
// warp reductions per value, one barrier, one atomic per value and block): of
// the run, maxip (max), the next hsml minimum and maximum and the VP time step
// (min); of the block's instance, the squared move of this update (max, into
// `move`), from which the step's end keeps the bounds on displacements and
// coordinates.  Values whose bit in `active` is clear are skipped.  Every
// thread of the block calls it.
constexpr int kBounds = 5;
__device__ __forceinline__ void block_bounds(Scalars *sc, unsigned long long *move, unsigned active,
                                             unsigned long long (&v)[kBounds]) {
    __shared__ unsigned long long part[kTile / 32][kBounds];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < kBounds; ++q) {
        if (!((active >> q) & 1u)) continue;
        const bool mn = (q == 1 || q == 3);
        const unsigned long long r = q == 0 ? (unsigned long long)__reduce_max_sync(0xffffffffu, (unsigned)v[0])
                                            : mn ? warp_least(v[q]) : warp_top(v[q]);
        if (lane == 0) part[w][q] = r;
    }
    __syncthreads();
    const int q = threadIdx.x;
    if (q < kBounds && ((active >> q) & 1u)) {
        const bool mn = (q == 1 || q == 3);
        unsigned long long r = part[0][q];
#pragma unroll
        for (int k = 1; k < kTile / 32; ++k) {
            const unsigned long long t = part[k][q];
            r = mn ? (t < r ? t : r) : (t > r ? t : r);
        }
        switch (q) {
            case 0: atomicMax(&sc->maxip, (int)r); break;
            case 1: atomicMin(&sc->acc_hmin, r); break;
            case 2: atomicMax(&sc->acc_hmax, r); break;
            case 3: atomicMin(&sc->acc_dt, r); break;
            default: atomicMax(move, r); break;
        }
    }
}

// Wall pairs of a particle (boundary_kernel.f90:5-45 calling boundary_force.f90
// once per pair): the sum of F_b, applied as -F_b / rho, and the acceleration
// terms added as they are.
struct WallSums {
    double fx = 0.0, fy = 0.0, gx = 0.0, gy = 0.0;
    int cnt = 0;
};

// What stress_finish will read of particle i, brought to the L1 cache while the
// pairs are summed.
template <class P>
__device__ __forceinline__ void prefetch_l1(const P *p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}
__device__ __forceinline__ void stress_prefetch(const StressArgs &a, int i) {
    const State &s = a.rhs, &b = a.base;
    prefetch_l1(&s.rho[i]);
    prefetch_l1(&s.h[i]);
    prefetch_l1(&s.A[i]);
    prefetch_l1(&a.div[i]);
    prefetch_l1(&a.rec.ta[i]);
    prefetch_l1(&a.rec.tb[i]);
    prefetch_l1(&s.vxy[i]);
    prefetch_l1(&b.m[i]);
    if (a.mode == EPI_CORRECT || a.mode == EPI_LEAP) {
        prefetch_l1(&b.xy[i]);
        prefetch_l1(&b.vxy[i]);
        prefetch_l1(&b.h[i]);
        prefetch_l1(&b.A[i]);
    }
}

// Everything of the stress pass after the pair sums S = sum_j m_j grad W_ij
// and T = sum_j m_j tau_j . grad W_ij of particle i: internal force, walls,
// drag, rates and the integrator epilogue with the bounds reductions.
// Called by every thread of the block (dead lanes with live = false).
// `walls`: its wall sums.
template <class W>
__device__ __forceinline__ void stress_finish(const StressArgs &a, int i, bool live, int ki, const Inst &I,
                                              const W &walls, double xi, double yi, double hi, double Sx,
                                              double Sy, double Tx, double Ty, int cnt) {
    const State &s = a.rhs;
    const Phys &P = a.P;
    // everything else the epilogue reads, before anything that could hold it up
    const State &b = a.base;
    const bool own = a.mode == EPI_PREDICT || a.mode == EPI_EULER || a.mode == EPI_RATES;   // (base is the rhs state)
    const double rho = s.rho[i], hh = s.h[i], AA = s.A[i], dv = a.div[i];
    const double2 ta = a.rec.ta[i], tb = a.rec.tb[i], vi = s.vxy[i];
    double2 xy0 = make_double2(xi, yi), v0 = vi;
    double h0 = hh, A0 = AA;
    if (!own) {
        xy0 = b.xy[i];
        v0 = b.vxy[i];
        h0 = b.h[i];
        A0 = b.A[i];
    }
    double mn = b.m[i];
    const double dt = a.sc->dt;
    const double ih = 1.0 / hh, irho = 1.0 / rho;
    const double fi = (P.pa_sph == 2) ? P.inv_rho_ice * ih : rho * P.inv_rho_ice * ih;
    double ax = fi * fma(ta.x, Sx, fma(ta.y, Sy, Tx));
    double ay = fi * fma(ta.y, Sx, fma(tb.x, Sy, Ty));
    const double vxi = vi.x, vyi = vi.y;
    walls.add(irho, ax, ay, cnt);
    // drag, wind_forcing.f90:35-51 and water_drag.f90:35-53 (off at t <= 0)
    const double tnow = I.t;
    if (P.wind_force && tnow > 0.0) {
        double wu, wv;
        wind_at(I, xi, yi, &wu, &wv);
        const double ru = wu - vxi, rv = wv - vyi;
        const double k = P.k_wind * ih;
        ax += k * ru * fabs(ru);
        ay += k * rv * fabs(rv);
    }
    if (P.water_force && tnow > 0.0) {
        const double ru = P.current_u - vxi, rv = P.current_v - vyi;
        const double k = P.k_water * ih;
        ax += k * ru * fabs(ru);
        ay += k * rv * fabs(rv);
    }
    // regularisation, single_step.f90:99-101 (after the drag): the
    // artificial viscosity into dv/dt, the XSPH sum into dx/dt
    // (regularization.f90:93, then single_step.f90:106: dxdt = -chi xsph + v)
    double dxdt = vxi, dydt = vyi;
    if (a.reg) {
        const size_t M = (size_t)a.maxn;
        if (P.art_visc == 1 || P.art_visc == 2) {
            ax += a.reg[i];
            ay += a.reg[M + i];
        }
        if (P.xsph) {
            dxdt = -(P.chi * a.reg[2 * M + i]) + vxi;
            dydt = -(P.chi * a.reg[3 * M + i]) + vyi;
        }
    }
    // prognostic rates, single_step.f90:104-106
    const double dhdt = -hh * dv * irho;
    const double dAdt = -AA * dv * irho;
    if (a.mode == EPI_RATES) {
        block_max_i32(&a.sc->maxip, live ? cnt : 0);
        if (live) {
            const size_t M = (size_t)a.maxn;
            a.rates[i] = ax;
            a.rates[M + i] = ay;
            a.rates[2 * M + i] = dhdt;
            a.rates[3 * M + i] = dAdt;
            if (a.reg && P.xsph) {   // dx/dt in place of the XSPH sum
                a.reg[2 * M + i] = dxdt;
                a.reg[3 * M + i] = dydt;
            }
        }
        return;
    }
    const double x0 = xy0.x, y0 = xy0.y, vx0 = v0.x, vy0 = v0.y;
    double xn, yn, vxn, vyn, hn, An;
    if (a.mode == EPI_PREDICT) {
        // time_integration.f90:207-215 (and the leap-frog's first half, :333-341)
        xn = x0 + dxdt * dt / 2.0;
        yn = y0 + dydt * dt / 2.0;
        vxn = vx0 + ax * dt / 2.0;
        vyn = vy0 + ay * dt / 2.0;
        hn = h0 + dhdt * dt / 2.0;
        An = A0 + dAdt * dt / 2.0;
    } else if (a.mode == EPI_EULER) {
        // euler_scheme, time_integration.f90:117-125
        xn = x0 + dxdt * dt;
        yn = y0 + dydt * dt;
        vxn = vx0 + ax * dt;
        vyn = vy0 + ay * dt;
        hn = h0 + dhdt * dt;
        An = A0 + dAdt * dt;
    } else if (a.mode == EPI_LEAP) {
        // leapfrog_scheme, time_integration.f90:361-369 (vx0: the step-start
        // velocity, dxdt: the half-step right-hand side's dx/dt)
        vxn = vx0 + ax * dt;
        vyn = vy0 + ay * dt;
        hn = h0 + dhdt * dt;
        xn = x0 + (vx0 + dxdt) * dt / 2.0;
        yn = y0 + (vy0 + dydt) * dt / 2.0;
        An = A0 + dAdt * dt;
    } else {
        // time_integration.f90:236-259
        const double x12 = x0 + dxdt * dt / 2.0, y12 = y0 + dydt * dt / 2.0;
        const double vx12 = vx0 + ax * dt / 2.0, vy12 = vy0 + ay * dt / 2.0;
        const double h12 = h0 + dhdt * dt / 2.0, A12 = A0 + dAdt * dt / 2.0;
        xn = 2.0 * x12 - x0;
        yn = 2.0 * y12 - y0;
        vxn = 2.0 * vx12 - vx0;
        vyn = 2.0 * vy12 - vy0;
        hn = 2.0 * h12 - h0;
        An = 2.0 * A12 - A0;
    }
    if (An > 1.0) An = 1.0;
    // the step's last update: hsml, VP time step (after the corrector, the
    // Euler step or the leap-frog's second half).  `tail_later`: a
    // density-rate pass (k_density_rate) follows and does them, because the
    // final density (con_density), Benz's hsml or the Monaghan time step
    // with artificial viscosity needs the updated velocities of the
    // neighbours.
    const bool final_update = a.mode == EPI_CORRECT || a.mode == EPI_EULER || a.mode == EPI_LEAP;
    const bool den2 = P.den_alg == 2, den1 = P.den_alg == 1;
    const bool tail_later = final_update && ((den2 && a.mode != EPI_CORRECT) || den1 || P.sle == 1 ||
                                             (P.tse == 1 && P.artificial_visc));
    double rhon;
    if (den1) {
        rhon = s.rho[i];   // the density of the call, until the summation pass replaces it
    } else if (!den2) {
        rhon = hn * P.rho_ice;                                // density.f90:192
    } else if (a.mode == EPI_CORRECT) {
        // time_integration.f90:242-266: drho/dt of the corrector's density
        // call (half-step velocities and pairs) is the negated divergence
        // sum of this right-hand side
        const double r0 = b.rho[i];
        const double r12 = r0 + (-dv) * dt / 2.0;
        rhon = 2.0 * r12 - r0;
    } else {
        rhon = b.rho[i];   // rho_1, until k_density_rate adds drho/dt dt
    }
    const double hs_old = hi;
    if (P.sle != 2 && P.mass_from_area) {                     // mass_evolution.f90:66-69
        const double ar = kPi * ((P.alpha * hs_old) * (P.alpha * hs_old));
        mn = P.rho_ice * An * hn * ar;
    }
    double hsn = hs_old;
    if (final_update && !tail_later && P.sle == 2) {          // smoothing_length.f90:136-142
        hsn = sqrt(mn / rhon) * (double)P.hsml_multiplicity;
        if (hsn > P.max_hsml) hsn = P.max_hsml;
    }
    // how far this update moves the particle (a non-finite move flags its
    // basin below; an idle lane may see its particle updated)
    double m2 = (xn - x0) * (xn - x0) + (yn - y0) * (yn - y0);
    if (!live || !isfinite(m2)) m2 = 0.0;
    const bool bad = !(isfinite(xn) && isfinite(yn) && isfinite(vxn) && isfinite(vyn) &&
                       isfinite(hn) && isfinite(An));
    if (live && bad) {
        atomicOr(&a.sc->flags, FLAG_NONFINITE);
        atomicOr(&a.inst[ki].flags, FLAG_NONFINITE);
    }
    if (live) {
        const State &o = a.out;
        const double morn = mn / rhon;
        o.xy[i] = make_double2(xn, yn);
        o.vxy[i] = make_double2(vxn, vyn);
        o.mm[i] = make_double2(mn, morn);
        o.h[i] = hn;
        o.A[i] = An;
        o.rho[i] = rhon;
        if (P.sle != 2 && P.mass_from_area) o.m[i] = mn;
        if (o.hmm) o.hmm[i] = make_float4((float)hs_old, (float)mn, (float)morn, 0.0f);
        if (final_update && !tail_later && P.sle == 2) a.hs_next[i] = hsn;
    }
    // this step's bounds, one block-wide reduction
    const bool corr = final_update && !tail_later;
    unsigned active = 1u | 16u;
    unsigned long long v[kBounds] = {(unsigned long long)(live ? cnt : 0), ~0ull, 0ull, ~0ull, dbits(m2)};
    if (corr && P.sle == 2) {                                   // smoothing_length.f90:136-142
        active |= 2u | 4u;
        if (live) {
            v[1] = dbits(hsn);
            v[2] = dbits(hsn);
        }
    }
    if (corr && P.tse != 0) {                                   // time_step.f90:20-26
        active |= 8u;
        if (live) v[3] = dbits(dt_candidate(P, hsn, ax * ax + ay * ay, rhon, 0.0));
    }
    if (tail_later && P.tse == 1 && live) a.rates[i] = ax * ax + ay * ay;   // for k_density_rate
    Inst *Iw = a.inst + ki;
    block_bounds(a.sc, a.mode == EPI_PREDICT ? &Iw->half2_bits : &Iw->step2_bits, active, v);
}

}  // namespace pass

}  // namespace simp
