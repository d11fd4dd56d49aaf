// The two tile passes: one particle per thread, its neighbours' data in shared
// memory (tile.cuh).  Their physics is described in pass_common.cuh.  Each kernel
// function and precision is compiled in a source of its own (passes_*.cu), that
// is, into a module of its own, and a process loads only those it uses (the first
// context of a process: 10 ms; 28 with all of them in one, 18 with gathers).
#pragma once

#include <cmath>
#include <type_traits>

#include "pass_common.cuh"
#include "walls.cuh"

namespace simp {
namespace pass {

constexpr int kBlock = kTile;
// hsml of the halo's particles, where it varies.
__device__ __forceinline__ void tile_hsml(const Halo &h, const TileMem &m, const State &s) {
    for (int d = 0; d < h.nseg; ++d) {
        const int n = h.off[d + 1] - h.off[d];
        for (int k = threadIdx.x; k < n; k += kTile) {
            const double v = s.hs[h.lo[d] + k];
            m.hs[h.off[d] + k] = v;
        }
    }
}

// One word of a particle's candidates, slots [sl, sl + n), n <= 32: bit k set
// where candidate k is not certainly beyond mhsml + delta (FP32 with its
// proven margin).  Called by the whole warp (lanes with n = 0 take part).
template <bool UNIFORM>
__device__ __forceinline__ unsigned scan_word(const TileMem &m, int sl, int n, float xf, float yf, float hf,
                                              float delta, float grow) {
    const int top = __reduce_max_sync(0xffffffffu, n);
    if (n <= 0) sl = 0;   // (a batch may read up to 31 slots past the halo)
    const float2 *f = m.f();
    const float lim_u = (hf + delta) * (hf + delta) * grow;
    unsigned bits = 0u;
    for (int k0 = 0; k0 < top; k0 += 8) {
        unsigned b8 = 0u;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const float2 q = f[sl + k0 + u];
            const float dx = xf - q.x, dy = yf - q.y;
            const float sf = fmaf(dx, dx, dy * dy);
            float lim = lim_u;
            if (!UNIFORM) {
                const float mf = 0.5f * (hf + m.hf()[sl + k0 + u]) + delta;
                lim = mf * mf * grow;
            }
            if (sf <= lim) b8 |= 1u << u;
        }
        bits |= b8 << k0;
    }
    if (n < 32) bits &= (1u << max(n, 0)) - 1u;
    return bits;
}

// Builds the lists of a tile part whose xy records are in shared memory; a
// particle's candidates go to the shared list and to the tile's lists `out`,
// at its column.  Returns the particle's candidates, which may exceed
// kListRows (the list then holds the first ones).  Called by the whole block.
template <bool UNIFORM>
__device__ __noinline__ int build_lists(const Halo &h, const TileMem &m, const KinArgs &a, const Inst &I, int i,
                                        bool live, unsigned short *out, int column) {
    const int t = threadIdx.x;
    const double2 *xs = reinterpret_cast<const double2 *>(m.rec[0]);
    const int total = h.off[h.nseg];
    for (int k = t; k < total; k += kTile) {
        const double2 q = xs[k];
        m.f()[k] = make_float2((float)q.x, (float)q.y);
        if (!UNIFORM) m.hf()[k] = (float)m.hs[k];
    }
    __syncthreads();
    const int2 at = cell_at(I, a.cell[i]);
    const double2 xy = a.s.xy[i];
    const float xf = (float)xy.x, yf = (float)xy.y, hf = (float)a.s.hs[i];
    const float margin = prefilter_margin(bitsd(I.xabs_bits) + sqrt(bitsd(I.half2_bits)), I.hmin);
    const float grow = margin < 0.25f ? 1.0f + margin : INFINITY;
    const float delta = (float)I.delta;
    const int own = slot_of(h, i);
    int cnt = 0;
    for (int d = 0; d < h.nseg; ++d) {
        int j0, j1;
        stencil_range(I, a.cell_start, at, h.nseg / 2, d, j0, j1);
        int left = live ? j1 - j0 : 0;
        int sl = left > 0 ? slot_of(h, j0) : 0;
        while (__any_sync(0xffffffffu, left > 0)) {
            unsigned bits = scan_word<UNIFORM>(m, sl, min(left, 32), xf, yf, hf, delta, grow);
            const int self = own - sl;
            if (self >= 0 && self < 32) bits &= ~(1u << self);
            while (bits != 0u) {
                const int k = __ffs(bits) - 1;
                bits &= bits - 1u;
                if (cnt < kListRows) {
                    m.list[list_at(cnt, t)] = (unsigned short)(sl + k);
                    out[list_at(cnt, column)] = (unsigned short)(sl + k);
                }
                ++cnt;
            }
            sl += 32;
            left -= 32;
        }
    }
    return cnt;
}

// Programmatic dependent launch: a pass's blocks may start while the last
// blocks of the kernel before still run, and wait here before they read what
// it wrote (with ordinary loads: the wait does not order those of the read-only
// path, which are for data that nothing writes while a kernel runs).  The
// kernels after it may follow once every block is this far (so that everything
// before the previous kernel has ended).
__device__ __forceinline__ void pass_begin() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Per-neighbour scalars of a slot: the FP64 records for the plain form, the
// packed FP32 copies for the mixed form.  (Where hsml is one value in every
// basin a neighbour's is not read.)
template <class T>
struct Rec;
template <>
struct Rec<double> {
    static constexpr int stress_arrays = 3;   // xy, (tau11, tau12), (tau22, m)
    static __device__ __forceinline__ double own_h(const State &s, int i) { return s.hs[i]; }
    static __device__ __forceinline__ const void *kin_src(const State &s) { return s.mm; }
    template <bool UNIFORM>
    static __device__ __forceinline__ void kin(const TileMem &t, int sl, double &m, double &mor, double &h) {
        const double2 q = reinterpret_cast<const double2 *>(t.rec[2])[sl];
        m = q.x;
        mor = q.y;
        h = UNIFORM ? 0.0 : t.hs[sl];
    }
    template <bool UNIFORM>
    static __device__ __forceinline__ void stress(const TileMem &t, int sl, double &m, double &t11, double &t12,
                                                  double &t22, double &h) {
        const double2 a = reinterpret_cast<const double2 *>(t.rec[1])[sl];
        const double2 b = reinterpret_cast<const double2 *>(t.rec[2])[sl];
        m = b.y;
        t11 = a.x;
        t12 = a.y;
        t22 = b.x;
        h = UNIFORM ? 0.0 : t.hs[sl];
    }
    static constexpr double band = kBand;
};
template <>
struct Rec<float> {
    static constexpr int stress_arrays = 2;   // xy, (tau11, tau12, tau22, m)
    static __device__ __forceinline__ float own_h(const State &s, int i) { return s.hsf[i]; }
    static __device__ __forceinline__ const void *kin_src(const State &s) { return s.hmm; }
    template <bool UNIFORM>
    static __device__ __forceinline__ void kin(const TileMem &t, int sl, float &m, float &mor, float &h) {
        const float4 q = reinterpret_cast<const float4 *>(t.rec[2])[sl];
        h = q.x;
        m = q.y;
        mor = q.z;
    }
    template <bool UNIFORM>
    static __device__ __forceinline__ void stress(const TileMem &t, int sl, float &m, float &t11, float &t12,
                                                  float &t22, float &h) {
        const float4 q = reinterpret_cast<const float4 *>(t.rec[1])[sl];
        m = q.w;
        t11 = q.x;
        t12 = q.y;
        t22 = q.z;
        h = UNIFORM ? 0.0f : (float)t.hs[sl];
    }
    // (differences and hsml rounded to FP32: within 2^-20 of the exact ratio)
    static constexpr float band = 0x1p-18f;
};

// A candidate against the exact criterion's band: 1 certainly a pair, 0
// certainly none, 2 within the band (or not a number).
template <class T, bool UNIFORM>
__device__ __forceinline__ int classify(T dx, T dy, T hi, T hj, T mh2_u) {
    const T s = fma(dx, dx, dy * dy);
    T mh2 = mh2_u;
    if (!UNIFORM) {
        const T mh = T(0.5) * (hi + hj);
        mh2 = mh * mh;
    }
    if (s < mh2 * (T(1) - Rec<T>::band)) return 1;
    return s > mh2 * (T(1) + Rec<T>::band) ? 0 : 2;
}

constexpr int kHaloWords = sizeof(Halo) / sizeof(int);
constexpr int kWallWords = 2 * kMaxWallRows;
__device__ __forceinline__ int halo_word(const void *h, int k) { return reinterpret_cast<const int *>(h)[k]; }

// The largest squared distance of the tile's particles from where they were
// sorted, rounded up, as a float's bits.  Called by the whole block.
inline __device__ __noinline__ void tile_moved(const State &s, const double2 *xyr, int p0, int p1, unsigned &out) {
    const int t = threadIdx.x, i = p0 + t;
    if (t == 0) out = 0u;
    __syncthreads();
    float d2 = 0.0f;
    if (i < p1) {
        const double2 a = s.xy[i], b = xyr[i];
        const double dx = a.x - b.x, dy = a.y - b.y;
        d2 = __double2float_ru(fma(dx, dx, dy * dy));
        if (!(d2 >= 0.0f)) d2 = INFINITY;
    }
    const unsigned most = __reduce_max_sync(0xffffffffu, __float_as_uint(d2));
    if ((t & 31) == 0) atomicMax(&out, most);
    __syncthreads();
}

// Whether a basin's lists hold every pair of this right-hand side (Inst).
// In a step's second right-hand side they are at most as old as the first.
__device__ __forceinline__ bool lists_valid(const Inst &I, bool second) {
    if (!I.list_ok && !second) return false;
    const double room = 0.5 * I.delta * (1.0 - 1e-9) - (I.list_ok ? I.list_d : 0.0);
    return room >= 0.0 && (!second || bitsd(I.half2_bits) <= room * room);
}

// The sums of a particle without a list, from its stencil.  A call in FP64,
// inlined in the mixed form, whose five blocks per SM leave no registers for one
// (us per step, called and inlined: FP64 262,144 particles 157 and 160, 1,048,576
// 568 and 582; mixed 262,144 178 and 158, 1,048,576 613 and 556).
template <class T, int SKF, int HS>
__device__ __forceinline__ KinSums<T> kin_stencil(const KinArgs &a, const Inst &I, const Halo &h, int i) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr bool UNIFORM = HS == HSML_ONE;
    const State &s = a.s;
    const void *src[3] = {s.xy, s.vxy, Rec<T>::kin_src(s)};
    const Around w(h, tile_mem(smem, a.cap, 3, UNIFORM), src, s);
    const double2 xy = s.xy[i], vi = s.vxy[i];
    PairGrad<T, SKF, HS> grad;
    grad.init(a.P, I, Rec<T>::own_h(s, i));
    KinSums<T> ks;
    stencil_pairs<UNIFORM>(w, s, I, a.cell_start, i, a.cell[i], [&](int q, int) {
        const double2 x = reinterpret_cast<const double2 *>(w.m.rec[0])[q];
        const double2 v = reinterpret_cast<const double2 *>(w.m.rec[1])[q];
        T mj, mrj, hj;
        Rec<T>::template kin<UNIFORM>(w.m, q, mj, mrj, hj);
        const T dx = (T)(xy.x - x.x), dy = (T)(xy.y - x.y);
        const T g = grad(a.P, fma(dx, dx, dy * dy), hj);
        ks.add(true, g * dx, g * dy, (T)(vi.x - v.x), (T)(vi.y - v.y), mj, mrj);
    });
    return ks;
}
template <class T, int SKF, int HS>
__device__ __noinline__ KinSums<T> kin_stencil_call(const KinArgs &a, const Inst &I, const Halo &h, int i) {
    return kin_stencil<T, SKF, HS>(a, I, h, i);
}

// Kinematic pass over tiles.  Bound by shared memory and latency: a block waits
// for its tile's copies, then reads three 16-byte records per pair at slots that
// have no order, so that their banks collide (L1 57% busy in FP64, 73% mixed;
// issue slots 32% and 54%).  Two candidates at a time put six such reads in
// flight.  262,144 particles, FP64: 79 -> 38 us per pass against gathers from
// global memory; mixed at 1,048,576: 237 -> 124 us.
template <class T, int SKF, int HS, int BLOCKS>
__global__ void __launch_bounds__(kBlock, BLOCKS) k_kinematic(const __grid_constant__ KinArgs a) {
    constexpr bool UNIFORM = HS == HSML_ONE;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Halo h;
    __shared__ __align__(8) unsigned long long bar;
    __shared__ int rows_max, failed;
    __shared__ unsigned moved2;
    const int t = threadIdx.x;
    const Chunk ch = a.chunks[blockIdx.x];   // (of the last sort)
    const int shift = part_shift(ch);
    if (t == 0) bar_init(&bar);
    pass_begin();
    const Inst &I = a.inst[a.single ? 0 : ch.q];
    const State &s = a.s;
    const Phys &P = a.P;
    Halo *halos = reinterpret_cast<Halo *>(a.halos) + (size_t)blockIdx.x * kParts;
    const int first = t < kHaloWords ? halo_word(halos, t) : 0;   // (read along with the instance)
    if (t == kTile - 1) failed = failed_before(a.sc);
    if (ch.spare >= I.spares) return;   // (an unused spare tile)
    unsigned short *lists = a.pl.slot + (size_t)blockIdx.x * kListRows * kTile;
    // a basin whose state turned non-finite is not searched any more (its
    // stencil would span its whole grid); it is only carried until retired
    if (inst_dead(I.flags)) {
        if (t == 0) {
            Halo none{};
            none.kind = HALO_NONE;
            none.size = ch.p1 - ch.p0;
            halos[0] = none;
        }
        const int i = ch.p0 + t;
        if (i >= ch.p1) return;
        kin_rheology(a, i, -0.0, -0.0, -0.0, -0.0);
        return;
    }
    const bool build = !lists_valid(I, a.second);
    const TileMem m = tile_mem(smem, a.cap, 3, UNIFORM);
    unsigned parity = 0u;
    if (build) tile_moved(s, a.xyr, ch.p0, ch.p1, moved2);
    for (int p0 = ch.p0; p0 < ch.p1;) {
        if (!build) {
            if (t < kHaloWords)
                reinterpret_cast<int *>(&h)[t] = p0 == ch.p0 ? first : halo_word(&halos[(p0 - ch.p0) >> shift], t);
        } else if (t < 32) {
            make_halo(I, a.cell_start, a.bstart, a.cell, p0, ch.p1, shift, a.cap,
                      sqrt((double)__uint_as_float(moved2)) * (1.0 + 1e-6), h,
                      reinterpret_cast<HaloWalls *>(a.halo_walls)[(size_t)blockIdx.x * kParts + ((p0 - ch.p0) >> shift)]);
            if (t == 0) rows_max = 0;
        }
        __syncthreads();
        if (failed < 2 * p0) return;
        const void *src[3] = {s.xy, s.vxy, Rec<T>::kin_src(s)};
        const bool fits = h.kind == HALO_TILE;
        if (fits && t < 32) tile_fetch(h, m, src, 0, build ? 1 : 3, lists, build ? 0 : h.rows, &bar);
        const bool live = t < h.size;
        const int i = p0 + (live ? t : 0);
        double2 xy = s.xy[i], vi = s.vxy[i];
        if (sizeof(T) == sizeof(float) && a.prefetch) {   // (the plain form has no register to spare)
            prefetch_l1(&s.h[i]);
            prefetch_l1(&s.A[i]);
            prefetch_l1(&s.rho[i]);
            prefetch_l1(&s.mm[i]);
        }
        const T hiT = Rec<T>::own_h(s, i);
        PairGrad<T, SKF, HS> grad;
        grad.init(P, I, hiT);
        const bool rule = rule_on(I);
        KinSums<T> ks;     // -div and the velocity gradient, negated
        auto terms = [&](bool in, T dx, T dy, double2 v, T mj, T mrj, T hj) {
            const T g = grad(P, fma(dx, dx, dy * dy), hj);
            ks.add(in, g * dx, g * dy, (T)(vi.x - v.x), (T)(vi.y - v.y), mj, mrj);
        };
        int cnt = 0;       // candidates in the particle's list
        if (fits) {
            if (!UNIFORM) tile_hsml(h, m, s);
            if (!build && live) cnt = a.pl.count[i];
            if (!copies_arrive(&bar, parity, 2 * p0, &failed, &a.sc->flags)) cnt = 0;
            parity ^= 1u;
            if (!UNIFORM || build) __syncthreads();
            if (build) {
                cnt = build_lists<UNIFORM>(h, m, a, I, i, live, lists, i - ch.p0);
                const int rows = __reduce_max_sync(0xffffffffu, cnt);
                if ((t & 31) == 0) atomicMax(&rows_max, rows);
                // (the FP32 copies make way for the records)
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncthreads();
                if (failed <= 2 * p0) return;
                if (t == 0) h.rows = min(rows_max, kListRows);
                if (t < 32) tile_fetch(h, m, src, 1, 3, lists, 0, &bar);
                if (live) a.pl.count[i] = cnt;
                if (!copies_arrive(&bar, parity, 2 * p0 + 1, &failed, &a.sc->flags)) cnt = 0;
                parity ^= 1u;
                __syncthreads();
            }
        }
        if (build && t == 0) halos[(p0 - ch.p0) >> shift] = h;
        if (fits && cnt <= kListRows) {
            const double2 *xs = reinterpret_cast<const double2 *>(m.rec[0]);
            const double2 *vs = reinterpret_cast<const double2 *>(m.rec[1]);
            const T mh2_u = hiT * hiT;
            // (a list just built stands at the thread's own column, a copied
            // one at the particle's)
            const ushort2 *col = reinterpret_cast<const ushort2 *>(m.list) + (build ? t : i - ch.p0);
            // two candidates at a time, so that their chains overlap
            for (int k = 0; k < cnt; k += 2) {
                const ushort2 w = col[(k >> 1) * kTile];
                const int q0 = w.x, q1 = k + 1 < cnt ? w.y : w.x;
                if (!SIMP_IN_RANGE(q0, 0, h.off[h.nseg], SITE_TILE) || !SIMP_IN_RANGE(q1, 0, h.off[h.nseg], SITE_TILE))
                    continue;
                const double2 x0 = xs[q0], x1 = xs[q1], v0 = vs[q0], v1 = vs[q1];
                T m0, r0, h0, m1, r1, h1;
                Rec<T>::template kin<UNIFORM>(m, q0, m0, r0, h0);
                Rec<T>::template kin<UNIFORM>(m, q1, m1, r1, h1);
                const T dx0 = (T)(xy.x - x0.x), dy0 = (T)(xy.y - x0.y);
                const T dx1 = (T)(xy.x - x1.x), dy1 = (T)(xy.y - x1.y);
                int in0 = classify<T, UNIFORM>(dx0, dy0, hiT, h0, mh2_u);
                int in1 = k + 1 < cnt ? classify<T, UNIFORM>(dx1, dy1, hiT, h1, mh2_u) : 0;
                if (((in0 | in1) & 2) || rule) {
                    const int in = exact_two(s, I, rule, i, h, q0, q1, in0, in1);
                    in0 = in & 1;
                    in1 = in >> 1;
                    reload(xy, &s.xy[i]);
                    reload(vi, &s.vxy[i]);
                }
                terms(in0 != 0, dx0, dy0, v0, m0, r0, h0);
                terms(in1 != 0, dx1, dy1, v1, m1, r1, h1);
            }
        } else if (live) {
            ks = sizeof(T) == sizeof(double) ? kin_stencil_call<T, SKF, HS>(a, I, h, i) : kin_stencil<T, SKF, HS>(a, I, h, i);
        }
        if (live) {
            const double c = -grad.common(I);
            kin_rheology(a, i, c * ks.dv.get(), c * ks.g1.get(), c * ks.g23.get(), c * ks.g4.get());
        }
        p0 += h.size;
        if (p0 < ch.p1) {
            // the next part's copies write where this one's reads were
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
        }
    }
}

// The stress pass's, and how many pairs it has.
template <class T, int SKF, int HS>
__device__ __forceinline__ StressSums<T> stress_stencil(const StressArgs &a, const Inst &I, const Halo &h, int i) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr bool UNIFORM = HS == HSML_ONE;
    const State &s = a.rhs;
    const void *src[3] = {s.xy, a.rec.tq ? (const void *)a.rec.tq : (const void *)a.rec.ta, a.rec.tb};
    const Around w(h, tile_mem(smem, a.cap, Rec<T>::stress_arrays, UNIFORM), src, s);
    const double2 xy = s.xy[i];
    PairGrad<T, SKF, HS> grad;
    grad.init(a.P, I, Rec<T>::own_h(s, i));
    StressSums<T> ss;
    stencil_pairs<UNIFORM>(w, s, I, a.cell_start, i, a.cell[i], [&](int q, int) {
        const double2 x = reinterpret_cast<const double2 *>(w.m.rec[0])[q];
        T mj, t11, t12, t22, hj;
        Rec<T>::template stress<UNIFORM>(w.m, q, mj, t11, t12, t22, hj);
        const T dx = (T)(xy.x - x.x), dy = (T)(xy.y - x.y);
        const T g = grad(a.P, fma(dx, dx, dy * dy), hj);
        ss.add(true, g * dx, g * dy, mj, t11, t12, t22);
        ++ss.pairs;
    });
    return ss;
}

template <class T, int SKF, int HS>
__device__ __noinline__ StressSums<T> stress_stencil_call(const StressArgs &a, const Inst &I, const Halo &h, int i) {
    return stress_stencil<T, SKF, HS>(a, I, h, i);
}

// Stress pass over the same tiles, then the epilogue, whose twenty own values
// are loaded together ahead of the walls and the update (68 -> 50 us against
// loading each where it is used).  Half of a block's time is the latency of its
// copies and of that epilogue (issue slots 30%, L1 52%).  262,144 particles,
// FP64: 71 -> 45 us per pass against gathers from global memory; mixed at
// 1,048,576: 192 -> 149 us.
template <class T, int SKF, int HS, int BLOCKS>
__global__ void __launch_bounds__(kBlock, BLOCKS) k_stress(const __grid_constant__ StressArgs a) {
    constexpr bool UNIFORM = HS == HSML_ONE;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Halo h;
    __shared__ HaloWalls hw;
    __shared__ int failed;
    __shared__ __align__(8) unsigned long long bar;
    const int t = threadIdx.x;
    const Chunk ch = a.chunks[blockIdx.x];   // (of the last sort)
    const int shift = part_shift(ch);
    if (t == 0) bar_init(&bar);
    pass_begin();
    const Inst &I = a.inst[a.single ? 0 : ch.q];
    const Halo *halos = reinterpret_cast<const Halo *>(a.halos) + (size_t)blockIdx.x * kParts;
    const HaloWalls *walls = reinterpret_cast<const HaloWalls *>(a.halo_walls) + (size_t)blockIdx.x * kParts;
    // (read along with the instance; the second warp reads the walls)
    const int first = t < kHaloWords ? halo_word(halos, t)
                      : BLOCKS == 4 && t >= 32 && t < 32 + kWallWords ? halo_word(walls, t - 32) : 0;
    if (t == kTile - 1) failed = failed_before(a.sc);
    if (ch.spare >= I.spares) return;   // (an unused spare tile)
    const State &s = a.rhs;
    const Phys &P = a.P;
    // (of a dead basin the kinematic pass wrote records without walls; its flags
    // are not asked here, because other blocks set them while this one runs and
    // the walls' barriers need every thread to decide alike)
    const bool have_walls = (P.boundary_pressure || P.boundary_friction) && a.nb > 0;
    using Walls = typename std::conditional<sizeof(T) == sizeof(float), WallShared, WallRegs>::type;
    constexpr int arrays = Rec<T>::stress_arrays;
    const TileMem m = tile_mem(smem, a.cap, arrays, UNIFORM);
    unsigned parity = 0u;
    for (int p0 = ch.p0; p0 < ch.p1;) {
        const int part = (p0 - ch.p0) >> shift;
        if (t < kHaloWords) reinterpret_cast<int *>(&h)[t] = part == 0 ? first : halo_word(&halos[part], t);
        if (BLOCKS == 4 && t >= 32 && t < 32 + kWallWords)
            reinterpret_cast<int *>(&hw)[t - 32] = part == 0 ? first : halo_word(&walls[part], t - 32);
        __syncthreads();
        if (failed < 2 * p0) return;
        const bool tile = h.kind == HALO_TILE;
        const void *src[3] = {s.xy, a.rec.tq ? (const void *)a.rec.tq : (const void *)a.rec.ta, a.rec.tb};
        if (tile && t < 32) {
            tile_fetch(h, m, src, 0, arrays, a.pl.slot + (size_t)blockIdx.x * kListRows * kTile, h.rows, &bar);
        }
        const bool live = t < h.size;
        const int i = p0 + (live ? t : h.size - 1);   // idle lanes mirror the part's last particle
        if (a.prefetch) stress_prefetch(a, i);
        if (BLOCKS == 4 && have_walls && h.walls) wall_prefetch(a, hw, a.bstart[I.base], i);
        double2 xy = s.xy[i];
        double hi = s.hs[i];
        const T hiT = Rec<T>::own_h(s, i);
        StressSums<T> ss;
        PairGrad<T, SKF, HS> grad;
        grad.init(P, I, hiT);
        auto terms = [&](bool in, T dx, T dy, T mj, T t11, T t12, T t22, T hj) {
            const T g = grad(P, fma(dx, dx, dy * dy), hj);
            ss.add(in, g * dx, g * dy, mj, t11, t12, t22);
            ss.pairs += in;
        };
        int cnt = live && h.kind != HALO_NONE ? kListRows + 1 : 0;   // candidates in its list
        if (tile) {
            if (!UNIFORM) tile_hsml(h, m, s);
            if (live) cnt = a.pl.count[i];
            if (!copies_arrive(&bar, parity, 2 * p0, &failed, &a.sc->flags)) cnt = 0;
            parity ^= 1u;
            if (!UNIFORM) __syncthreads();
        }
        if (cnt <= kListRows) {
            const bool rule = rule_on(I);
            const double2 *xs = reinterpret_cast<const double2 *>(m.rec[0]);
            const ushort2 *col = reinterpret_cast<const ushort2 *>(m.list) + (i - ch.p0);
            const T mh2_u = hiT * hiT;
            // two candidates at a time, so that their chains overlap
            for (int k = 0; k < cnt; k += 2) {
                const ushort2 w = col[(k >> 1) * kTile];
                const int q0 = w.x, q1 = k + 1 < cnt ? w.y : w.x;
                if (!SIMP_IN_RANGE(q0, 0, h.off[h.nseg], SITE_TILE) || !SIMP_IN_RANGE(q1, 0, h.off[h.nseg], SITE_TILE))
                    continue;
                const double2 x0 = xs[q0], x1 = xs[q1];
                T m0, a0, b0, c0, h0, m1, a1, b1, c1, h1;
                Rec<T>::template stress<UNIFORM>(m, q0, m0, a0, b0, c0, h0);
                Rec<T>::template stress<UNIFORM>(m, q1, m1, a1, b1, c1, h1);
                const T dx0 = (T)(xy.x - x0.x), dy0 = (T)(xy.y - x0.y);
                const T dx1 = (T)(xy.x - x1.x), dy1 = (T)(xy.y - x1.y);
                int in0 = classify<T, UNIFORM>(dx0, dy0, hiT, h0, mh2_u);
                int in1 = k + 1 < cnt ? classify<T, UNIFORM>(dx1, dy1, hiT, h1, mh2_u) : 0;
                if (((in0 | in1) & 2) || rule) {
                    const int in = exact_two(s, I, rule, i, h, q0, q1, in0, in1);
                    in0 = in & 1;
                    in1 = in >> 1;
                    reload(xy, &s.xy[i]);
                }
                terms(in0 != 0, dx0, dy0, m0, a0, b0, c0, h0);
                terms(in1 != 0, dx1, dy1, m1, a1, b1, c1, h1);
            }
        } else {
            ss = sizeof(T) == sizeof(double) ? stress_stencil_call<T, SKF, HS>(a, I, h, i)
                                             : stress_stencil<T, SKF, HS>(a, I, h, i);
        }
        // (a retired basin's particles are not written any more: their state
        // stays as it was until the batch's next compaction drops them)
        double S[4];
        auto pair_sums = [&] {
            const double c = grad.common(I);
            S[0] = c * ss.sx.get();
            S[1] = c * ss.sy.get();
            S[2] = c * ss.tx.get();
            S[3] = c * ss.ty.get();
        };
        if (Walls::kKeep) pair_sums();
        Walls wl;
        if (have_walls && h.walls) {
            int bytes = (int)stress_smem_bytes(a.cap, arrays, UNIFORM);
            __syncthreads();
            double *keep = reinterpret_cast<double *>(smem + bytes) - 4 * kTile + t;
            if (Walls::kKeep) {
                bytes -= 4 * kTile * (int)sizeof(double);
#pragma unroll
                for (int k = 0; k < 4; ++k) keep[k * kTile] = S[k];
            }
            wl.set(reinterpret_cast<WallTile *>(smem),
                   wall_sums<SKF, BLOCKS == 4>(a, I, h.walls, hw, p0, h.size, i, xy, hi, smem, bytes));
            if (Walls::kKeep) {
#pragma unroll
                for (int k = 0; k < 4; ++k) S[k] = keep[k * kTile];
                reload(xy, &s.xy[i]);
                reload(hi, &s.hs[i]);
            }
        }
        if (!Walls::kKeep) pair_sums();
        stress_finish(a, i, live && !(I.flags & FLAG_RETIRED), ch.q, I, wl, xy.x, xy.y, hi, S[0], S[1], S[2], S[3],
                      ss.pairs);
        p0 += h.size;
        if (p0 < ch.p1) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
        }
    }
}

// The passes of one kernel function and precision, by hsml form and resident
// blocks per SM.
template <class T, int SKF, int HS>
PassForm pass_form_of(int blocks) {
    if constexpr (sizeof(T) == sizeof(float))
        if (blocks == 5) return {k_kinematic<T, SKF, HS, 5>, k_stress<T, SKF, HS, 5>};
    return {k_kinematic<T, SKF, HS, 4>, k_stress<T, SKF, HS, 4>};
}
template <class T, int SKF>
PassForm pass_form(int hs, int blocks) {
    if (hs == HSML_ONE) return pass_form_of<T, SKF, HSML_ONE>(blocks);
    if (hs == HSML_VARIED || SKF == 0) return pass_form_of<T, SKF, HSML_VARIED>(blocks);   // (the generic kernels' arithmetic is one)
    return pass_form_of<T, SKF, SKF ? HSML_EITHER : HSML_VARIED>(blocks);
}

}  // namespace pass
}  // namespace simp
