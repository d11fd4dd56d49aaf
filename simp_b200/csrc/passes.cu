// Pair passes: one particle per thread, its neighbours' data in shared memory
// (tile.cuh).  The physics of both passes is described in pass_common.cuh.
#include <cmath>
#include <type_traits>

#include "pass_common.cuh"
#include "walls.cuh"

namespace simp {

namespace {

using namespace pass;

constexpr int kBlock = kTile;
// Resident blocks per SM the register allocation aims at.  4 (128 registers)
// holds the pair math of two candidates: FP64 always (5 and 6
// blocks per step at 262,144 particles: 160 -> 168 and 234 us; the reference's
// switches at 90,007: 131 -> 154 and 197).  The mixed form takes 5 above
// kSmallTiles tiles, where more of them at a time begin to pay; up to 4,000 or so
// it depends on how full the last wave is (592 tiles a wave with 4, 740 with 5).
// us per step with 4 and 5: 57,600 particles 56 and 66, 102,400 88 and 98, 131,044
// 92 and 106, 160,000 116 and 111, 200,704 127 and 143, 262,144 162 and 163,
// 640,000 366 and 364, 1,048,576 560 and 548.
constexpr int kSmallTiles = 1024;

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
__device__ __noinline__ void tile_moved(const State &s, const double2 *xyr, int p0, int p1, unsigned &out) {
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
// have no order, so that their banks collide (L1 55% busy in FP64, 70% mixed;
// issue slots 31% and 51%).  Two candidates at a time put six such reads in
// flight.  262,144 particles, FP64: 79 -> 40 us per pass against gathers from
// global memory; mixed at 1,048,576: 237 -> 132 us.
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
            const double c = -grad.common();
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
// copies and of that epilogue (issue slots 29%, L1 50%).  262,144 particles,
// FP64: 71 -> 44 us per pass against gathers from global memory; mixed at
// 1,048,576: 192 -> 147 us.
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
            const double c = grad.common();
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

// Regularisation of a right-hand side (regularization.f90, called by
// single_step.f90:99-101), per particle i over the pairs the kinematic pass
// just found, in FP64 in both precision forms:
//   XSPH (:45-95)  xs_i = sum_j m_j (v_i - v_j) W_ij / ((rho_i + rho_j) / 2)
//   artificial viscosity, av_i = -sum_j m_j pi_ij grad_i W_ij with
//     Hernquist-Katz (:102-213): pi_ij = lv_i / rho_i^2 + lv_j / rho_j^2,
//       lv = (alpha_pi hsml c |d| + beta_pi (|d| hsml)^2) rho, d the
//       velocity divergence (the kinematic pass's sum over rho) where it is
//       negative, else 0;
//     Monaghan (:220-308): pi_ij = (beta_pi iota^2 - alpha_pi iota
//       (c_i + c_j) / 2) / ((rho_i + rho_j) / 2), iota = hsml_ij v_r /
//       (r_ij^2 + (0.01 hsml_ij)^2), v_r = (v_i - v_j) . (x_i - x_j);
//     for pairs with (v_i - v_j) . (x_i - x_j) <= 0, else pi_ij = 0.
// The reference runs both loops serially over its pair list, where pi_ij
// keeps the previous pair's value for a pair outside the criterion and XSPH
// adds the same-signed term to both particles; the gather here evaluates
// every pair on its own (zero outside the criterion, XSPH antisymmetric).
struct RegArgs {
    State s;
    const double *div;   // the kinematic pass's -sum_j m_j (v_i - v_j) . grad W
    PairList pl;
    const int *cell_start, *cell;
    const Chunk *chunks;
    const unsigned char *halos;
    int cap;
    const Inst *inst;
    Scalars *sc;
    Phys P;
    double *reg;
    int maxn;
};

// lv / rho^2 of the Hernquist-Katz viscosity of particle k
__device__ __forceinline__ double hk_lv_r2(const Phys &P, const State &s, const double *div, int k) {
    const double rho = s.rho[k], hs = s.hs[k];
    double d = div[k] / rho;
    if (d >= 0.0) d = 0.0;
    const double c = sound_speed_held(P, rho);
    const double ad = fabs(d);
    const double lv = (P.alpha_pi * hs * c * ad + P.beta_pi * ((ad * hs) * (ad * hs))) * rho;
    return lv / (rho * rho);
}

// The tiles of the two passes below hold, beside the records (xy, vxy) and
// hsml, some FP64 values per particle, each worked out once per tile instead
// of once per pair: fill(j, k) writes those of particle j at slot k.
template <class F>
__device__ __forceinline__ void tile_fill(const Halo &h, F &&fill) {
    for (int d = 0; d < h.nseg; ++d) {
        const int n = h.off[d + 1] - h.off[d];
        for (int k = threadIdx.x; k < n; k += kTile) fill(h.lo[d] + k, h.off[d] + k);
    }
}
constexpr int kAuxArrays = 3;
constexpr size_t aux_smem_bytes(int cap) {
    return tile_smem_bytes(cap, 2, false) + (size_t)kAuxArrays * cap * sizeof(double);
}
static_assert(aux_smem_bytes(kMostHaloCap) <= kMostTileSmem, "ctx.h: kMostHaloCap");

// Copies a tile part's halo record, records and lists to shared memory and
// fills the other values.  Called by the whole block; false, for all of it,
// where a copy did not arrive, now or in an earlier pass.
template <class F>
__device__ __forceinline__ bool aux_tile(const Halo *rec, Halo &h, const TileMem &m, const State &g, const double2 *vxy,
                                         const unsigned short *lists, unsigned long long *bar, unsigned &parity,
                                         Scalars *sc, F &&fill) {
    __shared__ int failed;
    const int t = threadIdx.x;
    if (t < (int)(sizeof(Halo) / sizeof(int))) reinterpret_cast<int *>(&h)[t] = reinterpret_cast<const int *>(rec)[t];
    if (t == kTile - 1) failed = failed_before(sc);
    __syncthreads();
    if (failed < 0) return false;
    if (h.kind != HALO_TILE) return true;
    const void *src[3] = {g.xy, vxy, nullptr};
    if (t < 32) tile_fetch(h, m, src, 0, 2, lists, h.rows, bar);
    tile_hsml(h, m, g);
    tile_fill(h, fill);
    copies_arrive(bar, parity, 0, &failed, &sc->flags);
    parity ^= 1u;
    __syncthreads();
    return failed == kNoneFailed;
}

// Pairs of a particle of such a tile: f(j, slot, x_j, v_j, h_j), slot -1 where
// there is no tile.
template <class F>
__device__ __forceinline__ void aux_pairs(const Halo &h, const TileMem &m, const State &g, const double2 *vxy,
                                          const Inst &I, const int *cell_start, const int *cell, const int *count,
                                          int i, int column, F &&f) {
    const int cnt = h.kind == HALO_TILE ? count[i] : kListRows + 1;
    if (h.kind != HALO_NONE && cnt > kListRows) {
        const void *src[3] = {g.xy, vxy, nullptr};
        const Around w(h, m, src, g);
        stencil_pairs<false>(w, g, I, cell_start, i, cell[i], [&](int q, int j) {
            f(j, w.h ? q : -1, reinterpret_cast<const double2 *>(w.m.rec[0])[q],
              reinterpret_cast<const double2 *>(w.m.rec[1])[q], w.m.hs[q]);
        });
    } else if (h.kind == HALO_TILE) {
        const double2 p = g.xy[i];
        const double hi = g.hs[i];
        const bool rule = rule_on(I);
        const double2 *xs = reinterpret_cast<const double2 *>(m.rec[0]);
        const double2 *vs = reinterpret_cast<const double2 *>(m.rec[1]);
        for (int k = 0; k < cnt; ++k) {
            const int q = m.list[list_at(k, column)];
            if (!SIMP_IN_RANGE(q, 0, h.off[h.nseg], SITE_TILE)) continue;
            const double2 x = xs[q];
            const double hj = m.hs[q];
            const int in = classify<double, false>(p.x - x.x, p.y - x.y, hi, hj, 0.0);
            if (in == 0) continue;
            if (in == 2 || rule)
                if (!exact_pair(g, I, rule, i, particle_of(h, q))) continue;
            f(particle_of(h, q), q, x, vs[q], hj);
        }
    }
}

__global__ void __launch_bounds__(kBlock) k_regularize(const __grid_constant__ RegArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Halo h;
    __shared__ __align__(8) unsigned long long bar;
    const int t = threadIdx.x;
    const Chunk ch = a.chunks[blockIdx.x];
    const int shift = part_shift(ch);
    const State &s = a.s;
    const Phys &P = a.P;
    const size_t M = (size_t)a.maxn;
    const Inst &I = a.inst[ch.q];
    if (ch.spare >= I.spares) return;   // (an unused spare tile)
    const bool dead = inst_dead(I.flags);
    const Halo *halos = reinterpret_cast<const Halo *>(a.halos) + (size_t)blockIdx.x * kParts;
    const TileMem m = tile_mem(smem, a.cap, 2, false);
    double *rho_s = reinterpret_cast<double *>(smem + tile_smem_bytes(a.cap, 2, false));
    double *m_s = rho_s + a.cap, *v_s = m_s + a.cap;   // v: lv / rho^2 (Hernquist-Katz) or the sound speed (Monaghan)
    auto visc = [&](int j, double rho) {
        return P.art_visc == 1 ? hk_lv_r2(P, s, a.div, j) : sound_speed_held(P, rho);
    };
    if (t == 0) bar_init(&bar);
    unsigned parity = 0u;
    for (int p0 = ch.p0; p0 < ch.p1;) {
        if (!aux_tile(&halos[(p0 - ch.p0) >> shift], h, m, s, s.vxy, a.pl.slot + (size_t)blockIdx.x * kListRows * kTile, &bar,
                      parity, a.sc, [&](int j, int k) {
                          const double rho = s.rho[j];
                          rho_s[k] = rho;
                          m_s[k] = s.m[j];
                          v_s[k] = visc(j, rho);
                      }))
            return;
        const bool live = t < h.size;
        const int i = p0 + t;
        if (live) {
            const double2 xy = s.xy[i], v = s.vxy[i];
            const double xi = xy.x, yi = xy.y, vxi = v.x, vyi = v.y;
            const double hi = s.hs[i], inv_hi = 1.0 / hi, rhoi = s.rho[i];
            const double vi = visc(i, rhoi);
            Sum<double> avx, avy, xsx, xsy;
            if (!dead)
                aux_pairs(h, m, s, s.vxy, I, a.cell_start, a.cell, a.pl.count, i, i - ch.p0,
                          [&](int j, int slot, double2 q, double2 w, double hj) {
                    const double dx = xi - q.x, dy = yi - q.y;
                    const double dvx = vxi - w.x, dvy = vyi - w.y;
                    const double rhoj = slot >= 0 ? rho_s[slot] : s.rho[j], mj = slot >= 0 ? m_s[slot] : s.m[j];
                    const PairGeom<double> pg = pair_geom<double, true>(P, dx, dy, hi, inv_hi, hj);
                    if (P.xsph) {
                        const double rbar = 0.5 * (rhoi + rhoj), c = mj * pg.w / rbar;
                        xsx.madd(dvx, c);
                        xsy.madd(dvy, c);
                    }
                    const double vr = dvx * dx + dvy * dy;
                    if ((P.art_visc == 1 || P.art_visc == 2) && vr <= 0.0) {
                        const double vj = slot >= 0 ? v_s[slot] : visc(j, rhoj);
                        double pij;
                        if (P.art_visc == 1) {
                            pij = vi + vj;
                        } else {
                            const double hij = __dmul_rn(__dadd_rn(hi, hj), 0.5);
                            const double scor = (double)0.01f * hij;
                            const double iota = hij * vr / fma(dx, dx, fma(dy, dy, scor * scor));
                            pij = (P.beta_pi * (iota * iota) - P.alpha_pi * iota * (vi + vj) / 2.0) / ((rhoi + rhoj) / 2.0);
                        }
                        avx.madd(-(mj * pij), pg.gfac * pg.dx);
                        avy.madd(-(mj * pij), pg.gfac * pg.dy);
                    }
                });
            a.reg[i] = avx.get();
            a.reg[M + i] = avy.get();
            a.reg[2 * M + i] = xsx.get();
            a.reg[3 * M + i] = xsy.get();
        }
        p0 += h.size;
        if (p0 < ch.p1) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
        }
    }
}

// Density rate drho/dt_i = sum_j m_j (v_i - v_j) . grad_i W_ij over the
// pairs of the right-hand side just evaluated, with the velocities the
// integrator has just written: con_density (density.f90:107-165, called
// after each update, time_integration.f90:128-133, 218-223, 344-349, 372-377)
// and the same sum in Benz_hsml (smoothing_length.f90:62-80).  The pair
// geometry and hsml are those of the right-hand side's state (the reference
// reuses that right-hand side's p_i, p_j and dwdx); the masses are the
// current ones at the call: the right-hand side's for con_density (called
// before mass_evolution), the updated ones for Benz_hsml's own sum (called
// after it).  The sum is FP64 in both precision forms.
//   rho_upd: 0 none, 1 rho = rho_1 + drho/dt dt / 2, 2 rho = rho_1 + drho/dt dt;
//   tail: the step's final hsml (Benz, or Marquis with the new density),
//   its bounds and the VP time step, which the stress epilogue left out.
struct DensArgs {
    State g;             // right-hand side state (positions, hsml, masses)
    State v;             // updated state: velocities in, rho and views out
    const double *mj;    // neighbour masses of the sum
    const double *rho1;  // step-start density
    double *acc;         // Benz's drhodt when den_alg != 2 (kept across steps)
    const double *a2;    // |dv/dt|^2 of the last right-hand side (tse = 1)
    double *hs_next;
    PairList pl;
    const int *cell_start, *cell;
    const Chunk *chunks;
    const unsigned char *halos;
    int cap;
    const Inst *inst;
    Scalars *sc;
    Phys P;
    int rho_upd, tail;
    int dt_div;          // the Monaghan time step's divergence (artificial viscosity)
    // summation density (den_alg = 1, density.f90:41-100): rho_out =
    // (k0 m_i + sum_j m_j W_ij) / (k0 m_i / rho_i + sum_j m_j W_ij / rho_j)
    // over the right-hand side's pairs and kernel values, with the masses
    // m_sum and densities rho_in at the reference's density call; rho_out
    // is o.rho (then m/rho and the packed copies follow) or a scratch array
    // that k_commit_rho copies in
    int sum_mode;
    const double *m_sum, *rho_in;
    double *rho_out;
    // its self term kernel_zero(i) m_i: the reference keeps kernel_zero per
    // particle and sets it in each right-hand side's pair loop for the p_i
    // of every pair, W(0) at the pair's hsml (kernel.f90:503, set to 0 by
    // initialize.f90:60), so a particle that is p_i of no pair keeps an
    // earlier value.  Which particle of a pair is p_i follows the search:
    // direct_find (nnps.f90:41-148) the lower index; the bucket search
    // (nnps.f90:259-411) the lower index within one bucket, else the
    // particle whose bucket has the other's to its right, above, above
    // right or above left.  Of several pairs the serial pair order's last
    // gives the value (it matters only where hsml varies)
    double *k0;
    const int *id;
};

// One part of a tile, particles [p0, p0 + h.size).
__device__ __forceinline__ void density_rate(const DensArgs &a, const Halo &h, const TileMem &m, const double *mj_s,
                                             const double *w_s, const double *rho_s, const Chunk &ch, int p0) {
    const int i = p0 + min((int)threadIdx.x, h.size - 1);   // idle lanes mirror the part's last particle
    const State &g = a.g;
    const Phys &P = a.P;
    const Inst &I = a.inst[ch.q];
    const bool live = (int)threadIdx.x < h.size && !(I.flags & FLAG_RETIRED);   // (a retired basin is not written)
    const bool dead = inst_dead(I.flags);
    const double2 gxy = g.xy[i], vxy = a.v.vxy[i];
    const double xi = gxy.x, yi = gxy.y, hi = g.hs[i];
    const double inv_hi = 1.0 / hi;
    const double vxi = vxy.x, vyi = vxy.y;
    Sum<double> r, rt, num, den;
    // p_i rule of the summation density's kernel_zero (DensArgs)
    const int idi = a.sum_mode ? a.id[i] : 0;
    const long long bxi = (a.sum_mode && P.nnps == 2) ? ref_bin(xi, I.bs) : 0;
    const long long byi = (a.sum_mode && P.nnps == 2) ? ref_bin(yi, I.bs) : 0;
    long long last = -1;   // (position in the serial pair order, category then index)
    double h_last = 0.0;
    auto add = [&](int j, int slot, double2 q, double2 v, double hj) {
        const double mj = slot >= 0 ? mj_s[slot] : a.mj[j];
        PairGeom<double> pg;
        if (a.sum_mode) {
            pg = pair_geom<double, true>(P, xi - q.x, yi - q.y, hi, inv_hi, hj);
            const double mw = (slot >= 0 ? w_s[slot] : a.m_sum[j]) * pg.w;
            num.madd(mw, 1.0);
            den.madd(mw / (slot >= 0 ? rho_s[slot] : a.rho_in[j]), 1.0);
            const int idj = a.id[j];
            int cat = -1;
            if (P.nnps != 2) {
                cat = idj > idi ? 0 : -1;
            } else {
                const long long dx = ref_bin(q.x, I.bs) - bxi, dy = ref_bin(q.y, I.bs) - byi;
                if (dx == 0 && dy == 0) cat = idj > idi ? 0 : -1;
                else if (dy == 0 && dx == 1) cat = 1;     // right
                else if (dy == 1 && dx == 0) cat = 2;     // up
                else if (dy == 1 && dx == 1) cat = 3;     // up-right
                else if (dy == 1 && dx == -1) cat = 4;    // up-left
            }
            const long long key = cat < 0 ? -1 : ((long long)cat << 32) | (long long)(unsigned)idj;
            if (key > last) {
                last = key;
                h_last = hj;
            }
        } else {
            pg = pair_geom<double, false>(P, xi - q.x, yi - q.y, hi, inv_hi, hj);
        }
        const double dvx = vxi - v.x, dvy = vyi - v.y;
        const double t = fma(dvx, pg.gfac * pg.dx, dvy * (pg.gfac * pg.dy));
        r.madd(mj, t);
        // time_step.f90:93-109: the current masses (after mass_evolution)
        if (a.dt_div) rt.madd(slot >= 0 && !a.sum_mode ? w_s[slot] : a.v.m[j], t);
    };
    if (!dead && (int)threadIdx.x < h.size)
        aux_pairs(h, m, g, a.v.vxy, I, a.cell_start, a.cell, a.pl.count, i, i - ch.p0, add);
    const double drhodt = r.get();
    const double dt = a.sc->dt;
    const State &o = a.v;
    double rhon = o.rho[i];
    if (a.sum_mode) {
        double k0 = a.k0[i];
        if (last >= 0) k0 = kernel_zero(P, (hi + h_last) / 2.0);   // nnps.f90:278
        const double k0m = k0 * a.m_sum[i];
        rhon = (k0m + num.get()) / (k0m / a.rho_in[i] + den.get());
        if (live) {
            a.k0[i] = k0;
            a.rho_out[i] = rhon;
            if (a.rho_out == o.rho) {
                refresh_views(o, i);
            }
        }
    } else if (a.rho_upd && live) {
        rhon = (a.rho_upd == 1) ? a.rho1[i] + drhodt * dt / 2.0 : a.rho1[i] + drhodt * dt;
        o.rho[i] = rhon;
        refresh_views(o, i);
    }
    if (!a.tail) return;
    const double hs_old = g.hs[i];
    double hsn = hs_old;
    if (P.sle == 1) {
        // Benz_hsml, smoothing_length.f90:82-94.  Without con_density the
        // reference adds to its drhodt array, never cleared: kept per
        // particle across steps (and re-sorts) here.
        double d = drhodt;
        if (a.acc) {
            d = a.acc[i] + drhodt;
            if (live) a.acc[i] = d;
        }
        const double dhs = -hs_old * d / 2.0 / rhon;
        hsn = hs_old + dhs * dt;
        if (hsn < 0.0) hsn = hsn - dhs * dt;
    } else if (P.sle == 2) {                                   // smoothing_length.f90:136-142
        hsn = sqrt(o.m[i] / rhon) * (double)P.hsml_multiplicity;
        if (hsn > P.max_hsml) hsn = P.max_hsml;
    }
    if (live && P.sle != 0) a.hs_next[i] = hsn;
    // (dead lanes contribute neutral values: the particle they mirror may
    // already have been updated by its own thread)
    unsigned active = 0u;
    unsigned long long v[kBounds] = {0ull, ~0ull, 0ull, ~0ull, 0ull};
    if (P.sle != 0) {
        active |= 2u | 4u;
        if (live) {
            v[1] = dbits(hsn);
            v[2] = dbits(hsn);
        }
    }
    if (P.tse != 0) {                                          // time_step.f90:20-26
        active |= 8u;
        // |div v| = |sum_j m_j (v_i - v_j) . grad W| / rho_i (time_step.f90:108-111)
        const double adiv = a.dt_div ? fabs(rt.get() / rhon) : 0.0;
        if (live) v[3] = dbits(dt_candidate(P, hsn, P.tse == 1 ? a.a2[i] : 0.0, rhon, adiv));
    }
    block_bounds(a.sc, nullptr, active, v);
}

__global__ void __launch_bounds__(kBlock) k_density_rate(const __grid_constant__ DensArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Halo h;
    __shared__ __align__(8) unsigned long long bar;
    const int t = threadIdx.x;
    const Chunk ch = a.chunks[blockIdx.x];
    const int shift = part_shift(ch);
    if (ch.spare >= a.inst[ch.q].spares) return;   // (an unused spare tile)
    const Halo *halos = reinterpret_cast<const Halo *>(a.halos) + (size_t)blockIdx.x * kParts;
    const TileMem m = tile_mem(smem, a.cap, 2, false);
    double *mj_s = reinterpret_cast<double *>(smem + tile_smem_bytes(a.cap, 2, false));
    double *w_s = mj_s + a.cap, *rho_s = w_s + a.cap;   // w: the summation's mass, or the time step's
    const double *w_src = a.sum_mode ? a.m_sum : a.dt_div ? a.v.m : nullptr;
    if (t == 0) bar_init(&bar);
    unsigned parity = 0u;
    for (int p0 = ch.p0; p0 < ch.p1;) {
        if (!aux_tile(&halos[(p0 - ch.p0) >> shift], h, m, a.g, a.v.vxy, a.pl.slot + (size_t)blockIdx.x * kListRows * kTile,
                      &bar, parity, a.sc, [&](int j, int k) {
                          mj_s[k] = a.mj[j];
                          if (w_src) w_s[k] = w_src[j];
                          if (a.sum_mode) rho_s[k] = a.rho_in[j];
                      }))
            return;
        density_rate(a, h, m, mj_s, w_s, rho_s, ch, p0);
        p0 += h.size;
        if (p0 < ch.p1) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
        }
    }
}

// The summation density written to scratch by the second of two passes
// into the state (the first pass read the state's density).
__global__ void k_commit_rho(int n, const double *__restrict__ src, State o, const int *__restrict__ pinst,
                             const Inst *__restrict__ inst) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || (inst[pinst[i]].flags & FLAG_RETIRED)) return;
    const double r = src[i];
    o.rho[i] = r;
    refresh_views(o, i);
}

// New hsml of the next step (sle = 1, 2) and its FP32 copy.
__global__ void __launch_bounds__(256) k_commit_hsml(int n, const double *__restrict__ hs_next, State s0, Scalars *sc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    // how far any hsml grew, for the Verlet lists' bound (NaN: as infinity)
    double grown = i < n ? hs_next[i] - s0.hs[i] : 0.0;
    if (!(grown <= 1e300)) grown = INFINITY;
    block_max_u64(&sc->acc_dh, dbits(fmax(grown, 0.0)));
    if (i >= n) return;
    const double v = hs_next[i];
    const float vf = (float)v;
    s0.hs[i] = v;
    s0.hsf[i] = vf;
    if (s0.hmm) s0.hmm[i].x = vf;
}

// End of a predictor-corrector step: time_step's new dt, current_time += dt
// (time_integration.f90:71, using the dt computed at the end of the step),
// and the new hsml bounds.
// (One basin per context when tse = 2 or sle != 0: instance 0 carries its
// hsml bounds.)  Every instance's current_time advances by the same dt.
constexpr int kFinishThreads = 256;
__global__ void __launch_bounds__(kFinishThreads) k_step_finish(Scalars *sc, Inst *inst, int ninst, int tse,
                                                                int sle) {
    pass_begin();
    __shared__ double dt, grown;
    if (threadIdx.x == 0) {
        grown = 0.0;
        if (tse != 0) {
            sc->dt = bitsd(sc->acc_dt);
            sc->acc_dt = dbits(INFINITY);
        }
        dt = sc->dt;
        sc->t = sc->t + dt;
        if (sle != 0) {
            sc->hmin = bitsd(sc->acc_hmin);
            sc->hmax = fmax(sc->hmax, bitsd(sc->acc_hmax));
            sc->bs = 2.0 * sc->hmin;
            sc->acc_hmin = dbits(INFINITY);
            sc->acc_hmax = 0ull;
            grown = bitsd(sc->acc_dh);
            sc->acc_dh = 0ull;
            inst[0].hmin = sc->hmin;
            inst[0].hmax = sc->hmax;
            inst[0].bs = sc->bs;
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < ninst; k += kFinishThreads) {
        Inst &I = inst[k];
        I.t = I.t + dt;
        // the Verlet lists: built in this step unless they were valid before
        // it; stale when the step's second right-hand side had to build its
        // own, or when another step like this one could outrun them
        const double half = sqrt(bitsd(I.half2_bits)), step = sqrt(bitsd(I.step2_bits));
        const double old = I.list_ok ? I.list_d : 0.0;
        const double moved = old + step + 0.5 * grown;
        const double room = 0.5 * I.delta * (1.0 - 1e-9) - old;   // (as lists_valid)
        I.list_ok = (room >= 0.0 && bitsd(I.half2_bits) <= room * room && 2.0 * (moved + half) <= I.delta) ? 1 : 0;
        I.list_d = moved;
        // displacement since the sort and largest coordinate: each step adds
        // the farthest any particle moved in it
        I.disp += step;
        I.xabs_bits = dbits(bitsd(I.xabs_bits) + step);
        I.half2_bits = 0ull;
        I.step2_bits = 0ull;
    }
}

// The Euler step writes its result into S1 (S0 is read by the pair sums of
// the same pass); this copies it back, with the packed copies.
__global__ void k_copy_s1_to_s0(int n, State s1, State s0) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    s0.xy[i] = s1.xy[i];
    s0.vxy[i] = s1.vxy[i];
    s0.mm[i] = s1.mm[i];
    s0.h[i] = s1.h[i];
    s0.A[i] = s1.A[i];
    s0.rho[i] = s1.rho[i];
    if (s1.m != s0.m) s0.m[i] = s1.m[i];
    if (s0.hmm) s0.hmm[i] = s1.hmm[i];
}

// (FLAG_TIMEOUT stays until the state is set anew: what the passes keep from one
// step to the next may be incomplete)
__global__ void k_reset_stats(Scalars *sc) {
    sc->maxip = 0;
    sc->minip = 0x7fffffff;
    sc->sumip = 0ull;
    sc->noip = 0;
    sc->flags &= FLAG_TIMEOUT;
}

inline int nblk(long long n, int b) { return (int)((n + b - 1) / b); }

// The chunks of the current layout: src holds, per basin in memory order, its
// offset, particles, first chunk and slot.
__device__ __forceinline__ int4 chunk_basin(int c, int nsrc, const int4 *src) {
    int lo = 0, hi = nsrc - 1;   // the last basin whose first chunk is at or before c
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (src[mid].z <= c) lo = mid;
        else hi = mid - 1;
    }
    return src[lo];
}
__global__ void k_chunks(int nchunks, int nsrc, const int4 *__restrict__ src, int size, Chunk *__restrict__ chunks) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nchunks) return;
    const int4 b = chunk_basin(c, nsrc, src);
    const int k = c - b.z, tiles = (b.y + size - 1) / size;
    if (k < tiles) chunks[c] = Chunk{b.x + k * size, min(b.x + (k + 1) * size, b.x + b.y), b.w, -1};
    else chunks[c] = Chunk{0, 0, b.w, k - tiles};
}

// Cuts the tiles of the basins just sorted whose halo would not fit: a sparse
// cell row's tile spans many cells of its full neighbour rows.  One warp per tile
// cuts it from the front, each time the longest power of two of particles that
// fits, down to single ones (65,536 particles, one of whose cell rows holds a few
// of them: 57 us per step; 112 when parts of 8 were the shortest, one of which
// then read its neighbours from global memory).  The parts go to the basin's
// spare tiles, so that they run beside the others; what finds no room there stays
// together and is worked off part by part.
constexpr int kSplitWarps = 4;
__global__ void __launch_bounds__(32 * kSplitWarps)
    k_split(int nchunks, int nsrc, const int4 *__restrict__ src, int size, Chunk *__restrict__ chunks, DueMask due,
            Inst *inst, const int *__restrict__ cell_start, const int *__restrict__ cell, int cap) {
    static_assert(kTile == 128, "sizes tried");
    __shared__ unsigned char starts[kSplitWarps][kTile];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * kSplitWarps + w;
    if (c >= nchunks) return;
    const int4 b = chunk_basin(c, nsrc, src);
    const int k = c - b.z, tiles = (b.y + size - 1) / size;
    if (k >= tiles || !((due.w[b.w >> 6] >> (b.w & 63)) & 1ull)) return;
    Inst &I = inst[b.w];
    const int p0 = b.x + k * size, p1 = min(p0 + size, b.x + b.y);
    const int R = stencil_radius(I.hmax, inst_disp(I), inst_grid(I, cell_start), I.hmax + I.delta);
    int parts = 0;
    for (int p = p0; p < p1;) {
        // (lane k tries 128 >> k; nothing fits: the rest stays one part)
        const int e = min(p + (kTile >> min(lane, 7)), p1);
        bool fits = false;
        if (lane < 8 && R <= kMaxRadius) {
            int lo[kMaxSeg], off[kMaxSeg + 1];
            fits = halo_ranges(I, cell_start, cell[p], cell[e - 1], R, lo, off) <= cap;
        }
        const unsigned ok = __ballot_sync(0xffffffffu, fits);
        if (lane == 0) starts[w][parts] = (unsigned char)(p - p0);
        ++parts;
        p = ok ? min(p + (kTile >> (__ffs(ok) - 1)), p1) : p1;
    }
    __syncwarp();
    const int extra = parts - 1, room = spare_tiles(tiles);
    int at = 0;
    if (lane == 0 && extra > 0) at = atomicAdd(&I.spares, extra);
    at = __shfl_sync(0xffffffffu, at, 0);
    const int more = max(min(extra, room - at), 0);   // parts that get a tile of their own
    auto start = [&](int q) { return q <= more && q < parts ? p0 + starts[w][q] : p1; };
    for (int q = 1 + lane; q <= more; q += 32)
        chunks[b.z + tiles + at + q - 1] = Chunk{start(q), start(q + 1), b.w, at + q - 1};
    if (lane == 0) chunks[c] = Chunk{p0, start(1), b.w, -1};
}

// Halo slots of a tile in shared memory.  Three rows of cells around 128
// particles take up to 520 slots at hsml = 2.4 spacings and 650 at the
// reference's 3 spacings; five rows (after more motion), or a sparse row's tile
// among full ones, about 850.  A context of up to kSmallTiles has room for the
// latter (40,401 particles with the density passes: 158 -> 137 us per step); a
// larger one is faster with what shared memory then leaves to the L1 cache
// (1,048,576 particles, us per step with room for 528, 576, 640, 832: FP64 541,
// 542, 547, 563, mixed 528, 531, 560, 579), but not with less than 576 where
// particles move: a fifth of hsml between sorts, FP64 1066, 908, 916, 936, mixed
// 1046, 892, 935, 973; or at 2.6 spacings, FP64 596, 544, 548, 564.
int tile_cap(const simp_ctx *c) {
    if (c->halo_cap > 0) return c->halo_cap;
    if (c->nchunks <= kSmallTiles) return 832;
    return c->uniform ? 576 : 704;
}

// Whether a pass fetches its epilogue's values ahead of its pairs: where they
// come from DRAM, which is where the arrays of a step (about 280 bytes per
// particle) outgrow two thirds of L2.  us per step without and with it, FP64 and
// mixed: 176,400 particles 122.3 and 122.9, 114.9 and 116.5; 262,144 158.6 and
// 159.8, 162.2 and 164.0; 313,600 189.4 and 188.7, 201.5 and 200.8; 399,424 237.9
// and 234.1, 250.6 and 249.2; 1,048,576 558 and 548, 560 and 546.
bool prefetch_own(const simp_ctx *c) { return 280.0 * c->n > 2.0 / 3.0 * c->l2_bytes; }

TauRec tau_rec(simp_ctx *c) {
    TauRec r;
    r.ta = c->tau_a;
    r.tb = c->tau_b;
    r.tq = c->tau_q;
    return r;
}

PairList pair_list(simp_ctx *c) {
    PairList pl;
    pl.slot = c->pair_slot;
    pl.count = c->pair_count;
    return pl;
}

// Launches a kernel that calls pass_begin, overlapping the one before it where
// the context says so (within a step graph: after the kernel before it, which
// may be any).
template <class... P, class... A>
void launch_pass(simp_ctx *c, void (*k)(P...), int grid, int block, size_t smem, const A &...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = c->overlap_launches ? 1 : 0;
    cudaLaunchKernelEx(&cfg, k, args...);   // (an error is found by the caller's next check)
}

// The passes' form of a context's current layout, for f.
template <class T_, int SKF, int HS, int BLOCKS>
struct Form {
    using T = T_;
    static constexpr int skf = SKF, hs = HS, blocks = BLOCKS;
};
template <class T, int SKF, int BLOCKS, class F>
void with_hsml_form(const simp_ctx *c, F &&f) {
    if (c->uniform) f(Form<T, SKF, HSML_ONE, BLOCKS>());
    else if (c->max_inst == 1 || SKF == 0) f(Form<T, SKF, HSML_VARIED, BLOCKS>());   // (the generic kernels' arithmetic is one)
    else f(Form<T, SKF, SKF ? HSML_EITHER : HSML_VARIED, BLOCKS>());
}
template <int SKF, class F>
void with_kernel_form(const simp_ctx *c, F &&f) {
    if (c->prm.precision != SIMP_PREC_MIXED) with_hsml_form<double, SKF, 4>(c, f);
    else if (c->nchunks <= kSmallTiles) with_hsml_form<float, SKF, 4>(c, f);
    else with_hsml_form<float, SKF, 5>(c, f);
}
template <class F>
void with_form(const simp_ctx *c, F &&f) {
    switch (skf_compiled(c->prm.skf)) {
        case SIMP_SKF_CUBIC: with_kernel_form<SIMP_SKF_CUBIC>(c, f); break;
        case SIMP_SKF_WENDLAND_C6: with_kernel_form<SIMP_SKF_WENDLAND_C6>(c, f); break;
        default: with_kernel_form<0>(c, f);
    }
}

}  // namespace

void launch_chunks(simp_ctx *c) {
    if (c->nchunks == 0) return;
    k_chunks<<<nblk(c->nchunks, 256), 256, 0, c->stream>>>(c->nchunks, c->nsrc, c->chunk_src, kTile, c->chunks);
    c->launches += 1;
}
void launch_split(simp_ctx *c, const DueMask &due) {
    if (c->nchunks == 0) return;
    k_split<<<nblk(c->nchunks, kSplitWarps), 32 * kSplitWarps, 0, c->stream>>>(
        c->nchunks, c->nsrc, c->chunk_src, kTile, c->chunks, due, c->inst_dev, c->cell_start, c->cell, tile_cap(c));
    c->launches += 1;
}

namespace {
__global__ void k_uncut(Inst *inst, int ninst) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= ninst) return;
    inst[q].list_ok = 0;
    inst[q].spares = 0;
}
}  // namespace
void launch_recut(simp_ctx *c) {
    k_uncut<<<nblk(c->ninst, 128), 128, 0, c->stream>>>(c->inst_dev, c->ninst);
    c->launches += 1;
    launch_chunks(c);
    DueMask all;
    for (unsigned long long &w : all.w) w = ~0ull;
    launch_split(c, all);
}

// Lets the kernels of the current layout's form take their shared memory.  Only
// those: asking loads a kernel, and loading every form with the first context of
// a process took 28 to 39 ms instead of 12.
int passes_configure(simp_ctx *c) {
    const int form = (c->uniform ? 1 : 0) | (c->nchunks <= kSmallTiles ? 2 : 0);
    if (c->pass_form == form) return SIMP_OK;
    cudaError_t e = cudaSuccess;
    auto allow = [&](auto *k) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostTileSmem);
    };
    with_form(c, [&](auto w) {
        using W = decltype(w);
        allow(k_kinematic<typename W::T, W::skf, W::hs, W::blocks>);
        allow(k_stress<typename W::T, W::skf, W::hs, W::blocks>);
    });
    // (the passes that enqueue_step and simp_gpu_single_step may add)
    const simp_params &p = c->prm;
    if (c->reg) allow(k_regularize);
    if (p.den_alg == 1 || p.den_alg == 2 || p.sle == 1 || (p.tse == 1 && p.artificial_visc)) allow(k_density_rate);
    if (e != cudaSuccess) return simp_cuda_check(c, e, "cudaFuncSetAttribute (tile shared memory)");
    c->pass_form = form;
    return SIMP_OK;
}

void launch_kinematic(simp_ctx *c, const State &s, bool diag, bool second) {
    SIMP_RANGE("kinematic pass");
    if (c->nchunks == 0) return;
    KinArgs a{};
    a.s = s;
    a.cell_start = c->cell_start;
    a.bstart = c->bcell_start;
    a.inst = c->inst_dev;
    a.cell = c->cell;
    a.P = c->phys;
    a.sc = c->sc;
    a.div = c->div;
    a.rec = tau_rec(c);
    a.diag = diag ? c->diag : nullptr;
    a.pl = pair_list(c);
    a.maxn = c->maxn;
    a.single = c->max_inst == 1;
    a.prefetch = prefetch_own(c);
    a.chunks = c->chunks;
    a.halos = c->halos;
    a.xyr = c->xyr;
    a.halo_walls = c->halo_walls;
    a.cap = tile_cap(c);
    a.second = second ? 1 : 0;
    with_form(c, [&](auto w) {
        using W = decltype(w);
        launch_pass(c, k_kinematic<typename W::T, W::skf, W::hs, W::blocks>, c->nchunks, kTile,
                    tile_smem_bytes(a.cap, 3, c->uniform), a);
    });
    c->launches += 1;
}

void launch_stress(simp_ctx *c, const State &rhs, const State &base, EpiMode mode) {
    SIMP_RANGE("stress pass");
    if (c->nchunks == 0) return;
    StressArgs a{};
    a.rhs = rhs;
    a.base = base;
    a.out = (mode == EPI_PREDICT || mode == EPI_EULER) ? c->s1 : c->s0;
    a.cell_start = c->cell_start;
    a.inst = c->inst_dev;
    a.cell = c->cell;
    a.bx = c->bx;
    a.by = c->by;
    a.bm = c->bm;
    a.bnx = c->bnx;
    a.bny = c->bny;
    a.bstart = c->bcell_start;
    a.nb = c->nb;
    a.P = c->phys;
    a.sc = c->sc;
    a.div = c->div;
    a.rec = tau_rec(c);
    a.pl = pair_list(c);
    a.rates = c->rates;
    a.reg = c->reg;
    a.hs_next = c->tmp;   // hsml of the next step (committed by launch_step_finish)
    a.maxn = c->maxn;
    a.mode = mode;
    a.single = c->max_inst == 1;
    a.prefetch = prefetch_own(c);
    a.chunks = c->chunks;
    a.halos = c->halos;
    a.halo_walls = c->halo_walls;
    a.cap = tile_cap(c);
    with_form(c, [&](auto w) {
        using W = decltype(w);
        launch_pass(c, k_stress<typename W::T, W::skf, W::hs, W::blocks>, c->nchunks, kTile,
                    stress_smem_bytes(a.cap, Rec<typename W::T>::stress_arrays, c->uniform), a);
    });
    c->launches += 1;
}

void launch_regularize(simp_ctx *c, const State &s) {
    if (!c->reg) return;
    SIMP_RANGE("regularisation pass");
    RegArgs a{};
    a.s = s;
    a.div = c->div;
    a.pl = pair_list(c);
    a.cell_start = c->cell_start;
    a.cell = c->cell;
    a.chunks = c->chunks;
    a.halos = c->halos;
    a.cap = tile_cap(c);
    a.inst = c->inst_dev;
    a.sc = c->sc;
    a.P = c->phys;
    a.reg = c->reg;
    a.maxn = c->maxn;
    k_regularize<<<c->nchunks, kTile, aux_smem_bytes(a.cap), c->stream>>>(a);
    c->launches += 1;
}

void launch_density_rate(simp_ctx *c, const State &g, const State &v, int rho_upd, bool tail) {
    SIMP_RANGE("density-rate pass");
    DensArgs a{};
    a.g = g;
    a.v = v;
    a.rho1 = c->s0.rho;
    a.acc = c->drhodt;
    a.mj = c->drhodt ? v.m : g.m;
    a.a2 = c->rates;
    a.hs_next = c->tmp;
    a.pl = pair_list(c);
    a.cell_start = c->cell_start;
    a.cell = c->cell;
    a.chunks = c->chunks;
    a.halos = c->halos;
    a.cap = tile_cap(c);
    a.inst = c->inst_dev;
    a.sc = c->sc;
    a.P = c->phys;
    a.rho_upd = rho_upd;
    a.tail = tail ? 1 : 0;
    a.dt_div = (tail && c->prm.tse == 1 && c->prm.artificial_visc) ? 1 : 0;
    k_density_rate<<<c->nchunks, kTile, aux_smem_bytes(a.cap), c->stream>>>(a);
    c->launches += 1;
}

void launch_sum_density(simp_ctx *c, const State &g, const State &v, const double *m_sum, const double *rho_in,
                        double *rho_out, bool tail) {
    SIMP_RANGE("summation-density pass");
    DensArgs a{};
    a.g = g;
    a.v = v;
    a.rho1 = c->s0.rho;
    a.acc = c->drhodt;
    a.mj = c->drhodt ? v.m : g.m;
    a.a2 = c->rates;
    a.hs_next = c->tmp;
    a.pl = pair_list(c);
    a.cell_start = c->cell_start;
    a.cell = c->cell;
    a.chunks = c->chunks;
    a.halos = c->halos;
    a.cap = tile_cap(c);
    a.inst = c->inst_dev;
    a.sc = c->sc;
    a.P = c->phys;
    a.rho_upd = 0;
    a.tail = tail ? 1 : 0;
    a.dt_div = (tail && c->prm.tse == 1 && c->prm.artificial_visc) ? 1 : 0;
    a.sum_mode = 1;
    a.m_sum = m_sum;
    a.rho_in = rho_in;
    a.rho_out = rho_out;
    a.k0 = c->k0;
    a.id = c->id;
    k_density_rate<<<c->nchunks, kTile, aux_smem_bytes(a.cap), c->stream>>>(a);
    c->launches += 1;
}

void launch_commit_rho(simp_ctx *c, const double *src, const State &o) {
    k_commit_rho<<<nblk(c->n, 256), 256, 0, c->stream>>>(c->n, src, o, c->pinst, c->inst_dev);
    c->launches += 1;
}

void launch_step_finish(simp_ctx *c) {
    if (c->prm.sle != 0) {
        k_commit_hsml<<<nblk(c->n, 256), 256, 0, c->stream>>>(c->n, c->tmp, c->s0, c->sc);
        c->launches += 1;
    }
    launch_pass(c, k_step_finish, 1, kFinishThreads, 0, c->sc, c->inst_dev, c->ninst, (int)c->prm.tse, (int)c->prm.sle);
    c->launches += 1;
}

void launch_copy_s1_to_s0(simp_ctx *c) {
    k_copy_s1_to_s0<<<nblk(c->n, 256), 256, 0, c->stream>>>(c->n, c->s1, c->s0);
    c->launches += 1;
}

void launch_reset_stats(simp_ctx *c) {
    k_reset_stats<<<1, 1, 0, c->stream>>>(c->sc);
    c->launches += 1;
}

}  // namespace simp
