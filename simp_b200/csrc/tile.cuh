// Tiles of the pair passes.
//
// A tile is up to kTile consecutive particles of one basin, one per thread of
// a block.  Particles are stored in cell order, row-major, so the cells within
// R of a tile's cells are 2R + 1 runs of consecutive cell keys, hence 2R + 1
// contiguous index ranges (its halo), whether or not the tile wraps from one
// cell row into the next.  A block copies its halo's records to shared memory
// (one bulk copy per range and array) and the pair arithmetic gathers from
// there: a gather from global memory waits for its slowest lane's L2 miss on
// nearly every pair (12 of 17 cycles between a warp's instructions, at issue
// slots 25% and L1 40% busy), one from shared memory never does.
//
// The candidates of a particle are a Verlet list of slots, 16 bits each, copied
// to shared memory with the halo.  A kinematic pass whose basin's lists are
// stale first builds them (k_kinematic: the cell stencil against FP32 copies).
// The exact FP64 criterion is applied to every candidate in each pass.
// Candidates are in increasing index order, so the sums depend neither on the
// tile shape nor on when a list was built.
//
// A particle of more than kListRows candidates finds its pairs in the halo's cell
// stencil, whatever the others of its tile do (65,536 particles, FP64, with 48
// neighbours each: 221 us per step, 341 when such a particle sent its tile to
// global memory and 254 with lists per particle in global memory).  A tile whose
// halo exceeds the shared-memory capacity (a sparse cell row next to full ones) is
// cut (k_split); one that comes to exceed it later, by motion, is taken in parts
// one after another.  What still does not fit, or has a stencil radius above
// kMaxRadius, reads its neighbours from global memory.  The arithmetic and its
// order are the same everywhere.
#pragma once

#include "pass_common.cuh"

namespace simp {
namespace pass {

constexpr int kMaxRadius = 2;
constexpr int kMaxSeg = 2 * kMaxRadius + 1;

// The halo of a tile or part of one, one record per part.
enum : int { HALO_NONE = 0, HALO_TILE = 1, HALO_GLOBAL = 2 };
struct Halo {
    int kind, nseg;
    int walls;                 // cells around its own that hold every wall pair, 0: none
    int rows;                  // longest list of one of its particles, kListRows at most
    int lo[kMaxSeg];           // first particle of each range
    int off[kMaxSeg + 1];      // its first slot, and the total
    int size;                  // particles in this part of the tile
};
static_assert(sizeof(Halo) == kHaloBytes, "ctx.h: kHaloBytes");
// A halo's walls, by cell row: from the basin's first, and how many (-1 in the
// first row: more rows than there is room for).
constexpr int kMaxWallRows = 7;
struct HaloWalls {
    int lo[kMaxWallRows], n[kMaxWallRows];
    int spare[2];
};
static_assert(sizeof(HaloWalls) == kHaloWallBytes, "ctx.h: kHaloWallBytes");

// Place of candidate k in a particle's list (PairList): consecutive candidates
// of a thread share a 32-bit word.
__host__ __device__ __forceinline__ int list_at(int k, int column) { return ((k >> 1) * kTile + column) * 2 + (k & 1); }

// Bulk copies to shared memory, completing on an mbarrier.
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(unsigned long long *bar) {
    asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void bar_expect(unsigned long long *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
// Waits for the barrier's phase; gives up after a bounded number of tries, which
// take 4 us each: about a second.
constexpr int kWaitTries = 1 << 18;
__device__ __forceinline__ bool bar_wait(unsigned long long *bar, unsigned parity) {
    for (int k = 0; k < kWaitTries; ++k) {
        unsigned ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// The wait for a tile's copies.  Where they do not arrive, the step reports it,
// and the thread gives them as long again to end, marks its block and goes on
// without pairs, so that the block's barriers still meet.  The block leaves as a
// whole where it next looks at the mark, behind a barrier: the mark is the least
// `at` of a wait that failed, so that a thread that looks late does not see one
// of a wait that others have reached since.
constexpr int kNoneFailed = 0x7fffffff;
inline __device__ __noinline__ void copies_failed(unsigned long long *bar, unsigned parity, int at, int *failed, int *flags) {
    atomicOr(flags, FLAG_TIMEOUT);
    bar_wait(bar, parity);
    atomicMin(failed, at);
}
__device__ __forceinline__ bool copies_arrive(unsigned long long *bar, unsigned parity, int at, int *failed, int *flags) {
    if (bar_wait(bar, parity)) return true;
    copies_failed(bar, parity, at, failed, flags);
    return false;
}
// A block's mark at its start: where copies of an earlier pass did not arrive its
// records may be missing, and there is nothing to do.  Asked by one thread, since
// other blocks may set the flag meanwhile.
__device__ __forceinline__ int failed_before(const Scalars *sc) {
    return (*(const volatile int *)&sc->flags & FLAG_TIMEOUT) ? -1 : kNoneFailed;
}

// Shared memory of a tile: records of 16 bytes per particle by array (xy and
// the pass's own), hsml where it varies, and the lists.  While lists are built
// the FP32 copies stand where the pass's own records go.
struct TileMem {
    unsigned char *rec[3];
    double *hs;
    unsigned short *list;           // kListRows slots per thread
    __device__ __forceinline__ float2 *f() const { return reinterpret_cast<float2 *>(rec[2]); }
    __device__ __forceinline__ float *hf() const { return reinterpret_cast<float *>(rec[1]); }
};

__host__ __device__ constexpr size_t tile_smem_bytes(int cap, int arrays, bool uniform) {
    return (size_t)cap * (16 * arrays + (uniform ? 0 : 8)) + (size_t)kListRows * kTile * sizeof(unsigned short);
}

__device__ __forceinline__ TileMem tile_mem(unsigned char *p, int cap, int arrays, bool uniform) {
    TileMem m;
    for (int a = 0; a < 3; ++a) m.rec[a] = p + (size_t)(a < arrays ? a : 0) * 16 * cap;
    p += (size_t)16 * cap * arrays;
    m.hs = reinterpret_cast<double *>(p);
    if (!uniform) p += (size_t)cap * sizeof(double);
    m.list = reinterpret_cast<unsigned short *>(p);
    return m;
}

// The ranges of a halo of radius R around cells ka .. kb, and their total.
__device__ __forceinline__ int halo_ranges(const Inst &I, const int *cell_start, int ka, int kb, int R, int (&lo)[kMaxSeg],
                                           int (&off)[kMaxSeg + 1]) {
    const int end = I.base + I.ncx * I.ncy, nseg = 2 * R + 1;
    int a[kMaxSeg], b[kMaxSeg];
#pragma unroll
    for (int d = 0; d < kMaxSeg; ++d) {
        if (d >= nseg) break;
        const int sh = (d - R) * I.ncx;
        a[d] = cell_start[clampi(ka + sh - R, I.base, end)];
        b[d] = cell_start[clampi(kb + sh + R + 1, I.base, end)];
    }
    int total = 0, past = 0;
#pragma unroll
    for (int d = 0; d < kMaxSeg; ++d) {
        if (d >= nseg) break;
        // (a tile of more than a cell row: its ranges meet)
        lo[d] = max(a[d], past);
        off[d] = total;
        total += max(b[d] - lo[d], 0);
        past = max(b[d], past);
    }
    off[nseg] = total;
    return total;
}

// Parts of a tile begin at multiples of 8 particles, or anywhere in a tile of 16
// or fewer: either way it has at most 16 parts, and records.
constexpr int kParts = kTile / kPartMin;
__device__ __forceinline__ int part_shift(const Chunk &ch) { return ch.p1 - ch.p0 <= kParts ? 0 : 3; }
static_assert(kPartMin == 1 << 3, "part_shift");

// The halo of the longest part of a tile from p0 on that fits (up to p1, parts in
// steps of 1 << shift), and its walls, if it has any.  `moved`: how far any of the
// tile's particles is from where it was sorted.  Called by a warp: a lane per
// size, and a lane per row of walls (262,144 particles that move a fifth of hsml
// between sorts, so that lists are built in every step, FP64, at 528 slots: 288 us
// per step; 343 with one thread that halved the size until it fitted).
inline __device__ __noinline__ void make_halo(const Inst &I, const int *cell_start, const int *bstart, const int *cell, int p0,
                                       int p1, int shift, int cap, double moved, Halo &h, HaloWalls &hw) {
    const int lane = threadIdx.x & 31;
    const Grid g = inst_grid(I, cell_start);
    // The farthest of a basin's particles are few: with the tile's own distance
    // for one side of a pair, the tiles of the others keep a smaller radius (one
    // particle in a thousand moves a fifth of hsml between sorts, FP64: 262,144
    // particles 243 -> 208 us per step, 1,048,576 875 -> 692).
    const double disp = inst_disp(I);
    const int R = stencil_radius(I.hmax, 0.5 * (fmin(moved, disp) + disp), g, I.hmax + I.delta);
    const int e = min(p0 + max((kParts - lane) << shift, 1), p1);
    const int ka = cell[p0], ke = cell[e - 1], end = I.base + I.ncx * I.ncy;
    int lo[kMaxSeg], off[kMaxSeg + 1];
    const bool fits = lane < kParts && R <= kMaxRadius && halo_ranges(I, cell_start, ka, ke, R, lo, off) <= cap;
    const unsigned ok = __ballot_sync(0xffffffffu, fits);
    // (the longest; if none fits the shortest, or all where the radius is too wide)
    const int w = ok ? __ffs(ok) - 1 : R <= kMaxRadius ? kParts - 1 : 0;
    if (lane == w) {
        h.kind = fits ? HALO_TILE : HALO_GLOBAL;
        h.nseg = 2 * R + 1;
        h.rows = 0;
        h.size = e - p0;
        if (fits) {
#pragma unroll
            for (int d = 0; d < kMaxSeg; ++d) {
                if (d >= 2 * R + 1) break;
                h.lo[d] = lo[d];
                h.off[d + 1] = off[d + 1];
            }
            h.off[0] = 0;
        }
    }
    // walls within b_length of any place its particles take while the lists
    // stay valid (they move less than delta)
    const int kb = __shfl_sync(0xffffffffu, ke, w);
    const int Rb = wall_radius(disp, g, I.b_length + I.delta), rows = 2 * Rb + 1;
    auto first = [&](int d) { return bstart[clampi(ka + (d - Rb) * I.ncx - Rb, I.base, end)]; };
    auto past = [&](int d) { return bstart[clampi(kb + (d - Rb) * I.ncx + Rb + 1, I.base, end)]; };
    bool any = false;
    for (int d = lane; d < rows; d += 32) any = any || past(d) > first(d);
    any = __any_sync(0xffffffffu, any);
    if (lane == 0) h.walls = any ? Rb : 0;
    if (!any) return;
    // each row's, from where the rows before it end
    const int b0 = lane < rows ? first(lane) : 0, b1 = lane < rows ? past(lane) : 0, b_first = bstart[I.base];
    int upto = b1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto = max(upto, u);
    }
    const int before = max(__shfl_up_sync(0xffffffffu, upto, 1), 0);
    if (lane < kMaxWallRows) {
        const int b = lane > 0 ? max(b0, before) : b0;
        hw.lo[lane] = b - b_first;
        hw.n[lane] = lane == 0 && rows > kMaxWallRows ? -1 : max(b1 - b, 0);
    }
}

// Slot of particle j, which the halo holds.
__device__ __forceinline__ int slot_of(const Halo &h, int j) {
    int s = h.off[0] + j - h.lo[0];
#pragma unroll
    for (int d = 1; d < kMaxSeg; ++d)
        if (d < h.nseg && j >= h.lo[d]) s = h.off[d] + j - h.lo[d];
    return s;
}
__device__ __forceinline__ int particle_of(const Halo &h, int slot) {
    int j = h.lo[0] + slot - h.off[0];
#pragma unroll
    for (int d = 1; d < kMaxSeg; ++d)
        if (d < h.nseg && slot >= h.off[d]) j = h.lo[d] + slot - h.off[d];
    return j;
}

// Column and row of cell ci, and the candidate range d of a particle there:
// [j0, j1).
__device__ __forceinline__ int2 cell_at(const Inst &I, int ci) {
    const int local = ci - I.base;
    if (!SIMP_IN_RANGE(local, 0, (long long)I.ncx * I.ncy, SITE_CELL)) return make_int2(0, -kMaxSeg);
    const int cy = local / I.ncx;
    return make_int2(local - cy * I.ncx, cy);
}
__device__ __forceinline__ void stencil_range(const Inst &I, const int *cell_start, int2 at, int R, int d, int &j0,
                                              int &j1) {
    const int cy = at.y + d - R;
    j0 = j1 = 0;
    if (cy < 0 || cy >= I.ncy) return;
    const int k = I.base + cy * I.ncx;
    j0 = cell_start[k + max(at.x - R, 0)];
    j1 = cell_start[k + min(at.x + R, I.ncx - 1) + 1];
}

// Starts the copies of record arrays [a0, a1) of the halo and of `rows` rows
// of its lists.  Called by the first warp.
__device__ __forceinline__ void tile_fetch(const Halo &h, const TileMem &m, const void *const (&src)[3], int a0, int a1,
                                           const unsigned short *list, int rows, unsigned long long *bar) {
    const int lane = threadIdx.x & 31, arrays = a1 - a0;
    const unsigned list_bytes = (unsigned)(((rows + 1) & ~1) * kTile * sizeof(unsigned short));
    if (lane == 0) bar_expect(bar, (unsigned)h.off[h.nseg] * 16u * (unsigned)arrays + list_bytes);
    __syncwarp();
    if (lane == 31 && rows > 0) bulk_copy(m.list, list, list_bytes, bar);
    if (lane < h.nseg * arrays) {
        const int d = lane / arrays, a = a0 + lane - d * arrays;
        const int n = h.off[d + 1] - h.off[d];
        if (n > 0)
            bulk_copy(m.rec[a] + (size_t)16 * h.off[d],
                      reinterpret_cast<const unsigned char *>(src[a]) + (size_t)16 * h.lo[d], 16u * (unsigned)n, bar);
    }
}

// Half width of the band around mhsml^2 within which a squared distance needs
// the exact criterion (the fma'd squares are within 2^-50 of the exact ratio).
constexpr double kBand = 0x1p-40;

// The exact reference criterion (nnps.f90:277-281 and the bucket rule).
inline __device__ __noinline__ bool exact_pair(const State &s, const Inst &I, bool rule, int i, int j) {
    const double2 p = s.xy[i], q = s.xy[j];
    double r;
    const double mh = __dmul_rn(__dadd_rn(s.hs[i], s.hs[j]), 0.5);
    if (!pair_test(__dsub_rn(p.x, q.x), __dsub_rn(p.y, q.y), mh, &r)) return false;
    return !rule || bin_rule_ok(make_bin_rule(I.bs, p.x, p.y, I.hmax), q.x, q.y);
}
// The same for two candidates at slots q0 and q1, as classified: bit 0 and bit 1
// set where they are pairs.
inline __device__ __noinline__ int exact_two(const State &s, const Inst &I, bool rule, int i, const Halo &h, int q0, int q1,
                                      int in0, int in1) {
    if (in0) in0 = in0 == 1 && !rule ? 1 : exact_pair(s, I, rule, i, particle_of(h, q0));
    if (in1) in1 = in1 == 1 && !rule ? 1 : exact_pair(s, I, rule, i, particle_of(h, q1));
    return in0 | in1 << 1;
}
// A particle's own value loaded again after a call, so that no register (nor a
// store to local memory) holds it over the call.
__device__ __forceinline__ void reload(double2 &v, const double2 *p) {
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
}
__device__ __forceinline__ void reload(double &v, const double *p) {
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
}
__device__ __forceinline__ bool rule_on(const Inst &I) { return I.hmax >= I.bs * (1.0 - 1e-6); }

// Where a particle without a list finds its candidates: its tile's halo, or for
// a tile without one (h null) global memory, whose arrays then stand in `m`.
struct Around {
    const Halo *h;
    TileMem m;
    __device__ __forceinline__ Around(const Halo &halo, const TileMem &tile, const void *const (&src)[3], const State &s)
        : h(halo.kind == HALO_TILE ? &halo : nullptr), m(tile) {
        if (h) return;
        for (int a = 0; a < 3; ++a) m.rec[a] = (unsigned char *)src[a];
        m.hs = (double *)s.hs;
    }
};

// Pairs of particle i over its cell stencil, in increasing index order: f(q, j),
// q its place in `w`.  The halo covers the stencil it was made with, which holds
// every pair as long as lists built then would.
template <bool UNIFORM, class F>
__device__ __forceinline__ void stencil_pairs(const Around &w, const State &s, const Inst &I, const int *cell_start,
                                              int i, int ci, F &&f) {
    const double2 p = s.xy[i];
    const double hi = s.hs[i];
    const bool rule = rule_on(I);
    const int2 at = cell_at(I, ci);
    const int R = w.h ? w.h->nseg / 2 : stencil_radius(I.hmax, inst_disp(I), inst_grid(I, cell_start), 0.0);
    const double2 *xs = reinterpret_cast<const double2 *>(w.m.rec[0]);
    for (int d = 0; d < 2 * R + 1; ++d) {
        int j0, j1;
        stencil_range(I, cell_start, at, R, d, j0, j1);
        const int shift = w.h && j0 < j1 ? slot_of(*w.h, j0) - j0 : 0;
#pragma unroll 4
        for (int j = j0; j < j1; ++j) {
            const double2 q = xs[j + shift];
            const double dx = p.x - q.x, dy = p.y - q.y, mh = UNIFORM ? hi : 0.5 * (hi + w.m.hs[j + shift]);
            const double d2 = fma(dx, dx, dy * dy);
            if (d2 > mh * mh * (1.0 + kBand) || j == i) continue;
            if (!(d2 < mh * mh * (1.0 - kBand)) || rule)
                if (!exact_pair(s, I, rule, i, j)) continue;
            f(j + shift, j);
        }
    }
}

}  // namespace pass
}  // namespace simp
