// Wall pairs of a tile's particles.
//
// Few tiles of a large basin have any, but those hold the pass up: one thread
// per particle left a wall's particles with up to seven pairs each, a square
// root and a division per pair in a chain, while the other threads waited.  So
// the block lists the walls near the tile, marks each particle's pairs
// (comparisons only), takes the pairs one per thread whichever particle they
// belong to, and each particle sums its own in the walls' order.  Bound by the
// latency of five such phases.  Per step with walls on four sides, against one
// thread per particle: FP64 2,500 particles 59 -> 46 us, 65,536 82 -> 65,
// 262,144 188 -> 161, 600,011 372 -> 347; mixed 24,649 67 -> 54, 262,144
// 189 -> 169, 1,048,576 569 -> 554.
#pragma once

#include "tile.cuh"

namespace simp {
namespace pass {

constexpr int kWallCap = 128;
constexpr int kWallPairs = 1024;
struct WallTile {
    int n;                             // walls, -1: too many
    int pairs;                         // pairs with them, -1: too many
    int part[kTile / 32];              // (of the scan)
    unsigned short first[kTile + 1];   // each particle's first pair, and the total
    unsigned short pair[kWallPairs];   // particle | wall << 7
    int id[kWallCap];
    double x[kWallCap], y[kWallCap], m[kWallCap];
    double2 own[kTile];                // the particles' positions, then (mixed form) their sums fx, fy
    double own_m[kTile], own_h[kTile]; // mass and hsml, then the sums gx, gy
    int cnt[kTile];
};
static_assert(kTile <= 128 && kWallCap <= 128, "WallTile::pair");
// Shared memory of the stress pass: its tile's, and at least what the wall sums
// put in its place (the pair sums behind them).
__host__ __device__ constexpr size_t stress_smem_bytes(int cap, int arrays, bool uniform) {
    const size_t tile = tile_smem_bytes(cap, arrays, uniform), walls = sizeof(WallTile) + 4 * kTile * sizeof(double);
    return tile > walls ? tile : walls;
}

__device__ __forceinline__ int warp_scan(int v, int lane) {   // inclusive
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

// Wall k of the part's, in their order, or -1 behind the last (HaloWalls).
__device__ __forceinline__ int wall_at(const HaloWalls &h, int b_first, int k) {
    int b = -1;
#pragma unroll
    for (int d = 0; d < kMaxWallRows; ++d) {
        const int n = h.n[d];
        if (k >= 0 && k < n) b = b_first + h.lo[d] + k;
        k -= n;
    }
    return b;
}
// Brings what wall_sums reads first to the L1 cache, while the pairs are summed.
__device__ __forceinline__ void wall_prefetch(const StressArgs &a, const HaloWalls &h, int b_first, int i) {
    const int b = wall_at(h, b_first, threadIdx.x);
    if (b >= 0) {
        prefetch_l1(&a.bx[b]);
        prefetch_l1(&a.by[b]);
        prefetch_l1(&a.bm[b]);
    }
    prefetch_l1(&a.rhs.m[i]);
}
// The part's walls.  Called by the whole block, which synchronises before they
// are read.
__device__ __forceinline__ void wall_list(const StressArgs &a, const HaloWalls &h, int b_first, WallTile &w) {
    static_assert(kWallCap <= kTile, "one wall per thread");
    const int t = threadIdx.x, b = t < kWallCap ? wall_at(h, b_first, t) : -1;
    if (b >= 0) {
        w.id[t] = b;
        w.x[t] = a.bx[b];
        w.y[t] = a.by[b];
        w.m[t] = a.bm[b];
    }
    if (t == 0) {
        int n = 0;
        for (int d = 0; d < kMaxWallRows; ++d) n += h.n[d];
        w.n = h.n[0] >= 0 && n <= kWallCap ? n : -1;
    }
}

// The same from the cell lists, for a part with cells ka .. kb whose walls lie
// within Rb cells (Halo.walls).  Called by the whole block, which synchronises
// before they are read.
__device__ __forceinline__ void wall_find(const StressArgs &a, const Inst &I, int Rb, int ka, int kb, WallTile &w) {
    const int end = I.base + I.ncx * I.ncy, rows = 2 * Rb + 1, lane = threadIdx.x & 31;
    // one lane per cell row: its walls, from where the rows before it end
    int b0 = 0, b1 = 0;
    if (lane < rows) {
        const int sh = (lane - Rb) * I.ncx;
        b0 = a.bstart[clampi(ka + sh - Rb, I.base, end)];
        b1 = a.bstart[clampi(kb + sh + Rb + 1, I.base, end)];
    }
    int past = b1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, past, o);
        if (lane >= o) past = max(past, u);
    }
    const int before = __shfl_up_sync(0xffffffffu, past, 1);
    if (lane > 0) b0 = max(b0, before);
    const int c = max(b1 - b0, 0), upto = warp_scan(c, lane);
    const int n = rows <= 32 ? __shfl_sync(0xffffffffu, upto, 31) : kWallCap + 1;
    for (int d = 0; d < rows && n <= kWallCap; ++d) {
        const int from = __shfl_sync(0xffffffffu, b0, d), m = __shfl_sync(0xffffffffu, c, d);
        const int at = __shfl_sync(0xffffffffu, upto, d) - m;
        for (int k = threadIdx.x; k < m; k += kTile) {
            w.id[at + k] = from + k;
            w.x[at + k] = a.bx[from + k];
            w.y[at + k] = a.by[from + k];
            w.m[at + k] = a.bm[from + k];
        }
    }
    if (threadIdx.x == 0) w.n = n <= kWallCap ? n : -1;
}

// Marks the pairs of a part's particles with the listed walls.  `room`: pairs
// there is room for.  Called by the whole block, which synchronises before the
// pairs are read.
__device__ __forceinline__ void wall_pairs(const StressArgs &a, const Inst &I, bool live, int i, double2 p, double hi,
                                           int room, WallTile &w) {
    const int t = threadIdx.x, lane = t & 31;
    const double bl = I.b_length, near = bl * bl * (1.0 - kBand), far = bl * bl * (1.0 + kBand);
    w.own[t] = p;
    w.own_m[t] = a.rhs.m[i];
    w.own_h[t] = hi;
    // without branches, so that the walls' comparisons overlap
    constexpr int words = kWallCap / 32;
    unsigned hit[words] = {}, edge = 0u;
#pragma unroll
    for (int g = 0; g < words; ++g) {
        const int n = min(w.n - 32 * g, 32);
        unsigned bits = 0u;
#pragma unroll 8
        for (int k = 0; k < n; ++k) {
            const double dx = __dsub_rn(w.x[32 * g + k], p.x), dy = __dsub_rn(w.y[32 * g + k], p.y);
            const double s = fma(dx, dx, dy * dy);
            bits |= (s <= far ? 1u : 0u) << k;
            edge |= (s <= far && !(s < near)) ? 1u : 0u;
        }
        hit[g] = live ? bits : 0u;
    }
    const BinRule bb = make_bin_rule(I.bs, p.x, p.y, bl);
    if (edge || bb.on) {   // the exact criterion, for all of the particle's
#pragma unroll
        for (int g = 0; g < words; ++g)
            for (unsigned b = hit[g]; b; b &= b - 1) {
                const int k = 32 * g + __ffs(b) - 1;
                double d;
                if (!pair_test(__dsub_rn(w.x[k], p.x), __dsub_rn(w.y[k], p.y), bl, &d) ||
                    !bin_rule_ok(bb, w.x[k], w.y[k]))
                    hit[g] &= ~(b & (0u - b));
            }
    }
    int c = 0;
#pragma unroll
    for (int g = 0; g < words; ++g) c += __popc(hit[g]);
    const int upto = warp_scan(c, lane);
    if (lane == 31) w.part[t / 32] = upto;
    __syncthreads();
    int at = upto - c, total = 0;
#pragma unroll
    for (int q = 0; q < kTile / 32; ++q) {
        const int p = w.part[q];
        if (q < t / 32) at += p;
        total += p;
    }
    w.first[t] = (unsigned short)at;
    const bool fits = w.n >= 0 && total <= room;
    if (t == 0) {
        w.first[kTile] = (unsigned short)total;
        w.pairs = fits ? total : -1;
    }
    if (!fits) return;
#pragma unroll
    for (int g = 0; g < words; ++g)
        for (unsigned b = hit[g]; b; b &= b - 1) w.pair[at++] = (unsigned short)(t | (32 * g + __ffs(b) - 1) << 7);
}

// One wall pair (boundary_force.f90: bfa 1 bf_Monaghan :38-102, 2 bf_Wang
// :109-176, 3 bf_Marquis :183-225).
template <int SKF>
__device__ __noinline__ WallSums wall_pair(const StressArgs &a, double bl, int i, double mi, double hi, int b,
                                           double mb, double bdx, double bdy) {
    const Phys &P = a.P;
    WallSums w;
    double d = 0.0;
    pair_test(bdx, bdy, bl, &d);
    if (P.bfa == 1) {
        if (P.boundary_pressure) {
            const double bw = boundary_w<SKF>(P, d, hi);
            const double coef = P.kappa_n * bw * 2.0 * mb / ((mi + mb) * (d * d));
            w.fx = coef * bdx;
            w.fy = coef * bdy;
        }
        if (P.boundary_friction) {   // :85-100
            const double rho = a.rhs.rho[i];
            const double2 v = a.rhs.vxy[i];
            const double sh = (double)P.scale_h;
            const double t = boundary_fdwdq<SKF>(P, d, hi) / bl;
            const double bwx = -(t * (bdx / d) * sh), bwy = -(t * (bdy / d) * sh);
            const double v_r = v.x * bdx + v.y * bdy;
            const double pi_aj = P.kappa_t * sound_speed(P, rho) * v_r / d / rho;
            w.gx = (-1.0 * mb * pi_aj * bwx) / rho;
            w.gy = (-1.0 * mb * pi_aj * bwy) / rho;
        }
    } else if (P.bfa == 2) {
        if (P.boundary_pressure) {   // :146-172
            const double2 v = a.rhs.vxy[i];
            const double dt = a.sc->dt;
            const double nx = a.bnx[b], ny = a.bny[b];
            const double v1 = nx * v.x + ny * v.y;
            double v2 = sqrt(v.x * v.x + v.y * v.y) - v1;
            const double F1 = mi * v1 / dt;
            double F2 = mi * v2 / dt;
            if (P.boundary_friction && fabs(v2) > fabs(P.xi * v1)) {
                v2 = v2 * P.xi * fabs(F1 / F2);
                F2 = mi * v2 / dt;
            }
            w.gx = F1 * nx + F2 * ny;
            w.gy = F1 * ny - F2 * nx;
        }
    } else if (!P.boundary_pressure && P.boundary_friction) {   // :212-222
        const double2 v = a.rhs.vxy[i];
        w.gx = -(v.x * (1.0 - d / bl));
        w.gy = -(v.y * (1.0 - d / bl));
    }
    return w;
}

// A particle's wall pairs one after another, where a tile has too many.  The
// same terms in the same order.
template <int SKF>
__device__ __noinline__ WallSums wall_serial(const StressArgs &a, const Inst &I, int i) {
    const double2 p = a.rhs.xy[i];
    const Grid g = inst_grid(I, a.cell_start);
    WallSums w;
    w.cnt = for_each_wall(a.bx, a.by, a.bstart, g, a.cell[i], wall_radius(inst_disp(I), g, I.b_length),
                          make_bin_rule(I.bs, p.x, p.y, I.b_length), p.x, p.y, I.b_length,
                          [&](int b, double bdx, double bdy, double) {
                              const WallSums c = wall_pair<SKF>(a, I.b_length, i, a.rhs.m[i], a.rhs.hs[i], b, a.bm[b],
                                                                bdx, bdy);
                              w.fx += c.fx;
                              w.fy += c.fy;
                              w.gx += c.gx;
                              w.gy += c.gy;
                          });
    return w;
}

// Whether the walls come with the halo or from the cell lists: in the mixed form
// of five blocks per SM those hide the cell lists' two more loads in a row, and
// the halo's cost registers it does not have (1,048,576 particles: 552 us per
// step from the cell lists, 562 with the halo); everywhere else they come with
// the halo (FP64 at 262,144: 157 -> 153, at 2,500: 43 -> 40).
//
// The wall sums of a part's particles, thread t's particle p0 + t.  Works in
// `bytes` of shared memory that the block no longer needs.  Called by the whole
// block.
template <int SKF, bool LISTED>
__device__ __forceinline__ WallSums wall_sums(const StressArgs &a, const Inst &I, int Rb, const HaloWalls &h, int p0,
                                              int size, int i, double2 p,
                                              double hi, unsigned char *smem, int bytes) {
    WallTile &w = *reinterpret_cast<WallTile *>(smem);
    double *res = reinterpret_cast<double *>(smem + sizeof(WallTile));
    const int t = threadIdx.x;
    const bool live = t < size;
    // which sums the parameters give terms to
    const bool f = a.P.bfa == 1 && a.P.boundary_pressure, g = a.P.bfa != 1 || a.P.boundary_friction;
    const int room = (bytes - (int)sizeof(WallTile)) / (16 * max(1, (int)f + (int)g));
    if (LISTED) wall_list(a, h, a.bstart[I.base], w);
    else wall_find(a, I, Rb, a.cell[p0], a.cell[p0 + size - 1], w);
    __syncthreads();
    wall_pairs(a, I, live, i, p, hi, min(kWallPairs, room), w);
    __syncthreads();
    WallSums s;
    const int n = w.pairs;
    if (n < 0) {
        if (live) s = wall_serial<SKF>(a, I, p0 + t);
        return s;
    }
    double *rg = res + (f ? 2 * n : 0);
    for (int k = t; k < n; k += kTile) {
        const int e = w.pair[k], q = e & 127, b = e >> 7;
        const double2 p = w.own[q];
        const WallSums c = wall_pair<SKF>(a, I.b_length, p0 + q, w.own_m[q], w.own_h[q], w.id[b], w.m[b],
                                          __dsub_rn(w.x[b], p.x), __dsub_rn(w.y[b], p.y));
        if (f) {
            res[k] = c.fx;
            res[n + k] = c.fy;
        }
        if (g) {
            rg[k] = c.gx;
            rg[n + k] = c.gy;
        }
    }
    __syncthreads();
    const int k1 = w.first[t + 1];
    for (int k = w.first[t]; k < k1; ++k) {
        ++s.cnt;
        if (f) {
            s.fx += res[k];
            s.fy += res[n + k];
        }
        if (g) {
            s.gx += rg[k];
            s.gy += rg[n + k];
        }
    }
    return s;
}
// Where the epilogue finds them, so that the registers they take cost tiles
// without walls little: in FP64 in registers, while the pair sums wait in
// shared memory (kKeep); in the mixed form, with fewer registers, in shared
// memory themselves.  Per step FP64 at 600,011: 353 us against 362 with the
// other way and 358 with neither; mixed at 1,048,576: 555 against 557 and 560.
struct WallRegs {
    static constexpr bool kKeep = true;
    WallSums s;
    __device__ __forceinline__ void set(WallTile *, const WallSums &v) { s = v; }
    __device__ __forceinline__ void add(double irho, double &ax, double &ay, int &cnt) const {
        ax = ax - s.fx * irho + s.gx;
        ay = ay - s.fy * irho + s.gy;
        cnt += s.cnt;
    }
};
struct WallShared {
    static constexpr bool kKeep = false;
    const WallTile *w = nullptr;
    __device__ __forceinline__ void set(WallTile *t, const WallSums &v) {   // (others have read `own`)
        t->own[threadIdx.x] = make_double2(v.fx, v.fy);
        t->own_m[threadIdx.x] = v.gx;
        t->own_h[threadIdx.x] = v.gy;
        t->cnt[threadIdx.x] = v.cnt;
        w = t;
    }
    __device__ __forceinline__ void add(double irho, double &ax, double &ay, int &cnt) const {
        if (!w) return;
        const double2 f = w->own[threadIdx.x];
        ax = ax - f.x * irho + w->own_m[threadIdx.x];
        ay = ay - f.y * irho + w->own_h[threadIdx.x];
        cnt += w->cnt[threadIdx.x];
    }
};

}  // namespace pass
}  // namespace simp
