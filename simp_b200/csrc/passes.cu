// The passes that go over tiles (tile.cuh) besides the two of every right-hand
// side (pass_kernels.cuh), the end of a step, the tiles' table, and all launches.
#include <cmath>

#include "pass_kernels.cuh"

namespace simp {

namespace {

using namespace pass;

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

// The passes' form of a context's current layout.
PassForm form_of(const simp_ctx *c) {
    const bool mixed = c->prm.precision == SIMP_PREC_MIXED;
    const int hs = c->uniform ? HSML_ONE : c->max_inst == 1 ? HSML_VARIED : HSML_EITHER;
    const int blocks = mixed && c->nchunks > kSmallTiles ? 5 : 4;
    switch (skf_compiled(c->prm.skf)) {
        case SIMP_SKF_CUBIC: return mixed ? passes_cubic_mixed(hs, blocks) : passes_cubic_fp64(hs, blocks);
        case SIMP_SKF_WENDLAND_C6: return mixed ? passes_wendland_mixed(hs, blocks) : passes_wendland_fp64(hs, blocks);
        default: return mixed ? passes_generic_mixed(hs, blocks) : passes_generic_fp64(hs, blocks);
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
    const PassForm f = form_of(c);
    allow(f.kin);
    allow(f.stress);
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
    launch_pass(c, form_of(c).kin, c->nchunks, kTile, tile_smem_bytes(a.cap, 3, c->uniform), a);
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
    const int arrays = c->prm.precision == SIMP_PREC_MIXED ? Rec<float>::stress_arrays : Rec<double>::stress_arrays;
    launch_pass(c, form_of(c).stress, c->nchunks, kTile, stress_smem_bytes(a.cap, arrays, c->uniform), a);
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
