// Cell list of the neighbour search (replaces nnps.f90:155-517 bucket_search).
//
// The reference bins particles into square buckets of side 2 * min(hsml)
// serially and scans a half stencil of buckets (nnps.f90:211-412).  Here the
// particles are sorted once into a uniform grid of side cs = (1 + skin) *
// max(hsml) and stay in that order; each pair pass scans the (2R+1)^2 cells
// around a particle, R computed on the device from the exact bounds hmax and
// the maximal displacement since the sort (common.cuh: stencil_radius), so
// the cell list is a superset of every pair at every step without a host
// round trip.  The exact reference criterion (and its bucket rule) is applied
// per candidate in the passes, so the pair set equals the reference's.
//
// Sort: counting sort on cell keys (one radix digit of width log2(ncells)):
// key histogram, exclusive prefix scan, scatter, then a per-cell sort by
// original particle index so the order is deterministic.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "ctx.h"

namespace simp {

namespace {

constexpr int kScanBlock = 256;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanBlock * kScanItems;

// Exclusive scan, phase 1: per-tile sums.
__global__ void scan_tile_sums(const int *__restrict__ in, int n, int *__restrict__ sums) {
    __shared__ int red[kScanBlock / 32];
    const int base = blockIdx.x * kScanTile;
    int s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int i = base + k * kScanBlock + threadIdx.x;
        s += (i < n) ? in[i] : 0;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = (threadIdx.x < kScanBlock / 32) ? red[threadIdx.x] : 0;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) sums[blockIdx.x] = s;
    }
}

// Block-wide exclusive scan of one value per thread; returns the total.
__device__ int block_exclusive_scan(int v, int *smem_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) smem_warp[warp] = incl;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    if (warp == 0) {
        int w = (lane < nw) ? smem_warp[lane] : 0;
        int wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < nw) smem_warp[lane] = wi - w;
        if (lane == 31) smem_warp[32] = wi;
    }
    __syncthreads();
    const int res = smem_warp[warp] + incl - v;
    __syncthreads();
    return res;  // the block total stays in smem_warp[32] until the next call
}

// Phase 2: exclusive scan of the tile sums in one block (sequential chunks).
__global__ void scan_sums(int *sums, int nt) {
    __shared__ int sw[33];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nt; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const int v = (i < nt) ? sums[i] : 0;
        const int ex = block_exclusive_scan(v, sw);
        const int tot = sw[32];
        __syncthreads();
        if (i < nt) sums[i] = ex + carry;
        __syncthreads();
        if (threadIdx.x == 0) carry += tot;
        __syncthreads();
    }
}

// Phase 3: scan within tiles plus tile offset; out has n + 1 entries.
__global__ void scan_tiles(const int *__restrict__ in, int n, const int *__restrict__ sums,
                           int *__restrict__ out) {
    __shared__ int sw[33];
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    int v[kScanItems];
    int loc = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int i = base + k;
        v[k] = (i < n) ? in[i] : 0;
        loc += v[k];
    }
    const int ex = block_exclusive_scan(loc, sw) + sums[blockIdx.x];
    int run = ex;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int i = base + k;
        if (i < n) out[i] = run;
        run += v[k];
    }
}

__global__ void scan_total(const int *__restrict__ in, int n, int *__restrict__ out) {
    out[n] = (n > 0) ? out[n - 1] + in[n - 1] : 0;
}

// Cell key of each particle from its sort position and its instance's grid;
// particles being removed (instance -1) go to the dump key after all cells.
__global__ void k_keys(int n, const double2 *__restrict__ xyr, const int *__restrict__ pinst, const Inst *__restrict__ inst, int dump_key,
                       int *__restrict__ key, int *__restrict__ cnt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int q = pinst[i];
    int k = dump_key;
    if (q >= 0) {
        const Inst &I = inst[q];
        const int cx = clampi((int)floor((xyr[i].x - I.x0) * I.inv_cs), 0, I.ncx - 1);
        const int cy = clampi((int)floor((xyr[i].y - I.y0) * I.inv_cs), 0, I.ncy - 1);
        k = I.base + cy * I.ncx + cx;
    }
    key[i] = k;
    atomicAdd(&cnt[k], 1);
}

// Instances due for a re-sort take their current positions as sort positions and
// the largest coordinate from them (k_reset_inst_disp has set it to 0); a basin
// flagged non-finite keeps its old (finite) ones.  Whole warps.
__global__ void k_refresh_sortpos(int n, const int *__restrict__ pinst, DueMask due, Inst *inst,
                                  const double2 *__restrict__ xy, double2 *__restrict__ xyr) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int q = i < n ? pinst[i] : -1;
    if (q >= 0 && (!((due.w[q >> 6] >> (q & 63)) & 1ull) || inst_dead(inst[q].flags))) q = -1;
    unsigned long long far = 0ull;
    if (q >= 0) {
        const double2 p = xy[i];
        xyr[i] = p;
        far = dbits(fmax(fabs(p.x), fabs(p.y)));
    }
    // one atomic per warp where it holds one basin, and none where the bound is
    // there already
    const int q0 = __reduce_max_sync(0xffffffffu, q);
    if (__all_sync(0xffffffffu, q == q0 || q < 0)) {
        const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(far >> 32));
        const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(far >> 32) == hi ? (unsigned)far : 0u);
        far = (unsigned long long)hi << 32 | lo;
        q = (threadIdx.x & 31) == 0 ? q0 : -1;
    }
    if (q >= 0 && *(volatile unsigned long long *)&inst[q].xabs_bits < far) atomicMax(&inst[q].xabs_bits, far);
}

__global__ void k_reset_inst_disp(Inst *inst, int ninst, DueMask due) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= ninst) return;
    if (!((due.w[q >> 6] >> (q & 63)) & 1ull)) return;
    inst[q].disp = 0.0;
    inst[q].list_ok = 0;   // (its particles take new places)
    inst[q].spares = 0;
    if (!inst_dead(inst[q].flags)) inst[q].xabs_bits = 0ull;
}

__global__ void k_scatter(int n, const int *__restrict__ key, const int *__restrict__ start,
                          int *__restrict__ cnt, int *__restrict__ perm) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int k = key[i];
    const int slot = atomicSub(&cnt[k], 1) - 1;
    const int pos = start[k] + slot;
    if (!SIMP_IN_RANGE(pos, 0, n, SITE_SORT)) return;
    perm[pos] = i;
}

// Sort each cell's entries by original particle index (insertion sort; a
// cell holds a few tens of particles).
__global__ void k_cell_sort(int ncells, const int *__restrict__ start, int *__restrict__ perm,
                            const int *__restrict__ id) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    const int a = start[c], b = start[c + 1];
    for (int k = a + 1; k < b; ++k) {
        const int v = perm[k];
        const int kv = id[v];
        int j = k - 1;
        while (j >= a && id[perm[j]] > kv) { perm[j + 1] = perm[j]; --j; }
        perm[j + 1] = v;
    }
}

constexpr int kPairs = 3, kFields = 7;   // (the last two fields only with Benz's kept drhodt and the kept kernel_zero)
struct Gather {
    const double2 *psrc[kPairs];
    double2 *pdst[kPairs];
    const double *src[kFields];
    double *dst[kFields];
};

__device__ __forceinline__ bool is_due(const DueMask &m, int q) {
    return q >= 0 && ((m.w[q >> 6] >> (q & 63)) & 1ull);
}

// Positions of the new order whose particle may differ from the old one:
// every position from `from` on (an admission appends a basin there; a
// removal shifts the basins after it down), and those of the due basins
// (each basin keeps its range of positions; the others keep their order).
__device__ __forceinline__ bool moves(int from, const DueMask &due, const int *pinst, int k) {
    return k >= from || is_due(due, pinst[k]);
}

// New order into scratch.
__global__ void k_gather(int kept, int from, DueMask due, const int *__restrict__ perm, Gather gd,
                         const int *__restrict__ key, int *__restrict__ cell_out, const int *__restrict__ id_in,
                         int *__restrict__ id_out, const int *__restrict__ pinst_in, int *__restrict__ pinst_out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= kept || !moves(from, due, pinst_in, k)) return;
    const int o = perm[k];
#pragma unroll
    for (int a = 0; a < kPairs; ++a) gd.pdst[a][k] = gd.psrc[a][o];
#pragma unroll
    for (int a = 0; a < kFields; ++a)
        if (gd.src[a]) gd.dst[a][k] = gd.src[a][o];
    cell_out[k] = key[o];
    id_out[k] = id_in[o];
    pinst_out[k] = pinst_in[o];
}

// Scratch back into the state arrays (pointers stay fixed so the captured
// step graph remains valid), with the FP32 copies of the moved particles.
__global__ void k_put_back(int kept, int from, DueMask due, Gather gd, State s, const int *__restrict__ id_new,
                           int *__restrict__ id, const int *__restrict__ pinst_new, int *__restrict__ pinst) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= kept || !moves(from, due, pinst, k)) return;
#pragma unroll
    for (int a = 0; a < kPairs; ++a) const_cast<double2 *>(gd.psrc[a])[k] = gd.pdst[a][k];
#pragma unroll
    for (int a = 0; a < kFields; ++a)
        if (gd.src[a]) const_cast<double *>(gd.src[a])[k] = gd.dst[a][k];
    id[k] = id_new[k];
    pinst[k] = pinst_new[k];
    refresh_views(s, k);
}

inline int nblk(long long n, int b) { return (int)((n + b - 1) / b); }

}  // namespace

size_t scan_tmp_bytes(int n) {
    const int nt = (n + kScanTile - 1) / kScanTile;
    return (size_t)(nt + 1) * sizeof(int);
}

// Exclusive scan of n ints into out[0..n] (out[n] = total).
void launch_scan_i32(const int *in, int *out, int n, void *tmp, cudaStream_t s) {
    const int nt = std::max(1, (n + kScanTile - 1) / kScanTile);
    int *sums = (int *)tmp;
    scan_tile_sums<<<nt, kScanBlock, 0, s>>>(in, n, sums);
    scan_sums<<<1, 1024, 0, s>>>(sums, nt);
    scan_tiles<<<nt, kScanBlock, 0, s>>>(in, n, sums, out);
    scan_total<<<1, 1, 0, s>>>(in, n, out);
}

// Sorts the particles into cell order (instance-major keys, within a cell by
// global id).  Instances in `due` re-bin at their current positions; the
// others keep their sort positions, so their order does not change.
// Positions from `from` on are rewritten (after an admission or a removal:
// the first position whose basin changed), before it only the due
// instances' ranges move.  Particles of removed instances (instance -1) end
// up after all others and are dropped: c->n shrinks to the kept count.
int rebuild(simp_ctx *c, const DueMask &due, int from) {
    SIMP_RANGE("re-sort");
    const int n = c->n;
    cudaStream_t s = c->stream;
    const int B = 256;
    const int nkeys = c->total_cells + 1;   // + the dump key
    const size_t MX = (size_t)std::max(c->maxn, c->maxnb);
    int *key = c->itmp;
    int *id_new = c->itmp + MX;
    int *pinst_new = c->itmp + 2 * MX;
    int kept = 0;
    for (const InstHost &h : c->insts)
        if (h.active) kept += h.n;
    if (n > 0) {
        k_reset_inst_disp<<<nblk(c->ninst, 128), 128, 0, s>>>(c->inst_dev, c->ninst, due);
        k_refresh_sortpos<<<nblk(n, B), B, 0, s>>>(n, c->pinst, due, c->inst_dev, c->s0.xy, c->xyr);
        SIMP_CUDA(c, cudaMemsetAsync(c->cnt, 0, sizeof(int) * (size_t)nkeys, s));
        k_keys<<<nblk(n, B), B, 0, s>>>(n, c->xyr, c->pinst, c->inst_dev, c->total_cells, key, c->cnt);
        launch_scan_i32(c->cnt, c->cell_start, nkeys, c->scan_tmp, s);
        k_scatter<<<nblk(n, B), B, 0, s>>>(n, key, c->cell_start, c->cnt, c->perm);
        // (the dump key is not ordered: its particles are dropped)
        if (c->total_cells > 0)
            k_cell_sort<<<nblk(c->total_cells, 128), 128, 0, s>>>(c->total_cells, c->cell_start, c->perm, c->id);
        double2 *pairs[kPairs] = {c->s0.xy, c->s0.vxy, c->xyr};
        double *fields[kFields] = {c->s0.m, c->s0.rho, c->s0.h, c->s0.A, c->s0.hs, c->drhodt, c->k0};
        Gather gd;
        for (int a = 0; a < kPairs; ++a) {
            gd.psrc[a] = pairs[a];
            gd.pdst[a] = reinterpret_cast<double2 *>(c->tmp) + (size_t)a * MX;
        }
        for (int a = 0; a < kFields; ++a) {
            gd.src[a] = fields[a];
            gd.dst[a] = c->tmp + (size_t)(2 * kPairs + a) * MX;
        }
        c->launches += 7 + kScanKernels;
        if (kept > 0) {
            k_gather<<<nblk(kept, B), B, 0, s>>>(kept, from, due, c->perm, gd, key, c->cell, c->id, id_new,
                                                 c->pinst, pinst_new);
            c->launches += 1;
            k_put_back<<<nblk(kept, B), B, 0, s>>>(kept, from, due, gd, c->s0, id_new, c->id, pinst_new, c->pinst);
            c->launches += 1;
        }
    } else {
        SIMP_CUDA(c, cudaMemsetAsync(c->cell_start, 0, sizeof(int) * (size_t)(nkeys + 1), s));
    }
    c->n = kept;
    DueMask cut = due;
    if (c->chunks_new) std::memset(&cut, 0xff, sizeof(cut));   // (the tiles of every basin)
    launch_split(c, cut);
    c->chunks_new = false;
    SIMP_CUDA(c, cudaGetLastError());
    c->rebuilds += 1;
    return SIMP_OK;
}

}  // namespace simp
