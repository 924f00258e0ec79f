// mps_neighbors.cu -- hash, sort, reorder and neighbour lists (NEIGHBOR,
// functions.cu:2788-2929; the reference GPU path's calcHash / sort_by_key /
// findCellStart / createNeighbourArrays, neighbour_parallel.cu:37-199).
//
// Per step:
//   1. k_hash      exact FP64 cell number of every particle on both grids
//                  (Laplacian grid = primary order, PND grid = index only),
//                  bucket counts by atomics;
//   2. scan        exclusive prefix sums of the counts (cell starts);
//   3. k_scatter   particles into their cell bucket (arbitrary order);
//   4. k_rank      order inside a bucket by (x, original id) on both grids,
//                  so that every x-triple of cells is sorted by x; NEIGHBOR's
//                  own order, (cell, id) -- the stable counting sort of the
//                  reference's insertion loop (functions.cu:2820) -- is
//                  formed when a permutation is downloaded;
//   5. k_gather    reorder the persistent particle state into cell order;
//   6. k_lists     both lists, membership decided with the reference's exact
//                  FP64 arithmetic over x-windowed runs of cells: a group of
//                  lanes per particle, or in larger 3D scenes a particle per
//                  lane (k_lists_lane).  Exported rows are put back in the
//                  reference's scan order (x offset outermost, then y, z;
//                  ascending id inside a cell).
#include <cmath>
#include <cstdio>
#include <type_traits>

#include "mps_internal.cuh"

using namespace vmps;

namespace {

template <int DIM>
__global__ void k_hash(int n, Grid gl, Grid gs, const double* __restrict__ x,
                       const double* __restrict__ y, const double* __restrict__ z,
                       int* __restrict__ cell_l, int* __restrict__ cell_s,
                       int* __restrict__ cnt_l, int* __restrict__ cnt_s,
                       int* __restrict__ bpos_l, int* __restrict__ bpos_s, unsigned int* err)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double xi = x[i], yi = y[i], zi = DIM == 3 ? z[i] : 0.0;
    int a, b, c;
    bool ok = cell_coords<DIM>(gl, xi, yi, zi, a, b, c);
    int Cl = a + (b - 1) * gl.ncx + (c - 1) * gl.ncx * gl.ncy;
    ok = cell_coords<DIM>(gs, xi, yi, zi, a, b, c) && ok;
    int Cs = a + (b - 1) * gs.ncx + (c - 1) * gs.ncx * gs.ncy;
    if (!ok) set_error(err, MPS_ERR_CELL);
    cell_l[i] = Cl;
    cell_s[i] = Cs;
    bpos_l[i] = atomicAdd(&cnt_l[Cl], 1);
    bpos_s[i] = atomicAdd(&cnt_s[Cs], 1);
}

// three-phase exclusive scan (tile sums, scan of tile sums, tile rescans)
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ int block_exclusive_scan(int v, int* sh, int* total)
{
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) sh[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int s = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : 0;
        int si = s;
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, si, o);
            if (lane >= o) si += t;
        }
        sh[lane] = si - s;
        if (lane == 31) sh[32] = si;
    }
    __syncthreads();
    int r = inc - v + sh[wid];
    if (total) *total = sh[32];
    __syncthreads();
    return r;
}

// up to two scans per launch, one per blockIdx.y
struct Scans {
    int m[2];
    const int* in[2];
    int* out[2];
    int* tile_sum[2];
};

__global__ void k_scan_tiles(Scans a)
{
    __shared__ int sh[33];
    const int m = a.m[blockIdx.y];
    const int* __restrict__ in = a.in[blockIdx.y];
    int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    if ((int)blockIdx.x * kScanTile >= m) return;
    int s = 0;
    for (int k = 0; k < kScanItems; k++)
        if (base + k < m) s += in[base + k];
    int tot;
    block_exclusive_scan(s, sh, &tot);
    if (threadIdx.x == 0) a.tile_sum[blockIdx.y][blockIdx.x] = tot;
}

__global__ void k_scan_sums(Scans a)
{
    __shared__ int sh[33];
    int* tile_sum = a.tile_sum[blockIdx.y];
    const int tiles = (a.m[blockIdx.y] + kScanTile - 1) / kScanTile;
    int carry = 0;
    for (int base = 0; base < tiles; base += kScanThreads) {
        int i = base + threadIdx.x;
        int v = i < tiles ? tile_sum[i] : 0;
        int tot;
        int e = block_exclusive_scan(v, sh, &tot);
        if (i < tiles) tile_sum[i] = e + carry;
        carry += tot;
        __syncthreads();
    }
}

__global__ void k_scan_apply(Scans a)
{
    __shared__ int sh[33];
    const int m = a.m[blockIdx.y];
    const int* __restrict__ in = a.in[blockIdx.y];
    int* __restrict__ out = a.out[blockIdx.y];
    int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    if ((int)blockIdx.x * kScanTile >= m) return;
    int vals[kScanItems];
    int s = 0;
    for (int k = 0; k < kScanItems; k++) {
        vals[k] = (base + k < m) ? in[base + k] : 0;
        s += vals[k];
    }
    int e = block_exclusive_scan(s, sh, nullptr) + a.tile_sum[blockIdx.y][blockIdx.x];
    for (int k = 0; k < kScanItems; k++) {
        if (base + k < m) out[base + k] = e;
        e += vals[k];
    }
}

// short arrays: one block per scan, tile after tile, in one launch
constexpr int kScanSmall = 4 * kScanTile;
__global__ void __launch_bounds__(kScanThreads) k_scan_small(Scans a)
{
    __shared__ int sh[33];
    const int m = a.m[blockIdx.y];
    const int* __restrict__ in = a.in[blockIdx.y];
    int* __restrict__ out = a.out[blockIdx.y];
    int carry = 0;
    for (int tile = 0; tile < m; tile += kScanTile) {
        const int base = tile + threadIdx.x * kScanItems;
        int vals[kScanItems], s = 0, tot;
        for (int k = 0; k < kScanItems; k++) {
            vals[k] = (base + k < m) ? in[base + k] : 0;
            s += vals[k];
        }
        int e = block_exclusive_scan(s, sh, &tot) + carry;
        for (int k = 0; k < kScanItems; k++) {
            if (base + k < m) out[base + k] = e;
            e += vals[k];
        }
        carry += tot;
    }
}

// Unsigned key whose integer order is the order of the doubles (-0 just
// below +0, NaNs at the ends), so that (key, id) is a strict total order
// even on a state that has gone non-finite: every bucket position is taken
// exactly once.
__device__ __forceinline__ unsigned long long order_key(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

__global__ void k_scatter(int n, const int* __restrict__ cell_l, const int* __restrict__ cell_s,
                          const int* __restrict__ bpos_l, const int* __restrict__ bpos_s,
                          const int* __restrict__ cst_l, const int* __restrict__ cst_s,
                          const int* __restrict__ oid, const double* __restrict__ x,
                          int* __restrict__ bslot_l, int* __restrict__ boid_l,
                          unsigned long long* __restrict__ bx_l, int* __restrict__ bslot_s,
                          int* __restrict__ boid_s, unsigned long long* __restrict__ bx_s)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int o = oid[i];
    int q = cst_l[cell_l[i]] + bpos_l[i];
    bslot_l[q] = i;
    boid_l[q] = o;
    const unsigned long long key = order_key(x[i]);
    bx_l[q] = key;
    int qs = cst_s[cell_s[i]] + bpos_s[i];
    bslot_s[qs] = i;
    boid_s[qs] = o;
    bx_s[qs] = key;
}

// Rank inside the bucket by (x, original id) on both grids, so that every
// cell's particles lie in ascending x and each x-triple of cells is sorted
// by x (the list passes window their candidate runs on x).  Laplacian grid
// (the memory order): src[new] = old slot and inv[old] = new.  PND grid:
// perm_tmp[position] = old slot and key_s[position] = x's order key.
// NEIGHBOR's own orders, (cell, id) on each grid (the stable counting sort
// of the reference's insertion loop, functions.cu:2820), are formed when
// the permutations are downloaded.
__global__ void k_rank(int n, const int* __restrict__ cell_l, const int* __restrict__ cell_s,
                       const int* __restrict__ cst_l, const int* __restrict__ cnt_l,
                       const int* __restrict__ cst_s, const int* __restrict__ cnt_s,
                       const int* __restrict__ bslot_l, const int* __restrict__ boid_l,
                       const unsigned long long* __restrict__ bx_l,
                       const int* __restrict__ bslot_s, const int* __restrict__ boid_s,
                       const unsigned long long* __restrict__ bx_s,
                       int* __restrict__ src, int* __restrict__ inv, int* __restrict__ perm_tmp,
                       unsigned long long* __restrict__ key_s)
{
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    // one grid per blockIdx.y: the two walks side by side, not one after the other
    if (blockIdx.y == 0) {
        int s = bslot_l[q], me = boid_l[q];
        const unsigned long long xm = bx_l[q];
        int c = cell_l[s];
        int b = cst_l[c], e = b + cnt_l[c], r = 0;
        for (int t = b; t < e; t++) {
            const unsigned long long xt = bx_l[t];
            r += (xt < xm || (xt == xm && boid_l[t] < me));
        }
        src[b + r] = s;
        inv[s] = b + r;
    } else {
        int s = bslot_s[q], me = boid_s[q];
        const unsigned long long xm = bx_s[q];
        int c = cell_s[s];
        int b = cst_s[c], e = b + cnt_s[c], r = 0;
        for (int t = b; t < e; t++) {
            const unsigned long long xt = bx_s[t];
            r += (xt < xm || (xt == xm && boid_s[t] < me));
        }
        perm_tmp[b + r] = s;
        key_s[b + r] = xm;
    }
}

// The persistent fields, old and new order: 15 doubles (x y z u v w p pnew phat
// un vn wn rho n pold) and 6 ints (ptype, id, cell numbers, scene, owned)
constexpr int kGatherD = 15, kGatherI = 6;
struct GatherSet {
    const double* from_d[kGatherD];
    double* to_d[kGatherD];
    const int* from_i[kGatherI];
    int* to_i[kGatherI];
};
// what else follows from the new order: the packed copies that the neighbour
// sums gather from, and the PND grid's order in new slots
struct GatherPack {
    double4 *P4, *U4;
    float4 *P4f, *U4f;  // U4f: mixed precision only
    double x0, y0, z0;
    const int *inv, *perm_old;
    int* perm;
};

// One pass for the reorder, the packed copies and the translated PND order (five
// launches and a second reading of the positions and velocities before; all loads
// of a particle are issued before its first store, 2D dam of 1.9 k particles 13 ->
// 5 us)
__global__ void k_gather(int n, const int* __restrict__ src, GatherSet g, GatherPack q)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int s = src[k];
    const int old = q.perm_old[k];
    double d[kGatherD];
    int v[kGatherI];
#pragma unroll
    for (int a = 0; a < kGatherD; a++) d[a] = __ldg(g.from_d[a] + s);
#pragma unroll
    for (int a = 0; a < kGatherI; a++) v[a] = __ldg(g.from_i[a] + s);
    const int slot = q.inv[old];
#pragma unroll
    for (int a = 0; a < kGatherD; a++) g.to_d[a][k] = d[a];
#pragma unroll
    for (int a = 0; a < kGatherI; a++) g.to_i[a][k] = v[a];
    q.P4[k] = make_double4(d[0], d[1], d[2], (double)v[0]);
    q.U4[k] = make_double4(d[3], d[4], d[5], 0.0);
    q.P4f[k] = make_float4((float)(d[0] - q.x0), (float)(d[1] - q.y0), (float)(d[2] - q.z0),
                           (float)v[0]);
    if (q.U4f) q.U4f[k] = make_float4((float)d[3], (float)d[4], (float)d[5], 0.f);
    q.perm[k] = slot;
}

__global__ void k_scene_ranges_init(int ns, int n, int* __restrict__ first, int* __restrict__ last)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < ns) { first[k] = n; last[k] = 0; }
}

// slot range [first, last) of each scene after the reorder: only the particles
// at a scene's boundaries touch the two words (an atomic per particle on one
// address took 435 us for 64 scenes of 5.4 k particles)
__global__ void k_scene_ranges(int n, const int* __restrict__ scene, int* __restrict__ first,
                               int* __restrict__ last)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    int s = scene[k];
    if (k == 0 || scene[k - 1] != s) atomicMin(&first[s], k);
    if (k == n - 1 || scene[k + 1] != s) atomicMax(&last[s], k + 1);
}

// One list, G lanes per particle, row-major.  Membership is the reference's
// exact FP64 rule (3D: d <= cut, self included; 2D: d < cut, self excluded)
// over the 3x3(x3) cells around the particle's cell (functions.cu:2854-2918).
// The three cells of one (y, z) offset are consecutive in the grid's order
// (cells are numbered x fastest), so they are scanned as one range; cells
// whose box lies farther than the cutoff from the particle are left out.
// Inside a cell the order is by x, so a range is sorted by x and shrinks to
// the x-window [x_i - r, x_i + r], r the largest |dx| that the particle's
// distance to the range's (y, z) cells leaves under the cutoff
// (conservative margins); the lanes of the group find the windows of their
// runs (lane l: runs l, l + G, ...) by binary searches over the order keys
// of x.  Rows are stored in scan order (y, z outer, memory order inside);
// the reference's own order (x offset outermost, ascending id per cell) is
// restored when lists are exported (mps_download_lists).
// 6 resident blocks per SM (40 registers).  Both lists, us, at 4 / 6 / 8 blocks (32
// registers, spills): 3D, 54 k particles 142 / 148 / 159; 2D, 345 k 159 / 151 / 149, 1.9 k
// 20 / 20 / 23
template <int DIM, int G, bool PERM>
__global__ void __launch_bounds__(256, 6) k_lists(int n, Grid g, double cut, float cut_lo, float cut_hi, int cap,
                        const double4* __restrict__ P4, const float4* __restrict__ P4f,
                        const int* __restrict__ cell, const int* __restrict__ cst,
                        const int* __restrict__ cnt, const int* __restrict__ perm,
                        const unsigned long long* __restrict__ keys, const double* __restrict__ xs,
                        int* __restrict__ out, int* __restrict__ len, int* len_max, int which,
                        unsigned int* err)
{
    // The warp's 32 / G groups step through their runs together (every
    // loop trip count is the warp's largest, lanes past their own run's end
    // idle): divergent groups would replay each ballot and shuffle once per
    // group.  Groups past the last row take part with empty runs.
    Grp<G> q;
    const bool live = q.gid < n;
    const int i = live ? (int)q.gid : 0;
    double4 pi = P4[i];
    float4 fi = P4f[i];
    int C = cell[i] - 1;
    int ic = C % g.ncx + 1, jc = (C / g.ncx) % g.ncy + 1, kc = C / (g.ncx * g.ncy) + 1;
    int m1 = (ic == 1) ? 0 : -1, m2 = (ic == g.ncx) ? 0 : 1;
    int m3 = (jc == 1) ? 0 : -1, m4 = (jc == g.ncy) ? 0 : 1;
    int m5 = 0, m6 = 0;
    if (DIM == 3) { m5 = (kc == 1) ? 0 : -1; m6 = (kc == g.ncz) ? 0 : 1; }
    // distances from the particle to the faces of its own cell; a margin of
    // 1e-9 cell sizes keeps the culling conservative under rounding
    const double mx = 1e-9 * g.re, mz = 1e-9 * g.rez;
    double lox = pi.x - (g.xmin + (ic - 1) * g.re) - mx, hix = (g.xmin + ic * g.re) - pi.x - mx;
    double loy = pi.y - (g.ymin + (jc - 1) * g.re) - mx, hiy = (g.ymin + jc * g.re) - pi.y - mx;
    double loz = 0, hiz = 0;
    if (DIM == 3) {
        loz = pi.z - (g.zmin + (kc - 1) * g.rez) - mz;
        hiz = (g.zmin + kc * g.rez) - pi.z - mz;
    }
    auto gap2 = [](int off, double lo, double hi) {
        double d = off < 0 ? lo : (off > 0 ? hi : 0.0);
        return d > 0 ? d * d : 0.0;
    };
    const double gxl = gap2(-1, lox, hix), gxh = gap2(1, lox, hix);
    const int ndp = m6 - m5 + 1, nt = live ? (m4 - m3 + 1) * ndp : 0;
    // the windows of this lane's runs t = lane, lane + G, ...
    constexpr int NT = DIM == 3 ? 9 : 3;
    constexpr int R = (NT + G - 1) / G;
    int wb[R], we[R];
#pragma unroll
    for (int u = 0; u < R; u++) {
        const int t = q.lane + u * G;
        wb[u] = 0;
        we[u] = 0;
        if (t >= nt) continue;
        const int cu = m3 + t / ndp, dp = m5 + t % ndp;
        const double gyz = gap2(cu, loy, hiy) + (DIM == 3 ? gap2(dp, loz, hiz) : 0.0);
        if (gyz > cut) continue;
        const int rlo = (m1 < 0 && gyz + gxl <= cut) ? -1 : 0;
        const int rhi = (m2 > 0 && gyz + gxh <= cut) ? 1 : 0;
        const int Cr = ic + (jc - 1 + cu) * g.ncx + (kc - 1 + dp) * g.ncx * g.ncy;
        // |dx| above r puts the pair beyond the cutoff with room for every
        // rounding of the distance
        const double r = sqrt(cut - gyz) * (1.0 + 1e-12) + mx;
        const unsigned long long klo = order_key(pi.x - r), khi = order_key(pi.x + r);
        int lo_a = cst[Cr + rlo], hi_a = cst[Cr + rhi] + cnt[Cr + rhi];
        int lo_b = lo_a, hi_b = hi_a;
        while (lo_a < hi_a || lo_b < hi_b) {
            const int ma = (lo_a + hi_a) >> 1, mb = (lo_b + hi_b) >> 1;
            const bool sa = lo_a < hi_a, sb = lo_b < hi_b;
            const unsigned long long va = sa ? (PERM ? keys[ma] : order_key(xs[ma])) : 0ull;
            const unsigned long long vb = sb ? (PERM ? keys[mb] : order_key(xs[mb])) : 0ull;
            if (sa) { if (va < klo) lo_a = ma + 1; else hi_a = ma; }
            if (sb) { if (vb <= khi) lo_b = mb + 1; else hi_b = mb; }
        }
        wb[u] = lo_a;
        we[u] = max(lo_a, lo_b);
    }
    int* row = out + (size_t)i * cap;
    int k = 0;
    const unsigned full = 0xffffffffu;
#pragma unroll
    for (int t = 0; t < NT; t++) {
        const int src_lane = (int)q.base + t % G;
        const int b = __shfl_sync(full, wb[t / G], src_lane);
        const int e = __shfl_sync(full, we[t / G], src_lane);
        const int trips = __reduce_max_sync(full, (e - b + G - 1) / G);
        for (int it = 0; it < trips; it++) {
            const int jj = b + it * G + q.lane;
            const bool valid = jj < e;
            bool in = false;
            int j = 0;
            if (valid) {
                j = PERM ? perm[jj] : jj;
                // FP32 screen; the exact FP64 rule decides only inside
                // the screening margin [cut_lo, cut_hi]
                const float4 fj = P4f[j];
                const float ex = fj.x - fi.x, ey = fj.y - fi.y,
                            ez = DIM == 3 ? fj.z - fi.z : 0.f;
                // fused multiply-adds: fewer roundings than the bound assumes
                const float f2 = __fmaf_rn(ez, ez, __fmaf_rn(ey, ey, __fmul_rn(ex, ex)));
                if (f2 < cut_lo) {
                    in = (DIM == 3) || (j != i);
                } else if (f2 <= cut_hi) {
                    const double4 pj = P4[j];
                    const double d2 = dist2<DIM>(pj.x - pi.x, pj.y - pi.y,
                                                 DIM == 3 ? pj.z - pi.z : 0.0);
                    in = (DIM == 3) ? (d2 <= cut) : (j != i && d2 < cut);
                }
            }
            const unsigned m = (__ballot_sync(full, in) >> q.base) & ((1u << G) - 1u);
            if (in) {
                const int pos = k + __popc(m & ((1u << q.lane) - 1u));
                if (pos < cap) row[pos] = j;
            }
            k += __popc(m);
        }
    }
    // the longest row: one atomic per warp instead of one per particle
    const int km = __reduce_max_sync(full, live ? k : 0);
    if ((threadIdx.x & 31) == 0) atomicMax(&len_max[which], km);
    if (live && q.lane == 0) {
        if (k > cap) {
            set_error(err, MPS_ERR_LIST_OVERFLOW);
            k = cap;
        }
        len[i] = k;
    }
}

// One list in 3D, one particle per lane: a warp takes 32 consecutive particles
// of the grid's order and walks the candidates of their common row of cells
// together.  Membership is the reference's exact FP64 rule (d <= cut, self
// included) over the 3x3x3 cells around each particle's cell
// (functions.cu:2854-2918), as k_lists has it, and rows come out entry for entry
// the same.  Bound by instruction issue: 17 k warp instructions per 32 particles
// of the Laplacian list against 50 k with four particles of a cell per warp and a
// ballot per particle and 32 candidates.
//
// The three (or more) cells of one (y, z) offset are consecutive in the grid's
// order (cells are numbered x fastest) and sorted by x through, so the warp's
// candidates there lie in one window [x_min - r, x_max + r], r the largest
// |dx| that the nearest of its particles to that row leaves under the cutoff
// (conservative margins); lane t finds row t's window by binary searches over
// the order keys of x.  Candidates are staged 64 at a time in shared memory,
// as coordinates that every lane reads by broadcast: a candidate costs one
// FP32 distance per lane for 32 pairs, in packed FP32 arithmetic (sm_100's f32x2)
// and without a branch, a ballot or a compaction.  Candidates out of reach of
// the box around the warp's particles are dropped as they are staged.  A
// lane appends its members to its own column of a shared buffer
// (conflict-free) and writes them to its row eight at a time, one 32-byte
// store each.  A pair whose FP32 distance lies in the screening margin, or
// that could sit two cells apart along x, is decided by the FP64 rule.
// Warps that straddle rows of cells take one row after another.
//
// Rows are stored in scan order (y, z outer, memory order inside); the
// reference's own order (x offset outermost, ascending id per cell) is
// restored when lists are exported (mps_download_lists).
// entries a lane may hold back: with 48 a block takes 7.1 KB of shared memory and 1 KB
// reserved, and 28 blocks (warps) fit an SM (1.6 M dam, Laplacian and PND list 1328 /
// 524 us; 56 entries, 24 blocks, 1372 / 527; 64 entries, 22 blocks, 1419 / 545)
constexpr int kListBuf = 48;
constexpr int kListFlush = kListBuf - 32;  // flushed once a lane holds more (32 candidates add at most 32)
// cells a warp's particles may span along x in one pass: a sparse row's next
// particles may be a whole tank away, and the pass would walk all between
// (Laplacian list of the 476 k-particle dam 717 us unlimited, 457 with 3 cells)
constexpr int kSpanL = 2, kSpanS = 4;

struct ListArgs {
    int n, cap, which;
    Grid g;
    double cut;           // squared cutoff
    float mid, margin;    // FP32 d2 - mid beyond -margin / margin decides by itself
    float x_safe;         // FP32 |dx| up to this: at most one cell apart along x
};

// unsigned key whose order is the order of the floats, and back
__device__ __forceinline__ unsigned float_key(float v)
{
    const unsigned b = __float_as_uint(v);
    return (b >> 31) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float float_of(unsigned k)
{
    return __uint_as_float((k >> 31) ? (k & 0x7fffffffu) : ~k);
}

// two FP32 values in one register pair (sm_100's packed arithmetic: the same
// roundings as the scalar instructions, half the issue slots)
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// candidate j into the lane's column: stored always, kept when in (t <= margin)
__device__ __forceinline__ void append(unsigned& wp, int j, float t, float margin)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.le.f32 p, %2, %3;\n\tst.shared.u32 [%0], %1;\n\t"
                 "@p add.u32 %0, %0, 128;\n\t}"
                 : "+r"(wp) : "r"(j), "f"(t), "f"(margin) : "memory");
}

template <bool PERM>
__global__ void __launch_bounds__(32, 32) k_lists_lane(
    ListArgs A, const double4* __restrict__ P4, const float4* __restrict__ P4f,
    const double* __restrict__ xs, const unsigned long long* __restrict__ keys,
    const int* __restrict__ perm, const int* __restrict__ cell, const int* __restrict__ cst,
    const int* __restrict__ cnt, int* __restrict__ out, int* __restrict__ len, int* len_max,
    unsigned int* err)
{
    constexpr unsigned full = 0xffffffffu;
    __shared__ __align__(16) float s_pos[4][64];  // x, y, z and the bits of the id
    __shared__ int s_buf[kListBuf + 1][32];  // (one store past the last entry)
    const int lane = threadIdx.x;
    const Grid& g = A.g;
    const int pos = blockIdx.x * 32 + lane;
    const bool live = pos < A.n;
    const int i = live ? (PERM ? perm[pos] : pos) : 0;
    const int c0 = cell[i] - 1;
    const int rowid = c0 / g.ncx, ic = c0 - rowid * g.ncx + 1;
    const double4 pi = ld4(P4 + i);
    const float4 fi = P4f[i];
    // high halves of order keys: bounds of a coordinate over lanes by integer
    // reductions (rounded outwards by at most 2^-20 of its value)
    auto hi_key = [](double v) { return (unsigned)(order_key(v) >> 32); };
    auto from_key = [](unsigned hi, bool up) {
        const unsigned long long k = ((unsigned long long)hi << 32) | (up ? 0xffffffffull : 0ull);
        return __longlong_as_double((long long)((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k));
    };
    unsigned lt_mask;  // lanes below this one
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt_mask));
    int* const row = out + (size_t)i * A.cap;
    int kept = 0;                     // entries written to the row
    int* const col = &s_buf[0][lane];
    const unsigned col_at = (unsigned)__cvta_generic_to_shared(col);
    unsigned wp = col_at;             // shared address of the column's next free entry
    // write the column's full groups of eight (and, at the end, the rest),
    // and move what is left to its front
    auto flush = [&](bool last) {
        const int have = (int)(wp - col_at) >> 7;
        const int groups = (last ? have + 7 : have) >> 3;
        const int most = __reduce_max_sync(full, groups);
        for (int q = 0; q < most; q++) {
            if (q < groups) {
                int v[8];
#pragma unroll
                for (int t = 0; t < 8; t++) v[t] = col[(q * 8 + t) * 32];
                if (kept + 8 <= A.cap)
                    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                                 :: "l"(row + kept), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                                    "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                                 : "memory");
                kept += 8;
            }
        }
        if (last) {
            kept += have - groups * 8;
            return;
        }
        const int rest = have & 7;
        if (groups > 0)
            for (int t = 0; t < rest; t++) col[t * 32] = col[(groups * 8 + t) * 32];
        wp = col_at + rest * 128;
    };
    unsigned todo = __ballot_sync(full, live);
    while (todo) {
        // the lanes whose particles lie in the first one's row of cells, at
        // most kSpan cells on
        const int lead = __ffs(todo) - 1;
        const int rid = __shfl_sync(full, rowid, lead), ic_lo = __shfl_sync(full, ic, lead);
        const bool act = live && (todo >> lane & 1u) && rowid == rid && ic - ic_lo <= (PERM ? kSpanS : kSpanL);
        todo &= ~__ballot_sync(full, act);
        const int ic_hi = __reduce_max_sync(full, act ? ic : 0);
        auto low = [&](double v) {
            return from_key(__reduce_min_sync(full, act ? hi_key(v) : full), false);
        };
        auto high = [&](double v) {
            return from_key(__reduce_max_sync(full, act ? hi_key(v) : 0u), true);
        };
        const double x_lo = low(pi.x), x_hi = high(pi.x), y_lo = low(pi.y), y_hi = high(pi.y);
        const double z_lo = low(pi.z), z_hi = high(pi.z);
        // the FP32 box of the particles
        auto lowf = [&](float v) {
            return float_of(__reduce_min_sync(full, act ? float_key(v) : full));
        };
        auto highf = [&](float v) {
            return float_of(__reduce_max_sync(full, act ? float_key(v) : 0u));
        };
        const float fx_lo = lowf(fi.x), fx_hi = highf(fi.x), fy_lo = lowf(fi.y), fy_hi = highf(fi.y);
        const float fz_lo = lowf(fi.z), fz_hi = highf(fi.z);
        const int jc = rid % g.ncy + 1, kc = rid / g.ncy + 1;
        const int m3 = (jc == 1) ? 0 : -1, m4 = (jc == g.ncy) ? 0 : 1;
        const int m5 = (kc == 1) ? 0 : -1, m6 = (kc == g.ncz) ? 0 : 1;
        const int ndp = m6 - m5 + 1, nt = (m4 - m3 + 1) * ndp;
        // lane t: the candidate window of row t of cells
        int rb = 0, re = 0, rc = 0;
        if (lane < nt) {
            const int cu = m3 + lane / ndp, dp = m5 + lane % ndp;
            const double mx = 1e-9 * g.re, mz = 1e-9 * g.rez;
            // distance from the particles to the row, squared; a margin of
            // 1e-9 cell sizes keeps it conservative under rounding
            auto gap2 = [](int off, double below, double above) {
                const double d = off < 0 ? below : (off > 0 ? above : 0.0);
                return d > 0 ? d * d : 0.0;
            };
            double gyz = gap2(cu, y_lo - (g.ymin + (jc - 1) * g.re) - mx,
                              (g.ymin + jc * g.re) - y_hi - mx);
            gyz += gap2(dp, z_lo - (g.zmin + (kc - 1) * g.rez) - mz,
                            (g.zmin + kc * g.rez) - z_hi - mz);
            if (!(gyz > A.cut)) {
                const int first = (jc - 1 + cu) * g.ncx + (kc - 1 + dp) * g.ncx * g.ncy;
                const int ca = first + max(ic_lo - 1, 1), cb = first + min(ic_hi + 1, g.ncx);
                // |dx| above r puts a pair beyond the cutoff with room for
                // every rounding of the distance
                const double r = sqrt(A.cut - gyz) * (1.0 + 1e-12) + mx;
                const unsigned long long klo = order_key(x_lo - r), khi = order_key(x_hi + r);
                int lo_a = cst[ca], hi_a = cst[cb] + cnt[cb];
                int lo_b = lo_a, hi_b = hi_a;
                while (lo_a < hi_a || lo_b < hi_b) {
                    const int ma = (lo_a + hi_a) >> 1, mb = (lo_b + hi_b) >> 1;
                    const bool sa = lo_a < hi_a, sb = lo_b < hi_b;
                    const unsigned long long va = sa ? (PERM ? keys[ma] : order_key(xs[ma])) : 0ull;
                    const unsigned long long vb = sb ? (PERM ? keys[mb] : order_key(xs[mb])) : 0ull;
                    if (sa) { if (va < klo) lo_a = ma + 1; else hi_a = ma; }
                    if (sb) { if (vb <= khi) lo_b = mb + 1; else hi_b = mb; }
                }
                rb = lo_a;
                re = max(lo_a, lo_b);
                rc = first;
            }
        }
        // lanes of other rows see nothing within reach
        const float fx = act ? -fi.x : 1e30f;
        const bool spans = ic_lo != ic_hi;
        // a pair that FP32 leaves open, by the exact rule: -1 in, 1 out
        auto decide = [&](float t, float e, int j) {
            if (!(t <= A.margin) || !(fabsf(t) <= A.margin || fabsf(e) > A.x_safe)) return t;
            const double4 pj = ld4(P4 + j);
            const double d2 = dist2<3>(pj.x - pi.x, pj.y - pi.y, pj.z - pi.z);
            const int dc = (cell[j] - 1) % g.ncx + 1 - ic;
            const bool in = d2 <= A.cut && dc >= -1 && dc <= 1;
            return in ? -1e30f : 1e30f;
        };
        // the windows' candidates, 64 at a time; the next batch's positions
        // travel while this one is tested
        int t = -1, b = 0, e = 0;
        int own_b = 0, own_e = 0;  // the row's candidates within a cell of the lane's
        auto next = [&]() {  // advance to the next batch [b, min(b + 64, e))
            b += 64;
            while (b >= e && ++t < nt) {
                b = __shfl_sync(full, rb, t);
                e = __shfl_sync(full, re, t);
                if (spans && b < e) {
                    const int first = __shfl_sync(full, rc, t);
                    const int cb = first + min(ic + 1, g.ncx);
                    own_b = act ? cst[first + max(ic - 1, 1)] : 0;
                    own_e = act ? cst[cb] + cnt[cb] : 0;
                }
            }
            return t < nt;
        };
        float4 f[2];
        int id[2] = {0, 0};
        auto fetch = [&]() {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int jj = b + h * 32 + lane;
                f[h] = make_float4(1e30f, 1e30f, 1e30f, 0.f);
                if (jj < e) {
                    id[h] = PERM ? perm[jj] : jj;
                    f[h] = P4f[id[h]];
                }
            }
        };
        bool more = next();
        if (more) fetch();
        while (more) {
            // a warp over several cells of the row (the cutoff is longer than a
            // cell): lanes more than a cell away from all of the
            // batch sit it out, and a batch that straddles some lane's limit
            // checks its pairs' |dx|
            float ox = fx;
            bool mixed = false;
            if (spans) {
                const int last = min(b + 64, e);
                const bool none = b >= own_e || last <= own_b;
                if (none) ox = 1e30f;
                mixed = __any_sync(full, act && !none && (b < own_b || last > own_e));
            }
            // keep the candidates within reach of the particles' box: its FP32
            // distance, in the pairs' own arithmetic, is at most each pair's
            int m = 0;
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float gx = fmaxf(fmaxf(fx_lo - f[h].x, f[h].x - fx_hi), 0.f);
                const float gy = fmaxf(fmaxf(fy_lo - f[h].y, f[h].y - fy_hi), 0.f);
                float gd = __fmaf_rn(gy, gy, __fmaf_rn(gx, gx, -A.mid));
                const float gz = fmaxf(fmaxf(fz_lo - f[h].z, f[h].z - fz_hi), 0.f);
                gd = __fmaf_rn(gz, gz, gd);
                const bool reach = gd <= A.margin;
                const unsigned who = __ballot_sync(full, reach);
                if (reach) {
                    const int p = m + __popc(who & lt_mask);
                    s_pos[0][p] = f[h].x;
                    s_pos[1][p] = f[h].y;
                    s_pos[2][p] = f[h].z;
                    s_pos[3][p] = __int_as_float(id[h]);
                }
                m += __popc(who);
            }
            if (lane < (-m & 3)) s_pos[0][m + lane] = 1e30f;  // fill the last four
            __syncwarp();
            more = next();
            if (more) fetch();
            const f32x2 ox2 = pack2(ox, ox), oy2 = pack2(-fi.y, -fi.y), oz2 = pack2(-fi.z, -fi.z);
            const f32x2 mid2 = pack2(-A.mid, -A.mid);
            auto scan = [&](auto check, int from, int to) {
                constexpr bool CHK = decltype(check)::value;
                const float* const c = s_pos[0];
                for (int q = from; q < to; q += 4) {
                    const ulonglong2 cx = *reinterpret_cast<const ulonglong2*>(c + q);
                    const ulonglong2 cy = *reinterpret_cast<const ulonglong2*>(c + 64 + q);
                    const ulonglong2 cz = *reinterpret_cast<const ulonglong2*>(c + 128 + q);
                    const int4 cj = *reinterpret_cast<const int4*>(c + 192 + q);
                    // d2 - mid of four pairs; fused multiply-adds: no more
                    // roundings than the bound assumes
                    const f32x2 ex0 = add2(cx.x, ox2), ex1 = add2(cx.y, ox2);
                    const f32x2 ey0 = add2(cy.x, oy2), ey1 = add2(cy.y, oy2);
                    const f32x2 ez0 = add2(cz.x, oz2), ez1 = add2(cz.y, oz2);
                    f32x2 d0 = fma2(ey0, ey0, fma2(ex0, ex0, mid2));
                    f32x2 d1 = fma2(ey1, ey1, fma2(ex1, ex1, mid2));
                    d0 = fma2(ez0, ez0, d0);
                    d1 = fma2(ez1, ez1, d1);
                    float t0, t1, t2, t3;
                    unpack2(d0, t0, t1);
                    unpack2(d1, t2, t3);
                    const float near = fminf(fminf(fabsf(t0), fabsf(t1)), fminf(fabsf(t2), fabsf(t3)));
                    float e0 = 0.f, e1 = 0.f, e2 = 0.f, e3 = 0.f, far = 0.f;
                    if (CHK) {
                        unpack2(ex0, e0, e1);
                        unpack2(ex1, e2, e3);
                        far = fmaxf(fmaxf(t0 <= A.margin ? fabsf(e0) : 0.f, t1 <= A.margin ? fabsf(e1) : 0.f),
                                    fmaxf(t2 <= A.margin ? fabsf(e2) : 0.f, t3 <= A.margin ? fabsf(e3) : 0.f));
                    }
                    if (near <= A.margin || (CHK && far > A.x_safe)) {
                        t0 = decide(t0, e0, cj.x);
                        t1 = decide(t1, e1, cj.y);
                        t2 = decide(t2, e2, cj.z);
                        t3 = decide(t3, e3, cj.w);
                    }
                    append(wp, cj.x, t0, A.margin);
                    append(wp, cj.y, t1, A.margin);
                    append(wp, cj.z, t2, A.margin);
                    append(wp, cj.w, t3, A.margin);
                }
            };
            for (int h = 0; h < m; h += 32) {
                const int to = min(h + 32, m);
                if (mixed) scan(std::true_type(), h, to);
                else scan(std::false_type(), h, to);
                if (__any_sync(full, wp > col_at + kListFlush * 128)) flush(false);
            }
        }
    }
    flush(true);
    const int longest = __reduce_max_sync(full, live ? kept : 0);
    if (lane == 0) atomicMax(&len_max[A.which], longest);
    if (live) {
        if (kept > A.cap) {
            set_error(err, MPS_ERR_LIST_OVERFLOW);
            kept = A.cap;
        }
        len[i] = kept;
    }
}

// 3D scenes of this many particles on take one particle per lane
// (k_lists_lane); smaller ones, and 2D, lane groups (k_lists): a lane walks all
// the candidates of its warp's 32 particles, about 100 us however few warps there
// are, and in 2D, with a fifth of the candidates per particle, the groups are as
// fast.  Laplacian and PND list, us, groups against lanes: 54 k particles 95 / 50
// against 107 / 49, 125 k 223 / 89 against 152 / 65, 476 k 852 / 319 (groups of
// four particles of a cell per warp) against 445 / 177; 2D, 345 k 121 / 52
// against 113 / 67
constexpr int kLaneMin = 65536;
// lanes per particle of the groups on the Laplacian grid: 16 in 3D (54 k
// particles: 95 us; 8 lanes 99, 4 lanes 121), in 2D 4 from kLarge2 particles on (86 k:
// 29.5 us; 8 lanes 35.5, 16 lanes 49) and 8 below (15 k: 11.1 us; 16 lanes 13.4, 4
// lanes 13.3; 1.9 k: 8.7, 7.2 and 12.1)
constexpr int kListG3 = 16, kListG2 = 8, kListG2Large = 4, kLarge2 = 65536;

void scan(mps_ctx* ctx, Scans a, int count)
{
    int m = a.m[0];
    for (int k = 1; k < count; k++) m = std::max(m, a.m[k]);
    if (m <= kScanSmall) {
        k_scan_small<<<dim3(1, count), kScanThreads, 0, ctx->stream>>>(a);
        vmps_count_launch(1);
        return;
    }
    const int tiles = (m + kScanTile - 1) / kScanTile;
    for (int k = 0; k < count; k++) a.tile_sum[k] = ctx->scan_tmp + (size_t)k * ctx->scan_pitch;
    k_scan_tiles<<<dim3(tiles, count), kScanThreads, 0, ctx->stream>>>(a);
    k_scan_sums<<<dim3(1, count), kScanThreads, 0, ctx->stream>>>(a);
    k_scan_apply<<<dim3(tiles, count), kScanThreads, 0, ctx->stream>>>(a);
    vmps_count_launch(3);
}

}  // namespace

int vmps_scan(mps_ctx* ctx, int m, const int* in, int* out)
{
    Scans a{};
    a.m[0] = m;
    a.in[0] = in;
    a.out[0] = out;
    scan(ctx, a, 1);
    return MPS_OK;
}

// Persistent fields carried through the reorder (all other fields are
// recomputed each step before use).
static void persistent_set(mps_ctx* ctx, GatherSet& g, std::vector<void**>& slots,
                           std::vector<void*>& alts)
{
    slots.clear();
    double** d[kGatherD] = {&ctx->x, &ctx->y, &ctx->z, &ctx->u, &ctx->v, &ctx->w, &ctx->p,
                            &ctx->pnew, &ctx->phat, &ctx->un, &ctx->vn, &ctx->wn, &ctx->rho,
                            &ctx->nd, &ctx->pold};
    int** ii[kGatherI] = {&ctx->ptype, &ctx->oid, &ctx->cell_l, &ctx->cell_s, &ctx->scene,
                          &ctx->own};
    for (int a = 0; a < kGatherD; a++) {
        g.from_d[a] = *d[a];
        g.to_d[a] = (double*)alts[a];
        slots.push_back((void**)d[a]);
    }
    for (int a = 0; a < kGatherI; a++) {
        g.from_i[a] = *ii[a];
        g.to_i[a] = (int*)alts[kGatherD + a];
        slots.push_back((void**)ii[a]);
    }
}

// Alternate buffers for the reorder live in ctx->owned after the primaries;
// they are registered by vmps_alloc_reorder() in mps_context.cu.
extern std::vector<void*>& vmps_reorder_alts(mps_ctx* ctx);

// Exchange the persistent fields with their alternates (the reorder wrote
// the alternates).  A replayed step graph skips the capture-time host code,
// so the graph path calls this once per replay.
void vmps_reorder_swap(mps_ctx* ctx)
{
    GatherSet g;
    std::vector<void**> slots;
    std::vector<void*>& alts = vmps_reorder_alts(ctx);
    persistent_set(ctx, g, slots, alts);
    for (size_t a = 0; a < slots.size(); a++) {
        void* old = *slots[a];
        *slots[a] = alts[a];
        alts[a] = old;
    }
    ctx->swaps++;
}

int vmps_neighbors(mps_ctx* ctx)
{
    const int n = ctx->n;
    cudaStream_t st = ctx->stream;
    int nb = grid_blocks(n);
    // both grids' counts and the longest rows lie side by side
    VMPS_CUDA(ctx, cudaMemsetAsync(ctx->cnt_l, 0,
                                   sizeof(int) * ((size_t)ctx->gl.tnc + ctx->gs.tnc + 6), st));
    if (ctx->cfg.dim == 3)
        k_hash<3><<<nb, kBlock, 0, st>>>(n, ctx->gl, ctx->gs, ctx->x, ctx->y, ctx->z, ctx->cell_l,
                                         ctx->cell_s, ctx->cnt_l, ctx->cnt_s, ctx->bpos_l,
                                         ctx->bpos_s, ctx->d_err);
    else
        k_hash<2><<<nb, kBlock, 0, st>>>(n, ctx->gl, ctx->gs, ctx->x, ctx->y, ctx->z, ctx->cell_l,
                                         ctx->cell_s, ctx->cnt_l, ctx->cnt_s, ctx->bpos_l,
                                         ctx->bpos_s, ctx->d_err);
    vmps_count_launch(1);
    Scans cells{};
    cells.m[0] = ctx->gl.tnc + 2;
    cells.in[0] = ctx->cnt_l;
    cells.out[0] = ctx->cst_l;
    cells.m[1] = ctx->gs.tnc + 2;
    cells.in[1] = ctx->cnt_s;
    cells.out[1] = ctx->cst_s;
    scan(ctx, cells, 2);
    k_scatter<<<nb, kBlock, 0, st>>>(n, ctx->cell_l, ctx->cell_s, ctx->bpos_l, ctx->bpos_s,
                                     ctx->cst_l, ctx->cst_s, ctx->oid, ctx->x, ctx->bslot_l,
                                     ctx->boid_l, ctx->bx_l, ctx->bslot_s, ctx->boid_s,
                                     ctx->bx_s);
    k_rank<<<dim3(nb, 2), kBlock, 0, st>>>(n, ctx->cell_l, ctx->cell_s, ctx->cst_l, ctx->cnt_l, ctx->cst_s,
                                  ctx->cnt_s, ctx->bslot_l, ctx->boid_l, ctx->bx_l,
                                  ctx->bslot_s, ctx->boid_s, ctx->bx_s, ctx->src, ctx->inv,
                                  ctx->perm_s_tmp, ctx->key_s);
    vmps_count_launch(2);
    // reorder persistent state into cell order
    GatherSet g;
    std::vector<void**> slots;
    std::vector<void*>& alts = vmps_reorder_alts(ctx);
    persistent_set(ctx, g, slots, alts);
    const mps_config& f = ctx->cfg;
    const GatherPack pk{ctx->P4, ctx->U4, ctx->P4f, f.precision >= 1 ? ctx->U4f : nullptr, f.xmin,
                        f.ymin, f.dim == 3 ? f.zmin : 0.0, ctx->inv, ctx->perm_s_tmp, ctx->perm_s};
    k_gather<<<nb, kBlock, 0, st>>>(n, ctx->src, g, pk);
    vmps_count_launch(1);
    vmps_reorder_swap(ctx);
    if (ctx->nscenes > 1) {
        k_scene_ranges_init<<<grid_blocks(ctx->nscenes), kBlock, 0, st>>>(ctx->nscenes, n,
                                                                          ctx->sfirst, ctx->slast);
        k_scene_ranges<<<nb, kBlock, 0, st>>>(n, ctx->scene, ctx->sfirst, ctx->slast);
        vmps_count_launch(2);
    }
    if (ctx->profile) VMPS_CUDA(ctx, cudaEventRecord(ctx->ev[6], st));
    {
        const bool three = ctx->cfg.dim == 3;
        const double* x = ctx->x;
        if (three && n >= kLaneMin) {
            auto args = [&](int cap, int which, const Grid& g, double cut) {
                // screening margin around the cutoff, rounded outwards, and the
                // FP32 |dx| that leaves two particles at most a cell apart
                const double u = std::ldexp(1.0, -24);
                const double de = 2 * (ctx->cfg.xmax - ctx->cfg.xmin) * u + std::sqrt(cut) * u;
                const double m = ctx->screen_abs + cut * 2 * u;
                return ListArgs{n, cap, which, g, cut, (float)cut,
                                std::nextafter((float)m, INFINITY),
                                (float)(g.re * (1 - 1e-5) - 2 * de)};
            };
            const int nw = (n + 31) / 32;
            k_lists_lane<false><<<nw, 32, 0, st>>>(
                args(ctx->cap_l, 0, ctx->gl, ctx->cut_l), ctx->P4, ctx->P4f, x, nullptr, nullptr,
                ctx->cell_l, ctx->cst_l, ctx->cnt_l, ctx->nbr_l, ctx->len_l, ctx->len_max, ctx->d_err);
            k_lists_lane<true><<<nw, 32, 0, st>>>(
                args(ctx->cap_s, 1, ctx->gs, ctx->cut_s), ctx->P4, ctx->P4f, x, ctx->key_s,
                ctx->perm_s, ctx->cell_s, ctx->cst_s, ctx->cnt_s, ctx->nbr_s, ctx->len_s,
                ctx->len_max, ctx->d_err);
        } else {
            // screening window, rounded outwards to float
            auto lo = [&](double c) { return std::nextafter((float)(c - ctx->screen_abs), 0.f); };
            auto hi = [&](double c) { return std::nextafter((float)(c + ctx->screen_abs), INFINITY); };
            auto blocks = [&](int g) { return (int)(((long)n * g + kBlock - 1) / kBlock); };
            const bool large = n >= kLarge2;
            (three ? k_lists<3, kListG3, false>
                   : large ? k_lists<2, kListG2Large, false> : k_lists<2, kListG2, false>)
                <<<blocks(three ? kListG3 : large ? kListG2Large : kListG2), kBlock, 0, st>>>(
                    n, ctx->gl, ctx->cut_l, lo(ctx->cut_l), hi(ctx->cut_l), ctx->cap_l, ctx->P4,
                    ctx->P4f, ctx->cell_l, ctx->cst_l, ctx->cnt_l, nullptr, nullptr, x, ctx->nbr_l,
                    ctx->len_l, ctx->len_max, 0, ctx->d_err);
            constexpr int G3 = SmallG<3>::G, G2 = SmallG<2>::G;
            const bool wide = ctx->tune_small_wide != 0;
            auto small = three ? (wide ? k_lists<3, 2 * G3, true> : k_lists<3, G3, true>)
                               : (wide ? k_lists<2, 2 * G2, true> : k_lists<2, G2, true>);
            small<<<blocks((three ? G3 : G2) * (wide ? 2 : 1)), kBlock, 0, st>>>(
                n, ctx->gs, ctx->cut_s, lo(ctx->cut_s), hi(ctx->cut_s), ctx->cap_s, ctx->P4,
                ctx->P4f, ctx->cell_s, ctx->cst_s, ctx->cnt_s, ctx->perm_s, ctx->key_s, x,
                ctx->nbr_s, ctx->len_s, ctx->len_max, 1, ctx->d_err);
        }
    }
    vmps_count_launch(2);
    if (ctx->profile) {
        VMPS_CUDA(ctx, cudaEventRecord(ctx->ev[7], st));
        VMPS_CUDA(ctx, cudaEventSynchronize(ctx->ev[7]));
        float ms = 0;
        VMPS_CUDA(ctx, cudaEventElapsedTime(&ms, ctx->ev[6], ctx->ev[7]));
        ctx->lists_ms += ms;
        ctx->lists_launches++;
    }
    // mps_step_io's velocities and pressure, copied while the lists were
    // built, go into the new order (nothing above reads them)
    if (ctx->state_defer) {
        int r = vmps_state_apply(ctx);
        if (r != MPS_OK) return r;
    }
    VMPS_CUDA(ctx, cudaGetLastError());
    return MPS_OK;
}
