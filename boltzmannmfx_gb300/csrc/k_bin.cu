// k_bin.cu -- counting-sort binning of the slots into columns, the prefix
// scan, the deterministic in-column order, the caller-order <-> slot-order
// moves, and the neighbour-list export.
//
// Replaces AMReX's neighbour machinery as BMX drives it every step
// (clearNeighbors / Redistribute / fillNeighbors / buildNeighborList,
// src/des/bmx_pc_interaction.cpp:97-103): bins are the level's cells, the
// pair predicate is BMXCheckPair(DEM::neighborhood, false)
// (src/des/bmx_pc.H:55-82), periodic images come from a one-cell halo
// (src/des/bmx_pc.cpp:23).  All of it is integer / byte work bounded by HBM
// and L2 bandwidth; nothing here is a contraction.
#include <algorithm>
#include <atomic>

#include <cooperative_groups.h>

#include "bmxg_pdl.cuh"
#include "bmxg_stencil.cuh"

namespace bmxg {

namespace {

__global__ void k_bin(const DevState S, int b)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n; i += gridDim.x * blockDim.x) {
        const DevGeom &G = geom_of(S, i);
        rebin_slot(S, G, i, S.x[b][i], S.y[b][i], S.z[b][i], S.rad[i], b);
    }
}

// ---- exclusive scan of n ints into n+1 offsets ----------------------------
// Three passes: tile sums, a scan of the tile sums, the scan of each tile with
// its offset.  A thread holds four consecutive counts, read and written as one
// 16-byte vector (coalesced across the warp); a tile is 1024 counts.
constexpr int kScanBlock = 256;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanBlock * kScanItems;

__device__ __forceinline__ int block_exclusive_scan(int v, int &total)
{
    __shared__ int warp_sums[kScanBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = (lane < kScanBlock / 32) ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < kScanBlock / 32) warp_sums[lane] = w;
    }
    __syncthreads();
    const int before = (warp > 0) ? warp_sums[warp - 1] : 0;
    total = warp_sums[kScanBlock / 32 - 1];
    __syncthreads();
    return before + x - v;
}

// this thread's four counts (zero past n): one vector load where all four lie inside
__device__ __forceinline__ int4 scan_load4(const int *__restrict__ in, int n, int base)
{
    if (base + 3 < n) return __ldg(reinterpret_cast<const int4 *>(in + base));
    int4 v = make_int4(0, 0, 0, 0);
    if (base < n) v.x = in[base];
    if (base + 1 < n) v.y = in[base + 1];
    if (base + 2 < n) v.z = in[base + 2];
    return v;
}

__global__ void k_scan_reduce(const int *__restrict__ in, int n, int *__restrict__ bsum, const int *gate)
{
    if (gate && !*gate) return;
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    const int4 v = scan_load4(in, n, base);
    int total;
    block_exclusive_scan(v.x + v.y + v.z + v.w, total);
    if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}

// one block of 1024 threads over the nb tile sums: each thread sums a
// contiguous segment (its loads independent of each other), one block-wide
// scan joins the segments, each thread writes its segment's offsets
constexpr int kTopBlock = 1024;

__global__ void __launch_bounds__(kTopBlock) k_scan_top(int *bsum, int nb, const int *gate)
{
    if (gate && !*gate) return;
    __shared__ int warp_sums[kTopBlock / 32];
    const int seg = (nb + kTopBlock - 1) / kTopBlock;
    const int b0 = min((int)threadIdx.x * seg, nb), b1 = min(b0 + seg, nb);
    int s = 0;
#pragma unroll 8
    for (int k = b0; k < b1; ++k) s += bsum[k];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = warp_sums[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    int run = ((warp > 0) ? warp_sums[warp - 1] : 0) + x - s;
    for (int k = b0; k < b1; ++k) {
        const int v = bsum[k];
        bsum[k] = run;
        run += v;
    }
    if (threadIdx.x == 0) bsum[nb] = warp_sums[kTopBlock / 32 - 1];
}

__global__ void k_scan_apply(const int *__restrict__ in, int n, const int *__restrict__ bsum,
                             int *__restrict__ out, const int *gate)
{
    if (gate && !*gate) return;
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    const int4 v = scan_load4(in, n, base);
    int total;
    const int run = block_exclusive_scan(v.x + v.y + v.z + v.w, total) + bsum[blockIdx.x];
    const int4 o = make_int4(run, run + v.x, run + v.x + v.y, run + v.x + v.y + v.z);
    if (base + 3 < n) {
        *reinterpret_cast<int4 *>(out + base) = o;
    } else {
        if (base < n) out[base] = o.x;
        if (base + 1 < n) out[base + 1] = o.y;
        if (base + 2 < n) out[base + 2] = o.z;
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = bsum[gridDim.x];
}

// The end of a step: its counters into last_* and cleared, the rod queue emptied.
__device__ __forceinline__ void publish_counters(DevCounters *c, RodCtl *rctl)
{
    c->last_out_of_domain = c->out_of_domain;
    c->last_edge_ghost = c->edge_ghost;
    c->last_bond_repairs = c->bond_repairs;
    c->out_of_domain = 0ull;
    c->edge_ghost = 0ull;
    c->pairs = 0ull;
    c->bond_repairs = 0ull;
    c->moved = 0ull;
    if (rctl) {
        rctl->ncontact = 0;
        rctl->nbond = 0;
        rctl->n64 = 0;
    }
}

// ---- long columns ------------------------------------------------------------
// A slot's rank in its column counted over all of the column's keys is work of the
// square of its length: columns of tall domains.  Their keys are first put into
// ascending order kRun at a time (one warp per run of them from the column's start),
// then a rank is a binary search per run, eight reads for 128 keys.  In the cluster sort,
// whose 16 SMs counted slower than the separate kernels' blocks do, 60 000 FP64 spheres in
// 1 / 4 / 16 / 64 columns, 5 steps: 54.4 / 16.2 / 5.35 / 2.12 -> 12.8 / 4.46 / 1.93 / 1.23 ms
// (separate kernels, every key counted: 16.6 / 5.21 / 2.25 / 1.37); runs of 32: 33.9 / 10.4 /
// 3.32 / 1.46.  In a tile of 50 451 + 62 038 in 36 columns 2006 -> 1653 us (cell by cell 1791).
// Whether a state has such columns its sorts say in DevCounters::long_column, which the host
// reads with the other counters.
// kLongColumn: 65 000 spheres at 253 / 112 a column, 5 steps, from 128 slots on
// 980 / 836, from 512 on 1075 / 786 us.
constexpr int kRun = 128;

// The warp sorts the run at t (keys t .. end - 1, at most kRun of them): a bitonic
// network over four keys a lane, key e of the run in lane e & 31.
__device__ __forceinline__ void sort_run(unsigned long long *lkey, int t, int end)
{
    constexpr int M = kRun / 32;
    const int lane = threadIdx.x & 31;
    unsigned long long v[M];
#pragma unroll
    for (int j = 0; j < M; ++j) v[j] = (t + lane + 32 * j < end) ? lkey[t + lane + 32 * j] : ~0ull;
#pragma unroll
    for (int k = 2; k <= kRun; k <<= 1)
#pragma unroll
        for (int d = k >> 1; d > 0; d >>= 1)
#pragma unroll
            for (int j = 0; j < M; ++j) {
                const bool up = ((lane + 32 * j) & k) == 0;
                if (d >= 32) {
                    const int q = j | (d >> 5);
                    if (q == j) continue;
                    const unsigned long long lo = min(v[j], v[q]), hi = max(v[j], v[q]);
                    v[j] = up ? lo : hi;
                    v[q] = up ? hi : lo;
                } else {
                    const unsigned long long o = __shfl_xor_sync(0xffffffffu, v[j], d);
                    v[j] = (up == ((lane & d) == 0)) ? min(v[j], o) : max(v[j], o);
                }
            }
#pragma unroll
    for (int j = 0; j < M; ++j)
        if (t + lane + 32 * j < end) lkey[t + lane + 32 * j] = v[j];
}

// Keys below `key` among s0 .. s1 - 1, the runs from s0 in order.
__device__ __forceinline__ int rank_in_runs(const unsigned long long *lkey, int s0, int s1, unsigned long long key)
{
    int rank = 0;
    for (int t = s0; t < s1; t += kRun) {
        const int m = min(kRun, s1 - t);
        int c = 0;
#pragma unroll
        for (int d = kRun; d > 0; d >>= 1)
            if (c + d <= m && lkey[t + c + d - 1] < key) c += d;
        rank += c;
    }
    return rank;
}

// ---- scatter into columns, then the deterministic in-column order --------
// Arrival order from the atomics is arbitrary; k_canon ranks every slot by
// its (z bin, original index) key among the members of its column, which is
// the order AMReX's serial binning gives (ascending index within a bin).
// With key scratch (S.lkey: a context's state) the scatter leaves each slot's
// key at the position it drew and the rank is counted over the column's keys;
// without it (a bare caller's scratch) the slot index goes there and the
// rank gathers each member's key.
__global__ void k_scatter(const DevState S, int b)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n; i += gridDim.x * blockDim.x) {
        const int c = S.col[b][i];
        const int r = atomicSub(&S.colcnt[c], 1) - 1;  // leaves colcnt at zero
        const int t = S.colstart[b][c] + r;
        if (r == kLongColumn) S.cnt->long_column = 1ull;
        if (t >= 0 && t < S.n) {
            if (S.lkey) S.lkey[t] = col_key(S.iz[b][i], S.orig ? S.orig[i] : i);
            else S.tmp[t] = i;
        } else {
            atomicAdd(&S.cnt->bad_index, 1ULL);
        }
    }
}

// (one column per blockIdx.x; the warps of blockIdx.y's blocks take its runs in turn)
__global__ void __launch_bounds__(256) k_sort_runs(const DevState S, int b)
{
    const int s0 = max(S.colstart[b][blockIdx.x], 0), s1 = min(S.colstart[b][blockIdx.x + 1], S.n);
    const int w = (blockIdx.y * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.y * blockDim.x) >> 5;
    for (int t = s0 + w * kRun; t < s1; t += nw * kRun) sort_run(S.lkey, t, s1);
}

__global__ void k_canon(const DevState S, int b, int publish, int runs)
{
    if (publish && blockIdx.x == 0 && threadIdx.x == 0) publish_counters(S.cnt, S.rctl);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n; i += gridDim.x * blockDim.x) {
        const int c = S.col[b][i];
        const int s0 = max(S.colstart[b][c], 0), s1 = min(S.colstart[b][c + 1], S.n);
        const int izi = S.iz[b][i];
        const unsigned long long key = col_key(izi, S.orig ? S.orig[i] : i);
        int rank = 0;
        if (runs) {
            rank = rank_in_runs(S.lkey, s0, s1, key);
        } else if (S.lkey) {
            for (int t = s0; t < s1; ++t) rank += (__ldg(&S.lkey[t]) < key);
        } else {
            for (int t = s0; t < s1; ++t) {
                const int j = S.tmp[t];
                if ((unsigned)j < (unsigned)S.n) rank += (col_key(S.iz[b][j], S.orig[j]) < key);
            }
        }
        const int t = s0 + rank;
        if (t >= s1) {  // i is not among its column's members: inconsistent counts
            atomicAdd(&S.cnt->bad_index, 1ULL);
            continue;
        }
        S.perm[b][t] = i;
        if (S.srel[b]) {
            S.srel[b][t] = S.rel[b][i];
            S.siz[b][t] = izi;
            S.rank[b][i] = t;
        }
    }
}

// ---- the whole sort in one thread-block cluster ----------------------------
// Column offsets (a scan of the counts), the scatter of the keys and the
// in-column ranks of k_scan_* / k_scatter / k_canon in one launch: the blocks
// of one cluster share the scan through distributed shared memory and pass
// from phase to phase at the cluster's hardware barrier.  For states that a
// cluster's threads hold at kSortItems each, the five launches are bound by
// launch and drain latency, not by work: 2000 spheres, 100 FP64 steps and the
// load 3.91 -> 3.17 ms (with the counters' clearing nodes gone, 39 -> 31 us a step),
// 20 000-sphere adjoint over 40 steps 11.8 -> 10.4 ms.
struct SortJob {
    int n, ncols;
    const int *col, *iz, *orig;  // orig null: the index itself
    int *colcnt, *colstart;
    unsigned long long *lkey;
    int *perm;
    const float4 *rel;           // with srel: the sorted copies
    float4 *srel;
    int *siz, *rank;
    DevCounters *cnt;
    RodCtl *rctl;
    int publish;
};
constexpr int kSortBlock = 1024;
constexpr int kSortItems = 4;    // slots per thread
// Columns per thread at most: their scan runs on 16 SMs.  20 FP64 steps of 500 / 20 000 slots in
// 62 500 columns 355 / 438 us (separate kernels 413 / 448), in 129 600 391 / 511 (355 / 438), in
// 250 000 597 / 721 (365 / 439; 511 / 672 before the cluster sort).
constexpr int kSortCols = 4;
constexpr int kSortCluster = 16; // blocks at most (a non-portable size)

// The rest of k_sort_cluster, after the keys' scatter, for a state with long
// columns; at: the places the thread's slots drew.  (Of an instantiation of its own: in
// the common kernel it cost every sort 0.3 us in line, as a function 1.6.)
__device__ __forceinline__ void rank_long(const SortJob &J, int g, int T, int4 at)
{
    for (int k = 0; k < kSortItems; ++k) {  // a run is sorted by the warp whose slot drew its first place
        const int i = g + k * T;
        int t = k == 0 ? at.x : (k == 1 ? at.y : (k == 2 ? at.z : at.w)), end = 0;
        if (i < J.n) {
            const int c = J.col[i];
            const int s0 = max(J.colstart[c], 0);
            end = min(J.colstart[c + 1], J.n);
            if (end - s0 <= kLongColumn || ((t - s0) & (kRun - 1)) || t < s0 || t >= end) end = 0;
        }
        for (unsigned m = __ballot_sync(0xffffffffu, end > 0); m; m &= m - 1) {
            const int from = __ffs(m) - 1;
            sort_run(J.lkey, __shfl_sync(0xffffffffu, t, from), __shfl_sync(0xffffffffu, end, from));
        }
    }
    cooperative_groups::this_cluster().sync();
    for (int i = g; i < J.n; i += T) {
        const int c = J.col[i], z = J.iz[i];
        const int s0 = max(J.colstart[c], 0), s1 = min(J.colstart[c + 1], J.n);
        const unsigned long long key = col_key(z, J.orig ? J.orig[i] : i);
        int r = 0;
        if (s1 - s0 > kLongColumn) r = rank_in_runs(J.lkey, s0, s1, key);
        else
            for (int t = s0; t < s1; ++t) r += (J.lkey[t] < key);
        const int t = s0 + r;
        if (t >= s1) {  // i is not among its column's members: inconsistent counts
            atomicAdd(&J.cnt->bad_index, 1ULL);
            continue;
        }
        J.perm[t] = i;
        if (J.srel) {
            J.srel[t] = J.rel[i];
            J.siz[t] = z;
            J.rank[i] = t;
        }
    }
}

template <bool LONG>
__global__ void __launch_bounds__(kSortBlock) k_sort_cluster(const SortJob J)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ int warp_sums[kSortBlock / 32];
    __shared__ int block_sum;
    const int nb = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int T = nb * kSortBlock, g = rank * kSortBlock + tid;
    chain_wait();
    if (J.publish && g == 0) publish_counters(J.cnt, J.rctl);
    // this thread's slots, loaded while the scan runs
    int c[kSortItems], z[kSortItems], o[kSortItems], at[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const int i = g + k * T;
        c[k] = -1;
        if (i < J.n) {
            c[k] = J.col[i];
            z[k] = J.iz[i];
            o[k] = J.orig ? J.orig[i] : i;
        }
    }
    // the block's columns: consecutive ones per thread
    const int per = (J.ncols + T - 1) / T;
    const int q0 = min((rank * kSortBlock + tid) * per, J.ncols), q1 = min(q0 + per, J.ncols);
    int s = 0;
    for (int q = q0; q < q1; ++q) s += J.colcnt[q];
    int x = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = warp_sums[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= d) w += y;
        }
        warp_sums[lane] = w;
        if (lane == 31) block_sum = w;
    }
    cl.sync();
    int run = ((warp > 0) ? warp_sums[warp - 1] : 0) + x - s;
    {   // the sums of the cluster's earlier blocks
        int v = (lane < rank) ? *cl.map_shared_rank(&block_sum, lane) : 0;  // (at most 16 blocks)
        run += __reduce_add_sync(0xffffffffu, v);
    }
    for (int q = q0; q < q1; ++q) {
        const int v = J.colcnt[q];
        J.colstart[q] = run;
        run += v;
    }
    if (q0 < J.ncols && q1 == J.ncols) J.colstart[J.ncols] = run;
    cl.sync();
    bool is_long = false;
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        if (c[k] < 0) continue;
        const int r = atomicSub(&J.colcnt[c[k]], 1) - 1;  // leaves colcnt at zero
        const int t = J.colstart[c[k]] + r;
        if (t >= 0 && t < J.n) J.lkey[t] = col_key(z[k], o[k]);
        else atomicAdd(&J.cnt->bad_index, 1ULL);
        if (LONG) at[k] = t;
        is_long |= r == kLongColumn;
    }
    if (is_long) J.cnt->long_column = 1ull;  // (one slot of each long column)
    cl.sync();
    if constexpr (LONG) {
        rank_long(J, g, T, make_int4(at[0], at[1], at[2], at[3]));
        return;
    }
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        if (c[k] < 0) continue;
        const int i = g + k * T;
        const int s0 = max(J.colstart[c[k]], 0), s1 = min(J.colstart[c[k] + 1], J.n);
        const unsigned long long key = col_key(z[k], o[k]);
        int r = 0;
        for (int t = s0; t < s1; ++t) r += (J.lkey[t] < key);
        const int t = s0 + r;
        if (t >= s1) {  // i is not among its column's members: inconsistent counts
            atomicAdd(&J.cnt->bad_index, 1ULL);
            continue;
        }
        J.perm[t] = i;
        if (J.srel) {
            J.srel[t] = J.rel[i];
            J.siz[t] = z[k];
            J.rank[i] = t;
        }
    }
}

// caller-order variants used once by set_state (orig == caller index)
__global__ void k_user_bin(const DevState S, const double *ux, const double *uy, const double *uz,
                           int *ucol, int *uiz)
{
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < S.n; u += gridDim.x * blockDim.x) {
        const DevGeom &G = geom_of(S, u);  // colony slot ranges equal caller ranges
        const int bx = bin_of_fast(ux[u], G.plo[0], G.dxi[0], G.plof[0], G.dxif[0], 1, G.n[0]);
        const int by = bin_of_fast(uy[u], G.plo[1], G.dxi[1], G.plof[1], G.dxif[1], 1, G.n[1]);
        const int bz = bin_of_fast(uz[u], G.plo[2], G.dxi[2], G.plof[2], G.dxif[2], 1, G.n[2]);
        const int c = column_of(G, bx, by);
        ucol[u] = c;
        uiz[u] = bz;
        atomicAdd(&S.colcnt[c], 1);
    }
}

// counting sort of the caller's particles into the columns (arrival order
// from the atomics): each particle's (z bin, caller index) key at the
// position it drew
__global__ void k_user_scatter(const DevState S, const int *ucol, const int *uiz, const int *colstart)
{
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < S.n; u += gridDim.x * blockDim.x) {
        const int c = ucol[u];
        const int r = atomicSub(&S.colcnt[c], 1) - 1;
        if (r == kLongColumn) S.cnt->long_column = 1ull;
        const int t = colstart[c] + r;
        if (t >= 0 && t < S.n) S.lkey[t] = col_key(uiz[u], u);
        else atomicAdd(&S.cnt->bad_index, 1ULL);
    }
}

__global__ void k_gather_d(double *dst, const double *src, const int *perm, int n, int planes)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const int u = perm[s];
        for (int k = 0; k < planes; ++k) dst[(size_t)k * n + s] = src[(size_t)k * n + u];
    }
}

__global__ void k_scatter_d(double *dst, const double *src, const int *orig, int n, int planes)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const int u = orig[s];
        for (int k = 0; k < planes; ++k) dst[(size_t)k * n + u] = src[(size_t)k * n + s];
    }
}

__global__ void k_scatter_f2d(double *dst, const float *src, const int *orig, int n)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x)
        dst[orig[s]] = (double)src[s];
}

// Neighbour list of every slot in the reference's order; indices and counts
// are in caller order.  Only pairs passing BMXCheckPair (|r|^2 <= neighborhood,
// evaluated in FP64 on the image positions) are listed.
__global__ void k_pairs(const DevState S, const DevParams P, int a, int64_t *cnt_or_offs, int *idx,
                        int8_t *img, int mode)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n; i += gridDim.x * blockDim.x) {
        const DevGeom &G = geom_of(S, i);
        int bx, by;
        col_to_bxy(G, S.col[a][i], bx, by);
        const double xi = S.x[a][i], yi = S.y[a][i], zi = S.z[a][i];
        int64_t o = (mode == 1) ? cnt_or_offs[S.orig[i]] : 0;
        int64_t c = 0;
        visit_stencil(S, G, a, i, bx, by, S.iz[a][i], [&](int j, int, int, int, int sx, int sy) {
            const double xj = sx ? S.x[a][j] + (double)sx * G.len[0] : S.x[a][j];
            const double yj = sy ? S.y[a][j] + (double)sy * G.len[1] : S.y[a][j];
            const double dx = xi - xj, dy = yi - yj, dz = zi - S.z[a][j];
            const double r2 = dx * dx + dy * dy + dz * dz;
            if (r2 <= P.nbh) {
                if (mode == 1) {
                    idx[o] = S.orig[j];
                    img[o] = (int8_t)((sx + 1) + 3 * (sy + 1));
                    ++o;
                }
                ++c;
            }
        });
        if (mode == 0) cnt_or_offs[S.orig[i]] = c;
    }
}

// Checks of a caller's state before it is loaded: cell types outside
// {YEAST, FUNGI}, whether any FUNGI segment is present, the largest radius
// (non-negative doubles order as their bit patterns) and whether any radius
// is NaN.  out: {bad, fungi, rmax bits, nan}, zeroed by the caller.
struct StateFlags {
    unsigned bad = 0, fungi = 0, nan = 0;
    unsigned long long rmax = 0;
    __device__ __forceinline__ void see(int ct, double r)
    {
        bad |= ((unsigned)ct > 1u) ? 1u : 0u;
        fungi |= (ct == 1) ? 1u : 0u;
        nan |= (r != r) ? 1u : 0u;
        if (r > 0.0) rmax = max(rmax, (unsigned long long)__double_as_longlong(r));
    }
    // (every thread of the block; one atomic of each a block)
    __device__ __forceinline__ void publish(unsigned long long *out)
    {
        __shared__ unsigned long long most[32];
        __shared__ unsigned flags[32];
        const unsigned all = __reduce_or_sync(0xffffffffu, bad | (fungi << 1) | (nan << 2));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) rmax = max(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
        if ((threadIdx.x & 31) == 0) {
            most[threadIdx.x >> 5] = rmax;
            flags[threadIdx.x >> 5] = all;
        }
        __syncthreads();
        if (threadIdx.x) return;
        unsigned f = all;
        for (int v = 1; v < (int)(blockDim.x >> 5); ++v) {
            rmax = max(rmax, most[v]);
            f |= flags[v];
        }
        if (f & 1u) atomicOr(&out[0], 1ull);
        if (f & 2u) atomicOr(&out[1], 1ull);
        if (rmax > *static_cast<volatile unsigned long long *>(&out[2])) atomicMax(&out[2], rmax);
        if (f & 4u) atomicOr(&out[3], 1ull);
    }
};

// Whether a load repeats the device state bit for bit: each slot's position
// (buffer a), radius and cell type against the caller's arrays at its caller
// index.  *diff becomes nonzero on the first difference.  chk (with r and ct; may be
// null): the checks of those as well, in the same pass (in one of their own before it
// the load of an unchanged state of 300 000 spheres took 168 us, 152 without).
__global__ void k_same_state(const DevState S, int a, const double *__restrict__ x, const double *__restrict__ y,
                             const double *__restrict__ z, const double *__restrict__ r, const int *__restrict__ ct,
                             unsigned long long *diff, unsigned long long *chk)
{
    unsigned d = 0;
    StateFlags f;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < S.n; s += gridDim.x * blockDim.x) {
        const int i = S.orig[s];
        if ((unsigned)i >= (unsigned)S.n) {
            d = 1u;
            continue;
        }
        // (a null field is not compared: a load compares each field as its copy lands)
        if (x) d |= (__double_as_longlong(x[i]) != __double_as_longlong(S.x[a][s])) ? 1u : 0u;
        if (y) d |= (__double_as_longlong(y[i]) != __double_as_longlong(S.y[a][s])) ? 1u : 0u;
        if (z) d |= (__double_as_longlong(z[i]) != __double_as_longlong(S.z[a][s])) ? 1u : 0u;
        if (r) d |= (__double_as_longlong(r[i]) != __double_as_longlong(S.rad[s])) ? 1u : 0u;
        if (ct) d |= (ct[i] != (int)S.ctype[s]) ? 1u : 0u;
        if (chk) f.see(ct[i], r[i]);
    }
    if (chk) f.publish(chk);
    d = __reduce_or_sync(0xffffffffu, d);
    if ((threadIdx.x & 31) == 0 && d) atomicOr(diff, 1ull);
}

__global__ void k_check_state(const int *__restrict__ ct, const double *__restrict__ r, int n,
                              unsigned long long *out)
{
    StateFlags f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) f.see(ct[i], r[i]);
    f.publish(out);
}

// Caller particle u's slot: its column's start + its rank among the
// column's keys (z bin, then caller index): uperm[slot] = u.
__global__ void k_user_canon(const DevState S, const int *ucol, const int *uiz, const int *colstart, int *uperm)
{
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < S.n; u += gridDim.x * blockDim.x) {
        const int c = ucol[u];
        const int s0 = max(colstart[c], 0), s1 = min(colstart[c + 1], S.n);
        const unsigned long long key = col_key(uiz[u], u);
        int rank = 0;
        for (int t = s0; t < s1; ++t) rank += (__ldg(&S.lkey[t]) < key);
        if (s0 + rank < s1) uperm[s0 + rank] = u;
        else atomicAdd(&S.cnt->bad_index, 1ULL);
    }
}

// Slot s of a freshly sorted state holds caller particle uperm[s]: its
// position, radius and cell type are gathered from the caller-order arrays,
// its bins are the caller-order bins of the sort, its column order is the
// sort's (perm = identity, colstart = the sort's offsets, copied by the
// caller), and its offsets and counters are place_slot's.  Velocities the caller
// gives are gathered, the others zero.
struct VelSrc {
    const double *v[6];
};

__global__ void k_load_slots(const DevState S, const double *ux, const double *uy, const double *uz,
                             const double *ur, const int *uct, const VelSrc V, const int *ucol, const int *uiz,
                             const int *uperm)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < S.n; s += gridDim.x * blockDim.x) {
        const DevGeom &G = geom_of(S, s);
        const int u = uperm[s];
        const double x = ux[u], y = uy[u], z = uz[u], r = ur[u];
        S.x[0][s] = x;
        S.y[0][s] = y;
        S.z[0][s] = z;
        S.rad[s] = r;
        S.ctype[s] = (int8_t)uct[u];
        S.orig[s] = u;
        S.vx[s] = V.v[0] ? V.v[0][u] : 0.0;
        S.vy[s] = V.v[1] ? V.v[1][u] : 0.0;
        S.vz[s] = V.v[2] ? V.v[2][u] : 0.0;
        S.wx[s] = V.v[3] ? V.v[3][u] : 0.0;
        S.wy[s] = V.v[4] ? V.v[4][u] : 0.0;
        S.wz[s] = V.v[5] ? V.v[5][u] : 0.0;
        int bx, by;
        col_to_bxy(G, ucol[u], bx, by);
        const int bz = uiz[u];
        place_slot(S, G, s, x, y, z, r, 0, 0, bx, by, bz, true, false);
        S.perm[0][s] = s;
        if (S.srel[0]) {
            S.srel[0][s] = S.rel[0][s];
            S.siz[0][s] = bz;
            S.rank[0][s] = s;
        }
    }
}

}  // namespace

int launch_load_slots(const DevState &S, const double *ux, const double *uy, const double *uz, const double *ur,
                      const int *uct, const double *const v[6], const int *ucol, const int *uiz, const int *uperm,
                      int grid, int block, cudaStream_t st)
{
    const VelSrc V{{v[0], v[1], v[2], v[3], v[4], v[5]}};
    k_load_slots<<<grid, block, 0, st>>>(S, ux, uy, uz, ur, uct, V, ucol, uiz, uperm);
    return 1;
}

int launch_check_state(const int *ct, const double *r, int n, unsigned long long *out, int grid, int block,
                       cudaStream_t st)
{
    k_check_state<<<grid, block, 0, st>>>(ct, r, n, out);
    return 1;
}

int launch_same_state(const DevState &S, int a, const double *x, const double *y, const double *z, const double *r,
                      const int *ct, unsigned long long *diff, unsigned long long *chk, int grid, int block,
                      cudaStream_t st)
{
    k_same_state<<<grid, block, 0, st>>>(S, a, x, y, z, r, ct, diff, chk);
    return 1;
}

int launch_bin(const DevState &S, int b, int grid, int block, cudaStream_t st)
{
    k_bin<<<grid, block, 0, st>>>(S, b);
    return 1;
}

size_t scan_scratch_ints(int n)
{
    return (size_t)((n + kScanTile - 1) / kScanTile) + 2;
}

int launch_scan(const int *in, int *out, int n, int *scratch, cudaStream_t st, const int *gate)
{
    const int nb = (n + kScanTile - 1) / kScanTile;
    if (nb == 0) {
        cudaMemsetAsync(out, 0, sizeof(int), st);
        return 0;
    }
    k_scan_reduce<<<nb, kScanBlock, 0, st>>>(in, n, scratch, gate);
    k_scan_top<<<1, kTopBlock, 0, st>>>(scratch, nb, gate);
    k_scan_apply<<<nb, kScanBlock, 0, st>>>(in, n, scratch, out, gate);
    return 3;
}

// Whether the current device takes the sort's cluster, looked up once per device.
static bool sort_cluster_fits()
{
    static std::atomic<int> known[64];  // 0: not looked up yet, 1: no, 2: yes
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    int v = known[dev].load(std::memory_order_relaxed);
    if (v) return v == 2;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)kSortCluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)kSortCluster);
    cfg.blockDim = dim3(kSortBlock);
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int fit = 0;
    const bool yes = cudaFuncSetAttribute(k_sort_cluster<false>, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                          1) == cudaSuccess &&
                     cudaOccupancyMaxActiveClusters(&fit, k_sort_cluster<false>, &cfg) == cudaSuccess && fit > 0 &&
                     cudaFuncSetAttribute(k_sort_cluster<true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                         cudaSuccess &&
                     cudaOccupancyMaxActiveClusters(&fit, k_sort_cluster<true>, &cfg) == cudaSuccess && fit > 0;
    if (!yes) (void)cudaGetLastError();
    known[dev].store(yes ? 2 : 1, std::memory_order_relaxed);
    return yes;
}

// Runs the job in one cluster where it fits (J.lkey set); false: the caller's
// separate kernels.
static bool sort_in_cluster(const SortJob &J, bool long_cols, cudaStream_t st)
{
    constexpr int T = kSortCluster * kSortBlock;
    if (!J.lkey || J.n > T * kSortItems || J.ncols > T * kSortCols || !sort_cluster_fits()) return false;
    // no more blocks than the slots and columns fill
    int use = kSortCluster;
    while (use > 1 && J.n <= (use / 2) * kSortBlock && J.ncols <= (use / 2) * kSortBlock * 4) use /= 2;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)use;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // (launch_after)
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)use);
    cfg.blockDim = dim3(kSortBlock);
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, long_cols ? k_sort_cluster<true> : k_sort_cluster<false>, J);  // (an error is the launch status the caller reads)
    return true;
}

int launch_rebuild(const DevState &S, int b, int *scan_scratch, int grid, int block, cudaStream_t st, bool publish)
{
    const SortJob J{S.n,       S.ncols_total, S.col[b], S.iz[b],  S.orig, S.colcnt, S.colstart[b],  S.lkey, S.perm[b],
                    S.rel[b],  S.srel[b],     S.siz[b], S.rank[b], S.cnt, S.rctl,   publish ? 1 : 0};
    if (sort_in_cluster(J, S.long_cols, st)) return 1;
    const int k = launch_scan(S.colcnt, S.colstart[b], S.ncols_total, scan_scratch, st);
    k_scatter<<<grid, block, 0, st>>>(S, b);
    const bool runs = S.lkey && S.long_cols;
    if (runs)
        k_sort_runs<<<dim3(S.ncols_total, std::max(1, std::min(64, S.n / S.ncols_total / (2 * kRun)))), 256, 0, st>>>(S, b);
    k_canon<<<grid, block, 0, st>>>(S, b, publish ? 1 : 0, runs ? 1 : 0);
    return k + 2 + (runs ? 1 : 0);
}

int launch_user_bin(const DevState &S, const double *ux, const double *uy, const double *uz, int *ucol,
                     int *uiz, int grid, int block, cudaStream_t st)
{
    k_user_bin<<<grid, block, 0, st>>>(S, ux, uy, uz, ucol, uiz);
    return 1;
}

int launch_user_sort(const DevState &S, const int *ucol, const int *uiz, int *colstart, int *scan_scratch,
                     int *uperm, int grid, int block, cudaStream_t st)
{
    const SortJob J{S.n,     S.ncols_total, ucol,    uiz,     nullptr, S.colcnt, colstart, S.lkey, uperm,
                    nullptr, nullptr,       nullptr, nullptr, S.cnt,   nullptr,  0};
    // (what this sort will find out the last load of the size or the average says for now;
    // above 32 768 slots a long column that neither shows costs more than looking out for it)
    const bool runs = S.long_cols || S.n > 32768 || S.n / std::max(S.ncols_total, 1) > kLongColumn;
    if (sort_in_cluster(J, runs, st)) return 1;
    const int k = launch_scan(S.colcnt, colstart, S.ncols_total, scan_scratch, st);
    k_user_scatter<<<grid, block, 0, st>>>(S, ucol, uiz, colstart);
    k_user_canon<<<grid, block, 0, st>>>(S, ucol, uiz, colstart, uperm);
    return k + 2;
}

int launch_gather_d(double *dst, const double *src, const int *perm, int n, int grid, int block, cudaStream_t st,
                    int planes)
{
    k_gather_d<<<grid, block, 0, st>>>(dst, src, perm, n, planes);
    return 1;
}

int launch_scatter_d(double *dst, const double *src, const int *orig, int n, int grid, int block, cudaStream_t st,
                     int planes)
{
    k_scatter_d<<<grid, block, 0, st>>>(dst, src, orig, n, planes);
    return 1;
}

int launch_scatter_f2d(double *dst, const float *src, const int *orig, int n, int grid, int block,
                       cudaStream_t st)
{
    k_scatter_f2d<<<grid, block, 0, st>>>(dst, src, orig, n);
    return 1;
}

int launch_pairs(const DevState &S, const DevParams &P, int a, int64_t *cnt_or_offs, int *idx, int8_t *img,
                  int mode, int grid, int block, cudaStream_t st)
{
    k_pairs<<<grid, block, 0, st>>>(S, P, a, cnt_or_offs, idx, img, mode);
    return 1;
}

}  // namespace bmxg
