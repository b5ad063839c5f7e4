// k_list.cu -- sphere steps over a neighbour list with a skin: the FP32F form, and
// FP64 steps on the same list (k_list64_step).
//
// The force acts only on pairs closer than rA = r_i + r_j + bw
// (maxInteractionDistance and the gate r^2 <= (r_lm - 1e-15)^2,
// bmx_cell_interaction_K.H:23-40, bmx_pc_interaction.cpp:212).  When the
// largest rA is at most the smallest bin width, any pair that close sits in
// neighbouring bins, so the reference's stencil list holds it whatever the
// binning is.  The list built here holds every pair closer than rA + skin
// at build time; while no pair's separation has changed by the skin since,
// it still holds every pair closer than rA.  The pair set of a step is
// therefore the reference's; only the FP32 rounding of the pair math (the
// precision form) differs from it.
//
// State: while the list path runs, positions live in 64-bit fixed point
// (FxGeom: one unit is span / 2^64, 7e-21 cm on a 0.128 cm box, finer than
// the FP64 ulp anywhere above 2^-9 cm) as a 16-byte record per slot (the high
// 32 bits of x, y, z and the FP32 radius) and three 32-bit low words.  A
// step reads and writes those 28 bytes, reads the list and writes the FP32
// velocity; a neighbour's offset is the int32 difference of two high words
// (exact; the minimum periodic image by the unsigned wrap), converted once to
// FP32 -- one 16-byte gather per neighbour, the same line its owner reads.
// The FP32 increment, scaled to units to 2^-44 of itself, is added exactly:
// no rounding accumulates in the positions, and no FP64 instruction runs
// (GB300 issues FP64 at 1/64 of the FP32 rate).  The FP64 positions are converted from the
// fixed point whenever anything reads them (launch_list_to_fp64), and to it
// when the list path starts.
// k_list_decide bounds the separation change of every pair from the spread
// of each step's increments and asks for a build when the bound reaches the
// skin (or after max_age steps); inside a CUDA graph the build kernels sit
// in a conditional node that the decision switches, so a step without a
// build launches two kernels.
//
// Build: bins from the high words (integer arithmetic, consistent with the
// positions), a counting sort into the x-y columns, the in-column order by z
// bin and caller index (deterministic lists and FP32 summation order), the 3D
// cells' offsets from the sorted z bins, and the stencil walk that keeps
// every candidate within rA + skin on exact fixed-point differences.
//
// Roofline: the step kernel streams 28 bytes of position state in and out,
// the list in and the FP32 velocity out; the neighbour records it gathers
// are L2-resident.  HBM bound, no contraction.
#include <algorithm>

#include "bmxg_fx.cuh"
#include "bmxg_pdl.cuh"
#include "bmxg_stencil.cuh"

namespace bmxg {

namespace {

// Order-preserving unsigned key of a float (and back): atomicMin / atomicMax
// on the keys order the floats.
__device__ __forceinline__ unsigned fkey(float f)
{
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ __forceinline__ float funkey(unsigned k)
{
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

constexpr unsigned kKeyPosInf = 0xff800000u;  // fkey(+inf)
constexpr unsigned kKeyNegInf = 0x007fffffu;  // fkey(-inf)

// An FP32 increment f in fixed-point units, f 2^64 / span, with the constant
// as an FP32 pair c + cl (2^-48 of it): p = f c rounded, its exact error from
// an FMA, plus f cl; each part rounded to the nearest unit.  Within 2^-44 of
// the increment (and a few units: ~1e-19 cm on a 0.128 cm box), far below
// the FP64 position's own rounding; the sum into the position is exact, so
// no rounding accumulates however small the increment is against the
// position.  An increment of a quarter span or more (or a non-finite one)
// sets `big`.
__device__ __forceinline__ long long fx_inc(float f, float c, float cl, bool &big)
{
    const float p = __fmul_rn(f, c);
    if (!(fabsf(p) < 4.6116860184273879e18f)) {  // 2^62
        big = true;
        return 0ll;
    }
    const float r = __fmaf_rn(f, cl, __fmaf_rn(f, c, -p));
    // the remainder (|r| <= 2^-24 |p| + |f cl| < 2^31 below |p| = 2^54) converted
    // to a 32-bit integer: the same value, one 64-bit conversion (an FP64-pipe
    // instruction on GB300) fewer
    if (fabsf(p) < 1.8014398509481984e16f) return __float2ll_rn(p) + (long long)__float2int_rn(r);  // 2^54
    return __float2ll_rn(p) + __float2ll_rn(r);
}

// The common case of fx_inc, |p| = |f c| < 2^54.
__device__ __forceinline__ long long fx_inc_small(float f, float c, float cl, float p)
{
    return __float2ll_rn(p) + (long long)__float2int_rn(__fmaf_rn(f, cl, __fmaf_rn(f, c, -p)));
}

// The bound: for any pair, the separation change since the build is, per
// component, at most the sum over steps of the spread (largest minus
// smallest) of that step's increments; its length at most the length of
// those sums.  Unlike twice the largest displacement, it does not count a
// drift common to all slots (here: the rise of the slots below the growth
// surface).  Each step adds eps_step per component for the FP32 rounding of
// the pair offsets the gate sees.
// It also clears the per-step counters (no memset nodes in the step), counts
// the call's steps down and names the buffer the step reads, so that steps can
// be enqueued without knowing which of them will run: see kDecideStall.
__global__ void k_list_decide(ListCtl *c, DevCounters *cnt, cudaGraphConditionalHandle h, int mode)
{
    chain_wait();
    if (mode == kDecideOne) c->left += 1;
    bool run = c->left > 0 && !c->bail && !(c->whole && c->overflow);
    bool rb = false;
    if (run) {
        bool need = c->need != 0;
        if (!need) {
            float r2 = 0.0f;
            float rg[3];
            for (int k = 0; k < 3; ++k) {
                const unsigned lo = c->inc_min[k], hi = c->inc_max[k];
                // no slot reported (empty state): no spread
                const float spread = (hi >= lo) ? (funkey(hi) - funkey(lo)) : 0.0f;
                rg[k] = c->range[k] + spread * 1.000001f + c->eps_step;
                r2 += rg[k] * rg[k];
                c->inc_min[k] = kKeyPosInf;
                c->inc_max[k] = kKeyNegInf;
                c->range[k] = rg[k];
            }
            const float acc = sqrtf(r2);
            const int age = c->age + 1;
            need = c->force != 0 || !(acc <= c->skin) || age > c->max_age;
            c->acc = acc;
            c->age = age;
        }
        if (need && mode != kDecideStall) {
            rb = true;
            need = false;
            for (int k = 0; k < 3; ++k) c->range[k] = 0.0f;
            c->acc = 0.0f;
            c->age = 0;
            c->force = 0;
            c->builds += 1;
            c->overflow = 0ull;
        }
        c->need = need ? 1 : 0;
        run = !need;
        if (run) {
            cnt->out_of_domain = 0ull;
            cnt->edge_ghost = 0ull;
            cnt->pairs = 0ull;
            cnt->bond_repairs = 0ull;
            cnt->moved = 0ull;
            c->left -= 1;
            const int par = c->par;
            c->cur = par;
            c->par = par ^ 1;
        }
    }
    c->active = run ? 1 : 0;
    c->rebuild = rb ? 1 : 0;
    if (mode == kDecideCond || mode == kDecideOne) cudaGraphSetConditional(h, rb ? 1u : 0u);
}

// Colony of index i for a kernel whose blocks take consecutive indices, one
// per thread: one binary search per block (the colonies of a block's range
// are few), then each thread steps forward.  Slot order and the list's sorted
// order hold the colonies in the same ranges (a colony's particles stay
// together under the sort), so either index works.  Every thread of the
// block must call it (it synchronises the block).
__device__ __forceinline__ int block_colony(const DevState &S, int i)
{
    __shared__ int c0;
    if (threadIdx.x == 0) c0 = colony_of(S.cbase, S.ncol, min((int)(blockIdx.x * blockDim.x), S.n - 1));
    __syncthreads();
    int c = c0;
    while (c + 1 < S.ncol && __ldg(&S.cbase[c + 1]) <= i) ++c;
    return c;
}

// Bin of a high word: a periodic axis spans the domain (bin = h n / 2^32);
// a closed axis has the domain in [2^30, 2^31), clamped to 1..n.
__device__ __forceinline__ int fx_bin(unsigned h, int nb, int per)
{
    if (per) return (int)__umulhi(h, (unsigned)nb) + 1;
    const long long d = (long long)h - (1ll << 30);
    if (d < 0) return 1;
    const long long b = (d * nb) >> 30;
    return (b >= nb) ? nb : (int)b + 1;
}

// Bins of the step's fixed-point positions (buffer lctl->cur) into the list bins (kListBins
// buffer) and the column counts.
__global__ void k_list_rebin(const DevState S)
{
    if (!S.lctl->rebuild) return;
    const int a = S.lctl->cur;
    constexpr int B = kListBins;
    if (blockIdx.x == 0 && threadIdx.x == 0) S.lctl->body_runs += 1ull;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int col = block_colony(S, i);
    if (i < S.n) {
        const DevGeom &G = S.geoms[col];
        const FxGeom &F = S.fxg[col];
        const int4 h = S.fxh[a][i];
        const int bx = fx_bin((unsigned)h.x, F.n[0], F.per[0]);
        const int by = fx_bin((unsigned)h.y, F.n[1], F.per[1]);
        const int bz = fx_bin((unsigned)h.z, F.n[2], F.per[2]);
        const int c = column_of(G, bx, by);
        S.col[B][i] = c;
        S.iz[B][i] = bz;
        atomicAdd(&S.colcnt[c], 1);
    }
}

// The order key of a slot inside its column: z bin, then caller index (the
// sorted order is column, z bin, caller index, as the 3D cells hold it).
__device__ __forceinline__ unsigned long long list_key(int bz, int orig)
{
    return ((unsigned long long)(unsigned)bz << 32) | (unsigned)orig;
}

// counting sort into the columns (arrival order from the atomics): each slot's
// key at the position it drew
__global__ void k_list_scatter(const DevState S)
{
    if (!S.lctl->rebuild) return;
    constexpr int B = kListBins;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < S.n) {
        const int c = S.col[B][i];
        const int r = atomicSub(&S.colcnt[c], 1) - 1;  // leaves colcnt at zero
        const int t = S.colstart[B][c] + r;
        if (t >= 0 && t < S.n) S.lkey[t] = list_key(S.iz[B][i], S.orig[i]);
        else atomicAdd(&S.cnt->bad_index, 1ULL);
    }
}

// deterministic order inside a column (z bin, then ascending original index:
// the slot's rank among its column's keys), and the sorted copies the build
// walks: the position record, z bin, slot, and each slot's rank
__global__ void k_list_canon(const DevState S)
{
    if (!S.lctl->rebuild) return;
    const int a = S.lctl->cur;
    constexpr int B = kListBins;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < S.n) {
        const int c = S.col[B][i];
        const int bz = S.iz[B][i];
        const int s0 = max(S.colstart[B][c], 0), s1 = min(S.colstart[B][c + 1], S.n);
        const unsigned long long me = list_key(bz, S.orig[i]);
        int rank = 0;
        for (int t = s0; t < s1; ++t) rank += (__ldg(&S.lkey[t]) < me);
        const int t = s0 + rank;
        if (t >= s1) {  // i is not among its column's members: inconsistent counts
            atomicAdd(&S.cnt->bad_index, 1ULL);
        } else {
            S.perm[B][t] = i;
            reinterpret_cast<int4 *>(S.srel[B])[t] = S.fxh[a][i];
            S.siz[B][t] = bz;
            S.rank[B][i] = t;
        }
        if ((i & 31) == 0) S.xcnt[i >> 5] = 0;  // the build adds up each group's entries
    }
}

// The 3D cells' offsets in the sorted copies from the columns' sorted z bins:
// cell (column, z) starts at the column's first position whose z bin is z or
// more.  One thread per column of the colony blockIdx.x (kCellsBlock columns
// per block, blocks strided over blockIdx.y) walks its column's members once
// and leaves the offsets of kCellsZ z bins at a time in shared memory; the
// block then writes its columns' cells, which lie together, in whole rows.
// The last entry (one past the last cell) is n.
constexpr int kCellsBlock = 128;
constexpr int kCellsZ = 32;  // one z bin per lane in the write-out

__global__ void __launch_bounds__(kCellsBlock) k_list_cells(const DevState S)
{
    if (!S.lctl->rebuild) return;
    constexpr int B = kListBins;
    constexpr int R = kCellsZ + 1;  // row pitch (no bank conflicts between the columns' rows)
    __shared__ int off[kCellsBlock * R];
    const DevGeom &G = S.geoms[blockIdx.x];
    const int nz = G.n[2];
    const int ncols = G.n[0] * G.n[1];
    for (int q0 = blockIdx.y * kCellsBlock; q0 < ncols; q0 += gridDim.y * kCellsBlock) {  // same trip count
        const int q = q0 + threadIdx.x;
        const int nq = min(kCellsBlock, ncols - q0);
        // t: the column's first position whose z bin (v; past the column's
        // end: above every bin) is not below the current z
        int t = 0, s1 = 0;
        if (q < ncols) {
            t = max(__ldg(&S.colstart[B][G.col_base + q]), 0);
            s1 = min(__ldg(&S.colstart[B][G.col_base + q + 1]), S.n);
        }
        int v = (t < s1) ? __ldg(&S.siz[B][t]) : 0x7fffffff;
        for (int zc = 0; zc < nz; zc += kCellsZ) {
            const int zl = min(kCellsZ, nz - zc);
            if (q < ncols) {
                for (int k = 0; k < zl; ++k) {
                    const int z = zc + k + 1;
                    while (v < z) {
                        ++t;
                        v = (t < s1) ? __ldg(&S.siz[B][t]) : 0x7fffffff;
                    }
                    off[threadIdx.x * R + k] = t;
                }
            }
            __syncthreads();
            // the block's cells of this z range: a warp writes one column's zl
            // cells at a time, lane k the k-th (a whole row; the columns' rows
            // lie one after another when nz <= kCellsZ)
            const int lane = threadIdx.x & 31;
            int *dst = S.cellstart + G.cell_base + (size_t)q0 * nz + zc;
            if (lane < zl)
                for (int cq = threadIdx.x >> 5; cq < nq; cq += kCellsBlock / 32)
                    dst[(size_t)cq * nz + lane] = off[cq * R + lane];
            __syncthreads();
        }
    }
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) S.cellstart[S.ncells_total] = S.n;
}

// Visit the slots of the 3 x 3 neighbour columns of bin (bx, by), z bins
// izi - 1 .. izi + 1 (periodic images included), as contiguous cell ranges
// of the sorted copies: f(u) for each sorted position u but the slot's own
// self_t (SKIP_SELF; otherwise f sees it too and excludes it itself).  Order:
// x rows outermost, then y, then z, ascending caller index within a cell.
template <bool SKIP_SELF = true, class F>
__device__ __forceinline__ void visit_cells(const DevState &S, const DevGeom &G, int self_t, int bx, int by, int izi,
                                            F &&f)
{
    const int *__restrict__ cs = S.cellstart;
    const int nz = G.n[2];
    const int z0 = max(izi - 1, 1), z1 = min(izi + 1, nz);
    for (int dxs = -1; dxs <= 1; ++dxs) {
        int sx = bx + dxs;
        if (sx < 1 || sx > G.n[0]) {
            if (!G.per[0]) continue;
            sx += (sx < 1) ? G.n[0] : -G.n[0];
        }
        for (int dys = -1; dys <= 1; ++dys) {
            int sy = by + dys;
            if (sy < 1 || sy > G.n[1]) {
                if (!G.per[1]) continue;
                sy += (sy < 1) ? G.n[1] : -G.n[1];
            }
            const int cb = G.cell_base + ((sx - 1) * G.n[1] + (sy - 1)) * nz;
            const int hi = __ldg(&cs[cb + z1]);
            for (int u = __ldg(&cs[cb + z0 - 1]); u < hi; ++u) {
                if (SKIP_SELF && u == self_t) continue;
                f(u);
            }
        }
    }
}

// Entries of slot i's list past the inline ones that the step takes from
// the compacted list (none for a slot whose list overflowed: it walks).
__device__ __forceinline__ int list_extra(int cnt)
{
    return (cnt > kNbrInline && cnt <= kNbrCap) ? cnt - kNbrInline : 0;
}

// List build: every slot (in sorted order, so a warp's lanes share cells)
// keeps the neighbours closer than rA + skin on the exact fixed-point
// differences of the high words (+ a slack of four units per component and
// the FP32 rounding of the test), and its list length.  The rounding margin:
// the offsets' unit factors are scaled by 1 - 1e-6 (r^2 by 1 - 2e-6), against
// at most ~4e-7 of relative FP32 rounding in r^2 and in the bound squared;
// the slot's own record passes the test (distance 0) and is dropped after it.
__global__ void __launch_bounds__(256, 6) k_list_build(const DevState S, const DevParams P)
{
    if (!S.lctl->rebuild) return;
    constexpr int B = kListBins;
    const int n = S.n;
    const float reach = P.bw32 + S.lctl->skin;
    const int4 *__restrict__ sg = reinterpret_cast<const int4 *>(S.srel[B]);
    unsigned long long over = 0;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int col = block_colony(S, t);  // the sorted order keeps the colonies' ranges
    if (t < n) {
        const int i = S.perm[B][t];
        const DevGeom &G = S.geoms[col];
        const FxGeom &F = S.fxg[col];
        int bx, by;
        col_to_bxy(G, S.col[B][i], bx, by);
        const int izi = S.siz[B][t];
        const int4 me = sg[t];
        const float ri = __int_as_float(me.w);
        const float ci = ri + (reach + 4.0f * (F.uh[0] + F.uh[1] + F.uh[2]));  // the bound less r_j
        const float ux = F.uh[0] * 0.999999f, uy = F.uh[1] * 0.999999f, uz = F.uh[2] * 0.999999f;
        int c = 0;
        int4 rec = make_int4(0, 0, 0, 0);
        visit_cells<false>(S, G, t, bx, by, izi, [&](int s) {
            const int4 q = __ldg(&sg[s]);
            const float ex = (float)(me.x - q.x) * ux;
            const float ey = (float)(me.y - q.y) * uy;
            const float ez = (float)(me.z - q.z) * uz;
            const float r2f = __fmaf_rn(ex, ex, __fmaf_rn(ey, ey, __fmul_rn(ez, ez)));
            const float lim = __int_as_float(q.w) + ci;
            if (!(r2f <= lim * lim) || s == t) return;
            const int e = __ldg(&S.perm[B][s]);
            if (c == 0) rec.y = e;
            else if (c == 1) rec.z = e;
            else if (c == 2) rec.w = e;
            else if (c < kNbrCap) S.nbr[(size_t)(c - kNbrInline) * n + i] = e;
            ++c;
        });
        rec.x = min(c, 255);
        S.lrec[i] = rec;
        if (c > kNbrCap) ++over;
        const int x = list_extra(rec.x);  // its group's count of entries past the inline ones
        if (x) atomicAdd(&S.xcnt[i >> 5], x);
    }
    if (over) atomicAdd(&S.lctl->overflow, over);
}

// Gated pairs of a step, recorded when the context asks (S.pcap): per slot,
// the count and the neighbour slots the step accumulated, in its order.
struct PairRec {
    int *cap;
    int i, k;
    __device__ __forceinline__ void add(int j)
    {
        if (cap && k < kPairCap) cap[(size_t)i * (kPairCap + 1) + 1 + k] = j;
        ++k;
    }
    __device__ __forceinline__ void done()
    {
        if (cap) cap[(size_t)i * (kPairCap + 1)] = k;
    }
};

// Compaction of the list entries past the inline ones, per group of 32
// consecutive slots (the step's warps): the groups' counts (added up by
// k_list_build into counts that k_list_canon zeroed), then (after their
// exclusive scan into xoff) each slot's entries copied from the build's
// planes to xlist[xoff[group] + the entries of the group's earlier slots].
// One slot per thread, whole warps.

__global__ void k_list_xcopy(const DevState S)
{
    if (!S.lctl->rebuild) return;
    const int n = S.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int x = (i < n) ? list_extra(S.lrec[i].x & 0xff) : 0;
    int o = x;  // inclusive scan over the warp
    for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, o, d);
        if (lane >= d) o += v;
    }
    if (x) {
        int *dst = S.xlist + __ldg(&S.xoff[i >> 5]) + (o - x);
        for (int k = 0; k < x; ++k) dst[k] = __ldg(&S.nbr[(size_t)k * n + i]);
    }
    // the slot's place in its group's run beside the list length (bits 8-17:
    // at most 31 x 29 entries precede it)
    if (i < n) S.lrec[i].x = (S.lrec[i].x & 0xff) | ((o - x) << 8);
}

// FP32F sphere step over the list: pair offsets from the fixed-point high
// words, pair math and wall law in FP32, the increments added in 64-bit fixed
// point (the periodic wrap is the unsigned wrap; the domain test of the
// closed z axis compares the high word).
// Each block takes a contiguous chunk of slots (a multiple of 32), so a
// thread's colony is found by one binary search and then by stepping forward
// from the last one.  The list metadata and the first entries come in one
// 16-byte record; the rest (a slot's list is mostly 0 to 3 long, rarely up to
// a dozen) from the compacted list, where a warp's entries lie together: a
// few sectors per warp, not one per entry as a plane per list position would
// cost.
// Bound: instruction issue (60 % of the slots) and the loads' latency, at 2.5 TB/s of
// HBM traffic.  What it measured on 2.75 million slots in 256 colonies: 84 us a step
// with the colony searched before the first loads, the low words' loads met after the
// pairs, the tail of a list one entry at a time and the range test per increment; 80
// with the loads first and the low words on their way into L2 (in registers: 86), 77
// with the tail in fours, 73 with one range test.  Five blocks of 256 instead of six
// (no spill): 81; eight (32 registers): 83.
template <bool CAP, bool PERSIST>
__global__ void __launch_bounds__(256, 6) k_list_step(const DevState S, const DevParams P, float dtf, int chunk)
{
    chain_wait();
    if (!S.lctl->active) return;  // (a stalled step, or one past the call's last)
    constexpr int B = kListBins;
    const int a = S.lctl->cur, b = a ^ 1;
    const int n = S.n;
    const float bwf = P.bw32, kf = P.k32;
    const float zkf = P.z_k32, zbwf = P.z_bw32, zgf = P.z_g32;
    const int4 *__restrict__ ga = S.fxh[a];
    const unsigned *__restrict__ la = S.fxl[a];
    // smallest and largest increment per component (order-preserving keys),
    // per warp in shared memory: reduced over the warp after each pass, so
    // that no register holds them through the list walk
    __shared__ unsigned wmin[32][3], wmax[32][3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane < 3) {
        wmin[w][lane] = kKeyPosInf;
        wmax[w][lane] = kKeyNegInf;
    }
    __syncwarp();
    // the chunks of consecutive slots this block takes: its own, or (persistent)
    // the next from the dispenser until none is left
    __shared__ int s_chunk;
    const int nchunks = (n + chunk - 1) / chunk;
    int ck = blockIdx.x;
    if (PERSIST) {
        if (threadIdx.x == 0) s_chunk = (int)atomicAdd(&S.lctl->next_chunk, 1u);
        __syncthreads();
        ck = s_chunk;
    }
    while (ck < nchunks) {
    const int i0 = ck * chunk;
    const int i1 = min(i0 + chunk, n);
    // the colony of the thread's slot and the first slot of the next one, kept in
    // registers: the common step compares against it instead of loading it
    int colony = -1, cnext = 0;
    for (int base = i0; base < i1; base += blockDim.x) {  // same trip count for every thread
        const int i = base + threadIdx.x;
        const bool act = i < i1;
        unsigned lo0 = kKeyPosInf, lo1 = kKeyPosInf, lo2 = kKeyPosInf;
        unsigned hi0 = kKeyNegInf, hi1 = kKeyNegInf, hi2 = kKeyNegInf;
        int4 h = make_int4(0, 0, 0, 0);
        int cnt = 0;
        float ux = 0.0f, uy = 0.0f, uz = 0.0f;
        float gx = 0.0f, gy = 0.0f, gz = 0.0f;
        PairRec pr{CAP ? S.pcap : nullptr, i, 0};
        // the pair term: offset from the high words, the gate r < rA, F / r
        auto term = [&](const int4 me, const int4 q, float tx, float ty, float tz, float &ex, float &ey, float &ez,
                        float &Fi) -> bool {
            ex = (float)(me.x - q.x) * tx;
            ey = (float)(me.y - q.y) * ty;
            ez = (float)(me.z - q.z) * tz;
            const float r2f = __fmaf_rn(ex, ex, __fmaf_rn(ey, ey, __fmul_rn(ez, ez)));
            const float rSf = __fadd_rn(__int_as_float(me.w), __int_as_float(q.w));
            const float rAf = __fadd_rn(rSf, bwf);
            if (!(r2f < __fmul_rn(rAf, rAf))) return false;
            float inv;  // (r^2 is 0 or normal: the high word's unit squared is, list_skin)
            asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(r2f));
            const float rn = __fmul_rn(r2f, inv);
            const float d1 = __fsub_rn(rn, rAf);
            const float Fm = __fmul_rn(__fmul_rn(__fmul_rn(-kf, d1), d1), __fsub_rn(rn, rSf));
            Fi = __fmul_rn(Fm, inv);
            return true;
        };
        auto pair = [&](int j, const int4 q) {
            float ex, ey, ez, Fi;
            if (!term(h, q, ux, uy, uz, ex, ey, ez, Fi)) return;
            if (CAP) pr.add(j);
            gx = __fmaf_rn(Fi, ex, gx);
            gy = __fmaf_rn(Fi, ey, gy);
            gz = __fmaf_rn(Fi, ez, gz);
        };
        int4 rec = make_int4(0, 0, 0, 0);
        int xo = 0;
        if (act) {
            rec = __ldg(&S.lrec[i]);
            h = ga[i];
            xo = __ldg(&S.xoff[i >> 5]);
            // (read after the pairs; held in registers from here they cost occupancy)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(la + i));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(la + n + i));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(la + 2 * (size_t)n + i));
            if (colony < 0) {
                colony = colony_of(S.cbase, S.ncol, i);
                cnext = (colony + 1 < S.ncol) ? __ldg(&S.cbase[colony + 1]) : 0x7fffffff;
            }
            while (i >= cnext) {
                ++colony;
                cnext = (colony + 1 < S.ncol) ? __ldg(&S.cbase[colony + 1]) : 0x7fffffff;
            }
            cnt = rec.x & 0xff;
            const float4 fu = *reinterpret_cast<const float4 *>(S.fxg[colony].uh);
            ux = fu.x;
            uy = fu.y;
            uz = fu.z;
        }
        if (act) {
            if (cnt <= kNbrCap) {
                // the inline entries: their gathers go out together
                const int4 z4 = make_int4(0, 0, 0, 0);
                const int4 p0 = (cnt > 0) ? __ldg(&ga[rec.y]) : z4;
                const int4 p1 = (cnt > 1) ? __ldg(&ga[rec.z]) : z4;
                const int4 p2 = (cnt > 2) ? __ldg(&ga[rec.w]) : z4;
                if (cnt > 0) pair(rec.y, p0);
                if (cnt > 1) pair(rec.z, p1);
                if (cnt > 2) pair(rec.w, p2);
                // this slot's entries past the inline ones, from its place in
                // its warp's run of the compacted list
                const int xl = list_extra(cnt);
                if (xl) {
                    const int *xs = S.xlist + xo + ((rec.x >> 8) & 0x3ff);
                    int k = 0;
                    // four entries in flight at a time (past the end: the first of
                    // the four again, dropped): the list loads and the neighbour
                    // gathers are independent across entries
                    for (; k < xl; k += 4) {
                        const int m = xl - k;
                        const int e0 = __ldg(xs + k), e1 = __ldg(xs + k + (m > 1 ? 1 : 0));
                        const int e2 = __ldg(xs + k + (m > 2 ? 2 : 0)), e3 = __ldg(xs + k + (m > 3 ? 3 : 0));
                        const int4 q0 = __ldg(&ga[e0]);
                        const int4 q1 = __ldg(&ga[e1]);
                        const int4 q2 = __ldg(&ga[e2]);
                        const int4 q3 = __ldg(&ga[e3]);
                        pair(e0, q0);
                        if (m > 1) pair(e1, q1);
                        if (m > 2) pair(e2, q2);
                        if (m > 3) pair(e3, q3);
                    }
                }
            } else {  // list overflow: walk the build's cells with the current records
                const DevGeom &G = S.geoms[colony];
                int bx, by;
                col_to_bxy(G, S.col[B][i], bx, by);
                visit_cells(S, G, S.rank[B][i], bx, by, S.iz[B][i], [&](int s) {
                    const int j = __ldg(&S.perm[B][s]);
                    pair(j, __ldg(&ga[j]));
                });
            }
        }
        if (act) {
            const FxGeom &F = S.fxg[colony];
            if (CAP) pr.done();
            const unsigned zw = F.zw;
            const float ri = __int_as_float(h.w);
            const float dzw = (float)(int)((unsigned)h.z - zw) * uz;
            const float vx = gx, vy = gy, vz = gz + wall_law32(dzw, ri, zkf, zbwf, zgf);
            const float ix = dtf * vx, iy = dtf * vy, iz = dtf * vz;
            bool big = false;
            const float4 fc = *reinterpret_cast<const float4 *>(F.c);
            const float4 fl = *reinterpret_cast<const float4 *>(F.cl);
            unsigned long long nx = fx_join((unsigned)h.x, la[i]);
            unsigned long long ny = fx_join((unsigned)h.y, la[n + i]);
            unsigned long long nz = fx_join((unsigned)h.z, la[2 * (size_t)n + i]);
            const float px = __fmul_rn(ix, fc.x), py = __fmul_rn(iy, fc.y), pz = __fmul_rn(iz, fc.z);
            if (fabsf(px) < 1.8014398509481984e16f && fabsf(py) < 1.8014398509481984e16f &&
                fabsf(pz) < 1.8014398509481984e16f) {  // 2^54 (fx_inc's common case)
                nx += (unsigned long long)fx_inc_small(ix, fc.x, fl.x, px);
                ny += (unsigned long long)fx_inc_small(iy, fc.y, fl.y, py);
                nz += (unsigned long long)fx_inc_small(iz, fc.z, fl.z, pz);
            } else {
                nx += (unsigned long long)fx_inc(ix, fc.x, fl.x, big);
                ny += (unsigned long long)fx_inc(iy, fc.y, fl.y, big);
                nz += (unsigned long long)fx_inc(iz, fc.z, fl.z, big);
            }
            const unsigned hz = (unsigned)(nz >> 32);
            // the domain [plo, phi) of a closed axis is the high word in [2^30, 2^31)
            if (hz - (1u << 30) >= (1u << 30)) {
                atomicAdd(&S.cnt->out_of_domain, 1ULL);
                // within three quarters of a length of the domain, or the fixed point's range ends
                if (hz < (1u << 28) || hz >= 0xf0000000u) atomicAdd(&S.cnt->range, 1ULL);
            }
            S.fxh[b][i] = make_int4((int)(nx >> 32), (int)(ny >> 32), (int)hz, h.w);
            unsigned *lb = S.fxl[b];
            lb[i] = (unsigned)nx;
            lb[n + i] = (unsigned)ny;
            lb[2 * (size_t)n + i] = (unsigned)nz;
            S.vxf[i] = vx;
            S.vyf[i] = vy;
            S.vzf[i] = vz;
            lo0 = hi0 = fkey(ix);
            lo1 = hi1 = fkey(iy);
            lo2 = hi2 = fkey(iz);
            if (!isfinite(ix + iy + iz) || big) {
                atomicAdd(&S.cnt->nonfinite, 1ULL);
                lo0 = 0u;  // spreads the bound: the next step rebuilds
                hi0 = 0xffffffffu;
            }
        }
        lo0 = __reduce_min_sync(0xffffffffu, lo0);
        hi0 = __reduce_max_sync(0xffffffffu, hi0);
        lo1 = __reduce_min_sync(0xffffffffu, lo1);
        hi1 = __reduce_max_sync(0xffffffffu, hi1);
        lo2 = __reduce_min_sync(0xffffffffu, lo2);
        hi2 = __reduce_max_sync(0xffffffffu, hi2);
        if (lane == 0) {
            wmin[w][0] = min(wmin[w][0], lo0);
            wmax[w][0] = max(wmax[w][0], hi0);
            wmin[w][1] = min(wmin[w][1], lo1);
            wmax[w][1] = max(wmax[w][1], hi1);
            wmin[w][2] = min(wmin[w][2], lo2);
            wmax[w][2] = max(wmax[w][2], hi2);
        }
    }
    if (!PERSIST) break;
    __syncthreads();  // every thread has read s_chunk
    if (threadIdx.x == 0) s_chunk = (int)atomicAdd(&S.lctl->next_chunk, 1u);
    __syncthreads();
    ck = s_chunk;
    }
    if (PERSIST && threadIdx.x == 0) {
        // the last block to find the dispenser empty resets it for the next launch
        __threadfence();
        if (atomicAdd(&S.lctl->done_blocks, 1u) == gridDim.x - 1) {
            S.lctl->next_chunk = 0u;
            S.lctl->done_blocks = 0u;
            __threadfence();
        }
    }
    // then over the block: six atomics per block, not per warp (updates of
    // one address serialise in its L2 slice)
    __syncthreads();
    if (threadIdx.x < 3) {
        const int k = threadIdx.x;
        unsigned lo = kKeyPosInf, hi = kKeyNegInf;
        for (int v = 0; v < nw; ++v) {
            lo = min(lo, wmin[v][k]);
            hi = max(hi, wmax[v][k]);
        }
        if (hi >= lo) {
            atomicMin(&S.lctl->inc_min[k], lo);
            atomicMax(&S.lctl->inc_max[k], hi);
        }
    }
}

// The two ends of the list path, in integer arithmetic (GB300 issues FP64 at
// a small fraction of the FP32 rate; only an origin other than 0 costs one
// FP64 addition or subtraction per coordinate).
//
// fixed point of a coordinate: (x - o) 2^64 / span, rounded, mod 2^64 on a
// periodic axis, else clamped to the range [0, 2^64) (a closed axis's range
// is four domain lengths from one length below plo).  With d = x - o =
// md 2^ed and 2^64 / span = mc 2^ec the value is md mc 2^(ed + ec): a 117-bit
// product shifted into place.
__device__ __forceinline__ unsigned long long to_fx(double x, const FxGeom &F, int ax)
{
    const double d = F.ozero[ax] ? x : x - F.o[ax];
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    const int be = (int)((b >> 52) & 0x7ffu);
    if (be == 0) return 0ull;  // zero (and subnormals)
    const bool neg = (b >> 63) != 0ull;
    const unsigned long long md = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    const unsigned long long hi = __umul64hi(md, F.mc[ax]), lo = md * F.mc[ax];
    const int r = -((be - 1075) + F.ec[ax]);  // X = (hi:lo) >> r
    unsigned long long X;
    bool over = false;
    if (r <= 0) {
        over = true;
        X = 0ull;
    } else if (r < 64) {
        over = (hi >> r) != 0ull;
        X = (hi << (64 - r)) | (lo >> r);
        X += (lo >> (r - 1)) & 1ull;  // round half up
    } else if (r < 128) {
        X = (r == 64) ? hi : (hi >> (r - 64));
        X += (r == 64) ? (lo >> 63) : ((hi >> (r - 65)) & 1ull);
    } else {
        X = 0ull;
    }
    if (F.per[ax]) return neg ? 0ull - X : X;  // the unsigned wrap is the periodic wrap
    if (neg) return 0ull;
    return over ? ~0ull : X;
}

// ---- FP64 steps over the list ------------------------------------------------
// The plain form on the same list: the list is a superset of the pairs within the
// cutoff for as long as the bound holds, whoever moves the slots, so an FP64 step
// needs no re-binning, sort and stencil walk either.  What it must keep is the
// reference's summation order, which follows the CURRENT bins (27 bins around
// the slot's own in walk order, ascending caller index within one): each pair
// that passes the FP64 gate gets that order as its key, from its bins
// re-derived out of the FP64 positions (bin_of_fast: exact, no FP64 arithmetic),
// and a slot adds its terms by ascending key.  The keys of a list ascend as it was
// built and rarely stop doing so between builds; then the slot selects by key.
// Image membership is the reference's (the image's bin from its shifted FP64
// position).  So the result is bit-identical to the per-step path's.
// Each step also writes the slots' coordinates above the domain's corner in
// FP32 (rel; c = plo + coordinate within 2^-23 of the magnitudes), which the next
// step screens its entries with.
// Bound: FP64 issue (2 lanes a clock per SM) of the pairs that pass the screen and
// of the update, then the screen's loads; 688 000 slots in 64 colonies step in 187 us
// (per-step path 295 with its rebuild), 400 000 in 81.  Blocks of 64 slots: the
// pairs of a block spread evenly over its threads; ten blocks fit an SM (96 registers:
// 2 million slots 372 us; eight at 119 386, twelve at 80 381; the entries' gathers four at
// a time 373).  The
// staging holds a whole list: with room for 12 entries and a serial way out the few
// slots beyond it (2 % of a dense colony's blocks held one) kept the kernel for
// 520 us.  A state with an overflowed list (over 32 slots within the cutoff and the
// skin of one) steps on the per-step path, whose walk is one thread's or warp's.
constexpr int kList64Block = 64;
constexpr int kList64Pairs = 4;  // evaluated at once, per slot on average (more: in batches of slots)

// FP32 coordinates of a position; false when the list does not cover it: a
// closed axis more than 0.7 of a length outside the domain, or not finite.
__device__ __forceinline__ bool coords32(const DevGeom &G, double x, double y, double z, float &cx, float &cy,
                                         float &cz)
{
    cx = d2f_rn(x) - G.plof[0];
    cy = d2f_rn(y) - G.plof[1];
    cz = d2f_rn(z) - G.plof[2];
    bool in = finite_bits(x) && finite_bits(y) && finite_bits(z);
    const float c[3] = {cx, cy, cz};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float len = G.dxf[d] * (float)G.n[d];
        in = in && c[d] > -0.7f * len && c[d] < 1.7f * len;
    }
    return in;
}

// Whether the state's positions resolve in FP32 coordinates, and those coordinates.
__global__ void k_list64_begin(const DevState S, int a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int col = block_colony(S, i);
    if (i < S.n) {
        float cx, cy, cz;
        if (!coords32(S.geoms[col], S.x[a][i], S.y[a][i], S.z[a][i], cx, cy, cz)) S.lctl->bail = 1;
        S.rel[a][i] = make_float4(cx, cy, cz, d2f_rn(S.rad[i]));
    }
}

// Sum of the terms t0 .. t0 + m - 1 by ascending key (the keys of a slot's
// pairs differ; ~0: no term).
__device__ __forceinline__ void add_by_key(const unsigned long long *key, const double *term, int pitch, int t0, int m,
                                           double &fx, double &fy, double &fz)
{
    unsigned long long last = 0ull;
    bool ordered = true;
    for (int k = t0; k < t0 + m; ++k) {
        const unsigned long long q = key[k];
        if (q == ~0ull) continue;
        ordered = ordered && q >= last;
        last = q;
    }
    if (ordered) {
        for (int k = t0; k < t0 + m; ++k) {
            if (key[k] == ~0ull) continue;
            fx += term[k];
            fy += term[pitch + k];
            fz += term[2 * pitch + k];
        }
        return;
    }
    last = 0ull;
    for (int r = 0; r < m; ++r) {
        unsigned long long best = ~0ull;
        int at = -1;
        for (int k = t0; k < t0 + m; ++k)
            if (key[k] < best && (r == 0 || key[k] > last)) {
                best = key[k];
                at = k;
            }
        if (at < 0) break;
        last = best;
        fx += term[at];
        fy += term[pitch + at];
        fz += term[2 * pitch + at];
    }
}

// The FP64 term of a slot (position and radius o, bins ob, colony geometry Q) on
// j, and the pair's place in the reference's order (~0: not in the list or
// beyond the cutoff).
__device__ __forceinline__ unsigned long long pair_by_list64(const DevState &S, const DevParams &P, int a,
                                                             const double *o, const int4 ob, const DevGeom &Q, int j,
                                                             int code, double *t)
{
    const int sx = code / 3 - 1, sy = code % 3 - 1;
    const double x = S.x[a][j], y = S.y[a][j], z = S.z[a][j];
    const double xj = sx ? image_coord(x, Q.len[0], sx) : x;
    const double yj = sy ? image_coord(y, Q.len[1], sy) : y;
    if (!sphere_pair64(P, 1, o[0] - xj, o[1] - yj, o[2] - z, o[3], S.rad[j], t)) return ~0ull;
    // (an image is listed when its source's own bin is the face's and its shifted
    // position is in the halo cell; image_bin clamps, and a position beyond a face,
    // as a load may hold, has partners farther in than the face's bin)
    int jx = bin_of_fast(x, Q.plo[0], Q.dxi[0], Q.plof[0], Q.dxif[0], 1, Q.n[0]);
    int jy = bin_of_fast(y, Q.plo[1], Q.dxi[1], Q.plof[1], Q.dxif[1], 1, Q.n[1]);
    if (sx) {
        if (jx != (sx < 0 ? Q.n[0] : 1)) return ~0ull;
        jx = sx < 0 ? 0 : Q.n[0] + 1;
        if (image_bin(Q, 0, xj) != jx) return ~0ull;
    }
    if (sy) {
        if (jy != (sy < 0 ? Q.n[1] : 1)) return ~0ull;
        jy = sy < 0 ? 0 : Q.n[1] + 1;
        if (image_bin(Q, 1, yj) != jy) return ~0ull;
    }
    const int jz = bin_of_fast(z, Q.plo[2], Q.dxi[2], Q.plof[2], Q.dxif[2], 1, Q.n[2]);
    const int d0 = jx - ob.x + 1, d1 = jy - ob.y + 1, d2 = jz - ob.z + 1;
    if ((unsigned)d0 > 2u || (unsigned)d1 > 2u || (unsigned)d2 > 2u) return ~0ull;  // not a stencil pair
    return ((unsigned long long)(d0 * 9 + d1 * 3 + d2) << 32) | (unsigned)S.orig[j];
}

__global__ void __launch_bounds__(kList64Block, 10) k_list64_step(const DevState S, const DevParams P, double dt)
{
    constexpr int B = kList64Block, cap = B * kList64Pairs;
    static_assert(kNbrCap <= cap, "a slot's pairs fit a batch");
    chain_wait();
    // (a stalled step, or one past the call's last; an overflowed list)
    if (!S.lctl->active || S.lctl->overflow) return;
    const int a = S.lctl->cur, b = a ^ 1;
    __shared__ int stage[kNbrCap][B];
    __shared__ unsigned char codes[kNbrCap][B];
    __shared__ double opos[B][4];
    __shared__ int4 obin[B];
    __shared__ double term[3 * cap];
    __shared__ unsigned long long key[cap];
    __shared__ int orun[B + 1], wsum[B / 32];
    __shared__ unsigned wmin[B / 32][3], wmax[B / 32][3];
    const int n = S.n;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int i = blockIdx.x * B + tid;
    const bool act = i < n;
    const int colony = block_colony(S, i);
    const float4 *__restrict__ ca = S.rel[a];
    double xi = 0.0, yi = 0.0, zi = 0.0, ri = 0.0;
    int xl = 0, bx = 1, by = 1, bz = 1;
    const DevGeom &G = S.geoms[act ? colony : 0];
    if (act) {
        const int4 rec = __ldg(&S.lrec[i]);
        const float4 me = ca[i];
        xi = S.x[a][i];
        yi = S.y[a][i];
        zi = S.z[a][i];
        ri = S.rad[i];
        bx = bin_of_fast(xi, G.plo[0], G.dxi[0], G.plof[0], G.dxif[0], 1, G.n[0]);
        by = bin_of_fast(yi, G.plo[1], G.dxi[1], G.plof[1], G.dxif[1], 1, G.n[1]);
        bz = bin_of_fast(zi, G.plo[2], G.dxi[2], G.plof[2], G.dxif[2], 1, G.n[2]);
        const float lenx = G.dxf[0] * (float)G.n[0], leny = G.dxf[1] * (float)G.n[1];
        // the FP32 coordinates' rounding (2^-23 of the magnitudes each, four of them per
        // axis with the subtraction's) and 2e-6 of the bound's own
        const float mag = fabsf(G.plof[0]) + fabsf(G.plof[1]) + fabsf(G.plof[2]) +
                          2.0f * (lenx + leny + G.dxf[2] * (float)G.n[2]);
        const float ci = (me.w + P.bw32) * 1.000002f + 2.0e-6f * (G.dxf[0] + G.dxf[1] + G.dxf[2]) + 4.8e-7f * mag;
        auto entry = [&](int j) {
            const float4 q = __ldg(&ca[j]);
            float ex = me.x - q.x, ey = me.y - q.y;
            const float ez = me.z - q.z;
            int sx = 0, sy = 0;
            if (G.per[0] && fabsf(ex) > 0.5f * lenx) {
                sx = ex < 0.0f ? -1 : 1;
                ex -= (float)sx * lenx;
            }
            if (G.per[1] && fabsf(ey) > 0.5f * leny) {
                sy = ey < 0.0f ? -1 : 1;
                ey -= (float)sy * leny;
            }
            const float r2f = __fmaf_rn(ex, ex, __fmaf_rn(ey, ey, __fmul_rn(ez, ez)));
            const float lim = q.w + ci;
            if (!(r2f > lim * lim)) {
                stage[xl][tid] = j;
                codes[xl][tid] = (unsigned char)((sx + 1) * 3 + (sy + 1));
                ++xl;
            }
        };
        const int len = rec.x & 0xff;
        if (len > 0) entry(rec.y);
        if (len > 1) entry(rec.z);
        if (len > 2) entry(rec.w);
        const int m = list_extra(len);
        const int *xs = S.xlist + (m ? __ldg(&S.xoff[i >> 5]) + ((rec.x >> 8) & 0x3ff) : 0);
        for (int k = 0; k < m; ++k) entry(__ldg(xs + k));
    }
    opos[tid][0] = xi;
    opos[tid][1] = yi;
    opos[tid][2] = zi;
    opos[tid][3] = ri;
    obin[tid] = make_int4(bx, by, bz, colony);
    // the block's run of staged pairs: slot by slot in thread order
    int xo = xl;
    for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, xo, d);
        if (lane >= d) xo += v;
    }
    if (lane == 31) wsum[w] = xo;
    __syncthreads();
    for (int v = 0; v < w; ++v) xo += wsum[v];
    orun[tid + 1] = xo;
    if (tid == 0) orun[0] = 0;
    __syncthreads();
    xo -= xl;
    double fx = 0.0, fy = 0.0, fz = 0.0;
    // one pair per thread, a slot's terms added by its thread; in batches of
    // slots when the block's pairs are more than the terms' room
    for (int s0 = 0; s0 < B;) {
        const int t0 = orun[s0];
        int s1 = B;
        if (orun[B] - t0 > cap)
            for (s1 = s0 + 1; orun[s1 + 1] - t0 <= cap;) ++s1;
        const int t1 = orun[s1];
        for (int t = t0 + tid; t < t1; t += B) {
            int o = 0;  // the slot that owns pair t
#pragma unroll
            for (int s2 = B / 2; s2 >= 1; s2 >>= 1)
                if (orun[o + s2] <= t) o += s2;
            const int k = t - orun[o];
            double tt[3] = {0.0, 0.0, 0.0};
            key[t - t0] = pair_by_list64(S, P, a, opos[o], obin[o], S.geoms[obin[o].w], stage[k][o], codes[k][o], tt);
            term[t - t0] = tt[0];
            term[cap + t - t0] = tt[1];
            term[2 * cap + t - t0] = tt[2];
        }
        __syncthreads();
        if (tid >= s0 && tid < s1) add_by_key(key, term, cap, xo - t0, xl, fx, fy, fz);
        __syncthreads();
        s0 = s1;
    }
    unsigned lo[3] = {kKeyPosInf, kKeyPosInf, kKeyPosInf}, hi[3] = {kKeyNegInf, kKeyNegInf, kKeyNegInf};
    if (act) {
        // evaluateSurfaceForce, sphere branch, the update and the wrap, as k_sphere64
        const double vx = plus_zero(fx);
        const double vy = plus_zero(fy);
        const double vz = fz + wall_law(zi, ri, P);
        const double ix = dt * vx, iy = dt * vy, iz = dt * vz;
        double nx = xi + ix;
        double ny = yi + iy;
        const double nz = zi + iz;
        if (G.per[0]) nx = wrap1(nx, G.plo[0], G.phi[0], G.len[0]);
        if (G.per[1]) ny = wrap1(ny, G.plo[1], G.phi[1], G.len[1]);
        S.x[b][i] = nx;
        S.y[b][i] = ny;
        S.z[b][i] = nz;
        S.vx[i] = vx;
        S.vy[i] = vy;
        S.vz[i] = vz;
        float cx, cy, cz;
        if (!coords32(G, nx, ny, nz, cx, cy, cz)) S.lctl->bail = 1;
        S.rel[b][i] = make_float4(cx, cy, cz, d2f_rn(ri));
        count_slot(S, G, nx, ny, nz,
                   bin_of_fast(nx, G.plo[0], G.dxi[0], G.plof[0], G.dxif[0], 1, G.n[0]),
                   bin_of_fast(ny, G.plo[1], G.dxi[1], G.plof[1], G.dxif[1], 1, G.n[1]), true);
        lo[0] = hi[0] = fkey(d2f_rn(ix));
        lo[1] = hi[1] = fkey(d2f_rn(iy));
        lo[2] = hi[2] = fkey(d2f_rn(iz));
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = __reduce_min_sync(0xffffffffu, lo[k]);
        hi[k] = __reduce_max_sync(0xffffffffu, hi[k]);
        if (lane == 0) {
            wmin[w][k] = lo[k];
            wmax[w][k] = hi[k];
        }
    }
    __syncthreads();
    if (tid < 3) {
        unsigned l = kKeyPosInf, h = kKeyNegInf;
        for (int v = 0; v < B / 32; ++v) {
            l = min(l, wmin[v][tid]);
            h = max(h, wmax[v][tid]);
        }
        if (h >= l) {
            atomicMin(&S.lctl->inc_min[tid], l);
            atomicMax(&S.lctl->inc_max[tid], h);
        }
    }
}

// The build's fixed-point positions from the FP64 ones (the high words alone).
__global__ void k_list64_fx(const DevState S)
{
    if (!S.lctl->rebuild) return;
    const int a = S.lctl->cur;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int col = block_colony(S, i);
    if (i < S.n) {
        const FxGeom &F = S.fxg[col];
        S.fxh[a][i] = make_int4((int)(to_fx(S.x[a][i], F, 0) >> 32), (int)(to_fx(S.y[a][i], F, 1) >> 32),
                                (int)(to_fx(S.z[a][i], F, 2) >> 32), __float_as_int(d2f_rn(S.rad[i])));
    }
}

// Fixed-point positions of buffer a from its FP64 positions and the radii
__global__ void k_list_init(const DevState S, int a)
{
    const int n = S.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int col = block_colony(S, i);
    if (i < n) {
        const FxGeom &F = S.fxg[col];
        const unsigned long long X = to_fx(S.x[a][i], F, 0);
        const unsigned long long Y = to_fx(S.y[a][i], F, 1);
        const unsigned long long Z = to_fx(S.z[a][i], F, 2);
        S.fxh[a][i] = make_int4((int)(X >> 32), (int)(Y >> 32), (int)(Z >> 32), __float_as_int(d2f_rn(S.rad[i])));
        S.fxl[a][i] = (unsigned)X;
        S.fxl[a][n + i] = (unsigned)Y;
        S.fxl[a][2 * (size_t)n + i] = (unsigned)Z;
    }
}

// FP64 positions of buffer a from its fixed-point positions
__global__ void k_list_to_fp64(const DevState S, int a)
{
    const int n = S.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int col = block_colony(S, i);
    if (i < n) {
        const FxGeom &F = S.fxg[col];
        const int4 h = S.fxh[a][i];
        S.x[a][i] = from_fx(fx_join((unsigned)h.x, S.fxl[a][i]), F, 0);
        S.y[a][i] = from_fx(fx_join((unsigned)h.y, S.fxl[a][n + i]), F, 1);
        S.z[a][i] = from_fx(fx_join((unsigned)h.z, S.fxl[a][2 * (size_t)n + i]), F, 2);
    }
}

// One axis of the same conversion, the value also scattered to the caller's
// order (out[orig[i]]): a store of the state converts and gathers in one pass.
__global__ void k_list_to_fp64_axis(const DevState S, int a, int ax, double *out)
{
    const int n = S.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int col = block_colony(S, i);
    if (i < n) {
        const FxGeom &F = S.fxg[col];
        const int4 h = S.fxh[a][i];
        const unsigned hi = (unsigned)(ax == 0 ? h.x : (ax == 1 ? h.y : h.z));
        const double v = from_fx(fx_join(hi, S.fxl[a][(size_t)ax * n + i]), F, ax);
        (ax == 0 ? S.x : (ax == 1 ? S.y : S.z))[a][i] = v;
        const int o = S.orig[i];
        if ((unsigned)o < (unsigned)n) out[o] = v;
    }
}

}  // namespace

int launch_list_decide(const DevState &S, unsigned long long cond, int mode, cudaStream_t st)
{
    launch_after(k_list_decide, 1, 1, 0, st, S.lctl, S.cnt, (cudaGraphConditionalHandle)cond, mode);
    return 1;
}

int launch_list64_begin(const DevState &S, int a, cudaStream_t st)
{
    k_list64_begin<<<(S.n + 255) / 256, 256, 0, st>>>(S, a);
    return 1;
}

int launch_list64_fx(const DevState &S, cudaStream_t st)
{
    k_list64_fx<<<(S.n + 255) / 256, 256, 0, st>>>(S);
    return 1;
}

int launch_list64_step(const DevState &S, const DevParams &P, double dt, cudaStream_t st, bool chained)
{
    const int grid = (S.n + kList64Block - 1) / kList64Block;
    if (chained) launch_after(k_list64_step, grid, kList64Block, 0, st, S, P, dt);
    else k_list64_step<<<grid, kList64Block, 0, st>>>(S, P, dt);
    return 1;
}

int launch_list_init(const DevState &S, int a, int grid, int block, cudaStream_t st)
{
    (void)grid;  // one slot per thread
    k_list_init<<<(S.n + block - 1) / block, block, 0, st>>>(S, a);
    return 1;
}

int launch_list_to_fp64(const DevState &S, int a, int grid, int block, cudaStream_t st)
{
    (void)grid;  // one slot per thread
    k_list_to_fp64<<<(S.n + block - 1) / block, block, 0, st>>>(S, a);
    return 1;
}

int launch_list_to_fp64_axis(const DevState &S, int a, int ax, double *out, int block, cudaStream_t st)
{
    k_list_to_fp64_axis<<<(S.n + block - 1) / block, block, 0, st>>>(S, a, ax, out);
    return 1;
}

int launch_list_build(const DevState &S, const DevParams &P, int build_block, cudaStream_t st)
{
    k_list_build<<<(S.n + build_block - 1) / build_block, build_block, 0, st>>>(S, P);
    return 1;
}

int launch_list_rebuild(const DevState &S, const DevParams &P, int *scan_scratch, int grid, int block,
                        int build_block, cudaStream_t st)
{
    const int *gate = &S.lctl->rebuild;
    // one slot per thread (a block's colonies from one search)
    const int g1 = (S.n + block - 1) / block;
    k_list_rebin<<<g1, block, 0, st>>>(S);
    int k = 1 + launch_scan(S.colcnt, S.colstart[kListBins], S.ncols_total, scan_scratch, st, gate);
    k_list_scatter<<<g1, block, 0, st>>>(S);
    k_list_canon<<<g1, block, 0, st>>>(S);
    // the cell offsets: a block per kCellsBlock columns of the largest colony
    const dim3 gc(S.ncol, std::max(1, std::min(65535, (S.cols_max + kCellsBlock - 1) / kCellsBlock)));
    k_list_cells<<<gc, kCellsBlock, 0, st>>>(S);
    // the build: one slot per thread in small blocks (the stencil walks
    // differ in length from slot to slot; small blocks on a grid of every
    // slot let the scheduler balance them)
    launch_list_build(S, P, build_block, st);
    // the entries past the inline ones, compacted per group of 32 slots
    const int gx = (S.n + 127) / 128;
    k = k + launch_scan(S.xcnt, S.xoff, (S.n + 31) / 32, scan_scratch, st, gate);
    k_list_xcopy<<<gx, 128, 0, st>>>(S);
    return k + 5;
}

int launch_list_step(const DevState &S, const DevParams &P, double dt, int grid, int block, int passes,
                     cudaStream_t st, bool persistent, bool chained)
{
    // passes of the block per chunk (passes <= 0: the rule): short enough that
    // the block scheduler evens out the uneven list lengths of the colonies
    // (one wave of long chunks ends on its slowest block), long enough to
    // amortise the colony search and the block's reduction of the increment
    // spreads.  The rule: two, or one when two would leave fewer than four
    // waves of 1536 threads per SM (grid = the SM count).
    int chunk = block * passes;
    if (passes <= 0) {
        const int two = (S.n + 2 * block - 1) / (2 * block);
        chunk = (two >= 4 * (1536 / block) * grid) ? 2 * block : block;
    }
    const int nb = (S.n + chunk - 1) / chunk;
    if (persistent) {
        // one wave: the blocks that fit on the SMs at once (1536 threads per SM)
        const int wave = std::max(1, std::min(nb, grid * (1536 / block)));
        if (S.pcap) k_list_step<true, true><<<wave, block, 0, st>>>(S, P, (float)dt, chunk);
        else k_list_step<false, true><<<wave, block, 0, st>>>(S, P, (float)dt, chunk);
    } else {
        if (chained && !S.pcap) launch_after(k_list_step<false, false>, nb, block, 0, st, S, P, (float)dt, chunk);
        else if (S.pcap) k_list_step<true, false><<<nb, block, 0, st>>>(S, P, (float)dt, chunk);
        else k_list_step<false, false><<<nb, block, 0, st>>>(S, P, (float)dt, chunk);
    }
    return 1;
}

}  // namespace bmxg
