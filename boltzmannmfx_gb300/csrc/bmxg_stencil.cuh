// bmxg_stencil.cuh -- the neighbour traversal every kernel shares, and the
// per-slot rebin.  Translation units that include this are compiled with
// -fmad=false so that every FP64 expression rounds exactly like the host
// oracle's (FP32 code uses explicit __fmaf_rn where it wants a fused op).
#pragma once
#include <algorithm>

#include "bmxg_kernels.cuh"

namespace bmxg {

// Whether the periodic image of slot j under shift (sx, sy) lies in stencil
// row (ii, jj): the image's bin is computed from its shifted FP64 position,
// as AMReX bins its ghost copies.
__device__ __forceinline__ bool image_in_row(const DevState &S, const DevGeom &G, int a, int j,
                                             int ii, int jj, int sx, int sy)
{
    if (sx) {
        if (image_bin(G, 0, image_coord(S.x[a][j], G.len[0], sx)) != ii) return false;
    }
    if (sy) {
        if (image_bin(G, 1, image_coord(S.y[a][j], G.len[1], sy)) != jj) return false;
    }
    return true;
}

// Visit slot i's neighbour candidates in the order of the reference's
// neighbour list: stencil bins x outermost, then y, then z, ascending
// original index within a bin (AMReX NeighborList over the 27 bins around
// the particle's bin, periodic images from the one-cell halo).  Each column is
// entered by binary search at its first entry of z bin izi - 1.
// f(j, dxs, dys, dzs, sx, sy): dxs/dys/dzs = neighbour bin minus own bin,
// sx/sy = image shift in units of the domain length.
template <class F>
__device__ __forceinline__ void visit_stencil(const DevState &S, const DevGeom &G, int a, int i,
                                              int bx, int by, int izi, F &&f)
{
    const int *__restrict__ perm = S.perm[a];
    const int *__restrict__ cs = S.colstart[a];
    const int *__restrict__ izs = S.iz[a];
    for (int ii = bx - 1; ii <= bx + 1; ++ii) {
        for (int jj = by - 1; jj <= by + 1; ++jj) {
            int cc, sx, sy;
            if (!stencil_row(G, ii, jj, cc, sx, sy)) continue;
            const int t1 = __ldg(&cs[cc + 1]);
            int t0 = __ldg(&cs[cc]);
            for (int hi2 = t1; t0 < hi2;) {  // first entry of z bin >= izi - 1
                const int mid = (t0 + hi2) >> 1;
                if (__ldg(&izs[__ldg(&perm[mid])]) < izi - 1) t0 = mid + 1;
                else hi2 = mid;
            }
            for (int t = t0; t < t1; ++t) {
                const int j = __ldg(&perm[t]);
                const int dzs = __ldg(&izs[j]) - izi;
                if (dzs > 1) break;  // a column is sorted by z-bin: the rest is out of reach
                if (dzs < -1) continue;
                if (j == i) continue;
                if ((sx | sy) && !image_in_row(S, G, a, j, ii, jj, sx, sy)) continue;
                f(j, ii - bx, jj - by, dzs, sx, sy);
            }
        }
    }
}

// First t in [lo, hi) with siz[t] >= v (siz ascends over the range).
__device__ __forceinline__ int first_at_least(const int *__restrict__ siz, int lo, int hi, int v)
{
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(&siz[mid]) < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// The same walk over the column-sorted copies (siz / srel, filled by the
// rebuild): f(t, dxs, dys, dzs, sx, sy) gets the sorted index t of each
// candidate (its slot is perm[t]).  An x-row's three columns by-1..by+1 are
// consecutive column ids, so away from the periodic faces a row is three
// back-to-back runs of one contiguous range; each run is ordered by z-bin
// and is entered by binary search at its first entry of z-bin izi - 1 (a
// column can be many bins tall), and left at the first entry above izi + 1.
// self_t = rank of the slot itself.  Order of candidates: identical to
// visit_stencil.
template <class F>
__device__ __forceinline__ void visit_sorted(const DevState &S, const DevGeom &G, int a, int self_t, int bx,
                                             int by, int izi, F &&f)
{
    const int *__restrict__ cs = S.colstart[a];
    const int *__restrict__ siz = S.siz[a];
    for (int ii = bx - 1; ii <= bx + 1; ++ii) {
        int srcx = ii, sx = 0;
        if (ii == 0) {
            if (!G.per[0]) continue;
            srcx = G.n[0];
            sx = -1;
        } else if (ii == G.n[0] + 1) {
            if (!G.per[0]) continue;
            srcx = 1;
            sx = 1;
        }
        if (sx == 0 && by >= 2 && by <= G.n[1] - 1) {
            const int c = column_of(G, srcx, by - 1);
            int lo = __ldg(&cs[c]);
            for (int dys = -1; dys <= 1; ++dys) {
                const int hi = __ldg(&cs[c + dys + 2]);
                for (int t = first_at_least(siz, lo, hi, izi - 1); t < hi; ++t) {
                    const int dzs = __ldg(&siz[t]) - izi;
                    if (dzs > 1) break;
                    if (dzs < -1 || t == self_t) continue;
                    f(t, ii - bx, dys, dzs, 0, 0);
                }
                lo = hi;
            }
        } else {
            for (int jj = by - 1; jj <= by + 1; ++jj) {
                int cc, ssx, sy;
                if (!stencil_row(G, ii, jj, cc, ssx, sy)) continue;
                const int t1 = __ldg(&cs[cc + 1]);
                for (int t = first_at_least(siz, __ldg(&cs[cc]), t1, izi - 1); t < t1; ++t) {
                    const int dzs = __ldg(&siz[t]) - izi;
                    if (dzs > 1) break;
                    if (dzs < -1 || t == self_t) continue;
                    if ((ssx | sy) && !image_in_row(S, G, a, __ldg(&S.perm[a][t]), ii, jj, ssx, sy)) continue;
                    f(t, ii - bx, jj - by, dzs, ssx, sy);
                }
            }
        }
    }
}

// Walk the stencil over the column-sorted copies when the state has them
// (SORTED), else over perm (callers that provide no sorted buffers).  f gets
// the candidate's FP32 offsets, a functor returning its slot, and the shifts.
template <bool SORTED, class F>
__device__ __forceinline__ void walk(const DevState &S, const DevGeom &G, int a, int i, int bx, int by, int izi,
                                     F &&f)
{
    if constexpr (SORTED) {
        visit_sorted(S, G, a, S.rank[a][i], bx, by, izi, [&](int t, int dxs, int dys, int dzs, int sx, int sy) {
            f(__ldg(&S.srel[a][t]), [&]() { return __ldg(&S.perm[a][t]); }, dxs, dys, dzs, sx, sy);
        });
    } else {
        visit_stencil(S, G, a, i, bx, by, izi, [&](int j, int dxs, int dys, int dzs, int sx, int sy) {
            f(__ldg(&S.rel[a][j]), [&]() { return j; }, dxs, dys, dzs, sx, sy);
        });
    }
}

// Grown-box bin (bx, by) of a slot from its column id.
__device__ __forceinline__ void col_to_bxy(const DevGeom &G, int col, int &bx, int &by)
{
    const int q = col - G.col_base;
    bx = q / G.n[1] + 1;
    by = q - (bx - 1) * G.n[1] + 1;
}

// ---- a stencil walk with one warp per neighbour column ----------------------
// A block holds NS slots (a multiple of 32) and nine warps; warp w walks neighbour column w
// (x offset w / 3 - 1, y offset w % 3 - 1, the order of the reference's list)
// for all of them, one slot per lane, 32 at a time, and stages the candidates that pass the
// caller's FP32 screen.  Nine short independent walks instead of one long
// chain of dependent loads per slot, and a warp's lanes read the same or
// adjacent columns.
constexpr int kWalkCols = 9;
constexpr int kWalkBlock = 32 * kWalkCols;
// Candidates staged per slot and column (sphere step, adjoint): one word
// each, in the room of six of two words.  A slot with more in some column is walked again by
// one lane while the block waits.  Adjoint of 20 000 / 50 000 spheres over 20 steps, ms: at 10
// a column 2.3 / 4.0 (6.3 / 6.3 with six), 2.7 / 4.8 at 15 (8.8 / 11.6; one thread per slot with
// its pairs staged by the block 6.5 / 7.7), 3.4 / 10.4 at 24 (15.4 / 22.4); 1.77 / 3.06 at 3 (1.76 /
// 3.06).  14: 3.5 / 10.4 at 24, 1.79 / 3.07 at 3.
constexpr int kWalkStage = 12;

// Blocks an SM a launch of `blocks` is compiled for, `least` to 5: as few (as many
// registers a thread, as few spills) as hold the grid in the fewest waves.  The
// blocks do about the same work, so a wave that is nearly empty costs as much
// as a full one.  Measured, us: k_sphere64w, 3 / 4 / 5 blocks an SM: 10 000 slots (3 blocks for
// each SM) 14.7 / 14.9 / 15.1, 15 000 (4) 22.7 / 15.3 / 16.9, 20 000 (5) 22.8 / 22.2 / 16.8, 25 000
// (6) 22.7 / 22.8 / 23.9, 32 768 (7) 29.5 / 23.1 / 25.1; the adjoint's two kernels with 3 and 2 / 3 and
// 3 / 5 and 5, forward and backward of 40 steps: 9000 slots 2634 / 2686 / 2923, 14 000 3171 / 2767 /
// 3252, 24 000 4651 / 4307 / 3595, 48 000 7500 / 7120 / 5794.
inline int wave_fit(int blocks, int least, int nsm)
{
    nsm = std::max(nsm, 1);
    int best = least;
    for (int k = least + 1; k <= 5; ++k)
        if ((blocks + nsm * k - 1) / (nsm * k) < (blocks + nsm * best - 1) / (nsm * best)) best = k;
    return best;
}

// One column of one slot: up to four entries are loaded before any is used.
// f(t, dzs) for every entry of z bins izi - 1 .. izi + 1 but the slot itself.
template <class F>
__device__ __forceinline__ void walk_column(const DevState &S, int a, int lo, int hi, int self_t, int izi, F &&f)
{
    const int *__restrict__ siz = S.siz[a];
    const float4 *__restrict__ srel = S.srel[a];
    if (hi - lo > 8) {  // (a column can be many bins tall)
        int l = lo, h = hi;
        while (l < h) {
            const int mid = (l + h) >> 1;
            if (__ldg(&siz[mid]) < izi - 1) l = mid + 1;
            else h = mid;
        }
        lo = l;
    }
    for (int t = lo; t < hi; t += 4) {
        int z[4];
        float4 q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int u = min(t + k, hi - 1);
            z[k] = __ldg(&siz[u]) - izi;
            q[k] = __ldg(&srel[u]);
        }
        if (z[0] > 1) break;  // sorted by z bin: the rest is out of reach
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (t + k < hi && z[k] >= -1 && z[k] <= 1 && t + k != self_t) f(t + k, q[k], z[k]);
    }
}

// A staged candidate: slot j and its code; in one word where the slots are below 2^28
// and the code is an image's (0..8).
__device__ __forceinline__ void put_entry(int2 &e, int j, int code) { e = make_int2(j, code); }
__device__ __forceinline__ void put_entry(unsigned &e, int j, int code) { e = (unsigned)j | ((unsigned)code << 28); }
__device__ __forceinline__ int2 get_entry(const int2 &e) { return e; }
__device__ __forceinline__ int2 get_entry(unsigned e) { return make_int2((int)(e & 0xfffffffu), (int)(e >> 28)); }

// Shared memory of a block's walk over NS slots (32 per pass of the warps): per
// column and slot the staged candidates (slot of the neighbour, image code)
// and, after walk_scan, the end of the column's run among the slot's pairs;
// the slots' first pairs.
template <int NS, int STAGE, class Entry = int2>
struct WalkMem {
    Entry stage[kWalkCols * NS][STAGE];
    int end[kWalkCols][NS];
    int first[NS + 1];
    int over[NS];  // the slot staged too many in some column: no pairs here
    int wsum[NS / 32];
};

// After every warp wrote its counts into end[w][slot] (more than STAGE, or
// more than `most` in all: overflow): the counts into runs, over the whole
// block (it synchronises).
template <int NS, int STAGE, class Entry>
__device__ __forceinline__ void walk_scan(WalkMem<NS, STAGE, Entry> &M, int most = 0x7fffffff)
{
    const int tid = threadIdx.x, lane = tid & 31;
    __syncthreads();
    int x = 0, mine = 0;
    if (tid < NS) {
        int run = 0;
        bool over = false;
#pragma unroll
        for (int w = 0; w < kWalkCols; ++w) {
            const int c = M.end[w][tid];
            over |= c > STAGE;
            run += c;
            M.end[w][tid] = run;
        }
        over |= run > most;
        M.over[tid] = over ? 1 : 0;
        mine = over ? 0 : run;
        x = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (NS == 32) M.first[tid + 1] = x;
        else if (lane == 31) M.wsum[tid >> 5] = x;
        if (tid == 0) M.first[0] = 0;
    }
    __syncthreads();
    if (NS > 32) {
        if (tid < NS) {
            for (int v = 0; v < (tid >> 5); ++v) x += M.wsum[v];
            M.first[tid + 1] = x;
        }
        __syncthreads();
    }
}

// Pair t of the block: its slot o and its staged candidate.
template <int NS, int STAGE, class Entry>
__device__ __forceinline__ int2 walk_pair(const WalkMem<NS, STAGE, Entry> &M, int t, int &o)
{
    o = 0;
#pragma unroll
    for (int d = NS / 2; d >= 1; d >>= 1)
        if (M.first[o + d] <= t) o += d;
    const int k = t - M.first[o];
    int w = 0, at = 0;
#pragma unroll
    for (int v = 0; v < kWalkCols - 1; ++v) {
        const int e = M.end[v][o];
        if (e <= k) {
            w = v + 1;
            at = e;
        }
    }
    return get_entry(M.stage[w * NS + o][k - at]);
}

// The column of warp w around slot i's bin (false: outside a closed face).
__device__ __forceinline__ bool walk_target(const DevState &S, const DevGeom &G, int a, int bx, int by, int w, int &ii,
                                            int &jj, int &lo, int &hi, int &sx, int &sy)
{
    ii = bx + w / 3 - 1;
    jj = by + w % 3 - 1;
    int cc;
    if (!stencil_row(G, ii, jj, cc, sx, sy)) return false;
    lo = __ldg(&S.colstart[a][cc]);
    hi = __ldg(&S.colstart[a][cc + 1]);
    return true;
}

// The FP32 screen of the FP64 pair walks: false only when the candidate is
// certainly beyond the cutoff r_i + r_j + bw, from the FP32 offsets to the bin
// corners (o: the neighbour bin's minus the slot's) with an absolute slack of 8
// ulp of the largest bin width that bounds their error; the FP64 gate decides
// the rest.
__device__ __forceinline__ bool near_pair32(const float4 me, const float4 q, float ox, float oy, float oz, float bwf,
                                            float slack)
{
    const float ex = (me.x - q.x) - ox;
    const float ey = (me.y - q.y) - oy;
    const float ez = (me.z - q.z) - oz;
    const float r2f = __fmaf_rn(ex, ex, __fmaf_rn(ey, ey, __fmul_rn(ez, ez)));
    const float lim = __fadd_rn(__fadd_rn(__fadd_rn(me.w, q.w), bwf), slack);
    return !(r2f > __fmul_rn(lim, lim));
}

__device__ __forceinline__ float screen_slack(const DevGeom &G)
{
    return 8.0f * 1.1920929e-7f * fmaxf(G.dxf[0], fmaxf(G.dxf[1], G.dxf[2]));
}

// The block's walk of buffer a: every slot's candidates staged, the runs of
// pairs set up (walk_scan).  own(s, i, colony): the first warp, for each slot.
template <int NS, int STAGE, class Entry, class Own>
__device__ __forceinline__ void walk_block(const DevState &S, int a, float bwf, WalkMem<NS, STAGE, Entry> &M, Own &&own)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int g = 0; g < NS; g += 32) {
        const int s = g + lane;
        const int i = blockIdx.x * NS + s;
        int cnt = 0;
        if (i < S.n) {
            const int col = colony_of(S.cbase, S.ncol, i);
            const DevGeom &G = S.geoms[col];
            int bx, by;
            col_to_bxy(G, S.col[a][i], bx, by);
            const int izi = S.iz[a][i];
            const float4 me = S.rel[a][i];
            const int self_t = S.rank[a][i];
            if (w == 0) own(s, i, col);
            const float slack = screen_slack(G), dzb = G.dxf[2];
            const float ox = (float)(w / 3 - 1) * G.dxf[0], oy = (float)(w % 3 - 1) * G.dxf[1];
            int ii, jj, lo, hi, sx, sy;
            if (walk_target(S, G, a, bx, by, w, ii, jj, lo, hi, sx, sy)) {
                walk_column(S, a, lo, hi, self_t, izi, [&](int t, const float4 q, int dzs) {
                    if (!near_pair32(me, q, ox, oy, (float)dzs * dzb, bwf, slack)) return;
                    const int j = __ldg(&S.perm[a][t]);
                    if ((sx | sy) && !image_in_row(S, G, a, j, ii, jj, sx, sy)) return;
                    if (cnt < STAGE) put_entry(M.stage[w * NS + s][cnt], j, (sx + 1) * 3 + (sy + 1));
                    ++cnt;
                });
            }
        }
        M.end[w][s] = cnt;
    }
    walk_scan(M);
}

// The block's staged pairs, one per thread: eval(o, e, t) computes pair e of
// slot o into t[NT] (false: no term); add(t, stride) adds one pair's terms to
// the sums of slot threadIdx.x, in staging order (the slots' threads are the
// block's first NS).  term: NT x kWalkBlock values.
template <int NT, int NS, int STAGE, class Entry, class Eval, class Add>
__device__ __forceinline__ void walk_pairs(const WalkMem<NS, STAGE, Entry> &M, double *term, unsigned char *opass, Eval &&eval,
                                           Add &&add)
{
    const int tid = threadIdx.x;
    const int total = M.first[NS];
    for (int t0 = 0; t0 < total; t0 += kWalkBlock) {
        const int t = t0 + tid;
        if (t < total) {
            int o;
            const int2 e = walk_pair(M, t, o);
            double tt[NT];
            for (int c = 0; c < NT; ++c) tt[c] = 0.0;
            opass[tid] = eval(o, e, tt) ? 1 : 0;
            for (int c = 0; c < NT; ++c) term[c * kWalkBlock + tid] = tt[c];
        }
        __syncthreads();
        if (tid < NS) {
            const int k1 = min(M.first[tid + 1], t0 + kWalkBlock);
            for (int k = max(M.first[tid], t0); k < k1; ++k)
                if (opass[k - t0]) add(term + (k - t0));
        }
        if (t0 + kWalkBlock < total) __syncthreads();
    }
}

// Counters of a slot at (x, y, z) in bins bx, by: out-of-domain z, non-finite
// positions, images that leave their halo cell.
__device__ __forceinline__ void count_slot(const DevState &S, const DevGeom &G, double x, double y, double z, int bx,
                                           int by, bool count_domain)
{
    if (count_domain) {
        // inside for certain from the FP32 values (truncated z within 2^-21 of the
        // magnitudes), else the FP64 test
        const float zf = d2f_trunc(z);
        const float m = 4.8e-7f * (fabsf(zf) + fabsf(G.plof[2]) + fabsf(G.phif[2]));
        const bool sure = G.phif[2] > G.plof[2] && zf - m > G.plof[2] && zf + m < G.phif[2];
        if (!sure && !(z >= G.plo[2] && z < G.phi[2])) atomicAdd(&S.cnt->out_of_domain, 1ULL);
    }
    if (!finite_bits(x) || !finite_bits(y) || !finite_bits(z)) atomicAdd(&S.cnt->nonfinite, 1ULL);
    if (G.per[0] && (bx == 1 || bx == G.n[0])) {
        const int sx = (bx == 1) ? 1 : -1;
        const int gb = image_bin(G, 0, image_coord(x, G.len[0], sx));
        if (gb != (sx > 0 ? G.n[0] + 1 : 0)) atomicAdd(&S.cnt->edge_ghost, 1ULL);
    }
    if (G.per[1] && (by == 1 || by == G.n[1])) {
        const int sy = (by == 1) ? 1 : -1;
        const int gb = image_bin(G, 1, image_coord(y, G.len[1], sy));
        if (gb != (sy > 0 ? G.n[1] + 1 : 0)) atomicAdd(&S.cnt->edge_ghost, 1ULL);
    }
}

// Bin a slot at position (x, y, z): column and z bin into buffer bb, FP32
// offsets from the bin corner into buffer rb, column count; flag
// out-of-domain z, images that leave their halo cell, and non-finite positions.
// place_slot does the same for bins already known.
__device__ __forceinline__ void place_slot(const DevState &S, const DevGeom &G, int i, double x, double y,
                                           double z, double r, int bb, int rb, int bx, int by, int bz,
                                           bool count_domain, bool count_col)
{
    const int c = column_of(G, bx, by);
    S.col[bb][i] = c;
    S.iz[bb][i] = bz;
    // bin corners from the geometry's table (the same FP64 formula, evaluated
    // once on the host), the conversions and tests from the bits: FP64
    // arithmetic here is the three differences (GB300 issues FP64 at a small
    // fraction of the FP32 rate)
    auto corner = [&](int d, int bin) {
        return (bin >= 1 && bin <= G.ncorner[d]) ? G.corner[d][bin - 1] : G.plo[d] + (double)(bin - 1) * G.dx[d];
    };
    const double cx = corner(0, bx), cy = corner(1, by), cz = corner(2, bz);
    S.rel[rb][i] = make_float4(d2f_rn(x - cx), d2f_rn(y - cy), d2f_rn(z - cz), d2f_rn(r));
    if (count_col) atomicAdd(&S.colcnt[c], 1);
    count_slot(S, G, x, y, z, bx, by, count_domain);
}

__device__ __forceinline__ void rebin_slot_into(const DevState &S, const DevGeom &G, int i, double x, double y,
                                                double z, double r, int bb, int rb, bool count_domain = true,
                                                bool count_col = true)
{
    const int bx = bin_of_fast(x, G.plo[0], G.dxi[0], G.plof[0], G.dxif[0], 1, G.n[0]);
    const int by = bin_of_fast(y, G.plo[1], G.dxi[1], G.plof[1], G.dxif[1], 1, G.n[1]);
    const int bz = bin_of_fast(z, G.plo[2], G.dxi[2], G.plof[2], G.dxif[2], 1, G.n[2]);
    place_slot(S, G, i, x, y, z, r, bb, rb, bx, by, bz, count_domain, count_col);
}

// Bin a slot into buffer b (bins and offsets).
__device__ __forceinline__ void rebin_slot(const DevState &S, const DevGeom &G, int i, double x, double y,
                                           double z, double r, int b)
{
    rebin_slot_into(S, G, i, x, y, z, r, b, b);
}

// Growth-surface cubic law of one site at height z
// (bmx_cell_interaction_K.H:1019-1030, :1099-1121).  The branches above and
// below the surface are one product c t t w with selected factors (the same
// roundings; a warp whose lanes differ would issue both branches), and the
// comparisons read the bits: FP64 instructions are what the callers run out of.
__device__ __forceinline__ double wall_law(double z, double rS, const DevParams &P)
{
    const double dz = z - P.z_wall;
    const double rA = rS + P.z_bw;
    const bool below = le_bits(dz, 0.0);
    const bool near = !below && lt_bits(dz, rA) && !is_nan_bits(dz);
    const double t = near ? dz - rA : rA;
    const double w = near ? dz - rS : rS;
    double v = (near ? -P.z_k : P.z_k) * t * t * w;
    if (!below && !near) v = 0.0;
    v -= P.z_gk * rA * rA * rS;
    return v;
}

// The FP64 term of a sphere pair at separation (dx, dy, dz), in the reference's
// operation order: false when the pair is not in the neighbour list or beyond
// the cutoff, else the three products F u_x, F u_y, F u_z that the gather adds.
__device__ __forceinline__ bool sphere_pair64(const DevParams &P, int nbh_trivial, double dx, double dy, double dz,
                                              double ri, double rj, double *t)
{
    const double r2 = dx * dx + dy * dy + dz * dz;
    if (!nbh_trivial && !(r2 <= P.nbh)) return false;  // not in the neighbour list
    const double rlm = ri + rj + P.bw;                  // maxInteractionDistance
    if (!le_nonneg(r2, (rlm - kSmall) * (rlm - kSmall))) return false;
    const double rS = ri + rj;
    const double rA = rS + P.bw;
    Divisor by;
    const double rn = sqrt_rn(r2, &by);
    const double ux = div_by(dx, by), uy = div_by(dy, by), uz = div_by(dz, by);
    const double F = lt_bits(rn, rA) ? -P.k * (rn - rA) * (rn - rA) * (rn - rS) : 0.0;
    t[0] = F * ux;
    t[1] = F * uy;
    t[2] = F * uz;
    return true;
}

// Exact float -> double conversion with integer operations (GB300's FP64
// pipe is the scarce resource here), on the two 32-bit words: for a normal
// float the high word is the sign, then exponent and mantissa shifted down by
// three with the exponent rebased by 1023 - 127, and the low word the last
// three mantissa bits.  Subnormal floats flush to a signed zero; infinities
// and NaNs keep their payload.
__device__ __forceinline__ double f2d_int(float f)
{
    const unsigned u = __float_as_uint(f);
    const unsigned sgn = u & 0x80000000u, a = u & 0x7fffffffu;
    unsigned hi = sgn | ((a >> 3) + 0x38000000u);
    unsigned lo = u << 29;
    if (a < 0x00800000u) {
        hi = sgn;
        lo = 0u;
    } else if (a >= 0x7f800000u) {
        hi = sgn | 0x7ff00000u | ((a & 0x7fffffu) >> 3);
    }
    return __hiloint2double((int)hi, (int)lo);
}

// growth-surface cubic law in FP32 (bmx_cell_interaction_K.H:1019-1030)
__device__ __forceinline__ float wall_law32(float dz, float rS, float zk, float zbw, float zg)
{
    const float rA = rS + zbw;
    float v;
    if (dz > 0.0f && dz < rA) v = -zk * (dz - rA) * (dz - rA) * (dz - rS);
    else if (dz <= 0.0f) v = zk * rA * rA * rS;
    else v = 0.0f;
    return v - zg * zk * rA * rA * rS;
}

__device__ __forceinline__ const DevGeom &geom_of(const DevState &S, int i)
{
    return S.geoms[colony_of(S.cbase, S.ncol, i)];
}

}  // namespace bmxg
