// k_sphere.cu -- fused sphere step: force gather over the neighbour stencil,
// growth-surface force, overdamped update, periodic wrap and rebin, one pass.
//
// Replaces, for YEAST-only states, the force lambda of
// src/des/bmx_pc_interaction.cpp:170-279 (evaluateForce's sphere branch,
// src/chemistry/bmx_cell_interaction_K.H:243-276, and evaluateSurfaceForce's
// sphere branch, :1009-1030) and the update lambda (:311-436), followed by
// the periodic wrap of the trailing Redistribute (:485-486).
//
// Forms:
//  FP64  (plain, k_sphere64) every pair that can pass the reference's cutoff
//        test is evaluated in FP64 with the reference's operation order (this
//        file is compiled with -fmad=false), accumulated in list order: the
//        result is bit-identical to the host oracle.  Pairs are first
//        screened in FP32 from the bin-relative offsets with an absolute
//        slack that bounds the FP32 error, so only pairs that are certainly
//        beyond the cutoff skip the FP64 test.
//  FP32F (precision form, k_sphere32) pair math and wall law in FP32 on
//        FP64-differenced bin-relative offsets; the position accumulation
//        stays FP64.  GB300 issues FP64 at 1/64 of the FP32 rate, so the
//        per-particle epilogue avoids FP64 too: the bin-relative offsets are
//        advanced in FP32 and re-derived exactly from the FP64 position
//        (exact FP64 re-binning) every kResyncEvery-th step and whenever a
//        particle comes within a guard band of a bin face, where its bin
//        might change.  Away from the faces the FP64 bin cannot change, so
//        the neighbour lists stay exactly the reference's.
// Roofline: HBM / L2 bound gather; no dense contraction, so no tensor cores.
#include <atomic>

#include "bmxg_pdl.cuh"
#include "bmxg_stencil.cuh"

namespace bmxg {

namespace {

// The FP64 pair term of slot i (at xi, yi, zi, radius ri, colony geometry
// G) from neighbour j under image shift (sx, sy).
__device__ __forceinline__ bool sphere_term64(const DevState &S, const DevGeom &G, const DevParams &P, int a,
                                              double xi, double yi, double zi, double ri, int j, int sx, int sy,
                                              double *t)
{
    const double xj = sx ? image_coord(S.x[a][j], G.len[0], sx) : S.x[a][j];
    const double yj = sy ? image_coord(S.y[a][j], G.len[1], sy) : S.y[a][j];
    return sphere_pair64(P, G.nbh_trivial, xi - xj, yi - yj, zi - S.z[a][j], ri, S.rad[j], t);
}

// FP64 plain step.  Each thread walks its slot's stencil and screens the
// candidates in FP32 (FP32 and integer work); the few that can pass the
// cutoff (about 1.3 per slot on the colonies) are staged in shared memory,
// and the block then evaluates its slots' staged pairs together, one per
// thread, so that the FP64 gate, square root and divisions run in full warps
// (GB300 issues FP64 at 2 lanes per clock per SM whatever the mask: a thread
// walking its own candidates keeps 8 of 32 lanes busy in those instructions),
// and a warp whose share of a round is empty skips it.  Each slot then adds
// its pairs' terms in walk order -- the same FP64 values in the same order as
// a walk that evaluates each pair when it meets it, so the result stays
// bit-identical to the oracle.  A slot with more than kStage64 candidates walks
// again and evaluates them itself, in order.
// Bound: the walk's loads and instructions (FP64 pipe 37 % busy).  The walk over
// the sorted copies takes a column at a time, four entries in flight, and three blocks of
// 256 threads fit an SM (80 registers): 500 000 slots 223 -> 172 us, 2 million 687 -> 507,
// 688 000 in 64 colonies 379 -> 245 against entry by entry with the crowded slots'
// evaluation inside the walk (128 registers).  64 registers: 183; the next column's bounds
// a column ahead: 179; three columns unrolled: 216.
// A staged candidate is one word: its slot (below 2^30) and whether it is an image along
// x and y; which one the slot's own bin says (a periodic axis has three bins or more).
// 24 of them in the room of 12 of two words, whose crowded slots' second walk cost more than
// staging saved: a load and 24 steps of 50 000 spheres, 15 / 24 a column, 3.51 / 5.06 -> 2.03 /
// 2.72 ms, 2 million 29.1 / 60.2 -> 28.0 / 40.9; 3 a column 1.18 / 14.3 -> 1.18 / 14.4.
constexpr int kStage64 = 24;

// dynamic shared memory of k_sphere64 for a block of `block` threads
__host__ __device__ constexpr size_t sphere64_smem(int block)
{
    return (size_t)block * (kStage64 * sizeof(unsigned) + 4 * sizeof(double) + 3 * sizeof(double) + 4 * sizeof(int)) +
           2 * 32 * sizeof(int);
}

template <bool SORTED>
__global__ void __launch_bounds__(256, 3) k_sphere64(const DevState S, const DevParams P, double dt, int a)
{
    // per thread: its staged candidates (j, image code); its slot's position,
    // radius, colony and run of staged pairs (for the block's evaluation);
    // one round's terms and gate results
    extern __shared__ __align__(16) unsigned char sm64[];
    const int B = blockDim.x, tid = threadIdx.x;
    const int lane = tid & 31, w = tid >> 5, nw = B >> 5;
    unsigned *stage = reinterpret_cast<unsigned *>(sm64);
    double *opos = reinterpret_cast<double *>(stage + (size_t)B * kStage64);  // 4 per thread: x, y, z, r
    double *term = opos + 4 * B;                                               // 3 per thread
    int *ocol = reinterpret_cast<int *>(term + 3 * B);
    int *orun = ocol + B;   // first staged pair of the slot in the block's run
    int *oimg = orun + B;   // the shifts its images have: (sx + 1) * 3 + (sy + 1)
    int *opass = oimg + B;  // the round's gate result per thread
    int *wsum = opass + B;  // per warp: staged pairs, then their exclusive scan
    const int b = a ^ 1;
    const float bwf = P.bw32;
    if (SORTED) chain_wait();
    for (int base = blockIdx.x * B; base < S.n; base += gridDim.x * B) {
        const int i = base + tid;
        const bool act = i < S.n;
        double xi = 0.0, yi = 0.0, zi = 0.0, ri = 0.0;
        double fx = 0.0, fy = 0.0, fz = 0.0;
        int col = 0, cnt = 0, bx = 1, by = 1;
        if (act) {
            col = colony_of(S.cbase, S.ncol, i);
            const DevGeom &G = S.geoms[col];
            col_to_bxy(G, S.col[a][i], bx, by);
            const int izi = S.iz[a][i];
            xi = S.x[a][i];
            yi = S.y[a][i];
            zi = S.z[a][i];
            ri = S.rad[i];
            const float4 me = S.rel[a][i];
            const float slack = screen_slack(G), dzb = G.dxf[2];
            unsigned *mine = stage + (size_t)tid * kStage64;
            auto take = [&](int j, int sx, int sy) {
                if (cnt < kStage64) mine[cnt] = (unsigned)j | (sx ? 1u << 30 : 0u) | (sy ? 1u << 31 : 0u);
                ++cnt;
            };
            if constexpr (SORTED) {
                const int self_t = S.rank[a][i];
                for (int c = 0; c < kWalkCols; ++c) {
                    const float ox = (float)(c / 3 - 1) * G.dxf[0], oy = (float)(c % 3 - 1) * G.dxf[1];
                    int ii, jj, lo, hi, sx, sy;
                    if (!walk_target(S, G, a, bx, by, c, ii, jj, lo, hi, sx, sy)) continue;
                    walk_column(S, a, lo, hi, self_t, izi, [&](int t, const float4 q, int dzs) {
                        if (!near_pair32(me, q, ox, oy, (float)dzs * dzb, bwf, slack)) return;
                        const int j = __ldg(&S.perm[a][t]);
                        if ((sx | sy) && !image_in_row(S, G, a, j, ii, jj, sx, sy)) return;
                        take(j, sx, sy);
                    });
                }
            } else {
                walk<false>(S, G, a, i, bx, by, izi, [&](const float4 q, auto slot, int dxs, int dys, int dzs, int sx,
                                                         int sy) {
                    if (near_pair32(me, q, (float)dxs * G.dxf[0], (float)dys * G.dxf[1], (float)dzs * dzb, bwf, slack))
                        take(slot(), sx, sy);
                });
            }
            if (cnt > kStage64)  // too many for the stage: the whole walk, each pair evaluated as it is met
                walk<SORTED>(S, G, a, i, bx, by, izi, [&](const float4 q, auto slot, int dxs, int dys, int dzs, int sx,
                                                          int sy) {
                    if (!near_pair32(me, q, (float)dxs * G.dxf[0], (float)dys * G.dxf[1], (float)dzs * dzb, bwf, slack))
                        return;
                    double t[3];
                    if (sphere_term64(S, G, P, a, xi, yi, zi, ri, slot(), sx, sy, t)) {
                        fx += t[0];
                        fy += t[1];
                        fz += t[2];
                    }
                });
        }
        // the block's run of staged pairs: slot by slot in thread order
        const int xl = (cnt <= kStage64) ? cnt : 0;
        int xo = xl;
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, xo, d);
            if (lane >= d) xo += v;
        }
        if (lane == 31) wsum[w] = xo;
        opos[4 * tid] = xi;
        opos[4 * tid + 1] = yi;
        opos[4 * tid + 2] = zi;
        opos[4 * tid + 3] = ri;
        ocol[tid] = col;
        oimg[tid] = (bx == 1 ? 0 : 6) + (by == 1 ? 0 : 2);
        __syncthreads();
        if (tid == 0) {
            int run = 0;
            for (int v = 0; v < nw; ++v) {
                const int c = wsum[v];
                wsum[32 + v] = run;
                run += c;
            }
            wsum[31] = run;  // (nw <= 8: slot 31 is free) the block's total
        }
        __syncthreads();
        const int xt = wsum[31];
        xo += wsum[32 + w] - xl;
        orun[tid] = xo;
        __syncthreads();
        for (int t0 = 0; t0 < xt; t0 += B) {
            const int t = t0 + tid;
            int pass = 0;
            double tt[3] = {0.0, 0.0, 0.0};
            if (t0 + 32 * w < xt) {  // a warp with no pair in this round skips it
                if (t < xt) {
                    int o = 0;  // the slot that owns pair t: the last thread whose run starts at or before t
                    for (int s2 = 1 << (31 - __clz(max(B - 1, 1))); s2 >= 1; s2 >>= 1)
                        if (o + s2 < B && orun[o + s2] <= t) o += s2;
                    const unsigned e = stage[(size_t)o * kStage64 + (t - orun[o])];
                    const int im = oimg[o];
                    pass = sphere_term64(S, S.geoms[ocol[o]], P, a, opos[4 * o], opos[4 * o + 1], opos[4 * o + 2],
                                         opos[4 * o + 3], (int)(e & 0x3fffffffu), (e >> 30) & 1u ? im / 3 - 1 : 0,
                                         e >> 31 ? im % 3 - 1 : 0, tt)
                               ? 1
                               : 0;
                }
            }
            term[3 * tid] = tt[0];
            term[3 * tid + 1] = tt[1];
            term[3 * tid + 2] = tt[2];
            opass[tid] = pass;
            __syncthreads();
            const int k1 = min(xo + xl, t0 + B);
            for (int k = max(xo, t0); k < k1; ++k) {
                if (!opass[k - t0]) continue;
                fx += term[3 * (k - t0)];
                fy += term[3 * (k - t0) + 1];
                fz += term[3 * (k - t0) + 2];
            }
            __syncthreads();
        }
        if (act) {
            const DevGeom &G = S.geoms[col];
            // evaluateSurfaceForce, sphere branch: vcom = (0, 0, wall), vrot = 0
            const double vx = plus_zero(fx);
            const double vy = plus_zero(fy);
            const double vz = fz + wall_law(zi, ri, P);
            double nx = xi + dt * vx;
            double ny = yi + dt * vy;
            const double nz = zi + dt * vz;
            if (G.per[0]) nx = wrap1(nx, G.plo[0], G.phi[0], G.len[0]);
            if (G.per[1]) ny = wrap1(ny, G.plo[1], G.phi[1], G.len[1]);
            S.x[b][i] = nx;
            S.y[b][i] = ny;
            S.z[b][i] = nz;
            S.vx[i] = vx;
            S.vy[i] = vy;
            S.vz[i] = vz;
            rebin_slot(S, G, i, nx, ny, nz, ri, b);
        }
        __syncthreads();  // the next pass reuses the stage and the slot records
    }
}

// The same step with one warp per neighbour column (bmxg_stencil.cuh): the
// staged pairs one per thread over the block, the sums and the slots' updates
// in its first warps.  Same pairs, same FP64 operations, same order of the sums.
template <int NS, int STAGE, int RESIDENT>
__global__ void __launch_bounds__(kWalkBlock, RESIDENT) k_sphere64w(const DevState S, const DevParams P, double dt, int a)
{
    extern __shared__ __align__(16) unsigned char smw[];
    auto &M = *reinterpret_cast<WalkMem<NS, STAGE, unsigned> *>(smw);
    __shared__ double opos[NS][4];
    __shared__ int ocol[NS];
    __shared__ double term[3 * kWalkBlock];
    __shared__ unsigned char opass[kWalkBlock];
    const int tid = threadIdx.x;
    const int b = a ^ 1;
    chain_wait();
    walk_block(S, a, P.bw32, M, [&](int s, int i, int col) {
        opos[s][0] = S.x[a][i];
        opos[s][1] = S.y[a][i];
        opos[s][2] = S.z[a][i];
        opos[s][3] = S.rad[i];
        ocol[s] = col;
    });
    double fx = 0.0, fy = 0.0, fz = 0.0;
    walk_pairs<3>(
        M, term, opass,
        [&](int o, int2 e, double *t) {
            return sphere_term64(S, S.geoms[ocol[o]], P, a, opos[o][0], opos[o][1], opos[o][2], opos[o][3], e.x,
                                 e.y / 3 - 1, e.y % 3 - 1, t);
        },
        [&](const double *t) {
            fx += t[0];
            fy += t[kWalkBlock];
            fz += t[2 * kWalkBlock];
        });
    const int i = blockIdx.x * NS + tid;
    if (tid >= NS || i >= S.n) return;
    const DevGeom &G = S.geoms[ocol[tid]];
    const double xi = opos[tid][0], yi = opos[tid][1], zi = opos[tid][2], ri = opos[tid][3];
    if (M.over[tid]) {  // a crowded column: the whole walk, each pair evaluated as it is met
        int bx, by;
        col_to_bxy(G, S.col[a][i], bx, by);
        const float4 me = S.rel[a][i];
        const float slack = screen_slack(G);
        walk<true>(S, G, a, i, bx, by, S.iz[a][i], [&](const float4 q, auto slot, int dxs, int dys, int dzs, int sx,
                                                       int sy) {
            if (!near_pair32(me, q, (float)dxs * G.dxf[0], (float)dys * G.dxf[1], (float)dzs * G.dxf[2], P.bw32, slack))
                return;
            double t[3];
            if (sphere_term64(S, G, P, a, xi, yi, zi, ri, slot(), sx, sy, t)) {
                fx += t[0];
                fy += t[1];
                fz += t[2];
            }
        });
    }
    // evaluateSurfaceForce, sphere branch: vcom = (0, 0, wall), vrot = 0
    const double vx = plus_zero(fx);
    const double vy = plus_zero(fy);
    const double vz = fz + wall_law(zi, ri, P);
    double nx = xi + dt * vx;
    double ny = yi + dt * vy;
    const double nz = zi + dt * vz;
    if (G.per[0]) nx = wrap1(nx, G.plo[0], G.phi[0], G.len[0]);
    if (G.per[1]) ny = wrap1(ny, G.plo[1], G.phi[1], G.len[1]);
    S.x[b][i] = nx;
    S.y[b][i] = ny;
    S.z[b][i] = nz;
    S.vx[i] = vx;
    S.vy[i] = vy;
    S.vz[i] = vz;
    rebin_slot(S, G, i, nx, ny, nz, ri, b);
}

template <bool SORTED>
__global__ void __launch_bounds__(256, 5) k_sphere32(const DevState S, const DevParams P, float dtf, int a,
                                                  int resync)
{
    const int b = a ^ 1;
    // the FP32 roundings come from the host (a conversion is an FP64-pipe
    // instruction, and threads without a slot would issue them too)
    const float bwf = P.bw32, kf = P.k32;
    const float zkf = P.z_k32, zbwf = P.z_bw32, zgf = P.z_g32;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n; i += gridDim.x * blockDim.x) {
        const DevGeom &G = geom_of(S, i);
        const int col = S.col[a][i];
        int bx, by;
        col_to_bxy(G, col, bx, by);
        const int izi = S.iz[a][i];
        const float4 me = S.rel[a][i];
        const float dxb = G.dxf[0], dyb = G.dxf[1], dzb = G.dxf[2];
        float gx = 0.0f, gy = 0.0f, gz = 0.0f;
        walk<SORTED>(S, G, a, i, bx, by, izi, [&](const float4 q, auto slot, int dxs, int dys, int dzs, int sx, int sy) {
            const float ex = (me.x - q.x) - (float)dxs * dxb;
            const float ey = (me.y - q.y) - (float)dys * dyb;
            const float ez = (me.z - q.z) - (float)dzs * dzb;
            const float r2f = __fmaf_rn(ex, ex, __fmaf_rn(ey, ey, __fmul_rn(ez, ez)));
            const float rAf = __fadd_rn(__fadd_rn(me.w, q.w), bwf);
            if (!(r2f < __fmul_rn(rAf, rAf))) return;
            if (!G.nbh_trivial) {  // BMXCheckPair, exactly (FP64)
                const int j = slot();
                const double xj = sx ? S.x[a][j] + (double)sx * G.len[0] : S.x[a][j];
                const double yj = sy ? S.y[a][j] + (double)sy * G.len[1] : S.y[a][j];
                const double dx = S.x[a][i] - xj, dy = S.y[a][i] - yj, dz = S.z[a][i] - S.z[a][j];
                if (!(dx * dx + dy * dy + dz * dz <= P.nbh)) return;
            }
            const float inv = rsqrtf(r2f);
            const float rn = __fmul_rn(r2f, inv);
            const float rSf = __fadd_rn(me.w, q.w);
            const float d1 = __fsub_rn(rn, rAf);
            const float F = __fmul_rn(__fmul_rn(__fmul_rn(-kf, d1), d1), __fsub_rn(rn, rSf));
            const float Fi = __fmul_rn(F, inv);
            gx = __fmaf_rn(Fi, ex, gx);
            gy = __fmaf_rn(Fi, ey, gy);
            gz = __fmaf_rn(Fi, ez, gz);
        });
        // wall: height above the surface from the bin face's height (float
        // pair) and the FP32 offset, FP64 only where no table entry exists
        float dzw;
        if (izi < G.nwz) {
            const float2 c = G.wz[izi];
            dzw = (c.x + me.z) + c.y;
        } else {
            dzw = (float)(S.z[a][i] - P.z_wall);
        }
        const float vx = gx, vy = gy, vz = gz + wall_law32(dzw, me.w, zkf, zbwf, zgf);
        const float ix = dtf * vx, iy = dtf * vy, iz = dtf * vz;
        // FP64 position accumulation
        double nx = S.x[a][i] + f2d_int(ix);
        double ny = S.y[a][i] + f2d_int(iy);
        const double nz = S.z[a][i] + f2d_int(iz);
        S.vxf[i] = vx;
        S.vyf[i] = vy;
        S.vzf[i] = vz;
        // FP32 offsets; exact FP64 re-binning near a bin face or on re-sync steps
        const float4 r = make_float4(me.x + ix, me.y + iy, me.z + iz, me.w);
        const float g0 = 1e-4f * dxb, g1 = 1e-4f * dyb, g2 = 1e-4f * dzb;
        const bool inside = !resync && r.x >= g0 && r.x <= dxb - g0 && r.y >= g1 && r.y <= dyb - g1 &&
                            r.z >= g2 && r.z <= dzb - g2;
        if (inside) {
            S.x[b][i] = nx;
            S.y[b][i] = ny;
            S.z[b][i] = nz;
            S.rel[b][i] = r;
            S.col[b][i] = col;
            S.iz[b][i] = izi;
            atomicAdd(&S.colcnt[col], 1);
            if (!isfinite(vx + vy + vz)) atomicAdd(&S.cnt->nonfinite, 1ULL);
        } else {
            if (G.per[0]) nx = wrap1(nx, G.plo[0], G.phi[0], G.len[0]);
            if (G.per[1]) ny = wrap1(ny, G.plo[1], G.phi[1], G.len[1]);
            S.x[b][i] = nx;
            S.y[b][i] = ny;
            S.z[b][i] = nz;
            rebin_slot(S, G, i, nx, ny, nz, S.rad[i], b);
        }
    }
}

}  // namespace

// A kernel's dynamic shared memory above the default 48 KB: the attribute,
// once per device (known: a bit per device, set twice at worst).
template <class K>
static void allow_smem_once(K kernel, size_t bytes, std::atomic<unsigned long long> &known)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    if (dev < 64 && ((known.load(std::memory_order_relaxed) >> dev) & 1ull)) return;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess &&
        dev < 64)
        known.fetch_or(1ull << dev, std::memory_order_relaxed);
}

// Which FP64 kernel a sorted state takes: one warp per neighbour column where
// the slots are too few for a thread each to hide the walk's dependent loads,
// one thread per slot above, where the walk's instructions count and not its
// latency.  Measured, us a load and 40 steps, one thread per slot / one warp per
// column, 3 and 10 slots a column: 16 000 slots 1365, 2068 / 911, 1086, 32 768 1597,
// 2303 / 1402, 1654, 48 000 1776, 2485 / 1651, 2007, 56 000 1866, 2694 / 1904, 2317, 80 000
// 1954, 2884 / 2400, 3018.
constexpr int kColumnSlots64 = 49152;
static_assert(kColumnSlots64 < (1 << 28), "a staged slot in 28 bits");

int launch_sphere_step(const DevState &S, const DevParams &P, double dt, int a, int precision, int grid,
                       int block, cudaStream_t st, int resync, bool pinned)
{
    const bool sorted = S.srel[a] != nullptr;  // the context keeps sorted copies; bare callers do not
    if (precision == BMXG_FP64_FORM) {
        if (sorted && !pinned && S.n <= kColumnSlots64) {
            const int blocks = (S.n + 31) / 32, fit = wave_fit(blocks, 3, S.nsm);
            launch_after(fit == 3 ? k_sphere64w<32, kWalkStage, 3>
                                  : (fit == 4 ? k_sphere64w<32, kWalkStage, 4> : k_sphere64w<32, kWalkStage, 5>),
                         blocks, kWalkBlock, sizeof(WalkMem<32, kWalkStage, unsigned>), st, S, P, dt, a);
            return 1;
        }
        // (block a multiple of 32, at most 256: the block stages and evaluates its pairs together)
        const size_t smem = sphere64_smem(block);
        if (sorted) {
            static std::atomic<unsigned long long> known{0};
            allow_smem_once(k_sphere64<true>, sphere64_smem(256), known);
            launch_after(k_sphere64<true>, grid, block, smem, st, S, P, dt, a);
        } else {
            static std::atomic<unsigned long long> known{0};
            allow_smem_once(k_sphere64<false>, sphere64_smem(256), known);
            k_sphere64<false><<<grid, block, smem, st>>>(S, P, dt, a);
        }
    } else {
        if (sorted) k_sphere32<true><<<grid, block, 0, st>>>(S, P, (float)dt, a, resync);
        else k_sphere32<false><<<grid, block, 0, st>>>(S, P, (float)dt, a, resync);
    }
    return 1;
}

}  // namespace bmxg
