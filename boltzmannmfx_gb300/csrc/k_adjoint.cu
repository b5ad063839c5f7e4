// k_adjoint.cu -- the differentiation form: an FP64 sphere step with the
// contact-parameter extensions, and its hand-written adjoint.
//
// Forward law (spheres; the reference law of
// src/chemistry/bmx_cell_interaction_K.H:243-276 and :1009-1030 when
// damping = mu = adhesion = 0, bit for bit):
//   f(r)   = -k (r - rA)^2 (r - rS) - k bw abar (r - rA)^2        r < rA
//   Ft(r)  = f(r) / (1 + gamma (m_i + m_j))      two-body overdamped dashpot
//   v_i    = m_i sum_j Ft(r_ij) u_ij + wall(z_i) e_z
//   x_i'   = x_i + dt v_i                        (then the periodic wrap)
// with abar = (a_i + a_j)/2 (per-particle adhesion energy, in units of the
// band's spring energy), m_i = 1/(6 pi mu r_i) for mu > 0 and 1 otherwise
// (drag folded into k, as the reference does).
//
// Adjoint of one step, lam' = dL/dx_{t+1}:
//   lam_k = lam'_k + dt [ sum_j J_kj (m_k lam'_k - m_j lam'_j) + wall'(z_k) lam'_kz e_z ]
//   J = Ft' u u^T + (Ft / r)(I - u u^T)   (symmetric, J_kj = J_jk)
// a gather over the same neighbour walk as the forward step -- no atomics.
// Parameter gradients are accumulated per slot across steps (deterministic)
// and reduced once at the end.
#include <algorithm>

#include "bmxg_pdl.cuh"
#include "bmxg_stencil.cuh"

namespace bmxg {

namespace {

struct PairLaw {
    double f, df, fk, fa;  // f, df/dr, df/dk, df/dabar
};

__device__ __forceinline__ PairLaw pair_law(double r, double rS, double rA, double k, double bw, double abar)
{
    PairLaw q{0.0, 0.0, 0.0, 0.0};
    if (r < rA) {
        const double e = r - rA, g = r - rS;
        q.f = -k * e * e * g - k * bw * abar * e * e;
        q.df = -k * (2.0 * e * g + e * e) - 2.0 * k * bw * abar * e;
        q.fk = -e * e * g - bw * abar * e * e;
        q.fa = -k * bw * e * e;
    }
    return q;
}

__device__ __forceinline__ double mobility_of(double r, double mu)
{
    return mu > 0.0 ? div_rn(1.0, 6.0 * kPi * mu * r) : 1.0;
}

__device__ __forceinline__ double wall_slope(double z, double rS, const DevParams &P)
{
    const double dz = z - P.z_wall;
    const double rA = rS + P.z_bw;
    if (dz > 0.0 && dz < rA) return -P.z_k * (2.0 * (dz - rA) * (dz - rS) + (dz - rA) * (dz - rA));
    return 0.0;
}

// near_pair32 by bin offsets
__device__ __forceinline__ bool near32(const float4 me, const float4 q, int dxs, int dys, int dzs, const DevGeom &G,
                                       float bwf, float slack)
{
    return near_pair32(me, q, (float)dxs * G.dxf[0], (float)dys * G.dxf[1], (float)dzs * G.dxf[2], bwf, slack);
}

// ---- staged pair evaluation ----------------------------------------------
// One thread per slot walks its stencil and screens the candidates in FP32;
// the survivors (about one per slot) are staged in shared memory and the
// block then evaluates its staged pairs one per thread, so that the FP64 pair
// arithmetic runs in full warps instead of one walk iteration at a time with
// a lane or two active (GB300 issues FP64 at 2 lanes per clock per SM whatever
// the mask).  Each slot adds its pairs' terms in walk order: the same values
// in the same order as a walk that evaluates each pair when it meets it.  A
// slot with more than kStageD candidates evaluates them itself, in order.
constexpr int kStageD = 16;

// dynamic shared memory of a staged kernel: block B, NO owner values and NT
// terms per thread
__host__ __device__ constexpr size_t staged_smem(int B, int NO, int NT)
{
    return (size_t)B * (kStageD * sizeof(int2) + (NO + NT) * sizeof(double) + 4 * sizeof(int)) +
           64 * sizeof(int);
}

struct StageMem {
    int2 *stage;   // per thread: its staged candidates (j, image code)
    double *own;   // per thread: NO values of its slot for the evaluating thread
    double *term;  // per thread: NT terms of the pair it evaluated this round
    int *ocol, *orun, *olen, *opass, *wsum;
};

__device__ __forceinline__ StageMem stage_mem(unsigned char *sm, int B, int NO, int NT)
{
    StageMem M;
    M.stage = reinterpret_cast<int2 *>(sm);
    M.own = reinterpret_cast<double *>(M.stage + (size_t)B * kStageD);
    M.term = M.own + (size_t)NO * B;
    M.ocol = reinterpret_cast<int *>(M.term + (size_t)NT * B);
    M.orun = M.ocol + B;
    M.olen = M.orun + B;
    M.opass = M.olen + B;
    M.wsum = M.opass + B;
    return M;
}

// After every thread has staged its cnt candidates (and written its owner
// values and colony), the block evaluates the staged pairs one per thread:
// eval(o, e, t) computes pair e of owner thread o into t[NT] (false: no term);
// add(t) adds one term to the calling thread's sums, in staging order.
template <int NT, class Eval, class Add>
__device__ __forceinline__ void staged_pairs(const StageMem &M, int cnt, Eval &&eval, Add &&add)
{
    const int B = blockDim.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = B >> 5;
    const int xl = (cnt <= kStageD) ? cnt : 0;
    int xo = xl;
    for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, xo, d);
        if (lane >= d) xo += v;
    }
    if (lane == 31) M.wsum[w] = xo;
    M.olen[tid] = xl;
    __syncthreads();
    if (tid == 0) {
        int run = 0;
        for (int v = 0; v < nw; ++v) {
            const int c = M.wsum[v];
            M.wsum[32 + v] = run;
            run += c;
        }
        M.wsum[31] = run;  // (at most 8 warps: slot 31 is free) the block's total
    }
    __syncthreads();
    const int xt = M.wsum[31];
    xo += M.wsum[32 + w] - xl;
    M.orun[tid] = xo;
    __syncthreads();
    for (int t0 = 0; t0 < xt; t0 += B) {
        const int t = t0 + tid;
        int pass = 0;
        double tt[NT];
        for (int c = 0; c < NT; ++c) tt[c] = 0.0;
        if (t0 + 32 * w < xt && t < xt) {  // (a warp with no pair in this round skips it)
            int o = 0;  // the slot that owns pair t: the last thread whose run starts at or before t
            for (int s2 = 1 << (31 - __clz(max(B - 1, 1))); s2 >= 1; s2 >>= 1)
                if (o + s2 < B && M.orun[o + s2] <= t) o += s2;
            pass = eval(o, M.stage[(size_t)o * kStageD + (t - M.orun[o])], tt) ? 1 : 0;
        }
        for (int c = 0; c < NT; ++c) M.term[(size_t)NT * tid + c] = tt[c];
        M.opass[tid] = pass;
        __syncthreads();
        const int k1 = min(xo + xl, t0 + B);
        for (int k = max(xo, t0); k < k1; ++k)
            if (M.opass[k - t0]) add(&M.term[(size_t)NT * (k - t0)]);
        __syncthreads();
    }
}

// The forward pair term of slot i on neighbour j (image shift sx, sy): the
// three products F u that the walk adds (false: outside the list or the cutoff).
__device__ __forceinline__ bool dfwd_term(const DevState &S, const DevGeom &G, const DevParams &P,
                                          const DiffParams &D, int a, double xi, double yi, double zi, double ri,
                                          double mi, double ai, int j, int sx, int sy, double *t)
{
    const double xj = sx ? image_coord(S.x[a][j], G.len[0], sx) : S.x[a][j];
    const double yj = sy ? image_coord(S.y[a][j], G.len[1], sy) : S.y[a][j];
    const double dx = xi - xj, dy = yi - yj, dz = zi - S.z[a][j];
    const double r2 = dx * dx + dy * dy + dz * dz;
    if (!G.nbh_trivial && !(r2 <= P.nbh)) return false;
    const double rj = S.rad[j];
    const double rlm = ri + rj + P.bw;
    if (!le_nonneg(r2, (rlm - kSmall) * (rlm - kSmall))) return false;
    const double rS = ri + rj, rA = rS + P.bw;
    Divisor by;
    const double rn = sqrt_rn(r2, &by);
    const double ux = div_by(dx, by), uy = div_by(dy, by), uz = div_by(dz, by);
    const double abar = 0.5 * (ai + (D.adh ? D.adh[j] : 0.0));
    const PairLaw q = pair_law(rn, rS, rA, P.k, P.bw, abar);
    const double s = div_rn(1.0, 1.0 + D.gamma * (mi + mobility_of(rj, D.mu)));
    const double F = mi * (q.f * s);
    t[0] = F * ux;
    t[1] = F * uy;
    t[2] = F * uz;
    return true;
}

// The adjoint pair term of slot k on neighbour j: its contribution to the
// gathered J w (t[0..2]) and to the stiffness, damping, drag and adhesion
// slopes (t[3..6]) (false: no contribution).
__device__ __forceinline__ bool dadj_term(const DevState &S, const DevGeom &G, const DevParams &P,
                                          const DiffParams &D, int a, const double *lin, int n,
                                          const double *o, int j, int sx, int sy, double *t)
{
    // o: xk, yk, zk, rk, mk, dmk, ak, lk[3]
    const double xk = o[0], yk = o[1], zk = o[2], rk = o[3], mk = o[4], dmk = o[5], ak = o[6];
    const double lk[3] = {o[7], o[8], o[9]};
    const double xj = sx ? image_coord(S.x[a][j], G.len[0], sx) : S.x[a][j];
    const double yj = sy ? image_coord(S.y[a][j], G.len[1], sy) : S.y[a][j];
    const double d[3] = {xk - xj, yk - yj, zk - S.z[a][j]};
    const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    if (!G.nbh_trivial && !(r2 <= P.nbh)) return false;
    const double rj = S.rad[j];
    const double rlm = rk + rj + P.bw;
    if (!le_nonneg(r2, (rlm - kSmall) * (rlm - kSmall))) return false;
    const double rS = rk + rj, rA = rS + P.bw;
    Divisor by;
    const double rn = sqrt_rn(r2, &by);
    if (!lt_bits(rn, rA)) return false;  // f, f' and all parameter slopes vanish
    const double u[3] = {div_by(d[0], by), div_by(d[1], by), div_by(d[2], by)};
    const double mj = mobility_of(rj, D.mu);
    const double dmj = D.mu > 0.0 ? div_rn(-mj, D.mu) : 0.0;
    const double abar = 0.5 * (ak + (D.adh ? D.adh[j] : 0.0));
    const PairLaw q = pair_law(rn, rS, rA, P.k, P.bw, abar);
    const double M = mk + mj;
    const double s = div_rn(1.0, 1.0 + D.gamma * M);
    const double Ft = q.f * s, dFt = q.df * s;
    const double lj[3] = {lin[j], lin[(size_t)n + j], lin[(size_t)2 * n + j]};
    // w = m_k lam'_k - m_j lam'_j ; J w = dFt u (u.w) + (Ft/r)(w - u (u.w))
    double w[3];
    for (int c = 0; c < 3; ++c) w[c] = mk * lk[c] - mj * lj[c];
    const double uw = u[0] * w[0] + u[1] * w[1] + u[2] * w[2];
    const double fr = div_by(Ft, by);
    for (int c = 0; c < 3; ++c) t[c] = dFt * u[c] * uw + fr * (w[c] - u[c] * uw);
    // parameter slopes of v_k (this pair's term m_k Ft u), against lam'_k
    const double lu = lk[0] * u[0] + lk[1] * u[1] + lk[2] * u[2];
    t[3] = mk * (q.fk * s) * lu;
    t[4] = mk * (-q.f * M * s * s) * lu;
    t[5] = (dmk * Ft + mk * (-q.f * s * s * D.gamma * (dmk + dmj))) * lu;
    // adhesion of k enters both v_k and v_j through abar = (a_k + a_j)/2
    t[6] = 0.5 * (q.fa * s) * uw;
    return true;
}

// forward step of the differentiable form (reads buffer a, writes b, rebins)
template <bool SORTED>
__global__ void __launch_bounds__(256) k_dfwd(const DevState S, const DevParams P, DiffParams D, double dt, int a)
{
    extern __shared__ __align__(16) unsigned char smd[];
    constexpr int NO = 6, NT = 3;
    const int B = blockDim.x, tid = threadIdx.x;
    const StageMem M = stage_mem(smd, B, NO, NT);
    const int b = a ^ 1;
    const float bwf = P.bw32;
    for (int base = blockIdx.x * B; base < S.n; base += gridDim.x * B) {
        const int i = base + tid;
        const bool act = i < S.n;
        double xi = 0.0, yi = 0.0, zi = 0.0, ri = 0.0, mi = 0.0, ai = 0.0;
        double fx = 0.0, fy = 0.0, fz = 0.0;
        int col = 0, cnt = 0;
        if (act) {
            col = colony_of(S.cbase, S.ncol, i);
            const DevGeom &G = S.geoms[col];
            int bx, by;
            col_to_bxy(G, S.col[a][i], bx, by);
            xi = S.x[a][i];
            yi = S.y[a][i];
            zi = S.z[a][i];
            ri = S.rad[i];
            mi = mobility_of(ri, D.mu);
            ai = D.adh ? D.adh[i] : 0.0;
            const float4 me = S.rel[a][i];
            const float slack = screen_slack(G);
            int2 *mine = M.stage + (size_t)tid * kStageD;
            auto eval = [&](int j, int sx, int sy) {
                double t[3];
                if (dfwd_term(S, G, P, D, a, xi, yi, zi, ri, mi, ai, j, sx, sy, t)) {
                    fx += t[0];
                    fy += t[1];
                    fz += t[2];
                }
            };
            walk<SORTED>(S, G, a, i, bx, by, S.iz[a][i], [&](const float4 qr, auto slot, int dxs, int dys, int dzs,
                                                             int sx, int sy) {
                if (!near32(me, qr, dxs, dys, dzs, G, bwf, slack)) return;
                const int j = slot();
                if (cnt < kStageD) {
                    mine[cnt] = make_int2(j, (sx + 1) * 3 + (sy + 1));
                } else {
                    if (cnt == kStageD)  // too many for the stage: the staged ones first, in order
                        for (int k = 0; k < kStageD; ++k) eval(mine[k].x, mine[k].y / 3 - 1, mine[k].y % 3 - 1);
                    eval(j, sx, sy);
                }
                ++cnt;
            });
        }
        double *own = M.own + (size_t)NO * tid;
        own[0] = xi;
        own[1] = yi;
        own[2] = zi;
        own[3] = ri;
        own[4] = mi;
        own[5] = ai;
        M.ocol[tid] = col;
        staged_pairs<NT>(
            M, cnt,
            [&](int o, int2 e, double *t) {
                const double *oo = M.own + (size_t)NO * o;
                return dfwd_term(S, S.geoms[M.ocol[o]], P, D, a, oo[0], oo[1], oo[2], oo[3], oo[4], oo[5], e.x,
                                 e.y / 3 - 1, e.y % 3 - 1, t);
            },
            [&](const double *t) {
                fx += t[0];
                fy += t[1];
                fz += t[2];
            });
        if (act) {
            const DevGeom &G = S.geoms[col];
            const double vx = plus_zero(fx), vy = plus_zero(fy), vz = fz + wall_law(zi, ri, P);
            double nx = xi + dt * vx, ny = yi + dt * vy;
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

// adjoint of the step taken from buffer a (positions x_t, bins of x_t)
template <bool SORTED>
__global__ void __launch_bounds__(256) k_dadj(const DevState S, const DevParams P, DiffParams D, double dt, int a,
                                             const double *__restrict__ lin, double *__restrict__ lout,
                                             double *__restrict__ gacc, double *__restrict__ gadh)
{
    extern __shared__ __align__(16) unsigned char smd[];
    constexpr int NO = 10, NT = 7;
    const int B = blockDim.x, tid = threadIdx.x;
    const StageMem M = stage_mem(smd, B, NO, NT);
    const int n = S.n;
    const float bwf = P.bw32;
    for (int base = blockIdx.x * B; base < n; base += gridDim.x * B) {
        const int k = base + tid;
        const bool act = k < n;
        double o[NO];
        for (int c = 0; c < NO; ++c) o[c] = 0.0;
        double acc[3] = {0.0, 0.0, 0.0};
        double gk = 0.0, gg = 0.0, gm = 0.0, ga = 0.0;
        int col = 0, cnt = 0;
        auto add = [&](const double *t) {
            for (int c = 0; c < 3; ++c) acc[c] += t[c];
            gk += t[3];
            gg += t[4];
            gm += t[5];
            ga += t[6];
        };
        if (act) {
            col = colony_of(S.cbase, S.ncol, k);
            const DevGeom &G = S.geoms[col];
            int bx, by;
            col_to_bxy(G, S.col[a][k], bx, by);
            const double rk = S.rad[k];
            const double mk = mobility_of(rk, D.mu);
            o[0] = S.x[a][k];
            o[1] = S.y[a][k];
            o[2] = S.z[a][k];
            o[3] = rk;
            o[4] = mk;
            o[5] = D.mu > 0.0 ? div_rn(-mk, D.mu) : 0.0;
            o[6] = D.adh ? D.adh[k] : 0.0;
            o[7] = lin[k];
            o[8] = lin[(size_t)n + k];
            o[9] = lin[(size_t)2 * n + k];
            const float4 me = S.rel[a][k];
            const float slack = screen_slack(G);
            int2 *mine = M.stage + (size_t)tid * kStageD;
            auto eval = [&](int j, int sx, int sy) {
                double t[NT];
                if (dadj_term(S, G, P, D, a, lin, n, o, j, sx, sy, t)) add(t);
            };
            walk<SORTED>(S, G, a, k, bx, by, S.iz[a][k], [&](const float4 qr, auto slot, int dxs, int dys, int dzs,
                                                             int sx, int sy) {
                if (!near32(me, qr, dxs, dys, dzs, G, bwf, slack)) return;
                const int j = slot();
                if (cnt < kStageD) {
                    mine[cnt] = make_int2(j, (sx + 1) * 3 + (sy + 1));
                } else {
                    if (cnt == kStageD)
                        for (int q = 0; q < kStageD; ++q) eval(mine[q].x, mine[q].y / 3 - 1, mine[q].y % 3 - 1);
                    eval(j, sx, sy);
                }
                ++cnt;
            });
        }
        for (int c = 0; c < NO; ++c) M.own[(size_t)NO * tid + c] = o[c];
        M.ocol[tid] = col;
        staged_pairs<NT>(
            M, cnt,
            [&](int ow, int2 e, double *t) {
                return dadj_term(S, S.geoms[M.ocol[ow]], P, D, a, lin, n, M.own + (size_t)NO * ow, e.x,
                                 e.y / 3 - 1, e.y % 3 - 1, t);
            },
            add);
        if (act) {
            const double wz = wall_slope(o[2], o[3], P);
            lout[k] = o[7] + dt * acc[0];
            lout[(size_t)n + k] = o[8] + dt * acc[1];
            lout[(size_t)2 * n + k] = o[9] + dt * (acc[2] + wz * o[9]);
            gacc[k] += dt * gk;
            gacc[(size_t)n + k] += dt * gg;
            gacc[(size_t)2 * n + k] += dt * gm;
            gadh[k] += dt * ga;
        }
        __syncthreads();
    }
}

// The same two kernels with one warp per neighbour column (bmxg_stencil.cuh),
// for sizes whose walks are bound by their dependent loads: same pairs, same
// FP64 operations, same order of the sums.
template <int NS, int STAGE, int RESIDENT>
__global__ void __launch_bounds__(kWalkBlock, RESIDENT) k_dfwdw(const DevState S, const DevParams P, DiffParams D, double dt,
                                                         int a)
{
    extern __shared__ __align__(16) unsigned char smw[];
    auto &M = *reinterpret_cast<WalkMem<NS, STAGE, unsigned> *>(smw);
    __shared__ double own[6][NS];
    __shared__ int ocol[NS];
    __shared__ double term[3 * kWalkBlock];
    __shared__ unsigned char opass[kWalkBlock];
    const int tid = threadIdx.x;
    const int b = a ^ 1;
    chain_wait();
    walk_block(S, a, P.bw32, M, [&](int s, int i, int col) {
        const double ri = S.rad[i];
        own[0][s] = S.x[a][i];
        own[1][s] = S.y[a][i];
        own[2][s] = S.z[a][i];
        own[3][s] = ri;
        own[4][s] = mobility_of(ri, D.mu);
        own[5][s] = D.adh ? D.adh[i] : 0.0;
        ocol[s] = col;
    });
    double fx = 0.0, fy = 0.0, fz = 0.0;
    walk_pairs<3>(
        M, term, opass,
        [&](int o, int2 e, double *t) {
            return dfwd_term(S, S.geoms[ocol[o]], P, D, a, own[0][o], own[1][o], own[2][o], own[3][o], own[4][o],
                             own[5][o], e.x, e.y / 3 - 1, e.y % 3 - 1, t);
        },
        [&](const double *t) {
            fx += t[0];
            fy += t[kWalkBlock];
            fz += t[2 * kWalkBlock];
        });
    const int i = blockIdx.x * NS + tid;
    if (tid >= NS || i >= S.n) return;
    const DevGeom &G = S.geoms[ocol[tid]];
    const double xi = own[0][tid], yi = own[1][tid], zi = own[2][tid], ri = own[3][tid];
    if (M.over[tid]) {  // a crowded column: the whole walk, each pair evaluated as it is met
        int bx, by;
        col_to_bxy(G, S.col[a][i], bx, by);
        const float4 me = S.rel[a][i];
        const float slack = screen_slack(G);
        walk<true>(S, G, a, i, bx, by, S.iz[a][i], [&](const float4 q, auto slot, int dxs, int dys, int dzs, int sx,
                                                       int sy) {
            if (!near32(me, q, dxs, dys, dzs, G, P.bw32, slack)) return;
            double t[3];
            if (dfwd_term(S, G, P, D, a, xi, yi, zi, ri, own[4][tid], own[5][tid], slot(), sx, sy, t)) {
                fx += t[0];
                fy += t[1];
                fz += t[2];
            }
        });
    }
    const double vx = plus_zero(fx), vy = plus_zero(fy), vz = fz + wall_law(zi, ri, P);
    double nx = xi + dt * vx, ny = yi + dt * vy;
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

template <int NS, int STAGE, int RESIDENT>
__global__ void __launch_bounds__(kWalkBlock, RESIDENT) k_dadjw(const DevState S, const DevParams P, DiffParams D, double dt,
                                                         int a, const double *lin, double *lout, double *gacc, double *gadh)
{
    constexpr int NO = 10, NT = 7;
    extern __shared__ __align__(16) unsigned char smw[];
    auto &M = *reinterpret_cast<WalkMem<NS, STAGE, unsigned> *>(smw);
    __shared__ double own[NS][NO + 1];  // (odd pitch: no bank conflicts between the slots' rows)
    __shared__ int ocol[NS];
    __shared__ double term[NT * kWalkBlock];
    __shared__ unsigned char opass[kWalkBlock];
    const int tid = threadIdx.x;
    const int n = S.n;
    chain_wait();
    walk_block(S, a, P.bw32, M, [&](int s, int k, int col) {
        double *o = own[s];
        const double rk = S.rad[k];
        const double mk = mobility_of(rk, D.mu);
        o[0] = S.x[a][k];
        o[1] = S.y[a][k];
        o[2] = S.z[a][k];
        o[3] = rk;
        o[4] = mk;
        o[5] = D.mu > 0.0 ? div_rn(-mk, D.mu) : 0.0;
        o[6] = D.adh ? D.adh[k] : 0.0;
        o[7] = lin[k];
        o[8] = lin[(size_t)n + k];
        o[9] = lin[(size_t)2 * n + k];
        ocol[s] = col;
    });
    double acc[NT];
    for (int c = 0; c < NT; ++c) acc[c] = 0.0;
    walk_pairs<NT>(
        M, term, opass,
        [&](int ow, int2 e, double *t) {
            return dadj_term(S, S.geoms[ocol[ow]], P, D, a, lin, n, own[ow], e.x, e.y / 3 - 1, e.y % 3 - 1, t);
        },
        [&](const double *t) {
            for (int c = 0; c < NT; ++c) acc[c] += t[c * kWalkBlock];
        });
    const int k = blockIdx.x * NS + tid;
    if (tid >= NS || k >= n) return;
    const double *o = own[tid];
    if (M.over[tid]) {
        const DevGeom &G = S.geoms[ocol[tid]];
        int bx, by;
        col_to_bxy(G, S.col[a][k], bx, by);
        const float4 me = S.rel[a][k];
        const float slack = screen_slack(G);
        walk<true>(S, G, a, k, bx, by, S.iz[a][k], [&](const float4 q, auto slot, int dxs, int dys, int dzs, int sx,
                                                       int sy) {
            if (!near32(me, q, dxs, dys, dzs, G, P.bw32, slack)) return;
            double t[NT];
            if (dadj_term(S, G, P, D, a, lin, n, o, slot(), sx, sy, t))
                for (int c = 0; c < NT; ++c) acc[c] += t[c];
        });
    }
    const double wz = wall_slope(o[2], o[3], P);
    lout[k] = o[7] + dt * acc[0];
    lout[(size_t)n + k] = o[8] + dt * acc[1];
    lout[(size_t)2 * n + k] = o[9] + dt * (acc[2] + wz * o[9]);
    gacc[k] += dt * acc[3];
    gacc[(size_t)n + k] += dt * acc[4];
    gacc[(size_t)2 * n + k] += dt * acc[5];
    gadh[k] += dt * acc[6];
}

// Deterministic sum of per-slot gradient planes: every block of a plane sums a
// fixed share of it, the second kernel the blocks' sums, each in a fixed order
// (one block over all planes took 114 us for 20 000 slots; 6 us for both).  The
// rounding of every addition is kept beside the sum (two_add, the exact difference
// of Knuth's sum), so the order costs no digits: the result is the planes' sum
// rounded about once, however the shares fall.
constexpr int kReduceThreads = 256;

__device__ __forceinline__ void two_add(double &s, double &c, double v)
{
    const double t = s + v, z = t - s;
    c += (s - (t - z)) + (v - z);
    s = t;
}

// The block's sum and what its roundings left, in thread 0.
__device__ __forceinline__ void block_sum(double &s, double &c, double (*sh)[2])
{
    sh[threadIdx.x][0] = s;
    sh[threadIdx.x][1] = c;
    __syncthreads();
    for (int w = kReduceThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            two_add(s, c, sh[threadIdx.x + w][0]);
            c += sh[threadIdx.x + w][1];
            sh[threadIdx.x][0] = s;
            sh[threadIdx.x][1] = c;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kReduceThreads) k_dreduce(const double *gacc, int n, double *out)
{
    __shared__ double sh[kReduceThreads][2];
    const int p = blockIdx.y;
    double s = 0.0, c = 0.0;
    for (int i = blockIdx.x * kReduceThreads + threadIdx.x; i < n; i += gridDim.x * kReduceThreads)
        two_add(s, c, gacc[(size_t)p * n + i]);
    block_sum(s, c, sh);
    if (threadIdx.x == 0) {
        double *o = out + 4 + 2 * (p * kReduceBlocks + blockIdx.x);
        o[0] = s;
        o[1] = c;
    }
}

__global__ void __launch_bounds__(kReduceThreads) k_dreduce_top(double *out, int blocks)
{
    __shared__ double sh[kReduceThreads][2];
    const int p = blockIdx.x;
    const double *o = out + 4 + 2 * (p * kReduceBlocks + min((int)threadIdx.x, blocks - 1));
    const bool mine = (int)threadIdx.x < blocks;
    double s = mine ? o[0] : 0.0, c = mine ? o[1] : 0.0;
    block_sum(s, c, sh);
    if (threadIdx.x == 0) out[p] = finite_bits(s) ? s + c : s;
}

}  // namespace

// a kernel's dynamic shared memory above the default 48 KB (the launches
// that need it: 256-thread blocks)
template <class K>
void allow_smem(K kernel, size_t need)
{
    if (need > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need);
}

// The kernels with a warp per neighbour column up to here, above with a thread per
// slot.  Forward and backward of 20 steps, one thread per slot / a warp per column, us, 3 and 10
// slots a column: 20 000 slots 3347, 5257 / 1758, 2352, 65 000 3888, 6208 / 3590, 4844, 100 000 5924,
// 9445 / 5314, 7299, 130 000 6133, 9931 / 6242, 8668, 200 000 7928, 13 295 / 8671, 12 101.
constexpr int kAdjointColumns = 114688;
static_assert(kAdjointColumns < (1 << 28), "a staged slot in 28 bits");

int launch_dfwd(const DevState &S, const DevParams &P, const DiffParams &D, double dt, int a, int grid, int block,
                cudaStream_t st, bool pinned)
{
    const size_t smem = staged_smem(block, 6, 3);
    if (S.srel[a] && !pinned && S.n <= kAdjointColumns) {
        const int blocks = (S.n + 31) / 32, fit = wave_fit(blocks, 3, S.nsm);
        launch_after(fit == 3 ? k_dfwdw<32, kWalkStage, 3>
                              : (fit == 4 ? k_dfwdw<32, kWalkStage, 4> : k_dfwdw<32, kWalkStage, 5>),
                     blocks, kWalkBlock, sizeof(WalkMem<32, kWalkStage, unsigned>), st, S, P, D, dt, a);
    } else if (S.srel[a]) {
        allow_smem(k_dfwd<true>, smem);
        k_dfwd<true><<<grid, block, smem, st>>>(S, P, D, dt, a);
    } else {
        allow_smem(k_dfwd<false>, smem);
        k_dfwd<false><<<grid, block, smem, st>>>(S, P, D, dt, a);
    }
    return 1;
}

int launch_dadj(const DevState &S, const DevParams &P, const DiffParams &D, double dt, int a, const double *lin,
                double *lout, double *gacc, double *gadh, int grid, int block, cudaStream_t st, bool pinned)
{
    const size_t smem = staged_smem(block, 10, 7);
    if (S.srel[a] && !pinned && S.n <= kAdjointColumns) {
        const int blocks = (S.n + 31) / 32, fit = wave_fit(blocks, 2, S.nsm);
        launch_after(fit == 2 ? k_dadjw<32, kWalkStage, 2>
                              : (fit == 3 ? k_dadjw<32, kWalkStage, 3>
                                          : (fit == 4 ? k_dadjw<32, kWalkStage, 4> : k_dadjw<32, kWalkStage, 5>)),
                     blocks, kWalkBlock, sizeof(WalkMem<32, kWalkStage, unsigned>), st, S, P, D, dt, a, lin, lout,
                     gacc, gadh);
    } else if (S.srel[a]) {
        allow_smem(k_dadj<true>, smem);
        k_dadj<true><<<grid, block, smem, st>>>(S, P, D, dt, a, lin, lout, gacc, gadh);
    } else {
        allow_smem(k_dadj<false>, smem);
        k_dadj<false><<<grid, block, smem, st>>>(S, P, D, dt, a, lin, lout, gacc, gadh);
    }
    return 1;
}

int launch_dreduce(const double *gacc, int n, int planes, double *out, cudaStream_t st)
{
    static_assert(kReduceBlocks <= kReduceThreads, "one thread per block sum");
    const int blocks = std::max(1, std::min(kReduceBlocks, (n + kReduceThreads - 1) / kReduceThreads));
    k_dreduce<<<dim3(blocks, planes), kReduceThreads, 0, st>>>(gacc, n, out);
    k_dreduce_top<<<planes, kReduceThreads, 0, st>>>(out, blocks);
    return 2;
}

}  // namespace bmxg
