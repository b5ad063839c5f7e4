// k_rod.cu -- the step for states that hold rod segments (FUNGI), alone or
// mixed with spheres: deterministic bond bookkeeping, the segment-segment
// closest-point contact / bonded-spring force gather with the wall force,
// and the update with the orientation rotation.
//
// Replaces, for FUNGI, the force lambda of src/des/bmx_pc_interaction.cpp:170-279
// with evaluateForce's rod branch (src/chemistry/bmx_cell_interaction_K.H:277-993)
// and evaluateSurfaceForce's rod branch (:1031-1282), and the update lambda
// (bmx_pc_interaction.cpp:311-436) with its orientation rotation (:334-431).
//
// Design notes
//  * The reference edits bond tables from inside its parallel pair loop; its
//    edits of the neighbour j land on a by-value copy (bmx_pc_interaction.cpp:188)
//    and do not persist, so the lasting effect is "each segment repairs its
//    own table".  k_rod_book does exactly that, reading the neighbours'
//    tables as they were at the start of the step (buffer a) and writing the
//    segment's own table to buffer b -- deterministic, and equal to the
//    reference's serial CPU result.
//  * Only segment i's velocity is produced per pair (the j-side accumulation
//    is disabled in the reference, bmx_pc_interaction.cpp:251-261), and the
//    mobility of segment i is linear in its two site forces:
//      vel = 1/2 (Dii + Dij)(f1 + f2),  rot = 1/2 r x (Dii - Dij)(f1 - f2)_perp
//    with Dii = d0 I and Dij = db I + (da - db) n n^T (the rotated tensors of
//    :812-882).  The kernel therefore sums f1 + f2 and f1 - f2 over the pairs
//    and applies the mobility once per segment: the same result up to
//    rounding, without two 3x3 tensor rotations per pair.
//  * FP32F: contact pair math in FP32 on the FP64-differenced bin-relative
//    offsets; pairs whose segments are near-parallel (det < 0.05 Aii Ajj,
//    where the closest-point solve loses precision), pairs whose closest
//    points are within 1 % of the segment lengths (touching or crossing
//    segments, where the separation's direction is end-point rounding noise)
//    and bonded pairs (a spring on the difference of two coincident end
//    points) are done in FP64.
#include "bmxg_stencil.cuh"

namespace bmxg {

namespace {

// FP32 axis and length of a segment
__device__ __forceinline__ float4 rod_axis32(const double4_32a &tr, double L)
{
    return make_float4(d2f_rn(tr.y * tr.z), d2f_rn(tr.y * tr.w), d2f_rn(tr.x), d2f_rn(L));
}

template <class T>
__device__ __forceinline__ bool in01(T t) { return le_q(T(0), t) && le_q(t, T(1)); }

template <class T>
__device__ __forceinline__ T sq3(T a, T b, T c) { return a * a + b * b + c * c; }

// Closest points of segments (a1,a2) and (b1,b2): the case structure of
// evaluateMinimumDistance (bmx_cell_interaction_K.H:51-221), including the
// exact zero tests on Aij and det and the unconstrained result for Aij == 0.
template <class T>
__device__ void min_distance(const T *a1, const T *a2, const T *b1, const T *b2, T &tau_i, T &tau_j)
{
    T ri[3], rj[3], w[3];
    for (int k = 0; k < 3; ++k) {
        ri[k] = a2[k] - a1[k];
        rj[k] = b2[k] - b1[k];
        w[k] = a1[k] - b1[k];
    }
    T rirj = T(0);
    for (int k = 0; k < 3; ++k) rirj += ri[k] * rj[k];
    const T Aii = sq3(ri[0], ri[1], ri[2]);
    const T Ajj = sq3(rj[0], rj[1], rj[2]);
    const T Aij = -rirj;
    const T det = Aii * Ajj - Aij * Aij;
    const T Bi = -(w[0] * ri[0] + w[1] * ri[1] + w[2] * ri[2]);
    const T Bj = w[0] * rj[0] + w[1] * rj[1] + w[2] * rj[2];
    T ti = T(0), tj = T(0);
    bool search = false;
    if (zero_q(Aij)) {
        ti = qdiv(Bi, Aii);
        tj = qdiv(Bj, Ajj);
    } else if (zero_q(det)) {
        const T t0 = qdiv(Bj, Ajj);
        if (in01(t0)) { ti = T(0); tj = t0; }
        else {
            const T t1 = qdiv(Bj + rirj, Ajj);
            if (in01(t1)) { ti = T(1); tj = t1; }
            else search = true;
        }
    } else {
        ti = qdiv(Ajj * Bi - Aij * Bj, det);
        tj = qdiv(Aii * Bj - Aij * Bi, det);
        if (in01(ti)) {
            if (lt_q(tj, T(0)) || lt_q(T(1), tj)) {
                const T t0 = qdiv(Bi, Aii), t1 = qdiv(Bi + rirj, Aii);
                if (in01(t0) && in01(t1)) {
                    const T s0 = sq3(a1[0] + t0 * ri[0] - b1[0], a1[1] + t0 * ri[1] - b1[1],
                                     a1[2] + t0 * ri[2] - b1[2]);
                    const T s1 = sq3(a1[0] + t1 * ri[0] - b2[0], a1[1] + t1 * ri[1] - b2[1],
                                     a1[2] + t1 * ri[2] - b2[2]);
                    if (lt_q(s0, s1)) { tj = T(0); ti = t0; } else { tj = T(1); ti = t1; }
                } else if (in01(t0)) { tj = T(0); ti = t0; }
                else if (in01(t1)) { tj = T(1); ti = t1; }
                else search = true;
            }
        } else if (in01(tj)) {
            const T t0 = qdiv(Bj, Ajj), t1 = qdiv(Bj + rirj, Ajj);
            if (in01(t0) && in01(t1)) {
                const T s0 = sq3(b1[0] + t0 * rj[0] - a1[0], b1[1] + t0 * rj[1] - a1[1],
                                 b1[2] + t0 * rj[2] - a1[2]);
                const T s1 = sq3(b1[0] + t1 * rj[0] - a2[0], b1[1] + t1 * rj[1] - a2[1],
                                 b1[2] + t1 * rj[2] - a2[2]);
                if (lt_q(s0, s1)) { ti = T(0); tj = t0; } else { ti = T(1); tj = t1; }
            } else if (in01(t0)) { ti = T(0); tj = t0; }
            else if (in01(t1)) { ti = T(1); tj = t1; }
            else search = true;
        } else {
            search = true;
        }
    }
    if (search) {
        T m[4];
        m[0] = sq3(a1[0] - b1[0], a1[1] - b1[1], a1[2] - b1[2]);
        m[1] = sq3(a1[0] - b2[0], a1[1] - b2[1], a1[2] - b2[2]);
        m[2] = sq3(a2[0] - b1[0], a2[1] - b1[1], a2[2] - b1[2]);
        m[3] = sq3(a2[0] - b2[0], a2[1] - b2[1], a2[2] - b2[2]);
        int best = 0;
        for (int k = 1; k < 4; ++k)
            if (lt_q(m[k], m[best])) best = k;
        ti = (best >= 2) ? T(1) : T(0);
        tj = (best & 1) ? T(1) : T(0);
    }
    tau_i = ti;
    tau_j = tj;
}

// Site forces on segment i from segment j (j's centre at the origin, i's at
// r12): a bonded linear spring between the bonded sites (si, sj in {1,2}),
// otherwise the cubic contact law at the closest points split (1-tau, tau)
// (bmx_cell_interaction_K.H:552-772).  Returns f1 (site 1) and f2 (site 2).
template <class T>
__device__ void rod_site_forces(const T *r12, const T *ni, T Li, const T *nj, T Lj, T rS, T rA, T k,
                                int si, int sj, T kb, T *f1, T *f2, T *r_out = nullptr)
{
    T e1[3], e2[3], g1[3], g2[3];
    for (int d = 0; d < 3; ++d) {
        e1[d] = r12[d] - T(0.5) * ni[d] * Li;
        e2[d] = r12[d] + T(0.5) * ni[d] * Li;
        g1[d] = T(-0.5) * nj[d] * Lj;
        g2[d] = T(0.5) * nj[d] * Lj;
        f1[d] = T(0);
        f2[d] = T(0);
    }
    if ((si == 1 || si == 2) && (sj == 1 || sj == 2)) {
        const T *ea = (si == 1) ? e1 : e2;
        const T *eb = (sj == 1) ? g1 : g2;
        T *f = (si == 1) ? f1 : f2;
        for (int d = 0; d < 3; ++d) f[d] -= kb * (ea[d] - eb[d]);
        return;
    }
    T ti, tj;
    min_distance(e1, e2, g1, g2, ti, tj);
    T dv[3];
    for (int d = 0; d < 3; ++d) dv[d] = (e1[d] + ti * (e2[d] - e1[d])) - (g1[d] + tj * (g2[d] - g1[d]));
    const T r = qsqrt(dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2]);
    if (r_out) *r_out = r;
    // r <= 1e-8: the reference keeps the unnormalised separation (its
    // fallback direction goes to shadowing locals, :744-746); so do we.
    if (lt_q(T(1.0e-8), r)) {
        dv[0] = qdiv(dv[0], r);
        dv[1] = qdiv(dv[1], r);
        dv[2] = qdiv(dv[2], r);
    }
    const T F = lt_q(r, rA) ? -k * (r - rA) * (r - rA) * (r - rS) : T(0);
    if (!zero_q(F)) {
        for (int d = 0; d < 3; ++d) {
            f1[d] += F * dv[d] * (T(1) - ti);
            f2[d] += F * dv[d] * ti;
        }
    }
}

// The bonded spring of rod_site_forces alone (si, sj in {1, 2}): the two bonded
// ends with its operations, the other two left out.
__device__ __forceinline__ void rod_spring(const double *r12, const double *ni, double Li, const double *nj, double Lj,
                                           int si, int sj, double kb, double *f1, double *f2)
{
    for (int d = 0; d < 3; ++d) {
        const double hi = 0.5 * ni[d] * Li, hj = 0.5 * nj[d] * Lj;
        const double ea = (si == 1) ? r12[d] - hi : r12[d] + hi;
        const double eb = (sj == 1) ? -hj : hj;
        const double f = 0.0 - kb * (ea - eb);
        f1[d] = (si == 1) ? f : 0.0;
        f2[d] = (si == 1) ? 0.0 : f;
    }
}

__device__ __forceinline__ int find_in_table(const int *tb, int id, int cpu)
{
    const int nb = min(tb[0], 4);
    for (int k = 0; k < nb; ++k)
        if (tb[1 + k] == id && tb[5 + k] == cpu) return k;
    return -1;
}

// The site of the first entry of a register-held table tb (n_bnds, ids[4],
// cpus[4], sites[4]) that names (id, cpu), or 0: the same answer as
// tb[9 + find_in_table(...)], by selects over constant indices so the table
// never goes to local memory.
__device__ __forceinline__ int table_site(const int *tb, int id, int cpu)
{
    const int nb = min(tb[0], 4);
    int site = 0;
#pragma unroll
    for (int k = 3; k >= 0; --k)
        if (k < nb && tb[1 + k] == id && tb[5 + k] == cpu) site = tb[9 + k];
    return site;
}

__device__ __forceinline__ int find_in_plane_table(const int *tab, int n, int j, int id, int cpu)
{
    const int nb = min(__ldg(&tab[j]), 4);
    for (int k = 0; k < nb; ++k)
        if (__ldg(&tab[(size_t)(1 + k) * n + j]) == id && __ldg(&tab[(size_t)(5 + k) * n + j]) == cpu) return k;
    return -1;
}

// the same over a table written by this kernel
__device__ __forceinline__ int find_in_slot_table(const int *tab, int n, int j, int id, int cpu)
{
    const int nb = min(tab[j], 4);
    for (int k = 0; k < nb; ++k)
        if (tab[(size_t)(1 + k) * n + j] == id && tab[(size_t)(5 + k) * n + j] == cpu) return k;
    return -1;
}

// exact FP64 separation of slot i from the (image of) slot j, as the
// reference's loop computes it (bmx_pc_interaction.cpp:191-197)
__device__ __forceinline__ double sep64(const DevState &S, const DevGeom &G, int a, int j, int sx, int sy,
                                        double xi, double yi, double zi, double *d)
{
    const double xj = sx ? S.x[a][j] + (double)sx * G.len[0] : S.x[a][j];
    const double yj = sy ? S.y[a][j] + (double)sy * G.len[1] : S.y[a][j];
    d[0] = xi - xj;
    d[1] = yi - yj;
    d[2] = zi - S.z[a][j];
    return d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
}

// The interaction gate r^2 <= (r_lm - 1e-15)^2 (and BMXCheckPair's
// r^2 <= neighborhood) decided from the FP32 bin offsets where they settle it:
// the offsets are the FP64 differences rounded once, so the FP32 separation
// is within ~1e-9 cm of the exact one, and a pair more than 1e-5 r_lm from
// the gate is decided without FP64 arithmetic; the others take the exact
// FP64 test.  Returns the decision and the FP32 separation r12f.
__device__ __forceinline__ bool rod_gate(const DevState &S, const DevGeom &G, const DevParams &P, int a, int j,
                                         int dxs, int dys, int dzs, int sx, int sy, float4 me, float Lif, float Ljf,
                                         double xi, double yi, double zi, double Li, float *r12f)
{
    const float4 q = __ldg(&S.rel[a][j]);
    r12f[0] = (me.x - q.x) - (float)dxs * G.dxf[0];
    r12f[1] = (me.y - q.y) - (float)dys * G.dxf[1];
    r12f[2] = (me.z - q.z) - (float)dzs * G.dxf[2];
    const float r2f = r12f[0] * r12f[0] + r12f[1] * r12f[1] + r12f[2] * r12f[2];
    if (G.nbh_trivial) {
        const float rlmf = 1.5f * (Lif + Ljf) + P.bw32;
        const float lo = rlmf * (1.0f - 1.0e-5f), hi = rlmf * (1.0f + 1.0e-5f);
        if (r2f <= lo * lo) return true;
        if (r2f > hi * hi) return false;
    }
    double d[3];
    const double r2 = sep64(S, G, a, j, sx, sy, xi, yi, zi, d);
    if (!G.nbh_trivial && !(r2 <= P.nbh)) return false;
    const double rlm = 1.5 * (Li + S.clen[j]) + P.bw;
    return r2 <= (rlm - kSmall) * (rlm - kSmall);
}

// Whether two segments are certainly beyond the contact range `reach` (then the
// contact force is exactly zero), in FP32: q = the separation at a candidate
// (s, t) of the closest points bounds the distance from above, and since
// |w + s u - t v|^2 is convex, its slopes at (s, t) bound it from below over
// the whole square.  The rounding of the FP32 offsets and axes enters with 4e-6 of
// the squared lengths, far above it.  (Segments whose axes may be exactly
// perpendicular are never clear: the reference then takes the closest points of
// the unbounded lines.)
__device__ __forceinline__ bool rod_clear32(const float *r12, const float4 axi, const float4 axj, float reach)
{
    const float u[3] = {axi.x * axi.w, axi.y * axi.w, axi.z * axi.w};
    const float v[3] = {axj.x * axj.w, axj.y * axj.w, axj.z * axj.w};
    float w[3];
    float aa = 0.0f, bb = 0.0f, cc = 0.0f, dd = 0.0f, ee = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        w[k] = r12[k] - 0.5f * u[k] + 0.5f * v[k];
        aa = __fmaf_rn(u[k], u[k], aa);
        bb = __fmaf_rn(u[k], v[k], bb);
        cc = __fmaf_rn(v[k], v[k], cc);
        dd = __fmaf_rn(u[k], w[k], dd);
        ee = __fmaf_rn(v[k], w[k], ee);
    }
    if (!(bb * bb > 1.0e-8f * aa * cc)) return false;
    const float det = aa * cc - bb * bb;
    float s = (det > 1.0e-5f * aa * cc) ? __saturatef(__fdividef(bb * ee - cc * dd, det)) : 0.5f;
    const float t = __saturatef(__fdividef(bb * s + ee, cc));
    s = __saturatef(__fdividef(bb * t - dd, aa));
    float f = 0.0f, gs = 0.0f, gt = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float q = w[k] + s * u[k] - t * v[k];
        f = __fmaf_rn(q, q, f);
        gs = __fmaf_rn(2.0f * u[k], q, gs);
        gt = __fmaf_rn(-2.0f * v[k], q, gt);
    }
    const float low = f - fmaxf(gs * s, -gs * (1.0f - s)) - fmaxf(gt * t, -gt * (1.0f - t)) - 4.0e-6f * (aa + cc + f);
    return low > 1.01f * reach * reach && reach >= 0.0f;  // (not finite: not clear)
}

// ---- bookkeeping ----------------------------------------------------------
// The bookkeeping of segment i by a walk of its stencil: flag resets, position
// fix-up, half-bond repair of its own table (buffer b).
__device__ void book_slot(const DevState &S, const DevParams &P, int a, int i)
{
    const int b = a ^ 1;
    const int n = S.n;
    S.fflag[i] = 0;  // flag resets of bmx_pc_interaction.cpp:178-180
    S.sflag[i] = 0;
    S.nflag[i] = 0;
    int tb[13];
    for (int k = 0; k < 13; ++k) tb[k] = S.tab[a][(size_t)k * n + i];
    if (S.ctype[i] == kFungi) {
        const DevGeom &G = geom_of(S, i);
        int bx, by;
        col_to_bxy(G, S.col[a][i], bx, by);
        const double xi = S.x[a][i], yi = S.y[a][i], zi = S.z[a][i];
        const double Li = S.clen[i];
        const float Lif = d2f_rn(Li);
        const float4 me = S.rel[a][i];
        const int iid = S.id[i], icpu = S.cpu[i];
        const int fs = S.fix_site[i];
        int pos = S.position[i];
        bool any = false;
        int rep = 0;
        visit_stencil(S, G, a, i, bx, by, S.iz[a][i], [&](int j, int dxs, int dys, int dzs, int sx, int sy) {
            if (S.ctype[j] != kFungi) return;
            float r12f[3];
            if (!rod_gate(S, G, P, a, j, dxs, dys, dzs, sx, sy, me, Lif, d2f_rn(S.clen[j]), xi, yi, zi, Li, r12f))
                return;
            any = true;
            const int jid = S.id[j], jcpu = S.cpu[j];
            // position fix-up (bmx_cell_interaction_K.H:338-362); the
            // neighbour's position is only tested against TIP, which no
            // thread writes, so reading it while others update theirs is safe
            if (pos == kSecond1 || pos == kSecond2) {
                const int site = (pos == kSecond1) ? 1 : 2;
                const int nb = min(tb[0], 4);
                int k = 0;
                for (; k < nb; ++k)
                    if (tb[1 + k] == jid && tb[5 + k] == jcpu && tb[9 + k] == site) break;
                if (k < nb && S.position[j] != kTip) pos = kInterior;
            }
            // half-bond repair of i (:370-467)
            const bool i_to_j = find_in_table(tb, jid, jcpu) >= 0;
            const bool j_to_i = find_in_plane_table(S.tab[a], n, j, iid, icpu) >= 0;
            if (!i_to_j && j_to_i) {
                const int nb = tb[0];
                if (nb >= 0 && nb < 4) {
                    const int isite = (fs == 0) ? (tb[9] == 1 ? 2 : 1) : fs;
                    tb[1 + nb] = jid;
                    tb[5 + nb] = jcpu;
                    tb[9 + nb] = isite;
                    tb[0] = nb + 1;
                    ++rep;
                }
            }
        });
        S.position[i] = pos;
        if (any)
            for (int k = 0; k < 6; ++k) S.dltd[(size_t)k * n + i] = -1;
        if (rep) atomicAdd(&S.cnt->bond_repairs, (unsigned long long)rep);
    }
    for (int k = 0; k < 13; ++k) S.tab[b][(size_t)k * n + i] = tb[k];
}

// (contexts without room for the pipelines' queues)
__global__ void k_rod_book_plain(const DevState S, const DevParams P, int a)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n; i += gridDim.x * blockDim.x) book_slot(S, P, a, i);
}

// The bookkeeping and the queue of gated pairs, one warp per neighbour column
// (bmxg_stencil.cuh): the walk is a chain of dependent loads (candidate, its
// type, its ids, its bond table), which 50 000 segments on one thread each do
// not hide.  A segment whose own table an unmutual bond will change (rare), or
// with more candidates than the staging or kRodCap holds, takes book_slot's walk
// for the bookkeeping; in the latter case its pairs are not queued (rcnt tells
// the segment kernel to walk).  Every other segment's table stays as it was.
// The block's pairs go to the queue together: contacts from the front, pairs
// that the segment's table bonds from the back, so that the pair kernels' warps
// run one kind.  The FP64 step of 50 000 segments, 10 steps and the load, 2.70 ->
// 2.30 ms, FP32F, 20 steps, 3.80 -> 3.14 ms, with the pair kernels below (the
// bookkeeping alone 54 -> 46 us).
constexpr int kRodStage = 12;

__global__ void __launch_bounds__(kWalkBlock, 3) k_rod_book(const DevState S, const DevParams P, int a)
{
    extern __shared__ __align__(16) unsigned char smw[];
    auto &M = *reinterpret_cast<WalkMem<32, kRodStage> *>(smw);
    __shared__ int tb[13][32];
    __shared__ int repair[32], fixed[32], any[32];
    __shared__ int nq[2], at[2];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int b = a ^ 1;
    const int n = S.n;
    const int i = blockIdx.x * 32 + lane;
    for (int k = w; k < 13; k += kWalkCols)
        if (i < n) tb[k][lane] = S.tab[a][(size_t)k * n + i];
    if (w == 0) {
        repair[lane] = 0;
        fixed[lane] = 0;
        any[lane] = 0;
    }
    if (tid < 2) nq[tid] = 0;
    __syncthreads();
    int cnt = 0;
    if (i < n && S.ctype[i] == kFungi) {
        const DevGeom &G = geom_of(S, i);
        int bx, by;
        col_to_bxy(G, S.col[a][i], bx, by);
        const int izi = S.iz[a][i];
        const double xi = S.x[a][i], yi = S.y[a][i], zi = S.z[a][i];
        const double Li = S.clen[i];
        const float4 axi = S.axf[a][i];
        const float4 me = S.rel[a][i];
        const int iid = S.id[i], icpu = S.cpu[i];
        const int pos = S.position[i];
        const int second = (pos == kSecond1) ? 1 : (pos == kSecond2 ? 2 : 0);
        const int nb = min(tb[0][lane], 4);
        int ii, jj, lo, hi, sx, sy;
        if (walk_target(S, G, a, bx, by, w, ii, jj, lo, hi, sx, sy)) {
            const int dxs = w / 3 - 1, dys = w % 3 - 1;
            walk_column(S, a, lo, hi, S.rank[a][i], izi, [&](int t, const float4 q, int dzs) {
                const int j = __ldg(&S.perm[a][t]);
                if (S.ctype[j] != kFungi) return;
                if ((sx | sy) && !image_in_row(S, G, a, j, ii, jj, sx, sy)) return;
                float r12f[3];
                const float4 axj = __ldg(&S.axf[a][j]);
                if (!rod_gate(S, G, P, a, j, dxs, dys, dzs, sx, sy, me, axi.w, axj.w, xi, yi, zi, Li, r12f)) return;
                any[lane] = 1;
                const int jid = S.id[j], jcpu = S.cpu[j];
                // the first entry of i's table that names j (table_site), and whether
                // one with the position's site does (the position fix-up)
                int site = 0;
                bool mine = false, at_site = false;
                for (int k = nb - 1; k >= 0; --k)
                    if (tb[1 + k][lane] == jid && tb[5 + k][lane] == jcpu) {
                        mine = true;
                        site = tb[9 + k][lane];
                        at_site |= site == second;
                    }
                if (second && at_site && S.position[j] != kTip) fixed[lane] = 1;
                const bool half = !mine && find_in_plane_table(S.tab[a], n, j, iid, icpu) >= 0;
                if (half) repair[lane] = 1;
                // a contact out of range adds exact zeros: not queued
                if (!half && site != 1 && site != 2 && rod_clear32(r12f, axi, axj, me.w + q.w + P.bw32)) return;
                if (cnt < kRodStage) {
                    const int code = ((dxs + 1) * 9 + (dys + 1) * 3 + (dzs + 1)) | (((sx + 1) * 3 + (sy + 1)) << 5) |
                                     (((site == 1 || site == 2) ? site : 0) << 9);
                    M.stage[w * 32 + lane][cnt] = make_int2(j, code);
                }
                ++cnt;
            });
        }
    }
    M.end[w][lane] = cnt;
    walk_scan(M, kRodCap);
    // the slots' own records
    if (i < n) {
        const bool walked = M.over[lane] || repair[lane];
        if (walked) {
            if (w == 0) book_slot(S, P, a, i);
        } else {
            for (int k = w; k < 13; k += kWalkCols) S.tab[b][(size_t)k * n + i] = tb[k][lane];
            if (w == 4) {
                S.fflag[i] = 0;  // flag resets of bmx_pc_interaction.cpp:178-180
                S.sflag[i] = 0;
                S.nflag[i] = 0;
                if (fixed[lane]) S.position[i] = kInterior;
            }
            if (w == 5 && any[lane])
                for (int k = 0; k < 6; ++k) S.dltd[(size_t)k * n + i] = -1;
        }
        if (w == 7) S.rcnt[i] = M.over[lane] ? kRodCap + 1 : M.end[kWalkCols - 1][lane];
    }
    // the queue: one reservation per block and end
    __syncthreads();  // (the repaired tables, written above, are read below)
    const int total = M.first[32];
    for (int t0 = 0; t0 < total; t0 += kWalkBlock) {
        const int t = t0 + tid;
        int o = 0, kind = -1, k = 0, mine = 0;
        int2 e = make_int2(0, 0);
        if (t < total) {
            e = walk_pair(M, t, o);
            k = t - M.first[o];
            if (repair[o]) {  // the site in the repaired table
                const int q = blockIdx.x * 32 + o;
                const int jb = find_in_slot_table(S.tab[b], n, q, S.id[e.x], S.cpu[e.x]);
                const int site = jb >= 0 ? S.tab[b][(size_t)(9 + jb) * n + q] : 0;
                e.y = (e.y & 0x1ff) | (((site == 1 || site == 2) ? site : 0) << 9);
            }
            kind = ((e.y >> 9) & 3) ? 1 : 0;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const unsigned m = __ballot_sync(0xffffffffu, kind == q);
            int base = 0;
            if (lane == 0 && m) base = atomicAdd(&nq[q], __popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (kind == q) mine = base + __popc(m & ((1u << lane) - 1u));
        }
        __syncthreads();
        if (tid < 2) {
            at[tid] = nq[tid] ? atomicAdd(tid ? &S.rctl->nbond : &S.rctl->ncontact, nq[tid]) : 0;
            nq[tid] = 0;
        }
        __syncthreads();
        if (kind >= 0) {
            const size_t slot = kind ? (size_t)n * kRodCap - 1 - (size_t)(at[1] + mine) : (size_t)(at[0] + mine);
            S.rwork[slot] = make_int4(blockIdx.x * 32 + o, k, e.x, e.y);
        }
        if (t0 + kWalkBlock < total) __syncthreads();
    }
}

// ---- per-segment mobility -----------------------------------------------------
// Mobility of a segment from its area, length and the viscosity
// (bmx_cell_interaction_K.H:812-840): d0 for the segment as a sphere of the
// same area, da along and db across its axis.  Stored as the combinations the
// force gather applies, (d0 + db, da - db, (d0 - db) / 2), each the FP64
// expression the gather evaluated per step before; none of the inputs changes
// during a step, so it runs when a state or the parameters load.
__device__ __forceinline__ double4_32a rod_mobility(int ctype, double Li, double sarea, const DevParams &P)
{
    double4_32a m = make_trig(0.0, 0.0, 0.0, 0.0);
    if (ctype == kFungi) {
        const double area = sarea / 2.0;
        const double arad = sqrt(area / (4.0 * kPi));
        const double d0 = 1.0 / (6.0 * kPi * arad * P.visc);
        double da, db;
        if (Li > 2.0 * arad) {
            da = (Li * Li - 2.0 * arad * arad / 3.0) / (4.0 * kPi * pow(Li, 3.0) * P.visc);
            db = (Li * Li + 2.0 * arad * arad / 3.0) / (8.0 * kPi * pow(Li, 3.0) * P.visc);
        } else {
            da = (1.0 - 3.0 * Li / (16.0 * arad)) / (6.0 * kPi * arad * P.visc);
            db = (1.0 - 9.0 * Li / (32.0 * arad)) / (6.0 * kPi * arad * P.visc);
        }
        m = make_trig(d0 + db, da - db, 0.5 * (d0 - db), 0.0);
    }
    return m;
}

__global__ void k_rod_mobility(const DevState S, const DevParams P)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n; i += gridDim.x * blockDim.x)
        S.mob[i] = rod_mobility(S.ctype[i], S.clen[i], S.area[i], P);
}

// The segments' fields of a load, gathered into slot order in one pass (18
// fields: one launch instead of a copy and a gather each), with the trig of
// the angles and the mobility.
__global__ void __launch_bounds__(128) k_load_rods(const DevState S, const DevParams P, const RodFields F,
                                                   const int *__restrict__ uperm)
{
    const size_t n = (size_t)S.n;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < S.n; s += gridDim.x * blockDim.x) {
        const int u = uperm[s];
        const double L = F.clen ? F.clen[u] : 0.0, area = F.area ? F.area[u] : 0.0;
        const double th = F.theta ? F.theta[u] : 0.0, ph = F.phi ? F.phi[u] : 0.0;
        S.clen[s] = L;
        S.area[s] = area;
        S.bscale[s] = F.bscale ? F.bscale[u] : 1.0;
        S.theta[0][s] = th;
        S.phi[0][s] = ph;
        S.id[s] = F.id ? F.id[u] : 0;
        S.cpu[s] = F.cpu ? F.cpu[u] : 0;
        S.fuse_tip[s] = F.fuse_tip ? F.fuse_tip[u] : 0;
        S.position[s] = F.position ? F.position[u] : 0;
        S.fix_site[s] = F.fix_site ? F.fix_site[u] : 0;
        S.fflag[s] = F.fflag ? F.fflag[u] : 0;
        S.sflag[s] = F.sflag ? F.sflag[u] : 0;
        S.nflag[s] = F.nflag ? F.nflag[u] : 0;
#pragma unroll
        for (int k = 0; k < 6; ++k) S.dltd[k * n + s] = F.dltd ? F.dltd[k * n + u] : -1;
        // bond table planes: n_bnds, ids[4], cpus[4], sites[4]
        int *tab = S.tab[0];
        tab[s] = F.n_bnds ? F.n_bnds[u] : 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            tab[(1 + k) * n + s] = F.seg_id1 ? F.seg_id1[k * n + u] : 0;
            tab[(5 + k) * n + s] = F.seg_id2 ? F.seg_id2[k * n + u] : 0;
            tab[(9 + k) * n + s] = F.site ? F.site[k * n + u] : 0;
        }
        double st, ct, sp, cp;
        sincos(th, &st, &ct);
        sincos(ph, &sp, &cp);
        const double4_32a tr = make_trig(ct, st, cp, sp);
        S.trig[0][s] = tr;
        S.axf[0][s] = rod_axis32(tr, L);
        S.mob[s] = rod_mobility(S.ctype[s], L, area, P);
    }
}

// Velocity (acc[0..2]) and rotation (acc[3..5]) of a segment in FP32 from its
// site-force sums Sv = sum f1 + f2 and Dv = sum f1 - f2, its mobility m and
// the growth-surface force on its two sites (bmx_cell_interaction_K.H:812-882,
// :1067-1281), the axis from ni and L instead of the difference of the two
// site positions (which FP32 would round at the magnitude of the position);
// dzc = centre height above the surface, rounded once from FP64.
__device__ __forceinline__ void rod_velocity32(const float *ni, float L, const float *Sv, const float *Dv,
                                               const double4_32a &m, float dzc, float rS, const DevParams &P,
                                               float *acc)
{
    const float m0 = d2f_rn(m.x), m1 = d2f_rn(m.y), m2 = d2f_rn(m.z);
    const float ns = ni[0] * Sv[0] + ni[1] * Sv[1] + ni[2] * Sv[2];
    float ax[3];
    for (int k = 0; k < 3; ++k) {
        acc[k] = 0.5f * (m0 * Sv[k] + m1 * ns * ni[k]);
        ax[k] = -ni[k] * L;  // site 1 minus site 2
    }
    acc[3] = m2 * (ax[1] * Dv[2] - ax[2] * Dv[1]);
    acc[4] = m2 * (ax[2] * Dv[0] - ax[0] * Dv[2]);
    acc[5] = m2 * (ax[0] * Dv[1] - ax[1] * Dv[0]);
    const float h = 0.5f * ni[2] * L;
    float w1[3] = {0.0f, 0.0f, wall_law32(dzc - h, rS, P.z_k32, P.z_bw32, P.z_g32)};
    float w2[3] = {0.0f, 0.0f, wall_law32(dzc + h, rS, P.z_k32, P.z_bw32, P.z_g32)};
    const float ra = sqrtf(ax[0] * ax[0] + ax[1] * ax[1] + ax[2] * ax[2]);
    const float un[3] = {ax[0] / ra, ax[1] / ra, ax[2] / ra};
    const float fn = (w1[2] - w2[2]) * un[2];
    float vw[3];
    for (int k = 0; k < 3; ++k) {
        w1[k] -= 0.5f * fn * un[k];
        w2[k] += 0.5f * fn * un[k];
        vw[k] = 0.5f * (w1[k] + w2[k]);
    }
    for (int k = 0; k < 3; ++k) {
        w1[k] -= 0.5f * vw[k];
        w2[k] -= 0.5f * vw[k];
    }
    acc[0] += vw[0];
    acc[1] += vw[1];
    acc[2] += vw[2];
    acc[3] += 0.5f * ((ax[1] * w1[2] - ax[2] * w1[1]) - (ax[1] * w2[2] - ax[2] * w2[1]));
    acc[4] += 0.5f * ((ax[2] * w1[0] - ax[0] * w1[2]) - (ax[2] * w2[0] - ax[0] * w2[2]));
    acc[5] += 0.5f * ((ax[0] * w1[1] - ax[1] * w1[0]) - (ax[0] * w2[1] - ax[1] * w2[0]));
}

// The same in FP64 (the plain form), from the two site positions as the
// reference computes them.
__device__ __forceinline__ void rod_velocity64(const double *ni, double Li, const double *Sv, const double *Dv,
                                               const double4_32a &mb, double xi, double yi, double zi, double ri,
                                               const DevParams &P, double *acc)
{
    const double ns = ni[0] * Sv[0] + ni[1] * Sv[1] + ni[2] * Sv[2];
    double rv[3];
    for (int k = 0; k < 3; ++k) {
        acc[k] = 0.5 * (mb.x * Sv[k] + mb.y * ns * ni[k]);
        rv[k] = (-0.5 * ni[k] * Li) - (0.5 * ni[k] * Li);  // site 1 minus site 2
    }
    const double c = mb.z;
    acc[3] = c * (rv[1] * Dv[2] - rv[2] * Dv[1]);
    acc[4] = c * (rv[2] * Dv[0] - rv[0] * Dv[2]);
    acc[5] = c * (rv[0] * Dv[1] - rv[1] * Dv[0]);
    // growth-surface force on both sites (bmx_cell_interaction_K.H:1067-1281;
    // its mobility block :1176-1265 is overwritten there and has no effect)
    double u1[3], u2[3], ax[3];
    const double pc[3] = {xi, yi, zi};
    for (int k = 0; k < 3; ++k) {
        u1[k] = pc[k] - 0.5 * ni[k] * Li;
        u2[k] = pc[k] + 0.5 * ni[k] * Li;
        ax[k] = u1[k] - u2[k];
    }
    double w1[3] = {0.0, 0.0, wall_law(u1[2], ri, P)};
    double w2[3] = {0.0, 0.0, wall_law(u2[2], ri, P)};
    Divisor by;
    (void)sqrt_rn(ax[0] * ax[0] + ax[1] * ax[1] + ax[2] * ax[2], &by);
    const double un[3] = {div_by(ax[0], by), div_by(ax[1], by), div_by(ax[2], by)};
    const double fn = (w1[0] - w2[0]) * un[0] + (w1[1] - w2[1]) * un[1] + (w1[2] - w2[2]) * un[2];
    double vw[3];
    for (int k = 0; k < 3; ++k) {
        w1[k] -= 0.5 * fn * un[k];
        w2[k] += 0.5 * fn * un[k];
    }
    for (int k = 0; k < 3; ++k) vw[k] = 0.5 * (w1[k] + w2[k]);
    for (int k = 0; k < 3; ++k) {
        w1[k] -= 0.5 * vw[k];
        w2[k] -= 0.5 * vw[k];
    }
    double rw[3];
    rw[0] = 0.5 * (ax[1] * w1[2] - ax[2] * w1[1]);
    rw[1] = 0.5 * (ax[2] * w1[0] - ax[0] * w1[2]);
    rw[2] = 0.5 * (ax[0] * w1[1] - ax[1] * w1[0]);
    rw[0] += -0.5 * (ax[1] * w2[2] - ax[2] * w2[1]);
    rw[1] += -0.5 * (ax[2] * w2[0] - ax[0] * w2[2]);
    rw[2] += -0.5 * (ax[0] * w2[1] - ax[1] * w2[0]);
    for (int k = 0; k < 3; ++k) {
        acc[k] += vw[k];
        acc[3 + k] += rw[k];
    }
}

// ---- force gather ----------------------------------------------------------
// The force gather of slot i by a walk of its stencil (fc, fix_site).
template <int PREC>
__device__ __forceinline__ void rod_force_slot(const DevState &S, const DevParams &P, int a, int i)
{
    const int b = a ^ 1;
    const int n = S.n;
    {
        const DevGeom &G = geom_of(S, i);
        int bx, by;
        col_to_bxy(G, S.col[a][i], bx, by);
        const int izi = S.iz[a][i];
        const double xi = S.x[a][i], yi = S.y[a][i], zi = S.z[a][i];
        const double ri = S.rad[i];
        const int ti = S.ctype[i];
        double acc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (ti == kYeast) {
            visit_stencil(S, G, a, i, bx, by, izi, [&](int j, int, int, int, int sx, int sy) {
                if (S.ctype[j] != kYeast) return;  // mixed pairs: no force (cutoff 0)
                double d[3];
                const double r2 = sep64(S, G, a, j, sx, sy, xi, yi, zi, d);
                if (!G.nbh_trivial && !(r2 <= P.nbh)) return;
                const double rj = S.rad[j];
                const double rlm = ri + rj + P.bw;
                if (!(r2 <= (rlm - kSmall) * (rlm - kSmall))) return;
                const double rS = ri + rj, rA = rS + P.bw;
                Divisor by;
                const double rn = sqrt_rn(r2, &by);
                const double ux = div_by(d[0], by), uy = div_by(d[1], by), uz = div_by(d[2], by);
                const double F = lt_bits(rn, rA) ? -P.k * (rn - rA) * (rn - rA) * (rn - rS) : 0.0;
                acc[0] += F * ux;
                acc[1] += F * uy;
                acc[2] += F * uz;
            });
            acc[2] += wall_law(zi, ri, P);
        } else if (ti == kFungi) {
            const double Li = S.clen[i];
            const double4_32a tri = S.trig[a][i];  // (ct, st, cp, sp)
            const double ni[3] = {tri.y * tri.z, tri.y * tri.w, tri.x};
            const int iid = S.id[i], icpu = S.cpu[i];
            const int itip = S.fuse_tip[i];
            const double bsi = S.bscale[i];
            int tb[13];
#pragma unroll
            for (int k = 0; k < 13; ++k) tb[k] = S.tab[b][(size_t)k * n + i];
            const float4 me = S.rel[a][i];
            const float4 axi = S.axf[a][i];  // FP32 axis and length
            double Sv[3] = {0.0, 0.0, 0.0}, Dv[3] = {0.0, 0.0, 0.0};
            float Svf[3] = {0.0f, 0.0f, 0.0f}, Dvf[3] = {0.0f, 0.0f, 0.0f};  // the FP32F pairs' sums
            visit_stencil(S, G, a, i, bx, by, izi, [&](int j, int dxs, int dys, int dzs, int sx, int sy) {
                if (S.ctype[j] != kFungi) return;
                const float4 axj = __ldg(&S.axf[a][j]);
                float r12f[3];
                if (!rod_gate(S, G, P, a, j, dxs, dys, dzs, sx, sy, me, axi.w, axj.w, xi, yi, zi, Li, r12f)) return;
                // bonds: mutual entries in both (repaired) tables
                int si = 0, sj = 0;
                double kb = P.k_bond;
                const int isite = table_site(tb, S.id[j], S.cpu[j]);
                if (isite != 0) {  // (an entry of site 0 bonds nothing either way)
                    const int jb = find_in_plane_table(S.tab[b], n, j, iid, icpu);
                    if (jb >= 0) {
                        si = isite;
                        sj = __ldg(&S.tab[b][(size_t)(9 + jb) * n + j]);
                        const int jtip = S.fuse_tip[j];
                        if ((itip > 0 && itip == si) || (jtip > 0 && jtip == sj)) kb = bsi * S.bscale[j] * kb;
                    }
                }
                if (PREC == BMXG_FP32F_FORM) {
                    // the pair in FP32 from the bin offsets and this step's FP32 axes,
                    // except: bonded pairs (their spring acts on the difference of
                    // two coincident end points, which FP32 end points would swamp
                    // with rounding noise: k_bond x ulp of the segment length),
                    // near-parallel segments (det < 0.05 Aii Ajj of the closest-point
                    // system: the FP64 solve) and touching or crossing segments
                    // (closest points within 1 % of the lengths: the direction of an
                    // FP32 separation is end-point rounding noise there)
                    const float nif[3] = {axi.x, axi.y, axi.z};
                    const float njf[3] = {axj.x, axj.y, axj.z};
                    const float rij = nif[0] * njf[0] + nif[1] * njf[1] + nif[2] * njf[2];
                    const bool bonded = (si == 1 || si == 2) && (sj == 1 || sj == 2);
                    if (!bonded && 1.0f - rij * rij >= 0.05f) {
                        const float rSf = me.w + __ldg(&S.rel[a][j]).w;
                        float g1[3], g2[3], rf;
                        // (not bonded: the spring constant is not used)
                        rod_site_forces<float>(r12f, nif, axi.w, njf, axj.w, rSf, rSf + P.bw32, P.k32, si, sj,
                                               0.0f, g1, g2, &rf);
                        if (rf >= 0.01f * (axi.w + axj.w)) {
                            for (int k = 0; k < 3; ++k) {
                                Svf[k] += g1[k] + g2[k];
                                Dvf[k] += g1[k] - g2[k];
                            }
                            return;
                        }
                    }
                }
                double d[3];
                sep64(S, G, a, j, sx, sy, xi, yi, zi, d);
                const double4_32a trj = S.trig[a][j];
                const double rS = ri + S.rad[j];
                const double rA = rS + P.bw;
                const double nj[3] = {trj.y * trj.z, trj.y * trj.w, trj.x};
                double f1[3], f2[3];
                rod_site_forces<double>(d, ni, Li, nj, S.clen[j], rS, rA, P.k, si, sj, kb, f1, f2);
                for (int k = 0; k < 3; ++k) {
                    Sv[k] += f1[k] + f2[k];
                    Dv[k] += f1[k] - f2[k];
                }
            });
            // mobility of segment i (bmx_cell_interaction_K.H:812-840), k_rod_mobility
            const double4_32a mb = S.mob[i];
            if (PREC == BMXG_FP32F_FORM) {
                // the FP64 pairs' sums plus the FP32 pairs' (exactly converted), rounded
                // once; velocity, rotation and the surface force in FP32
                float sv[3], dv[3], af[6];
                for (int k = 0; k < 3; ++k) {
                    sv[k] = d2f_rn(Sv[k] + f2d_int(Svf[k]));
                    dv[k] = d2f_rn(Dv[k] + f2d_int(Dvf[k]));
                }
                const float nif[3] = {axi.x, axi.y, axi.z};
                rod_velocity32(nif, axi.w, sv, dv, mb, d2f_rn(zi - P.z_wall), me.w, P, af);
                for (int k = 0; k < 6; ++k) acc[k] = f2d_int(af[k]);
                S.fix_site[i] = 0;  // evaluateSurfaceForce (bmx_cell_interaction_K.H:1060)
                for (int c = 0; c < 6; ++c) S.fc[(size_t)c * n + i] = acc[c];
                return;
            }
            rod_velocity64(ni, Li, Sv, Dv, mb, xi, yi, zi, ri, P, acc);
            S.fix_site[i] = 0;  // evaluateSurfaceForce (:1060)
        }
        for (int c = 0; c < 6; ++c) S.fc[(size_t)c * n + i] = acc[c];
    }
}

// The plain FP64 form without pair lists (no room for them).
__global__ void __launch_bounds__(128) k_rod_force(const DevState S, const DevParams P, int a)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n; i += gridDim.x * blockDim.x)
        rod_force_slot<BMXG_FP64_FORM>(S, P, a, i);
}

// ---- flat pipelines -----------------------------------------------------------
// With every segment's gated pairs queued by k_rod_book, the force gather runs
// flat, one pair per thread in full warps, instead of one stencil walk per
// thread (whose lanes diverge over pair counts and, in the FP32F form, over the
// FP32 and FP64 paths; GB300 issues FP64 at 2 lanes per clock per SM whatever
// the mask, and the FP64 walk kept 6 of 32 lanes busy).
// Plain FP64 form: k_rod_pair64 evaluates every pair, k_rod_seg adds a
// segment's pairs in list order (the walk's FP64 values in the walk's order:
// bit-identical to it).  50 000 segments in 500 trees, 10 steps and the load:
// 8.29 -> 3.35 ms when the walk became this pipeline.
// FP32F form:
//   k_rod_pair32  contacts in FP32 where the form allows (else queued for FP64),
//                 bonded pairs' springs in FP64;
//   k_rod_pair64q the queued contacts in FP64;
//   k_rod_seg     per segment: its pairs' f1 + f2 and f1 - f2 summed in FP64 in
//                 list order, then mobility and surface force in FP32, and the
//                 update.
// Each pair writes its own place, so the sums do not depend on the order in
// which the queues filled.

__device__ __forceinline__ void decode_pair(int code, int &dxs, int &dys, int &dzs, int &sx, int &sy)
{
    const int c = code & 31, s = (code >> 5) & 15;
    dxs = c / 9 - 1;
    dys = (c / 3) % 3 - 1;
    dzs = c % 3 - 1;
    sx = s / 3 - 1;
    sy = s % 3 - 1;
}

__device__ __forceinline__ void put_pair(const DevState &S, int i, int k, const double *sv, const double *dv)
{
    const size_t n = (size_t)S.n;
    for (int c = 0; c < 3; ++c) {
        S.rres[((size_t)c * kRodCap + k) * n + i] = sv[c];
        S.rres[((size_t)(3 + c) * kRodCap + k) * n + i] = dv[c];
    }
}

// Entry t of the queue: the contacts, then the bonded pairs.
__device__ __forceinline__ int4 rod_entry(const DevState &S, int t, int ncontact)
{
    return S.rwork[t < ncontact ? (size_t)t : (size_t)S.n * kRodCap - 1 - (size_t)(t - ncontact)];
}

// The bonded sites of a pair that i's repaired table bonds at isite: both when
// j's repaired table names i too.
__device__ __forceinline__ bool mutual_sites(const DevState &S, int b, int i, int j, int isite, int &si, int &sj)
{
    si = sj = 0;
    if (!isite) return false;
    const int jb = find_in_plane_table(S.tab[b], S.n, j, S.id[i], S.cpu[i]);
    if (jb < 0) return false;
    const int s2 = __ldg(&S.tab[b][(size_t)(9 + jb) * S.n + j]);
    if (s2 != 1 && s2 != 2) return false;
    si = isite;
    sj = s2;
    return true;
}

// The pair of a queue entry in FP64 (bonded: si, sj in {1, 2}).
__device__ __forceinline__ void rod_pair_fp64(const DevState &S, const DevParams &P, int a, const int4 e, int si,
                                              int sj)
{
    const int i = e.x, j = e.z;
    int dxs, dys, dzs, sx, sy;
    decode_pair(e.w, dxs, dys, dzs, sx, sy);
    const DevGeom &G = geom_of(S, i);
    double d[3];
    sep64(S, G, a, j, sx, sy, S.x[a][i], S.y[a][i], S.z[a][i], d);
    const double4_32a tri = S.trig[a][i], trj = S.trig[a][j];
    const double ni[3] = {tri.y * tri.z, tri.y * tri.w, tri.x};
    const double nj[3] = {trj.y * trj.z, trj.y * trj.w, trj.x};
    double f1[3], f2[3], sv[3], dv[3];
    if (si && sj) {
        double kb = P.k_bond;  // fusing tips (bmx_cell_interaction_K.H:552-600)
        const int itip = S.fuse_tip[i], jtip = S.fuse_tip[j];
        if ((itip > 0 && itip == si) || (jtip > 0 && jtip == sj)) kb = S.bscale[i] * S.bscale[j] * kb;
        rod_spring(d, ni, S.clen[i], nj, S.clen[j], si, sj, kb, f1, f2);
    } else {
        const double rS = S.rad[i] + S.rad[j];
        const double rA = rS + P.bw;
        rod_site_forces<double>(d, ni, S.clen[i], nj, S.clen[j], rS, rA, P.k, 0, 0, 0.0, f1, f2);
    }
    for (int c = 0; c < 3; ++c) {
        sv[c] = f1[c] + f2[c];
        dv[c] = f1[c] - f2[c];
    }
    put_pair(S, i, e.y, sv, dv);
}

__global__ void __launch_bounds__(256) k_rod_pair32(const DevState S, const DevParams P, int a)
{
    const int b = a ^ 1;
    const int nc = S.rctl->ncontact, total = nc + S.rctl->nbond;
    const int lane = threadIdx.x & 31;
    for (int t0 = blockIdx.x * blockDim.x; t0 < total; t0 += gridDim.x * blockDim.x) {
        const int t = t0 + threadIdx.x;
        bool q64 = false;
        if (t < total) {
            const int4 e = rod_entry(S, t, nc);
            const int i = e.x, j = e.z;
            int si, sj;
            if (mutual_sites(S, b, i, j, (e.w >> 9) & 3, si, sj)) {
                rod_pair_fp64(S, P, a, e, si, sj);
            } else {
                int dxs, dys, dzs, sx, sy;
                decode_pair(e.w, dxs, dys, dzs, sx, sy);
                const DevGeom &G = geom_of(S, i);
                const float4 me = S.rel[a][i], q = __ldg(&S.rel[a][j]);
                // the offsets of the gate (rod_gate), recomputed
                float r12f[3] = {(me.x - q.x) - (float)dxs * G.dxf[0], (me.y - q.y) - (float)dys * G.dxf[1],
                                 (me.z - q.z) - (float)dzs * G.dxf[2]};
                // FP32 unless near-parallel or touching (as rod_force_slot)
                q64 = true;
                const float4 axi = S.axf[a][i], axj = __ldg(&S.axf[a][j]);
                const float nif[3] = {axi.x, axi.y, axi.z};
                const float njf[3] = {axj.x, axj.y, axj.z};
                const float rij = nif[0] * njf[0] + nif[1] * njf[1] + nif[2] * njf[2];
                if (1.0f - rij * rij >= 0.05f) {
                    const float rSf = me.w + q.w;
                    float g1[3], g2[3], rf;
                    rod_site_forces<float>(r12f, nif, axi.w, njf, axj.w, rSf, rSf + P.bw32, P.k32, 0, 0, 0.0f, g1,
                                           g2, &rf);
                    if (rf >= 0.01f * (axi.w + axj.w)) {
                        double sv[3], dv[3];
                        for (int c = 0; c < 3; ++c) {
                            sv[c] = f2d_int(g1[c] + g2[c]);
                            dv[c] = f2d_int(g1[c] - g2[c]);
                        }
                        put_pair(S, i, e.y, sv, dv);
                        q64 = false;
                    }
                }
            }
        }
        // queue the FP64 contacts, one atomic per warp
        const unsigned qm = __ballot_sync(0xffffffffu, q64);
        if (qm) {
            int base = 0;
            if (lane == 0) base = atomicAdd(&S.rctl->n64, __popc(qm));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (q64) S.rq64[base + __popc(qm & ((1u << lane) - 1u))] = t;
        }
    }
}

__global__ void __launch_bounds__(64) k_rod_pair64q(const DevState S, const DevParams P, int a)
{
    const int nc = S.rctl->ncontact, nw = S.rctl->n64;
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += gridDim.x * blockDim.x)
        rod_pair_fp64(S, P, a, rod_entry(S, S.rq64[w], nc), 0, 0);
}

__global__ void __launch_bounds__(64) k_rod_pair64(const DevState S, const DevParams P, int a)
{
    const int b = a ^ 1;
    const int nc = S.rctl->ncontact, total = nc + S.rctl->nbond;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const int4 e = rod_entry(S, t, nc);
        int si, sj;
        mutual_sites(S, b, e.x, e.z, (e.w >> 9) & 3, si, sj);
        rod_pair_fp64(S, P, a, e, si, sj);
    }
}

// ---- update ---------------------------------------------------------------
// The update of slot i from its velocity fc[0..2] and rotation fc[3..5].
__device__ __forceinline__ void rod_update_slot(const DevState &S, double dt, int a, int i, const double *fc)
{
    const int b = a ^ 1;
    const DevGeom &G = geom_of(S, i);
    const double v[3] = {fc[0], fc[1], fc[2]}, w[3] = {fc[3], fc[4], fc[5]};
    S.vx[i] = v[0];
    S.vy[i] = v[1];
    S.vz[i] = v[2];
    S.wx[i] = w[0];
    S.wy[i] = w[1];
    S.wz[i] = w[2];
    double nx = S.x[a][i] + dt * v[0];
    double ny = S.y[a][i] + dt * v[1];
    const double nz = S.z[a][i] + dt * v[2];
    double th = S.theta[a][i], ph = S.phi[a][i];
    double4_32a tr = S.trig[a][i];
    if (S.ctype[i] == kFungi) {
        // rotate the axis by |omega| dt (bmx_pc_interaction.cpp:334-431)
        const double ct = tr.x, st = tr.y, cp = tr.z, sp = tr.w;
        const double R[3][3] = {{cp * st, -sp, -cp * ct}, {sp * st, cp, -sp * ct}, {ct, 0.0, st}};
        double om[3];
        for (int r = 0; r < 3; ++r) {
            om[r] = 0.0;
            for (int c = 0; c < 3; ++c) om[r] += R[c][r] * w[c];
        }
        const double L = S.clen[i];
        om[0] = 0.0;
        const double oL = div_rn(2.0, L * L);
        om[1] *= oL;
        om[2] *= oL;
        Divisor by;
        const double on = sqrt_rn(om[1] * om[1] + om[2] * om[2], &by);
        if (on > 0.0) {
            om[1] = div_by(om[1], by);
            om[2] = div_by(om[2], by);
        }
        const double c = om[2], s = om[1];
        const double Q[3][3] = {{1.0, 0.0, 0.0}, {0.0, c, -s}, {0.0, s, c}};
        const double ang = on * dt;
        double sa, ca;
        sincos(ang, &sa, &ca);  // one argument reduction for both
        const double u[3] = {ca, sa, 0.0};
        double q[3], nd[3];
        for (int r = 0; r < 3; ++r) {
            q[r] = 0.0;
            for (int cc = 0; cc < 3; ++cc) q[r] += Q[cc][r] * u[cc];
        }
        for (int r = 0; r < 3; ++r) {
            nd[r] = 0.0;
            for (int cc = 0; cc < 3; ++cc) nd[r] += R[r][cc] * q[cc];
        }
        th = acos(nd[2]);
        const double rho = sqrt_rn(nd[0] * nd[0] + nd[1] * nd[1], &by);
        if (rho > 0.0) nd[0] = div_by(nd[0], by);
        ph = acos(nd[0]);
        if (nd[1] < 0.0) ph = 2.0 * kPi - ph;
        double st2, ct2, sp2, cp2;
        sincos(th, &st2, &ct2);
        sincos(ph, &sp2, &cp2);
        tr = make_trig(ct2, st2, cp2, sp2);
    }
    S.theta[b][i] = th;
    S.phi[b][i] = ph;
    S.trig[b][i] = tr;
    S.axf[b][i] = rod_axis32(tr, S.clen[i]);
    if (G.per[0]) nx = wrap1(nx, G.plo[0], G.phi[0], G.len[0]);
    if (G.per[1]) ny = wrap1(ny, G.plo[1], G.phi[1], G.len[1]);
    S.x[b][i] = nx;
    S.y[b][i] = ny;
    S.z[b][i] = nz;
    rebin_slot(S, G, i, nx, ny, nz, S.rad[i], b);
}

// (contexts without room for the pipelines' queues, after k_rod_force)
__global__ void k_rod_update(const DevState S, double dt, int a)
{
    const size_t n = (size_t)S.n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n; i += gridDim.x * blockDim.x) {
        double fc[6];
        for (int c = 0; c < 6; ++c) fc[c] = S.fc[c * n + i];
        rod_update_slot(S, dt, a, i, fc);
    }
}

// A segment's pairs summed in list order, as the walk adds them, then mobility,
// surface force and update in one pass (the six force planes between a segment
// and an update kernel never leave the registers).  Spheres of a mixed state,
// and segments with more pairs than the queue holds: the walk.
template <int PREC>
__global__ void __launch_bounds__(64) k_rod_seg(const DevState S, const DevParams P, double dt, int a)
{
    const size_t n = (size_t)S.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S.n) return;
    double fc[6];
    const int cnt = S.rcnt[i];
    if (S.ctype[i] != kFungi || cnt > kRodCap) {
        rod_force_slot<PREC>(S, P, a, i);
        for (int c = 0; c < 6; ++c) fc[c] = S.fc[c * n + i];
    } else {
        double Sv[3] = {0.0, 0.0, 0.0}, Dv[3] = {0.0, 0.0, 0.0};
        for (int k = 0; k < cnt; ++k)
            for (int c = 0; c < 3; ++c) {
                Sv[c] += S.rres[((size_t)c * kRodCap + k) * n + i];
                Dv[c] += S.rres[((size_t)(3 + c) * kRodCap + k) * n + i];
            }
        if (PREC == BMXG_FP64_FORM) {
            const double4_32a tri = S.trig[a][i];
            const double ni[3] = {tri.y * tri.z, tri.y * tri.w, tri.x};
            rod_velocity64(ni, S.clen[i], Sv, Dv, S.mob[i], S.x[a][i], S.y[a][i], S.z[a][i], S.rad[i], P, fc);
        } else {
            const float4 axi = S.axf[a][i];
            float sv[3], dv[3], af[6];
            for (int c = 0; c < 3; ++c) {
                sv[c] = d2f_rn(Sv[c]);
                dv[c] = d2f_rn(Dv[c]);
            }
            const float nif[3] = {axi.x, axi.y, axi.z};
            rod_velocity32(nif, axi.w, sv, dv, S.mob[i], d2f_rn(S.z[a][i] - P.z_wall), S.rel[a][i].w, P, af);
            for (int c = 0; c < 6; ++c) fc[c] = f2d_int(af[c]);
        }
        S.fix_site[i] = 0;  // evaluateSurfaceForce (bmx_cell_interaction_K.H:1060)
    }
    rod_update_slot(S, dt, a, i, fc);
}

// ---- InitBonds ---------------------------------------------------------------
// Start-up bond detection (bmx_pc_interaction.cpp:500-626 with fixBonds,
// bmx_cell_interaction_K.H:1287-1440): for every listed FUNGI-FUNGI pair
// within the interaction gate, the four end pairs (i1,j1), (i2,j1), (i1,j2),
// (i2,j2) are tried in that order and the first closer than rlim appends
// (id_j, cpu_j, site of i) to i's table.  As in the force gather, the
// neighbour is a copy, so only i's own table changes; each thread owns its
// row and appends in the reference's list order.  A fifth bond (past the
// reference's four table slots) is counted, not written.
__global__ void k_init_bonds(const DevState S, const DevParams P, int a, double rlim,
                             unsigned long long *counts)
{
    const int n = S.n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (S.ctype[i] != kFungi) continue;
        const DevGeom &G = geom_of(S, i);
        int bx, by;
        col_to_bxy(G, S.col[a][i], bx, by);
        const double xi = S.x[a][i], yi = S.y[a][i], zi = S.z[a][i];
        const double Li = S.clen[i];
        const double4_32a tri = S.trig[a][i];
        const double ni[3] = {tri.y * tri.z, tri.y * tri.w, tri.x};
        int nb = S.tab[a][i];
        unsigned long long add = 0, over = 0;
        visit_stencil(S, G, a, i, bx, by, S.iz[a][i], [&](int j, int, int, int, int sx, int sy) {
            if (S.ctype[j] != kFungi) return;
            double d[3];
            const double r2 = sep64(S, G, a, j, sx, sy, xi, yi, zi, d);
            if (!G.nbh_trivial && !(r2 <= P.nbh)) return;
            const double Lj = S.clen[j];
            const double rlm = 1.5 * (Li + Lj) + P.bw;
            if (!(r2 <= (rlm - kSmall) * (rlm - kSmall))) return;
            const double4_32a trj = S.trig[a][j];
            const double nj[3] = {trj.y * trj.z, trj.y * trj.w, trj.x};
            double e[4][3];  // i1, i2, j1, j2 with j's centre at the origin
            for (int k = 0; k < 3; ++k) {
                e[0][k] = d[k] - 0.5 * ni[k] * Li;
                e[1][k] = d[k] + 0.5 * ni[k] * Li;
                e[2][k] = -0.5 * nj[k] * Lj;
                e[3][k] = 0.5 * nj[k] * Lj;
            }
            for (int m = 0; m < 4; ++m) {
                const int si = (m & 1) + 1, sj = (m >> 1) + 1;  // (1,1) (2,1) (1,2) (2,2)
                const double *p = e[si - 1], *q = e[1 + sj];
                const double rx = p[0] - q[0], ry = p[1] - q[1], rz = p[2] - q[2];
                if (sqrt(rx * rx + ry * ry + rz * rz) < rlim) {
                    if (nb >= 0 && nb < 4) {
                        S.tab[a][(size_t)(1 + nb) * n + i] = S.id[j];
                        S.tab[a][(size_t)(5 + nb) * n + i] = S.cpu[j];
                        S.tab[a][(size_t)(9 + nb) * n + i] = si;
                        ++nb;
                        ++add;
                    } else {
                        ++over;
                    }
                    break;
                }
            }
        });
        S.tab[a][i] = nb;
        if (add) atomicAdd(&counts[0], add);
        if (over) atomicAdd(&counts[1], over);
    }
}

// ---- ParticleExchange --------------------------------------------------------
// One substep of BMXParticleContainer::ParticleExchange (bmx_pc_xchng.cpp:13-257)
// with initExchange / evaluateExchange / applyIncrements
// (bmx_chem_K.H:1949-2126): over the step's neighbour list, every FUNGI
// segment i sums, for each listed FUNGI neighbour j that i and j both hold in
// their bond tables, -d / vol_i with d = (c_i - c_j) * area * mt * dt
// (area = pi (r_i^2 + r_j^2) / 2), d clamped so that neither side loses more
// than its concentration over its bond count, and adds the sum to its
// concentrations.  The reference's write to j's increment goes to a by-value
// neighbour copy and is lost; the result reads only concentrations from
// before the substep, so the kernel writes a separate output.  Same
// arithmetic, in the same order, as the reference (FP64, no contraction).
__global__ void k_exchange(const DevState S, const DevParams P, int a, const double *vol, const double *conc,
                           double *out, double dt, double mtA, double mtB, double mtC)
{
    const int n = S.n;
    const double pi = 3.14159265358979323846;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double a1 = conc[i], b1 = conc[(size_t)n + i], c1 = conc[(size_t)2 * n + i];
        double inc[3] = {0.0, 0.0, 0.0};
        if (S.ctype[i] == kFungi) {
            const DevGeom &G = geom_of(S, i);
            int bx, by;
            col_to_bxy(G, S.col[a][i], bx, by);
            const double xi = S.x[a][i], yi = S.y[a][i], zi = S.z[a][i];
            int tb[13];
            for (int k = 0; k < 13; ++k) tb[k] = S.tab[a][(size_t)k * n + i];
            const int iid = S.id[i], icpu = S.cpu[i];
            const double r1 = S.rad[i], v1 = vol[i];
            const double area1 = pi * r1 * r1;
            const double ni = (double)tb[0];
            visit_stencil(S, G, a, i, bx, by, S.iz[a][i], [&](int j, int, int, int, int sx, int sy) {
                if (S.ctype[j] != kFungi) return;
                if (!G.nbh_trivial) {  // BMXCheckPair: j is in i's list only within the neighbourhood
                    double d[3];
                    if (!(sep64(S, G, a, j, sx, sy, xi, yi, zi, d) <= P.nbh)) return;
                }
                if (find_in_table(tb, S.id[j], S.cpu[j]) < 0) return;
                if (find_in_plane_table(S.tab[a], n, j, iid, icpu) < 0) return;
                const double a2 = conc[j], b2 = conc[(size_t)n + j], c2 = conc[(size_t)2 * n + j];
                const double r2 = S.rad[j], v2 = vol[j];
                const double area2 = pi * r2 * r2;
                const double area = 0.5 * (area1 + area2);
                const double nj = (double)S.tab[a][j];
                double dA = (a1 - a2) * area * mtA * dt;
                double dB = (b1 - b2) * area * mtB * dt;
                double dC = (c1 - c2) * area * mtC * dt;
                if (dA / v1 > a1 / ni) dA = a1 * v1 / ni;
                if (-dA / v2 > a2 / nj) dA = -a2 * v2 / nj;
                if (dB / v1 > b1 / ni) dB = b1 * v1 / ni;
                if (-dB / v2 > b2 / nj) dB = -b2 * v2 / nj;
                if (dC / v1 > c1 / ni) dC = c1 * v1 / ni;
                if (-dC / v2 > c2 / nj) dC = -c2 * v2 / nj;
                inc[0] -= dA / v1;
                inc[1] -= dB / v1;
                inc[2] -= dC / v1;
            });
        }
        out[i] = a1 + inc[0];
        out[(size_t)n + i] = b1 + inc[1];
        out[(size_t)2 * n + i] = c1 + inc[2];
    }
}

}  // namespace

int launch_exchange(const DevState &S, const DevParams &P, int a, const double *vol, const double *conc, double *out,
                    double dt, const double *xpar, int grid, int block, cudaStream_t st)
{
    k_exchange<<<grid, block, 0, st>>>(S, P, a, vol, conc, out, dt, xpar[0], xpar[1], xpar[2]);
    return 1;
}

int launch_rod_mobility(const DevState &S, const DevParams &P, int grid, int block, cudaStream_t st)
{
    k_rod_mobility<<<grid, block, 0, st>>>(S, P);
    return 1;
}

int launch_load_rods(const DevState &S, const DevParams &P, const RodFields &F, const int *uperm, int grid, int block,
                     cudaStream_t st)
{
    k_load_rods<<<grid, block, 0, st>>>(S, P, F, uperm);
    return 1;
}

int launch_rod_book(const DevState &S, const DevParams &P, int a, bool list, int grid, int block, cudaStream_t st)
{
    if (list) k_rod_book<<<(S.n + 31) / 32, kWalkBlock, sizeof(WalkMem<32, kRodStage>), st>>>(S, P, a);
    else k_rod_book_plain<<<grid, block, 0, st>>>(S, P, a);
    return 1;
}

int launch_rod_pairs(const DevState &S, const DevParams &P, double dt, int a, int precision, int nsm, int n,
                     cudaStream_t st)
{
    const int grid = (n + 63) / 64;
    if (precision == BMXG_FP64_FORM) {
        k_rod_pair64<<<nsm * 8, 64, 0, st>>>(S, P, a);
        k_rod_seg<BMXG_FP64_FORM><<<grid, 64, 0, st>>>(S, P, dt, a);
        return 2;
    }
    k_rod_pair32<<<nsm * 4, 128, 0, st>>>(S, P, a);
    k_rod_pair64q<<<nsm * 4, 64, 0, st>>>(S, P, a);
    k_rod_seg<BMXG_FP32F_FORM><<<grid, 64, 0, st>>>(S, P, dt, a);
    return 3;
}

int launch_rod_force(const DevState &S, const DevParams &P, int a, int grid, int block, cudaStream_t st)
{
    k_rod_force<<<grid, block, 0, st>>>(S, P, a);
    return 1;
}

int launch_rod_update(const DevState &S, double dt, int a, int grid, int block, cudaStream_t st)
{
    k_rod_update<<<grid, block, 0, st>>>(S, dt, a);
    return 1;
}

int launch_init_bonds(const DevState &S, const DevParams &P, int a, double rlim, unsigned long long *counts,
                      int grid, int block, cudaStream_t st)
{
    k_init_bonds<<<grid, block, 0, st>>>(S, P, a, rlim, counts);
    return 1;
}

}  // namespace bmxg
