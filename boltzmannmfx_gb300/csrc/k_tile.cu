// k_tile.cu -- the FP64 sphere step of one tile with the caller's ghost
// particles: AMReX's per-tile EvolveParticles (src/des/bmx_pc_interaction.cpp:
// 97-279 with the halo of one cell of src/des/bmx_pc.cpp:23), where
// fillNeighbors has put copies of the particles of the neighbouring tiles --
// periodic images already shifted by a domain length -- beside the tile's own.
//
// The tile's cells are the level's global cells (the particle's cell from the
// domain origin, as the whole-domain step bins it) offset by the tile's first
// cell; the grown box adds the one-cell halo that holds the ghosts.  A real
// particle walks the 27 cells around its own in the whole-domain step's
// order (x outermost, then y, then z, ascending index within a cell: the
// tile's reals in the caller's order, then its ghosts in theirs), and each
// pair is evaluated with the whole-domain step's FP64 operations on the
// ghost's given position.  So with the ghosts a whole-domain step would see
// (copies of every particle within one cell of the tile, images at x + s L),
// the tiles' results are bit-identical to the step of the whole domain.
//
// The tile is laid out as a state of its own: the grown tile's (x, y) cells are
// columns sorted by z cell and index, with FP32 offsets from the cells' corners,
// so that the step screens its candidates in FP32 and walks one column per warp
// as the whole-domain step of a small state does.  A call is a clear, four
// kernels and one read-back on a workspace the context keeps (18 allocations
// and a gather and a copy per array before): a quarter of a 20 000-sphere level
// (5000 reals and their ghosts) takes 68 us a call, 334 before (369 with one
// thread per real and the FP64 gate on every candidate and FP64 divisions).
#include "bmxg_stencil.cuh"

namespace bmxg {

namespace {

// Every particle (reals [0, nreal), then ghosts) into the workspace: its cell
// in the grown tile box, the column counts, its FP32 offsets.  bad[0] counts a
// real outside the tile or a ghost outside the halo, bad[1] a particle that is
// not a sphere (YEAST).
__global__ void __launch_bounds__(128) k_tile_bin(const TileCall C, const TileGeom T)
{
    const DevState &S = C.S;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= S.n) return;
    const bool real = p < C.nreal;
    const int q = real ? p : p - C.nreal;
    const double pos[3] = {real ? C.rx[q] : C.gx[q], real ? C.ry[q] : C.gy[q], real ? C.rz[q] : C.gz[q]};
    const double r = real ? C.rr[q] : C.gr[q];
    const int ct = real ? C.rct[q] : C.gct[q];
    int l[3];
    float rel[3];
    bool halo = false, out = false;
    for (int d = 0; d < 3; ++d) {
        // the whole-domain step's bin (1-based): a slot's own clamped to the
        // domain, a periodic image's the halo cell its shifted position is in
        const int gb = (real || !T.per[d]) ? bin_of(pos[d], T.plo[d], T.dxi[d], 1, T.n[d])
                                            : bin_of(pos[d], T.plo[d], T.dxi[d], 0, T.n[d] + 1);
        int lb = gb - T.lo[d];
        if (lb < 0 || lb > T.nt[d] + 1) {
            out = true;
            lb = min(max(lb, 0), T.nt[d] + 1);
        }
        if (lb == 0 || lb == T.nt[d] + 1) halo = true;
        l[d] = lb;
        // beyond its cell (clamped, or not finite): NaN, which no FP32 screen rejects
        const float f = (float)(pos[d] - (T.plo[d] + (double)(gb - 1) * T.dx[d]));
        rel[d] = (f >= -0.5f * T.dxf[d] && f <= 1.5f * T.dxf[d]) ? f : __int_as_float(0x7fc00000);
    }
    if (out || (real ? halo : !halo)) atomicAdd(&C.bad[0], 1ull);
    if (ct != kYeast) atomicAdd(&C.bad[1], 1ull);
    const int c = l[0] * (T.nt[1] + 2) + l[1];
    S.x[0][p] = pos[0];
    S.y[0][p] = pos[1];
    S.z[0][p] = pos[2];
    S.rad[p] = r;
    S.col[0][p] = c;
    S.iz[0][p] = l[2];
    S.rel[0][p] = make_float4(rel[0], rel[1], rel[2], d2f_rn(r));
    atomicAdd(&S.colcnt[c], 1);
}

// Slots are sorted positions, so a warp's lanes walk the same or adjacent
// columns; the ghosts among them idle.
template <int NS, int STAGE>
__global__ void __launch_bounds__(kWalkBlock, 3) k_tile_step(const TileCall C, const TileGeom T, const DevParams P,
                                                             double dt)
{
    extern __shared__ __align__(16) unsigned char smw[];
    auto &M = *reinterpret_cast<WalkMem<NS, STAGE> *>(smw);
    __shared__ double opos[NS][4];
    __shared__ double term[3 * kWalkBlock];
    __shared__ unsigned char opass[kWalkBlock];
    const DevState &S = C.S;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const float slack = 8.0f * 1.1920929e-7f * fmaxf(T.dxf[0], fmaxf(T.dxf[1], T.dxf[2]));
    // the candidates of slot i at sorted position t in column offset (dx, dy): f(candidate)
    auto column = [&](int t, int i, int dx, int dy, auto &&f) {
        const int c = S.col[0][i];
        const int lx = c / (T.nt[1] + 2) + dx, ly = c % (T.nt[1] + 2) + dy;
        // (a real outside its tile, an input error the call reports, has cells outside the grown box: skipped)
        if (lx < 0 || lx > T.nt[0] + 1 || ly < 0 || ly > T.nt[1] + 1) return;
        const int cc = lx * (T.nt[1] + 2) + ly;
        const float4 me = S.srel[0][t];
        const float ox = (float)dx * T.dxf[0], oy = (float)dy * T.dxf[1];
        walk_column(S, 0, __ldg(&S.colstart[0][cc]), __ldg(&S.colstart[0][cc + 1]), t, S.siz[0][t],
                    [&](int u, const float4 q, int dzs) {
                        if (near_pair32(me, q, ox, oy, (float)dzs * T.dxf[2], P.bw32, slack)) f(__ldg(&S.perm[0][u]));
                    });
    };
    for (int g = 0; g < NS; g += 32) {
        const int s = g + lane;
        const int t = blockIdx.x * NS + s;
        const int i = t < S.n ? S.perm[0][t] : S.n;
        int cnt = 0;
        if (i < C.nreal) {
            if (w == 0) {
                opos[s][0] = S.x[0][i];
                opos[s][1] = S.y[0][i];
                opos[s][2] = S.z[0][i];
                opos[s][3] = S.rad[i];
            }
            column(t, i, w / 3 - 1, w % 3 - 1, [&](int j) {
                if (cnt < STAGE) M.stage[w * NS + s][cnt] = make_int2(j, 0);
                ++cnt;
            });
        }
        M.end[w][s] = cnt;
    }
    walk_scan(M);
    // the whole-domain step's pair term (sphere_term64), on the ghost's given position
    auto pair = [&](int s, int j, double *t) {
        return sphere_pair64(P, T.nbh_trivial, opos[s][0] - S.x[0][j], opos[s][1] - S.y[0][j],
                             opos[s][2] - S.z[0][j], opos[s][3], S.rad[j], t);
    };
    double fx = 0.0, fy = 0.0, fz = 0.0;
    walk_pairs<3>(
        M, term, opass, [&](int o, int2 e, double *t) { return pair(o, e.x, t); },
        [&](const double *t) {
            fx += t[0];
            fy += t[kWalkBlock];
            fz += t[2 * kWalkBlock];
        });
    const int t = blockIdx.x * NS + tid;
    if (tid >= NS || t >= S.n) return;
    const int i = S.perm[0][t];
    if (i >= C.nreal) return;
    if (M.over[tid])  // a crowded column: every pair evaluated as it is met
        for (int c = 0; c < kWalkCols; ++c)
            column(t, i, c / 3 - 1, c % 3 - 1, [&](int j) {
                double q[3];
                if (pair(tid, j, q)) {
                    fx += q[0];
                    fy += q[1];
                    fz += q[2];
                }
            });
    // evaluateSurfaceForce (sphere branch), the update, and the periodic
    // wrap of the trailing Redistribute, as the whole-domain step
    const double xi = opos[tid][0], yi = opos[tid][1], zi = opos[tid][2];
    const double v0 = plus_zero(fx);
    const double v1 = plus_zero(fy);
    const double v2 = fz + wall_law(zi, opos[tid][3], P);
    double nx = xi + dt * v0;
    double ny = yi + dt * v1;
    const double nz = zi + dt * v2;
    if (T.per[0]) nx = wrap1(nx, T.plo[0], T.phi[0], T.len[0]);
    if (T.per[1]) ny = wrap1(ny, T.plo[1], T.phi[1], T.len[1]);
    if (!finite_bits(nx) || !finite_bits(ny) || !finite_bits(nz)) atomicAdd(&C.bad[2], 1ull);
    const size_t n = (size_t)C.nreal;
    C.out[i] = nx;
    C.out[n + i] = ny;
    C.out[2 * n + i] = nz;
    C.out[3 * n + i] = v0;
    C.out[4 * n + i] = v1;
    C.out[5 * n + i] = v2;
}

struct TileDst {
    double *d[6];
};

// the results into the caller's arrays, unless the input was bad
__global__ void __launch_bounds__(128) k_tile_out(const double *__restrict__ out, int n, const TileDst D,
                                                  const unsigned long long *bad)
{
    if (bad[0] || bad[1]) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
#pragma unroll
    for (int k = 0; k < 6; ++k) D.d[k][i] = out[(size_t)k * n + i];
}

}  // namespace

int launch_tile_step(const TileCall &C, const TileGeom &T, const DevParams &P, double dt, int *scan_scratch,
                     double *const dst[6], cudaStream_t st)
{
    const int n = C.S.n, blk = 128;
    k_tile_bin<<<(n + blk - 1) / blk, blk, 0, st>>>(C, T);
    int k = 1 + launch_rebuild(C.S, 0, scan_scratch, (n + blk - 1) / blk, blk, st);
    // 32 slots per block while that leaves SMs without work, then 128
    if (n <= kWalkNarrow) {
        k_tile_step<32, 6><<<(n + 31) / 32, kWalkBlock, sizeof(WalkMem<32, 6>), st>>>(C, T, P, dt);
    } else {
        static_assert(sizeof(WalkMem<128, 3>) + 128 * 32 + 3 * kWalkBlock * 8 + kWalkBlock <= 48 * 1024,
                      "within the default shared memory");
        k_tile_step<128, 3><<<(n + 127) / 128, kWalkBlock, sizeof(WalkMem<128, 3>), st>>>(C, T, P, dt);
    }
    ++k;
    if (dst) {
        const TileDst D{{dst[0], dst[1], dst[2], dst[3], dst[4], dst[5]}};
        k_tile_out<<<(C.nreal + blk - 1) / blk, blk, 0, st>>>(C.out, C.nreal, D, C.bad);
        ++k;
    }
    return k;
}

}  // namespace bmxg
