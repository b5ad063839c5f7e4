// k_io.cu -- the state out to caller order in one pass, and the reference's AoS
// records (amrex::Particle<nreal, nint>: pos, rdata, id, cpu, idata;
// src/chemistry/bmx_chem.H:16-17, 38-118) in and out.
//
// Both are gathers and scatters of a few hundred bytes per particle; a launch
// and a copy per field cost more than the bytes for all but the largest
// states: 50 000 segments, load, 10 FP64 steps and store 2.96 -> 2.71 ms.
// Records in host memory are read and written in place where the device
// shares the host's page tables (GB300: NVLink-C2C), and only the words the
// step uses: a step of 400 segments 687 -> 213 us, of 20 011 cells (with the
// caller's own 9 MB copy of them) 1442 -> 762 us, against packing loops on the
// host and a copy per field.  (A copy of whole records runs at 170 GB/s from
// pageable memory, 62 us each way for those cells; the words a sphere step reads
// and writes take 25 and 77 us.)
#include <algorithm>
#include <type_traits>

#include "bmxg_fx.cuh"
#include "bmxg_kernels.cuh"
#include "bmxg_stencil.cuh"

namespace bmxg {

namespace {

// realIdx and intIdx positions (src/chemistry/bmx_chem.H:38-118)
enum {
    R_radius = 0, R_c_length = 1, R_theta = 2, R_phi = 3, R_area = 4, R_velx = 6, R_bond_scale = 24
};
enum {
    I_cell_type = 5, I_n_bnds = 6, I_seg1_id1 = 7, I_seg1_id2 = 11, I_site1 = 15, I_position = 19, I_fuse_flag = 20,
    I_split_flag = 21, I_new_flag = 22, I_fuse_tip = 25, I_dltd_site1 = 26, I_fix_site = 32, I_id = 33, I_cpu = 34
};

template <bool FX, bool V32>
__global__ void __launch_bounds__(256) k_store(const DevState S, int a, const StoreFields F)
{
    const size_t n = (size_t)S.n;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < S.n; s += gridDim.x * blockDim.x) {
        const int u = S.orig[s];
        double x, y, z;
        if (FX) {
            const FxGeom &X = S.fxg[colony_of(S.cbase, S.ncol, s)];
            const int4 h = S.fxh[a][s];
            x = from_fx(fx_join((unsigned)h.x, S.fxl[a][s]), X, 0);
            y = from_fx(fx_join((unsigned)h.y, S.fxl[a][n + s]), X, 1);
            z = from_fx(fx_join((unsigned)h.z, S.fxl[a][2 * n + s]), X, 2);
            S.x[a][s] = x;
            S.y[a][s] = y;
            S.z[a][s] = z;
        }
        if ((unsigned)u >= (unsigned)S.n) continue;
        if (F.x) F.x[u] = FX ? x : S.x[a][s];
        if (F.y) F.y[u] = FX ? y : S.y[a][s];
        if (F.z) F.z[u] = FX ? z : S.z[a][s];
        if (F.v[0]) F.v[0][u] = V32 ? (double)S.vxf[s] : S.vx[s];
        if (F.v[1]) F.v[1][u] = V32 ? (double)S.vyf[s] : S.vy[s];
        if (F.v[2]) F.v[2][u] = V32 ? (double)S.vzf[s] : S.vz[s];
        if (F.v[3]) F.v[3][u] = S.wx[s];
        if (F.v[4]) F.v[4][u] = S.wy[s];
        if (F.v[5]) F.v[5][u] = S.wz[s];
        if (!S.has_rods) continue;
        if (F.theta) F.theta[u] = S.theta[a][s];
        if (F.phi) F.phi[u] = S.phi[a][s];
        const int *tab = S.tab[a];
        if (F.n_bnds) F.n_bnds[u] = tab[s];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (F.seg_id1) F.seg_id1[k * n + u] = tab[(1 + k) * n + s];
            if (F.seg_id2) F.seg_id2[k * n + u] = tab[(5 + k) * n + s];
            if (F.site) F.site[k * n + u] = tab[(9 + k) * n + s];
        }
        if (F.position) F.position[u] = S.position[s];
        if (F.fix_site) F.fix_site[u] = S.fix_site[s];
        if (F.fflag) F.fflag[u] = S.fflag[s];
        if (F.sflag) F.sflag[u] = S.sflag[s];
        if (F.nflag) F.nflag[u] = S.nflag[s];
        if (F.dltd) {
#pragma unroll
            for (int k = 0; k < 6; ++k) F.dltd[k * n + u] = S.dltd[k * n + s];
        }
    }
}

template <bool RODS>
__global__ void __launch_bounds__(128) k_aos_load(const unsigned char *rec, const AosLayout L, int n, double *d, int *o)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n) return;
    const size_t N = (size_t)n;
    const double *p = reinterpret_cast<const double *>(rec + (size_t)u * L.stride);
    const double *r = reinterpret_cast<const double *>(rec + (size_t)u * L.stride + L.rdata);
    const int *q = reinterpret_cast<const int *>(rec + (size_t)u * L.stride + L.idata);
    for (int k = 0; k < 3; ++k) d[k * N + u] = p[k];
    d[3 * N + u] = r[R_radius];
    for (int k = 0; k < 6; ++k) d[(9 + k) * N + u] = r[R_velx + k];
    o[u] = q[I_cell_type];
    if (!RODS) return;
    d[4 * N + u] = r[R_c_length];
    d[5 * N + u] = r[R_theta];
    d[6 * N + u] = r[R_phi];
    d[7 * N + u] = r[R_area];
    d[8 * N + u] = r[R_bond_scale];
    o[N + u] = q[I_id];
    o[2 * N + u] = q[I_cpu];
    o[3 * N + u] = q[I_n_bnds];
    for (int k = 0; k < 12; ++k) o[(4 + k) * N + u] = q[I_seg1_id1 + k];  // seg_id1, seg_id2, site
    o[16 * N + u] = q[I_position];
    o[17 * N + u] = q[I_fuse_tip];
    o[18 * N + u] = q[I_fix_site];
    o[19 * N + u] = q[I_fuse_flag];
    o[20 * N + u] = q[I_split_flag];
    o[21 * N + u] = q[I_new_flag];
    for (int k = 0; k < 6; ++k) o[(22 + k) * N + u] = q[I_dltd_site1 + k];
}

// pos, velx .. wz, theta, phi and the integer fields the step's pair loop and
// wall force write (spheres: the position, the velocity and the three flags,
// which a step clears)
__global__ void __launch_bounds__(128) k_aos_store(unsigned char *rec, const AosLayout L, const DevState S, int a)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S.n) return;
    const size_t n = (size_t)S.n;
    const int u = S.orig[s];
    if ((unsigned)u >= (unsigned)S.n) return;
    double *p = reinterpret_cast<double *>(rec + (size_t)u * L.stride);
    double *r = reinterpret_cast<double *>(rec + (size_t)u * L.stride + L.rdata);
    int *q = reinterpret_cast<int *>(rec + (size_t)u * L.stride + L.idata);
    p[0] = S.x[a][s];
    p[1] = S.y[a][s];
    p[2] = S.z[a][s];
    r[R_velx] = S.vx[s];
    r[R_velx + 1] = S.vy[s];
    r[R_velx + 2] = S.vz[s];
    if (!S.has_rods) {
        q[I_fuse_flag] = 0;
        q[I_split_flag] = 0;
        q[I_new_flag] = 0;
        return;
    }
    r[R_velx + 3] = S.wx[s];
    r[R_velx + 4] = S.wy[s];
    r[R_velx + 5] = S.wz[s];
    r[R_theta] = S.theta[a][s];
    r[R_phi] = S.phi[a][s];
    const int *tab = S.tab[a];
    q[I_n_bnds] = tab[s];
    for (int k = 0; k < 12; ++k) q[I_seg1_id1 + k] = tab[(1 + k) * n + s];
    q[I_position] = S.position[s];
    q[I_fix_site] = S.fix_site[s];
    q[I_fuse_flag] = S.fflag[s];
    q[I_split_flag] = S.sflag[s];
    q[I_new_flag] = S.nflag[s];
    for (int k = 0; k < 6; ++k) q[I_dltd_site1 + k] = S.dltd[k * n + s];
}

}  // namespace

namespace {

// One field of `PLANES` planes to caller order.
template <int PLANES, class D, class T>
__global__ void __launch_bounds__(256) k_scatter_field(D *dst, const T *src, const int *orig, int n)
{
    const int s = blockIdx.x * 256 + threadIdx.x;
    if (s >= n) return;
    const int u = orig[s];
    if ((unsigned)u >= (unsigned)n) return;
#pragma unroll
    for (int p = 0; p < PLANES; ++p) dst[(size_t)p * n + u] = (D)src[(size_t)p * n + s];
}

int store_pass(const DevState &S, int a, const StoreFields &F, bool fx, bool vel32, cudaStream_t st)
{
    const int grid = (S.n + 255) / 256;
    if (fx && vel32) k_store<true, true><<<grid, 256, 0, st>>>(S, a, F);
    else if (fx) k_store<true, false><<<grid, 256, 0, st>>>(S, a, F);
    else if (vel32) k_store<false, true><<<grid, 256, 0, st>>>(S, a, F);
    else k_store<false, false><<<grid, 256, 0, st>>>(S, a, F);
    return 1;
}

}  // namespace

size_t store_bytes(const StoreFields &F, int n)
{
    size_t each = 0;
    for (const double *f : {F.x, F.y, F.z, F.v[0], F.v[1], F.v[2], F.v[3], F.v[4], F.v[5], F.theta, F.phi})
        each += f ? 8 : 0;
    for (const int *f : {F.n_bnds, F.position, F.fix_site, F.fflag, F.sflag, F.nflag}) each += f ? 4 : 0;
    for (const int *f : {F.seg_id1, F.seg_id2, F.site}) each += f ? 16 : 0;
    return (each + (F.dltd ? 24 : 0)) * (size_t)n;
}

// In one pass while the fields' lines stay in L2 until they are whole, else a pass for each
// field, us: 3 / 6 / 9 fields of 1 million spheres 26 / 41 / 65 and 34 / 60 / 93, 1.5 million 33 / 64 /
// 183 and 43 / 89 / 135, 3 million 66 / 364 / 809 and 98 / 215 / 318; 2 million segments in random
// order, every field, 1465 and 420.
int launch_store(const DevState &S, int a, const StoreFields &F, bool fx, bool vel32, cudaStream_t st)
{
    if (fx || store_bytes(F, S.n) <= kScatterPass) return store_pass(S, a, F, fx, vel32, st);
    int k = 0;
    auto field = [&](auto *dst, const auto *src, auto planes) {
        if (!dst) return;
        k_scatter_field<decltype(planes)::value><<<(S.n + 255) / 256, 256, 0, st>>>(dst, src, S.orig, S.n);
        ++k;
    };
    const std::integral_constant<int, 1> one;
    const std::integral_constant<int, 4> four;
    const std::integral_constant<int, 6> six;
    field(F.x, S.x[a], one);
    field(F.y, S.y[a], one);
    field(F.z, S.z[a], one);
    if (vel32) {
        field(F.v[0], S.vxf, one);
        field(F.v[1], S.vyf, one);
        field(F.v[2], S.vzf, one);
    } else {
        field(F.v[0], S.vx, one);
        field(F.v[1], S.vy, one);
        field(F.v[2], S.vz, one);
    }
    field(F.v[3], S.wx, one);
    field(F.v[4], S.wy, one);
    field(F.v[5], S.wz, one);
    if (!S.has_rods) return k;
    const size_t n = (size_t)S.n;
    const int *tab = S.tab[a];
    field(F.theta, S.theta[a], one);
    field(F.phi, S.phi[a], one);
    field(F.n_bnds, tab, one);
    field(F.seg_id1, tab + n, four);
    field(F.seg_id2, tab + 5 * n, four);
    field(F.site, tab + 9 * n, four);
    field(F.position, S.position, one);
    field(F.fix_site, S.fix_site, one);
    field(F.fflag, S.fflag, one);
    field(F.sflag, S.sflag, one);
    field(F.nflag, S.nflag, one);
    field(F.dltd, S.dltd, six);
    return k;
}

int launch_aos_load(const unsigned char *rec, const AosLayout &L, int n, bool rods, double *d, int *i, cudaStream_t st)
{
    const int grid = (n + 127) / 128;
    if (rods) k_aos_load<true><<<grid, 128, 0, st>>>(rec, L, n, d, i);
    else k_aos_load<false><<<grid, 128, 0, st>>>(rec, L, n, d, i);
    return 1;
}

int launch_aos_store(unsigned char *rec, const AosLayout &L, const DevState &S, int a, cudaStream_t st)
{
    k_aos_store<<<(S.n + 127) / 128, 128, 0, st>>>(rec, L, S, a);
    return 1;
}

}  // namespace bmxg
