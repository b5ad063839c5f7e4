// bmxg_ctx.cu -- host side of the C ABI (include/bmxg.h): context lifetime,
// state upload / readback, the graph-captured step loop, neighbour-list
// export, statistics and the launch-shape autotuner.
//
// Stands behind BMXParticleContainer::EvolveParticles
// (src/des/bmx_pc.H:126-129, src/des/bmx_pc_interaction.cpp:13-495).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <type_traits>
#include <utility>
#include <vector>

#include "../../include/bmxg.h"
#include "bmxg_kernels.cuh"

using namespace bmxg;

namespace {

// What a step call reads back, in one copy.
struct StepBlock {
    DevCounters cnt;
    alignas(256) ListCtl ctl;  // (its atomics in lines of their own)
};

struct GraphKey {
    double dt;
    int precision;
    int parity;
    // -1: kResyncEvery steps (list steps: -2 with a build possible before each, -1 before the
    // first); 0 / 1: one step without / with the FP32F re-sync (list steps: 1 one that adds
    // itself to the call's steps, 2 one of those set before)
    int single;
    bool list;   // list steps (their kernels read the parity from the control block)
    bool operator<(const GraphKey &o) const
    {
        if (dt != o.dt) return dt < o.dt;
        if (precision != o.precision) return precision < o.precision;
        if (parity != o.parity) return parity < o.parity;
        if (single != o.single) return single < o.single;
        return list < o.list;
    }
};

struct Shape {
    int block = 256;
    int grid = 0;  // 0: derive from occupancy
};

// Buffers of the differentiation form, grown on demand.
struct AdjBuf {
    void *p = nullptr;
    size_t bytes = 0;
};
enum {
    kAdjCkpt,   // (nseg + 1) x 3n positions, slot order
    kAdjEnd,    // 3n: the trajectory's end
    kAdjLam0,   // adjoint of the positions, 3 planes
    kAdjLam1,
    kAdjAcc,    // 3n + n: parameter slopes and adhesion slope per slot
    kAdjOut,    // kReduceOut
    kAdjSeg,    // ckpt_every x 3n positions of one segment (no room for kAdjTrail)
    kAdjTrail,  // ckpt_every states of one segment with their columns sorted
    kAdjBufs
};

}  // namespace

struct bmxg_ctx {
    std::string err;
    bmxg_params prm{};
    int ncol = 0;
    std::vector<bmxg_geometry> geoms;
    int device = 0;
    int nsm = 0;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;

    // device allocations
    std::vector<void *> allocs;
    DevState S{};
    DevGeom *d_geoms = nullptr;
    int *d_cbase = nullptr;                 // ncol + 1 colony slot offsets (device)
    std::vector<int> h_cbase;
    std::vector<DevGeom> h_geoms;
    DevCounters *d_cnt = nullptr;
    DevCounters *h_cnt = nullptr;  // pinned (h_step's)
    StepBlock *d_step = nullptr, *h_step = nullptr;
    int *scan_scratch = nullptr;
    // staging in caller order
    double *ud = nullptr;  // n doubles
    int *uperm = nullptr;

    int64_t n = 0;
    bool have_state = false;
    bool stepped = false;
    int parity = 0;
    std::vector<int64_t> offsets;

    std::map<GraphKey, cudaGraphExec_t> graphs;
    std::map<GraphKey, int> graph_kernels;  // kernels per replay of each graph
    Shape sh_sphere[2], sh_rod, sh_misc;
    bool adj_pinned = false;  // sh_sphere[0]'s grid is the caller's (bmxg_set_shapes): the adjoint's too
    // list path shapes (bmxg_autotune): k_list_step's block and passes per
    // chunk (0: the launcher's rule), k_list_build's block
    int ls_block = kListStepBlock, ls_passes = 0, lb_block = kListBuildBlock;
    bool ls_persist = false;  // the list step as one wave of blocks taking chunks from a counter
    bmxg_stats stats{};
    int64_t launches = 0;                   // kernels enqueued (graph nodes counted per replay)
    bool profiling = false;
    std::vector<cudaEvent_t> kev;           // event pairs around the force kernel, profiling mode
    size_t kev_used = 0;

    // differentiation form
    double ext_gamma = 0.0, ext_mu = 0.0;
    double *d_adh = nullptr;                // per-slot adhesion in use (nullptr: zero)
    double *adh_buf = nullptr;              // its buffer, allocated with the state
    AdjBuf adj[kAdjBufs];                   // buffers of the trajectory and its adjoint (adj_buf)
    int traj_T = -1, traj_k = 0;
    double traj_dt = 0.0;

    bool rod_walk = false;    // no room for the rod pair lists: FP64 rod steps walk the stencil
    int64_t scratch_limit = -1;   // bmxg_set_scratch_limit
    bool vel32 = false;       // the last step's velocities are in the FP32F buffers
    bool vel64_zero = false;  // the FP64 velocity planes (vx .. wz) hold zeros: a load zeroed them
                              // and no kernel that writes them ran since
    int64_t step_count = 0;   // steps since set_state (FP32F re-sync schedule)

    // neighbour list with a skin (k_list.cu)
    int list_mode = 1;            // 1: sphere steps use the list where it is exact (FP64: and pays); 0: never
    bool list_on = false;         // the steps being enqueued use the list
    bool list_valid = false;      // the list and its frozen bins describe the state
    bool bins_exact = true;       // bins of buffer `parity` are the reference's (list steps freeze them)
    double rmax = 0.0;            // largest radius of the state
    int64_t ncells_total = 0;     // 3D cells over all colonies
    int *cell_scratch = nullptr;  // scan scratch of the list build (column counts, group entries)
    float skin_cur = 0.0f;        // skin of the list control block
    int list_prec = BMXG_FP32F;   // the form whose steps the list follows
    bool list_room = true;        // (false: no room for the list, FP64 steps go without)
    bool list64_bail = false;     // the loaded state left what FP64 list steps cover
    int64_t plain64 = 0;          // FP64 steps of this state's size that went without a list
    bool list64_live = false;     // FP64 steps follow a list; it has lasted list64_lived steps
    int64_t list64_lived = 0;
    int list64_short = 0;         // lists in a row that did not last kList64MinSteps steps
    int64_t list64_since = 0;     // FP64 steps in a row without one
    // list steps and the builds that fell due among them, over the last calls
    // (16 steps a build to begin with)
    double period_steps = 4.0, period_builds = 0.25;
    bool list_begun = false;      // the next build is the list's first (not one that fell due)
    int *h_run = nullptr;         // pinned: steps and buffer of a list call
    ListCtl *h_lctl = nullptr;    // pinned copy of the control block (h_step's)
    unsigned long long body_runs_seen = 0;  // list builds already counted as launches
    bool capturing = false;       // enqueue_step runs inside a graph capture
    bool list_one = false;        // ... of a list step that adds itself to the call's steps
    bool pair_capture = false;    // list steps record their gated pairs (S.pcap)
    bool pcap_valid = false;      // S.pcap holds the last step's gated pairs
    bool fx_ahead = false;        // list steps moved the fixed-point positions past the FP64 ones
    std::vector<FxGeom> h_fxg;    // per colony fixed-point geometry of the list path
    FxGeom *d_fxg = nullptr;
    cudaStream_t body_stream = nullptr;     // captures the bodies of conditional nodes

    // loads and stores of host arrays: the copies run on io_stream, overlapped
    // with the sort, gather and scatter kernels on `stream`; the device
    // staging is kept (and grown) across calls
    cudaStream_t io_stream = nullptr;
    cudaEvent_t io_ev[8] = {};
    char *io_buf = nullptr;
    size_t io_cap = 0;
    char *tile_buf = nullptr;               // workspace of the tile step, grown
    size_t tile_cap = 0;
    char *aos_buf = nullptr;                // planes (and staged records) of the AoS entry point, grown
    size_t aos_cap = 0;
    bool pageable = false;                  // the device reads pageable host memory in place
    unsigned long long *d_chk = nullptr;    // state-check flags (4) and the comparison of a load (1), device
    unsigned long long *h_chk = nullptr;    // and pinned host
};

namespace {

int sync_fp64(bmxg_ctx *ctx);
void list64_end(bmxg_ctx *ctx, bool poor = false);

// What a load checks of a state (launch_check_state), when the caller has done so.
struct StateCheck {
    bool rods;
    double rmax;
};
int load_state(bmxg_ctx *ctx, const bmxg_particles *p, const int64_t *colony_offsets, int where,
               const StateCheck *known);
int check_state(bmxg_ctx *ctx, const int *ct, const double *r, int64_t n, StateCheck *out);
int read_check(bmxg_ctx *ctx, StateCheck *out);

int fail(bmxg_ctx *c, int code, const std::string &msg)
{
    if (c) c->err = msg;
    return code;
}

#define CK(call)                                                                              \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess)                                                                \
            return fail(ctx, e_ == cudaErrorMemoryAllocation ? BMXG_ERR_OOM : BMXG_ERR_CUDA,  \
                        std::string(#call) + ": " + cudaGetErrorString(e_));                  \
    } while (0)

// Enqueue a launcher (it returns how many kernels it launched), count them,
// and turn a launch error into a status naming the launcher.
#define LAUNCH(call)                                                                             \
    do {                                                                                         \
        ctx->launches += (call);                                                                 \
        cudaError_t e_ = cudaPeekAtLastError();                                                  \
        if (e_ != cudaSuccess)                                                                   \
            return fail(ctx, BMXG_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

template <class T>
int dalloc(bmxg_ctx *ctx, T **p, size_t count)
{
    void *q = nullptr;
    if (count == 0) count = 1;
    CK(cudaMalloc(&q, count * sizeof(T)));
    ctx->allocs.push_back(q);
    *p = (T *)q;
    return BMXG_OK;
}

void drop_graphs(bmxg_ctx *ctx)
{
    for (auto &g : ctx->graphs) cudaGraphExecDestroy(g.second);
    ctx->graphs.clear();
    ctx->graph_kernels.clear();
}

// The trajectory is gone; its buffers stay for the next one while they are small
// (kAdjointKeep) and the state's arrays stay, else they are given back.
constexpr size_t kAdjointKeep = 256u << 20;

size_t adjoint_bytes(const bmxg_ctx *ctx)
{
    size_t held = 0;
    for (const AdjBuf &b : ctx->adj) held += b.bytes;
    return held;
}

void free_adj_buf(AdjBuf &b)
{
    if (b.p) cudaFree(b.p);  // (waits for the work that uses it)
    b = AdjBuf{};
}

void free_adjoint(bmxg_ctx *ctx, bool all = false)
{
    ctx->traj_T = -1;
    if (!all && adjoint_bytes(ctx) <= kAdjointKeep) return;
    for (AdjBuf &b : ctx->adj) free_adj_buf(b);
}

// The buffers of a reverse sweep alone, after it: the states of a segment can be
// half of the device's memory.  (The trajectory stays: another sweep may follow.)
struct SweepBufs {
    bmxg_ctx *ctx;
    ~SweepBufs()
    {
        for (int k : {kAdjTrail, kAdjSeg})
            if (adjoint_bytes(ctx) > kAdjointKeep) free_adj_buf(ctx->adj[k]);
    }
};

// What the last sort found (the captured steps hold the choice of its kernel).
void set_long_cols(bmxg_ctx *ctx, bool some)
{
    if ((ctx->S.long_cols != 0) == some) return;
    ctx->S.long_cols = some ? 1 : 0;
    drop_graphs(ctx);
}

// Device staging of at least `bytes` for host loads and stores.
int ensure_io(bmxg_ctx *ctx, size_t bytes)
{
    if (bytes <= ctx->io_cap) return BMXG_OK;
    CK(cudaStreamSynchronize(ctx->stream));
    CK(cudaStreamSynchronize(ctx->io_stream));
    if (ctx->io_buf) cudaFree(ctx->io_buf);
    ctx->io_buf = nullptr;
    ctx->io_cap = 0;
    CK(cudaMalloc(&ctx->io_buf, bytes));
    ctx->io_cap = bytes;
    return BMXG_OK;
}

// Waits for the load / store copies still reading or writing caller memory
// when a call returns early.
struct JoinIo {
    cudaStream_t s;
    ~JoinIo()
    {
        if (s) cudaStreamSynchronize(s);
    }
};

// Whether `need` bytes of buffers that a call can do without may be taken: up to the caller's
// limit, else one `share`-th of the device's free memory.
bool room_for(const bmxg_ctx *ctx, size_t need, size_t share)
{
    if (ctx->scratch_limit >= 0) return need <= (size_t)ctx->scratch_limit;
    size_t room = 0, all = 0;
    if (cudaMemGetInfo(&room, &all) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return need <= room / share;
}

void free_state(bmxg_ctx *ctx)
{
    drop_graphs(ctx);
    free_adjoint(ctx, true);
    ctx->d_adh = ctx->adh_buf = nullptr;  // lives in allocs
    for (void *p : ctx->allocs) cudaFree(p);
    ctx->allocs.clear();
    ctx->S = DevState{};
    ctx->rod_walk = false;
    ctx->list_room = true;
    ctx->plain64 = 0;
    list64_end(ctx);
    ctx->list64_short = 0;
    ctx->d_geoms = nullptr;
    ctx->d_cbase = nullptr;
    ctx->scan_scratch = nullptr;
    ctx->cell_scratch = nullptr;
    ctx->ud = nullptr;
    ctx->uperm = nullptr;
    ctx->have_state = false;
    ctx->list_valid = false;
    ctx->fx_ahead = false;
    ctx->d_fxg = nullptr;
    ctx->bins_exact = true;
}

int grid_for(bmxg_ctx *ctx, const Shape &s, int64_t n)
{
    int g = s.grid;
    if (g <= 0) g = ctx->nsm * std::max(1, 2048 / s.block);
    int64_t need = (n + s.block - 1) / s.block;
    if (need < 1) need = 1;
    return (int)std::min<int64_t>(g, need);
}

// Launch shape of the per-slot stencil kernels (spheres, the differentiation
// form): an autotuned shape when there is one; else one slot per thread in
// 64-thread blocks.  The stencil walks differ in length from slot to slot, and
// small blocks on a grid of every slot let the block scheduler balance them
// (2.73 M spheres: FP64 6.66 -> 5.94 ms, FP32F 657 -> 600 us per step, against
// 256-thread blocks striding over one wave).
void stencil_shape(bmxg_ctx *ctx, const Shape &s, int64_t n, int *grid, int *block)
{
    if (s.grid > 0) {
        *block = s.block;
        *grid = grid_for(ctx, s, n);
    } else {
        *block = kSphereBlock;
        *grid = (int)std::max<int64_t>(1, (n + kSphereBlock - 1) / kSphereBlock);
    }
}

DevParams dev_params(const bmxg_params &p) { return make_dev_params(p); }

int check_params(const bmxg_params *p)
{
    if (!p) return BMXG_ERR_ARG;
    const double v[10] = {p->bndry_width, p->stiffness,     p->z_wall,      p->z_bndry_width, p->z_stiffness,
                          p->z_gravity,   p->bond_strength, p->bond_cutoff, p->viscosity,     p->neighborhood};
    for (double x : v)
        if (!std::isfinite(x)) return BMXG_ERR_ARG;
    return BMXG_OK;
}

int check_geom(const bmxg_geometry &g, std::string &why)
{
    for (int d = 0; d < 3; ++d) {
        if (!(g.prob_hi[d] > g.prob_lo[d]) || !std::isfinite(g.prob_lo[d]) || !std::isfinite(g.prob_hi[d])) {
            why = "prob_hi must exceed prob_lo";
            return BMXG_ERR_ARG;
        }
        if (g.n_cell[d] < 1 || g.n_cell[d] > (1 << 20)) {
            why = "n_cell out of range";
            return BMXG_ERR_ARG;
        }
        if (g.is_periodic[d] && g.n_cell[d] < 3) {
            why = "a periodic direction needs n_cell >= 3";
            return BMXG_ERR_UNSUPPORTED;
        }
    }
    if (g.is_periodic[2]) {
        why = "z must be non-periodic (the growth surface sits in z)";
        return BMXG_ERR_UNSUPPORTED;
    }
    return BMXG_OK;
}

// Device geometry of each colony, with the column and slot numbering.
void build_geoms(bmxg_ctx *ctx)
{
    ctx->h_geoms.resize(ctx->ncol);
    ctx->h_fxg.resize(ctx->ncol);
    int col_base = 0;
    int64_t cell_base = 0;
    for (int c = 0; c < ctx->ncol; ++c) {
        const bmxg_geometry &g = ctx->geoms[c];
        DevGeom &G = ctx->h_geoms[c];
        std::memset(&G, 0, sizeof(G));
        double diag2 = 0.0;
        for (int d = 0; d < 3; ++d) {
            G.plo[d] = g.prob_lo[d];
            G.phi[d] = g.prob_hi[d];
            G.len[d] = g.prob_hi[d] - g.prob_lo[d];
            G.n[d] = g.n_cell[d];
            G.dx[d] = G.len[d] / (double)G.n[d];
            G.dxi[d] = 1.0 / G.dx[d];
            G.dxf[d] = (float)G.dx[d];
            G.plof[d] = (float)G.plo[d];
            G.dxif[d] = (float)G.dxi[d];
            G.phif[d] = (float)G.phi[d];
            // corners as the device computes them: a product, then a sum, each
            // rounded (volatile keeps the host compiler from fusing them)
            G.ncorner[d] = std::min(G.n[d], kCornerTable);
            for (int bi = 1; bi <= G.ncorner[d]; ++bi) {
                volatile double t = (double)(bi - 1) * G.dx[d];
                G.corner[d][bi - 1] = G.plo[d] + t;
            }
            G.per[d] = g.is_periodic[d] ? 1 : 0;
            diag2 += 4.0 * G.dx[d] * G.dx[d];
        }
        G.col_base = col_base;
        col_base += G.n[0] * G.n[1];
        G.cell_base = (int)std::min<int64_t>(cell_base, INT32_MAX);
        cell_base += (int64_t)G.n[0] * G.n[1] * G.n[2];
        G.slot_base = (int)ctx->offsets[c];
        G.slot_end = (int)ctx->offsets[c + 1];
        // two bins apart at most per axis: |r|^2 < 4 (dx^2 + dy^2 + dz^2)
        G.nbh_trivial = (ctx->prm.neighborhood >= diag2 * (1.0 + 1e-9)) ? 1 : 0;
        G.invny = 1.0f / (float)G.n[1];
        // 64-bit fixed point of the list path: a periodic axis spans the
        // domain, a closed one four lengths from one length below plo
        FxGeom &F = ctx->h_fxg[c];
        std::memset(&F, 0, sizeof(F));
        for (int d = 0; d < 3; ++d) {
            const double span = G.per[d] ? G.len[d] : 4.0 * G.len[d];
            F.o[d] = G.per[d] ? G.plo[d] : G.plo[d] - G.len[d];
            F.u[d] = std::ldexp(span, -64);
            F.uh[d] = (float)std::ldexp(span, -32);
            const long double cx = std::ldexp(1.0L / (long double)span, 64);
            F.c[d] = (float)cx;
            F.cl[d] = (float)(cx - (long double)F.c[d]);
            F.n[d] = G.n[d];
            F.per[d] = G.per[d];
            F.plo[d] = G.plo[d];
            F.phi[d] = G.phi[d];
            F.ozero[d] = F.o[d] == 0.0 ? 1 : 0;
            int k = 0;
            const double fr = std::frexp(span, &k);  // span = fr 2^k, fr in [0.5, 1)
            F.ms[d] = (unsigned long long)std::ldexp(fr, 53);
            F.es[d] = k - 53;
            // 2^64 / span = 2^(64 - es) / ms: q = 2^127 / ms, normalised to 64 bits
            const unsigned __int128 q = ((unsigned __int128)1 << 127) / F.ms[d];
            int bl = 0;
            for (unsigned __int128 v = q; v; v >>= 1) ++bl;
            const int sh = bl - 64;
            F.mc[d] = (unsigned long long)(q >> sh);
            F.ec[d] = (64 - F.es[d]) - 127 + sh;
        }
        {
            const long double t = ((long double)ctx->prm.z_wall - (long double)F.o[2]) / (long double)F.u[2];
            const long double hi = std::floor(t / 4294967296.0L);
            F.zw = (hi <= 0.0L) ? 0u : (hi >= 4294967295.0L ? 4294967295u : (unsigned)hi);
        }
        // height of each z-bin's lower face above the growth surface, with the
        // same FP64 face the re-binning uses, split into a float pair
        G.nwz = std::min(G.n[2] + 2, kWallTable);
        for (int bz = 0; bz < G.nwz; ++bz) {
            const double face = G.plo[2] + (double)(bz - 1) * G.dx[2];
            const double h = face - ctx->prm.z_wall;
            const float hi = (float)h;
            G.wz[bz] = make_float2(hi, (float)(h - (double)hi));
        }
    }
    ctx->ncells_total = cell_base;
}

}  // namespace

extern "C" {

int bmxg_version(void) { return BMXG_ABI_VERSION; }

const char *bmxg_last_error(const bmxg_ctx *ctx) { return ctx ? ctx->err.c_str() : "null context"; }

int bmxg_create(const bmxg_params *params, int32_t ncolonies, const bmxg_geometry *geoms, bmxg_ctx **out)
{
    if (!out) return BMXG_ERR_ARG;
    *out = nullptr;
    if (check_params(params) || ncolonies < 1 || !geoms) return BMXG_ERR_ARG;
    bmxg_ctx *ctx = new bmxg_ctx();
    ctx->prm = *params;
    ctx->ncol = ncolonies;
    ctx->geoms.assign(geoms, geoms + ncolonies);
    for (int c = 0; c < ncolonies; ++c) {
        std::string why;
        int rc = check_geom(ctx->geoms[c], why);
        if (rc) {
            delete ctx;
            return rc;
        }
    }
    int64_t cols = 0;
    for (auto &g : ctx->geoms) cols += (int64_t)g.n_cell[0] * g.n_cell[1];
    if (cols >= (1LL << 31) - 2) {
        delete ctx;
        return BMXG_ERR_UNSUPPORTED;
    }
    cudaError_t e = cudaGetDevice(&ctx->device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&ctx->nsm, cudaDevAttrMultiProcessorCount, ctx->device);
    int paged = 0;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&paged, cudaDevAttrPageableMemoryAccess, ctx->device);
    ctx->pageable = paged != 0;
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev0);
    if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev1);
    if (e == cudaSuccess) e = cudaMallocHost(&ctx->h_step, sizeof(StepBlock));
    if (e == cudaSuccess) {
        ctx->h_cnt = &ctx->h_step->cnt;
        ctx->h_lctl = &ctx->h_step->ctl;
    }
    if (e == cudaSuccess) e = cudaMallocHost(&ctx->h_run, 2 * sizeof(int));
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->body_stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->io_stream, cudaStreamNonBlocking);
    for (cudaEvent_t &ev : ctx->io_ev)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaMalloc(&ctx->d_chk, 5 * sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMallocHost(&ctx->h_chk, 5 * sizeof(unsigned long long));
    if (e != cudaSuccess) {
        ctx->err = cudaGetErrorString(e);
        bmxg_destroy(ctx);
        return BMXG_ERR_CUDA;
    }
    ctx->stream = ctx->own_stream;
    ctx->sh_sphere[0].block = 256;
    ctx->sh_sphere[1].block = 256;
    ctx->sh_rod.block = 32;  // rod walks: one warp per block balances best (FP64 890 -> 844 us, 50 k segments)
    ctx->sh_misc.block = 256;
    *out = ctx;
    return BMXG_OK;
}

void bmxg_destroy(bmxg_ctx *ctx)
{
    if (!ctx) return;
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    free_state(ctx);
    if (ctx->h_step) cudaFreeHost(ctx->h_step);
    if (ctx->h_run) cudaFreeHost(ctx->h_run);
    if (ctx->body_stream) cudaStreamDestroy(ctx->body_stream);
    if (ctx->io_stream) {
        cudaStreamSynchronize(ctx->io_stream);
        cudaStreamDestroy(ctx->io_stream);
    }
    for (cudaEvent_t ev : ctx->io_ev)
        if (ev) cudaEventDestroy(ev);
    if (ctx->io_buf) cudaFree(ctx->io_buf);
    if (ctx->aos_buf) cudaFree(ctx->aos_buf);
    if (ctx->tile_buf) cudaFree(ctx->tile_buf);
    if (ctx->d_chk) cudaFree(ctx->d_chk);
    if (ctx->h_chk) cudaFreeHost(ctx->h_chk);
    if (ctx->ev0) cudaEventDestroy(ctx->ev0);
    if (ctx->ev1) cudaEventDestroy(ctx->ev1);
    for (cudaEvent_t e : ctx->kev) cudaEventDestroy(e);
    if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
    delete ctx;
}

int bmxg_set_params(bmxg_ctx *ctx, const bmxg_params *params)
{
    if (!ctx) return BMXG_ERR_ARG;
    if (check_params(params)) return fail(ctx, BMXG_ERR_ARG, "non-finite force parameter");
    if (int rc = sync_fp64(ctx)) return rc;  // the list's fixed point restarts from the FP64 positions
    ctx->prm = *params;
    drop_graphs(ctx);
    list64_end(ctx);
    ctx->list_valid = false;
    if (ctx->have_state) {
        build_geoms(ctx);
        CK(cudaMemcpyAsync(ctx->d_geoms, ctx->h_geoms.data(), sizeof(DevGeom) * ctx->ncol,
                           cudaMemcpyHostToDevice, ctx->stream));
        CK(cudaMemcpyAsync(ctx->d_fxg, ctx->h_fxg.data(), sizeof(FxGeom) * ctx->ncol, cudaMemcpyHostToDevice,
                           ctx->stream));
        if (ctx->S.has_rods && ctx->n) {  // the segment mobilities depend on the viscosity
            const int blk = ctx->sh_misc.block, grd = grid_for(ctx, ctx->sh_misc, ctx->n);
            launch_rod_mobility(ctx->S, dev_params(ctx->prm), grd, blk, ctx->stream);
            CK(cudaGetLastError());
        }
        CK(cudaStreamSynchronize(ctx->stream));
    }
    return BMXG_OK;
}

int bmxg_set_stream(bmxg_ctx *ctx, void *stream)
{
    if (!ctx) return BMXG_ERR_ARG;
    cudaStream_t s = stream ? (cudaStream_t)stream : ctx->own_stream;
    if (s != ctx->stream) {
        CK(cudaStreamSynchronize(ctx->stream));
        ctx->stream = s;
        drop_graphs(ctx);
    }
    return BMXG_OK;
}

int bmxg_set_state(bmxg_ctx *ctx, const bmxg_particles *p, const int64_t *colony_offsets, int where)
{
    return load_state(ctx, p, colony_offsets, where, nullptr);
}

}  // extern "C"

namespace {

int load_state(bmxg_ctx *ctx, const bmxg_particles *p, const int64_t *colony_offsets, int where,
               const StateCheck *known)
{
    if (!ctx) return BMXG_ERR_ARG;
    (void)cudaGetLastError();  // drop a non-sticky error another library left on this thread
    if (!p || p->n < 0 || !p->x || !p->y || !p->z || !p->radius || !p->cell_type)
        return fail(ctx, BMXG_ERR_ARG, "x, y, z, radius and cell_type are required");
    if (p->n > (1LL << 30)) return fail(ctx, BMXG_ERR_UNSUPPORTED, "more than 2^30 particles");
    if (where != BMXG_HOST && where != BMXG_DEVICE) return fail(ctx, BMXG_ERR_ARG, "bad `where`");
    const int64_t n = p->n;
    std::vector<int64_t> off(ctx->ncol + 1, 0);
    if (ctx->ncol == 1) {
        off[1] = n;
    } else {
        if (!colony_offsets) return fail(ctx, BMXG_ERR_ARG, "colony_offsets required for several colonies");
        for (int c = 0; c <= ctx->ncol; ++c) off[c] = colony_offsets[c];
        if (off[0] != 0 || off[ctx->ncol] != n) return fail(ctx, BMXG_ERR_ARG, "colony_offsets must span 0..n");
        for (int c = 0; c < ctx->ncol; ++c)
            if (off[c + 1] < off[c]) return fail(ctx, BMXG_ERR_ARG, "colony_offsets must not decrease");
    }
    const cudaMemcpyKind kind = (where == BMXG_HOST) ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
    // A load of exactly the state the device holds (a caller that stores the
    // state after a step and loads it back unchanged before the next, as a
    // load-step-store loop does) keeps the slot order, the neighbour list and
    // its frozen frames: the loaded positions, radii and cell types are
    // compared bit for bit with the device state first (a state that passed
    // the checks below before).  Only for spheres and when the caller gives no
    // other field (which would overwrite device fields); what any load resets
    // is reset here as well.
    const bool only_required = !p->velx && !p->vely && !p->velz && !p->wx && !p->wy && !p->wz &&
                               !p->c_length && !p->theta && !p->phi && !p->area && !p->bond_scale &&
                               !p->id && !p->cpu && !p->n_bnds && !p->seg_id1 && !p->seg_id2 && !p->site &&
                               !p->position && !p->fuse_tip && !p->fix_site && !p->fuse_flag &&
                               !p->split_flag && !p->new_flag && !p->dltd;
    const bool same_cand = n && !known && only_required && ctx->have_state && ctx->n == n && ctx->offsets == off &&
                           !ctx->S.has_rods;
    // the comparison reads the device's FP64 positions
    if (same_cand) {
        if (int rc = sync_fp64(ctx)) return rc;
    }
    // Positions, radii and cell types: read in place from device arrays; host
    // arrays go to the staging, radii and cell types first on the compute
    // stream (the state checks need them), positions on the copy stream, so
    // that their copy overlaps the checks and the host's decisions below.
    const double *src_x = p->x, *src_y = p->y, *src_z = p->z, *src_r = p->radius;
    const int *src_ct = p->cell_type;
    JoinIo join{nullptr};
    cudaStream_t st0 = ctx->stream, st1 = ctx->io_stream;
    {   // staging of the positions, radii and cell types (36 B) and of the other fields (up to 200 B, 24 of them)
        auto staged = [&](const void *f, size_t align) {
            return f && (where == BMXG_HOST || reinterpret_cast<uintptr_t>(f) % align != 0);
        };
        size_t bytes = (where == BMXG_HOST) ? (size_t)n * 36 + 512 : 0;
        for (const double *f : {p->velx, p->vely, p->velz, p->wx, p->wy, p->wz, p->c_length, p->theta, p->phi,
                                p->area, p->bond_scale})
            if (staged(f, 8)) bytes += (size_t)n * 8 + 16;
        for (const int32_t *f : {p->id, p->cpu, p->fuse_tip, p->position, p->fix_site, p->fuse_flag, p->split_flag,
                                 p->new_flag, p->n_bnds})
            if (staged(f, 4)) bytes += (size_t)n * 4 + 16;
        for (const int32_t *f : {p->seg_id1, p->seg_id2, p->site})
            if (staged(f, 4)) bytes += (size_t)n * 16 + 16;
        if (staged(p->dltd, 4)) bytes += (size_t)n * 24 + 16;
        if (int rc0 = ensure_io(ctx, bytes)) return rc0;
    }
    if (n && where == BMXG_HOST) {
        double *bx = (double *)ctx->io_buf, *by = bx + n, *bz = by + n, *br = bz + n;
        int *bct = (int *)(br + n);
        CK(cudaEventRecord(ctx->io_ev[0], st0));  // earlier kernels on st0 are done with the staging
        CK(cudaStreamWaitEvent(st1, ctx->io_ev[0], 0));
        join.s = st1;
        CK(cudaMemcpyAsync(br, p->radius, sizeof(double) * n, kind, st0));
        CK(cudaMemcpyAsync(bct, p->cell_type, sizeof(int) * n, kind, st0));
        CK(cudaMemcpyAsync(bx, p->x, sizeof(double) * n, kind, st1));
        CK(cudaEventRecord(ctx->io_ev[6], st1));
        CK(cudaMemcpyAsync(by, p->y, sizeof(double) * n, kind, st1));
        CK(cudaEventRecord(ctx->io_ev[7], st1));
        CK(cudaMemcpyAsync(bz, p->z, sizeof(double) * n, kind, st1));
        CK(cudaEventRecord(ctx->io_ev[1], st1));
        src_x = bx;
        src_y = by;
        src_z = bz;
        src_r = br;
        src_ct = bct;
    }
    if (same_cand) {
        cudaStream_t st = ctx->stream;
        const int grd = grid_for(ctx, ctx->sh_misc, n), blk = ctx->sh_misc.block;
        const DevState &S = ctx->S;
        unsigned long long *diff = ctx->d_chk + 4;
        CK(cudaMemsetAsync(ctx->d_chk, 0, 5 * sizeof(unsigned long long), st));
        // (the checks of a full load go along: one read-back decides both)
        if (join.s) {  // each field as its copy lands: only the last comparison follows the copies
            LAUNCH(launch_same_state(S, ctx->parity, nullptr, nullptr, nullptr, src_r, src_ct, diff, ctx->d_chk, grd,
                                     blk, st));
            CK(cudaStreamWaitEvent(st, ctx->io_ev[6], 0));
            LAUNCH(launch_same_state(S, ctx->parity, src_x, nullptr, nullptr, nullptr, nullptr, diff, nullptr, grd,
                                     blk, st));
            CK(cudaStreamWaitEvent(st, ctx->io_ev[7], 0));
            LAUNCH(launch_same_state(S, ctx->parity, nullptr, src_y, nullptr, nullptr, nullptr, diff, nullptr, grd,
                                     blk, st));
            CK(cudaStreamWaitEvent(st, ctx->io_ev[1], 0));
            LAUNCH(launch_same_state(S, ctx->parity, nullptr, nullptr, src_z, nullptr, nullptr, diff, nullptr, grd,
                                     blk, st));
        } else {
            LAUNCH(launch_same_state(S, ctx->parity, src_x, src_y, src_z, src_r, src_ct, diff, ctx->d_chk, grd, blk,
                                     st));
        }
        CK(cudaMemcpyAsync(ctx->h_chk, ctx->d_chk, 5 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (ctx->h_chk[4] == 0) {
            // velocities to zero (unless no kernel wrote them since the last
            // load zeroed them) and the counters; stream-ordered before
            // whatever the caller enqueues next
            if (!ctx->vel64_zero)
                for (double *v : {S.vx, S.vy, S.vz, S.wx, S.wy, S.wz})
                    CK(cudaMemsetAsync(v, 0, sizeof(double) * n, st));
            CK(cudaMemsetAsync(ctx->d_cnt, 0, sizeof(DevCounters), st));
            CK(cudaGetLastError());
            ctx->vel64_zero = true;
            ctx->stepped = false;
            ctx->vel32 = false;
            ctx->pcap_valid = false;
            ctx->d_adh = nullptr;
            free_adjoint(ctx);
            std::memset(&ctx->stats, 0, sizeof(ctx->stats));
            ctx->stats.n_particles = n;
            return BMXG_OK;
        }
    }
    ctx->vel64_zero = false;  // (until the full load below has set every plane)
    // cell types decide which path runs (rods need their fields) and the
    // largest radius whether the FP32F list is exact: checked on the device,
    // one small read-back
    StateCheck chk{false, 0.0};
    if (known) {
        chk = *known;
    } else if (same_cand) {
        if (int rc0 = read_check(ctx, &chk)) return rc0;
    } else if (n) {
        if (int rc0 = check_state(ctx, src_ct, src_r, n, &chk)) return rc0;
    }
    const bool rods = chk.rods;
    const double rmax = chk.rmax;
    if (rods && (!p->c_length || !p->theta || !p->phi || !p->area || !p->id || !p->cpu || !p->n_bnds ||
                 !p->seg_id1 || !p->seg_id2 || !p->site))
        return fail(ctx, BMXG_ERR_ARG, "rod segments need c_length, theta, phi, area, id, cpu and the bond table");

    // Same particle count, colony layout and cell-type mix as the loaded
    // state: keep the device buffers (and the captured step graphs, which
    // only hold their addresses) and overwrite the contents.
    const bool reuse = ctx->have_state && ctx->n == n && ctx->offsets == off && ctx->S.has_rods == (rods ? 1 : 0);
    if (!reuse) {
        CK(cudaStreamSynchronize(ctx->stream));
        free_state(ctx);
    }
    ctx->n = n;
    ctx->offsets = off;
    build_geoms(ctx);
    int64_t ncols = 0;
    for (auto &g : ctx->geoms) ncols += (int64_t)g.n_cell[0] * g.n_cell[1];

    DevState &S = ctx->S;
    S.n = (int)n;
    S.ncol = ctx->ncol;
    S.ncols_total = (int)ncols;
    S.nsm = ctx->nsm;
    S.has_rods = rods ? 1 : 0;
    int rc = BMXG_OK;
#define AL(ptr, cnt)                       \
    do {                                   \
        rc = dalloc(ctx, &(ptr), (cnt));   \
        if (rc) return rc;                 \
    } while (0)
    if (!reuse) {
    AL(ctx->d_geoms, ctx->ncol);
    AL(ctx->d_fxg, ctx->ncol);
    AL(ctx->d_cbase, ctx->ncol + 1);
    AL(ctx->d_step, 1);
    ctx->d_cnt = &ctx->d_step->cnt;
    for (int k = 0; k < 2; ++k) {
        AL(S.x[k], n); AL(S.y[k], n); AL(S.z[k], n);
        AL(S.rel[k], n); AL(S.col[k], n); AL(S.iz[k], n);
        AL(S.perm[k], n); AL(S.colstart[k], ncols + 1);
        AL(S.srel[k], n); AL(S.siz[k], n); AL(S.rank[k], n);
    }
    AL(S.colcnt, ncols); AL(S.tmp, n); AL(S.lkey, n);
    AL(S.rad, n); AL(S.orig, n); AL(S.ctype, n);
    AL(S.vx, n); AL(S.vy, n); AL(S.vz, n); AL(S.wx, n); AL(S.wy, n); AL(S.wz, n);
    AL(S.vxf, n); AL(S.vyf, n); AL(S.vzf, n);
    AL(ctx->scan_scratch, scan_scratch_ints((int)ncols));
    AL(ctx->ud, n); AL(ctx->uperm, n);
    if (rods) {
        AL(S.clen, n); AL(S.area, n); AL(S.bscale, n);
        for (int k = 0; k < 2; ++k) { AL(S.theta[k], n); AL(S.phi[k], n); AL(S.trig[k], n); AL(S.tab[k], 13 * n); }
        AL(S.id, n); AL(S.cpu, n); AL(S.fuse_tip, n); AL(S.position, n); AL(S.fix_site, n);
        AL(S.fflag, n); AL(S.sflag, n); AL(S.nflag, n); AL(S.dltd, 6 * n); AL(S.fc, 6 * n); AL(S.mob, n);
        AL(S.axf[0], n); AL(S.axf[1], n);
    }
    }  // !reuse
#undef AL
    S.geoms = ctx->d_geoms;
    S.fxg = ctx->d_fxg;
    S.cbase = ctx->d_cbase;
    S.cnt = ctx->d_cnt;
    cudaStream_t st = ctx->stream;
    if (!reuse) {  // same colonies as the loaded state: the device copies are current
        CK(cudaMemcpyAsync(ctx->d_geoms, ctx->h_geoms.data(), sizeof(DevGeom) * ctx->ncol, cudaMemcpyHostToDevice,
                           st));
        CK(cudaMemcpyAsync(ctx->d_fxg, ctx->h_fxg.data(), sizeof(FxGeom) * ctx->ncol, cudaMemcpyHostToDevice, st));
        ctx->h_cbase.assign(off.begin(), off.end());
        CK(cudaMemcpyAsync(ctx->d_cbase, ctx->h_cbase.data(), sizeof(int) * (ctx->ncol + 1), cudaMemcpyHostToDevice,
                           st));
    }
    CK(cudaMemsetAsync(ctx->d_cnt, 0, sizeof(DevCounters), st));
    CK(cudaMemsetAsync(S.colcnt, 0, sizeof(int) * std::max<int64_t>(ncols, 1), st));
    if (n == 0) {
        CK(cudaMemsetAsync(S.colstart[0], 0, sizeof(int) * (ncols + 1), st));
        CK(cudaMemsetAsync(S.colstart[1], 0, sizeof(int) * (ncols + 1), st));
        CK(cudaStreamSynchronize(st));
        ctx->have_state = true;
        ctx->parity = 0;
        return BMXG_OK;
    }
    const int blk = ctx->sh_misc.block;
    const int grd = grid_for(ctx, ctx->sh_misc, n);
    if (join.s) CK(cudaStreamWaitEvent(st, ctx->io_ev[1], 0));  // staged positions
    // canonical order of the caller's particles
    LAUNCH(launch_user_bin(S, src_x, src_y, src_z, S.col[1], S.iz[1], grd, blk, st));
    LAUNCH(launch_user_sort(S, S.col[1], S.iz[1], S.colstart[0], ctx->scan_scratch, ctx->uperm, grd, blk, st));
    // positions, radii, cell types, bins and offsets into slot order in one
    // pass (slot s is sorted position s, so the sort's bins are the slots')
    // The other fields: read in place from device arrays (aligned ones), else
    // staged behind the positions; then gathered in one kernel.
    char *stage = ctx->io_buf + (((size_t)(where == BMXG_HOST ? n : 0) * 36 + 255) / 256) * 256;
    rc = BMXG_OK;
    auto field = [&](const void *src, size_t bytes, size_t align) -> const void * {
        if (!src || rc) return nullptr;
        if (where == BMXG_DEVICE && (reinterpret_cast<uintptr_t>(src) % align) == 0) return src;
        const cudaError_t e = cudaMemcpyAsync(stage, src, bytes, kind, st);
        if (e != cudaSuccess) {
            rc = fail(ctx, BMXG_ERR_CUDA, std::string("load of a field: ") + cudaGetErrorString(e));
            return nullptr;
        }
        const void *q = stage;
        stage += (bytes + 15) / 16 * 16;
        return q;
    };
    auto fd = [&](const double *src) { return static_cast<const double *>(field(src, sizeof(double) * n, 8)); };
    auto fi = [&](const int32_t *src, int planes) {
        return static_cast<const int *>(field(src, sizeof(int) * n * planes, 4));
    };
    const double *vel[6] = {fd(p->velx), fd(p->vely), fd(p->velz), fd(p->wx), fd(p->wy), fd(p->wz)};
    if (rc) return rc;
    // velocities that the gather of the positions has no room for in its pass: one by one
    // after it (3 million spheres with six: 652 us, 829 in one pass)
    const double *later[6] = {};
    size_t pass = (size_t)n * 36;
    for (int k = 0; k < 6; ++k) {
        if (!vel[k]) continue;
        pass += (size_t)n * sizeof(double);
        if (pass > kScatterPass) std::swap(vel[k], later[k]);
    }
    LAUNCH(launch_load_slots(S, src_x, src_y, src_z, src_r, src_ct, vel, S.col[1], S.iz[1], ctx->uperm, grd, blk,
                             st));
    double *const vdst[6] = {S.vx, S.vy, S.vz, S.wx, S.wy, S.wz};
    for (int k = 0; k < 6; ++k)
        if (later[k]) LAUNCH(launch_gather_d(vdst[k], later[k], ctx->uperm, (int)n, grd, blk, st));
    if (rods) {
        const RodFields F{fd(p->c_length), fd(p->area), fd(p->bond_scale), fd(p->theta), fd(p->phi),
                          fi(p->id, 1), fi(p->cpu, 1), fi(p->fuse_tip, 1), fi(p->position, 1), fi(p->fix_site, 1),
                          fi(p->fuse_flag, 1), fi(p->split_flag, 1), fi(p->new_flag, 1), fi(p->dltd, 6),
                          fi(p->n_bnds, 1), fi(p->seg_id1, 4), fi(p->seg_id2, 4), fi(p->site, 4)};
        if (rc) return rc;
        const int rblk = 128;
        LAUNCH(launch_load_rods(S, dev_params(ctx->prm), F, ctx->uperm, (int)((n + rblk - 1) / rblk), rblk, st));
    }
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(ctx->h_cnt, ctx->d_cnt, sizeof(DevCounters), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (ctx->h_cnt->bad_index) return fail(ctx, BMXG_ERR_STATE, "internal: inconsistent bin counts in the load sort");
    set_long_cols(ctx, ctx->h_cnt->long_column != 0);
    ctx->have_state = true;
    ctx->stepped = false;
    ctx->vel32 = false;
    ctx->vel64_zero = !p->velx && !p->vely && !p->velz && !p->wx && !p->wy && !p->wz;
    ctx->step_count = 0;
    ctx->list64_bail = false;
    list64_end(ctx);
    ctx->parity = 0;
    ctx->rmax = rmax;
    ctx->list_valid = false;
    ctx->pcap_valid = false;
    ctx->fx_ahead = false;
    ctx->bins_exact = true;
    ctx->d_adh = nullptr;  // per-particle adhesion must be given again for the new state
    free_adjoint(ctx);
    std::memset(&ctx->stats, 0, sizeof(ctx->stats));
    ctx->stats.n_particles = n;
    return BMXG_OK;
}

// The check's read-back (h_chk) as a StateCheck.
int read_check(bmxg_ctx *ctx, StateCheck *out)
{
    const unsigned long long *h = ctx->h_chk;
    if (h[0]) return fail(ctx, BMXG_ERR_ARG, "cell_type must be 0 or 1");
    out->rods = h[1] != 0;
    const uint64_t rb = h[2];
    std::memcpy(&out->rmax, &rb, sizeof(out->rmax));
    if (h[3]) out->rmax = std::nan("");
    return BMXG_OK;
}

// Cell types, presence of rods and the largest radius of device arrays in
// caller order (synchronises the stream).
int check_state(bmxg_ctx *ctx, const int *ct, const double *r, int64_t n, StateCheck *out)
{
    cudaStream_t st = ctx->stream;
    CK(cudaMemsetAsync(ctx->d_chk, 0, 4 * sizeof(unsigned long long), st));
    Shape sh;
    LAUNCH(launch_check_state(ct, r, (int)n, ctx->d_chk, grid_for(ctx, sh, n), sh.block, st));
    CK(cudaMemcpyAsync(ctx->h_chk, ctx->d_chk, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(ctx, BMXG_ERR_CUDA, std::string("state check: ") + cudaGetErrorString(e));
    return read_check(ctx, out);
}

constexpr int64_t kStoreFused = 65536;

// bmxg_get_state through one kernel: straight into device arrays, or into the
// staging and from there into host arrays.
int store_fused(bmxg_ctx *ctx, bmxg_particles *p, bool host, bool fx)
{
    const int64_t n = ctx->n;
    const DevState &S = ctx->S;
    cudaStream_t st = ctx->stream;
    struct Out {
        void *dst;
        char *from;
        size_t bytes;
    };
    std::vector<Out> outs;
    size_t used = 0;
    // spheres have no rod fields (those arrays are left alone)
    const bool rods = S.has_rods != 0;
    struct Want {
        void *dst;
        size_t bytes;
    };
    const size_t d8 = sizeof(double) * (size_t)n, i4 = sizeof(int) * (size_t)n;
    Want w[] = {{p->x, d8},          {p->y, d8},         {p->z, d8},
                {p->velx, d8},       {p->vely, d8},      {p->velz, d8},
                {p->wx, d8},         {p->wy, d8},        {p->wz, d8},
                {rods ? p->theta : nullptr, d8},         {rods ? p->phi : nullptr, d8},
                {rods ? p->n_bnds : nullptr, i4},        {rods ? p->seg_id1 : nullptr, 4 * i4},
                {rods ? p->seg_id2 : nullptr, 4 * i4},   {rods ? p->site : nullptr, 4 * i4},
                {rods ? p->position : nullptr, i4},      {rods ? p->fix_site : nullptr, i4},
                {rods ? p->fuse_flag : nullptr, i4},     {rods ? p->split_flag : nullptr, i4},
                {rods ? p->new_flag : nullptr, i4},      {rods ? p->dltd : nullptr, 6 * i4}};
    if (host) {
        for (const Want &q : w)
            if (q.dst) used += (q.bytes + 15) / 16 * 16;
        if (int rc = ensure_io(ctx, used)) return rc;
        used = 0;
    }
    void *at[sizeof(w) / sizeof(w[0])];
    for (size_t k = 0; k < sizeof(w) / sizeof(w[0]); ++k) {
        at[k] = w[k].dst;
        if (!host || !w[k].dst) continue;
        at[k] = ctx->io_buf + used;
        outs.push_back({w[k].dst, ctx->io_buf + used, w[k].bytes});
        used += (w[k].bytes + 15) / 16 * 16;
    }
    StoreFields F;
    F.x = (double *)at[0];
    F.y = (double *)at[1];
    F.z = (double *)at[2];
    for (int k = 0; k < 6; ++k) F.v[k] = (double *)at[3 + k];
    F.theta = (double *)at[9];
    F.phi = (double *)at[10];
    F.n_bnds = (int *)at[11];
    F.seg_id1 = (int *)at[12];
    F.seg_id2 = (int *)at[13];
    F.site = (int *)at[14];
    F.position = (int *)at[15];
    F.fix_site = (int *)at[16];
    F.fflag = (int *)at[17];
    F.sflag = (int *)at[18];
    F.nflag = (int *)at[19];
    F.dltd = (int *)at[20];
    if (fx && store_bytes(F, (int)n) + 3 * d8 > kScatterPass) {  // (a pass for each field: converted before them)
        if (int rc = sync_fp64(ctx)) return rc;
        fx = false;
    }
    LAUNCH(launch_store(S, ctx->parity, F, fx, ctx->vel32, st));
    if (fx) ctx->fx_ahead = false;
    for (const Out &o : outs) CK(cudaMemcpyAsync(o.dst, o.from, o.bytes, cudaMemcpyDeviceToHost, st));
    if (!rods && ctx->stepped)  // a step of spheres only clears the fusion flags (bmx_pc_interaction.cpp:178-180)
        for (int32_t *f : {p->fuse_flag, p->split_flag, p->new_flag}) {
            if (!f) continue;
            if (host) std::memset(f, 0, i4);
            else CK(cudaMemsetAsync(f, 0, i4, st));
        }
    CK(cudaStreamSynchronize(st));
    return BMXG_OK;
}

}  // namespace

extern "C" {

int bmxg_get_state(bmxg_ctx *ctx, bmxg_particles *p, int where)
{
    if (!ctx) return BMXG_ERR_ARG;
    (void)cudaGetLastError();  // drop a non-sticky error another library left on this thread
    if (!ctx->have_state) return fail(ctx, BMXG_ERR_STATE, "no state loaded");
    if (!p || p->n != ctx->n) return fail(ctx, BMXG_ERR_ARG, "particle count differs from the loaded state");
    if (where != BMXG_HOST && where != BMXG_DEVICE) return fail(ctx, BMXG_ERR_ARG, "bad `where`");
    // positions still in the list's fixed point are converted as they are
    // stored, where all three axes are asked for; otherwise first
    const bool fx_store = ctx->fx_ahead && p->x && p->y && p->z;
    if (!fx_store) {
        if (int rc = sync_fp64(ctx)) return rc;
    }
    const int64_t n = ctx->n;
    if (n == 0) return BMXG_OK;
    const DevState &S = ctx->S;
    cudaStream_t st = ctx->stream, st1 = ctx->io_stream;
    const bool host = where == BMXG_HOST;
    const int blk = ctx->sh_misc.block;
    const int grd = grid_for(ctx, ctx->sh_misc, n);
    const int a = ctx->parity;
    // Device arrays receive the caller-order scatter directly, every field in
    // one kernel.  Host arrays of rod states and of few particles go through
    // the same kernel into the staging, then out field by field; of many
    // spheres: each field is scattered into one of two staging halves on the
    // compute stream and copied out on the copy stream, so that the copy of one
    // field overlaps the scatter of the next (500 000 spheres: six scatters of
    // 6 us behind copies of 21 us; below kStoreFused the launches cost more).
    if (!host || S.has_rods || n <= kStoreFused) return store_fused(ctx, p, host, fx_store);
    JoinIo join{nullptr};
    int used = 0;
    {
        int rc0 = ensure_io(ctx, (size_t)n * 48 + 256);
        if (rc0) return rc0;
    }
    CK(cudaEventRecord(ctx->io_ev[0], st));
    CK(cudaStreamWaitEvent(st1, ctx->io_ev[0], 0));
    join.s = st1;
    char *half[2] = {ctx->io_buf, ctx->io_buf + (size_t)n * 24 + 128};
    // destination of the next field: the caller's array or a staging half
    cudaError_t wait_err = cudaSuccess;
    auto begin = [&](void *dst) -> void * {
        (void)dst;
        const int h = used & 1;
        if (used >= 2) {  // the half's previous copy-out is done
            const cudaError_t e = cudaStreamWaitEvent(st, ctx->io_ev[4 + h], 0);
            if (e != cudaSuccess) wait_err = e;
        }
        return half[h];
    };
    auto finish = [&](void *dst, size_t bytes) -> int {
        CK(wait_err);
        const int h = used & 1;
        CK(cudaEventRecord(ctx->io_ev[2 + h], st));
        CK(cudaStreamWaitEvent(st1, ctx->io_ev[2 + h], 0));
        CK(cudaMemcpyAsync(dst, half[h], bytes, cudaMemcpyDeviceToHost, st1));
        CK(cudaEventRecord(ctx->io_ev[4 + h], st1));
        ++used;
        return BMXG_OK;
    };
    auto out_d = [&](double *dst, const double *src) -> int {
        if (!dst || !src) return BMXG_OK;
        double *o = (double *)begin(dst);
        LAUNCH(launch_scatter_d(o, src, S.orig, (int)n, grd, blk, st));
        return finish(dst, sizeof(double) * n);
    };
    auto out_f = [&](double *dst, const float *src) -> int {  // FP32F velocities, widened
        if (!dst || !src) return BMXG_OK;
        double *o = (double *)begin(dst);
        LAUNCH(launch_scatter_f2d(o, src, S.orig, (int)n, grd, blk, st));
        return finish(dst, sizeof(double) * n);
    };
    int rc;
    if (fx_store) {
        double *dst[3] = {p->x, p->y, p->z};
        for (int ax = 0; ax < 3; ++ax) {
            double *o = (double *)begin(dst[ax]);
            LAUNCH(launch_list_to_fp64_axis(S, a, ax, o, blk, st));
            if ((rc = finish(dst[ax], sizeof(double) * n))) return rc;
        }
        ctx->fx_ahead = false;
    } else {
        if ((rc = out_d(p->x, S.x[a]))) return rc;
        if ((rc = out_d(p->y, S.y[a]))) return rc;
        if ((rc = out_d(p->z, S.z[a]))) return rc;
    }
    if (ctx->vel32) {
        if ((rc = out_f(p->velx, S.vxf))) return rc;
        if ((rc = out_f(p->vely, S.vyf))) return rc;
        if ((rc = out_f(p->velz, S.vzf))) return rc;
    } else {
        if ((rc = out_d(p->velx, S.vx))) return rc;
        if ((rc = out_d(p->vely, S.vy))) return rc;
        if ((rc = out_d(p->velz, S.vz))) return rc;
    }
    if ((rc = out_d(p->wx, S.wx))) return rc;
    if ((rc = out_d(p->wy, S.wy))) return rc;
    if ((rc = out_d(p->wz, S.wz))) return rc;
    if (ctx->stepped) {
        // spheres: the step only clears the fusion flags (bmx_pc_interaction.cpp:178-180)
        for (int32_t *f : {p->fuse_flag, p->split_flag, p->new_flag})
            if (f) std::memset(f, 0, sizeof(int32_t) * n);
    }
    CK(cudaStreamSynchronize(st));
    CK(cudaStreamSynchronize(st1));
    return BMXG_OK;
}

}  // extern "C"

namespace {

// Enqueue one DEM step reading buffer a.  resync: the FP32F sphere step
// re-derives every slot's offsets and bin from its FP64 position.
// profiling mode: an event pair around the force kernel of this step
void prof_events(bmxg_ctx *ctx, cudaEvent_t *k0, cudaEvent_t *k1)
{
    *k0 = *k1 = nullptr;
    if (!ctx->profiling) return;
    while (ctx->kev.size() < 2 * (ctx->kev_used + 1)) {
        cudaEvent_t e;
        if (cudaEventCreate(&e) != cudaSuccess) break;
        ctx->kev.push_back(e);
    }
    if (ctx->kev.size() >= 2 * (ctx->kev_used + 1)) {
        *k0 = ctx->kev[2 * ctx->kev_used];
        *k1 = ctx->kev[2 * ctx->kev_used + 1];
        ++ctx->kev_used;
    }
}

// ---- neighbour list with a skin ---------------------------------------
constexpr int kListMaxAge = 64;      // builds at least this often
// FP64 spheres step over the list where it is the faster path.  A load and 100 steps, per-step
// path / list, us, 3 and 10 slots a column: 16 000 slots 2008 / 2344, 2466 / 3443, 20 000 2374 /
// 2399, 3115 / 3733, 24 000 2501 / 2399, 2995 / 3330, 28 000 3101 / 2371, 3663 / 3416, 40 000 3996 /
// 2581, 6007 / 3755, 160 000 7459 / 5019, 12 292 / 8041, 400 000 13 864 / 9613, 22 939 / 15 815
// (between kList64Slots and kList64Sure it gains 4 % at best and loses up to 20 %: there
// it is for states that step for long).
// From a load on, with the build: 6 steps of 28 000 slots 396 / 377, 441 / 451, 40 000 476 /
// 410, 578 / 482, 400 000 1279 / 1069, 1791 / 1424; fewer steps keep the per-step path.
constexpr int kList64Slots = 16384;
constexpr int kList64Sure = 28672;
constexpr int kList64MinSteps = 6;
// Steps of a state's size that pay for the list's buffers and graphs.  In a fresh
// context, per-step path / list, us, 3 and 10 slots a column: 50 000 slots 13 steps 653 / 692,
// 933 / 837, 20 941 / 972, 1352 / 1210, 25 1115 / 996, 1638 / 1269; 100 000 20 1218 / 1346,
// 1760 / 1729, 25 1447 / 1413, 2110 / 1904; 200 000 10 1039 / 1107, 1511 / 1406, 13 1286 / 1194,
// 1879 / 1600; 400 000 8 1319 / 1274, 2010 / 1725; 900 000 6 1641 / 1726, 2617 / 2479, 8 2336 /
// 2007, 3656 / 3037.
inline double list64_pays_back(double n) { return n < kList64Sure ? 150.0 : std::min(26.0, 5.0 + 1.6e6 / n); }
// So few list steps go as a graph (with its conditional node) for each, more as graphs of
// kResyncEvery whose surplus steps return at once: the node costs 7 us, a surplus step its
// blocks' launch.  2 / 3 / 4 FP32F steps as singles and as one graph, us: 20 000 slots 53, 68,
// 84 and 55, 66, 66; 400 000 66, 92, 122 and 90, 92, 103; 700 000 78, 109, 133 and 115, 127, 139;
// 1 million 91, 129, 172 and 139, 155, 176.
inline int list_singles(int64_t n) { return n <= 400000 ? 2 : 4; }
// Fewer steps a build than this: graphs with a conditional node before every step, where
// none stalls.  48 FP32F steps with one node per graph / one per step, by steps a build, us:
// 2000 slots 5: 1033 / 1200, 4: 1203 / 1287, 3: 1474 / 1472, 2: 2108 / 1865, 1.2: 3201 / 2517;
// 200 000 slots 5: 1529 / 1681, 3: 2151 / 2058, 1.2: 4548 / 3658; 1 million 5: 3977 / 4018,
// 3: 5676 / 5092, 1.2: 12 479 / 9857.
constexpr double kStallPeriod = 4.0;
constexpr size_t kRodBytes = 4 + kRodCap * (sizeof(int4) + sizeof(int) + 6 * sizeof(double));  // rod queues, a segment
constexpr int kListMinSteps = 2;     // a shorter first call after a load runs the per-step path

// Skin of the list for the loaded state and parameters, or 0 where the list
// would not reproduce the reference's pair set: the largest cutoff
// 2 r_max + bw plus the skin must stay within the smallest bin width (so
// that every pair inside the cutoff is a stencil pair whatever the bins),
// BMXCheckPair must hold for every stencil pair, and the fixed point's high
// word must resolve offsets to 2^-20 of a bin (and its unit squared be a normal
// FP32 number: the step takes r^2 for one).
float list_skin(const bmxg_ctx *ctx)
{
    if (ctx->S.has_rods || ctx->n == 0 || ctx->n >= (1LL << kNbrShift)) return 0.0f;
    if (ctx->ncells_total >= (1LL << 30)) return 0.0f;  // 3D cell offsets of the build
    double skin = 1e300;
    for (const DevGeom &g : ctx->h_geoms) {
        if (!g.nbh_trivial) return 0.0f;
        const double dmin = std::min(g.dx[0], std::min(g.dx[1], g.dx[2]));
        const double rcut = 2.0 * ctx->rmax + ctx->prm.bndry_width;
        const double sk = std::min(0.25 * dmin, 0.95 * (dmin - rcut));
        if (!(sk >= 0.02 * dmin)) return 0.0f;
        for (int d = 0; d < 3; ++d) {
            const double unit = std::ldexp((g.per[d] ? 1.0 : 4.0) * g.len[d], -32);
            if (!(unit <= std::ldexp(dmin, -20) && unit >= std::ldexp(1.0, -62))) return 0.0f;
        }
        skin = std::min(skin, sk);
    }
    return (float)skin;
}

// The FP64 steps in a row over one list, or without one, end (poor: its builds fell due
// too often).
void list64_end(bmxg_ctx *ctx, bool poor)
{
    if (ctx->list64_live) ctx->list64_short = (poor || ctx->list64_lived < kList64MinSteps) ? ctx->list64_short + 1 : 0;
    ctx->list64_live = false;
    ctx->list64_lived = 0;
    ctx->list64_since = 0;
}

// Whether FP64 steps go over the list (which covers the state: list_skin).
// A list pays from kList64MinSteps on, and those are not known beforehand: a reader of
// the bins, another form or a load ends it, or the state moves so fast that it is built
// again too soon.  From the second list in a row that did not last, twice as many steps
// without one, or in the call, are asked for each time.  One step and an export of the
// neighbour list in turn, us: 20 000 slots 100 without, 154 with a list for every step, 400 000
// 230 and 263.
bool list64_pays(bmxg_ctx *ctx, int32_t nsteps)
{
    if (!ctx->list_room || ctx->list64_bail || ctx->n <= kList64Slots) return false;
    if (ctx->list_valid && ctx->list_prec == BMXG_FP64) return true;
    if (ctx->list64_since + nsteps < (int64_t)kList64MinSteps << std::min(std::max(ctx->list64_short - 1, 0), 10))
        return false;
    if (ctx->S.nbr) return true;
    const double steps = (double)(ctx->plain64 + nsteps), n = (double)ctx->n;
    if (steps < list64_pays_back(n)) return false;
    // (refused once, this state size goes without)
    const size_t need = (size_t)ctx->n * 320 + (size_t)ctx->ncells_total * sizeof(int);
    if (!room_for(ctx, need, 4)) ctx->list_room = false;
    return ctx->list_room;
}

// Allocate the list on first use; (re)initialise its control block when the
// state or the skin changed, asking the next step for a build.
int ensure_list(bmxg_ctx *ctx, float skin, int precision)
{
    DevState &S = ctx->S;
    if (!S.nbr) {
        int rc;
        if ((rc = dalloc(ctx, &S.nbr, (size_t)(kNbrCap - kNbrInline) * ctx->n))) return rc;
        if ((rc = dalloc(ctx, &S.lrec, ctx->n))) return rc;
        const size_t ngroups = ((size_t)ctx->n + 31) / 32;
        if ((rc = dalloc(ctx, &S.xcnt, ngroups))) return rc;
        if ((rc = dalloc(ctx, &S.xoff, ngroups + 1))) return rc;
        if ((rc = dalloc(ctx, &S.xlist, (size_t)(kNbrCap - kNbrInline) * ctx->n))) return rc;
        for (int k = 0; k < 2; ++k) {
            if ((rc = dalloc(ctx, &S.fxh[k], ctx->n))) return rc;
            if ((rc = dalloc(ctx, &S.fxl[k], 3 * (size_t)ctx->n))) return rc;
        }
        if ((rc = dalloc(ctx, &S.cellstart, ctx->ncells_total + 1))) return rc;
        // (the scratch serves the scan of the column counts and that of the groups' entries)
        const int nscan = (int)std::max<int64_t>(S.ncols_total, ((int64_t)ctx->n + 31) / 32);
        if ((rc = dalloc(ctx, &ctx->cell_scratch, scan_scratch_ints(nscan)))) return rc;
        S.lctl = &ctx->d_step->ctl;
        S.ncells_total = (int)ctx->ncells_total;
        S.cols_max = 0;
        for (const DevGeom &g : ctx->h_geoms) S.cols_max = std::max(S.cols_max, g.n[0] * g.n[1]);
        // offsets within [0, n] from the start, whatever a build leaves unwritten
        CK(cudaMemsetAsync(S.cellstart, 0, sizeof(int) * (ctx->ncells_total + 1), ctx->stream));
        ctx->list_valid = false;
        drop_graphs(ctx);  // captured kernels hold the state's pointers by value
    }
    if (ctx->list_valid && skin == ctx->skin_cur && ctx->list_prec == precision) return BMXG_OK;
    // (the other form's steps left their own positions ahead)
    if (int rc = sync_fp64(ctx)) return rc;
    ctx->list_prec = precision;
    double dmax = 0.0;
    for (const DevGeom &g : ctx->h_geoms) dmax = std::max(dmax, std::max(g.dx[0], std::max(g.dx[1], g.dx[2])));
    ListCtl h;
    std::memset(&h, 0, sizeof(h));
    h.skin = skin;
    h.eps_step = (float)(4.0e-7 * dmax);
    for (int k = 0; k < 3; ++k) {  // empty spreads (see k_list_decide)
        h.inc_min[k] = 0xff800000u;
        h.inc_max[k] = 0x007fffffu;
    }
    h.max_age = kListMaxAge;
    h.whole = precision == BMXG_FP64;
    h.force = 1;
    h.par = ctx->parity;
    CK(cudaMemcpyAsync(S.lctl, &h, sizeof(h), cudaMemcpyHostToDevice, ctx->stream));
    // the fixed-point positions (FP64 form: the screen's coordinates) start from
    // the FP64 ones
    if (precision == BMXG_FP32F)
        LAUNCH(launch_list_init(S, ctx->parity, grid_for(ctx, ctx->sh_misc, ctx->n), ctx->sh_misc.block,
                                ctx->stream));
    else {
        LAUNCH(launch_list64_begin(S, ctx->parity, ctx->stream));
        ctx->bins_exact = false;  // (in place of the offsets from the bins' corners)
    }
    ctx->fx_ahead = false;
    CK(cudaStreamSynchronize(ctx->stream));
    ctx->skin_cur = skin;
    ctx->body_runs_seen = 0;
    ctx->list_begun = true;
    ctx->list_valid = true;
    return BMXG_OK;
}

// Bins of buffer `parity` as the reference has them (after list steps froze
// them); every consumer of the bins other than a list step calls this.
// FP64 positions of buffer `parity` from the list path's fixed point, when
// list steps ran since they were last written; every reader of the FP64
// positions calls this first.
int sync_fp64(bmxg_ctx *ctx)
{
    if (!ctx->fx_ahead || !ctx->have_state || ctx->n == 0) return BMXG_OK;
    LAUNCH(launch_list_to_fp64(ctx->S, ctx->parity, grid_for(ctx, ctx->sh_misc, ctx->n), ctx->sh_misc.block,
                               ctx->stream));
    ctx->fx_ahead = false;
    return BMXG_OK;
}

int ensure_exact(bmxg_ctx *ctx)
{
    if (int rc = sync_fp64(ctx)) return rc;
    if (ctx->bins_exact || !ctx->have_state) return BMXG_OK;
    const int blk = ctx->sh_misc.block, grd = grid_for(ctx, ctx->sh_misc, ctx->n);
    LAUNCH(launch_bin(ctx->S, ctx->parity, grd, blk, ctx->stream));
    LAUNCH(launch_rebuild(ctx->S, ctx->parity, ctx->scan_scratch, grd, blk, ctx->stream));
    ctx->bins_exact = true;
    ctx->list_valid = false;
    return BMXG_OK;
}

// The same for a reader of the bins between steps.
int read_bins(bmxg_ctx *ctx)
{
    list64_end(ctx);
    return ensure_exact(ctx);
}

// Steps of a list call from here on: their number and the buffer the first reads.
int set_list_run(bmxg_ctx *ctx, int steps)
{
    ctx->h_run[0] = steps;
    ctx->h_run[1] = ctx->parity;
    static_assert(offsetof(ListCtl, par) == offsetof(ListCtl, left) + sizeof(int), "set together");
    CK(cudaMemcpyAsync(&ctx->S.lctl->left, ctx->h_run, 2 * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
    return BMXG_OK;
}

// One list step: decide, build when needed (capturing: a conditional node
// where `build`, else the step stalls), then the force / update kernel.  What
// ran is counted after the call (two kernels a step, the build's when it ran):
// a kernel of a step that did not run returns at once.
int enqueue_list_step(bmxg_ctx *ctx, double dt, int precision, bool build)
{
    const DevState &S = ctx->S;
    cudaStream_t st = ctx->stream;
    const DevParams P = dev_params(ctx->prm);
    // the decision kernel clears the per-step counters
    const int64_t n = ctx->n;
    const int mblk = ctx->sh_misc.block, mgrd = grid_for(ctx, ctx->sh_misc, n);
    if (ctx->capturing && !build) {
        launch_list_decide(S, 0, kDecideStall, st);
    } else if (ctx->capturing) {
        cudaStreamCaptureStatus cs;
        cudaGraph_t cg = nullptr;
        const cudaGraphNode_t *deps = nullptr;
        const cudaGraphEdgeData *ed = nullptr;
        size_t nd = 0;
        CK(cudaStreamGetCaptureInfo(st, &cs, nullptr, &cg, &deps, &ed, &nd));
        cudaGraphConditionalHandle h;
        CK(cudaGraphConditionalHandleCreate(&h, cg, 0, 0));
        launch_list_decide(S, (unsigned long long)h, ctx->list_one ? kDecideOne : kDecideCond, st);
        CK(cudaStreamGetCaptureInfo(st, &cs, nullptr, &cg, &deps, &ed, &nd));
        cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeIf;
        cp.conditional.size = 1;
        cudaGraphNode_t cn = nullptr;
        CK(cudaGraphAddNode(&cn, cg, deps, ed, nd, &cp));
        CK(cudaStreamUpdateCaptureDependencies(st, &cn, nullptr, 1, cudaStreamSetCaptureDependencies));
        CK(cudaStreamBeginCaptureToGraph(ctx->body_stream, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                         cudaStreamCaptureModeRelaxed));
        if (precision == BMXG_FP64) launch_list64_fx(S, ctx->body_stream);
        launch_list_rebuild(S, P, ctx->cell_scratch, mgrd, mblk, ctx->lb_block, ctx->body_stream);
        const cudaError_t e1 = cudaPeekAtLastError();
        cudaGraph_t body = nullptr;
        const cudaError_t e2 = cudaStreamEndCapture(ctx->body_stream, &body);
        if (e1 != cudaSuccess || e2 != cudaSuccess)
            return fail(ctx, BMXG_ERR_CUDA,
                        std::string("list build capture: ") + cudaGetErrorString(e1 != cudaSuccess ? e1 : e2));
    } else {
        launch_list_decide(S, 0, kDecideBuild, st);
        if (precision == BMXG_FP64) launch_list64_fx(S, st);
        launch_list_rebuild(S, P, ctx->cell_scratch, mgrd, mblk, ctx->lb_block, st);
        const cudaError_t e = cudaPeekAtLastError();
        if (e != cudaSuccess) return fail(ctx, BMXG_ERR_CUDA, std::string("list build: ") + cudaGetErrorString(e));
    }
    cudaEvent_t k0, k1;
    prof_events(ctx, &k0, &k1);
    if (k0) cudaEventRecord(k0, st);
    const bool chained = ctx->capturing && !build;
    if (precision == BMXG_FP64) launch_list64_step(S, P, dt, st, chained);
    else launch_list_step(S, P, dt, ctx->nsm, ctx->ls_block, ctx->ls_passes, st, ctx->ls_persist, chained);
    if (k1) cudaEventRecord(k1, st);
    const cudaError_t le = cudaPeekAtLastError();
    if (le != cudaSuccess) return fail(ctx, BMXG_ERR_CUDA, std::string("list step: ") + cudaGetErrorString(le));
    return BMXG_OK;
}

int enqueue_step(bmxg_ctx *ctx, double dt, int precision, int a, int resync)
{
    if (ctx->list_on) return enqueue_list_step(ctx, dt, precision, resync != 0);  // (list steps take no re-sync: a build)
    const DevState &S = ctx->S;
    cudaStream_t st = ctx->stream;
    const DevParams P = dev_params(ctx->prm);
    const int b = a ^ 1;
    const int64_t n = ctx->n;
    const int mblk = ctx->sh_misc.block, mgrd = grid_for(ctx, ctx->sh_misc, n);
    cudaEvent_t k0, k1;
    prof_events(ctx, &k0, &k1);
    if (!S.has_rods) {
        const Shape &sh = ctx->sh_sphere[precision == BMXG_FP32F ? 1 : 0];
        if (k0) cudaEventRecord(k0, st);
        int sg, sb;
        stencil_shape(ctx, sh, n, &sg, &sb);
        LAUNCH(launch_sphere_step(S, P, dt, a, precision, sg, sb, st, resync, sh.grid > 0));
        if (k1) cudaEventRecord(k1, st);
    } else {
        const int rg = grid_for(ctx, ctx->sh_rod, n);
        // the flat pipeline over the pairs the bookkeeping records
        const bool pipe = S.rwork != nullptr;
        LAUNCH(launch_rod_book(S, P, a, pipe, rg, ctx->sh_rod.block, st));
        if (k0) cudaEventRecord(k0, st);
        if (pipe) {
            LAUNCH(launch_rod_pairs(S, P, dt, a, precision, ctx->nsm, (int)n, st));
            if (k1) cudaEventRecord(k1, st);
        } else {
            LAUNCH(launch_rod_force(S, P, a, rg, ctx->sh_rod.block, st));
            if (k1) cudaEventRecord(k1, st);
            LAUNCH(launch_rod_update(S, dt, a, mgrd, mblk, st));
        }
    }
    LAUNCH(launch_rebuild(S, b, ctx->scan_scratch, mgrd, mblk, st, true));
    return BMXG_OK;
}

// (list steps take the buffer from the device: one graph serves either parity.
// A conditional node costs 6.6 us per evaluation even when false, so the graph of
// kResyncEvery list steps has one, before its first step; a step that finds a
// build due stalls, with the rest of the graph, until the next graph's.  200 000
// spheres, 100 steps, load and store: 2.19 -> 1.70 ms; 2.73 M in 256 colonies the
// same within noise, where a stalled launch of 10 700 blocks costs what it saves.
// Where builds fall due every few steps the stalls cost more than the nodes: see
// kStallPeriod)
int get_graph(bmxg_ctx *ctx, double dt, int precision, int parity, cudaGraphExec_t *out, int single = -1)
{
    if (ctx->list_on) {
        parity = 0;
        if (single >= 0) single = std::max(single, 1);
    }
    GraphKey key{dt, precision, parity, single, ctx->list_on};
    auto it = ctx->graphs.find(key);
    if (it != ctx->graphs.end()) {
        *out = it->second;
        return BMXG_OK;
    }
    // kResyncEvery steps (an even number, so the graph ends on the parity it
    // starts from); the FP32F re-sync falls on its last step
    cudaGraph_t g = nullptr;
    const int64_t before = ctx->launches;
    CK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    int rc2 = BMXG_OK;
    ctx->capturing = true;
    if (single >= 0)
    {
        ctx->list_one = ctx->list_on && single == 1;
        rc2 = enqueue_step(ctx, dt, precision, parity, single);
        ctx->list_one = false;
    }
    else
        for (int s = 0; s < kResyncEvery && !rc2; ++s)
            rc2 = enqueue_step(ctx, dt, precision, parity ^ (s & 1),
                               ctx->list_on ? s == 0 || single == -2 : s == kResyncEvery - 1);
    ctx->capturing = false;
    cudaError_t e = cudaStreamEndCapture(ctx->stream, &g);
    if (rc2) {
        if (g) cudaGraphDestroy(g);
        ctx->launches = before;
        return rc2;
    }
    ctx->graph_kernels[key] = (int)(ctx->launches - before);  // counted per replay instead
    ctx->launches = before;
    if (e != cudaSuccess) return fail(ctx, BMXG_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(e));
    cudaGraphExec_t ex = nullptr;
    e = cudaGraphInstantiate(&ex, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return fail(ctx, BMXG_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(e));
    ctx->graphs[key] = ex;
    *out = ex;
    return BMXG_OK;
}

// nsteps list steps, to the end or (FP64 form) until a slot left the range the
// list covers: *done of them ran (the stream is synchronised, h_cnt and h_lctl
// read back).  Graphs are launched for the steps left and for those that the
// builds due by then will stall, and again for what is still left.
int list_steps(bmxg_ctx *ctx, double dt, int32_t nsteps, int precision, int32_t *done)
{
    cudaStream_t st = ctx->stream;
    // a call of few steps sets nothing before them (the copy costs 3-6 us): none are
    // left over from the last, and the buffer is where that ended
    const bool few = !ctx->profiling && nsteps <= list_singles(ctx->n);
    if (!few)
        if (int rc = set_list_run(ctx, nsteps)) return rc;
    ctx->list_valid = false;  // until the steps have run
    int left = nsteps;
    double due = 0.0;  // builds of this call that fell due
    bool poor = false;
    while (left > 0) {
        cudaGraphExec_t g = nullptr;
        const double period = (ctx->period_steps + (nsteps - left)) / (ctx->period_builds + due);
        if (ctx->profiling) {  // launched one by one, with events around the force kernel
            for (int k = 0; k < left; ++k)
                if (int rc = enqueue_list_step(ctx, dt, precision, true)) return rc;
        } else if (few || (left < nsteps && left <= 4)) {  // (the last ones: none can stall)
            if (int rc = get_graph(ctx, dt, precision, 0, &g, few ? 1 : 2)) return rc;
            for (int k = 0; k < left; ++k) CK(cudaGraphLaunch(g, st));
        } else {
            const bool each = period < kStallPeriod;
            if (int rc = get_graph(ctx, dt, precision, 0, &g, each ? -2 : -1)) return rc;
            const double stalled = each ? 0.0 : 0.5 * (kResyncEvery - 1) * left / std::max(period, 1.0);
            const int graphs = std::max(1, (int)((left + stalled) / kResyncEvery + 0.5));
            for (int k = 0; k < graphs; ++k) CK(cudaGraphLaunch(g, st));
        }
        CK(cudaEventRecord(ctx->ev1, st));
        CK(cudaMemcpyAsync(ctx->h_step, ctx->d_step, sizeof(StepBlock), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        const int now = ctx->h_lctl->left;
        due = (double)(ctx->h_lctl->body_runs - ctx->body_runs_seen) - (ctx->list_begun ? 1.0 : 0.0);
        const bool over = precision == BMXG_FP64 && ctx->h_lctl->overflow;  // (the step of that build did not run)
        if (over || ctx->h_lctl->bail) {
            ctx->list64_bail = true;
            left = now + (over ? 1 : 0);
            break;
        }
        // (FP64: the rest of the call goes without)
        poor = precision == BMXG_FP64 && due >= 2.0 && (nsteps - now) < kList64MinSteps * due;
        if (poor) {
            left = now;
            break;
        }
        if (now >= left || now < 0) return fail(ctx, BMXG_ERR_STATE, "internal: list steps made no progress");
        left = now;
    }
    *done = nsteps - left;
    ctx->parity ^= *done & 1;
    ctx->step_count += *done;
    const unsigned long long runs = ctx->h_lctl->body_runs - ctx->body_runs_seen;
    ctx->body_runs_seen = ctx->h_lctl->body_runs;
    ctx->launches += (int64_t)runs * (kListBodyKernels + (precision == BMXG_FP64 ? 1 : 0)) + 2 * (int64_t)*done;
    ctx->list_begun = ctx->list_begun && runs == 0;
    ctx->period_steps += *done;
    ctx->period_builds += std::max(due, 0.0);
    while (ctx->period_steps > 64.0) {
        ctx->period_steps *= 0.5;
        ctx->period_builds *= 0.5;
    }
    ctx->stats.n_rebins += (int64_t)runs;
    if (*done > 0) {
        ctx->bins_exact = false;
        if (precision == BMXG_FP32F) ctx->fx_ahead = true;
    }
    ctx->list_valid = !(precision == BMXG_FP64 && (ctx->list64_bail || poor));
    if (precision == BMXG_FP64) {
        ctx->list64_live = true;
        ctx->list64_lived += *done;
        if (!ctx->list_valid) list64_end(ctx, poor);
    }
    return BMXG_OK;
}

// What a call of nsteps steps in this form needs before it enqueues them:
// the list or exact bins, the buffers of the path it takes (graphs captured
// before an allocation are dropped: they hold the state's pointers by value).
int step_setup(bmxg_ctx *ctx, int32_t nsteps, int32_t precision)
{
    if (precision == BMXG_FP32F) list64_end(ctx);
    float skin = (ctx->list_mode && (precision == BMXG_FP32F || list64_pays(ctx, nsteps))) ? list_skin(ctx) : 0.0f;
    if (skin > 0.0f && precision == BMXG_FP32F && !ctx->list_valid && nsteps < kListMinSteps && ctx->step_count == 0)
        skin = 0.0f;
    if (skin > 0.0f && precision == BMXG_FP64) {
        const size_t held = ctx->allocs.size();
        int rc = ensure_list(ctx, skin, precision);
        if (rc == BMXG_ERR_OOM) {  // no room for the list: FP64 steps go without
            while (ctx->allocs.size() > held) {
                cudaFree(ctx->allocs.back());
                ctx->allocs.pop_back();
            }
            (void)cudaGetLastError();
            ctx->S.nbr = nullptr;
            ctx->list_room = false;
            skin = 0.0f;
            rc = ensure_exact(ctx);
        }
        if (rc) return rc;
    } else if (skin > 0.0f) {
        int rc = ensure_list(ctx, skin, precision);
        if (rc) return rc;
    } else {
        int rc = ensure_exact(ctx);
        if (rc) return rc;
    }
    ctx->list_on = skin > 0.0f;
    ctx->pcap_valid = false;
    if (ctx->list_on && precision == BMXG_FP32F && ctx->pair_capture && !ctx->S.pcap) {
        int rc = dalloc(ctx, &ctx->S.pcap, (size_t)(kPairCap + 1) * ctx->n);
        if (rc) return rc;
        drop_graphs(ctx);
    }
    // the rod pipelines' buffers (the queue's length is an int), which the FP64 form can
    // do without
    if (ctx->S.has_rods && !ctx->S.rwork && precision == BMXG_FP64 && !ctx->rod_walk)
        ctx->rod_walk = ctx->n > (1LL << 26) || !room_for(ctx, (size_t)ctx->n * kRodBytes, 4);
    if (ctx->S.has_rods && !ctx->S.rwork && !(precision == BMXG_FP64 && ctx->rod_walk)) {
        const size_t n = (size_t)ctx->n;
        int4 *work = nullptr;
        int *cnt = nullptr, *q64 = nullptr;
        double *res = nullptr;
        RodCtl *ctl = nullptr;
        const size_t held = ctx->allocs.size();
        int rc = dalloc(ctx, &q64, n * kRodCap);
        if (!rc) rc = dalloc(ctx, &cnt, n);
        if (!rc) rc = dalloc(ctx, &res, n * kRodCap * 6);
        if (!rc) rc = dalloc(ctx, &work, n * kRodCap);
        if (!rc) rc = dalloc(ctx, &ctl, 1);
        if (rc) {
            // no room for the queues after all: the FP64 form walks
            while (ctx->allocs.size() > held) {
                cudaFree(ctx->allocs.back());
                ctx->allocs.pop_back();
            }
            (void)cudaGetLastError();
            if (precision != BMXG_FP64 || rc != BMXG_ERR_OOM) return rc;
            ctx->rod_walk = true;
            return BMXG_OK;
        }
        ctx->S.rq64 = q64;
        ctx->S.rcnt = cnt;
        ctx->S.rres = res;
        ctx->S.rwork = work;
        ctx->S.rctl = ctl;
        CK(cudaMemsetAsync(ctl, 0, sizeof(RodCtl), ctx->stream));  // (then emptied at the end of each step)
        drop_graphs(ctx);
    }
    return BMXG_OK;
}

}  // namespace

extern "C" {

int bmxg_prepare(bmxg_ctx *ctx, double dt, int32_t precision)
{
    if (!ctx) return BMXG_ERR_ARG;
    ctx->vel64_zero = false;  // (its kernels may write the FP64 velocity planes)
    (void)cudaGetLastError();  // drop a non-sticky error another library left on this thread
    if (!ctx->have_state) return fail(ctx, BMXG_ERR_STATE, "no state loaded");
    if (!std::isfinite(dt)) return fail(ctx, BMXG_ERR_ARG, "bad dt");
    if (precision != BMXG_FP64 && precision != BMXG_FP32F) return fail(ctx, BMXG_ERR_ARG, "bad precision");
    if (ctx->n == 0 || ctx->profiling) return BMXG_OK;
    const double subdt = dt / 1.0;
    if (int rc = step_setup(ctx, 2 * kResyncEvery, precision)) return rc;
    // the replayed graph of kResyncEvery steps and the one-step graphs (with and
    // without the re-sync), from either parity
    auto capture = [&]() -> int {
        for (int parity = 0; parity < 2; ++parity) {
            cudaGraphExec_t g = nullptr;
            if (int rc = get_graph(ctx, subdt, precision, parity, &g)) return rc;
            for (int resync = 0; resync < (ctx->list_on ? 3 : 2); ++resync)
                if (int rc = get_graph(ctx, subdt, precision, parity, &g, resync)) return rc;
            if (ctx->list_on && ctx->period_steps < kStallPeriod * ctx->period_builds)
                if (int rc = get_graph(ctx, subdt, precision, parity, &g, -2)) return rc;
        }
        return BMXG_OK;
    };
    if (int rc = capture()) return rc;
    if (!ctx->list_on || precision != BMXG_FP64) return BMXG_OK;
    // FP64 steps take the list where they are many enough (list64_pays): the others' graphs
    // too
    ctx->list_on = false;
    const int rc = capture();
    ctx->list_on = true;
    return rc;
}

int bmxg_step(bmxg_ctx *ctx, double dt, int32_t nsteps, int32_t precision)
{
    if (!ctx) return BMXG_ERR_ARG;
    // an FP32F sphere step writes the FP32 velocity planes only
    if (precision != BMXG_FP32F || ctx->S.has_rods) ctx->vel64_zero = false;
    (void)cudaGetLastError();  // drop a non-sticky error another library left on this thread
    if (!ctx->have_state) return fail(ctx, BMXG_ERR_STATE, "no state loaded");
    if (nsteps < 0 || !std::isfinite(dt)) return fail(ctx, BMXG_ERR_ARG, "bad dt or nsteps");
    if (precision != BMXG_FP64 && precision != BMXG_FP32F) return fail(ctx, BMXG_ERR_ARG, "bad precision");
    if (ctx->n == 0 || nsteps == 0) return BMXG_OK;
    // nsubsteps = ceil(dt / dtsolid) with dtsolid := dt, subdt = dt / nsubsteps
    // (bmx_pc_interaction.cpp:56-65): one substep of dt / 1
    const double subdt = dt / 1.0;
    // FP32F spheres use the neighbour list wherever it reproduces the pair set,
    // and where the steps are many enough to amortise a build: the first call
    // after a load, if shorter than kListMinSteps, takes the per-step path (a
    // load-step-store caller never reuses a list); later calls build one
    if (int rc = step_setup(ctx, nsteps, precision)) return rc;
    // the per-step counters (the end of each step clears them for the next)
    // (list steps clear them first)
    if (!ctx->list_on) CK(cudaMemsetAsync(ctx->d_cnt, 0, kStepCounters * sizeof(unsigned long long), ctx->stream));
    CK(cudaEventRecord(ctx->ev0, ctx->stream));
    int32_t left = nsteps;
    ctx->kev_used = 0;
    if (ctx->list_on) {
        int32_t done = 0;
        if (int rc = list_steps(ctx, subdt, nsteps, precision, &done)) return rc;
        left -= done;
        if (left > 0) {  // (FP64, out of the list's range) the rest on the per-step path
            if (int rc = ensure_exact(ctx)) return rc;
            ctx->list_on = false;
            CK(cudaMemsetAsync(ctx->d_cnt, 0, kStepCounters * sizeof(unsigned long long), ctx->stream));
        }
    }
    const bool by_list = ctx->list_on;
    const int32_t per_step = left;
    auto eager = [&]() -> int {  // one step on the re-sync schedule
        // re-sync on the last step of each kResyncEvery (not right after a load,
        // whose offsets are exact)
        const int resync = (ctx->step_count % kResyncEvery == kResyncEvery - 1) ? 1 : 0;
        if (ctx->profiling) {  // launched one by one, with events around the force kernel
            int rc = enqueue_step(ctx, subdt, precision, ctx->parity, resync);
            if (rc) return rc;
        } else {  // a captured one-step graph: one launch instead of the step's kernels and copies
            cudaGraphExec_t g1 = nullptr;
            int rc = get_graph(ctx, subdt, precision, ctx->parity, &g1, resync);
            if (rc) return rc;
            CK(cudaGraphLaunch(g1, ctx->stream));
            ctx->launches += ctx->graph_kernels[GraphKey{subdt, precision, ctx->parity, resync}];
        }
        ctx->parity ^= 1;
        ++ctx->step_count;
        --left;
        return BMXG_OK;
    };
    // eager steps up to the next re-sync boundary, graph replays of
    // kResyncEvery steps, eager remainder; every step eager when profiling
    while (left > 0 && (ctx->profiling || ctx->step_count % kResyncEvery != 0 || left < kResyncEvery)) {
        int rc = eager();
        if (rc) return rc;
    }
    if (left >= kResyncEvery) {
        cudaGraphExec_t g = nullptr, g_other = nullptr;
        int rc = get_graph(ctx, subdt, precision, ctx->parity, &g);
        // the other parity's graph too, so that a later call needs no capture
        if (!rc) rc = get_graph(ctx, subdt, precision, ctx->parity ^ 1, &g_other);
        if (rc) return rc;
        const int per = ctx->graph_kernels[GraphKey{subdt, precision, ctx->parity, -1}];
        while (left >= kResyncEvery) {
            CK(cudaGraphLaunch(g, ctx->stream));
            ctx->launches += per;
            ctx->step_count += kResyncEvery;
            left -= kResyncEvery;
        }
    }
    while (left > 0) {
        int rc = eager();
        if (rc) return rc;
    }
    ctx->vel32 = (precision == BMXG_FP32F) && !ctx->S.has_rods;
    ctx->pcap_valid = by_list && precision == BMXG_FP32F && ctx->S.pcap != nullptr;
    if (!by_list) {
        CK(cudaGetLastError());
        CK(cudaEventRecord(ctx->ev1, ctx->stream));
        CK(cudaMemcpyAsync(ctx->h_cnt, ctx->d_cnt, sizeof(DevCounters), cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        ctx->stats.n_rebins += per_step;
        if (ctx->h_cnt->long_column) set_long_cols(ctx, true);
        if (precision == BMXG_FP64) {
            ctx->plain64 += per_step;
            ctx->list64_since += per_step;
        }
        ctx->list_valid = false;
    }
    ctx->stepped = true;
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    ctx->stats.last_step_ms = ms;
    for (size_t k = 0; k < ctx->kev_used; ++k) {
        float km = 0.0f;
        if (cudaEventElapsedTime(&km, ctx->kev[2 * k], ctx->kev[2 * k + 1]) == cudaSuccess) {
            ctx->stats.main_kernel_ms += km;
            ctx->stats.main_kernel_launches += 1;
        }
    }
    ctx->kev_used = 0;
    ctx->stats.n_kernel_launches = ctx->launches;
    const DevCounters &hc = *ctx->h_cnt;
    ctx->stats.n_out_of_domain = (int64_t)(by_list ? hc.out_of_domain : hc.last_out_of_domain);
    ctx->stats.n_edge_ghost = (int64_t)(by_list ? hc.edge_ghost : hc.last_edge_ghost);
    ctx->stats.n_bond_repairs = (int64_t)(by_list ? hc.bond_repairs : hc.last_bond_repairs);
    if (ctx->h_cnt->bad_index) return fail(ctx, BMXG_ERR_STATE, "internal: inconsistent bin counts");
    if (ctx->h_cnt->nonfinite) return fail(ctx, BMXG_ERR_NONFINITE, "a step produced a non-finite position");
    if (ctx->h_cnt->range)
        return fail(ctx, BMXG_ERR_STATE, "a z left the FP32F list path's range (three quarters of a length past the domain)");
    return BMXG_OK;
}

int bmxg_evolve_particles(bmxg_ctx *ctx, double dt, double *cost_per_colony, int32_t *nsubsteps)
{
    if (!ctx) return BMXG_ERR_ARG;
    int rc = bmxg_step(ctx, dt, 1, BMXG_FP64);
    if (rc) return rc;
    if (nsubsteps) *nsubsteps = 1;
    if (cost_per_colony)  // "NumParticles" knapsack weight (bmx_pc_interaction.cpp:470-473)
        for (int c = 0; c < ctx->ncol; ++c) cost_per_colony[c] = (double)(ctx->offsets[c + 1] - ctx->offsets[c]);
    return BMXG_OK;
}

int bmxg_evolve_particles_aos(bmxg_ctx *ctx, void *particles, int64_t n, int32_t nreal, int32_t nint,
                              const int64_t *colony_offsets, double dt, double *cost_per_colony, int32_t *nsubsteps)
{
    if (!ctx || n < 0 || (n > 0 && !particles)) return BMXG_ERR_ARG;
    if (nreal <= 24 || nint <= 34) return BMXG_ERR_ARG;  // up to bond_scale and cpu (bmx_chem.H:38-118)
    AosLayout L;
    L.rdata = 3 * sizeof(double);
    L.idata = L.rdata + (size_t)nreal * sizeof(double) + 2 * sizeof(int);
    L.stride = (L.idata + (size_t)nint * sizeof(int) + 7) / 8 * 8;
    bmxg_particles s;
    std::memset(&s, 0, sizeof(s));
    s.n = n;
    if (n == 0 || n > (1LL << 30)) return bmxg_set_state(ctx, &s, colony_offsets, BMXG_DEVICE);  // (refused there)
    (void)cudaGetLastError();
    cudaStream_t st = ctx->stream;
    // the records in place where the device reads the host's pages, else staged whole
    const size_t N = (size_t)n;
    const bool in_place = ctx->pageable && (reinterpret_cast<uintptr_t>(particles) & 7u) == 0;
    const size_t planes = N * (15 * sizeof(double) + 28 * sizeof(int));
    const size_t rec_at = (planes + 255) / 256 * 256;
    const size_t need = rec_at + (in_place ? 0 : N * L.stride);
    if (need > ctx->aos_cap) {
        CK(cudaStreamSynchronize(st));
        if (ctx->aos_buf) cudaFree(ctx->aos_buf);
        ctx->aos_buf = nullptr;
        ctx->aos_cap = 0;
        CK(cudaMalloc(&ctx->aos_buf, need));
        ctx->aos_cap = need;
    }
    unsigned char *rec = in_place ? static_cast<unsigned char *>(particles)
                                  : reinterpret_cast<unsigned char *>(ctx->aos_buf + rec_at);
    if (!in_place) CK(cudaMemcpyAsync(rec, particles, N * L.stride, cudaMemcpyHostToDevice, st));
    double *d = reinterpret_cast<double *>(ctx->aos_buf);
    int *q = reinterpret_cast<int *>(d + 15 * N);
    // the first record's type says which fields to expect (the check decides)
    int32_t first = 0;
    std::memcpy(&first, static_cast<const unsigned char *>(particles) + L.idata + 5 * sizeof(int), sizeof(first));
    const bool guess = first == BMXG_FUNGI;
    LAUNCH(launch_aos_load(rec, L, (int)n, guess, d, q, st));
    StateCheck chk;
    if (int rc = check_state(ctx, q, d + 3 * N, n, &chk)) return rc;
    if (chk.rods && !guess) LAUNCH(launch_aos_load(rec, L, (int)n, true, d, q, st));
    s.x = d; s.y = d + N; s.z = d + 2 * N; s.radius = d + 3 * N;
    s.velx = d + 9 * N; s.vely = d + 10 * N; s.velz = d + 11 * N;
    s.wx = d + 12 * N; s.wy = d + 13 * N; s.wz = d + 14 * N;
    s.cell_type = q;
    if (chk.rods) {
        s.c_length = d + 4 * N; s.theta = d + 5 * N; s.phi = d + 6 * N; s.area = d + 7 * N; s.bond_scale = d + 8 * N;
        s.id = q + N; s.cpu = q + 2 * N; s.n_bnds = q + 3 * N;
        s.seg_id1 = q + 4 * N; s.seg_id2 = q + 8 * N; s.site = q + 12 * N;
        s.position = q + 16 * N; s.fuse_tip = q + 17 * N; s.fix_site = q + 18 * N;
        s.fuse_flag = q + 19 * N; s.split_flag = q + 20 * N; s.new_flag = q + 21 * N; s.dltd = q + 22 * N;
    }
    if (int rc = load_state(ctx, &s, colony_offsets, BMXG_DEVICE, &chk)) return rc;
    if (int rc = bmxg_evolve_particles(ctx, dt, cost_per_colony, nsubsteps)) return rc;
    LAUNCH(launch_aos_store(rec, L, ctx->S, ctx->parity, st));
    if (!in_place) CK(cudaMemcpyAsync(particles, rec, N * L.stride, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return BMXG_OK;
}

int bmxg_get_stats(const bmxg_ctx *ctx, bmxg_stats *out)
{
    if (!ctx || !out) return BMXG_ERR_ARG;
    *out = ctx->stats;
    out->n_kernel_launches = ctx->launches;
    return BMXG_OK;
}

int bmxg_set_profiling(bmxg_ctx *ctx, int32_t on)
{
    if (!ctx) return BMXG_ERR_ARG;
    ctx->profiling = on != 0;
    if (ctx->profiling) {
        ctx->stats.main_kernel_ms = 0.0;
        ctx->stats.main_kernel_launches = 0;
    }
    return BMXG_OK;
}

int bmxg_step_tile(bmxg_ctx *ctx, const bmxg_tile *tile, const bmxg_particles *reals, const bmxg_particles *ghosts,
                   double dt, int32_t where)
{
    if (!ctx) return BMXG_ERR_ARG;
    ctx->vel64_zero = false;  // (its kernels may write the FP64 velocity planes)
    (void)cudaGetLastError();  // drop a non-sticky error another library left on this thread
    if (!tile || !reals || reals->n < 0 || (ghosts && ghosts->n < 0)) return fail(ctx, BMXG_ERR_ARG, "bad arguments");
    if (where != BMXG_HOST && where != BMXG_DEVICE) return fail(ctx, BMXG_ERR_ARG, "bad `where`");
    if (!std::isfinite(dt)) return fail(ctx, BMXG_ERR_ARG, "bad dt");
    if (ctx->ncol != 1)
        return fail(ctx, BMXG_ERR_UNSUPPORTED, "a tile step takes a context of one geometry (the level's domain)");
    const int64_t nr = reals->n, ng = ghosts ? ghosts->n : 0;
    if (nr == 0) return BMXG_OK;
    if (!reals->x || !reals->y || !reals->z || !reals->radius || !reals->cell_type || !reals->velx || !reals->vely ||
        !reals->velz)
        return fail(ctx, BMXG_ERR_ARG, "reals need x, y, z, radius, cell_type and velx, vely, velz");
    if (ng && (!ghosts->x || !ghosts->y || !ghosts->z || !ghosts->radius || !ghosts->cell_type))
        return fail(ctx, BMXG_ERR_ARG, "ghosts need x, y, z, radius and cell_type");
    if (nr + ng >= (1LL << 30)) return fail(ctx, BMXG_ERR_UNSUPPORTED, "more than 2^30 particles in a tile");
    const bmxg_geometry &g = ctx->geoms[0];
    TileGeom T;
    std::memset(&T, 0, sizeof(T));
    double diag2 = 0.0;
    int64_t ncells = 1;
    for (int d = 0; d < 3; ++d) {
        T.plo[d] = g.prob_lo[d];
        T.phi[d] = g.prob_hi[d];
        T.len[d] = g.prob_hi[d] - g.prob_lo[d];
        T.n[d] = g.n_cell[d];
        const double dx = T.len[d] / (double)T.n[d];  // the whole-domain step's bin width and inverse
        T.dx[d] = dx;
        T.dxf[d] = (float)dx;
        T.dxi[d] = 1.0 / dx;
        T.per[d] = g.is_periodic[d] ? 1 : 0;
        if (tile->lo[d] < 0 || tile->hi[d] < tile->lo[d] || tile->hi[d] >= T.n[d])
            return fail(ctx, BMXG_ERR_ARG, "the tile is not a box of the domain's cells");
        T.lo[d] = tile->lo[d];
        T.nt[d] = tile->hi[d] - tile->lo[d] + 1;
        ncells *= T.nt[d] + 2;
        diag2 += 4.0 * dx * dx;
    }
    if (ncells >= (1LL << 30)) return fail(ctx, BMXG_ERR_UNSUPPORTED, "a tile of more than 2^30 cells");
    T.nbh_trivial = (ctx->prm.neighborhood >= diag2 * (1.0 + 1e-9)) ? 1 : 0;
    const int64_t nt = nr + ng;
    const int ncols = (T.nt[0] + 2) * (T.nt[1] + 2);
    cudaStream_t st = ctx->stream;
    // device arrays are read and written in place (aligned ones), others staged
    auto in_place = [&](const void *f, size_t align) {
        return where == BMXG_DEVICE && reinterpret_cast<uintptr_t>(f) % align == 0;
    };
    bool direct = true;
    for (const double *f : {reals->x, reals->y, reals->z, reals->radius, reals->velx, reals->vely, reals->velz})
        direct = direct && in_place(f, 8);
    direct = direct && in_place(reals->cell_type, 4);
    if (ng) {
        for (const double *f : {ghosts->x, ghosts->y, ghosts->z, ghosts->radius}) direct = direct && in_place(f, 8);
        direct = direct && in_place(ghosts->cell_type, 4);
    }
    // the workspace, kept by the context and grown: what a call clears first
    size_t used = 0;
    auto carve = [&](size_t bytes) {
        const size_t at = used;
        used += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t N = (size_t)nt, NR = (size_t)nr;
    const size_t o_bad = carve(3 * sizeof(unsigned long long) + sizeof(DevCounters));
    const size_t o_cnt = carve(sizeof(int) * ncols);
    const size_t cleared = used;
    const size_t o_pos = carve(sizeof(double) * 4 * N), o_out = carve(sizeof(double) * 6 * NR);
    const size_t o_rel = carve(sizeof(float4) * N), o_srel = carve(sizeof(float4) * N);
    const size_t o_key = carve(sizeof(unsigned long long) * N);
    const size_t o_int = carve(sizeof(int) * 5 * N);
    const size_t o_start = carve(sizeof(int) * (ncols + 1)), o_scan = carve(sizeof(int) * scan_scratch_ints(ncols));
    const size_t o_in = carve(direct ? 0 : 36 * N);
    if (used > ctx->tile_cap) {
        CK(cudaStreamSynchronize(st));
        if (ctx->tile_buf) cudaFree(ctx->tile_buf);
        ctx->tile_buf = nullptr;
        ctx->tile_cap = 0;
        if (cudaMalloc(&ctx->tile_buf, used) != cudaSuccess) {
            (void)cudaGetLastError();
            return fail(ctx, BMXG_ERR_OOM, "tile scratch");
        }
        ctx->tile_cap = used;
    }
    char *base = ctx->tile_buf;
    TileCall C;
    std::memset(&C, 0, sizeof(C));
    C.nreal = (int)nr;
    C.bad = reinterpret_cast<unsigned long long *>(base + o_bad);
    C.out = reinterpret_cast<double *>(base + o_out);
    DevState &S = C.S;
    S.n = (int)nt;
    S.ncol = 1;
    S.ncols_total = ncols;
    S.long_cols = nt / ncols > kLongColumn;  // (by the average: nothing was sorted before)
    S.cnt = reinterpret_cast<DevCounters *>(base + o_bad + 3 * sizeof(unsigned long long));
    S.x[0] = reinterpret_cast<double *>(base + o_pos);
    S.y[0] = S.x[0] + N;
    S.z[0] = S.y[0] + N;
    S.rad = S.z[0] + N;
    S.rel[0] = reinterpret_cast<float4 *>(base + o_rel);
    S.srel[0] = reinterpret_cast<float4 *>(base + o_srel);
    S.lkey = reinterpret_cast<unsigned long long *>(base + o_key);
    S.col[0] = reinterpret_cast<int *>(base + o_int);
    S.iz[0] = S.col[0] + N;
    S.perm[0] = S.iz[0] + N;
    S.siz[0] = S.perm[0] + N;
    S.rank[0] = S.siz[0] + N;
    S.colcnt = reinterpret_cast<int *>(base + o_cnt);
    S.colstart[0] = reinterpret_cast<int *>(base + o_start);
    cudaError_t e = cudaSuccess;
    char *stage = base + o_in;
    const cudaMemcpyKind kin = (where == BMXG_HOST) ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
    const cudaMemcpyKind kout = (where == BMXG_HOST) ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
    auto in = [&](const void *src, size_t bytes) -> const void * {
        if (direct || !bytes) return src;
        if (e == cudaSuccess) e = cudaMemcpyAsync(stage, src, bytes, kin, st);
        const void *q = stage;
        stage += bytes;
        return q;
    };
    auto in_d = [&](const double *src, size_t n) { return static_cast<const double *>(in(src, 8 * n)); };
    C.rx = in_d(reals->x, NR);
    C.ry = in_d(reals->y, NR);
    C.rz = in_d(reals->z, NR);
    C.rr = in_d(reals->radius, NR);
    if (ng) {
        C.gx = in_d(ghosts->x, ng);
        C.gy = in_d(ghosts->y, ng);
        C.gz = in_d(ghosts->z, ng);
        C.gr = in_d(ghosts->radius, ng);
        C.gct = static_cast<const int *>(in(ghosts->cell_type, 4 * (size_t)ng));
    }
    C.rct = static_cast<const int *>(in(reals->cell_type, 4 * NR));
    double *const dst[6] = {reals->x, reals->y, reals->z, reals->velx, reals->vely, reals->velz};
    if (e == cudaSuccess) e = cudaMemsetAsync(base, 0, cleared, st);
    if (e == cudaSuccess) {
        ctx->launches += launch_tile_step(C, T, dev_params(ctx->prm), dt / 1.0,
                                          reinterpret_cast<int *>(base + o_scan), direct ? dst : nullptr, st);
        e = cudaGetLastError();
    }
    unsigned long long *bad = ctx->h_chk;  // (pinned)
    if (e == cudaSuccess) e = cudaMemcpyAsync(bad, C.bad, 3 * sizeof(bad[0]), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess && !direct && !bad[0] && !bad[1]) {  // (non-finite positions are written, then reported)
        for (int k = 0; k < 6 && e == cudaSuccess; ++k)
            e = cudaMemcpyAsync(dst[k], C.out + (size_t)k * NR, 8 * NR, kout, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    if (e != cudaSuccess) return fail(ctx, BMXG_ERR_CUDA, std::string("tile step: ") + cudaGetErrorString(e));
    if (bad[1]) return fail(ctx, BMXG_ERR_UNSUPPORTED, "the tile step takes spheres (YEAST) only");
    if (bad[0])
        return fail(ctx, BMXG_ERR_ARG, "a real particle outside the tile or a ghost outside its one-cell halo");
    if (bad[2]) return fail(ctx, BMXG_ERR_NONFINITE, "a tile step produced a non-finite position");
    return BMXG_OK;
}

int bmxg_set_pair_capture(bmxg_ctx *ctx, int32_t on)
{
    if (!ctx) return BMXG_ERR_ARG;
    if ((on != 0) != ctx->pair_capture) drop_graphs(ctx);  // captured steps hold S by value
    ctx->pair_capture = on != 0;
    if (!ctx->pair_capture) ctx->S.pcap = nullptr;  // the buffer stays with the state's allocations
    ctx->pcap_valid = false;
    return BMXG_OK;
}

int bmxg_get_step_pairs(bmxg_ctx *ctx, int64_t *offs, int32_t *idx, int64_t cap, int64_t *total)
{
    if (!ctx) return BMXG_ERR_ARG;
    (void)cudaGetLastError();
    if (!offs || !total) return fail(ctx, BMXG_ERR_ARG, "offs and total are required");
    if (!ctx->pcap_valid || !ctx->S.pcap) return fail(ctx, BMXG_ERR_STATE, "no list step recorded with capture on");
    const int64_t n = ctx->n;
    const size_t w = kPairCap + 1;
    std::vector<int> rec((size_t)n * w), orig((size_t)n);
    cudaStream_t st = ctx->stream;
    CK(cudaMemcpyAsync(rec.data(), ctx->S.pcap, sizeof(int) * rec.size(), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(orig.data(), ctx->S.orig, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    std::vector<int64_t> slot_of((size_t)n);
    for (int64_t i = 0; i < n; ++i) slot_of[(size_t)orig[(size_t)i]] = i;
    offs[0] = 0;
    bool over = false;
    for (int64_t o = 0; o < n; ++o) {
        const int k = rec[(size_t)slot_of[(size_t)o] * w];
        over |= k > kPairCap;
        offs[o + 1] = offs[o] + std::min(k, kPairCap);
    }
    *total = offs[n];
    if (over) return fail(ctx, BMXG_ERR_CAPACITY, "a particle had more gated pairs than the capture holds");
    if (offs[n] > cap) return fail(ctx, BMXG_ERR_CAPACITY, "pair buffer too small");
    if (!idx) return BMXG_OK;
    for (int64_t o = 0; o < n; ++o) {
        const int *r = &rec[(size_t)slot_of[(size_t)o] * w];
        for (int k = 0; k < r[0]; ++k) idx[offs[o] + k] = orig[(size_t)r[1 + k]];
    }
    return BMXG_OK;
}

int bmxg_get_pairs(bmxg_ctx *ctx, int64_t *offs, int32_t *idx, int8_t *img, int64_t cap, int64_t *total)
{
    if (!ctx) return BMXG_ERR_ARG;
    (void)cudaGetLastError();  // drop a non-sticky error another library left on this thread
    if (!ctx->have_state) return fail(ctx, BMXG_ERR_STATE, "no state loaded");
    if (!offs || !total) return fail(ctx, BMXG_ERR_ARG, "offs and total are required");
    const int64_t n = ctx->n;
    offs[0] = 0;
    *total = 0;
    if (n == 0) return BMXG_OK;
    if (int rc0 = read_bins(ctx)) return rc0;
    cudaStream_t st = ctx->stream;
    const DevParams P = dev_params(ctx->prm);
    int64_t *d_offs = nullptr;
    CK(cudaMallocAsync((void **)&d_offs, sizeof(int64_t) * (n + 1), st));
    const int blk = ctx->sh_misc.block, grd = grid_for(ctx, ctx->sh_misc, n);
    ctx->launches += launch_pairs(ctx->S, P, ctx->parity, d_offs, nullptr, nullptr, 0, grd, blk, st);
    std::vector<int64_t> cnt((size_t)n);
    cudaError_t e = cudaMemcpyAsync(cnt.data(), d_offs, sizeof(int64_t) * n, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        cudaFreeAsync(d_offs, st);
        return fail(ctx, BMXG_ERR_CUDA, cudaGetErrorString(e));
    }
    for (int64_t i = 0; i < n; ++i) offs[i + 1] = offs[i] + cnt[(size_t)i];
    *total = offs[n];
    ctx->stats.n_pairs_last = offs[n];
    if (offs[n] > cap || !idx || !img) {
        cudaFreeAsync(d_offs, st);
        cudaStreamSynchronize(st);
        return (offs[n] > cap) ? fail(ctx, BMXG_ERR_CAPACITY, "pair buffer too small") : BMXG_OK;
    }
    int *d_idx = nullptr;
    int8_t *d_img = nullptr;
    const int64_t m = std::max<int64_t>(offs[n], 1);
    e = cudaMallocAsync((void **)&d_idx, sizeof(int) * m, st);
    if (e == cudaSuccess) e = cudaMallocAsync((void **)&d_img, m, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_offs, offs, sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        ctx->launches += launch_pairs(ctx->S, P, ctx->parity, d_offs, d_idx, d_img, 1, grd, blk, st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(idx, d_idx, sizeof(int) * offs[n], cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(img, d_img, offs[n], cudaMemcpyDeviceToHost, st);
    if (d_idx) cudaFreeAsync(d_idx, st);
    if (d_img) cudaFreeAsync(d_img, st);
    cudaFreeAsync(d_offs, st);
    cudaError_t e2 = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess) return fail(ctx, BMXG_ERR_CUDA, cudaGetErrorString(e));
    return BMXG_OK;
}

int bmxg_particle_exchange(bmxg_ctx *ctx, const double *vol, double *conc, double dt, const double *xpar,
                           int32_t where)
{
    if (!ctx) return BMXG_ERR_ARG;
    ctx->vel64_zero = false;  // (its kernels may write the FP64 velocity planes)
    (void)cudaGetLastError();  // drop a non-sticky error another library left on this thread
    if (!ctx->have_state) return fail(ctx, BMXG_ERR_STATE, "no state loaded");
    if (!vol || !conc || !xpar || !std::isfinite(dt)) return fail(ctx, BMXG_ERR_ARG, "vol, conc, xpar and a finite dt are required");
    if (where != BMXG_HOST && where != BMXG_DEVICE) return fail(ctx, BMXG_ERR_ARG, "bad `where`");
    const int64_t n = ctx->n;
    if (n == 0 || !ctx->S.has_rods) return BMXG_OK;  // only FUNGI segments exchange
    if (int rc0 = read_bins(ctx)) return rc0;
    cudaStream_t st = ctx->stream;
    const cudaMemcpyKind in = (where == BMXG_HOST) ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
    const cudaMemcpyKind back = (where == BMXG_HOST) ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
    double *buf = nullptr;  // caller-order staging (3n), slot-order vol (n), conc (3n), out (3n)
    CK(cudaMallocAsync((void **)&buf, sizeof(double) * 10 * n, st));
    double *stage = buf, *svol = buf + 3 * n, *sc = buf + 4 * n, *so = buf + 7 * n;
    const int blk = ctx->sh_misc.block, grd = grid_for(ctx, ctx->sh_misc, n);
    cudaError_t e = cudaMemcpyAsync(stage, vol, sizeof(double) * n, in, st);
    int launched = 0;
    if (e == cudaSuccess) {
        launched += launch_gather_d(svol, stage, ctx->S.orig, (int)n, grd, blk, st);
        e = cudaMemcpyAsync(stage, conc, sizeof(double) * 3 * n, in, st);
    }
    if (e == cudaSuccess) {
        for (int k = 0; k < 3; ++k)
            launched += launch_gather_d(sc + (size_t)k * n, stage + (size_t)k * n, ctx->S.orig, (int)n, grd, blk, st);
        launched += launch_exchange(ctx->S, dev_params(ctx->prm), ctx->parity, svol, sc, so, dt, xpar, grd, blk, st);
        for (int k = 0; k < 3; ++k)
            launched += launch_scatter_d(stage + (size_t)k * n, so + (size_t)k * n, ctx->S.orig, (int)n, grd, blk, st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(conc, stage, sizeof(double) * 3 * n, back, st);
    cudaFreeAsync(buf, st);
    const cudaError_t e2 = cudaStreamSynchronize(st);
    ctx->launches += launched;
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess) return fail(ctx, BMXG_ERR_CUDA, std::string("particle exchange: ") + cudaGetErrorString(e));
    return BMXG_OK;
}

int bmxg_set_list_mode(bmxg_ctx *ctx, int32_t mode)
{
    if (!ctx) return BMXG_ERR_ARG;
    if (mode != 0 && mode != 1) return fail(ctx, BMXG_ERR_ARG, "list mode must be 0 or 1");
    if (ctx->list_mode != mode) {
        ctx->list_mode = mode;
        list64_end(ctx);
        ctx->list_valid = false;
        drop_graphs(ctx);
    }
    return BMXG_OK;
}

int bmxg_set_scratch_limit(bmxg_ctx *ctx, int64_t bytes)
{
    if (!ctx) return BMXG_ERR_ARG;
    ctx->scratch_limit = bytes < 0 ? -1 : bytes;
    ctx->list_room = true;  // (refused ones are asked for again)
    ctx->rod_walk = false;
    return BMXG_OK;
}

int bmxg_init_bonds(bmxg_ctx *ctx, double rlim, int64_t *added, int64_t *overflow)
{
    if (!ctx) return BMXG_ERR_ARG;
    ctx->vel64_zero = false;  // (its kernels may write the FP64 velocity planes)
    (void)cudaGetLastError();  // drop a non-sticky error another library left on this thread
    if (added) *added = 0;
    if (overflow) *overflow = 0;
    if (!ctx->have_state) return fail(ctx, BMXG_ERR_STATE, "no state loaded");
    if (!(rlim > 0.0)) rlim = 1.0e-7;
    if (ctx->n == 0 || !ctx->S.has_rods) return BMXG_OK;
    if (int rc0 = read_bins(ctx)) return rc0;
    cudaStream_t st = ctx->stream;
    const DevParams P = dev_params(ctx->prm);
    unsigned long long *d_cnt = nullptr;
    CK(cudaMallocAsync((void **)&d_cnt, 2 * sizeof(unsigned long long), st));
    unsigned long long h_cnt[2] = {0, 0};
    cudaError_t e = cudaMemsetAsync(d_cnt, 0, 2 * sizeof(unsigned long long), st);
    if (e == cudaSuccess) {
        const int blk = ctx->sh_misc.block, grd = grid_for(ctx, ctx->sh_misc, ctx->n);
        ctx->launches += launch_init_bonds(ctx->S, P, ctx->parity, rlim, d_cnt, grd, blk, st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h_cnt, d_cnt, sizeof(h_cnt), cudaMemcpyDeviceToHost, st);
    cudaFreeAsync(d_cnt, st);
    cudaError_t e2 = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess) return fail(ctx, BMXG_ERR_CUDA, cudaGetErrorString(e));
    if (added) *added = (int64_t)h_cnt[0];
    if (overflow) *overflow = (int64_t)h_cnt[1];
    if (h_cnt[1]) return fail(ctx, BMXG_ERR_CAPACITY, "a segment end met more bonds than its four table slots");
    return BMXG_OK;
}

// The kernels that the cached shapes were timed on: entries of another set (before it
// was in the key, of kernels with one thread per slot alone) are timed again.
static constexpr int kTuneSet = 2;

int bmxg_autotune(bmxg_ctx *ctx, const char *cache_path)
{
    if (!ctx) return BMXG_ERR_ARG;
    ctx->vel64_zero = false;  // (its kernels may write the FP64 velocity planes)
    (void)cudaGetLastError();  // drop a non-sticky error another library left on this thread
    if (!ctx->have_state) return fail(ctx, BMXG_ERR_STATE, "no state loaded");
    if (ctx->n == 0 || ctx->S.has_rods) return BMXG_OK;
    if (int rc0 = read_bins(ctx)) return rc0;
    ctx->list_valid = false;  // the sweep writes the other buffer
    const int64_t n = ctx->n;
    char devname[256] = {0};
    {
        cudaDeviceProp prop;
        CK(cudaGetDeviceProperties(&prop, ctx->device));
        std::snprintf(devname, sizeof(devname), "%s", prop.name);
    }
    // the colony-size histogram (count per power-of-two size class) keys the
    // cache with the device and the particle count
    std::string hist;
    {
        int cls[64] = {0};
        for (int c = 0; c < ctx->ncol; ++c) {
            const int64_t m = ctx->offsets[c + 1] - ctx->offsets[c];
            int k = 0;
            while (k < 62 && (1LL << k) <= m) ++k;
            ++cls[k];
        }
        for (int k = 0; k < 64; ++k)
            if (cls[k]) hist += std::to_string(k) + ":" + std::to_string(cls[k]) + ",";
    }
    auto cache_read = [&]() {
        std::string txt;
        if (!cache_path) return txt;
        FILE *f = std::fopen(cache_path, "r");
        if (!f) return txt;
        char buf[4096];
        size_t r;
        while ((r = std::fread(buf, 1, sizeof(buf), f)) > 0) txt.append(buf, r);
        std::fclose(f);
        return txt;
    };
    auto cache_add = [&](const char *entry) {
        if (!cache_path) return;
        std::string txt = cache_read();
        const size_t close = txt.rfind('}');
        if (close == std::string::npos || txt.find('"') == std::string::npos)
            txt = std::string("{\n  ") + entry + "\n}\n";
        else
            txt = txt.substr(0, close) + ",\n  " + entry + "\n}\n";
        FILE *f = std::fopen(cache_path, "w");
        if (f) {
            std::fwrite(txt.data(), 1, txt.size(), f);
            std::fclose(f);
        }
    };
    // time `reps` launches after `warm` untimed ones (ms for the reps)
    auto timeit = [&](int warm, int reps, const std::function<int()> &launch, float *ms) -> int {
        for (int w = 0; w < warm; ++w) ctx->launches += launch();
        CK(cudaEventRecord(ctx->ev0, ctx->stream));
        for (int r = 0; r < reps; ++r) ctx->launches += launch();
        CK(cudaEventRecord(ctx->ev1, ctx->stream));
        CK(cudaEventSynchronize(ctx->ev1));
        CK(cudaGetLastError());
        CK(cudaEventElapsedTime(ms, ctx->ev0, ctx->ev1));
        return BMXG_OK;
    };
    char key[768];
    char entry[1024];
    const DevState &S = ctx->S;
    const DevParams P = dev_params(ctx->prm);
    // the per-step stencil kernels of both forms
    for (int prec = 0; prec < 2; ++prec) {
        std::snprintf(key, sizeof(key), "\"%s|sphere %d|%d|n=%lld|ncol=%d|h=%s\"", devname, kTuneSet, prec,
                      (long long)n, ctx->ncol, hist.c_str());
        {
            const std::string txt = cache_read();
            const size_t pos = txt.find(key);
            int bb = 0, gg = 0;
            if (pos != std::string::npos &&
                std::sscanf(txt.c_str() + pos + std::strlen(key), ": {\"block\": %d, \"grid\": %d}", &bb, &gg) == 2 &&
                bb > 0) {
                ctx->sh_sphere[prec].block = bb;
                ctx->sh_sphere[prec].grid = gg;
                if (prec == 0) ctx->adj_pinned = false;
                continue;
            }
        }
        // sweep: the kernel reads buffer a and writes buffer b, so repeated
        // launches leave the state as it was except for the column counters,
        // which are cleared afterwards
        float best = 1e30f;
        Shape bs = ctx->sh_sphere[prec];
        {   // the launch rule's own choice (grid 0)
            Shape sh = ctx->sh_sphere[prec];
            sh.grid = 0;
            int sg, sb;
            stencil_shape(ctx, sh, n, &sg, &sb);
            if (int rc = timeit(2, 5, [&]() { return launch_sphere_step(S, P, 0.0, ctx->parity, prec, sg, sb,
                                                                        ctx->stream, 0); }, &best))
                return rc;
            bs = sh;
        }
        const int blocks[] = {64, 128, 256};  // k_sphere is compiled with __launch_bounds__(256)
        for (int blk : blocks) {
            for (int mult = 1; mult <= 64; mult *= 2) {  // up to one slot per thread
                Shape sh;
                sh.block = blk;
                sh.grid = ctx->nsm * mult * std::max(1, 1024 / blk);
                const int grd = grid_for(ctx, sh, n);
                float ms = 0.0f;
                if (int rc = timeit(2, 5, [&]() { return launch_sphere_step(S, P, 0.0, ctx->parity, prec, grd, blk,
                                                                            ctx->stream, 0, true); }, &ms))
                    return rc;
                if (ms < best) {
                    best = ms;
                    bs = sh;
                }
            }
        }
        CK(cudaMemsetAsync(ctx->S.colcnt, 0, sizeof(int) * std::max(ctx->S.ncols_total, 1), ctx->stream));
        CK(cudaMemsetAsync(ctx->d_cnt, 0, sizeof(DevCounters), ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        ctx->sh_sphere[prec] = bs;
        if (prec == 0) ctx->adj_pinned = false;  // (the sweep does not time the adjoint)
        std::snprintf(entry, sizeof(entry), "%s: {\"block\": %d, \"grid\": %d, \"ms_per_5\": %.4f}", key, bs.block,
                      bs.grid, best);
        cache_add(entry);
    }
    // the FP32F list path: k_list_step's block and passes per chunk,
    // k_list_build's block
    const float skin = ctx->list_mode ? list_skin(ctx) : 0.0f;
    if (skin > 0.0f) {
        std::snprintf(key, sizeof(key), "\"%s|list %d|n=%lld|ncol=%d|h=%s\"", devname, kTuneSet, (long long)n, ctx->ncol,
                      hist.c_str());
        const std::string txt = cache_read();
        const size_t pos = txt.find(key);
        int sb = 0, sp = 0, bb = 0, pe = 0;
        if (pos != std::string::npos &&
            std::sscanf(txt.c_str() + pos + std::strlen(key),
                        ": {\"step_block\": %d, \"step_passes\": %d, \"step_persistent\": %d, \"build_block\": %d",
                        &sb, &sp, &pe, &bb) == 4 &&
            sb > 0 && bb > 0) {
            ctx->ls_block = sb;
            ctx->ls_passes = sp;
            ctx->ls_persist = pe != 0;
            ctx->lb_block = bb;
        } else {
            // a list built on the loaded positions; then the step launches read
            // buffer a and write buffer b (dt = 0), and the build launches
            // rewrite the same list: the loaded state is untouched, and the
            // list path starts afresh at the next step (list_valid = false), any other
            // reader of the bins re-bins first
            if (int rc = ensure_list(ctx, skin, BMXG_FP32F)) return rc;
            cudaStream_t st = ctx->stream;
            if (int rc = set_list_run(ctx, 1)) return rc;  // (the timed launches repeat that step)
            const int mblk = ctx->sh_misc.block, mgrd = grid_for(ctx, ctx->sh_misc, n);
            LAUNCH(launch_list_decide(S, 0, kDecideBuild, st));
            ctx->launches += launch_list_rebuild(S, P, ctx->cell_scratch, mgrd, mblk, ctx->lb_block, st);
            float best = 1e30f, best_b = 1e30f;
            int best_sb = ctx->ls_block, best_sp = ctx->ls_passes, best_bb = ctx->lb_block;
            bool best_pe = ctx->ls_persist;
            for (int blk : {64, 128, 256}) {
                // one block per chunk of 1, 2 or 4 passes; or one persistent wave
                // taking chunks of 2, 4 or 8 passes from the dispenser
                for (int pe = 0; pe < 2; ++pe) {
                    for (int passes : {1, 2, 4}) {
                        const int pp = pe ? 2 * passes : passes;
                        float ms = 0.0f;
                        if (int rc = timeit(2, 5, [&]() { return launch_list_step(S, P, 0.0, ctx->nsm, blk, pp,
                                                                                    st, pe != 0); }, &ms))
                            return rc;
                        if (ms < best) {
                            best = ms;
                            best_sb = blk;
                            best_sp = pp;
                            best_pe = pe != 0;
                        }
                    }
                }
                float ms = 0.0f;
                if (int rc = timeit(1, 3, [&]() { return launch_list_build(S, P, blk, st); }, &ms)) return rc;
                if (ms < best_b) {
                    best_b = ms;
                    best_bb = blk;
                }
            }
            CK(cudaMemsetAsync(ctx->d_cnt, 0, sizeof(DevCounters), st));
            CK(cudaStreamSynchronize(st));
            ctx->ls_block = best_sb;
            ctx->ls_passes = best_sp;
            ctx->ls_persist = best_pe;
            ctx->lb_block = best_bb;
            ctx->list_valid = false;
            ctx->bins_exact = false;  // (the builds left the list's in buffer kListBins)
            std::snprintf(entry, sizeof(entry),
                          "%s: {\"step_block\": %d, \"step_passes\": %d, \"step_persistent\": %d, \"build_block\": "
                          "%d, \"step_ms_per_5\": %.4f, \"build_ms_per_3\": %.4f}",
                          key, best_sb, best_sp, best_pe ? 1 : 0, best_bb, best, best_b);
            cache_add(entry);
        }
    }
    drop_graphs(ctx);
    return BMXG_OK;
}

int bmxg_set_shapes(bmxg_ctx *ctx, const bmxg_shapes *in)
{
    if (!ctx) return BMXG_ERR_ARG;
    if (!in) return fail(ctx, BMXG_ERR_ARG, "no shapes");
    auto block_ok = [](int b) { return b >= 32 && b <= 256 && b % 32 == 0; };
    for (int k = 0; k < 2; ++k)
        if (!block_ok(in->sphere_block[k]) || in->sphere_grid[k] < 0)
            return fail(ctx, BMXG_ERR_ARG, "sphere block: a multiple of 32 up to 256; grid >= 0");
    if (!block_ok(in->list_step_block) || !block_ok(in->list_build_block) || in->list_step_passes < 0 ||
        in->list_step_passes > 64)
        return fail(ctx, BMXG_ERR_ARG, "list blocks: a multiple of 32 up to 256; passes 0..64");
    // (a tuned FP64 shape handed back as it is stays one)
    if (in->sphere_block[0] != ctx->sh_sphere[0].block || in->sphere_grid[0] != ctx->sh_sphere[0].grid)
        ctx->adj_pinned = in->sphere_grid[0] > 0;
    for (int k = 0; k < 2; ++k) {
        ctx->sh_sphere[k].block = in->sphere_block[k];
        ctx->sh_sphere[k].grid = in->sphere_grid[k];
    }
    ctx->ls_block = in->list_step_block;
    ctx->ls_passes = in->list_step_passes;
    ctx->ls_persist = in->list_step_persistent != 0;
    ctx->lb_block = in->list_build_block;
    drop_graphs(ctx);
    return BMXG_OK;
}

int bmxg_get_shapes(const bmxg_ctx *ctx, bmxg_shapes *out)
{
    if (!ctx || !out) return BMXG_ERR_ARG;
    std::memset(out, 0, sizeof(*out));
    for (int k = 0; k < 2; ++k) {
        out->sphere_block[k] = ctx->sh_sphere[k].block;
        out->sphere_grid[k] = ctx->sh_sphere[k].grid;
    }
    out->list_step_block = ctx->ls_block;
    out->list_step_passes = ctx->ls_passes;
    out->list_build_block = ctx->lb_block;
    out->list_step_persistent = ctx->ls_persist ? 1 : 0;
    return BMXG_OK;
}

}  // extern "C"

// ---- differentiation form ----------------------------------------------------
extern "C" {

int bmxg_set_ext(bmxg_ctx *ctx, const bmxg_ext *ext)
{
    if (!ctx) return BMXG_ERR_ARG;
    if (!ext || !std::isfinite(ext->damping) || !std::isfinite(ext->mu) || ext->damping < 0.0 || ext->mu < 0.0)
        return fail(ctx, BMXG_ERR_ARG, "damping and mu must be finite and >= 0");
    if (!ctx->have_state) return fail(ctx, BMXG_ERR_STATE, "load the state before its extension parameters");
    (void)cudaGetLastError();
    ctx->ext_gamma = ext->damping;
    ctx->ext_mu = ext->mu;
    const int64_t n = ctx->n;
    if (ext->adhesion && n > 0) {
        if (!ctx->adh_buf) {
            int rc = dalloc(ctx, &ctx->adh_buf, n);
            if (rc) return rc;
        }
        ctx->d_adh = ctx->adh_buf;
        cudaStream_t st = ctx->stream;
        CK(cudaMemcpyAsync(ctx->ud, ext->adhesion, sizeof(double) * n, cudaMemcpyHostToDevice, st));
        LAUNCH(launch_gather_d(ctx->d_adh, ctx->ud, ctx->S.orig, (int)n, grid_for(ctx, ctx->sh_misc, n),
                               ctx->sh_misc.block, st));
        CK(cudaStreamSynchronize(st));
    } else {
        ctx->d_adh = nullptr;  // buffer (if any) stays allocated until the state is freed
    }
    ctx->traj_T = -1;
    return BMXG_OK;
}

}  // extern "C"

namespace {

// At least `count` values in buffer k.
template <class T>
int adj_buf(bmxg_ctx *ctx, int k, T **p, size_t count)
{
    AdjBuf &b = ctx->adj[k];
    const size_t need = std::max<size_t>(count, 1) * sizeof(T);
    if (b.bytes < need) {
        free_adj_buf(b);
        CK(cudaMalloc(&b.p, need));
        b.bytes = need;
    }
    *p = static_cast<T *>(b.p);
    return BMXG_OK;
}

// One state of a segment's recomputation: what a step reads of buffer a, so
// that the reverse sweep finds each step's positions binned and sorted as the
// recomputation left them.
struct Trail {
    size_t stride, o_pos, o_rel, o_srel, o_int, o_start;
    char *base = nullptr;
    size_t n;
    Trail(size_t n_, size_t ncols) : n(n_)
    {
        size_t at = 0;
        auto carve = [&](size_t bytes) {
            const size_t o = at;
            at += (bytes + 255) / 256 * 256;
            return o;
        };
        o_pos = carve(3 * sizeof(double) * n);
        o_rel = carve(sizeof(float4) * n);
        o_srel = carve(sizeof(float4) * n);
        o_int = carve(5 * sizeof(int) * n);
        o_start = carve(sizeof(int) * (ncols + 1));
        stride = at;
    }
    // entry k as buffer b of S
    void put(DevState &S, int b, size_t k) const
    {
        char *q = base + k * stride;
        S.x[b] = reinterpret_cast<double *>(q + o_pos);
        S.y[b] = S.x[b] + n;
        S.z[b] = S.y[b] + n;
        S.rel[b] = reinterpret_cast<float4 *>(q + o_rel);
        S.srel[b] = reinterpret_cast<float4 *>(q + o_srel);
        S.col[b] = reinterpret_cast<int *>(q + o_int);
        S.iz[b] = S.col[b] + n;
        S.perm[b] = S.iz[b] + n;
        S.siz[b] = S.perm[b] + n;
        S.rank[b] = S.siz[b] + n;
        S.colstart[b] = reinterpret_cast<int *>(q + o_start);
    }
};

DiffParams diff_params(const bmxg_ctx *ctx)
{
    return DiffParams{ctx->ext_gamma, ctx->ext_mu, ctx->d_adh};
}

// copy the positions of buffer b into 3 planes at dst (slot order)
int save_pos(bmxg_ctx *ctx, int b, double *dst)
{
    const size_t bytes = sizeof(double) * ctx->n;
    CK(cudaMemcpyAsync(dst, ctx->S.x[b], bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    CK(cudaMemcpyAsync(dst + ctx->n, ctx->S.y[b], bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    CK(cudaMemcpyAsync(dst + 2 * ctx->n, ctx->S.z[b], bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    return BMXG_OK;
}

// load 3 position planes into buffer 0 and rebuild its bins and column lists
int load_pos(bmxg_ctx *ctx, const double *src)
{
    const size_t bytes = sizeof(double) * ctx->n;
    const DevState &S = ctx->S;
    CK(cudaMemcpyAsync(S.x[0], src, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    CK(cudaMemcpyAsync(S.y[0], src + ctx->n, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    CK(cudaMemcpyAsync(S.z[0], src + 2 * ctx->n, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    const int mblk = ctx->sh_misc.block, mgrd = grid_for(ctx, ctx->sh_misc, ctx->n);
    LAUNCH(launch_bin(S, 0, mgrd, mblk, ctx->stream));
    LAUNCH(launch_rebuild(S, 0, ctx->scan_scratch, mgrd, mblk, ctx->stream));
    ctx->parity = 0;
    return BMXG_OK;
}

int dfwd_step(bmxg_ctx *ctx, const DevState &S, int a, double dt)
{
    const int mblk = ctx->sh_misc.block, mgrd = grid_for(ctx, ctx->sh_misc, ctx->n);
    const Shape &sh = ctx->sh_sphere[0];
    int sg, sb;
    stencil_shape(ctx, sh, ctx->n, &sg, &sb);
    LAUNCH(launch_dfwd(S, dev_params(ctx->prm), diff_params(ctx), dt, a, sg, sb, ctx->stream, ctx->adj_pinned));
    LAUNCH(launch_rebuild(S, a ^ 1, ctx->scan_scratch, mgrd, mblk, ctx->stream));
    return BMXG_OK;
}

}  // namespace

extern "C" {

int bmxg_forward(bmxg_ctx *ctx, double dt, int32_t nsteps, int32_t ckpt_every)
{
    if (!ctx) return BMXG_ERR_ARG;
    ctx->vel64_zero = false;  // (its kernels may write the FP64 velocity planes)
    if (!ctx->have_state) return fail(ctx, BMXG_ERR_STATE, "no state loaded");
    if (ctx->S.has_rods) return fail(ctx, BMXG_ERR_UNSUPPORTED, "the differentiation form covers spheres");
    if (nsteps < 0 || ckpt_every < 1 || !std::isfinite(dt)) return fail(ctx, BMXG_ERR_ARG, "bad dt, nsteps or ckpt_every");
    (void)cudaGetLastError();
    if (int rc0 = read_bins(ctx)) return rc0;
    ctx->list_valid = false;
    const int64_t n = ctx->n;
    free_adjoint(ctx);
    if (n == 0) {
        ctx->traj_T = nsteps;
        ctx->traj_k = ckpt_every;
        ctx->traj_dt = dt;
        return BMXG_OK;
    }
    const int nseg = (nsteps + ckpt_every - 1) / ckpt_every;
    int rc;
    double *ckpt = nullptr, *xT = nullptr;
    if ((rc = adj_buf(ctx, kAdjCkpt, &ckpt, (size_t)(nseg + 1) * 3 * n))) return rc;
    if ((rc = adj_buf(ctx, kAdjEnd, &xT, (size_t)3 * n))) return rc;
    const double subdt = dt / 1.0;
    CK(cudaEventRecord(ctx->ev0, ctx->stream));
    for (int t = 0; t < nsteps; ++t) {
        if (t % ckpt_every == 0 && (rc = save_pos(ctx, ctx->parity, ckpt + (size_t)(t / ckpt_every) * 3 * n)))
            return rc;
        if ((rc = dfwd_step(ctx, ctx->S, ctx->parity, subdt))) return rc;
        ctx->parity ^= 1;
    }
    if ((rc = save_pos(ctx, ctx->parity, xT))) return rc;
    CK(cudaEventRecord(ctx->ev1, ctx->stream));
    CK(cudaMemcpyAsync(ctx->h_cnt, ctx->d_cnt, sizeof(DevCounters), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    ctx->stats.last_step_ms = ms;
    ctx->stepped = true;
    ctx->traj_T = nsteps;
    ctx->traj_k = ckpt_every;
    ctx->traj_dt = subdt;
    ctx->vel32 = false;
    ctx->stats.n_kernel_launches = ctx->launches;
    if (ctx->h_cnt->bad_index) return fail(ctx, BMXG_ERR_STATE, "internal: inconsistent bin counts");
    if (ctx->h_cnt->nonfinite) return fail(ctx, BMXG_ERR_NONFINITE, "a step produced a non-finite position");
    return BMXG_OK;
}

int bmxg_backward(bmxg_ctx *ctx, const double *dL_dx, double *dL_dx0, double *dL_dparams, double *dL_dadhesion)
{
    if (!ctx) return BMXG_ERR_ARG;
    ctx->vel64_zero = false;  // (its kernels may write the FP64 velocity planes)
    if (ctx->traj_T < 0) return fail(ctx, BMXG_ERR_STATE, "bmxg_forward must run first");
    if (!dL_dx) return fail(ctx, BMXG_ERR_ARG, "dL_dx is required");
    (void)cudaGetLastError();
    const int64_t n = ctx->n;
    const int T = ctx->traj_T, K = ctx->traj_k;
    if (n == 0) {
        if (dL_dparams) dL_dparams[0] = dL_dparams[1] = dL_dparams[2] = 0.0;
        return BMXG_OK;
    }
    cudaStream_t st = ctx->stream;
    const DevState &S = ctx->S;
    int rc;
    ctx->list_valid = false;  // the recomputation rewrites buffer 0
    const size_t n3 = (size_t)3 * n;
    double *ckpt = nullptr, *xT = nullptr, *lam[2] = {nullptr, nullptr}, *gacc = nullptr, *gout = nullptr;
    if ((rc = adj_buf(ctx, kAdjCkpt, &ckpt, 0))) return rc;  // (the forward's)
    if ((rc = adj_buf(ctx, kAdjEnd, &xT, 0))) return rc;
    if ((rc = adj_buf(ctx, kAdjLam0, &lam[0], n3))) return rc;
    if ((rc = adj_buf(ctx, kAdjLam1, &lam[1], n3))) return rc;
    if ((rc = adj_buf(ctx, kAdjAcc, &gacc, n3 + n))) return rc;
    if ((rc = adj_buf(ctx, kAdjOut, &gout, kReduceOut))) return rc;
    double *gadh = gacc + n3;
    if ((rc = ensure_io(ctx, sizeof(double) * n3))) return rc;
    double *io = reinterpret_cast<double *>(ctx->io_buf);
    // A segment's states, sorted, where they take at most half of the free
    // memory (100 B per slot and step): the reverse sweep then runs one kernel
    // per step.  Otherwise the positions alone are kept (24 B) and binned and
    // sorted again.
    SweepBufs give_back{ctx};
    Trail trail((size_t)n, (size_t)S.ncols_total);
    double *segbuf = nullptr;
    const int kseg = std::min(K, std::max(T, 1));
    {
        const size_t need = trail.stride * (size_t)kseg;
        if (need <= ctx->adj[kAdjTrail].bytes || room_for(ctx, need, 2)) {
            if (adj_buf(ctx, kAdjTrail, &trail.base, need)) {
                (void)cudaGetLastError();
                trail.base = nullptr;
            }
        }
        if (!trail.base && (rc = adj_buf(ctx, kAdjSeg, &segbuf, (size_t)kseg * n3))) return rc;
    }
    const int mblk = ctx->sh_misc.block, mgrd = grid_for(ctx, ctx->sh_misc, n);
    CK(cudaEventRecord(ctx->ev0, st));
    // dL/dx_T, caller order -> slot order
    CK(cudaMemcpyAsync(io, dL_dx, sizeof(double) * n3, cudaMemcpyHostToDevice, st));
    LAUNCH(launch_gather_d(lam[0], io, S.orig, (int)n, mgrd, mblk, st, 3));
    CK(cudaMemsetAsync(gacc, 0, sizeof(double) * (n3 + n), st));
    int cur = 0;
    const DevParams P = dev_params(ctx->prm);
    const DiffParams D = diff_params(ctx);
    const Shape &sh = ctx->sh_sphere[0];
    int ag, ab;
    stencil_shape(ctx, sh, n, &ag, &ab);
    auto reverse = [&](const DevState &Q, int a) -> int {
        LAUNCH(launch_dadj(Q, P, D, ctx->traj_dt, a, lam[cur], lam[cur ^ 1], gacc, gadh, ag, ab, st,
                           ctx->adj_pinned));
        cur ^= 1;
        return BMXG_OK;
    };
    const int nseg = (T + K - 1) / K;
    for (int seg = nseg - 1; seg >= 0; --seg) {
        const int c0 = seg * K, c1 = std::min(c0 + K, T);
        const double *start = ckpt + (size_t)seg * n3;
        if (trail.base) {
            // recompute the segment's states from its checkpoint, entry by entry
            DevState Q = S;
            trail.put(Q, 0, 0);
            CK(cudaMemcpyAsync(Q.x[0], start, sizeof(double) * n3, cudaMemcpyDeviceToDevice, st));
            LAUNCH(launch_bin(Q, 0, mgrd, mblk, st));
            LAUNCH(launch_rebuild(Q, 0, ctx->scan_scratch, mgrd, mblk, st));
            for (int t = c0; t + 1 < c1; ++t) {
                trail.put(Q, 0, (size_t)(t - c0));
                trail.put(Q, 1, (size_t)(t - c0 + 1));
                if ((rc = dfwd_step(ctx, Q, 0, ctx->traj_dt))) return rc;
            }
            for (int t = c1 - 1; t >= c0; --t) {
                trail.put(Q, 0, (size_t)(t - c0));
                if ((rc = reverse(Q, 0))) return rc;
            }
            continue;
        }
        if ((rc = load_pos(ctx, start))) return rc;
        for (int t = c0; t < c1; ++t) {
            if ((rc = save_pos(ctx, ctx->parity, segbuf + (size_t)(t - c0) * n3))) return rc;
            if (t + 1 < c1) {
                if ((rc = dfwd_step(ctx, S, ctx->parity, ctx->traj_dt))) return rc;
                ctx->parity ^= 1;
            }
        }
        // reverse sweep through the segment
        for (int t = c1 - 1; t >= c0; --t) {
            if ((rc = load_pos(ctx, segbuf + (size_t)(t - c0) * n3))) return rc;
            if ((rc = reverse(S, 0))) return rc;
        }
    }
    LAUNCH(launch_dreduce(gacc, (int)n, 3, gout, st));
    CK(cudaEventRecord(ctx->ev1, st));
    if (dL_dx0) {
        LAUNCH(launch_scatter_d(io, lam[cur], S.orig, (int)n, mgrd, mblk, st, 3));
        CK(cudaMemcpyAsync(dL_dx0, io, sizeof(double) * n3, cudaMemcpyDeviceToHost, st));
    }
    if (dL_dadhesion) {
        LAUNCH(launch_scatter_d(ctx->ud, gadh, S.orig, (int)n, mgrd, mblk, st));
        CK(cudaMemcpyAsync(dL_dadhesion, ctx->ud, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
    }
    double g[3] = {0.0, 0.0, 0.0};
    CK(cudaMemcpyAsync(g, gout, sizeof(g), cudaMemcpyDeviceToHost, st));
    // leave the state at the end of the trajectory, as bmxg_forward did
    if ((rc = load_pos(ctx, xT))) return rc;
    CK(cudaStreamSynchronize(st));
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    ctx->stats.last_step_ms = ms;
    ctx->stats.n_kernel_launches = ctx->launches;
    if (dL_dparams) {
        dL_dparams[0] = g[0];
        dL_dparams[1] = g[1];
        dL_dparams[2] = ctx->ext_mu > 0.0 ? g[2] : 0.0;
    }
    return BMXG_OK;
}

}  // extern "C"
