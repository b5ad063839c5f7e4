// bmxg_kernels.cuh -- device state of a context and the host launchers of
// every kernel (internal to libbmxg; the public surface is include/bmxg.h).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "bmxg_dev.cuh"

namespace bmxg {

__host__ __device__ __forceinline__ double4_32a make_trig(double ct, double st, double cp, double sp)
{
    double4_32a t;
    t.x = ct;
    t.y = st;
    t.z = cp;
    t.w = sp;
    return t;
}

// Control block of the FP32F neighbour list with a skin (k_list.cu).  The
// list stays valid while no pair's separation has changed by the skin since
// it was built; acc bounds that change from above.
struct ListCtl {
    // per component, the smallest and largest position increment of the last
    // step over all slots (order-preserving integer keys of the floats); the
    // change of any pair's separation since the build is bounded per
    // component by the sum over steps of (largest - smallest)
    unsigned inc_min[3], inc_max[3];
    float range[3];        // those sums since the last build
    float acc;             // |range|: the bound on any pair's separation change
    float skin;            // list skin (cm)
    float eps_step;        // FP32 rounding of one position update, added per step
    int age;               // steps since the last build
    int max_age;           // rebuild at least this often (bounds FP32 offset drift)
    int force;             // rebuild at the next step (the state changed)
    int rebuild;           // this step's decision (read by the gated kernels)
    int need;              // a build is due; set where none can run, the steps stall until one can
    int left, par;         // steps left in the call and the buffer the next one reads (set by the host)
    int whole;             // the steps take no overflowed list (FP64 form)
    int bail;              // FP64 list steps: a slot left the range the list covers; no step runs any more
    int builds;            // builds decided so far
    unsigned long long body_runs;  // builds actually run (counted by the first build kernel)
    unsigned long long overflow;   // slots whose list exceeded the capacity (last build)
    // the persistent list step's chunk dispenser: the next chunk to hand out
    // and the blocks that found none left; the last of them resets both
    unsigned next_chunk, done_blocks;
    // Whether the step that follows runs (there are steps left, no build is due), and the
    // buffer it reads.  In a line of their own: every block of a step begins by reading
    // them and ends with an atomic on each of inc_min and inc_max, and the reads waited
    // behind those atomics where the line was the same.  1.1 million slots, calls of 1 / 12
    // FP32F steps 63.7 / 703 -> 55.2 / 611 us (56.5 / 652 with the buffer a kernel argument),
    // 1.6 million 77.9 / 948 -> 64.6 / 824, 500 000 51.0 / 407 -> 42.1 / 369.
    alignas(256) int active;
    int cur;
};
static_assert(offsetof(ListCtl, active) / 256 != offsetof(ListCtl, inc_max) / 256 &&
                  offsetof(ListCtl, cur) / 256 != offsetof(ListCtl, inc_max) / 256,
              "what a step's blocks read first lies apart from what they update last");

constexpr int kNbrCap = 32;          // list entries per slot (more: the slot walks its stencil)
constexpr int kNbrInline = 3;        // entries held in the slot's list record beside its metadata
constexpr int kNbrShift = 31;        // entries are slots below 2^31
constexpr int kPairCap = 32;         // gated pairs per slot the step records when asked
constexpr int kListBins = 0;         // list mode keeps its frozen bins in buffer 0
constexpr int kListStepBlock = 128;  // k_list_step's default block (at most 256; autotuned)
constexpr int kListBuildBlock = 128; // k_list_build's default block (one slot per thread; at most 256)
constexpr int kSphereBlock = 64;     // per-step sphere kernels' block (one slot per thread)
constexpr int kWalkNarrow = 65536;   // tile: 32 slots per block up to here, then 128
constexpr int kLongColumn = 160;     // slots of a column above which its runs are sorted (k_bin.cu)
constexpr int kRodCap = 32;          // gated pairs per segment the rod pipelines hold (more: the
                                     // segment walks its stencil in the segment kernel)

// Lengths of the rod pipelines' queues (k_rod.cu), emptied at the end of a step.
struct RodCtl {
    int ncontact;  // pairs from the front of rwork
    int nbond;     // pairs bonded by the segment's own table, from the back of rwork
    int n64;       // FP32F: contacts that need FP64 (rq64)
};

// Device pointers of one context.  [2] arrays are ping-pong buffers indexed
// by the step parity a (read) / b = a ^ 1 (write).
struct DevState {
    int n;             // particles (slots)
    int ncol;          // colonies
    int ncols_total;   // columns over all colonies
    int nsm;           // SMs of the device (launch rules count in waves of blocks over them)
    int long_cols;     // some column is longer than kLongColumn: what its sort found last
    const DevGeom *geoms;
    const int *cbase;  // ncol + 1: first slot of each colony, then n (a compact copy for colony lookups)
    DevCounters *cnt;

    double *x[2], *y[2], *z[2];
    float4 *rel[2];    // FP32 offsets from the slot's bin corner (x, y, z) + radius (w)
    int *col[2];       // global column of the slot
    int *iz[2];        // z bin (grown-box coordinates, 1..nz)
    int *perm[2];      // slots sorted by (column, z bin, original index)
    int *colstart[2];  // ncols_total + 1 offsets into perm
    int *colcnt;       // per-column counter, zero between uses
    int *tmp;          // scatter scratch, n entries
    // column-sorted copies (optional: null skips them): srel[t] = rel[perm[t]],
    // siz[t] = iz[perm[t]], rank[perm[t]] = t; the sphere kernels walk these
    // contiguously instead of chasing perm
    float4 *srel[2];
    int *siz[2];
    int *rank[2];

    double *rad;
    int *orig;         // slot -> caller's index
    int8_t *ctype;     // cell_type

    double *vx, *vy, *vz, *wx, *wy, *wz;  // step outputs (slot order)
    float *vxf, *vyf, *vzf;               // velocity output of the FP32F sphere step

    // rod segments (null when the state holds spheres only)
    int has_rods;
    double *clen, *area, *bscale;
    double *theta[2], *phi[2];
    double4_32a *trig[2];  // (cos theta, sin theta, cos phi, sin phi)
    int *id, *cpu, *fuse_tip;
    int *tab[2];       // 13 planes: n_bnds, ids[4], cpus[4], sites[4]
    int *position, *fix_site, *fflag, *sflag, *nflag;
    int *dltd;         // 6 planes
    double *fc;        // 6 planes, force gather of the rod path
    float4 *axf[2];    // FP32 axis (nx, ny, nz) and length of each segment
    double4_32a *mob;  // per segment: mobility (d0 + db, da - db, (d0 - db) / 2, 0) of its area,
                       // length and the viscosity (k_rod_mobility, on every state or parameter load)
    // rod pipelines (null until the first rod step): the queue of gated pairs
    // (i, k: the pair's place in the segment's list order, j, code: bin offsets
    // dx, dy, dz + 1 as a base-3 number in bits 0-4, image shifts sx, sy + 1 in
    // bits 5-8, the segment's bonded site in bits 9-10), written by k_rod_book
    int4 *rwork;       // kRodCap n entries
    int *rq64;         // FP32F: entries of rwork left to FP64
    int *rcnt;         // per segment: its gated pairs (more than kRodCap: it walks)
    double *rres;      // 6 x kRodCap planes of n: each pair's f1 + f2 (0-2), f1 - f2 (3-5)
    RodCtl *rctl;

    // FP32F neighbour list with a skin (null unless the context is in list mode)
    int *nbr;          // entries kNbrInline.. kNbrCap-1, one plane of n per entry: the
                       // neighbour slot (periodic images need no code: the fixed-point
                       // difference is the minimum image)
    int4 *lrec;        // per slot: x = list length (bits 0-7, saturating at 255) and the
                       // slot's place in its group's run of xlist (bits 8-17); y, z, w =
                       // the first kNbrInline entries
    // the entries past the inline ones, compacted for the step: per group of
    // 32 consecutive slots (one warp of k_list_step) the groups' entries lie
    // together, slot by slot in list order, from xoff[group] on
    int *xcnt;         // per group: its entries past the inline ones (then scanned into xoff)
    int *xoff;
    int *xlist;
    int4 *fxh[2];      // list path positions, ping-pong with x/y/z: high 32 bits of the
                       // 64-bit fixed-point x, y, z (FxGeom) and the FP32 radius bits --
                       // what a neighbour gathers
    unsigned *fxl[2];  // the low 32 bits, three planes of n (x, y, z)
    const FxGeom *fxg; // per colony
    int *pcap;         // null, or per slot 1 + kPairCap ints: the gated pairs of the last
                       // list step (count, then neighbour slots in accumulation order)
    unsigned long long *lkey;  // sort scratch, n (the load's sort and the list build): at each
                               // column position the counting sort gave a particle, its
                               // (z bin, caller index) key
    int *cellstart;    // ncells_total + 1 offsets of the cells in the sorted copies
    int ncells_total;
    int cols_max;      // largest column count of a colony
    ListCtl *lctl;
};

// Extension parameters of the differentiation form (k_adjoint.cu).
struct DiffParams {
    double gamma;        // two-body dashpot
    double mu;           // Stokes drag of spheres (0: mobility 1)
    const double *adh;   // per-slot adhesion energy (null: zero)
};

// ---- binning / counting sort (k_bin.cu) ----------------------------------
int launch_bin(const DevState &S, int b, int grid, int block, cudaStream_t st);
// gate (may be null): the kernels return at once when *gate == 0
int launch_scan(const int *in, int *out, int n, int *scratch, cudaStream_t st, const int *gate = nullptr);
size_t scan_scratch_ints(int n);
// publish: the end of a step (the counters into last_*, cleared, and the rod
// pipeline's queue emptied)
int launch_rebuild(const DevState &S, int b, int *scan_scratch, int grid, int block, cudaStream_t st,
                   bool publish = false);

// positions, radii, cell types, bins, offsets and identity column order of a
// freshly sorted state (buffer 0), gathered from the caller-order arrays
// (v: the six velocity fields, caller order; null: zeros)
int launch_load_slots(const DevState &S, const double *ux, const double *uy, const double *uz, const double *ur,
                      const int *uct, const double *const v[6], const int *ucol, const int *uiz, const int *uperm,
                      int grid, int block, cudaStream_t st);
// The fields of rod segments in caller order (device arrays; null: the field's
// default), gathered into slot order with the segments' trig and mobility.
struct RodFields {
    const double *clen, *area, *bscale, *theta, *phi;
    const int *id, *cpu, *fuse_tip, *position, *fix_site, *fflag, *sflag, *nflag, *dltd, *n_bnds, *seg_id1, *seg_id2,
        *site;
};
int launch_load_rods(const DevState &S, const DevParams &P, const RodFields &F, const int *uperm, int grid, int block,
                     cudaStream_t st);
// The state of buffer a scattered to caller order, the fields asked for (null: not).  fx: the positions come from the list's fixed point (the FP64
// ones are written too); vel32: the velocities from the FP32F planes.
struct StoreFields {
    double *x, *y, *z, *v[6], *theta, *phi;
    int *n_bnds, *seg_id1, *seg_id2, *site, *position, *fix_site, *fflag, *sflag, *nflag, *dltd;
};
// Bytes up to which one pass scatters several fields: past it their lines leave L2 (129 MB,
// the sources' lines with them) before they are whole.
constexpr size_t kScatterPass = 76u << 20;
size_t store_bytes(const StoreFields &F, int n);
int launch_store(const DevState &S, int a, const StoreFields &F, bool fx, bool vel32, cudaStream_t st);
// AoS records (k_io.cu): bytes per record, of rdata and idata in a record
struct AosLayout {
    size_t stride, rdata, idata;
};
// The records' fields into planes in caller order: 15 of doubles (x, y, z,
// radius, c_length, theta, phi, area, bond_scale, velx .. wz), 28 of ints
// (cell_type, id, cpu, n_bnds, seg_id1[4], seg_id2[4], site[4], position,
// fuse_tip, fix_site, fuse_flag, split_flag, new_flag, dltd[6]).  Without rods
// only the fields of spheres (the first four, the velocities, cell_type).
int launch_aos_load(const unsigned char *rec, const AosLayout &L, int n, bool rods, double *d, int *i, cudaStream_t st);
// What a step writes, from buffer a into the records.
int launch_aos_store(unsigned char *rec, const AosLayout &L, const DevState &S, int a, cudaStream_t st);
// *diff |= 1 when a given field (null: not compared) differs bit for bit from
// the device state of buffer a (slot s against caller index orig[s]); chk (null: not):
// launch_check_state's out, from the same pass over r and ct
int launch_same_state(const DevState &S, int a, const double *x, const double *y, const double *z, const double *r,
                      const int *ct, unsigned long long *diff, unsigned long long *chk, int grid, int block,
                      cudaStream_t st);
// state checks before a load: out[4] = {bad cell type, any FUNGI, largest radius bits, NaN radius}
int launch_check_state(const int *ct, const double *r, int n, unsigned long long *out, int grid, int block,
                       cudaStream_t st);

// caller-order staging -> slot order (set_state) and back (get_state)
int launch_user_bin(const DevState &S, const double *ux, const double *uy, const double *uz,
                     int *ucol, int *uiz, int grid, int block, cudaStream_t st);
// the caller's particles into column order: the column offsets and uperm[slot] =
// caller index (keys in lkey)
int launch_user_sort(const DevState &S, const int *ucol, const int *uiz, int *colstart, int *scan_scratch,
                     int *uperm, int grid, int block, cudaStream_t st);
// (planes of n each)
int launch_gather_d(double *dst, const double *src, const int *perm, int n, int grid, int block, cudaStream_t st,
                    int planes = 1);
int launch_scatter_d(double *dst, const double *src, const int *orig, int n, int grid, int block, cudaStream_t st,
                     int planes = 1);
int launch_scatter_f2d(double *dst, const float *src, const int *orig, int n, int grid, int block,
                       cudaStream_t st);

// neighbour-list export (k_bin.cu): mode 0 counts per caller index, mode 1 fills
int launch_pairs(const DevState &S, const DevParams &P, int a, int64_t *cnt_or_offs, int *idx,
                  int8_t *img, int mode, int grid, int block, cudaStream_t st);

// ---- spheres (k_sphere.cu) -----------------------------------------------
// force gather + wall + update + rebin of every slot, reading buffer a and
// writing buffer b; precision BMXG_FP64 / BMXG_FP32F
// resync (FP32F only): re-derive every slot's FP32 offsets and bin from its
// FP64 position this step
int launch_sphere_step(const DevState &S, const DevParams &P, double dt, int a, int precision,
                        int grid, int block, cudaStream_t st, int resync = 1, bool pinned = false);

// ---- FP32F neighbour list with a skin (k_list.cu) --------------------------
// decide: fold the last step's displacement into the bound and decide whether
// this step rebuilds.  What follows it in the stream: kDecideStall no build (a
// step that needs one does not run, nor the ones after it), kDecideCond a
// conditional node (cond) with the build, kDecideBuild the gated build kernels.
// kDecideOne: as kDecideCond, and the call's steps are one more (a call of few steps sets
// none before it).
enum { kDecideStall = 0, kDecideCond = 1, kDecideBuild = 2, kDecideOne = 3 };
int launch_list_decide(const DevState &S, unsigned long long cond, int mode, cudaStream_t st);
// fixed-point positions of buffer a from its FP64 positions and radii (when the
// list starts on a state), and back (whenever the FP64 positions are read)
int launch_list_init(const DevState &S, int a, int grid, int block, cudaStream_t st);
int launch_list_to_fp64(const DevState &S, int a, int grid, int block, cudaStream_t st);
// axis ax (0 x, 1 y, 2 z) of it, also scattered to out in the caller's order (out[orig[i]])
int launch_list_to_fp64_axis(const DevState &S, int a, int ax, double *out, int block, cudaStream_t st);
// rebuild (gated on lctl->rebuild): bins of buffer lctl->cur's positions into the
// list bins, column lists, and the list itself
// (returns the kernels it enqueues, kListBodyKernels)
int launch_list_rebuild(const DevState &S, const DevParams &P, int *scan_scratch, int grid, int block,
                        int build_block, cudaStream_t st);
// the list build kernel alone (gated on lctl->rebuild), build_block threads per block
int launch_list_build(const DevState &S, const DevParams &P, int build_block, cudaStream_t st);
constexpr int kListBodyKernels = 12;
// force + wall + update over the list, reading buffer lctl->cur and writing the
// other, or nothing when the step is not active (grid = the SM count; passes of the block per chunk of slots, <= 0: a rule;
// persistent: one wave of blocks taking chunks from a counter, else one block
// per chunk; chained: right after the decision kernel, no build between)
// FP64 form of the path: the FP32 coordinates the steps screen with (in rel) from
// buffer a's positions; the fixed-point positions of the build (first kernel of
// the build's body); the step.
int launch_list64_begin(const DevState &S, int a, cudaStream_t st);
int launch_list64_fx(const DevState &S, cudaStream_t st);
int launch_list64_step(const DevState &S, const DevParams &P, double dt, cudaStream_t st, bool chained);
int launch_list_step(const DevState &S, const DevParams &P, double dt, int grid, int block, int passes,
                     cudaStream_t st, bool persistent = false, bool chained = false);

// ---- one tile with the caller's ghosts (k_tile.cu) -------------------------
// The level's domain and the tile: cells are the domain's (1-based bins of
// the whole-domain step) offset by lo, the tile's first cell minus one, so
// that the tile's own cells are 1..nt and the one-cell halo 0 and nt + 1.
struct TileGeom {
    double plo[3], phi[3], len[3], dx[3], dxi[3];
    float dxf[3];
    int n[3], per[3];
    int lo[3], nt[3];
    int nbh_trivial;
};
// One tile call: the caller's arrays (device memory), the workspace as a state
// of the reals then the ghosts (buffer 0: positions, radii, columns of the
// grown tile, z bins, offsets, sort), the reals' results (6 planes) and flags.
struct TileCall {
    const double *rx, *ry, *rz, *rr, *gx, *gy, *gz, *gr;
    const int *rct, *gct;
    int nreal;
    DevState S;
    double *out;              // new x, y, z and velocity, nreal each
    unsigned long long *bad;  // [3]: a real outside the tile or a ghost outside the halo; a non-sphere;
                              // a non-finite new position
};
// bin, sort, step; then, with dst, the results into the caller's arrays unless
// the input was bad (dst[0..2] positions, [3..5] velocities)
int launch_tile_step(const TileCall &C, const TileGeom &T, const DevParams &P, double dt, int *scan_scratch,
                     double *const dst[6], cudaStream_t st);

// ---- rods and mixed states (k_rod.cu) ------------------------------------
int launch_rod_mobility(const DevState &S, const DevParams &P, int grid, int block, cudaStream_t st);
// list: also queue the segments' gated pairs for the pipelines
int launch_rod_book(const DevState &S, const DevParams &P, int a, bool list, int grid, int block, cudaStream_t st);
// the pipelines after the bookkeeping: the queued pairs, then per segment its
// sums, velocity and update (launch_rod_force and launch_rod_update without the queues)
int launch_rod_pairs(const DevState &S, const DevParams &P, double dt, int a, int precision, int nsm, int n,
                     cudaStream_t st);
int launch_rod_force(const DevState &S, const DevParams &P, int a, int grid, int block, cudaStream_t st);
int launch_rod_update(const DevState &S, double dt, int a, int grid, int block, cudaStream_t st);
// one ParticleExchange substep: conc / out 3 planes (A, B, C), slot order; xpar host
int launch_exchange(const DevState &S, const DevParams &P, int a, const double *vol, const double *conc, double *out,
                    double dt, const double *xpar, int grid, int block, cudaStream_t st);
// start-up bond detection; counts[0] += bonds added, counts[1] += bonds past four
int launch_init_bonds(const DevState &S, const DevParams &P, int a, double rlim, unsigned long long *counts,
                      int grid, int block, cudaStream_t st);

// ---- differentiation form (k_adjoint.cu) ---------------------------------
int launch_dfwd(const DevState &S, const DevParams &P, const DiffParams &D, double dt, int a, int grid, int block,
                cudaStream_t st, bool pinned = false);
int launch_dadj(const DevState &S, const DevParams &P, const DiffParams &D, double dt, int a, const double *lin,
                double *lout, double *gacc, double *gadh, int grid, int block, cudaStream_t st, bool pinned = false);
// out: kReduceOut values, the planes' sums first
constexpr int kReduceBlocks = 64;
constexpr int kReduceOut = 4 + 4 * 2 * kReduceBlocks;  // (up to four planes; a sum and its remainder)
int launch_dreduce(const double *gacc, int n, int planes, double *out, cudaStream_t st);

}  // namespace bmxg
