// kernels.h -- device buffers of a batch and the kernel launch wrappers.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "uegccd_internal.h"

namespace uegccd {

// The |q|^2 table's form in the ladders and the rings, and of the records both look it up with: 16
// copies in shared memory and |n|^2 carried in a record's fourth byte.
inline bool table16(int q2max, int n2max) { return q2max < 256 && n2max < 128; }
constexpr int kVtabSmemEntries = 1024;   // |q|^2 table entries a kernel stages in shared memory at most

// Raw device pointers of one batch (owned by the Batch object in capi.cu).
struct DevBatch {
    int nsolves = 0, nblocks = 0, ntiles = 0, nchunks = 0, nrchunks = 0, ntargets = 0;
    int max_v = 0;      // largest v_K
    // mosaics: block row and column sums, and per target the list of partials to add
    double *mpart = nullptr;
    int32_t *mt_start = nullptr, *mt_list = nullptr;
    // FP64 ladder tiles (ladder.cu): the FMA form's, then the DMMA form's, longest first
    LadderTile64 *ltiles = nullptr;
    int nltiles[2] = {0, 0};
    size_t ladder_smem[2] = {0, 0};
    int q2max = 0, n2max = 0;   // largest |q|^2 of the solves' tables, largest |n|^2
    int *vpk = nullptr;         // beside vir: the virtual's packed vector
    int2 *ppk = nullptr;        // beside pair_i / pair_j: theirs
    int4 *rowpk = nullptr;      // the same with i | j << 16 in the third word
    int max_occ = 0;    // largest NOcc
    int64_t namp = 0;
    SolveDev *solves = nullptr;
    BlockDev *blocks = nullptr;
    ChunkDev *chunks = nullptr;      // amplitude chunks
    ChunkDev *rchunks = nullptr;     // ring-intermediate chunks over (i, x, l)
    UTileDev *utiles = nullptr;      // tiles of the amplitudes i <= j (update.cu), solve after solve
    int nutiles = 0;
    int *utile_begin = nullptr;      // nsolves+1: first tile of each solve
    int2 *targets = nullptr;         // mosaic targets (solve, id)
    int16_t *pair_i = nullptr, *pair_j = nullptr, *vir = nullptr;
    int16_t *pcol = nullptr;          // beside vir: column of the partner d = K - c in the same block
    int32_t *pos = nullptr;          // dense (i,j,a) -> global packed index or -1
    int32_t *partner = nullptr;      // packed -> packed index of (i,j,b)
    AmpInfo *amps = nullptr;
    int4 *nv4 = nullptr;
    int *nvp = nullptr;              // the same vectors packed a component per byte (warp.cuh)
    double *eigen = nullptr, *vtab = nullptr;
    double *t = nullptr, *g = nullptr;
    double *jvv = nullptr, *joo = nullptr;
    // dRPA (on the first dRPA solve): k_drpa_sums' CTA list {solve, i, column range}, row and column
    // lookups, its U, S2 per (i, x) at phr0 + i*V + x - O, and Joo's terms per range; the count of
    // finished CTAs per range, then of finished ranges per solve
    int4 *drlist = nullptr;
    int ndrlist = 0, ndrranges = 0;
    DrpaSolveDev *drsolves = nullptr;
    int4 *drows = nullptr;
    int16_t *colpos = nullptr;
    double *dru = nullptr, *drs2 = nullptr, *drj = nullptr;
    int *drdone = nullptr;
    double *part_e = nullptr, *part_dt = nullptr, *part_r = nullptr;
    double *red = nullptr;           // 3 per solve: sum e, max dt, max |r|
    uint8_t *active = nullptr;       // per solve
    // particle-hole form of the ring terms
    int16_t *ph_i = nullptr, *ph_x = nullptr;   // row -> (i, x), rows grouped by Q
    int32_t *ridx_x = nullptr, *ridx_y = nullptr;  // at ph0 + row*O + k: index of t(ik, x), t(ki, x)
    RingPairDev *rpairs = nullptr;              // {Q, -Q} group pairs, by k_rings class and solve
    RingItemDev *ritems = nullptr;              // k_rings' CTAs, class by class
    RingRowDev *rrows = nullptr;                // beside ph_i, ph_x
    RingPairDev *spairs = nullptr;              // the same pairs in solve order (k_ring_stage: each
                                                // solve's amplitudes are gathered while in L2)
    // rings in the particle-hole layout (RingPairDev::xy0): xy holds the amplitudes each pair
    // multiplies, row by row (k_ring_stage gathers t into it before every ring launch); rx
    // the ring and crossed-ring G the pair forms, in the same places (k_update reads them).
    // Per (i, x) at phr0 + i*V + x - O: ph_a = the row's offset in xy/rx when (i, x) is in
    // its pair's group 1, else -1; ph_b = its column b in group 2, else -1.
    double *xy = nullptr, *rx = nullptr;
    int64_t xy_n = 0;
    int32_t *ph_a = nullptr, *ph_b = nullptr;
    int2 *rpos = nullptr;            // per amplitude i <= j, a <= b: where rx holds its and its partner's
    // mixed precision: tensor-core ladder tiles sorted by row tile (16, 32, 64)
    LadderTile *tctiles = nullptr;
    int ntc16 = 0, ntc32 = 0, ntc64 = 0;
    double *t_ref = nullptr, *g_ref = nullptr;  // refresh point of the defect correction
    int *tc_err = nullptr;
    // FP16 operands of the tensor-core ladder (allocated and built on first mixed use)
    TcTileDev *tcx = nullptr;        // beside tctiles
    WSlabDev *wslabs = nullptr;
    DTileDev *dtiles = nullptr;
    int nwslabs = 0, ndtiles = 0;
    int64_t w16_n = 0, d16_n = 0;    // halves
    int nscale = 0;
    void *w16 = nullptr, *d16 = nullptr;   // __half arrays
    float *dscale = nullptr;
    bool w16_valid = false;          // built for the current integral tables
    int nrpairs = 0;
    // ring pair classes by the rows of group 1 (kRingFrags): CTAs, shared memory, doubles a pair
    int nritems[6] = {0, 0, 0, 0, 0, 0};
    size_t ring_smem[6] = {0, 0, 0, 0, 0, 0};
    int ring_doubles[6] = {0, 0, 0, 0, 0, 0};
    int stage_threads = 128;                    // CTA size of k_ring_stage (tune_stage)
};
// FP64 ladders (ladder.cu): blocks with at most kLadderFmaRows rows i <= j take the FMA form,
// larger ones the DMMA form in tiles of at most kLadderMmaRows rows
constexpr int kLadderFmaRows = 4, kLadderMmaRows = 16;
// the FMA form's columns a tile (pairs of H included); the DMMA form's columns a pass for tiles
// of np rows
constexpr int kLadderFmaCols = 256;
constexpr int ladder_pass_cols(int np) { return np <= 8 ? 128 : 64; }
// dynamic shared memory for |q|^2 tables up to q2max, |n|^2 up to n2max and blocks of at most
// max_rows rows i <= j, launched in so many tiles; form 0 FMA, 1 DMMA
size_t ladder_smem_bytes(int q2max, int n2max, int max_rows, int form, int tiles);
void set_ladder_smem_limit(size_t bytes);
int ladder_chunk();   // virtuals per staged chunk of the DMMA form
// G of the rows i <= j: the particle-particle ladder of t (do_pp), the hole-hole one (do_hh); the
// DMMA form on st_mma.  Returns the launches.
int launch_ladder(const DevBatch &d, const double *t, int do_pp, int do_hh, double *g, cudaStream_t st,
                  cudaStream_t st_mma);
// Rings (rings.cu): pair classes by the fragments of eight rows that hold group 1
constexpr int kRingClasses = 6;
constexpr int kRingFrags[kRingClasses] = {1, 2, 3, 4, 6, 8};
int ring_class(int n1);             // -1: more than 64 rows (NOcc <= 64 keeps every group below)
int ring_pairs_per_pass(int c);     // pairs a CTA works on at a time
int ring_cta_threads(int pairs);    // the largest CTA of the classes that work on so many pairs at a time
int ring_doubles(int c, int max_n2);
size_t ring_smem_bytes(const DevBatch &d, int c, int max_n2);
void set_rings_smem_limit(size_t bytes);
// the classes go to the ns streams in turn, the largest first
int launch_rings(const DevBatch &d, const cudaStream_t *streams, int ns);
// Launch-shape autotuner, on the batch's current amplitudes: times k_ring_stage with 64, 128 and
// 256 threads per CTA (d.stage_threads) and keeps the fastest.  Results are the same.  Not inside
// a stream capture.  Returns a cudaError_t value.
int tune_stage(DevBatch &d, cudaStream_t st);

constexpr int kDiisMax = 16;   // DIIS history capacity (k_update and k_diis_* use the same bound)

// Live per-kernel timing with CUDA events on the launching stream (off unless enabled).
enum KernelId { KID_MP2 = 0, KID_ENERGY, KID_LADDER, KID_MOSAIC_S, KID_MOSAIC_RED, KID_DRPA_SUMS,
                KID_UPDATE, KID_REDUCE, KID_RINGS, KID_LADDER_TC, KID_RING_STAGE,
                KID_TAIL, KID_EXTRAP, KID_COUNT };
struct KernelTimer {
    bool on = false;
    cudaEvent_t ev[2 * 64];
    int kid[64];
    int n = 0;
    double ms[KID_COUNT] = {};
    long long launches[KID_COUNT] = {};
    void begin(int id, cudaStream_t st)
    {
        if (!on || n >= 64) return;
        kid[n] = id;
        cudaEventRecord(ev[2 * n], st);
    }
    void end(cudaStream_t st)
    {
        if (!on || n >= 64) return;
        cudaEventRecord(ev[2 * n + 1], st);
        n++;
    }
    // call after the stream is synchronised
    void collect()
    {
        for (int k = 0; k < n; k++) {
            float t = 0.f;
            if (cudaEventElapsedTime(&t, ev[2 * k], ev[2 * k + 1]) == cudaSuccess) {
                ms[kid[k]] += t;
                launches[kid[k]]++;
            } else {
                cudaGetLastError();  // a missing sample is not an error of the solve
            }
        }
        n = 0;
    }
};
extern const char *kKernelNames[KID_COUNT];

// Per-solve iteration state kept on the device (see k_tail).
struct IterState {
    int niter;      // NIter of the reference (1 before the first update)
    int status;     // 0 running, 1 converged, 2 MaxIter reached, 3 non-finite
    double e, dt;   // energy and max|dT| of the latest iteration
};

// Buffers of the device-side iteration control.
struct CtlBuffers {
    IterState *state = nullptr;
    uint8_t *applied = nullptr;  // the solves the iteration in flight updated
    int *stopped = nullptr;      // solves no longer iterating
    int *done = nullptr;         // host memory (page-locked): 1 when none is
    double *Bm = nullptr, *coef = nullptr, *part = nullptr;
    double *hist_t = nullptr;   // DIIS history: updated amplitudes t' (FP64)
    float *hist_e = nullptr;    // and error vectors e = t' - t (FP32: they only enter the B-matrix dots)
    double *rec_e = nullptr, *rec_dt = nullptr;
    int max_rec = 0;
};

struct TermFlags {
    int do_driver = 1, do_mosaic = 1, do_ladder = 1, do_pp = 1, do_hh = 1, do_ring = 1, do_xring = 1;
    int drpa = 0;
    int mixed = 0;  // particle-particle ladder on the tensor cores (defect correction on t - t_ref)
};

void launch_mp2(const DevBatch &d, cudaStream_t st);
void launch_reduce(const DevBatch &d, cudaStream_t st);
void launch_energy(const DevBatch &d, int kind, double csosex, cudaStream_t st);
// virtuals a CTA of k_drpa_sums takes at most
constexpr int kDrpaCols = 1024;
// d.t <- T2aaaa of d.t (t(ij,a) - t(ij,b))
void launch_to_aaaa(const DevBatch &d, cudaStream_t st);
// drows and colpos (pre-set to -1) of the dRPA sums from the blocks
void launch_drpa_tables(const DevBatch &d, cudaStream_t st);
// Side streams for the independent terms of a residual (nullptr: all on one stream).
constexpr int kSideStreams = 5;
struct Fork {
    cudaStream_t s[kSideStreams] = {};   // rings, mosaics, DMMA ladders, two more for the ring classes
    bool terms = false;                  // the terms beside each other, not the ring classes only
    cudaEvent_t start = nullptr, staged = nullptr, done[kSideStreams] = {};
};
// Residual of the selected terms for d.t; mode 0 also updates d.t (with DIIS: the history).
// fork: the ring classes and, with fork->terms, the terms run beside each other.  Returns launches.
struct CtlBuffers;
// diis/ndiis (mode 0 only): fuse the Pulay DIIS push into the update kernel
int launch_residual(const DevBatch &d, const TermFlags &f, int mode, double *g_out, cudaStream_t st,
                    KernelTimer *kt = nullptr, const CtlBuffers *diis = nullptr, int ndiis = 0,
                    const Fork *fork = nullptr);
void launch_pack(const DevBatch &d, int s, int namp, const double *dense, cudaStream_t st);
void launch_unpack_all(const DevBatch &d, const int64_t *dense_off, const double *t, double *out, cudaStream_t st);
// Structure-factor sums of solve `solve` from d.t: groups = its particle-hole groups
// {first row, rows}; grid = 5 arrays of (2S+1)^3 (SfSum, SfDSum, SfXSum, contributions,
// 1 where the reference's last contribution is a core pair), column-major from -S,
// zeroed by the caller; *err = 1 if a transfer falls outside.
void launch_sf(const DevBatch &d, const int2 *groups, int ngroups, int solve, int S, double *grid, int *err,
               cudaStream_t st);
// pos (pre-set to -1), amps, partner from the block structure; the particle-hole
// tables ph_a, ph_b (pre-set to -1) from the ring pairs; the ring gather indices
void launch_block_tables(const DevBatch &d, cudaStream_t st);
// rrows of the n ph rows (row0: each solve's first)
void launch_ring_rows(const DevBatch &d, int n, const int *row0, cudaStream_t st);
// mt_start / mt_list of the mosaic sums from the blocks (tbase: each solve's first target;
// lbase: its first list entry; smem: (max V + O) ints)
void launch_mosaic_targets(const DevBatch &d, const int *tbase, const int64_t *lbase, size_t smem, cudaStream_t st);
// Mixed precision: FP16 tcgen05 ladder of t - t_ref added to g (plus g_ref); writes the
// scaled FP16 d tiles first (d.w16 must be built).  Returns the launches.
int launch_ladder_tc(const DevBatch &d, const double *t_ref, const double *g_ref, int *err, cudaStream_t st);
// The static FP16 Coulomb slabs of the tensor-core ladder, from the current |q|^2 tables
void launch_w16_build(const DevBatch &d, cudaStream_t st);
// Refresh point: t_ref <- t and g_ref <- FP64 particle-particle ladder of t_ref.  Returns the launches.
int launch_refresh(const DevBatch &d, cudaStream_t st);
// Device-side iteration control
void launch_tail(const DevBatch &d, const CtlBuffers &c, double tol, int max_iter, int ndiis, int init,
                 cudaStream_t st);
// The element-wise kernels (update.cu): G, residual and update of the amplitudes i <= j, and the
// DIIS extrapolation; update_tiles hands (c0, nc, r0, nr) of each tile of a block to emit.
void launch_update(const DevBatch &d, const TermFlags &f, int mode, double *g_out, const CtlBuffers *diis, int ndiis,
                   cudaStream_t st);
void launch_extrap(const DevBatch &d, const CtlBuffers &c, int ndiis, cudaStream_t st);
void update_tiles(int rows, int v, void (*emit)(void *, int, int, int, int), void *to);
int launch_iteration(const DevBatch &d, const CtlBuffers &c, const TermFlags &f, double tol, int max_iter,
                     int ndiis, cudaStream_t st, KernelTimer *kt, const Fork *fork = nullptr);
void launch_unpack(const DevBatch &d, int s, int namp, const double *t, double *ab, double *ba, double *aa,
                   cudaStream_t st);

// Makes `dev` the calling thread's current CUDA device for the scope's lifetime and puts the
// previous one back at its end.  Every object of the library (batch, context, DIIS history)
// records the device it was created on, and every call on it runs under one of these, so a
// host thread whose current device differs (a fresh thread starts on device 0) still works on
// the object's own device.  rc is the cudaSetDevice status.
struct DeviceScope {
    int prev = -1, dev = -1;
    cudaError_t rc = cudaSuccess;
    explicit DeviceScope(int d) : dev(d)
    {
        if (d < 0) return;
        rc = cudaGetDevice(&prev);
        if (rc == cudaSuccess && prev != d) rc = cudaSetDevice(d);
        else if (rc == cudaSuccess) prev = -1;   // already current: nothing to restore
    }
    ~DeviceScope()
    {
        if (prev >= 0 && prev != dev) cudaSetDevice(prev);
    }
    DeviceScope(const DeviceScope &) = delete;
    DeviceScope &operator=(const DeviceScope &) = delete;
};

// The current device's index, or 0 when the query fails (for per-device caches).
inline int current_device()
{
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess) d = 0;
    return d;
}
constexpr int kMaxDevices = 64;

}  // namespace uegccd
