// nb_internal.h -- internal declarations shared by the engine's translation units.
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <cstddef>
#include <cstdint>
#include <functional>
#include <string>
#include <vector>

#include "../../include/nbody_c.h"

namespace nb {

// ---------------------------------------------------------------- errors
void set_error(const std::string &msg);
nb_status fail(nb_status s, const std::string &msg);
nb_status cuda_fail(cudaError_t e, const char *what);

#define NB_CUDA_TRY(call)                                                  \
    do {                                                                   \
        cudaError_t nb_e_ = (call);                                        \
        if (nb_e_ != cudaSuccess) return ::nb::cuda_fail(nb_e_, #call);    \
    } while (0)

// Counts one kernel launch of this library and checks the launch status.
void count_launch();
#define NB_LAUNCH_CHECK()                                                  \
    do {                                                                   \
        ::nb::count_launch();                                              \
        cudaError_t nb_e_ = cudaGetLastError();                            \
        if (nb_e_ != cudaSuccess) return ::nb::cuda_fail(nb_e_, "kernel launch"); \
    } while (0)

#define NB_TRY(call)                                                       \
    do {                                                                   \
        nb_status nb_s_ = (call);                                          \
        if (nb_s_ != NB_OK) return nb_s_;                                  \
    } while (0)

// An NVTX range over a host scope: the phases of a step (sort, build, walk,
// direct sum, serving tick) appear by name in timeline profilers and can be
// selected with ncu --nvtx --nvtx-include; a few nanoseconds when no tool is
// attached.
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};

// The first failed device-side index check of a translation unit of a
// checked build (nb_check.cuh): source line, index and bound.
struct DeviceCheck {
    int failed;
    int line;
    long long index;
    long long bound;
};
using CheckReader = nb_status (*)(DeviceCheck *out, bool clear);
// Called by every checked translation unit at load time.
void register_check_reader(const char *file, CheckReader reader);

// ---------------------------------------------------------------- memory
// A device buffer that grows on demand and is freed with its owner.
struct DevBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
    nb_status reserve(size_t want);
    void release();
    template <class T> T *as() const { return static_cast<T *>(ptr); }
};

struct DeviceProps {
    int device = 0;
    int num_sms = 0;
    int max_smem_optin = 0;
};
const DeviceProps &device_props();

// A pair of events recorded around the dominant kernel of a force evaluation
// (null members: not recorded).
struct KernelTimer {
    cudaEvent_t start = nullptr, stop = nullptr;
};

// The integrator's update of a body once its acceleration is known (nb_after.cuh):
// the kernel that finishes the acceleration applies it.  Planes by component.
struct AfterForce {
    enum Kind { kNone, kKick, kKickMean, kStage, kFinish };
    Kind kind = kNone;
    double h = 0.0;                 // the update's step
    double *x[3] = {}, *v[3] = {};  // written: velocities; positions too by kStage, kFinish
    const double *a0[3] = {};       // kKickMean: a(t); kFinish: the first stage's
    const double *x0[3] = {}, *v0[3] = {};  // kStage: the step's start
    const double *kv[3] = {};       // kStage: the stage's velocity; kFinish: the last one's
    const double *k2 = nullptr, *k3 = nullptr;  // kFinish: planes x y z vx vy vz ax ay az
    size_t ps = 0;                              // and their stride
    const double *m = nullptr;      // kStage, or null: the mirror split_positions
    float4 *hi = nullptr, *lo = nullptr;        // would make of the new positions
};

// ---------------------------------------------------------------- direct sum
// Mixed FP32/double-single all-pairs kernel.  hi/lo: float4 (x, y, z, m) and
// (x_lo, y_lo, z_lo, 0) of every body.  Writes G * sum into ax/ay/az (FP64).
// after.hi, after.lo: below kMixedPairsMin other arrays than hi, lo, since one launch
// reads every body's entry and writes the new ones.
// kMixedPairsMin: smallest system summed over unordered pairs, by several launches.  An
// evaluation takes 24.8 us there and 28.9 with ordered pairs at n = 4,000, 24.7 and
// 22.7 at 3,000.
constexpr int kMixedPairsMin = 4096;
nb_status direct_mixed(const float4 *hi, const float4 *lo, int n, double G, double eps2,
                       double *ax, double *ay, double *az, DevBuf &partials,
                       cudaStream_t st, const KernelTimer *timer = nullptr,
                       const AfterForce &after = AfterForce{});

// Thresholds of the sorted near/far kernels as (gap / D)^2, D the diameter of
// a warp's i-box: a j-chunk at least D/8 away takes the plain FP32 term, one
// at least D/4 away also drops the Newton step (kFarFactor = 1/8, kVeryFar =
// 1/4).
constexpr float kFarFactor2 = 0.015625f;
constexpr float kVeryFar2 = 0.0625f;
// Pairs of the sorted single-system kernel closer than R = min(kExact D,
// kExactSpacing s) (s: the mean body spacing in the warp's box) leave its FP32
// sum and are evaluated in double-single: they carry the largest terms of a
// body's sum, whose FP32 rounding would otherwise set its error.
constexpr float kExact2 = 0.015625f;        // kExact = 1/8
constexpr float kExactSpacing2 = 0.5625f;   // kExactSpacing = 3/4

// Hilbert-sorted near/far variant of the mixed path (nb_direct_sorted.cu).
struct BHTree;
struct SortedBuffers {
    DevBuf hi, lo, partials, boxes, tiles;
    DevBuf exact;  // the left-out pairs' sums, 3 n doubles per share (sorted order)
    DevBuf far, acc;  // the far kernel's partial planes, and their sums between passes
    cudaStream_t side[2] = {};  // the exact-pair and near kernels' streams
    cudaEvent_t fork = nullptr, join[2] = {};
    BHTree *sorter = nullptr;
    // The sort order is a performance device only (near/far decisions use
    // the current chunk boxes, any order gives results within tolerance), so
    // it is recomputed every kResortEvals force evaluations and when n
    // changes -- not at every call, and not on a load (the next periodic
    // re-sort adapts it to bodies that moved or were replaced).
    const uint32_t *order = nullptr;  // sorted index -> body (sorter-owned)
    const double *centre = nullptr;   // origin of the hi/lo split (sorter-owned)
    int order_n = -1;
    int evals_since_sort = 0;
    void invalidate_order() { order_n = -1; }
    void release();
};
// Bodies are sorted along a Hilbert curve; every warp re-centres the j-chunks
// (32 bodies) on its own (compact) i-box and runs the plain FP32 pair term on
// those that lie at least an eighth of the box diameter away; near chunks keep
// the double-single one.
nb_status direct_mixed_sorted(const double *x, const double *y, const double *z,
                              const double *m, int n, double G, double eps2, double *ax,
                              double *ay, double *az, SortedBuffers &b, cudaStream_t st,
                              const KernelTimer *timer = nullptr);
// Whether an evaluation of n bodies takes the sorted variant: flags
// NB_FLAG_MIXED_SORTED / NB_FLAG_MIXED_UNSORTED decide, else n >= kSortedMinBodies.
// Per evaluation of a Plummer sphere, unsorted / sorted, in us: 8,192 bodies 46 / 143,
// 16,384 134 / 221, 24,576 291 / 323, 32,768 500 / 501, 49,152 1103 / 919.  By time alone
// the line would lie at 32,768; it lies where it did when the unsorted sum took ordered
// pairs (201 / 194 us), since from there on results promise 1e-6 of every body's force,
// which the sorted kernel alone gives.
constexpr int kSortedMinBodies = 16384;
bool direct_sorted_enabled(int n, int flags);

// FP64 all-pairs kernel.
nb_status direct_fp64(const double *x, const double *y, const double *z, const double *m,
                      int n, double G, double eps2, double *ax, double *ay, double *az,
                      DevBuf &partials, cudaStream_t st, const KernelTimer *timer = nullptr,
                      const AfterForce &after = AfterForce{});

// Builds the float4 hi/lo mirror of FP64 positions + masses.
nb_status split_positions(const double *x, const double *y, const double *z,
                          const double *m, int n, float4 *hi, float4 *lo, cudaStream_t st);

// ---------------------------------------------------------------- integrators
// hi, lo (or null): the mirror split_positions would make of the new positions.
nb_status kick_drift(int kind, int n, double dt, double *x, double *y, double *z, double *vx,
                     double *vy, double *vz, const double *ax, const double *ay,
                     const double *az, double *oax, double *oay, double *oaz,
                     cudaStream_t st, const double *m = nullptr, float4 *hi = nullptr,
                     float4 *lo = nullptr);
nb_status kick(int kind, int n, double dt, double *vx, double *vy, double *vz,
               const double *ax, const double *ay, const double *az, const double *oax,
               const double *oay, const double *oaz, cudaStream_t st);

// An AfterForce as a launch of its own, after a force evaluation that did not
// apply it.
nb_status apply_after(const AfterForce &after, int n, const double *ax, const double *ay,
                      const double *az, cudaStream_t st);

// RK4 stage kernels.  stage 2/3/4 positions/velocities from the base state.
nb_status rk4_stage(int n, double h, const double *x, const double *y, const double *z,
                    const double *vx, const double *vy, const double *vz, const double *kvx,
                    const double *kvy, const double *kvz, const double *kax,
                    const double *kay, const double *kaz, double *ox, double *oy,
                    double *oz, double *ovx, double *ovy, double *ovz, cudaStream_t st);
nb_status rk4_combine(int n, double dt, double *x, double *y, double *z, double *vx,
                      double *vy, double *vz, const double *ax, const double *ay,
                      const double *az, const double *k2, const double *k3, const double *k4,
                      cudaStream_t st);

// One integrator step over the ten FP64 planes f (x y z vx vy vz ax ay az m)
// of n bodies; `force` evaluates accelerations of given positions.
struct StepBuffers {
    double *old_acc = nullptr;  // 3 planes (velocity Verlet)
    double *rk4 = nullptr;      // 27 planes (RK4 stages K2, K3, K4: x v a each)
    size_t ps = 0;              // plane stride in doubles
};
using ForceFn = std::function<nb_status(const double *, const double *, const double *,
                                        double *, double *, double *)>;
nb_status integrate_step(int integ, int n, double dt, double *const f[10], StepBuffers &b,
                         bool &forces_valid, const ForceFn &force, cudaStream_t st);

// ---------------------------------------------------------------- diagnostics
// Packed-FMA lane operations per second of the current device (a register-only
// probe kernel, best of three timed launches).
nb_status fp32_rate(double *lane_ops_per_s);
nb_status diagnostics(const double *x, const double *y, const double *z, const double *vx,
                      const double *vy, const double *vz, const double *m, int n, double G,
                      double eps2, DevBuf &scratch, cudaStream_t st, nb_diag *out);

// ---------------------------------------------------------------- batches
constexpr int kBatchBlockBodies = 256;  // four tiles of 64
// Smallest system summed over unordered pairs; smaller ones by rows (ordered
// pairs).  On the 1024-system ensemble (n log-uniform in [32, 4096], two RK4 steps)
// a line at 512 / 1024 / 2048 / beyond every system measured 7.58 / 7.69 / 8.12 /
// 9.15 ms (one i-tile at a time; at 1024 / 2048 7.04 / 7.51 ms with four i-bodies per
// lane).  Against 64 bits neither sum is better: over 12 systems each of 600 to 2,047
// bodies, Plummer and disk, the pairs' RMS error was 0.79 to 1.02 of the rows', the largest
// of a body 1.6e-7 to 3.6e-7 and 1.9e-7 to 3.9e-7 of its terms' magnitudes.  The line lies
// at 2048 so that smaller systems, in which one close pair can carry a body's whole
// force, keep the sums and so the trajectories they have had (of 30 ensembles, the
// largest difference of a velocity after two steps was 4.4e-8 of their scale with the line
// at 1024, 2.5e-8 at 2048).
constexpr int kBatchPairsMin = 2048;
// The server's jobs run many steps and may be dense disks, in which a close pair carries
// a force of 100: the two sums of the same terms are apart by 1.4e-7 of the velocities'
// scale after four steps of 1e-3 at n = 2705 (and as close to 64 bits: RMS errors of an
// acceleration 6.4e-8 by pairs, 6.6e-8 by rows for disks of 3,000).  Up to 4095 bodies
// their work is a few percent of the direct jobs' (a burst of 16 jobs: 15.7 ms, 15.5 by
// pairs from 1024), so they keep the rows that their trajectories have had.
constexpr int kServePairsMin = 4096;
// Largest system summed over unordered pairs: the table of its items grows as n^2 (8
// million at 2^20 bodies, 100 MB); larger ones go by rows, n / 32 items.
constexpr int kBatchPairsMax = 1 << 20;
// Partial planes of a pass over an ensemble's systems (a system needs 24 B a body and
// diagonal and side, 400 B a body at 4096 bodies; 4096 systems of 32 to 4096 bodies
// 0.55 GB, one pass).
constexpr size_t kBatchPlaneBytes = (size_t)1 << 30;
// A system of a batch: bodies [first, first + n) of the batch's pool; or, of one whose
// planes do not fit a pass, the diagonals [p0, p0 + np) alone.
struct SysDesc {
    int first;
    int n;
    int blocks = 0;       // blocks of kBatchBlockBodies; 0: summed by rows
    int tile0 = 0;        // first 64-body tile of the system
    // the place of its partial planes, 3 n entries each: the first sides of its diagonals,
    // then the second (which diagonal 0 has not)
    long long part0 = 0;
    int p0 = 0, np = 0;   // diagonals of its block pairs
    long long acc0 = 0;   // not all diagonals: its sums between passes
};
// One queue item: blocks a and (a + p) mod blocks of system `sys`; p < 0: the
// 32 rows from body 32 a.
struct PairItem {
    int sys;
    int a;
    int p;
};
// The systems are summed in passes, whose partial planes take turns in one buffer: a
// pass is a range of items of the pair kernel and one of (system, block, 0) entries for
// the combine.
struct BatchPass {
    int item0 = 0, items = 0;
    int block0 = 0, blocks = 0;
    bool parts = false;  // some diagonals of one system
};
// The work of a set of systems.  In: sys, first and n of each.
struct BatchWork {
    std::vector<SysDesc> sys;      // the systems, then descriptors of parts of them
    std::vector<PairItem> blocks;  // the combine's entries, pass by pass
    std::vector<PairItem> items;   // the pair kernel's, each pass by cost, largest first
    std::vector<BatchPass> passes;
    size_t part_bytes = 0;         // of the buffer of partial planes
    int num_tiles = 0;
};
// Systems by pairs: pairs_min to kBatchPairsMax bodies, one diagonal of which fits
// plane_bytes.  A system's result depends on it, pairs_min and plane_bytes alone.
void build_batch(BatchWork &w, int pairs_min, size_t plane_bytes);
// The work on the device.
struct BatchQueue {
    DevBuf d_sys, d_blocks, d_items;
    std::vector<BatchPass> passes;
    int num_tiles = 0;
    long long num_items = 0;
    float2 *part = nullptr;
    size_t bytes() const { return d_sys.bytes + d_blocks.bytes + d_items.bytes; }
    void release();
};
// Room for w in q, whose contents then are void.
nb_status reserve_batch(BatchQueue &q, const BatchWork &w);
// Uploads w (and waits for the copies); q.part is the caller's to set.
nb_status upload_batch(BatchQueue &q, const BatchWork &w, cudaStream_t st);
// Mixed-precision forces of all systems of the queue.
nb_status batch_forces(const float4 *hi, const float4 *lo, const BatchQueue &q, double G,
                       double eps2, double *ax, double *ay, double *az, int total,
                       cudaStream_t st, const KernelTimer *timer = nullptr);

// Hilbert-sorted variant of the batched forces (nb_batch.cu): each system's
// bodies are sorted along a Hilbert curve through its own cube; tile pairs far
// apart take the plain FP32 term.
struct BatchSorted {
    BHTree *sorter = nullptr;
    DevBuf body_sys, tiles, geom, boxes;
    const uint32_t *order = nullptr;  // sorted index -> body (sorter-owned)
    int num_sys = 0, num_tiles = 0, total = 0, key_shift = 0, first_shift = 0;
    void release();
};
// Device tables for the systems of d_sys (already uploaded with tile0).
nb_status batch_sorted_setup(BatchSorted &b, const SysDesc *d_sys, int num_sys, int num_tiles,
                             int total, cudaStream_t st);
// (Re)computes the order from the positions x, y, z.
nb_status batch_sorted_sort(BatchSorted &b, const SysDesc *d_sys, const double *x,
                            const double *y, const double *z, cudaStream_t st);
// a = G sum_j ... for every body, in the order of the last sort (hi/lo are
// scratch mirrors of total entries).
nb_status batch_sorted_forces(BatchSorted &b, const double *x, const double *y, const double *z,
                              const double *m, const BatchQueue &q, double G, double eps2,
                              float4 *hi, float4 *lo, double *ax, double *ay, double *az,
                              cudaStream_t st, const KernelTimer *timer);

// ---------------------------------------------------------------- Barnes-Hut
struct BHTree;  // opaque, defined in nb_bh.cu
BHTree *bh_create();
void bh_destroy(BHTree *t);
// Whether walks that would be ordered go one warp each (the same bits): less work, for a
// GPU that other trees fill, and a longer wait for a lone one.
void bh_prefer_serial(BHTree *t, bool serial);
// The tree object for other bodies: no topology, its counters at zero; its buffers stay.
nb_status bh_restart(BHTree *t, cudaStream_t st);
// Builds the tree of (x,y,z,m) and, when ax != nullptr, walks it writing
// G * acceleration (FP64) in the original body order.  reuse > 1: the tree is
// rebuilt every `reuse` walks; the walks in between keep its topology and
// refit monopoles and cell sides to the current positions.  quad: accepted
// cells act with their quadrupole moments too.  ref_open: the walk also opens,
// of every node it opens, the child toward the body (the reference's rule).
nb_status bh_compute(BHTree *t, const double *x, const double *y, const double *z,
                     const double *m, int n, double G, double eps2, double theta,
                     int leaf_capacity, double *ax, double *ay, double *az, cudaStream_t st,
                     const KernelTimer *timer = nullptr, int reuse = 1, bool quad = false,
                     bool ref_open = false, const AfterForce &after = AfterForce{});
// The device memory that bh_compute reserves at most for n bodies (every evaluation a
// build, no quadrupoles, the default opening rule).
size_t bh_bytes(int n, double theta, int leaf_capacity);
// The next bh_compute rebuilds (the bodies were replaced).
void bh_invalidate(BHTree *t);
// A replayed build changed the node count behind the host's back.
void bh_mark_count_stale(BHTree *t);
nb_status bh_info(BHTree *t, cudaStream_t st, nb_bh_info *info);
// Order of the bodies along the Hilbert curve through the 2^10-cell grid of the root cube
// (runs of sorted bodies fill compact regions): *order maps a sorted index to the
// original one; *root_centre points at the device copy of the root cube centre (3
// doubles), followed by the cube's side (a 4th double).  Both stay valid until the next
// call on t.
nb_status bh_hilbert_order(BHTree *t, const double *x, const double *y, const double *z, int n,
                           cudaStream_t st, const uint32_t **order, const double **root_centre);
// A stable sort of caller-made keys: bh_sort_buffers returns the key and
// value arrays (n entries) to fill on the device; bh_sort_keys then sorts them
// by the key bits [first_shift, 64) and returns the sorted values (valid until
// the next call on t).
nb_status bh_sort_buffers(BHTree *t, int n, uint64_t **keys, uint32_t **vals);
nb_status bh_sort_keys(BHTree *t, int n, int first_shift, cudaStream_t st,
                       const uint32_t **order);
nb_status bh_read_order(BHTree *t, cudaStream_t st, uint64_t *codes, uint32_t *order);
nb_status bh_read_nodes(BHTree *t, cudaStream_t st, int max_nodes, int *depth,
                        uint64_t *prefix, int *first, int *count, int *is_leaf, int *skip,
                        float *com_mass);

} // namespace nb

// The simulation object behind nb_sim*.
struct nb_sim {
    nb_config cfg{};
    size_t capacity = 0;
    size_t n = 0;
    cudaStream_t stream = nullptr;
    int device = 0;

    // FP64 state: x y z vx vy vz ax ay az m, each `capacity` doubles.
    nb::DevBuf state;
    double *f[10] = {};
    bool forces_valid = false;

    // Float4 mirrors for the mixed kernel.  An RK4 step below kMixedPairsMin bodies
    // alternates between two: a stage's launch reads one and writes the next stage's
    // positions to the other.
    nb::DevBuf split_hi[2], split_lo[2];
    nb::SortedBuffers sorted;        // Hilbert-sorted near/far variant of the mixed kernel
    nb::DevBuf partials;             // j-split partial sums
    nb::DevBuf old_acc;              // velocity-Verlet a(t)
    nb::DevBuf rk4;                  // RK4 stage states and accelerations
    nb::DevBuf diag_scratch;
    nb::BHTree *bh = nullptr;
    bool bh_serial = false;          // bh_prefer_serial; a captured step keeps its walk

    // One step as a CUDA graph (nb_step): captured on the second of two
    // consecutive eligible steps with the same integrator and dt, replayed
    // while they and the accelerations-valid flag stay the same; any load,
    // configuration or flag change drops it.
    cudaGraphExec_t step_graph = nullptr;
    int graph_integ = -1;
    double graph_dt = 0.0;
    bool graph_fv_before = false, graph_fv_after = false;  // forces_valid around the step
    uint64_t graph_kernels = 0;     // kernel nodes per replay (launch accounting)
    int warm_integ = -1;            // the last uncaptured eligible step
    double warm_dt = 0.0;
    bool graphs_off = false;        // a capture failed: run steps directly

    // Optional timing of the dominant force kernel (nb_profile_*).
    bool profiling = false;
    std::vector<nb::KernelTimer> timers;
    size_t timers_used = 0;

    double *x() const { return f[0]; }
    double *y() const { return f[1]; }
    double *z() const { return f[2]; }
    double *vx() const { return f[3]; }
    double *vy() const { return f[4]; }
    double *vz() const { return f[5]; }
    double *ax() const { return f[6]; }
    double *ay() const { return f[7]; }
    double *az() const { return f[8]; }
    double *m() const { return f[9]; }
};

namespace nb {
// Evaluates accelerations of positions (px,py,pz) with masses m into out* and
// applies `after`.  mirror: the one the mixed kernels read; split: it holds these
// positions already.
nb_status eval_forces(nb_sim *s, const double *px, const double *py, const double *pz,
                      double *oax, double *oay, double *oaz,
                      const AfterForce &after = AfterForce{}, bool split = false,
                      int mirror = 0);
// Drops the captured step graph (the next steps run directly).
void reset_step_graph(nb_sim *s);
// Kernel launches made by a graph replay (the launch counter's evidence).
void count_launches(uint64_t k);
}
