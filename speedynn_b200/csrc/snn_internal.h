// Internal declarations shared by the kernels (snn_kernels.cu) and the host
// driver (snn_api.cu).  Not part of the public ABI.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <vector>

namespace snn {

struct EventPair {
    cudaEvent_t a = nullptr, b = nullptr;
};

// A device allocation that buffers are carved from (snn_blocks.cu), with the
// stream and timing events of the handle that had it last.
struct Block {
    char *base = nullptr;
    size_t bytes = 0;
    int device = 0;
    unsigned long long id = 0;  // the driver's id of the allocation
    cudaStream_t stream = nullptr;
    std::vector<EventPair> events;
};
// A block of at least `bytes` bytes on the current device, a spare one if there is one.
cudaError_t block_acquire(int device, size_t bytes, Block *out);
// Give a block back: kept as a spare if it is small and nothing uses it any more (idle), else freed.
void block_release(Block &b, bool idle);
// Free the spare blocks of a device, or of all devices (device < 0).
void blocks_trim(int device);

// Selection state kept on the device so that a whole greedy step (score ->
// reduce -> select -> commit) runs without a host round trip.
struct State {
    int step;         // greedy steps completed
    int done;         // 1: selection finished (last step, auto stop or error)
    int error;        // SNN_ERR_NO_WINNER when no candidate had a finite error
    int winner;       // feature chosen by the last completed step
    int n_cand;       // candidates of the next step
    int best_k_last;  // best k of the last winner
    int num_final;    // features in the model after the last step
    int full_scan;    // 1: the sorted first steps or the pruned scan leave the step to the dense scorer
    int flat;         // the pruned scan's probe in this step: warps << 20, their estimated cost
};

// Everything a kernel needs, passed by value.
//
// Layout in HBM:
//   XT  [p][ldc]  neighbour (training) points, feature-major, zero padded
//   XV  [p][ldr]  scored points, feature-major (aliases XT in CV mode)
//   D   [n_rows][ldc]  committed FP32 distance matrix, row = scored point;
//                 +inf on excluded pairs (same CV fold) and on pad columns
//   pred [p][nk][n_rows]  kNN-mean prediction per (candidate slot, k, row)
struct Bufs {
    const float *XT;
    const float *XV;
    int ldc, ldr;
    const float *yc;
    const float *yr;
    float *D;
    int n_rows, n_cols, p;
    const int *kvals;
    int nk, kmax;
    float *pred;
    float *rmse32;
    double *rmse64;
    int *cands;       // current candidate list, in the order of perm
    int *prev_cands;  // candidate list of the last scored step
    const int *perm;  // all features, ascending training variance (ties: ascending id)
    int *mask;
    int *order;
    float *err;
    double *err64;
    int *stepk;
    State *st;
    int *nn_idx;      // optional [n_cand][n_rows][kmax]
    float *nn_dist;
    // losses beyond the default RMSE (nloss 0: RMSE only, nothing recorded)
    int nloss;
    const int *loss_ids;  // [nloss] reference loss ids; index 0 decides
    float *lossval;       // [nloss][n_cand][nk] this step's losses
    float *err_all;       // [nloss][p] the winners' losses, reference order l * p + i
    // backward: each (feature, row)'s k-th distance of the last step, [p][n_rows];
    // removing a feature only lowers distances, so it bounds the next step's k-th
    float *kth_prev;
    int use_prev;         // 1: this step may take its bounds from kth_prev
    const float *dmax;    // backward: per row, >= every finite committed distance (filter margin)
    int inject_stall;     // test hook, 0 off: block 0 never issues the copies of stage inject_stall - 1
    // optional filter counters of the TMA-fed scorer: [0] (row, chunk) pairs of
    // the full pass, [1] of them flagged by the filter, [2] holding an exact pass
    unsigned long long *fcount;
    // forward: kSeeds columns per row near it under the committed D, and their
    // distances [n_rows][kSeeds] (written by the previous step's commit); when
    // use_seeds is set the TMA-fed scorer takes its starting bounds from them
    const int *seeds;
    const float *seed_d;
    float *bound;  // forward: [p][n_rows] starting bounds of a seeded step (k_seed_bounds)
    int use_seeds;
    // the pruned scan (snn_scan.cu): the step's candidates packed [group][column][32];
    // backward: [group][column] extremes over the group's candidates, and per
    // feature (mean, min, max, -) of its training column
    float *xg;
    float2 *ext;
    const float4 *fstat;
    // forward problems that the scan leaves to k_walk: slot * n_rows + r of
    // each, how many, and every feature's sorted values with their columns
    // ([p][ldc], null where nothing is sorted)
    int *walk;
    int *n_walk;
    const float *sval;
    const int *sidx;
    // forward: each row's near columns as the last commit found them (null: none
    // kept): (column, distance) [n_rows][kNearList], all columns below near_info's y
    // if its x, their number, is at most kNearList; z: a distance below which about
    // a quarter of them lie; and what the next commit lists by (k_commit)
    int2 *near_list;
    float4 *near_info;
    float4 *near_next;
    int only_if_full;  // scoring kernels return at once unless st->full_scan is set
};

constexpr int kPadCols = 64;     // row stride multiple of the feature-major arrays / D
constexpr int kScoreMaxK = 256;  // largest k_max of the scoring kernel

// Launch shape of the scoring kernel: cc candidates per thread, `warps`
// warps per block (32 scored rows per block), dynamic shared memory bytes.
struct ScorePlan {
    int cc;
    int warps;
    int smem;
};
ScorePlan plan_score(int kmax, int p, int max_smem);

constexpr int kErrTimeout = -7;  // SNN_ERR_TIMEOUT: a bounded device wait gave up

// snn_last_error() plumbing shared by the C-ABI translation units.
int record_error(int code, const char *msg);
void clear_error();

// Warp-specialised TMA scoring (snn_score_tma.cu), k_max <= 64.
bool score_tma_supported(int kmax);  // kernel option 3: k_max <= 64
cudaError_t launch_score_tma(const Bufs &b, int n_cand, int backward, cudaStream_t s);
int score_tma_launches(int kmax, int n_cand, int backward);  // kernels one launch_score_tma issues
// Seeded forward steps: each candidate's starting bound from the seed columns, into b.bound.
// packed: b.xg holds the step's candidates (launch_pack_groups).
cudaError_t launch_seed_bounds(const Bufs &b, int n_cand, cudaStream_t s);

// Pruned scan (snn_scan.cu), k_max <= kScoreMaxK, given the packed candidates
// b.xg.  Where its starting bounds come from: nowhere else than b.kth_prev
// (backward, after a scored step), the seed columns b.seeds that the commit
// kept, or seed columns that the kernel finds itself.
enum { kNoSeeds = 0, kGivenSeeds = 1, kOwnSeeds = 2 };
inline int scan_groups(int n_cand) { return (n_cand + 31) / 32; }  // groups of at most 32 candidates
inline int scan_group_size(int n_cand) { return (n_cand + scan_groups(n_cand) - 1) / scan_groups(n_cand); }  // of a full group
cudaError_t launch_pack_groups(const Bufs &b, int n_cand, int backward, cudaStream_t s);
// May leave problems in b.walk for launch_walk (scan_leaves_walks).  gated: does
// nothing if State::full_scan is set (the dense scorer follows with only_if_full).
cudaError_t launch_scan(const Bufs &b, int n_cand, int backward, int seeding, bool gated, int max_smem, cudaStream_t s);
bool scan_leaves_walks(const Bufs &b, int n_cand, int backward);
// Estimates from a few rows what the scan would cost and sets State::full_scan
// if the dense scorer is faster; for problems where it may be (scan_worth_probing).
cudaError_t launch_scan_probe(const Bufs &b, int n_cand, int backward, int seeding, int max_smem, cudaStream_t s);
bool scan_worth_probing(const Bufs &b, int n_cand);
cudaError_t launch_walk(const Bufs &b, cudaStream_t s);

// Commit the winner into D (snn_commit.cu); forward commits given seed
// buffers also keep kSeeds near columns per row for the next step's bounds.
constexpr int kSeedsPerLane = 8;        // seed columns each lane of the commit keeps: the nearest of each eighth of its columns
constexpr int kSeeds = 32 * kSeedsPerLane;  // seed columns per row
// list: write b.near_list by the last such commit's b.near_next.  About 1,024
// columns are aimed at (768: fwd-64k 94.6, k = 50 271.9 ms a selection, 1,400:
// 95.3 and 272.0, 1,024: 93.9 and 267.8); kNearList leaves room for twice that.
constexpr int kNearList = 2048;
constexpr int kNearLeast = 256;  // a shorter list is not used: too many bounds reach beyond it, and the row is read for them
cudaError_t launch_commit(const Bufs &b, int backward, int *seeds, float *seed_d, bool list, cudaStream_t s);
// Known features (a warm start), in their order; start: from the empty matrix of
// a forward selection (D need not hold anything).
constexpr int kFeatureSeq = 16;
struct FeatureSeq {
    int n;
    int f[kFeatureSeq];
};
cudaError_t launch_commit_seq(const Bufs &b, const FeatureSeq &seq, int backward, bool start, int cv, int npf, int *seeds,
                              float *seed_d, cudaStream_t s);

// First forward step of a holdout problem from per-feature sorted training
// values (snn_sorted.cu): sort at load, then one thread per problem.
size_t sort_temp_bytes(int p, int ldc);
cudaError_t launch_sort_features(const Bufs &b, float *keys, int *vals, int *offsets, float *sv, int *si, void *temp,
                                 size_t temp_bytes, cudaStream_t s);
cudaError_t launch_first_step(const Bufs &b, const float *sv, const int *si, int n_cand, cudaStream_t s);
// The second step: walks of the first winner's sorted values (xs: n_cand x ldc
// floats of scratch for the candidates' values in that order; walked: a device
// counter).
cudaError_t launch_second_step(const Bufs &b, const float *sv, const int *si, float *xs, int n_cand,
                               unsigned long long *walked, cudaStream_t s);

cudaError_t launch_transpose(const float *X, int n, int p, float *XT, int ld, cudaStream_t s);
cudaError_t launch_init_forward(const Bufs &b, int cv, int npf, cudaStream_t s);
cudaError_t launch_full_distance(const Bufs &b, int cv, int npf, cudaStream_t s);
cudaError_t launch_score(const Bufs &b, int n_cand, const ScorePlan &plan, int backward, cudaStream_t s);
cudaError_t launch_reduce(const Bufs &b, int n_cand, cudaStream_t s);
cudaError_t launch_select(const Bufs &b, int n_cand, int it, int t, int total_steps, int backward,
                          int auto_feature, cudaStream_t s);
cudaError_t launch_reset_state(const Bufs &b, int backward, int total_steps, cudaStream_t s);
// Classification predictions from the kept neighbour lists (mode of the k labels).
cudaError_t launch_mode_predict(const Bufs &b, int n_cand, cudaStream_t s);
// Requested losses of every (candidate, k) prediction vector (b.nloss > 0).
cudaError_t launch_losses(const Bufs &b, int n_cand, cudaStream_t s);
// Per row of D: the largest finite entry (backward; D only shrinks afterwards).
cudaError_t launch_row_dmax(const Bufs &b, float *dmax, cudaStream_t s);
// Per-feature training variance (FP64 sums) into var[p], NaN for non-finite columns; with stat
// also (mean or 0, smallest, largest, 0) of the column.
cudaError_t launch_feature_variance(const Bufs &b, float *var, float4 *stat, cudaStream_t s);
// perm[0..p) = features by ascending var (NaN last, ties by id): the candidate slot order.
cudaError_t launch_feature_order(const float *var, int p, int *perm, cudaStream_t s);
// Record the features of seq as the winners of steps t, t + 1, ... without scoring them.
cudaError_t launch_force(const Bufs &b, const FeatureSeq &seq, int t, int total_steps, int backward, cudaStream_t s);

}  // namespace snn
