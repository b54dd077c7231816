// snn_scan.cu -- candidate scoring by a pruned scan (any k_max <= 256).
//
// The same result as snn_score_tma.cu: for every (scored row, candidate) the
// exact top-k_max list of d = fl(D[r,i] +/- fl((x_r,c - x_i,c)^2)) in the
// reference's stable (distance, index) order (speedynn/lib/cpu.c:128-168) and
// the kNN-mean predictions (cpu.c:56-66).  It needs a starting bound on each
// problem's k-th distance (the seed bounds of a forward step, the previous
// step's k-th distances of a backward step) and evaluates only the pairs that
// the bound leaves open.
//
// Why: with such a bound few pairs are open.  Forward, d >= D, so candidate c
// needs only the columns with D < its bound: on the fwd-64k data 1.5 % of the
// (row, column, candidate) triples at the third step, 0.26 % at the ninth.
// Backward, d = D - s >= D - max s: 0.8 % of bwd-50k's.  A dense scorer is
// bound by the FP32 pipe on the other 99 %.
//
// One warp per (scored row, group of up to 32 candidates), lane = candidate (small
// forward problems without walks: two warps):
//   * starting bounds: backward the previous step's k-th distances; forward from
//     the row's 256 seed columns, for k <= 16 by group minima, above (and where
//     nobody kept seeds) by putting the seed columns into the lists first;
//   * the warp streams its row of D, 512 columns at a time, and queues the
//     columns that any of its candidates may still take (the sign of D - H, H
//     the group's largest bound, which falls as the lists fill); forward, those of
//     two passes at once;
//   * queued columns are taken in batches, their candidate values gathered
//     together from `xg`, the candidates packed [group][column][32] (one aligned
//     128-byte line per column and group, so a gather is one full-width load);
//     every lane forms its candidate's exact distance and appends it to its
//     own buffer in shared memory if it may enter the list;
//   * forward, the commit may have listed the row's near columns, about 1,024, with
//     their distances (snn_commit.cu).  These are taken first, without gathers of D
//     (for long lists their nearest quarter before the others, in place of the
//     seeds), and the row is streamed only for bounds that reach beyond them: late
//     steps of fwd-64k 3.5 -> 2.2 ms, of k = 50 8.0 -> 5.8;
//   * forward without such a list, where the bounds reach beyond the row's 1,024
//     nearest columns (estimated from the seeds), the same in two passes over the
//     row (k = 50, third step of 50,021 x 24,989: 38 -> 30 ms);
//   * when a lane's buffer is half full, all lanes empty theirs together into
//     their lists, heaps of k_max (distance, column) keys in shared memory (four
//     children per node: k = 50 selection 335 -> 314 ms against two).  The
//     keys are ordered by distance, then column, which is the reference's
//     stable rule in whatever order the columns arrive;
//   * forward, a row that is an outlier in a feature leaves that candidate's
//     bound far above the others'.  Such problems are left to k_walk
//     (snn_sorted.cu), the split by the cost estimated from sampled columns;
//   * backward, H takes each candidate's largest possible s on the row; a
//     queued column is tested once more, with the group's extreme values in
//     that column (`ext`), before it is gathered.
// The insertion, the gather and the column test each stand once in the loop:
// with the insertion unrolled at every use the kernel waited for instructions
// 80 % of the time.
//
// What bounds it: instruction issue (72 % of the slots at half of fwd-64k, 37,000
// instructions per warp of 32,768 columns; 64 % backward, 49 % at k = 50, where
// the heaps leave 13 warps per SM) well above the D stream.  The gathers' latency
// is covered by the other warps: with them in flight through shared memory
// (cp.async, 8 to 16 columns ahead) fwd-64k took 110 to 112 ms against 110,
// backward 210 to 217 against 204.  Scoring of a whole fwd-64k selection 293 -> 50
// ms, a backward step of 25,003 x 12,502 7.0 -> 1.0 ms, a late k = 50 step of
// 50,021 x 24,989 57 -> 6 ms, a k = 150 step of 8,192 x 4,096 x 19 130 -> 3.2 ms.
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "snn_internal.h"
#include "snn_packed.cuh"

namespace snn {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kUnroll = 4;            // float4 loads of D per lane and pass of the loop
constexpr int kCols = 128 * kUnroll;  // columns per pass of the loop
constexpr int kQueue = 256;           // entries of a warp's column queues (a power of two, kSeeds at least)
constexpr float kCap = 0x1.fffffcp+127f;  // largest distance that can enter a list (items at FLT_MAX never do)
// Instructions of a warp, for choosing who walks (k_scan): a queued column, the
// start of a walk, a column of it, a column of another pass over the row (a walk's column: 1.6 instructions, but its gather of D fetches
// 64 bytes from memory, worth more; fwd-64k 120 ms a selection at 4, 118 at 9).
constexpr float kQueueCost = 14.0f, kWalkStart = 3000.0f, kWalkCost = 8.0f, kPassCost = 0.2f;
// Per column of a group: reading it, the second test, and the dense scorers' work
// per candidate (measured: 30,000 x 15,000 x 38 8 ms, the scan 14 with 68 % open).
constexpr float kReadCost = 0.25f, kTestCost = 4.0f, kDenseCost = 0.28f;
constexpr int kProbeRows = 64;
// The probe's warps and their cost share State::flat, so no more of them than 11
// bits count: above 1,023 candidates they are spread over fewer rows.  (With 32
// bits for each, the code of the instances changed: k = 150 0.5 % slower.)
constexpr int kProbeWarps = 2047;
static_assert(64 * kProbeWarps < 1 << 20, "their cost, at most 64 each, has 20 bits");
static_assert(kSeedsPerLane == 8, "the commit and the scan keep eight seeds per lane");
static_assert(kQueue >= kSeeds && kQueue >= 128 + 16 + 32, "room for a pass's columns");

// Order-preserving signed key of a float (no NaN), and back.
__device__ __forceinline__ int fkey(float v)
{
    const int u = __float_as_int(v);
    return u ^ ((u >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float fkey_inv(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

// List keys: (distance, column) as one unsigned 64-bit number.  Forward
// distances are >= +0, so their bits order like the values; backward ones may
// be negative.
template <bool BWD>
__device__ __forceinline__ unsigned long long pack_key(float d, int col)
{
    const unsigned u = BWD ? (unsigned)fkey(d) ^ 0x80000000u : __float_as_uint(d);
    return ((unsigned long long)u << 32) | (unsigned)col;
}
template <bool BWD>
__device__ __forceinline__ float key_dist(unsigned long long k)
{
    const unsigned u = (unsigned)(k >> 32);
    return BWD ? fkey_inv((int)(u ^ 0x80000000u)) : __uint_as_float(u);
}

// Put key in the place of entry i of the lane's max-heap h[0], h[32], ... (n
// entries, four children per node: half the dependent levels of a binary heap)
// and sink it.
__device__ __forceinline__ void sift_down(unsigned long long *h, int n, unsigned long long key, int i = 0)
{
    for (int c = 4 * i + 1; c < n; c = 4 * i + 1) {
        const unsigned long long *p = h + c * 32;
        const unsigned long long k0 = p[0], k1 = c + 1 < n ? p[32] : 0ull, k2 = c + 2 < n ? p[64] : 0ull,
                                 k3 = c + 3 < n ? p[96] : 0ull;
        const bool a = k1 > k0, d = k3 > k2;
        const unsigned long long ka = a ? k1 : k0, kd = d ? k3 : k2;
        const bool e = kd > ka;
        const unsigned long long k = e ? kd : ka;
        if (key >= k) break;
        h[i * 32] = k;
        i = c + (e ? (d ? 3 : 2) : (a ? 1 : 0));
    }
    h[i * 32] = key;
}

// Shared memory of a warp: heaps and buffers (two batches) of 32 lanes, and lists of columns.
size_t warp_smem(int K, int batch, int lists)
{
    return sizeof(unsigned long long) * 32 * (size_t)(K + 2 * batch) + sizeof(int) * (size_t)kQueue * lists;
}

__device__ __forceinline__ unsigned sign_in(unsigned m, float v) { return __funnelshift_l(__float_as_uint(v), m, 1); }

// What a kernel instance does before it scans the row (SEED): nothing
// (backward, bounds from the last step); bound every candidate's k-th distance
// by SEED group minima over the row's seed columns; or put the seed columns
// into the heaps.
constexpr int kSeedNone = 0, kSeedHeap = -1;

// kBatch queued columns are gathered together, and a lane buffers up to twice
// as many keys before they enter its heap.  Large problems take batches of 4 at
// 72 registers (two instances spill 4 bytes) and 28 warps per SM, which hide the
// gathers for one another (fwd-64k 118.0 ms a selection; batches of 8 with 20
// warps 122.7, with the loads of one batch under the work of the last one at 16
// warps 139.6); few rows (one_wave), whose time is the chain of gathers of one
// warp, take batches of 16 at up to 128 registers.  Instances that fill heaps
// from seeds (k > 16) rarely find shared memory for more than 24 warps (80
// registers).
constexpr int kBatchMany = 4, kBatchFew = 16, kWarpsMany = 28, kWarpsHeap = 24;
// ... and, forward from given bounds, two warps for each (row, group), each with
// every other pass over the row; the first one merges the lists (steps 3 to 8 of
// 2,000 x 1,000 x 20: 0.50 -> 0.39 ms; four warps 0.45; backward, where the work
// before the lists is short, it loses: 1,501 x 14 1.35 -> 1.50 ms a run).
constexpr int kMaxSplit = 2;

template <bool BWD, int SEED, int kBatch>
__global__ void __launch_bounds__(kBatch == kBatchMany ? 32 : 32 * kMaxSplit,
                                  kBatch != kBatchMany ? 16 / kMaxSplit : SEED == kSeedHeap ? kWarpsHeap : kWarpsMany)
    k_scan(Bufs b, int n_cand, int G, int gs, int walks, int own, int gated, int probe)
{
    constexpr int kBuf = 2 * kBatch;
    constexpr bool kHold = !BWD && kBatch == kBatchMany;  // push once per two passes (k = 50 of 50,021 x 24,989: 310 -> 303 ms)
    extern __shared__ __align__(16) unsigned char smraw[];
    if (b.st->done) return;
    if (gated && b.st->full_scan) return;  // the dense scorer takes the step
    constexpr bool kSplit = kBatch == kBatchFew && SEED > 0;
    // blocks of one warp for many: warps finish at different times
    const int lane = threadIdx.x & 31, w = kSplit ? threadIdx.x >> 5 : 0, warps = kSplit ? blockDim.x >> 5 : 1;
    // probe: only estimate, for rows that far apart, what the scan would cost
    const int r = blockIdx.x / G * (probe ? probe : 1), g = blockIdx.x % G;
    const int K = b.kmax;
    const size_t lists_at = sizeof(unsigned long long) * 32 * (size_t)(K + kBuf);
    const size_t wsmem = lists_at + sizeof(int) * kQueue;  // of a warp, where there are several
    unsigned long long *heap = reinterpret_cast<unsigned long long *>(smraw + w * wsmem) + lane;
    unsigned long long *buf = heap + (size_t)K * 32;
    int *queue = reinterpret_cast<int *>(smraw + w * wsmem + lists_at);
    int *wait = queue + kQueue;                  // backward: columns before the second test
    int *own_seed = queue + (BWD ? 2 : 1) * kQueue;  // kSeedHeap: the lanes' seed columns
    float *queue_d = reinterpret_cast<float *>(queue + kQueue);  // near columns: the queued columns' distances (own_seed's place)

    const int slot = g * gs + lane;
    const bool live = lane < gs && slot < n_cand;
    const int c = live ? __ldg(b.cands + slot) : 0;
    float xv = live ? __ldg(b.XV + (size_t)c * b.ldr + r) : NAN;
    const bool act = isfinite(xv);  // otherwise no distance of this candidate is below FLT_MAX
    if (!act) xv = NAN;             // never passes
    const size_t cr = (size_t)c * b.n_rows + r;
    const float *xg = b.xg + (size_t)g * b.ldc * 32 + lane;
    const float *Dr = b.D + (size_t)r * b.ldc;
    const float4 *row = reinterpret_cast<const float4 *>(Dr);
    const int n4 = b.ldc >> 2;

    // near: about the 1,024th smallest committed distance of the row.  A lane's
    // eight seeds are the minima of eight 256ths of the row, so the middle of them
    // is about the row's 172nd smallest distance and the largest about the 680th,
    // by the minimum of m independent values; the power law through the lanes'
    // means goes on to near (858 to 1,134 columns below it on average in the
    // steps of the fwd-64k and fwd-200k data).
    float near = INFINITY;
    auto set_near = [&](float d4, float d5, float d8) {
        float mid = 0.5f * (d4 + d5);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mid += __shfl_xor_sync(kFull, mid, o);
            d8 += __shfl_xor_sync(kFull, d8, o);
        }
        const float v = d8 * 0.03125f * powf(d8 / mid, 0.298f);  // ln(1024 / 680) / ln(680 / 172)
        if (v < FLT_MAX) near = v;  // otherwise (a lane without eight seeds, ties at 0): one stage for all columns
    };

    // The row's near columns, where the commit could list them all.
    constexpr bool kLists = !BWD && (SEED > 0 || SEED == kSeedHeap);
    bool listed = false;  // taking them now
    int n_near = 0;
    float quarter = 0.0f;
    if (kLists && b.near_list && !probe) {
        const float4 info = __ldg(b.near_info + r);
        listed = info.x <= (float)kNearList && info.x >= (float)kNearLeast && warps == 1;
        if (listed) {
            n_near = (int)info.x;
            near = info.y;
            quarter = info.z;
        }
    }

    // lim: distances above it cannot enter the lane's list.
    float lim = act ? kCap : -INFINITY;
    if (BWD && SEED == kSeedNone && act) lim = fminf(b.kth_prev[cr], kCap);
    if constexpr (SEED > 0) {
        // Any k distinct columns bound the k-th distance.  The minimum over each
        // group of 8 (k <= 8) or 4 seed columns belongs to another column, and the
        // k-th smallest of the 32 or 64 minima is nearly as tight as that of all 256
        // columns (for k = 10: the 4.2 % quantile of their distances instead of 3.9 %)
        // at an eighth or a quarter of the list insertions.
        constexpr int P = SEED <= 8 ? 8 : 4;
        float L[SEED];  // ascending; the first SEED - K entries -inf, so the k-th is the last
#pragma unroll
        for (int j = 0; j < SEED; ++j) L[j] = j < SEED - K ? -INFINITY : INFINITY;
        const int4 *seeds = reinterpret_cast<const int4 *>(b.seeds + (size_t)r * kSeeds);
        const float4 *seed_d4 = reinterpret_cast<const float4 *>(b.seed_d + (size_t)r * kSeeds);
        const float2 xv2 = make_float2(xv, xv);
        int4 ia = __ldg(seeds), ib = __ldg(seeds + 1);  // -1 for an absent column, its distance +inf
#pragma unroll 1
        for (int j = 0; j < kSeeds / 4; j += 2) {
            auto at = [&](int i) { return __ldg(xg + (size_t)max(i, 0) * 32); };
            const float2 x0 = make_float2(at(ia.x), at(ia.y)), x1 = make_float2(at(ia.z), at(ia.w));
            const float2 x2 = make_float2(at(ib.x), at(ib.y)), x3 = make_float2(at(ib.z), at(ib.w));
            const float4 da = __ldg(seed_d4 + j), db = __ldg(seed_d4 + j + 1);
            if (j + 2 < kSeeds / 4) {
                ia = __ldg(seeds + j + 2);
                ib = __ldg(seeds + j + 3);
            }
            auto least = [&](float4 d, float2 xa, float2 xb) {  // a NaN is left out, NaN if all are
                const float2 u = add2(make_float2(d.x, d.y), sq2(sub2(xv2, xa))), v = add2(make_float2(d.z, d.w), sq2(sub2(xv2, xb)));
                return fminf(fminf(u.x, u.y), fminf(v.x, v.y));
            };
            const float va = least(da, x0, x1), vb = least(db, x2, x3);
#pragma unroll
            for (int i = 0; i < 8; i += P) {
                // a group of missing values only (all NaN) counts as no column: as NaN it
                // would shift L and count a smaller entry twice
                const float v = fminf(P == 8 ? fminf(va, vb) : i ? vb : va, INFINITY);
                if (__any_sync(kFull, v < L[SEED - 1])) {
#pragma unroll
                    for (int q = SEED - 1; q > 0; --q) L[q] = fminf(L[q], fmaxf(L[q - 1], v));
                    L[0] = fminf(L[0], v);
                }
            }
        }
        const float *seed_d = b.seed_d + (size_t)r * kSeeds + lane;
        if (act) lim = fminf(L[SEED - 1], kCap);
        if (!listed) set_near(__ldg(seed_d + 3 * 32), __ldg(seed_d + 4 * 32), __ldg(seed_d + 7 * 32));
    }

    // The list starts as K sentinels at the (inclusive) bound, ordered after every
    // column; those left at the end are padding.
    // They give way from the last entry up, where a key sinks through few levels
    // or none; once all are gone (put is 0), a key replaces the largest entry.
    for (int j = 0; j < K; ++j) heap[j * 32] = pack_key<BWD>(lim, -1);
    // (Not in the large backward instance, whose registers are all in use.)
    constexpr bool kPut = !(BWD && SEED == kSeedNone && kBatch == kBatchMany);
    int put = kPut ? K - 1 : 0;
    auto enter = [&](unsigned long long key) {
        if (key < heap[put * 32]) {
            sift_down(heap, K, key, put);
            if (kPut) put = max(put - 1, 0);
        }
    };

    int qh = 0, qn = 0;  // queue: first entry, entries
    // kSeedHeap: the seed columns go through the queue before the row's others; the
    // lane keeps its own (the commit and this kernel give each lane the same
    // columns), ascending, to leave them out afterwards.
    // (Not with near columns: those make the start.)
    int nseed = 0;  // the lane's seed columns already passed, the next at own_seed[32 * nseed + lane]
    int noseed = listed ? kSeedsPerLane : 0;  // entries of own_seed without a column
    if (SEED == kSeedHeap && !listed) {
        int si[kSeedsPerLane];
        if (!own) {
            const float *seed_d = b.seed_d + (size_t)r * kSeeds + lane;
            if (!BWD) set_near(__ldg(seed_d + 3 * 32), __ldg(seed_d + 4 * 32), __ldg(seed_d + 7 * 32));
#pragma unroll
            for (int j = 0; j < kSeedsPerLane; ++j) si[j] = __ldg(b.seeds + (size_t)r * kSeeds + j * 32 + lane);
        } else {
            // nobody kept them: the same minima from a pass of its own (snn_commit.cu)
            float sv[kSeedsPerLane];
#pragma unroll
            for (int j = 0; j < kSeedsPerLane; ++j) {
                sv[j] = INFINITY;
                si[j] = -1;
            }
            const int part = ((n4 / 2 + 127) / 128) * 128;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll 4
                for (int q = h * part + lane; q < (h ? n4 : min(part, n4)); q += 32) {
                    const float4 d = __ldg(row + q);
                    const float v[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const bool less = v[e] < sv[4 * h + e];
                        sv[4 * h + e] = less ? v[e] : sv[4 * h + e];
                        si[4 * h + e] = less ? 4 * q + e : si[4 * h + e];
                    }
                }
            }
#pragma unroll
            for (int i = 1; i < kSeedsPerLane; ++i)
#pragma unroll
                for (int j = i; j > 0; --j) {
                    const bool swap = sv[j] < sv[j - 1];
                    const float lv = swap ? sv[j] : sv[j - 1], hv = swap ? sv[j - 1] : sv[j];
                    const int li = swap ? si[j] : si[j - 1], hi = swap ? si[j - 1] : si[j];
                    sv[j - 1] = lv;
                    sv[j] = hv;
                    si[j - 1] = li;
                    si[j] = hi;
                }
            if (!BWD) set_near(sv[3], sv[4], sv[7]);
        }
#pragma unroll
        for (int j = 0; j < kSeedsPerLane; ++j) {  // nearest first
            const unsigned m = __ballot_sync(kFull, si[j] >= 0);
            if (si[j] >= 0) queue[qn + __popc(m & ((1u << lane) - 1u))] = si[j];
            qn += __popc(m);
            noseed += si[j] >= 0 ? 0 : 1;
        }
        nseed = noseed;
#pragma unroll
        for (int i = 1; i < kSeedsPerLane; ++i)  // ascending, absent ones (-1) first
#pragma unroll
            for (int j = i; j > 0; --j) {
                const int lo = min(si[j - 1], si[j]), hi = max(si[j - 1], si[j]);
                si[j - 1] = lo;
                si[j] = hi;
            }
#pragma unroll
        for (int j = 0; j < kSeedsPerLane; ++j) own_seed[32 * j + lane] = si[j];
    }

    // Backward: each candidate's largest possible square on this row and the
    // row's extreme centred values (rounded outwards).
    float smax = 0.0f, amax = -INFINITY, amin = INFINITY, kmx = 0.0f;
    if constexpr (BWD) {
        if (act) {
            const float4 f = __ldg(b.fstat + c);  // mean, min, max of the training column
            const float um = fmaxf(__fsub_ru(xv, f.y), __fsub_ru(f.z, xv));
            smax = __fmul_ru(um, um);
            amax = __fsub_ru(xv, f.x);
            amin = __fsub_rd(xv, f.x);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            amax = fmaxf(amax, __shfl_xor_sync(kFull, amax, o));
            amin = fminf(amin, __shfl_xor_sync(kFull, amin, o));
        }
    }

    // No column with D >= H can enter a list of the queue's candidates: forward
    // d >= D; backward d <= lim means D - s < nextafter(lim) exactly (rounding is
    // monotone), and s <= smax.  kmx: the same for the second test.
    float H = 0.0f;
    auto update_H = [&] {
        if constexpr (BWD) {
            const float up = nextafterf(lim, INFINITY);
            H = __int_as_float(__reduce_max_sync(kFull, __float_as_int(fmaxf(__fadd_ru(up, smax), 0.0f))));
            kmx = fkey_inv(__reduce_max_sync(kFull, fkey(up)));
        } else {
            H = __int_as_float(__reduce_max_sync(kFull, __float_as_int(fmaxf(lim, 0.0f))) + 1);
        }
    };
    unsigned wide = 0u;  // forward: candidates left to k_walk, their lim -inf here
    // probe: the group's estimated instructions against the dense scorer's.  Where
    // most columns stay open (distances that hardly differ, as with two-valued
    // features committed; backward, features whose squares reach far) that one is
    // faster; the last of the probing warps decides, at ten sixteenths since ties make
    // a queued column dearer than estimated.
    auto vote = [&](float cost) {
        if (lane != 0) return;
        const float dense = kDenseCost * (float)gs * (K <= 16 ? 1.0f : K <= 32 ? 1.5f : 2.0f) * (float)b.n_cols;
        const int units = (int)fminf(16.0f * cost / dense, 64.0f);
        const int old = atomicAdd(&b.st->flat, (1 << 20) + units);  // of at most kProbeWarps warps
        if ((old >> 20) + 1 == (int)gridDim.x && (old & 0xfffff) + units > 10 * (int)gridDim.x) b.st->full_scan = 1;
    };
    auto choose_walks = [&] {
        // The split with the least estimated cost, from 128 sampled columns (64 for
        // the candidates' own squares): a queued column costs the group kQueueCost
        // instructions, a walk kWalkStart and kWalkCost for each column whose square
        // is within the candidate's bound.
        int cd = 0, cs = 0;  // sampled columns with D, with the square within the lane's bound
#pragma unroll 1
        for (int i = 0; i < 4; ++i) {
            const int j0 = i * (b.n_cols / 4);
            const float smp = __ldg(Dr + j0 + lane);
#pragma unroll 8
            for (int l = 0; l < 32; ++l) cd += __shfl_sync(kFull, smp, l) <= lim ? 1 : 0;
            if (walks) {
#pragma unroll 8
                for (int l = 0; l < 16; ++l) {
                    const float t = xv - __ldg(xg + (size_t)(j0 + l) * 32);
                    cs += t * t <= lim ? 1 : 0;
                }
            }
        }
        const float n = (float)b.n_cols;
        // if the candidates with more columns walk; beyond near the row is read once more
        float cost = kQueueCost / 128.0f * n * (float)cd + (lim >= near ? kPassCost * n : 0.0f);
        if (walks) {
            const float walk = kWalkStart + kWalkCost / 64.0f * n * (float)cs;
#pragma unroll 4
            for (int l = 0; l < 32; ++l) {
                const float wl = __shfl_sync(kFull, walk, l);
                cost += __shfl_sync(kFull, cd, l) > cd ? wl : 0.0f;
            }
        }
        // positive: the bits order like the values
        const int best = walks ? __reduce_min_sync(kFull, __float_as_int(cost)) : __reduce_max_sync(kFull, __float_as_int(cost));
        if (probe) {  // the near columns, taken first, at least halve what stays open (mixture-50k: a quarter)
            vote(__int_as_float(best) * (H > near ? 0.5f : 1.0f));
            return;
        }
        const int cut = __reduce_min_sync(kFull, __float_as_int(cost) == best ? cd : 999);
        wide = walks ? __ballot_sync(kFull, cd > cut) : 0u;
        if (wide) {
            int at = 0;
            if (lane == 0) at = atomicAdd(b.n_walk, __popc(wide));
            at = __shfl_sync(kFull, at, 0) + __popc(wide & ((1u << lane) - 1u));
            if ((wide >> lane) & 1u) {
                b.walk[at] = slot * b.n_rows + r;
                b.bound[cr] = lim;
                lim = -INFINITY;
            }
        }
    };
    // Backward's probe, lane = column: sampled columns queued, and kept by the second test.
    auto probe_backward = [&] {
        int c1 = 0, c2 = 0;
        for (int i = 0; i < 4; ++i) {
            const int j = i * (b.n_cols / 4) + lane;
            const float D = __ldg(Dr + j);
            const float2 x = __ldg(b.ext + (size_t)g * b.ldc + j);
            const float U = fmaxf(__fsub_ru(amax, x.x), __fsub_ru(x.y, amin));
            const bool q = D < H;
            c1 += __popc(__ballot_sync(kFull, q));
            c2 += __popc(__ballot_sync(kFull, q && __fsub_rn(D, __fmul_rn(U, U)) <= kmx));
        }
        vote((float)b.n_cols * (kReadCost + kTestCost / 128.0f * (float)c1 + kQueueCost / 128.0f * (float)c2));
    };

    int nb = 0;  // the lane's buffered keys
    int ah = 0, an = 0;  // backward: columns that wait for the second test
    auto flush = [&] {
        const int most = __reduce_max_sync(kFull, nb);
        for (int j = 0; j < most; ++j) {
            const unsigned long long key = j < nb ? buf[32 * j] : ~0ull;
            enter(key);
        }
        nb = 0;
        if (lim > -INFINITY) lim = key_dist<BWD>(heap[0]);
        update_H();
    };
    update_H();
    // Forward, two stages where the bounds still reach beyond near: its columns
    // first, which leaves nearly exact bounds for the split and for the others
    // (or none of them open).
    int stage = BWD || !(H > near) ? 2 : 0;  // 0: D < near, 1: the rest, 2: all in one
    bool close = SEED == kSeedHeap && listed;  // first only the nearest quarter of the near columns
    if constexpr (SEED != kSeedHeap) {
        if constexpr (BWD) {
            if (probe) probe_backward();
        } else if (probe || (stage == 2 && walks)) {
            choose_walks();
            update_H();
        }
        if (probe) return;
    }
    float4 nxt[kUnroll];
    // The next pass' columns.  Past the row any value does: they are masked.
    auto columns = [&](int q0) {
        if (q0 + kCols <= b.ldc) {
            const float4 *at = row + (q0 >> 2) + lane;
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) nxt[u] = __ldg(at + u * 32);
        } else {
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) nxt[u] = __ldg(row + min((q0 >> 2) + u * 32 + lane, n4 - 1));
        }
    };
    unsigned held = 0u;    // the columns of a pass, pushed together with those of the next
    bool second = false;
    // Near columns, four of 128 per lane and pass: nxt holds this pass' and the next's.
    const float4 *near4 = reinterpret_cast<const float4 *>(b.near_list + (size_t)r * kNearList) + 2 * lane;
    auto near_columns = [&](int q) {
        if (q + 4 * lane < n_near) {
            nxt[2] = __ldg(near4 + (q >> 1));
            nxt[3] = __ldg(near4 + (q >> 1) + 1);
        }
    };
    if (listed) {
        near_columns(0);
        nxt[0] = nxt[2];
        nxt[1] = nxt[3];
        near_columns(128);
    } else {
        columns(w * kCols);
    }
    // kSeedHeap: a pass for the seed columns first
    for (int q0 = SEED == kSeedHeap && !listed ? -kCols : w * kCols;; q0 += listed ? 128 : warps * kCols) {
        const bool last = q0 >= (listed ? n_near : b.ldc);  // no columns left: empty the queues
        const bool drainall = last || q0 < 0;
        unsigned m16 = 0u;  // bit 4u + e: this lane's column q0 + 128 u + 4 lane + e has D < H
        if (listed) {  // bit e: this lane's column e
            const float lo = close ? 0.0f : SEED == kSeedHeap ? quarter : 0.0f, hi = close ? fminf(quarter, H) : H;
            auto open = [&](float d) { return d < hi && d >= lo; };
            m16 = (open(nxt[0].y) ? 1u : 0u) | (open(nxt[0].w) ? 2u : 0u) | (open(nxt[1].y) ? 4u : 0u) | (open(nxt[1].w) ? 8u : 0u);
            const int left = n_near - q0 - 4 * lane;
            if (left < 4) m16 &= left > 0 ? (1u << left) - 1u : 0u;
        } else if (SEED != kSeedHeap || q0 >= 0) {
            // the sign of D - H, first column lowest
            auto below = [&](float limit) {
                const float2 nl = make_float2(-limit, -limit);
                unsigned m = 0u;
#pragma unroll
                for (int u = kUnroll - 1; u >= 0; --u) {
                    const float2 hi = add2(make_float2(nxt[u].z, nxt[u].w), nl), lo = add2(make_float2(nxt[u].x, nxt[u].y), nl);
                    m = sign_in(sign_in(sign_in(sign_in(m, hi.y), hi.x), lo.y), lo.x);
                }
                return m;
            };
            m16 = below(!BWD && stage == 0 ? fminf(H, near) : H);
            if (!BWD && stage == 1) m16 &= ~below(near);
            columns(q0 + warps * kCols);
            if (q0 + kCols > b.ldc) {  // past the row
#pragma unroll
                for (int u = 0; u < kUnroll; ++u)
                    if (q0 + 128 * u + 4 * lane >= b.ldc) m16 &= ~(15u << (4 * u));
            }
            if constexpr (SEED == kSeedHeap) {
                while (nseed < kSeedsPerLane) {
                    const int i = own_seed[32 * nseed + lane] - q0;
                    if (i >= kCols) break;
                    m16 &= ~(1u << (4 * (i >> 7) + (i & 3)));
                    ++nseed;
                }
            }
        }
        if (kHold && !second && !drainall && !listed) {
            held = m16;
            second = true;
            continue;
        }
        const unsigned m32 = kHold && !listed ? held | m16 << 16 : m16;  // bits 0 to 15: the pass before
        held = 0u;
        second = false;
        const int base = kHold && !listed ? q0 - warps * kCols : q0;
        // Rarely more columns than the queue has room for: then a pass, or 128, at a time.
        const unsigned cnt = __reduce_add_sync(kFull, __popc(m32 & 0xffffu) | __popc(m32 >> 16) << 16);
        const unsigned room = kQueue - kBatch - 32, c0 = cnt & 0xffffu, c1 = cnt >> 16;
        const int step = c0 + c1 <= room ? 32 : max(c0, c1) <= room ? 16 : 4;
        for (int part = 0; part < (kHold ? 32 : 16); part += step) {
            // each lane appends its columns, in no particular order
            unsigned mp = (m32 >> part) & (0xffffffffu >> (32 - step));
            for (unsigned any = __ballot_sync(kFull, mp != 0u); any; any = __ballot_sync(kFull, mp != 0u)) {
                if (mp) {
                    const int i = __ffs(mp) - 1 + part;
                    mp &= mp - 1;
                    const int at = __popc(any & ((1u << lane) - 1u));
                    int col = base + 128 * (i >> 2) + 4 * lane + (i & 3) + (kSplit ? (i >> 4) * (warps - 1) * kCols : 0);
                    if constexpr (BWD) wait[(ah + an + at) & (kQueue - 1)] = col;
                    else {
                        if (kLists && listed) {
                            const float4 v = i & 2 ? nxt[1] : nxt[0];
                            col = __float_as_int(i & 1 ? v.z : v.x);
                            queue_d[(qh + qn + at) & (kQueue - 1)] = i & 1 ? v.w : v.y;
                        }
                        queue[(qh + qn + at) & (kQueue - 1)] = col;
                    }
                }
                if constexpr (BWD) an += __popc(any);
                else qn += __popc(any);
            }
            __syncwarp();
            for (;;) {
                if constexpr (BWD) {
                    if (an >= (last ? 1 : 32)) {
                        // Second test, lane = column: an s of this column is at most U^2, U the
                        // larger of the two extreme differences (rounded up), so an entry needs
                        // D - fl(U^2) < nextafter(lim) for some candidate, and its rounding <= kmx.
                        const int n = min(an, 32);
                        const bool in = lane < n;
                        const int col = in ? wait[(ah + lane) & (kQueue - 1)] : 0;
                        const float D = __ldg(Dr + col);
                        const float2 x = __ldg(b.ext + (size_t)g * b.ldc + col);
                        const float U = fmaxf(__fsub_ru(amax, x.x), __fsub_ru(x.y, amin));
                        const bool keep = in && __fsub_rn(D, __fmul_rn(U, U)) <= kmx;
                        const unsigned m = __ballot_sync(kFull, keep);
                        if (keep) queue[(qh + qn + __popc(m & ((1u << lane) - 1u))) & (kQueue - 1)] = col;
                        qn += __popc(m);
                        ah = (ah + n) & (kQueue - 1);
                        an -= n;
                        __syncwarp();
                    }
                }
                while (qn >= (drainall ? 1 : kBatch)) {
                    // the first queued columns against every candidate of the group
                    const int n = min(qn, kBatch);
                    int col[kBatch];
                    float2 d[kBatch / 2], x[kBatch / 2];
#pragma unroll
                    for (int i = 0; i < kBatch; i += 4) {  // qh is a multiple of 4
                        const int4 v = *reinterpret_cast<const int4 *>(queue + ((qh + i) & (kQueue - 1)));
                        col[i] = v.x;
                        col[i + 1] = v.y;
                        col[i + 2] = v.z;
                        col[i + 3] = v.w;
                    }
                    if (n < kBatch) {
#pragma unroll
                        for (int i = 0; i < kBatch; ++i) col[i] = i < n ? col[i] : 0;
                    }
#pragma unroll
                    for (int i = 0; i < kBatch; i += 2) {
                        if (kLists && listed) d[i / 2] = *reinterpret_cast<const float2 *>(queue_d + ((qh + i) & (kQueue - 1)));
                        else d[i / 2] = make_float2(__ldg(Dr + col[i]), __ldg(Dr + col[i + 1]));
                        x[i / 2] = make_float2(__ldg(xg + (size_t)col[i] * 32), __ldg(xg + (size_t)col[i + 1] * 32));
                    }
                    qn -= n;
                    qh = qn ? (qh + n) & (kQueue - 1) : 0;
                    unsigned pm = 0u;
#pragma unroll
                    for (int i = 0; i < kBatch; i += 2) {
                        const float2 s = sq2(sub2(make_float2(xv, xv), x[i / 2]));
                        d[i / 2] = BWD ? sub2(d[i / 2], s) : add2(d[i / 2], s);
                        pm |= (d[i / 2].x <= lim ? 1u << i : 0u) | (d[i / 2].y <= lim ? 2u << i : 0u);
                    }
                    pm &= (1u << n) - 1u;
                    if (__any_sync(kFull, pm != 0u)) {
#pragma unroll
                        for (int i = 0; i < kBatch; ++i)
                            if ((pm >> i) & 1u) buf[32 * nb++] = pack_key<BWD>(i & 1 ? d[i / 2].y : d[i / 2].x, col[i]);
                    }
                    if (__any_sync(kFull, nb > kBuf - kBatch)) flush();
                }
                if (!BWD || an < (last ? 1 : 32)) break;
            }
        }
        if (SEED == kSeedHeap && q0 < 0) {  // the seeds are in
            flush();
            if constexpr (BWD) {
                if (probe) probe_backward();
            } else {
                stage = H > near ? 0 : 2;
                if (probe || (stage == 2 && walks)) {
                    choose_walks();
                    update_H();
                }
            }
            if (probe) return;
        }
        if (kLists && listed && !last) {
            nxt[0] = nxt[2];
            nxt[1] = nxt[3];
            near_columns(q0 + 256);
        }
        if (last) {
            if (SEED == kSeedHeap && close) {
                close = false;
                flush();
                near_columns(0);
                nxt[0] = nxt[2];
                nxt[1] = nxt[3];
                near_columns(128);
                q0 = -128;
                continue;
            }
            if (BWD || stage != 0) break;
            flush();
            if (walks) {
                choose_walks();
                update_H();
            }
            if (!(H > near)) break;
            stage = 1;
            listed = false;
            nseed = noseed;
            q0 = (w - warps) * kCols;
            columns(w * kCols);
        }
    }

    // Epilogue: each lane's list in ascending order, padding as (FLT_MAX, 0),
    // the k-th distance for the next backward step, the optional neighbour
    // dump, labels summed in rank order.
    for (int j = 0; j < nb; ++j) enter(buf[32 * j]);
    if constexpr (kSplit) {
        if (warps > 1) {
            __syncthreads();
            if (w > 0) return;
            for (int v = 1; v < warps; ++v) {
                const unsigned long long *other = reinterpret_cast<const unsigned long long *>(smraw + v * wsmem) + lane;
                for (int j = 0; j < K; ++j) {
                    const unsigned long long key = other[j * 32];
                    if ((int)(unsigned)key >= 0) enter(key);  // no sentinel
                }
            }
        }
    }
    if (!live || ((wide >> lane) & 1u)) return;
    for (int n = K - 1; n > 0; --n) {
        const unsigned long long end = heap[n * 32];
        heap[n * 32] = heap[0];
        sift_down(heap, n, end);
    }
    if (BWD) {
        const unsigned long long k = heap[(K - 1) * 32];
        b.kth_prev[cr] = (int)(unsigned)k >= 0 ? key_dist<BWD>(k) : FLT_MAX;
    }
    if (b.nn_idx) {
        const size_t o = ((size_t)slot * b.n_rows + r) * K;
        for (int j = 0; j < K; ++j) {
            const unsigned long long k = heap[j * 32];
            const int i = (int)(unsigned)k;
            b.nn_idx[o + j] = i >= 0 ? i : 0;
            b.nn_dist[o + j] = i >= 0 ? key_dist<BWD>(k) : FLT_MAX;
        }
    }
    float acc = 0.0f;
    float *pre = reinterpret_cast<float *>(heap);  // entry j's low word becomes the label sum of ranks 0..j
#pragma unroll 8
    for (int j = 0; j < K; ++j) {
        const int i = (int)(unsigned)heap[j * 32];
        acc = __fadd_rn(acc, __ldg(b.yc + (i >= 0 ? i : 0)));
        pre[j * 64] = acc;
    }
    for (int m = 0; m < b.nk; ++m) {
        const int k = __ldg(b.kvals + m);
        b.pred[((size_t)slot * b.nk + m) * b.n_rows + r] = __fdiv_rn(pre[(k - 1) * 64], (float)k);
    }
}

// xg[g][i][l] = X[cands[g * gs + l]][i] (0 past the group): the step's
// candidates packed for the scan's gathers, through 32 x 32 shared-memory
// tiles.  Backward also ext[g][i] = the smallest and largest value of column i
// over the group's candidates, each centred on its feature's mean (so that
// features on different levels share a useful range) with directed rounding;
// NaN values are left out, their distances never pass.
__global__ void __launch_bounds__(256) k_pack_groups(Bufs b, int n_cand, int gs, int backward)
{
    __shared__ float tile[32][33];
    if (b.st->done) return;
    const int i0 = blockIdx.x * 32, g = blockIdx.y;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int k = ty; k < 32; k += 8) {
        const int slot = g * gs + k;
        tile[k][tx] = k < gs && slot < n_cand ? __ldg(b.XT + (size_t)__ldg(b.cands + slot) * b.ldc + i0 + tx) : 0.0f;
    }
    __syncthreads();
    const bool mine = tx < gs && g * gs + tx < n_cand;
    const float mean = backward && mine ? __ldg(b.fstat + __ldg(b.cands + g * gs + tx)).x : NAN;
    for (int k = ty; k < 32; k += 8) {
        const size_t i = (size_t)g * b.ldc + i0 + k;
        const float v = tile[tx][k];
        b.xg[i * 32 + tx] = v;
        if (backward) {
            float lo = __fsub_rd(v, mean), hi = __fsub_ru(v, mean);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                lo = fminf(lo, __shfl_xor_sync(kFull, lo, o));
                hi = fmaxf(hi, __shfl_xor_sync(kFull, hi, o));
            }
            if (tx == 0) b.ext[i] = make_float2(lo, hi);
        }
    }
}

int sm_count_scan()
{
    static const int n = [] {  // initialised once, thread-safely
        int dev = 0, c = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
        return c > 0 ? c : 148;
    }();
    return n;
}

// At most one wave of warps at 28 per SM: a warp's chain of work is the kernel's
// time.  Long lists leave shared memory for fewer warps, four at k = 150, so there
// these rows are several waves, but the batches of 16 are the better ones all the
// same: scoring of six steps of 8,192 columns, k = 20, 50, 150, 256, with 500 rows
// forward 1.0, 1.6, 3.3, 6.0 against 1.7, 2.7, 5.3, 8.5 ms in batches of 4, with
// 4,096 rows 1.9, 3.9, 15.1, 28.0 against 2.6, 4.8, 18.5, 39.3, backward 2.7, 4.9,
// 14.3, 25.2 against 5.8, 5.8, 18.2, 38.8.
bool one_wave(const Bufs &b, int n_cand)
{
    return (long long)b.n_rows * scan_groups(n_cand) <= (long long)sm_count_scan() * kWarpsMany;
}

struct ScanCall {
    int n_cand;
    bool own;       // the kernel finds the seed columns itself
    bool gated;     // return at once if State::full_scan is set
    bool probe;     // only the probe's estimate
    int max_smem;
    cudaStream_t stream;
};

template <bool BWD, int SEED, int BATCH>
cudaError_t launch_batch(const Bufs &b, const ScanCall &c)
{
    const int G = scan_groups(c.n_cand), gs = scan_group_size(c.n_cand);
    int warps = 1;
    if (BATCH == kBatchFew && SEED > 0 && !scan_leaves_walks(b, c.n_cand, BWD)) {  // who walks is one warp's choice
        const long long room = (long long)sm_count_scan() * kWarpsMany / ((long long)b.n_rows * G);
        const int passes = (b.ldc + kCols - 1) / kCols;
        warps = (int)(room < kMaxSplit ? room : kMaxSplit);
        if (warps > passes) warps = passes;
    }
    const size_t smem = warps * warp_smem(b.kmax, BATCH, 1 + (BWD ? 1 : 0) + (SEED == kSeedHeap || (SEED > 0 && b.near_list) ? 1 : 0));
    const int probe_rows = G > kProbeWarps / kProbeRows ? (G < kProbeWarps ? kProbeWarps / G : 1) : kProbeRows;
    long long blocks = (long long)(c.probe ? probe_rows : b.n_rows) * G;
    if (c.probe && blocks > kProbeWarps) blocks = kProbeWarps;  // the first groups speak for the others
    if (smem > (size_t)c.max_smem || blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const int walks = scan_leaves_walks(b, c.n_cand, BWD);
    if (walks && !c.probe) {
        const cudaError_t e = cudaMemsetAsync(b.n_walk, 0, sizeof(int), c.stream);
        if (e != cudaSuccess) return e;
    }
    auto kern = k_scan<BWD, SEED, BATCH>;
    // The limit belongs to the function, not to this call, and an instance serves
    // many sizes: every call sets the same value, so that threads with other list
    // lengths do not take it away between here and the launch.
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, c.max_smem);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)blocks, 32 * warps, smem, c.stream>>>(b, c.n_cand, G, gs, walks, c.own ? 1 : 0, c.gated ? 1 : 0,
                                                   c.probe ? b.n_rows / probe_rows : 0);
    return cudaGetLastError();
}

template <bool BWD, int SEED>
cudaError_t launch_seeded(const Bufs &b, const ScanCall &c)
{
    return one_wave(b, c.n_cand) ? launch_batch<BWD, SEED, kBatchFew>(b, c) : launch_batch<BWD, SEED, kBatchMany>(b, c);
}

cudaError_t launch_any(const Bufs &b, int backward, int seeding, const ScanCall &c)
{
    if (backward) return seeding == kNoSeeds ? launch_seeded<true, kSeedNone>(b, c) : launch_seeded<true, kSeedHeap>(b, c);
    // lists of up to 16: bounds from group minima; longer ones start from the seeds themselves
    if (c.own || b.kmax > 16) return launch_seeded<false, kSeedHeap>(b, c);
    if (b.kmax <= 8) return launch_seeded<false, 8>(b, c);
    if (b.kmax <= 12) return launch_seeded<false, 12>(b, c);
    return launch_seeded<false, 16>(b, c);
}

}  // namespace

// One wave of warps gains from pruning even if every column is open (its time
// is one warp's chain of work: step 1 of a 3000-row CV problem, everything
// open, 0.36 against 0.58 ms), and lists above 64 have no dense scorer that
// comes near.
bool scan_worth_probing(const Bufs &b, int n_cand)
{
    return b.kmax <= 64 && b.n_cols >= 1024 && b.n_rows >= kProbeRows && !one_wave(b, n_cand);
}

bool scan_leaves_walks(const Bufs &b, int n_cand, int backward)
{
    return !backward && b.sval && b.kmax <= 64 && b.n_cols >= 4096 && (long long)n_cand * b.n_rows < 0x7fffffffLL;
}

cudaError_t launch_pack_groups(const Bufs &b, int n_cand, int backward, cudaStream_t s)
{
    k_pack_groups<<<dim3(b.ldc / 32, scan_groups(n_cand)), 256, 0, s>>>(b, n_cand, scan_group_size(n_cand), backward);
    return cudaGetLastError();
}

cudaError_t launch_scan(const Bufs &b, int n_cand, int backward, int seeding, bool gated, int max_smem, cudaStream_t s)
{
    return launch_any(b, backward, seeding, {n_cand, seeding == kOwnSeeds, gated, false, max_smem, s});
}

cudaError_t launch_scan_probe(const Bufs &b, int n_cand, int backward, int seeding, int max_smem, cudaStream_t s)
{
    return launch_any(b, backward, seeding, {n_cand, seeding == kOwnSeeds, false, true, max_smem, s});
}

}  // namespace snn
