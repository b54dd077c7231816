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
// One warp per (scored row, group of up to 32 candidates), lane = candidate:
//   * the warp streams its row of D, 512 columns at a time, and queues the
//     columns that any of its candidates may still take (the sign of D - H, H
//     the group's largest bound, which falls as the lists fill);
//   * queued columns are taken eight at a time, their candidate values gathered
//     together from `xg`, the candidates packed [group][column][32] (one aligned
//     128-byte line per column and group, so a gather is one full-width load);
//     every lane forms its candidate's exact distance and appends it to its
//     own buffer in shared memory if it may enter the list;
//   * when a lane's buffer is nearly full, all lanes empty theirs together into
//     their lists, heaps of k_max (distance, column) keys in shared memory.  The
//     keys are ordered by distance, then column, which is the reference's
//     stable rule in whatever order the columns arrive;
//   * forward, a row that is an outlier in some features leaves those
//     candidates' bounds far above the others'.  Such candidates ("wide") are
//     kept out of H and scanned with lane = column instead; the split minimises
//     the cost estimated from 256 sampled columns;
//   * backward, H takes each candidate's largest possible s on the row; a
//     queued column is tested once more, with the group's extreme values in
//     that column (`ext`), before it is gathered.
// The insertion, the gather and the column test each stand once in the loop:
// with the insertion unrolled at every use the kernel waited for instructions
// 80 % of the time.
//
// What bounds it: instruction issue (59 % of the slots on a 16,384 x 8,192 step
// with 14 warps per SM, each waiting for its own chain) well above the D stream
// (fwd-64k: 3 ms per late step, 1.3 ms of it the read of D).  Scoring of a whole
// fwd-64k selection 293 -> 80 ms, a step of bwd-50k's quarter size 7.0 -> 1.4 ms,
// a k = 150 step of 8,192 x 4,096 x 19 130 -> 8 ms.
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "snn_internal.h"

namespace snn {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kUnroll = 4;             // float4 loads of D per lane and pass of the loop
constexpr int kCols = 128 * kUnroll;   // columns per pass of the loop
constexpr int kQueue = 1024;           // entries of a warp's column queue (a power of two, above kCols + kBatch)
constexpr int kBatch = 8;              // queued columns gathered together
constexpr int kBuf = 16;               // distances a lane buffers before they enter its heap
constexpr int kTagShift = 26;          // queue entry: column, and above it 1 + lane of a wide candidate (0: the others)
constexpr int kWarps = 1;              // warps per block: they finish at different times

// Order-preserving signed key of a float (no NaN), and back.
__device__ __forceinline__ int fkey(float v)
{
    const int u = __float_as_int(v);
    return u ^ ((u >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float fkey_inv(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

// List keys: (distance, column) as one unsigned 64-bit number.
__device__ __forceinline__ unsigned long long pack_key(float d, int col)
{
    return ((unsigned long long)((unsigned)fkey(d) ^ 0x80000000u) << 32) | (unsigned)col;
}
__device__ __forceinline__ float key_dist(unsigned long long k) { return fkey_inv((int)((unsigned)(k >> 32) ^ 0x80000000u)); }

// Replace the root of the lane's max-heap h[0], h[32], ... (n entries) by key.
__device__ __forceinline__ void sift_down(unsigned long long *h, int n, unsigned long long key)
{
    int i = 0;
    for (;;) {
        int l = 2 * i + 1;
        if (l >= n) break;
        unsigned long long kl = h[l * 32];
        if (l + 1 < n) {
            const unsigned long long kr = h[(l + 1) * 32];
            if (kr > kl) {
                kl = kr;
                ++l;
            }
        }
        if (key >= kl) break;
        h[i * 32] = kl;
        i = l;
    }
    h[i * 32] = key;
}

// Shared memory of a warp: heaps and buffers of 32 lanes, column queue(s).
size_t warp_smem(int K, bool bwd)
{
    return sizeof(unsigned long long) * 32 * (size_t)(K + kBuf) + sizeof(int) * (size_t)kQueue * (bwd ? 2 : 1);
}

template <bool BWD>
__global__ void __launch_bounds__(32 * kWarps, 20) k_scan(Bufs b, int n_cand, int G, int gs, int wsmem, int wide_cost)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    if (b.st->done) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gw = blockIdx.x * (blockDim.x >> 5) + w;
    const int r = gw / G, g = gw % G;
    if (r >= b.n_rows) return;  // warp-uniform; nothing below synchronises the block
    const int K = b.kmax;
    unsigned long long *heap = reinterpret_cast<unsigned long long *>(smraw + (size_t)w * wsmem) + lane;
    unsigned long long *buf = heap + (size_t)K * 32;
    int *queue = reinterpret_cast<int *>(smraw + (size_t)w * wsmem + sizeof(unsigned long long) * 32 * (size_t)(K + kBuf));
    int *wait = queue + kQueue;  // backward: columns before the second test

    const int slot = g * gs + lane;
    const bool live = lane < gs && slot < n_cand;
    const int c = live ? __ldg(b.cands + slot) : 0;
    float xv = live ? __ldg(b.XV + (size_t)c * b.ldr + r) : NAN;
    const bool act = isfinite(xv);  // otherwise no distance of this candidate is below FLT_MAX
    if (!act) xv = NAN;             // never passes
    const size_t cr = (size_t)c * b.n_rows + r;
    const float *xg = b.xg + (size_t)g * b.ldc * 32 + lane;
    const float *Dr = b.D + (size_t)r * b.ldc;

    // lim: distances above it cannot enter the lane's list.  The list starts as K
    // sentinels at the (inclusive) bound, ordered after every column; those left
    // at the end are padding.
    float lim = -INFINITY;
    if (act) {
        lim = BWD ? b.kth_prev[cr] : b.bound[cr];
        if (!(lim < FLT_MAX)) lim = 0x1.fffffcp+127f;  // items at FLT_MAX never enter
    }
    for (int j = 0; j < K; ++j) heap[j * 32] = pack_key(lim, -1);

    const float4 *row = reinterpret_cast<const float4 *>(Dr);
    const int n4 = b.ldc >> 2;
    float4 nxt[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
        const int q = u * 32 + lane;
        nxt[u] = q < n4 ? __ldg(row + q) : make_float4(INFINITY, INFINITY, INFINITY, INFINITY);
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

    // Forward: which candidates are scanned with lane = column (wide): the cut
    // with the least estimated cost.  A wide candidate costs wide_cost sampled
    // columns, any other the sampled columns within its bound, the group the
    // most of them (launch_dir has the figures).
    unsigned wide = 0u;
    if constexpr (!BWD) {
        if (wide_cost > 0) {
            float smp[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) smp[i] = __ldg(Dr + (size_t)i * (b.n_cols / 8) + lane);
            int cnt = 0;  // sampled columns within the lane's bound
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll 4
                for (int l = 0; l < 32; ++l) cnt += __shfl_sync(kFull, smp[i], l) <= lim ? 1 : 0;
            int above = 0;  // candidates with more columns than this lane's
#pragma unroll 4
            for (int l = 0; l < 32; ++l) above += __shfl_sync(kFull, cnt, l) > cnt ? 1 : 0;
            const int best = __reduce_min_sync(kFull, ((wide_cost * above + cnt) << 9) | cnt);  // cost, then the cut
            wide = __ballot_sync(kFull, cnt > (best & 511));
        }
    }
    const bool reg = !((wide >> lane) & 1u);

    // No column with D >= H can enter a list of the queue's candidates: forward
    // d >= D; backward d <= lim means D - s < nextafter(lim) exactly (rounding is
    // monotone), and s <= smax.  kmx: the same for the second test.
    float H;
    auto update_H = [&] {
        if constexpr (BWD) {
            const float up = nextafterf(lim, INFINITY);
            H = __int_as_float(__reduce_max_sync(kFull, __float_as_int(fmaxf(__fadd_ru(up, smax), 0.0f))));
            kmx = fkey_inv(__reduce_max_sync(kFull, fkey(up)));
        } else {
            H = __int_as_float(__reduce_max_sync(kFull, reg ? __float_as_int(fmaxf(lim, 0.0f)) : 0) + 1);
        }
    };
    update_H();

    // Each lane appends the columns of its 16-bit mask (bit 4u + e: column
    // q0 + 128 u + 4 lane + e), in no particular order.
    auto push = [&](int *q, int tail, unsigned m16, int q0, int tag) {
        int n = 0;
        for (unsigned any = __ballot_sync(kFull, m16 != 0u); any; any = __ballot_sync(kFull, m16 != 0u)) {
            if (m16) {
                const int i = __ffs(m16) - 1;
                m16 &= m16 - 1;
                q[(tail + n + __popc(any & ((1u << lane) - 1u))) & (kQueue - 1)] =
                    (q0 + 128 * (i >> 2) + 4 * lane + (i & 3)) | tag;
            }
            n += __popc(any);
        }
        return n;
    };

    int qh = 0, qn = 0;  // queue: first entry, entries
    int ah = 0, an = 0;  // backward: columns that wait for the second test
    int nb = 0;          // the lane's buffered distances
    for (int q0 = 0;; q0 += kCols) {
        const bool last = q0 >= b.ldc;  // no columns left: empty the queues and buffers
        float4 cur[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            cur[u] = nxt[u];
            const int q = (q0 >> 2) + (kUnroll + u) * 32 + lane;
            nxt[u] = q < n4 ? __ldg(row + q) : make_float4(INFINITY, INFINITY, INFINITY, INFINITY);
        }
        unsigned todo = wide;
        for (int ph = -1;;) {  // -1: the columns of the group; then one wide candidate after the other
            if (ph < 0) {
                unsigned m16 = 0u;  // sign bits of D - H, first column lowest
#pragma unroll
                for (int u = kUnroll - 1; u >= 0; --u) {
                    m16 = __funnelshift_l(__float_as_uint(__fsub_rn(cur[u].w, H)), m16, 1);
                    m16 = __funnelshift_l(__float_as_uint(__fsub_rn(cur[u].z, H)), m16, 1);
                    m16 = __funnelshift_l(__float_as_uint(__fsub_rn(cur[u].y, H)), m16, 1);
                    m16 = __funnelshift_l(__float_as_uint(__fsub_rn(cur[u].x, H)), m16, 1);
                }
                if (q0 + kCols > b.ldc) {  // past the row
#pragma unroll
                    for (int u = 0; u < kUnroll; ++u)
                        if (q0 + 128 * u + 4 * lane >= b.ldc) m16 &= ~(15u << (4 * u));
                }
                if constexpr (BWD) an += push(wait, ah + an, m16, q0, 0);
                else qn += push(queue, qh + qn, m16, q0, 0);
            } else if constexpr (!BWD) {
                const float kw = __shfl_sync(kFull, lim, ph), xl = __shfl_sync(kFull, xv, ph);
                const float4 *xc = reinterpret_cast<const float4 *>(b.XT + (size_t)__shfl_sync(kFull, c, ph) * b.ldc);
                float4 x[kUnroll];
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) {
                    const int q = (q0 >> 2) + u * 32 + lane;
                    x[u] = q < n4 ? __ldg(xc + q) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                unsigned m16 = 0u;
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) {
                    const float t0 = __fsub_rn(xl, x[u].x), t1 = __fsub_rn(xl, x[u].y), t2 = __fsub_rn(xl, x[u].z),
                                t3 = __fsub_rn(xl, x[u].w);
                    m16 |= __fadd_rn(cur[u].x, __fmul_rn(t0, t0)) <= kw ? 1u << (4 * u) : 0u;
                    m16 |= __fadd_rn(cur[u].y, __fmul_rn(t1, t1)) <= kw ? 2u << (4 * u) : 0u;
                    m16 |= __fadd_rn(cur[u].z, __fmul_rn(t2, t2)) <= kw ? 4u << (4 * u) : 0u;
                    m16 |= __fadd_rn(cur[u].w, __fmul_rn(t3, t3)) <= kw ? 8u << (4 * u) : 0u;
                }
                // past the row the sums are +inf and never at or below kw
                qn += push(queue, qh + qn, m16, q0, (int)((unsigned)(ph + 1) << kTagShift));
            }
            for (;;) {
                if constexpr (BWD) {
                    if (an >= (last ? 1 : 32)) {
                        // Second test, lane = column: an s of this column is at most U^2, U the
                        // larger of the two extreme differences (rounded up), so an entry needs
                        // D - fl(U^2) < nextafter(lim) for some candidate, and its rounding <= kmx.
                        __syncwarp();
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
                    }
                }
                while (qn >= (last ? 1 : kBatch)) {
                    // the first queued columns against every candidate of the group
                    __syncwarp();
                    const int n = min(qn, kBatch);
                    float D[kBatch], x[kBatch];
#pragma unroll
                    for (int i = 0; i < kBatch; ++i) {
                        const int col = i < n ? queue[(qh + i) & (kQueue - 1)] & ((1 << kTagShift) - 1) : 0;
                        D[i] = __ldg(Dr + col);
                        x[i] = __ldg(xg + (size_t)col * 32);
                    }
#pragma unroll
                    for (int i = 0; i < kBatch; ++i) {
                        const float t = __fsub_rn(xv, x[i]);
                        const float s = __fmul_rn(t, t);
                        const float d = BWD ? __fsub_rn(D[i], s) : __fadd_rn(D[i], s);
                        if (d <= lim && i < n) {
                            const int e = queue[(qh + i) & (kQueue - 1)];
                            const int tag = (int)((unsigned)e >> kTagShift);
                            if (BWD || (tag ? tag == lane + 1 : reg)) buf[32 * nb++] = pack_key(d, e & ((1 << kTagShift) - 1));
                        }
                    }
                    qh = (qh + n) & (kQueue - 1);
                    qn -= n;
                    if (__any_sync(kFull, nb > kBuf - kBatch) || (last && qn == 0 && an == 0)) {
                        const int most = __reduce_max_sync(kFull, nb);
                        for (int j = 0; j < most; ++j) {
                            const unsigned long long key = j < nb ? buf[32 * j] : ~0ull;
                            if (key < heap[0]) sift_down(heap, K, key);
                        }
                        nb = 0;
                        if (act) lim = key_dist(heap[0]);
                        update_H();
                    }
                }
                if (!BWD || an < (last ? 1 : 32)) break;
            }
            if (BWD || todo == 0u) break;
            ph = __ffs(todo) - 1;
            todo &= todo - 1;
        }
        if (last) break;
    }

    // Epilogue: each lane's list in ascending order, padding as (FLT_MAX, 0),
    // the k-th distance for the next backward step, the optional neighbour
    // dump, labels summed in rank order.
    if (!live) return;
    for (int j = 0; j < nb; ++j)
        if (buf[32 * j] < heap[0]) sift_down(heap, K, buf[32 * j]);
    for (int n = K - 1; n > 0; --n) {
        const unsigned long long end = heap[n * 32];
        heap[n * 32] = heap[0];
        sift_down(heap, n, end);
    }
    if (BWD) {
        const unsigned long long k = heap[(K - 1) * 32];
        b.kth_prev[cr] = (int)(unsigned)k >= 0 ? key_dist(k) : FLT_MAX;
    }
    if (b.nn_idx) {
        const size_t o = ((size_t)slot * b.n_rows + r) * K;
        for (int j = 0; j < K; ++j) {
            const unsigned long long k = heap[j * 32];
            const int i = (int)(unsigned)k;
            b.nn_idx[o + j] = i >= 0 ? i : 0;
            b.nn_dist[o + j] = i >= 0 ? key_dist(k) : FLT_MAX;
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

template <bool BWD>
cudaError_t launch_dir(const Bufs &b, int n_cand, int G, int gs, int max_smem, cudaStream_t s)
{
    int warps = kWarps;
    const size_t per = warp_smem(b.kmax, BWD);
    while (warps > 1 && per * warps > (size_t)max_smem) --warps;
    if (per * warps > (size_t)max_smem) return cudaErrorInvalidConfiguration;
    const long long total = (long long)b.n_rows * G;
    const long long blocks = (total + warps - 1) / warps;
    if (total > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    auto kern = k_scan<BWD>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(per * warps));
    if (e != cudaSuccess) return e;
    // A queued column costs about 15 instructions, a sampled column stands for
    // n / 256 of them.  A wide candidate costs n / 8 instructions and, for each
    // of the k (1 + ln(n / k)) insertions that a list sees when columns come in
    // random order, a heap operation with one lane at work (about 80).  Without
    // the second term a k = 150 step of 8,192 x 4,096 took 50 ms instead of 8,
    // the third step of a k = 50 selection from 50,021 x 24,989 86 instead of 59.
    int wide_cost = 0;
    if (!BWD && b.n_cols >= 4096) {
        const double n = b.n_cols, k = b.kmax;
        wide_cost = (int)(2.5 + 1400.0 * k * (1.0 + log(n / k > 1.0 ? n / k : 1.0)) / n);
        if (wide_cost > 256) wide_cost = 0;
    }
    kern<<<(unsigned)blocks, 32 * warps, per * warps, s>>>(b, n_cand, G, gs, (int)per, wide_cost);
    return cudaGetLastError();
}

}  // namespace

bool scan_supported(int n_cols, int kmax) { return n_cols < (1 << kTagShift) && kmax >= 1 && kmax <= kScoreMaxK; }
int scan_groups(int n_cand) { return (n_cand + 31) / 32; }
int scan_group_size(int n_cand) { return (n_cand + scan_groups(n_cand) - 1) / scan_groups(n_cand); }

cudaError_t launch_pack_groups(const Bufs &b, int n_cand, int backward, cudaStream_t s)
{
    k_pack_groups<<<dim3(b.ldc / 32, scan_groups(n_cand)), 256, 0, s>>>(b, n_cand, scan_group_size(n_cand), backward);
    return cudaGetLastError();
}

cudaError_t launch_scan(const Bufs &b, int n_cand, int backward, int max_smem, cudaStream_t s)
{
    const int G = scan_groups(n_cand), gs = scan_group_size(n_cand);
    return backward ? launch_dir<true>(b, n_cand, G, gs, max_smem, s) : launch_dir<false>(b, n_cand, G, gs, max_smem, s);
}

}  // namespace snn
