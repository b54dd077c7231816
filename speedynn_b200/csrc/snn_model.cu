// snn_model.cu -- classification predictions and the reference's loss
// functions over every (candidate, k) prediction vector.
//
// Regression predictions (kNN means) come from the scoring kernels.  For the
// classification model (speedynn/lib/cpu.c:70-95) k_mode_predict replaces
// them with the mode of the k nearest labels, using the reference's rule
// (speedynn/lib/util.c:165-188): every label counts towards its first
// occurrence in rank order, and the first position with the strictly largest
// count wins.  k_losses evaluates the requested losses of
// speedynn/lib/loss_functions.c:6-183 with the reference's float/double
// operation order; loss 0 of the list decides best k and winner, as in
// cpu.c:104-120 and nearest_neighbors_feature_selection.c:316-330.
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "snn_internal.h"

namespace snn {

namespace {

// One thread per (candidate slot, scored row).  idx holds the row's k_max
// nearest training points in rank order.
__global__ void k_mode_predict(Bufs b, int n_cand)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)n_cand * b.n_rows) return;
    const int slot = (int)(t / b.n_rows), r = (int)(t % b.n_rows);
    const int *idx = b.nn_idx + ((size_t)slot * b.n_rows + r) * b.kmax;
    for (int m = 0; m < b.nk; ++m) {
        const int k = b.kvals[m];
        int best = 0, best_cnt = -1;
        // count of position i = number of j in [i, k) whose label first occurs at i
        for (int i = 0; i < k; ++i) {
            const float yi = __ldg(b.yc + idx[i]);
            bool first = true;
            for (int j = 0; j < i && first; ++j) first = __ldg(b.yc + idx[j]) != yi;
            if (!first) continue;  // counted at its first occurrence
            int cnt = 0;
            for (int j = i; j < k; ++j) cnt += __ldg(b.yc + idx[j]) == yi;
            if (cnt > best_cnt) {  // the first strict maximum in position order
                best_cnt = cnt;
                best = i;
            }
        }
        b.pred[((size_t)slot * b.nk + m) * b.n_rows + r] = __ldg(b.yc + idx[best]);
    }
}

// Order-preserving key of a float (NaN above +inf).
__device__ __forceinline__ uint32_t fkey(float v)
{
    const uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }

// Shared memory of a loss evaluation.
struct LossShared {
    uint32_t hist[256];
    uint32_t word[2];
    __align__(16) float term[1024];
    float sum;
    unsigned miss;
};

// Element of rank `rank` (0-based, ascending) of the n values val(i), by a
// most-significant-digit radix select over the keys; the whole block calls it.
// Lanes with the same digit add to its bin together (a classification's errors
// take a handful of values), and one warp searches the bins.
template <class F>
__device__ float block_select(int n, int rank, F val, LossShared &S)
{
    const int lane = threadIdx.x & 31;
    uint32_t prefix = 0u, mask = 0u;
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int d = threadIdx.x; d < 256; d += blockDim.x) S.hist[d] = 0u;
        __syncthreads();
        for (int i0 = 0; i0 < n; i0 += blockDim.x) {
            const int i = i0 + threadIdx.x;
            const uint32_t key = i < n ? fkey(val(i)) : 0u;
            const bool in = i < n && (key & mask) == prefix;
            const unsigned act = __ballot_sync(0xffffffffu, in);
            if (in) {
                const uint32_t d = (key >> shift) & 255u;
                const unsigned same = __match_any_sync(act, d);
                if (lane == __ffs(same) - 1) atomicAdd(S.hist + d, (uint32_t)__popc(same));
            }
        }
        __syncthreads();
        if (threadIdx.x < 32) {  // eight bins per lane
            uint32_t c[8], own = 0u;
#pragma unroll
            for (int q = 0; q < 8; ++q) own += c[q] = S.hist[8 * lane + q];
            uint32_t incl = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            uint32_t below = incl - own;
            if ((uint32_t)rank >= below && (uint32_t)rank < incl) {
                int q = 0;
#pragma unroll
                for (int e = 0; e < 7; ++e)
                    if (q == e && (uint32_t)rank >= below + c[e]) {
                        below += c[e];
                        ++q;
                    }
                S.word[0] = (uint32_t)(8 * lane + q);
                S.word[1] = (uint32_t)rank - below;
            }
        }
        __syncthreads();
        prefix |= S.word[0] << shift;
        mask |= 255u << shift;
        rank = (int)S.word[1];
        __syncthreads();
    }
    return fkey_inv(prefix);
}

// Sequential FP32 sum of term(0..n-1); the whole block calls it.  All threads
// form the terms, one adds them in order (one thread doing both waited for
// memory and a double division per row: 545 us for three losses of 2,501 rows,
// now 30).
template <class F>
__device__ float block_sum(int n, F term, LossShared &S)
{
    float sum = 0.0f;
    for (int i0 = 0; i0 < n; i0 += 1024) {
        const int cnt = min(1024, n - i0);
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) S.term[i] = term(i0 + i);
        __syncthreads();
        if (threadIdx.x == 0) {
            const float4 *v = reinterpret_cast<const float4 *>(S.term);
            int i = 0;
            for (; i + 16 <= cnt; i += 16) {
                float4 f[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) f[u] = v[(i >> 2) + u];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, f[u].x), f[u].y), f[u].z), f[u].w);
            }
            for (; i < cnt; ++i) sum = __fadd_rn(sum, S.term[i]);
            S.sum = sum;
        }
        __syncthreads();
    }
    return S.sum;
}

// speedynn/lib/loss_functions.c:88-111 (norm) and :66-86: median of the
// errors, then median of their distances to it (find_median = element n/2 of
// the sorted array, :173-183).
__device__ float mad_value(const float *pred, const float *y, int n, bool norm, LossShared &S)
{
    auto err = [&](int i) {
        const float t = y[i];
        const float d = __fsub_rn(t, pred[i]);
        return norm ? (float)__ddiv_rn((double)d, __dadd_rn(1.0, (double)t)) : d;
    };
    const float m1 = block_select(n, n / 2, err, S);
    auto dev = [&](int i) { return fabsf(__fsub_rn(err(i), m1)); };
    return block_select(n, n / 2, dev, S);
}

// The losses below are called by the whole block and valid in every thread.
__device__ float rmse_norm_value(const float *pred, const float *y, int n, LossShared &S)
{
    const float sum = block_sum(
        n,
        [&](int j) {
            const int i = n - 1 - j;  // loss_functions.c:55, descending
            const float t = y[i];
            const float tmp = (float)__ddiv_rn((double)__fsub_rn(t, pred[i]), __dadd_rn(1.0, (double)t));
            return __fmul_rn(tmp, tmp);
        },
        S);
    return (float)sqrt((double)__fdiv_rn(sum, (float)n));
}

__device__ float std_value(const float *pred, const float *y, int n, LossShared &S)
{
    const float mean = __fdiv_rn(block_sum(n, [&](int i) { return __fsub_rn(y[i], pred[i]); }, S), (float)n);
    // loss_functions.c:141 assigns instead of accumulating: only the last row counts
    const float a = __fsub_rn(__fsub_rn(y[n - 1], pred[n - 1]), mean);
    const float sum = __fdiv_rn(__fmul_rn(a, a), (float)(n - 1));
    return (float)sqrt((double)sum);
}

__device__ float rmse_value(const float *pred, const float *y, int n, LossShared &S)
{
    const float sum = block_sum(
        n,
        [&](int i) {
            const float tmp = __fsub_rn(y[i], pred[i]);
            return __fmul_rn(tmp, tmp);
        },
        S);
    return (float)sqrt((double)__fdiv_rn(sum, (float)n));
}

// loss_functions.c:113-127 passes the float difference to int abs(): on the
// host this truncates towards zero (x86 cvttss2si), and a difference that
// does not fit an int (or NaN) becomes INT_MIN, whose abs() stays negative.
// So a row counts as a miss iff 1 <= |t - p| < 2^31.
__device__ __forceinline__ unsigned zero_one_miss(float t, float p)
{
    const float a = fabsf(__fsub_rn(t, p));
    return (a >= 1.0f && a < 2147483648.0f) ? 1u : 0u;
}

// One block per (candidate slot, k index) and requested loss: that loss of that
// prediction vector into lossval[(l * n_cand + slot) * nk + m].  A non-RMSE
// deciding loss (index 0) also replaces rmse32/rmse64, which best k and the
// winner are chosen from (no other block reads them then).
__global__ void __launch_bounds__(256) k_losses(Bufs b, int n_cand, int l0)
{
    __shared__ LossShared S;
    if (b.st->done) return;  // nothing was predicted
    const int slot = blockIdx.x / b.nk, m = blockIdx.x % b.nk, l = l0 + blockIdx.y;
    const int n = b.n_rows;
    const float *pred = b.pred + ((size_t)slot * b.nk + m) * n;
    const float *y = b.yr;
    const int id = b.loss_ids[l];
    float v = NAN;
    if (id == 2 || id == 3) {
        v = mad_value(pred, y, n, id == 3, S);
    } else if (id == 6 || id == 7) {
        const float md = mad_value(pred, y, n, true, S), rn = rmse_norm_value(pred, y, n, S);
        if (id == 6) {
            const float sd = std_value(pred, y, n, S);
            v = (float)__dadd_rn(__dadd_rn(__ddiv_rn((double)rn, 0.19), __ddiv_rn((double)md, 0.041)),
                                 __ddiv_rn((double)sd, 0.16));
        } else {
            v = (float)__dadd_rn(__ddiv_rn((double)rn, 0.019), __ddiv_rn((double)md, 0.009));
        }
    } else if (id == 4) {
        if (threadIdx.x == 0) S.miss = 0u;
        __syncthreads();
        unsigned c = 0u;
        for (int i = threadIdx.x; i < n; i += blockDim.x) c += zero_one_miss(y[i], pred[i]);
        atomicAdd(&S.miss, c);
        __syncthreads();
        v = __fdiv_rn((float)S.miss, (float)n);  // adding 1.0f once per miss in row order is exact below 2^24 misses
    } else if (id == 0) {
        // rmse32 holds the RMSE unless a non-RMSE loss 0 replaces it
        v = b.loss_ids[0] == 0 ? b.rmse32[slot * b.nk + m] : rmse_value(pred, y, n, S);
    } else if (id == 1) {
        v = rmse_norm_value(pred, y, n, S);
    } else if (id == 5) {
        v = std_value(pred, y, n, S);
    } else if (id == 8) {
        const float rm = rmse_value(pred, y, n, S);
        v = __fadd_rn(rm, std_value(pred, y, n, S));
    }
    if (threadIdx.x == 0) {
        b.lossval[((size_t)l * n_cand + slot) * b.nk + m] = v;
        if (l == 0 && id != 0) {
            b.rmse32[slot * b.nk + m] = v;
            b.rmse64[slot * b.nk + m] = (double)v;
        }
    }
}

}  // namespace

cudaError_t launch_mode_predict(const Bufs &b, int n_cand, cudaStream_t s)
{
    const long long n = (long long)n_cand * b.n_rows;
    if (n <= 0) return cudaSuccess;
    k_mode_predict<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(b, n_cand);
    return cudaGetLastError();
}

cudaError_t launch_losses(const Bufs &b, int n_cand, cudaStream_t s)
{
    if (n_cand <= 0) return cudaSuccess;
    constexpr int kGridY = 65535;  // longer loss lists take several launches
    for (int l0 = 0; l0 < b.nloss; l0 += kGridY) {
        const int nl = b.nloss - l0 < kGridY ? b.nloss - l0 : kGridY;
        k_losses<<<dim3(n_cand * b.nk, nl), 256, 0, s>>>(b, n_cand, l0);
    }
    return cudaGetLastError();
}

}  // namespace snn
