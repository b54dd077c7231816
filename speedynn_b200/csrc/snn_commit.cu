// snn_commit.cu -- commit the winning feature into the distance matrix.
//
// k_commit: D <- fl(D +/- fl((x_r,w - x_i,w)^2)) in place for the winner w of
// the step that just ran (read from the device state, so the host never waits
// for it): speedynn/lib/cpu.c:217-231 and
// kernels/update_current_distance_matrix_float.cl:5-32, with the product and
// the sum rounded separately.  A warp streams one row with 16-byte loads and
// stores (HBM-bound: 8 bytes per entry).
//
// Seeds (forward steps only).  While it streams a row, each lane also keeps,
// for each of eight parts of the columns it visits (the four places of the
// float4 groups l, l+32, l+64, ... in either half of the row), the smallest new
// distance, so every row leaves 256 distinct real columns that lie near it
// under the committed features: seeds[r][j*32+l] and their distances
// seed_d[r][j*32+l] (lane l's j-th smallest; index -1 and +inf where a part has
// no finite distance).  The next forward scoring step bounds each candidate's
// k-th neighbour distance by distances over these columns (any k distinct
// columns bound it; near ones bound it tightly).  A minimum costs three
// instructions per column and no branch; the eight smallest of all the lane's
// columns are only a little nearer (fwd-64k, step 8: 0.06 against 0.07 % of the
// columns within the median candidate's bound), but their insertion ran for
// almost every group of some lane (a forward commit of 65,536 x 32,768 3.1 -> 2.8
// ms, 2.7 without seeds; of 5,003 x 2,501 59 -> 16 us).
#include <float.h>
#include <math.h>

#include "snn_internal.h"
#include "snn_packed.cuh"

namespace snn {

namespace {

__device__ __forceinline__ float sqdiff(float a, float b)
{
    const float t = __fsub_rn(a, b);
    return __fmul_rn(t, t);
}

// A lane's seeds of row r, ascending by distance, to their arrays.
__device__ __forceinline__ void store_seeds(float (&sv)[kSeedsPerLane], int (&si)[kSeedsPerLane], int *seeds, float *seed_d, int r,
                                            int lane)
{
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
#pragma unroll
    for (int j = 0; j < kSeedsPerLane; ++j) {
        seeds[(size_t)r * kSeeds + j * 32 + lane] = si[j];
        seed_d[(size_t)r * kSeeds + j * 32 + lane] = sv[j];
    }
}

// The middle and the largest of the lanes' sorted seeds, averaged: about the
// row's 172nd and 680th smallest distance; their power law goes on to the
// 1,024th (snn_scan.cu).  From these, what the next commit lists by: that
// distance, grown by 1.1 times what the last feature added (`last`: the same of
// the commit before, 0 on the first one, also after a warm start).  The factors
// are fitted to normal data; on others fewer lists may be usable (snn_get_near_lists),
// which costs time and nothing else.  The first features change the dimension most: on normal
// data the n-th part of the columns reaches about n times as far under two
// features as under one, and 4.5 times as far under three as under two (the
// median rows of fwd-64k and fwd-200k 72 and 50 for n of 64 and 49, then 5.1 and
// 4.4).  On those data 70 to 99 % of the lists hold 256 to kNearList columns,
// except after the fifth feature of fwd-200k (40 %).
__device__ __forceinline__ float4 near_of(const float (&sv)[kSeedsPerLane], float last, int n_cols)
{
    float mid = 0.5f * (sv[3] + sv[4]), far = sv[kSeedsPerLane - 1];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mid += __shfl_xor_sync(0xffffffffu, mid, o);
        far += __shfl_xor_sync(0xffffffffu, far, o);
    }
    const float near = far * 0.03125f * powf(far / mid, 0.298f);  // ln(1024 / 680) / ln(680 / 172)
    const float grow = !(last > 0.0f)         ? (float)n_cols * (1.0f / 800.0f)
                       : near > 8.0f * last ? 4.5f
                                            : 1.0f + 1.1f * fmaxf(near - last, 0.0f) / near;
    return make_float4(near, near * grow, mid * 0.03125f * grow, 0.0f);
}

// Three blocks of 256 threads per SM, each lane with four float4 loads of D in
// flight: the stream needs that many bytes in flight to stay HBM-bound (four
// blocks with two loads per lane while the seed lists take registers: 44.0
// against 43.0 ms of commits per fwd-64k selection).  LIST writes down the row's
// near columns on the way: 38.8 -> 41.0 ms of commits, 64.5 -> 49.6 of scoring.
template <bool BWD, bool SEEDS, bool LIST>
__global__ void __launch_bounds__(256, 3) k_commit(Bufs b, int *seeds, float *seed_d)
{
    if (b.st->done) return;
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const int w = b.st->winner;
    const float *xt = b.XT + (size_t)w * b.ldc;
    const float *xv = b.XV + (size_t)w * b.ldr;
    const float4 *xt4 = reinterpret_cast<const float4 *>(xt);
    const int n4 = b.ldc >> 2;
    constexpr int U = 4;  // float4 loads per lane in flight
    constexpr int H = SEEDS ? 2 : 1;  // parts of the row
    const int part = SEEDS ? ((n4 / 2 + 32 * U - 1) / (32 * U)) * (32 * U) : n4;
    for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < b.n_rows; r += gridDim.x * wpb) {
        const float a = __ldg(xv + r);
        float4 *row = reinterpret_cast<float4 *>(b.D + (size_t)r * b.ldc);
        float sv[kSeedsPerLane];
        int si[kSeedsPerLane];
#pragma unroll
        for (int j = 0; j < kSeedsPerLane; ++j) {
            sv[j] = INFINITY;
            si[j] = -1;
        }
        float4 by;
        int found = 0;  // columns below by.y
        int2 *list = nullptr;
        if (LIST) {
            by = b.near_next[r];
            list = b.near_list + (size_t)r * kNearList;
        }
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int end = h + 1 < H ? min(part, n4) : n4;
            for (int q0 = h * part; q0 < end; q0 += 32 * U) {
                float4 d[U], c[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int q = q0 + u * 32 + lane;
                    if (q < end) {
                        d[u] = __ldcs(row + q);
                        c[u] = __ldg(xt4 + q);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int q = q0 + u * 32 + lane;
                    if (q < end) {
                        if (BWD) {
                            d[u].x = __fsub_rn(d[u].x, sqdiff(a, c[u].x));
                            d[u].y = __fsub_rn(d[u].y, sqdiff(a, c[u].y));
                            d[u].z = __fsub_rn(d[u].z, sqdiff(a, c[u].z));
                            d[u].w = __fsub_rn(d[u].w, sqdiff(a, c[u].w));
                        } else {
                            d[u].x = __fadd_rn(d[u].x, sqdiff(a, c[u].x));
                            d[u].y = __fadd_rn(d[u].y, sqdiff(a, c[u].y));
                            d[u].z = __fadd_rn(d[u].z, sqdiff(a, c[u].z));
                            d[u].w = __fadd_rn(d[u].w, sqdiff(a, c[u].w));
                        }
                        __stcs(row + q, d[u]);
                        if (SEEDS) {
                            const float v[4] = {d[u].x, d[u].y, d[u].z, d[u].w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const int j = (4 * h + e) & (kSeedsPerLane - 1);
                                const bool near = v[e] < sv[j];  // strict: +inf and NaN never enter
                                sv[j] = near ? v[e] : sv[j];
                                si[j] = near ? q : si[j];
                            }
                        }
                    }
                }
                if (LIST) {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int q = q0 + u * 32 + lane;
                        const float v[4] = {d[u].x, d[u].y, d[u].z, d[u].w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const bool in = q < end && v[e] < by.y;
                            const unsigned m = __ballot_sync(0xffffffffu, in);
                            if (m) {
                                const int at = found + __popc(m & ((1u << lane) - 1u));
                                if (in && at < kNearList) list[at] = make_int2(4 * q + e, __float_as_int(v[e]));
                                found += __popc(m);
                            }
                        }
                    }
                }
            }
        }
        if (SEEDS) {
            // the float4 group of part 4 h + e -> its column
#pragma unroll
            for (int j = 0; j < kSeedsPerLane; ++j) si[j] = si[j] < 0 ? -1 : 4 * si[j] + (j & 3);
            store_seeds(sv, si, seeds, seed_d, r, lane);
            if (b.near_next) {
                const float4 next = near_of(sv, LIST ? by.x : 0.0f, b.n_cols);
                if (lane == 0) {
                    b.near_next[r] = next;
                    if (LIST) b.near_info[r] = make_float4(by.y < FLT_MAX ? (float)found : INFINITY, by.y, by.z, 0.0f);
                }
            }
        }
    }
}

// k_commit_seq: several known features at once (a warm start).  One commit per
// feature moves all of D twice for each; here a row's entry stays in a register
// while the features are added in their order with the same roundings, and a
// forward start from the empty matrix writes D without reading it.  Sixteen
// warps, a row each, share the features' values of 512 columns through shared
// memory (from L2 every row would fetch 4 bytes per feature and entry), two
// buffers filled by cp.async.  Seven features of a 65,536 x 32,768 matrix:
// 3.1 ms, 20.9 with the reset and seven commits (3.8 without packed pairs); its
// write alone takes 1.4.
constexpr int kSeqWarps = 16, kSeqCols = 512;

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(gmem) : "memory");
}

template <bool BWD, bool SEEDS, bool START>
__global__ void __launch_bounds__(32 * kSeqWarps, 2) k_commit_seq(Bufs b, const __grid_constant__ FeatureSeq seq, int cv,
                                                                   int npf, int *seeds, float *seed_d)
{
    extern __shared__ __align__(16) float xs[];  // [2][kFeatureSeq][kSeqCols]
    __shared__ float as[kSeqWarps][kFeatureSeq];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int r = blockIdx.x * kSeqWarps + w;
    const bool row_in = r < b.n_rows;
    if (row_in && lane < seq.n) as[w][lane] = __ldg(b.XV + (size_t)seq.f[lane] * b.ldr + r);
    const int lo = cv && row_in ? (r / npf) * npf : 0;
    const int n4 = b.ldc >> 2, chunks = (b.ldc + kSeqCols - 1) / kSeqCols;
    const int half = (chunks + 1) / 2;  // seeds: each place of the float4 groups, either half of the row
    auto fetch = [&](int c, int buf) {
        for (int e = threadIdx.x; e < seq.n * (kSeqCols / 4); e += 32 * kSeqWarps) {
            const int f = e / (kSeqCols / 4), q = c * (kSeqCols / 4) + e % (kSeqCols / 4);
            if (q < n4)
                cp_async16(xs + ((size_t)buf * kFeatureSeq + f) * kSeqCols + 4 * (e % (kSeqCols / 4)),
                           b.XT + (size_t)seq.f[f] * b.ldc + 4 * (size_t)q);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float sv[kSeedsPerLane];
    int si[kSeedsPerLane];
#pragma unroll
    for (int j = 0; j < kSeedsPerLane; ++j) {
        sv[j] = INFINITY;
        si[j] = -1;
    }
    fetch(0, 0);
    for (int c = 0; c < chunks; ++c) {
        if (c + 1 < chunks) fetch(c + 1, (c + 1) & 1);
        if (c + 1 < chunks) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (row_in) {
            float4 *row = reinterpret_cast<float4 *>(b.D + (size_t)r * b.ldc);
            float4 d[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int q = c * (kSeqCols / 4) + u * 32 + lane;
                if (START) {
                    float v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {  // as k_init_forward
                        const int i = 4 * q + e;
                        v[e] = i >= b.n_cols || (cv && (unsigned)(i - lo) < (unsigned)npf) ? INFINITY : 0.0f;
                    }
                    d[u] = make_float4(v[0], v[1], v[2], v[3]);
                } else if (q < n4) {
                    d[u] = __ldcs(row + q);
                }
            }
            const float *x0 = xs + (size_t)(c & 1) * kFeatureSeq * kSeqCols;
            for (int f = 0; f < seq.n; ++f) {
                const float a = as[w][f];
                const float4 *x4 = reinterpret_cast<const float4 *>(x0 + f * kSeqCols);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float4 x = x4[u * 32 + lane];
                    const float2 lo2 = sq2(sub2(make_float2(a, a), make_float2(x.x, x.y)));
                    const float2 hi2 = sq2(sub2(make_float2(a, a), make_float2(x.z, x.w)));
                    const float2 dl = make_float2(d[u].x, d[u].y), dh = make_float2(d[u].z, d[u].w);
                    const float2 nl = BWD ? sub2(dl, lo2) : add2(dl, lo2), nh = BWD ? sub2(dh, hi2) : add2(dh, hi2);
                    d[u] = make_float4(nl.x, nl.y, nh.x, nh.y);
                }
            }
            auto keep = [&](int h) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int q = c * (kSeqCols / 4) + u * 32 + lane;
                    const float v[4] = {d[u].x, d[u].y, d[u].z, d[u].w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int j = 4 * h + e;
                        const bool near = q < n4 && v[e] < sv[j];
                        sv[j] = near ? v[e] : sv[j];
                        si[j] = near ? 4 * q + e : si[j];
                    }
                }
            };
            if (SEEDS) {
                if (c < half) keep(0);
                else keep(1);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int q = c * (kSeqCols / 4) + u * 32 + lane;
                if (q < n4) __stcs(row + q, d[u]);
            }
        }
        __syncthreads();
    }
    if (SEEDS && row_in) store_seeds(sv, si, seeds, seed_d, r, lane);
}

int sm_count_commit()
{
    // initialised once, thread-safely (handles may be created from several threads)
    static const int n = [] {
        int dev = 0, c = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
        return c > 0 ? c : 148;
    }();
    return n;
}

}  // namespace

cudaError_t launch_commit(const Bufs &b, int backward, int *seeds, float *seed_d, bool list, cudaStream_t s)
{
    int grid = (b.n_rows + 7) / 8;
    const int cap = sm_count_commit() * 6;
    if (grid > cap) grid = cap;
    if (backward) k_commit<true, false, false><<<grid, 256, 0, s>>>(b, nullptr, nullptr);
    else if (seeds && seed_d && list) k_commit<false, true, true><<<grid, 256, 0, s>>>(b, seeds, seed_d);
    else if (seeds && seed_d) k_commit<false, true, false><<<grid, 256, 0, s>>>(b, seeds, seed_d);
    else k_commit<false, false, false><<<grid, 256, 0, s>>>(b, nullptr, nullptr);
    return cudaGetLastError();
}

cudaError_t launch_commit_seq(const Bufs &b, const FeatureSeq &seq, int backward, bool start, int cv, int npf, int *seeds,
                              float *seed_d, cudaStream_t s)
{
    const bool keep = !backward && seeds && seed_d;
    auto kern = backward ? k_commit_seq<true, false, false>
                : start  ? (keep ? k_commit_seq<false, true, true> : k_commit_seq<false, false, true>)
                         : (keep ? k_commit_seq<false, true, false> : k_commit_seq<false, false, false>);
    const size_t smem = sizeof(float) * 2 * kFeatureSeq * kSeqCols;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<(b.n_rows + kSeqWarps - 1) / kSeqWarps, 32 * kSeqWarps, smem, s>>>(b, seq, cv, npf, seeds, seed_d);
    return cudaGetLastError();
}

}  // namespace snn
