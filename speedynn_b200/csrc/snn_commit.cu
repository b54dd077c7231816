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

namespace snn {

namespace {

__device__ __forceinline__ float sqdiff(float a, float b)
{
    const float t = __fsub_rn(a, b);
    return __fmul_rn(t, t);
}

// Three blocks of 256 threads per SM, each lane with four float4 loads of D in
// flight: the stream needs that many bytes in flight to stay HBM-bound (four
// blocks with two loads per lane while the seed lists take registers: 44.0
// against 43.0 ms of commits per fwd-64k selection).
template <bool BWD, bool SEEDS>
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
            }
        }
        if (SEEDS) {
            // the float4 group of part 4 h + e -> its column; then ascending by distance
#pragma unroll
            for (int j = 0; j < kSeedsPerLane; ++j) si[j] = si[j] < 0 ? -1 : 4 * si[j] + (j & 3);
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
    }
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

cudaError_t launch_commit(const Bufs &b, int backward, int *seeds, float *seed_d, cudaStream_t s)
{
    int grid = (b.n_rows + 7) / 8;
    const int cap = sm_count_commit() * 6;
    if (grid > cap) grid = cap;
    if (backward) k_commit<true, false><<<grid, 256, 0, s>>>(b, nullptr, nullptr);
    else if (seeds && seed_d) k_commit<false, true><<<grid, 256, 0, s>>>(b, seeds, seed_d);
    else k_commit<false, false><<<grid, 256, 0, s>>>(b, nullptr, nullptr);
    return cudaGetLastError();
}

}  // namespace snn
