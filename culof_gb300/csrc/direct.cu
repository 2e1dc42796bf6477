// Exact k-NN of small inputs and few features (d <= 16, k <= 64) by two passes
// over all columns, nothing written in between.
//
// A warp takes R rows, its CTA stages the columns 512 at a time
// (dimension-major, two columns per lane). The first pass keeps the smallest
// distance of each of 32 (64) groups of columns per row, one (two) per lane;
// the k-th smallest of them bounds the row's k-th distance. The second pass
// computes the distances again and gathers the columns within the bound (about
// 31 at k = 20), which are sorted and written in the reference's slot order.
// Columns come in ascending index order, so one that only ties with the k-th
// of a full list cannot enter it: equal points stop gathering once they have
// k neighbours (6,000 equal points, d = 8: 221 us per scores call, 764 with every tie
// sorted in).
//
// What bounds it: the packed FP32 distances, 2 x 2d per 64 pairs and pass. The
// distance tile and radix select that it replaces here write and read every
// distance and spend a CTA of 256 threads with a dozen barriers on a row: 26 +
// 131 us at n = 3,001, d = 5, k = 15.
#include <algorithm>

#include "common.cuh"
#include "engine.cuh"
#include "fast.cuh"
#include "row_list.cuh"
#include "sweep_common.cuh"

namespace culof_gb300 {

namespace {

using sweep::fma2;
using sweep::dup2;
using sweep::sub2;

constexpr int kDirWarps = 8;
constexpr int kDirThreads = 32 * kDirWarps;
constexpr int kDirCols = 512;            // columns staged at a time
constexpr int kDirLd = kDirCols + 4;     // row stride: the d values of a point fall in different banks
constexpr int kDirBuf = 64;              // gathered keys per row before they are merged

// KR: list registers (k <= 32 KR); G: groups of columns per lane.
template <int DP, int KR, int G, int R>
__global__ void __launch_bounds__(kDirThreads)
direct_knn_kernel(const float* __restrict__ xc, int n, int d, int row_begin, int row_end, int k,
                  int32_t* __restrict__ nbr_idx, float* __restrict__ nbr_d2, float* __restrict__ kdist2) {
    __shared__ __align__(16) float cols[DP][kDirLd];
    __shared__ uint64_t buf[kDirWarps][R][kDirBuf];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row0 = row_begin + (static_cast<int>(blockIdx.x) * kDirWarps + warp) * R;
    uint64_t a[R][DP];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int f = 0; f < DP; ++f)
            a[r][f] = dup2(row0 + r < row_end && f < d ? xc[static_cast<int64_t>(row0 + r) * d + f] : 0.0f);
    if (d < DP)
        for (int i = tid; i < DP * kDirLd; i += kDirThreads) (&cols[0][0])[i] = 0.0f;  // padded dimensions stay zero

    // stage columns [c0, c0 + 512)
    const auto stage = [&](int c0) {
        __syncthreads();
        const int m = min(kDirCols, n - c0);
        const float* src = xc + static_cast<int64_t>(c0) * d;
        for (int i = tid; i < m * d; i += kDirThreads) cols[i % d][i / d] = src[i];
        __syncthreads();
    };
    // distance bits of row r to this lane's two columns of a step; all ones
    // for the row itself and past the last column
    const auto distances = [&](const uint64_t (&x)[DP], int r, int c, unsigned (&u)[2]) {
        uint64_t s = 0;
#pragma unroll
        for (int f = 0; f < DP; ++f) {
            const uint64_t t = sub2(a[r][f], x[f]);
            s = fma2(t, t, s);
        }
        u[0] = static_cast<unsigned>(s);
        u[1] = static_cast<unsigned>(s >> 32);
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (c + e >= n || c + e == row0 + r) u[e] = 0xFFFFFFFFu;
    };
    const auto load_columns = [&](int at, uint64_t (&x)[DP]) {
#pragma unroll
        for (int f = 0; f < DP; ++f) x[f] = *reinterpret_cast<const uint64_t*>(&cols[f][at]);
    };

    unsigned g[R][G];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < G; ++j) g[r][j] = 0xFFFFFFFFu;
    for (int c0 = 0; c0 < n; c0 += kDirCols) {
        stage(c0);
        const int steps = (min(kDirCols, n - c0) + 63) / 64;
#pragma unroll 1
        for (int st = 0; st < steps; ++st) {
            uint64_t x[DP];
            load_columns(64 * st + 2 * lane, x);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                unsigned u[2];
                distances(x, r, c0 + 64 * st + 2 * lane, u);
                g[r][0] = min(g[r][0], u[0]);
                g[r][G - 1] = min(g[r][G - 1], u[1]);
            }
        }
    }
    unsigned limit[R];  // distance bits of the columns still to be gathered lie below
    uint64_t b[R][KR];
    int pending[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const unsigned bound = warp_rank_value<G>(g[r], k - 1);  // (all ones: fewer than k groups)
        limit[r] = bound == 0xFFFFFFFFu ? bound : bound + 1u;
        pending[r] = 0;
#pragma unroll
        for (int j = 0; j < KR; ++j) b[r][j] = kKeyMax;
    }
    for (int c0 = 0; c0 < n; c0 += kDirCols) {
        if (n > kDirCols) stage(c0);
        const int steps = (min(kDirCols, n - c0) + 63) / 64;
#pragma unroll 1
        for (int st = 0; st < steps; ++st) {
            uint64_t x[DP];
            load_columns(64 * st + 2 * lane, x);
            const int c = c0 + 64 * st + 2 * lane;
            unsigned u[R][2];
            bool any = false;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                distances(x, r, c, u[r]);
                any |= min(u[r][0], u[r][1]) < limit[r];
            }
            if (!__any_sync(kFullMask, any)) continue;
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const bool in = u[r][e] < limit[r];
                    const unsigned m = __ballot_sync(kFullMask, in);
                    if (!m) continue;
                    if (pending[r] + __popc(m) > kDirBuf) {  // merge what is gathered
                        __syncwarp();
                        for (int e0 = 0; e0 < pending[r]; e0 += 32)
                            list_merge<KR>(b[r], e0 + lane < pending[r] ? buf[warp][r][e0 + lane] : kKeyMax);
                        pending[r] = 0;
                        // (strict: what is tested from here on lies above every
                        // merged index; this step's first columns are merged in
                        // only after its second ones were tested)
                        limit[r] = min(limit[r], list_kth_bits<KR>(b[r], k));
                        __syncwarp();
                    }
                    // (keys past a limit that has just tightened are kept: the list drops them)
                    if (in) buf[warp][r][pending[r] + __popc(m & ((1u << lane) - 1u))] = make_key(u[r][e], c + e);
                    pending[r] += __popc(m);
                }
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (row0 + r >= row_end) break;
        for (int e0 = 0; e0 < pending[r]; e0 += 32)
            list_merge<KR>(b[r], e0 + lane < pending[r] ? buf[warp][r][e0 + lane] : kKeyMax);
        emit_row<KR>(b[r], k, n, static_cast<unsigned>(row0 + r), nbr_idx, nbr_d2, kdist2);
    }
}

template <int DP, int R>
void launch_direct(const float* xc, int n, int d, int row_begin, int row_end, int k, int32_t* idx, float* d2, float* kd,
                   cudaStream_t s) {
    const unsigned grid = static_cast<unsigned>(ceil_div(row_end - row_begin, kDirWarps * R));
    if (k <= 24) direct_knn_kernel<DP, 1, 1, R><<<grid, kDirThreads, 0, s>>>(xc, n, d, row_begin, row_end, k, idx, d2, kd);
    else if (k <= 32) direct_knn_kernel<DP, 1, 2, R><<<grid, kDirThreads, 0, s>>>(xc, n, d, row_begin, row_end, k, idx, d2, kd);
    else direct_knn_kernel<DP, 2, 2, R><<<grid, kDirThreads, 0, s>>>(xc, n, d, row_begin, row_end, k, idx, d2, kd);
    CG_LAUNCH_CHECK();
}

template <int DP>
void dispatch_direct(const float* xc, int n, int d, int row_begin, int row_end, int k, int32_t* idx, float* d2,
                     float* kd, cudaStream_t s) {
    // two rows per warp share each staged column once there are enough rows
    // to fill the SMs (16 per SM: two CTAs of 8 warps)
    const int rows = row_end - row_begin;
    if (DP > 8 || rows <= 2432) launch_direct<DP, 1>(xc, n, d, row_begin, row_end, k, idx, d2, kd, s);
    else launch_direct<DP, 2>(xc, n, d, row_begin, row_end, k, idx, d2, kd, s);
}

}  // namespace

bool direct_supported(int64_t n, int d, int k) { return d <= 16 && k <= 64 && n <= (1 << 24); }

void direct_knn(const float* xc, int64_t n, int d, int64_t row_begin, int64_t row_end, int k, int32_t* idx, float* d2,
                float* kd, cudaStream_t s) {
    if (row_end <= row_begin) return;
    const int ni = static_cast<int>(n), b = static_cast<int>(row_begin), e = static_cast<int>(row_end);
    if (d <= 2) dispatch_direct<2>(xc, ni, d, b, e, k, idx, d2, kd, s);
    else if (d <= 4) dispatch_direct<4>(xc, ni, d, b, e, k, idx, d2, kd, s);
    else if (d <= 6) dispatch_direct<6>(xc, ni, d, b, e, k, idx, d2, kd, s);
    else if (d <= 8) dispatch_direct<8>(xc, ni, d, b, e, k, idx, d2, kd, s);
    else if (d <= 12) dispatch_direct<12>(xc, ni, d, b, e, k, idx, d2, kd, s);
    else dispatch_direct<16>(xc, ni, d, b, e, k, idx, d2, kd, s);
}

}  // namespace culof_gb300
