// The rows that leave the tensor path (tc_sweep.cu), against all points in
// FP32: the exact k nearest of a list of rows, its length known on the device
// only, for up to 256 features.
//
// A work item is 32 listed rows (four per warp) against a share of the columns,
// 128 at a time: the CTA stages 16 features of them (dimension-major), a lane
// takes four columns and carries the four rows' packed distances over the
// features. An eighth of the tiles is read first: the smallest distance of each
// of 32 (64) groups of their columns per row, whose k-th smallest bounds the
// row's k-th distance whatever the order of the columns. Then every tile: the
// columns within the bound are gathered, merged 64 at a time, and tighten it.
// Few rows split the columns (their CTAs would leave the chip idle); the last
// item of a group to finish merges the group's lists.
//
// What bounds it: the packed FP32 distances, 9/8 x 4d instructions per 128 columns
// and row. The FMA pipe is busy half of the time (barriers, list merges and a
// partly empty last wave take the rest). 20,000 Cauchy points of 32 features,
// which all leave, take 2.2 ms here (7.5 ms the call, 36.4 when their pairs were
// rescored one by one in the sweep, 19.4 when that had seven splits of the
// columns); 8,000 of 200 features 1.8 ms (2.0 the call; 2.9 when the distance
// tile and select took them).
#include <algorithm>

#include "common.cuh"
#include "engine.cuh"
#include "fast.cuh"
#include "row_list.cuh"
#include "sweep_common.cuh"

namespace culof_gb300 {

namespace {

using sweep::dup2;
using sweep::fma2;
using sweep::sub2;

constexpr int kLrWarps = 8;
constexpr int kLrThreads = 32 * kLrWarps;
constexpr int kLrRowsPer = 4;                      // rows per warp
constexpr int kLrRows = kLrWarps * kLrRowsPer;     // rows per item
constexpr int kLrCols = 128;                       // columns staged at a time
constexpr int kLrDims = 16;                        // features staged at a time, in two buffers
constexpr int kLrLd = kLrCols + 2;                 // (two columns' features lie in 32 banks, pairs stay aligned)
constexpr int kLrBuf = 64;                         // gathered keys per row before they are merged
constexpr int kLrSample = 8;                       // one tile in so many is read for the bounds
constexpr int kLrMaxSplits = 64;

template <int KR>
struct LostSmem {
    float cols[2][kLrDims][kLrLd];
    uint64_t list[kLrRows][32 * KR];
    uint64_t buf[kLrRows][kLrBuf];
    int pending[kLrRows];
    int last;
};

// Items per group of rows: one round of CTAs, or two where that is shorter (the
// groups alone from a whole round of them on), four tiles each at least. Every
// split gathers and merges some k ln(columns / k) keys of its own.
__host__ __device__ __forceinline__ int lost_splits(int groups, int slots, int nt) {
    const int one = groups >= slots ? 1 : slots / groups, two = groups >= slots ? 1 : 2 * slots / groups;
    const int want = two > 2 * one ? two : one;
    const int most = nt / 4 < kLrMaxSplits ? nt / 4 : kLrMaxSplits;
    return want < most ? want : most < 1 ? 1 : most;
}

// Four bytes into shared memory (zero if not in), not waited for.
__device__ __forceinline__ void copy4_async(float* dst, const float* src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(sweep::smem_u32(dst)), "l"(src), "r"(in ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int KR>
__device__ __forceinline__ void merge_gathered(uint64_t (&b)[KR], const uint64_t* list, const uint64_t* buf, int have) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < KR; ++j) b[j] = list[32 * j + lane];
    for (int e0 = 0; e0 < have; e0 += 32) list_merge<KR>(b, e0 + lane < have ? buf[e0 + lane] : kKeyMax);
}

// Gathers a row's columns below the limit (whole warp; u: the distance bits of
// this lane's four columns, ascending over e and, within e, over the lanes).
// Returns the limit. Columns come in ascending index order, so that it is strict:
// a merge takes in columns of the quarters before the last one only, and what
// is tested after it lies above them.
template <int KR>
__noinline__ __device__ unsigned lost_gather(uint64_t* list, uint64_t* buf, int* pending, unsigned u0, unsigned u1,
                                             unsigned u2, unsigned u3, unsigned limit, int c0, int k) {
    const int lane = threadIdx.x & 31;
    const unsigned u[4] = {u0, u1, u2, u3};
    int p = *pending;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const bool in = u[e] < limit;
        const unsigned m = __ballot_sync(kFullMask, in);
        if (!m) continue;
        if (p + __popc(m) > kLrBuf) {
            __syncwarp();
            uint64_t b[KR];
            merge_gathered<KR>(b, list, buf, p);
#pragma unroll
            for (int j = 0; j < KR; ++j) list[32 * j + lane] = b[j];
            limit = min(limit, list_kth_bits<KR>(b, k));
            p = 0;
            __syncwarp();
        }
        if (in) buf[p + __popc(m & ((1u << lane) - 1u))] = make_key(u[e], c0 + (e >> 1) * 64 + 2 * lane + (e & 1));
        p += __popc(m);
    }
    __syncwarp();
    if (lane == 0) *pending = p;
    __syncwarp();
    return limit;
}

template <int KR, int G>
__global__ void __launch_bounds__(kLrThreads, 2)
lost_rows_kernel(const float* __restrict__ xc, int64_t n, int d, int k, const int32_t* __restrict__ rows,
                 const int* __restrict__ count, uint64_t* __restrict__ scratch, int* __restrict__ arrived,
                 int32_t* __restrict__ nbr_idx, float* __restrict__ nbr_d2, float* __restrict__ kdist2) {
    extern __shared__ __align__(16) unsigned char lr_raw[];
    LostSmem<KR>& sh = *reinterpret_cast<LostSmem<KR>*>(lr_raw);
    uint64_t* row2 = reinterpret_cast<uint64_t*>(lr_raw + (sizeof(LostSmem<KR>) + 15) / 16 * 16);  // [kLrRows][dp]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int dp = (d + 1) & ~1;
    const int m = *count, nt = static_cast<int>((n + kLrCols - 1) / kLrCols);
    const int groups = (m + kLrRows - 1) / kLrRows;
    const int S = groups > 0 ? lost_splits(groups, gridDim.x, nt) : 1;
    for (int64_t item = blockIdx.x; item < static_cast<int64_t>(groups) * S; item += gridDim.x) {
        const int g = static_cast<int>(item / S), s = static_cast<int>(item % S);
        // the rows, each coordinate in both halves of a packed operand
        for (int i = warp; i < kLrRows; i += kLrWarps) {
            const int at = kLrRows * g + i;
            const int64_t row = at < m ? rows[at] : -1;
            for (int f = lane; f < dp; f += 32) row2[i * dp + f] = row >= 0 && f < d ? dup2(xc[row * d + f]) : 0;
#pragma unroll
            for (int j = 0; j < KR; ++j) sh.list[i][32 * j + lane] = kKeyMax;
            if (lane == 0) sh.pending[i] = 0;
        }
        int self[kLrRowsPer];
#pragma unroll
        for (int r = 0; r < kLrRowsPer; ++r) {
            const int at = kLrRows * g + kLrRowsPer * warp + r;
            self[r] = at < m ? rows[at] : -1;
        }
        const uint64_t* mine = row2 + kLrRowsPer * warp * dp;
        const int t0 = static_cast<int>(static_cast<int64_t>(nt) * s / S);
        const int t1 = static_cast<int>(static_cast<int64_t>(nt) * (s + 1) / S);

        // the item's tiles: first the sample, then all of them
        const int ns = (t1 - t0 + kLrSample - 1) / kLrSample, steps = ns + t1 - t0;
        const auto tile_of = [&](int q) { return q < ns ? t0 + kLrSample * q : t0 + q - ns; };
        // features [f0, f0 + kLrDims) of tile t's columns (zero past the last
        // feature and column), transposed on their way into shared memory
        const auto stage = [&](int buf, int t, int f0) {
            const int f = f0 + lane % kLrDims;
#pragma unroll
            for (int c = tid / kLrDims; c < kLrCols; c += kLrThreads / kLrDims) {
                const int64_t col = static_cast<int64_t>(t) * kLrCols + c;
                const bool in = col < n && f < d;
                copy4_async(&sh.cols[buf][lane % kLrDims][c], xc + (in ? col * d + f : 0), in);
            }
        };
        __syncthreads();
        stage(0, tile_of(0), 0);
        int buf = 0;
        unsigned limit[kLrRowsPer];  // distance bits of the columns still to be gathered lie below
        unsigned gm[kLrRowsPer][G];
#pragma unroll
        for (int r = 0; r < kLrRowsPer; ++r) {
            limit[r] = 0u;
#pragma unroll
            for (int j = 0; j < G; ++j) gm[r][j] = 0xFFFFFFFFu;
        }
#pragma unroll 1
        for (int q = 0; q < steps; ++q) {
            const int c0 = tile_of(q) * kLrCols;  // (n is at most 2^30)
            uint64_t acc[kLrRowsPer][2];
#pragma unroll
            for (int r = 0; r < kLrRowsPer; ++r) acc[r][0] = acc[r][1] = 0;
#pragma unroll 1
            for (int f0 = 0; f0 < d; f0 += kLrDims) {
                copies_done();
                __syncthreads();  // everyone's copies, and everyone is done with the other buffer
                if (f0 + kLrDims < d) stage(buf ^ 1, tile_of(q), f0 + kLrDims);
                else if (q + 1 < steps) stage(buf ^ 1, tile_of(q + 1), 0);
                const float(*cols)[kLrLd] = sh.cols[buf];
                buf ^= 1;
                const int fe = min(kLrDims, dp - f0);  // (a padded feature is zero in both: fma(0, 0, s) = s)
#pragma unroll 4
                for (int f = 0; f < fe; f += 2) {
                    uint64_t x[2][2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        x[e][0] = *reinterpret_cast<const uint64_t*>(&cols[f + e][2 * lane]);
                        x[e][1] = *reinterpret_cast<const uint64_t*>(&cols[f + e][64 + 2 * lane]);
                    }
#pragma unroll
                    for (int r = 0; r < kLrRowsPer; ++r) {  // the oracle's chain
                        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(mine + r * dp + f0 + f);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint64_t v = sub2(a.x, x[0][h]);
                            acc[r][h] = fma2(v, v, acc[r][h]);
                            v = sub2(a.y, x[1][h]);
                            acc[r][h] = fma2(v, v, acc[r][h]);
                        }
                    }
                }
            }
            if (q == ns) {
#pragma unroll
                for (int r = 0; r < kLrRowsPer; ++r) {
                    const unsigned bound = warp_rank_value<G>(gm[r], k - 1);  // (all ones: fewer than k groups)
                    limit[r] = self[r] < 0 ? 0u : bound == 0xFFFFFFFFu ? bound : bound + 1u;
                }
            }
#pragma unroll
            for (int r = 0; r < kLrRowsPer; ++r) {
                unsigned u[4];  // distance bits; all ones for the row itself and past the last column
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int c = c0 + (e >> 1) * 64 + 2 * lane + (e & 1);
                    u[e] = c >= n || c == self[r] ? 0xFFFFFFFFu : static_cast<unsigned>(acc[r][e >> 1] >> (32 * (e & 1)));
                }
                if (q < ns) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) gm[r][e * G / 4] = min(gm[r][e * G / 4], u[e]);
                } else if (__any_sync(kFullMask, min(min(u[0], u[1]), min(u[2], u[3])) < limit[r])) {
                    const int i = kLrRowsPer * warp + r;
                    limit[r] = lost_gather<KR>(sh.list[i], sh.buf[i], &sh.pending[i], u[0], u[1], u[2], u[3], limit[r], c0, k);
                }
            }
        }
#pragma unroll 1
        for (int r = 0; r < kLrRowsPer; ++r) {
            const int i = kLrRowsPer * warp + r, at = kLrRows * g + i;
            if (at >= m) break;
            uint64_t b[KR];
            merge_gathered<KR>(b, sh.list[i], sh.buf[i], sh.pending[i]);
            if (S == 1) {
                emit_row<KR>(b, k, n, static_cast<unsigned>(rows[at]), nbr_idx, nbr_d2, kdist2);
            } else {
#pragma unroll
                for (int j = 0; j < KR; ++j) scratch[((item * kLrRows + i) * KR + j) * 32 + lane] = b[j];
            }
        }
        __syncthreads();
        if (S == 1) continue;
        // the group's last item joins its lists
        if (tid == 0) {
            __threadfence();
            sh.last = atomicAdd(&arrived[g], 1) == S - 1 ? 1 : 0;
        }
        __syncthreads();
        if (sh.last) {
            __threadfence();
#pragma unroll 1
            for (int r = 0; r < kLrRowsPer; ++r) {
                const int i = kLrRowsPer * warp + r, at = kLrRows * g + i;
                if (at >= m) break;
                uint64_t b[KR];
#pragma unroll
                for (int j = 0; j < KR; ++j) b[j] = kKeyMax;
                for (int o = 0; o < S; ++o)
#pragma unroll
                    for (int j = 0; j < KR; ++j)
                        list_merge<KR>(b, __ldcg(scratch + (((static_cast<int64_t>(g) * S + o) * kLrRows + i) * KR + j) * 32 + lane));
                emit_row<KR>(b, k, n, static_cast<unsigned>(rows[at]), nbr_idx, nbr_d2, kdist2);
            }
        }
        __syncthreads();
    }
}

int lost_slots(int sms) { return std::min(2 * sms, kLostGroups); }

template <int KR, int G>
void launch_lost(const float* xc, int64_t n, int d, int k, const int32_t* rows, const int* count, uint64_t* scratch,
                 int* arrived, int sms, int32_t* idx, float* d2, float* kd, cudaStream_t s) {
    const size_t base = (sizeof(LostSmem<KR>) + 15) / 16 * 16, per_dim = sizeof(uint64_t) * kLrRows;
    set_max_dynamic_smem(reinterpret_cast<const void*>(lost_rows_kernel<KR, G>), static_cast<int>(base + per_dim * kMaxTensorD));
    // (as a dependent launch that starts under tc_final_kernel it cost passes that
    // overlap 1% at n = 200,000, d = 128; this way half a percent)
    lost_rows_kernel<KR, G><<<lost_slots(sms), kLrThreads, base + per_dim * ((d + 1) & ~1), s>>>(
        xc, n, d, k, rows, count, scratch, arrived, idx, d2, kd);
    CG_LAUNCH_CHECK();
}

}  // namespace

size_t lost_rows_bytes(int64_t n, int64_t max_rows, int k, int sms) {
    // (groups x splits, wherever the columns are split at all)
    const int64_t groups = ceil_div(max_rows, kLrRows), nt = ceil_div(n, kLrCols);
    const int64_t items = std::min<int64_t>(2 * lost_slots(sms), groups * std::max<int64_t>(1, std::min<int64_t>(kLrMaxSplits, nt / 4)));
    return sizeof(uint64_t) * static_cast<size_t>(items) * kLrRows * 32 * (k <= 32 ? 1 : 2);
}

void lost_rows(const float* xc, int64_t n, int d, int k, const int32_t* rows, const int* count, void* scratch,
               int* arrived, int sms, int32_t* idx, float* d2, float* kd, cudaStream_t s) {
    uint64_t* keys = static_cast<uint64_t*>(scratch);
    if (k <= 24) launch_lost<1, 1>(xc, n, d, k, rows, count, keys, arrived, sms, idx, d2, kd, s);
    else if (k <= 32) launch_lost<1, 2>(xc, n, d, k, rows, count, keys, arrived, sms, idx, d2, kd, s);
    else launch_lost<2, 2>(xc, n, d, k, rows, count, keys, arrived, sms, idx, d2, kd, s);
}

}  // namespace culof_gb300
