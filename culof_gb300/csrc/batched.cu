// Batched LOF over many independent problems in one persistent launch,
// replayed from a CUDA graph.
//
// The reference serves one problem per culof::lof call: a private stream and
// seven cudaMallocs per call (pipeline.cu:148-168), then the pipeline. A loop
// of such calls over thousands of small problems is bound by that per-call
// setup and by launches that cannot fill the GPU. Here one call takes all
// problems (points concatenated, per-problem offsets and k):
//   1. batched centring: the single-problem centring's arithmetic, in the
//      same order (chunks of kCenterChunk rows), for every problem at once;
//   2. a spatial order within each problem (Morton keys over its 8 widest
//      dimensions, two stable radix sorts);
//   3. the exact k-NN of every row among its problem's points: up to 16
//      features the row-pruned sweep (sweep_rows.cuh) over work items grouped
//      by list form; above, a persistent kernel whose CTAs pull (problem,
//      128-row tile) items from an atomic counter, largest problems first,
//      and visit the problem's column tiles nearest first into per-row lists
//      in shared memory (FP32 direct differences, the oracle's formula);
//   4. batched lrd and scores with the reference's FP64 sums.
// Every problem's scores are bit-identical to a single-problem call. The
// launch sequence of a given batch layout is captured once as a CUDA graph
// and replayed; on first sight of a layout a small autotuner times the k-NN
// kernel's variants (CTAs per SM) and keeps the fastest.
#include <algorithm>
#include <cstring>
#include <sstream>
#include <utility>
#include <vector>

#include "common.cuh"
#include "engine.cuh"
#include "fast.cuh"
#include "fp64.cuh"
#include "sweep_common.cuh"
#include "sweep_rows.cuh"

namespace culof_gb300 {

namespace {

using namespace sweep;

constexpr int kBM = 80;          // list capacity per row: k + 32 free slots (two CTAs per SM)
constexpr int kBMaxK = kBM - 32;
constexpr int kBMaxD = 64;

// ---- batched centring (prep.cu's arithmetic per problem) -------------------

// One thread per (global chunk, feature); chunk g belongs to problem cp[g].
template <bool kSquares>  // of x - mean, otherwise the sums of x
__global__ void bc_partials_kernel(const float* __restrict__ x, const int64_t* __restrict__ off, int d,
                                   const int* __restrict__ cp, const int64_t* __restrict__ coff, int64_t nchunks,
                                   const double* __restrict__ mean, double* __restrict__ partial) {
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= nchunks * d) return;
    const int64_t g = t / d;
    const int f = static_cast<int>(t % d);
    const int p = cp[g];
    const int64_t c = g - coff[p];
    const int64_t n = off[p + 1] - off[p];
    const float* xp = x + off[p] * d;
    const int64_t begin = c * kCenterChunk;
    const int64_t end = begin + kCenterChunk < n ? begin + kCenterChunk : n;
    double s = 0.0;
    const double m = kSquares ? mean[static_cast<int64_t>(p) * d + f] : 0.0;
    for (int64_t i = begin; i < end; i += 16) {  // 16 loads in flight
        const int len = end - i < 16 ? static_cast<int>(end - i) : 16;
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (j < len) v[j] = xp[(i + j) * d + f];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            if (j >= len) break;
            double a = widen(v[j]);
            if (kSquares) {
                a = __dsub_rn(a, m);
                a = __dmul_rn(a, a);
            }
            s = __dadd_rn(s, a);
        }
    }
    partial[t] = s;
}

__global__ void bc_finalize_kernel(const double* __restrict__ partial, const int64_t* __restrict__ off,
                                   const int64_t* __restrict__ coff, int num, int d, int mode,
                                   double* __restrict__ mean, double* __restrict__ inv_std) {
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= static_cast<int64_t>(num) * d) return;
    const int p = static_cast<int>(t / d);
    const int f = static_cast<int>(t % d);
    double total = 0.0;
    for (int64_t c = coff[p]; c < coff[p + 1]; ++c) total = __dadd_rn(total, partial[c * d + f]);
    const double dn = static_cast<double>(off[p + 1] - off[p]);
    if (mode == 0) {
        mean[t] = __ddiv_rn(total, dn);
        inv_std[t] = 1.0;
    } else {
        const double sd = __dsqrt_rn(__ddiv_rn(total, dn));
        inv_std[t] = (sd > 1e-12) ? __ddiv_rn(1.0, sd) : 1.0;
    }
}

// Each thread stays on one feature (the block's active threads and its stride
// are multiples of d); d <= kBMaxD. Bound by the FP64 units, one subtraction
// (and with kScale, normalising, one product) per value; a division of the
// place by d and conversions in FP64 took 105 us for 834,000 points of 16
// features, this takes 37.
constexpr int kApplyThreads = 256;
template <bool kScale>
__global__ void __launch_bounds__(kApplyThreads)
bc_apply_kernel(const float* __restrict__ x, int64_t ntot, int d, const int* __restrict__ pid,
                const double* __restrict__ mean, const double* __restrict__ inv_std, float* __restrict__ xc) {
    const int rows = kApplyThreads / d;  // rows per block and step
    const int r = static_cast<int>(threadIdx.x) / d, f = static_cast<int>(threadIdx.x) % d;
    if (r >= rows) return;
    const int64_t step = static_cast<int64_t>(gridDim.x) * rows;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * rows + r; i < ntot; i += step) {
        const int64_t pf = static_cast<int64_t>(pid[i]) * d + f;
        double w = __dsub_rn(widen(x[i * d + f]), mean[pf]);
        if (kScale) w = __dmul_rn(w, inv_std[pf]);
        xc[i * d + f] = narrow(w);
    }
}

// ---- spatial order within each problem -----------------------------------------

constexpr int kMortonDimsB = 8;

// One block per problem: per-dimension range of its centred points, then
// the (up to) 8 widest dimensions, widest first (ties by index). Latency:
// 1,024 threads with 8 loads in flight each (45 us for 256 problems of
// 834,000 points and 16 features; 256 threads, one load each, took 249).
constexpr int kMinMaxThreads = 1024;
__global__ void __launch_bounds__(kMinMaxThreads)
bm_minmax_kernel(const float* __restrict__ xc, const int64_t* __restrict__ off, int d,
                                 float* __restrict__ pmm, int* __restrict__ pdims) {
    __shared__ unsigned lo[kBMaxD], hi[kBMaxD];
    const int p = blockIdx.x;
    for (int f = threadIdx.x; f < d; f += blockDim.x) {
        lo[f] = 0xFFFFFFFFu;
        hi[f] = 0u;
    }
    __syncthreads();
    const int64_t b = off[p], e = off[p + 1];
    const int per = static_cast<int>(blockDim.x) / d * d;  // each thread stays on one feature
    if (static_cast<int>(threadIdx.x) < per) {
        const int f = static_cast<int>(threadIdx.x) % d;
        unsigned mn = 0xFFFFFFFFu, mx = 0u;
        const int64_t total = (e - b) * d;
        const float* xp = xc + b * d;
        for (int64_t t = threadIdx.x; t < total; t += static_cast<int64_t>(per) * 8) {
            float v[8];  // (past the end the first value again: min and max stay)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int64_t at = t + static_cast<int64_t>(j) * per;
                v[j] = xp[at < total ? at : t];
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const unsigned k = order_bits(v[j]);
                mn = min(mn, k);
                mx = max(mx, k);
            }
        }
        atomicMin(&lo[f], mn);
        atomicMax(&hi[f], mx);
    }
    __syncthreads();
    for (int f = threadIdx.x; f < d; f += blockDim.x) {
        pmm[(static_cast<int64_t>(p) * d + f) * 2] = order_value(lo[f]);
        pmm[(static_cast<int64_t>(p) * d + f) * 2 + 1] = order_value(hi[f]);
    }
    if (threadIdx.x == 0) {
        const int m = d < kMortonDimsB ? d : kMortonDimsB;
        int chosen[kMortonDimsB];
        for (int j = 0; j < m; ++j) {
            int best = -1;
            float span = -1.0f;
            for (int f = 0; f < d; ++f) {
                bool taken = false;
                for (int q = 0; q < j; ++q) taken |= chosen[q] == f;
                const float sp = order_value(hi[f]) - order_value(lo[f]);
                if (!taken && sp > span) {
                    span = sp;
                    best = f;
                }
            }
            // (ranges that are not numbers: the first feature not yet taken)
            for (int f = 0; best < 0; ++f) {
                bool taken = false;
                for (int q = 0; q < j; ++q) taken |= chosen[q] == f;
                if (!taken) best = f;
            }
            chosen[j] = best;
            pdims[p * kMortonDimsB + j] = best;
        }
    }
}

// Morton key of each point over its problem's chosen dimensions.
__global__ void bm_morton_kernel(const float* __restrict__ xc, int64_t ntot, int d, const int* __restrict__ pid,
                                 const float* __restrict__ pmm, const int* __restrict__ pdims,
                                 unsigned* __restrict__ keys, unsigned* __restrict__ vals) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < ntot;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int p = pid[i];
        const int m = d < kMortonDimsB ? d : kMortonDimsB;
        const int bits = (32 / m) < 10 ? 32 / m : 10;
        unsigned q[kMortonDimsB];
        for (int j = 0; j < m; ++j) {
            const int f = pdims[p * kMortonDimsB + j];
            const float lo = pmm[(static_cast<int64_t>(p) * d + f) * 2], hi = pmm[(static_cast<int64_t>(p) * d + f) * 2 + 1];
            const float span = hi - lo;
            float t = span > 0.0f ? (xc[i * d + f] - lo) / span : 0.0f;
            t = fminf(fmaxf(t, 0.0f), 1.0f);
            q[j] = static_cast<unsigned>(t * static_cast<float>((1u << bits) - 1u) + 0.5f);
        }
        unsigned key = 0u;
        for (int bt = bits - 1; bt >= 0; --bt)
            for (int j = 0; j < m; ++j) key = (key << 1) | ((q[j] >> bt) & 1u);
        keys[i] = key;
        vals[i] = static_cast<unsigned>(i);
    }
}

__global__ void bm_pidkey_kernel(int64_t ntot, const int* __restrict__ pid, const unsigned* __restrict__ vals,
                                 unsigned* __restrict__ keys) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < ntot;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        keys[i] = static_cast<unsigned>(pid[vals[i]]);
}

// Sorted coordinates and, per sorted position, the point's original index
// within its problem.
__global__ void bm_gather_kernel(const float* __restrict__ xc, int64_t ntot, int d, const unsigned* __restrict__ perm,
                                 const int* __restrict__ pid, const int64_t* __restrict__ off, float* __restrict__ xs,
                                 unsigned* __restrict__ lidx) {
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < ntot * d;
         t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t i = t / d;
        const int f = static_cast<int>(t % d);
        const unsigned src = perm[i];
        xs[t] = xc[static_cast<int64_t>(src) * d + f];
        if (f == 0) lidx[i] = static_cast<unsigned>(src - off[pid[src]]);
    }
}

// One CTA of 128 threads per (problem, tile of 128 sorted points): the column
// tile of the row-pruned sweep (small.cuh's layout) and its box.
template <int DP>
__global__ void __launch_bounds__(kCT) bm_tile_kernel(const float* __restrict__ xc, int d,
                                                      const unsigned* __restrict__ perm, const int64_t* __restrict__ off,
                                                      const int* __restrict__ tpid, const int64_t* __restrict__ toff,
                                                      float* __restrict__ tiles, float* __restrict__ boxes) {
    __shared__ float wb[kCT / 32][2][DP];
    const int64_t g = blockIdx.x;
    const int c = threadIdx.x, lane = c & 31, q = c >> 5;
    const int p = tpid[g];
    const int64_t pos = off[p] + (g - toff[p]) * kCT + c;
    const bool valid = pos < off[p + 1];
    const unsigned src = valid ? perm[pos] : 0u;
    float* tile = tiles + g * small::tile_floats(DP);
#pragma unroll
    for (int f = 0; f < DP; ++f) {
        const float v = (valid && f < d) ? xc[static_cast<int64_t>(src) * d + f] : 0.0f;
        tile[f * kCT + c] = (!valid && f == 0) ? __int_as_float(0x7fc00000) : v;
        float lo = valid ? v : __int_as_float(0x7f800000), hi = valid ? v : __int_as_float(0xff800000);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) {
            wb[q][0][f] = lo;
            wb[q][1][f] = hi;
        }
    }
    reinterpret_cast<unsigned*>(tile)[small::tile_index_off(DP) + c] =
        valid ? static_cast<unsigned>(src - off[p]) : kNoIndex;
    __syncthreads();
    if (c < small::kHalves * DP) {
        const int h = c / DP, f = c % DP;
        tile[small::tile_box_off(DP) + (h * DP + f) * 2] = fminf(wb[2 * h][0][f], wb[2 * h + 1][0][f]);
        tile[small::tile_box_off(DP) + (h * DP + f) * 2 + 1] = -fmaxf(wb[2 * h][1][f], wb[2 * h + 1][1][f]);
    }
    if (c < DP) {
        boxes[g * 2 * DP + c] = fminf(fminf(wb[0][0][c], wb[1][0][c]), fminf(wb[2][0][c], wb[3][0][c]));
        boxes[g * 2 * DP + DP + c] = fmaxf(fmaxf(wb[0][1][c], wb[1][1][c]), fmaxf(wb[2][1][c], wb[3][1][c]));
    }
}

// Batches of up to 16 features: one CTA per 64 rows of a problem, the
// row-pruned sweep over the problem's own tiles (sweep_rows.cuh). In the
// evaluated workload (256 problems, d = 16, three clusters and 2% outliers
// each) the boxes rule out the other clusters' tiles, two thirds of all pairs.
template <int DP, int KR, int G>
__global__ void __launch_bounds__(kThreads, DP <= 8 && KR == 1 ? 3 : 2)
batched_sweep_kernel(const float* __restrict__ tiles, const float* __restrict__ boxes, const int64_t* __restrict__ off,
                     const int* __restrict__ ks, const int64_t* __restrict__ nkoff, const int64_t* __restrict__ toff,
                     const uint2* __restrict__ items, int32_t* __restrict__ nbr_idx, float* __restrict__ nbr_d2,
                     float* __restrict__ kdist2, int* __restrict__ status) {
    constexpr int kRowsPer = 8;
    using Smem = small::SmallSmem<DP, KR, kRowsPer, kWarps>;
    extern __shared__ __align__(128) unsigned char bsw_raw[];
    Smem& sh = *reinterpret_cast<Smem*>(bsw_raw);
    constexpr int kPerTile = kCT / Smem::kRows;
    const uint2 it = items[blockIdx.x / kPerTile];
    const int p = static_cast<int>(it.x);
    small::SweepRows P{};
    P.n = off[p + 1] - off[p];
    P.base = static_cast<int64_t>(it.y) * kCT + static_cast<int>(blockIdx.x) % kPerTile * Smem::kRows;
    if (P.base >= P.n) return;
    P.nt = static_cast<int>((P.n + kCT - 1) / kCT);
    P.tiles = tiles + toff[p] * small::tile_floats(DP);
    P.boxes = boxes + toff[p] * 2 * DP;
    P.k = ks[p];
    P.segment = small::kSegTiles;
    P.nbr_idx = nbr_idx + nkoff[p];
    P.nbr_d2 = nbr_d2 + nkoff[p];
    P.kdist2 = kdist2 + off[p];
    P.status = status;
    small::sweep_rows<DP, KR, G, kRowsPer, kWarps, false>(sh, P);
}

// ---- persistent k-NN ---------------------------------------------------------

template <int DP>
struct BatchSmem {
    RowLists<kBM> L;
    uint64_t rows2[kRT][DP];         // this item's rows, each coordinate duplicated into both halves
    uint64_t cols2[kCT / 2][DP + 1];  // one column tile as packed column pairs (odd stride)
    int item;
};

// Append this lane's key for row r (if it beats the row's k-th key), keeping
// 32 free slots: warp-uniform.
__device__ __forceinline__ void offer(RowLists<kBM>& L, int r, uint64_t key, int k) {
    const int lane = threadIdx.x & 31;
    bool pass = key < L.kth[r];
    unsigned m = __ballot_sync(0xffffffffu, pass);
    if (!m) return;
    if (L.cnt[r] > kBM - 32) {
        compact_row<kBM>(L, r, k, 0.0f, 8);
        pass = key < L.kth[r];
        m = __ballot_sync(0xffffffffu, pass);
        if (!m) return;
    }
    const int c = L.cnt[r];
    if (pass) L.list[r][c + __popc(m & ((1u << lane) - 1u))] = key;
    __syncwarp();
    if (lane == 0) L.cnt[r] = c + __popc(m);
    __syncwarp();
}

// Offer a row's two keys (one warp-uniform test first).
__device__ __forceinline__ void offer_row(RowLists<kBM>& L, int r, const uint64_t (&key)[2], int k) {
    const uint64_t mn = key[1] < key[0] ? key[1] : key[0];
    if (!__any_sync(0xffffffffu, mn < L.kth[r])) return;
    offer(L, r, key[0], k);
    offer(L, r, key[1], k);
}

// Each warp owns 16 rows of the item. The CTA stages the problem's columns
// in tiles of 128 (packed column pairs in shared memory); per pass a lane
// holds a column pair in registers (packed f32x2 per dimension) and takes two
// rows at a time: two independent packed FMA chains. Distances are
// the oracle's direct-difference chain, exactly (per-lane IEEE sub.rn /
// fma.rn).
template <int DP>
__global__ void __launch_bounds__(kThreads, DP <= 32 ? 2 : 1)
batched_knn_kernel(const float* __restrict__ xc, const unsigned* __restrict__ lidx, const int64_t* __restrict__ off,
                   const int* __restrict__ ks, const int64_t* __restrict__ nkoff, const uint2* __restrict__ items,
                   int nitems, int d, unsigned* __restrict__ counter, int32_t* __restrict__ nbr_idx,
                   float* __restrict__ nbr_d2, float* __restrict__ kdist2) {
    extern __shared__ __align__(16) unsigned char braw[];
    BatchSmem<DP>& sh = *reinterpret_cast<BatchSmem<DP>*>(braw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kTile = 64;
    for (;;) {
        if (tid == 0) sh.item = static_cast<int>(atomicAdd(counter, 1u));
        __syncthreads();
        const int item = sh.item;
        if (item >= nitems) break;
        const int p = static_cast<int>(items[item].x);
        const int T = static_cast<int>(items[item].y);
        const int64_t base = off[p];
        const int n = static_cast<int>(off[p + 1] - base);
        const int k = ks[p];
        const float* xp = xc + base * d;
        const int r0 = T * kRT;
        for (int i = tid; i < kRT * DP; i += kThreads) {
            const int r = i / DP, f = i % DP;
            sh.rows2[r][f] = dup2((r0 + r < n && f < d) ? xp[static_cast<int64_t>(r0 + r) * d + f] : 0.0f);
        }
        if (tid < kRT) {
            sh.L.cnt[tid] = 0;
            sh.L.sorted[tid] = 0;
            sh.L.kth[tid] = kKeyMax;
            sh.L.row_norm[tid] = 0.0f;
        }
        __syncthreads();
        const int rw = warp * kRowsPerWarp;
        const unsigned* li = lidx + base;  // original index of each sorted position
        const int ntp = (n + kCT - 1) / kCT;
        // column tiles in spiral order from the item's own tile: near points
        // first, so the lists fill with good neighbours early
#pragma unroll 1
        for (int qt = 0; qt < ntp; ++qt) {
            const int ct = spiral_tile(T, qt, ntp);
            const int c0 = ct * kCT;
            // the CTA stages 128 columns (coalesced) as packed pairs
            for (int i = tid; i < kCT * DP; i += kThreads) {
                const int c = i / DP, f = i % DP;
                const float v = (c0 + c < n && f < d) ? xp[static_cast<int64_t>(c0 + c) * d + f] : 0.0f;
                reinterpret_cast<float*>(&sh.cols2[c >> 1][f])[c & 1] = v;
            }
            __syncthreads();
#pragma unroll 1
            for (int sub = 0; sub < kCT; sub += kTile) {
            uint64_t cp[DP];
            const int pr = (sub >> 1) + lane;  // column pair index in the tile
            const int cc = c0 + 2 * pr;
#pragma unroll
            for (int f = 0; f < DP; ++f) cp[f] = sh.cols2[pr][f];
            // per column: its original index in the key's low half, or all
            // ones (a key of kKeyMax) for columns beyond the problem
            const uint64_t cidx[2] = {cc < n ? static_cast<uint64_t>(li[cc]) : kKeyMax,
                                      cc + 1 < n ? static_cast<uint64_t>(li[cc + 1]) : kKeyMax};
            const bool own = c0 == r0;  // the only tile holding the rows' own points
#pragma unroll 1
            for (int rr = 0; rr < kRowsPerWarp; rr += 2) {
                const int r = rw + rr;
                if (r0 + r >= n) break;  // warp-uniform: rows beyond the problem
                uint64_t s[2] = {0, 0};
                // dimensions past d are zero in both operands: each adds
                // fma(0, 0, s) = s, so the chain over all DP equals the
                // oracle's chain over d
#pragma unroll
                for (int f = 0; f < DP; ++f) {
                    const uint64_t a0 = sh.rows2[r][f], a1 = sh.rows2[r + 1][f];
                    uint64_t t0, t1;
                    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(t0) : "l"(a0), "l"(cp[f]));
                    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(t1) : "l"(a1), "l"(cp[f]));
                    s[0] = fma2(t0, t0, s[0]);
                    s[1] = fma2(t1, t1, s[1]);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int gr = r0 + r + h;
                    if (gr >= n) break;  // warp-uniform
                    // a key can beat the row's k-th key only if its distance
                    // is at most the k-th distance: test the distances first
                    const uint64_t kk = sh.L.kth[r + h];
                    const float kd = kk == kKeyMax ? __int_as_float(0x7f800000) : __uint_as_float(key_bits(kk));
                    if (!__any_sync(0xffffffffu, (lo_f(s[h]) <= kd) | (hi_f(s[h]) <= kd))) continue;
                    uint64_t key[2] = {(static_cast<uint64_t>(__float_as_uint(lo_f(s[h]))) << 32) | cidx[0],
                                       (static_cast<uint64_t>(__float_as_uint(hi_f(s[h]))) << 32) | cidx[1]};
                    if (own) {  // a row is not its own neighbour
                        if (cc == gr) key[0] = kKeyMax;
                        if (cc + 1 == gr) key[1] = kKeyMax;
                    }
                    offer_row(sh.L, r + h, key, k);
                }
            }
            }
            __syncthreads();
        }
        // the k best per row, written in the reference's slot order
        for (int rr = 0; rr < kRowsPerWarp; ++rr) {
            const int r = rw + rr;
            if (r0 + r >= n) break;
            const int il = static_cast<int>(li[r0 + r]);  // the row's original index
            compact_row<kBM>(sh.L, r, k, 0.0f, 8);
            const uint64_t kth = sh.L.list[r][k - 1];
            const uint32_t kbits = key_bits(kth);
            int below = 0;
            for (int e = lane; e < k; e += 32) below += key_bits(sh.L.list[r][e]) < kbits ? 1 : 0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) below += __shfl_xor_sync(0xffffffffu, below, o);
            int32_t* oi = nbr_idx + nkoff[p];
            float* od = nbr_d2 + nkoff[p];
            for (int e = lane; e < k; e += 32) {
                const uint64_t y = sh.L.list[r][e];
                int slot = e;
                if (e < below) {
                    const uint32_t yi = key_index(y);
                    slot = 0;
                    for (int q = 0; q < below; ++q) slot += key_index(sh.L.list[r][q]) < yi ? 1 : 0;
                }
                oi[static_cast<int64_t>(slot) * n + il] = static_cast<int32_t>(key_index(y));
                od[static_cast<int64_t>(slot) * n + il] = __uint_as_float(key_bits(y));
            }
            if (lane == 0) kdist2[base + il] = __uint_as_float(kbits);
        }
        __syncthreads();
    }
}

// ---- batched lrd and scores (lof.cu's arithmetic, local indices) -------------

__global__ void bl_lrd_kernel(int64_t ntot, const int* __restrict__ pid, const int64_t* __restrict__ off,
                              const int* __restrict__ ks, const int64_t* __restrict__ nkoff,
                              const int32_t* __restrict__ nbr_idx, const float* __restrict__ nbr_d2,
                              const float* __restrict__ kdist2, float* __restrict__ lrd) {
    const int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (g >= ntot) return;
    const int p = pid[g];
    const int64_t base = off[p];
    const int64_t n = off[p + 1] - base, i = g - base;
    const int k = ks[p];
    const int32_t* ni = nbr_idx + nkoff[p];
    const float* nd = nbr_d2 + nkoff[p];
    double sum = 0.0;
    for (int t = 0; t < k; ++t) {
        const int64_t o = static_cast<int64_t>(t) * n + i;
        const int32_t j = ni[o];
        const float kj = (j >= 0 && j < n) ? kdist2[base + j] : __int_as_float(0x7fc00000);
        sum = __dadd_rn(sum, __dsqrt_rn(widen(fmaxf(kj, nd[o]))));
    }
    lrd[g] = __double2float_rn(__ddiv_rn(1.0, __dadd_rn(__ddiv_rn(sum, static_cast<double>(k)), 1e-10)));
}

__global__ void bl_score_kernel(int64_t ntot, const int* __restrict__ pid, const int64_t* __restrict__ off,
                                const int* __restrict__ ks, const int64_t* __restrict__ nkoff,
                                const int32_t* __restrict__ nbr_idx, const float* __restrict__ lrd,
                                float* __restrict__ scores) {
    const int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (g >= ntot) return;
    const int p = pid[g];
    const int64_t base = off[p];
    const int64_t n = off[p + 1] - base, i = g - base;
    const int k = ks[p];
    const int32_t* ni = nbr_idx + nkoff[p];
    const double self = widen(lrd[g]), y = __ddiv_rn(1.0, self);
    const bool quick = quotient_quick(y);
    double sum = 0.0;
    for (int t = 0; t < k; ++t) {
        const int32_t j = ni[static_cast<int64_t>(t) * n + i];
        sum = __dadd_rn(sum, quotient((j >= 0 && j < n) ? lrd[base + j] : __int_as_float(0x7fc00000), self, y, quick));
    }
    scores[g] = __double2float_rn(__ddiv_rn(sum, static_cast<double>(k)));
}

__global__ void pid_kernel(const int64_t* __restrict__ off, int num, int* __restrict__ pid) {
    // one block per problem
    for (int p = blockIdx.x; p < num; p += gridDim.x)
        for (int64_t i = off[p] + threadIdx.x; i < off[p + 1]; i += blockDim.x) pid[i] = p;
}

int dp_for(int d) { return d <= 32 ? 32 : 64; }  // (up to 16 features: the sweep)

template <int DP>
void launch_knn(int grid, const BatchDev& b, cudaStream_t s) {
    const size_t smem = sizeof(BatchSmem<DP>);
    set_max_dynamic_smem(reinterpret_cast<const void*>(batched_knn_kernel<DP>), static_cast<int>(smem));
    batched_knn_kernel<DP><<<grid, kThreads, smem, s>>>(b.xs, b.lidx, b.off, b.ks, b.nkoff, b.items, b.nitems, b.d,
                                                       b.counter, b.nbr, b.d2, b.kd);
    CG_LAUNCH_CHECK();
}

constexpr int kSweepMaxD = 16;  // more features take batched_knn_kernel
int sweep_dp(int d) { return d <= 4 ? 4 : d <= 8 ? 8 : d <= 12 ? 12 : 16; }

// The items of one list form, [first, first + count). one_cta: shared memory
// padded so that a single CTA fits on an SM.
template <int DP, int KR, int G>
void launch_sweep(const BatchDev& b, int first, int count, bool one_cta, int* status, cudaStream_t s) {
    if (count == 0) return;
    size_t smem = sizeof(small::SmallSmem<DP, KR, 8, kWarps>);
    set_max_dynamic_smem(reinterpret_cast<const void*>(batched_sweep_kernel<DP, KR, G>), 227 * 1024);
    if (one_cta) smem = std::max<size_t>(smem, 120 * 1024);
    batched_sweep_kernel<DP, KR, G><<<static_cast<unsigned>(count) * 2, kThreads, smem, s>>>(
        b.tiles, b.tbox, b.off, b.ks, b.nkoff, b.toff, b.items + first, b.nbr, b.d2, b.kd, status);
    CG_LAUNCH_CHECK();
}
template <int DP>
void launch_sweeps(const BatchDev& b, bool one_cta, int* status, cudaStream_t s) {
    launch_sweep<DP, 2, 2>(b, 0, b.group[0], one_cta, status, s);
    launch_sweep<DP, 1, 2>(b, b.group[0], b.group[1], one_cta, status, s);
    launch_sweep<DP, 1, 1>(b, b.group[0] + b.group[1], b.group[2], one_cta, status, s);
}
template <int DP>
void launch_tiles(const BatchDev& b, const unsigned* perm, cudaStream_t s) {
    bm_tile_kernel<DP><<<static_cast<unsigned>(b.ntiles), kCT, 0, s>>>(b.xc, b.d, perm, b.off, b.tpid, b.toff, b.tiles,
                                                                       b.tbox);
    CG_LAUNCH_CHECK();
}

int grid_cap(int64_t items) {
    int64_t g = ceil_div(items, 256);
    if (g > 152 * 16) g = 152 * 16;
    return static_cast<int>(g < 1 ? 1 : g);
}

}  // namespace

// ---- host orchestration --------------------------------------------------------

void Engine::batch_plan(int num, const int64_t* offsets, const int* ks, int d, bool normalize) {
    if (num < 1) throw Error(kInvalidArgument, "num_problems must be >= 1");
    if (!offsets || !ks) throw Error(kInvalidArgument, "offsets and ks must not be null");
    if (d < 1 || d > kBMaxD) throw Error(kInvalidArgument, "the batched path takes 1 <= n_dims <= 64");
    if (offsets[0] != 0) throw Error(kInvalidArgument, "offsets[0] must be 0");
    BatchPlan P;  // (a refused layout leaves the planned one as it was)
    P.num = num;
    P.d = d;
    P.normalize = normalize;
    P.off.assign(offsets, offsets + num + 1);
    P.ks.assign(ks, ks + num);
    P.nkoff.assign(num + 1, 0);
    P.coff.assign(num + 1, 0);
    P.toff.assign(num + 1, 0);
    std::vector<int> tp;
    std::vector<std::pair<int64_t, uint2>> items;
    std::vector<int> cp;
    for (int p = 0; p < num; ++p) {
        const int64_t n = offsets[p + 1] - offsets[p];
        const int k = ks[p];
        if (n < 2 || n > 0x7FFFFFFFll) {
            std::ostringstream os;
            os << "problem " << p << ": n_points must be >= 2 (got " << n << ")";
            throw Error(kInvalidArgument, os.str());
        }
        if (k < 1 || k >= n || k > kBMaxK) {
            std::ostringstream os;
            os << "problem " << p << ": k must satisfy 1 <= k <= n_points - 1 and k <= " << kBMaxK << " (got k=" << k
               << ", n_points=" << n << ")";
            throw Error(kInvalidArgument, os.str());
        }
        P.nkoff[p + 1] = P.nkoff[p] + n * k;
        const int64_t chunks = ceil_div(n, kCenterChunk);
        P.coff[p + 1] = P.coff[p] + chunks;
        for (int64_t c = 0; c < chunks; ++c) cp.push_back(p);
        const int64_t tiles = ceil_div(n, kRT);
        P.toff[p + 1] = P.toff[p] + tiles;
        for (int64_t t = 0; t < tiles; ++t) {
            items.push_back({n, make_uint2(static_cast<unsigned>(p), static_cast<unsigned>(t))});
            tp.push_back(p);
        }
    }
    // largest problems first: their items are the longest, the tail stays short
    std::stable_sort(items.begin(), items.end(),
                     [](const std::pair<int64_t, uint2>& a, const std::pair<int64_t, uint2>& b) { return a.first > b.first; });
    // the sweep's list forms (k > 32, k > 24, the rest) are launched one after
    // another, each largest problems first
    const auto form = [&](const std::pair<int64_t, uint2>& it) {
        const int k = ks[it.second.x];
        return k > 32 ? 0 : k > 24 ? 1 : 2;
    };
    if (d <= kSweepMaxD)
        std::stable_sort(items.begin(), items.end(),
                         [&](const std::pair<int64_t, uint2>& a, const std::pair<int64_t, uint2>& b) { return form(a) < form(b); });
    // From here to the end no layout is planned: a call that runs out of memory
    // leaves nothing that a later one could match.
    bgraph_valid_ = false;
    btuned_ = false;
    bplan_.num = 0;
    for (int& g : bdev_.group) g = 0;
    for (const auto& it : items) ++bdev_.group[form(it)];
    P.items.resize(items.size());
    for (size_t i = 0; i < items.size(); ++i) P.items[i] = items[i].second;
    P.ntot = offsets[num];
    P.nchunks = P.coff[num];
    // device copies of the plan (synchronous, before any capture)
    cudaStream_t s = stream_;
    BatchDev& b = bdev_;
    b.off = bplan_off_.as<int64_t>(num + 1);
    b.nkoff = bplan_nkoff_.as<int64_t>(num + 1);
    b.coff = bplan_coff_.as<int64_t>(num + 1);
    b.ks = bplan_ks_.as<int>(num);
    b.items = bplan_items_.as<uint2>(P.items.size());
    b.cp = bplan_cp_.as<int>(cp.size() ? cp.size() : 1);
    b.toff = bplan_toff_.as<int64_t>(num + 1);
    b.tpid = bplan_tpid_.as<int>(tp.size());
    b.ntiles = static_cast<int64_t>(tp.size());
    CG_CUDA(cudaMemcpyAsync(b.toff, P.toff.data(), sizeof(int64_t) * (num + 1), cudaMemcpyHostToDevice, s));
    CG_CUDA(cudaMemcpyAsync(b.tpid, tp.data(), sizeof(int) * tp.size(), cudaMemcpyHostToDevice, s));
    CG_CUDA(cudaMemcpyAsync(b.off, P.off.data(), sizeof(int64_t) * (num + 1), cudaMemcpyHostToDevice, s));
    CG_CUDA(cudaMemcpyAsync(b.nkoff, P.nkoff.data(), sizeof(int64_t) * (num + 1), cudaMemcpyHostToDevice, s));
    CG_CUDA(cudaMemcpyAsync(b.coff, P.coff.data(), sizeof(int64_t) * (num + 1), cudaMemcpyHostToDevice, s));
    CG_CUDA(cudaMemcpyAsync(b.ks, P.ks.data(), sizeof(int) * num, cudaMemcpyHostToDevice, s));
    CG_CUDA(cudaMemcpyAsync(b.items, P.items.data(), sizeof(uint2) * P.items.size(), cudaMemcpyHostToDevice, s));
    CG_CUDA(cudaMemcpyAsync(b.cp, cp.data(), sizeof(int) * cp.size(), cudaMemcpyHostToDevice, s));
    b.nitems = static_cast<int>(P.items.size());
    b.d = d;
    // workspaces
    b.pid = bpid_.as<int>(P.ntot);
    b.xc = bxc_.as<float>(static_cast<size_t>(P.ntot) * d);
    b.partial = bpartial_.as<double>(static_cast<size_t>(P.nchunks) * d);
    b.mean = bmean_.as<double>(static_cast<size_t>(num) * d);
    b.inv = binv_.as<double>(static_cast<size_t>(num) * d);
    b.nbr = bnbr_.as<int32_t>(P.nkoff[num]);
    b.d2 = bd2_.as<float>(P.nkoff[num]);
    b.kd = bkd_.as<float>(P.ntot);
    b.lrd = blrd_.as<float>(P.ntot);
    b.counter = bcounter_.as<unsigned>(1);
    const bool sweep = d <= kSweepMaxD;
    const int width = sweep ? sweep_dp(d) : d;  // of a box
    b.xs = sweep ? nullptr : bxs_.as<float>(static_cast<size_t>(P.ntot) * d);
    if (sweep) b.tiles = btiles_.as<float>(static_cast<size_t>(b.ntiles) * small::tile_floats(width));
    b.lidx = blidx_.as<unsigned>(P.ntot);
    b.pmm = bpmm_.as<float>(static_cast<size_t>(num) * d * 2);
    b.pdims = bpdims_.as<int>(static_cast<size_t>(num) * kMortonDimsB);
    b.skeys = bskeys_.as<unsigned>(2 * static_cast<size_t>(P.ntot));
    b.svals = bsvals_.as<unsigned>(2 * static_cast<size_t>(P.ntot));
    b.scounts = bscounts_.as<unsigned>(sort_pairs_counts(P.ntot));
    b.tbox = btbox_.as<float>(static_cast<size_t>(b.ntiles) * 2 * width);
    pid_kernel<<<num < 4096 ? num : 4096, 256, 0, s>>>(b.off, num, b.pid);
    CG_LAUNCH_CHECK();
    CG_CUDA(cudaStreamSynchronize(s));
    bplan_ = std::move(P);
}

void Engine::batch_launch(const float* d_x, float* d_scores) {
    const BatchPlan& P = bplan_;
    BatchDev& b = bdev_;
    cudaStream_t s = stream_;
    const int d = P.d;
    const int64_t cd = P.nchunks * d;
    const unsigned pgrid = static_cast<unsigned>(ceil_div(cd, 64));  // a chain of kCenterChunk additions per thread
    bc_partials_kernel<false><<<pgrid, 64, 0, s>>>(d_x, b.off, d, b.cp, b.coff, P.nchunks, nullptr, b.partial);
    CG_LAUNCH_CHECK();
    bc_finalize_kernel<<<static_cast<unsigned>(ceil_div(static_cast<int64_t>(P.num) * d, 128)), 128, 0, s>>>(
        b.partial, b.off, b.coff, P.num, d, 0, b.mean, b.inv);
    CG_LAUNCH_CHECK();
    if (P.normalize) {
        bc_partials_kernel<true><<<pgrid, 64, 0, s>>>(d_x, b.off, d, b.cp, b.coff, P.nchunks, b.mean, b.partial);
        CG_LAUNCH_CHECK();
        bc_finalize_kernel<<<static_cast<unsigned>(ceil_div(static_cast<int64_t>(P.num) * d, 128)), 128, 0, s>>>(
            b.partial, b.off, b.coff, P.num, d, 1, b.mean, b.inv);
        CG_LAUNCH_CHECK();
    }
    if (P.normalize)
        bc_apply_kernel<true><<<grid_cap(P.ntot * d), kApplyThreads, 0, s>>>(d_x, P.ntot, d, b.pid, b.mean, b.inv, b.xc);
    else
        bc_apply_kernel<false><<<grid_cap(P.ntot * d), kApplyThreads, 0, s>>>(d_x, P.ntot, d, b.pid, b.mean, b.inv, b.xc);
    CG_LAUNCH_CHECK();
    // spatial order within each problem: Morton keys, stable sort by key,
    // then stable sort by problem (keeps each problem's range in place)
    bm_minmax_kernel<<<P.num, kMinMaxThreads, 0, s>>>(b.xc, b.off, d, b.pmm, b.pdims);
    CG_LAUNCH_CHECK();
    bm_morton_kernel<<<grid_cap(P.ntot), 256, 0, s>>>(b.xc, P.ntot, d, b.pid, b.pmm, b.pdims, b.skeys, b.svals);
    CG_LAUNCH_CHECK();
    unsigned* vs = nullptr;
    unsigned* ks1 = sort_pairs_stable(b.skeys, b.svals, b.skeys + P.ntot, b.svals + P.ntot, P.ntot, 32, b.scounts, s, &vs);
    unsigned* kother = ks1 == b.skeys ? b.skeys + P.ntot : b.skeys;
    unsigned* vother = vs == b.svals ? b.svals + P.ntot : b.svals;
    bm_pidkey_kernel<<<grid_cap(P.ntot), 256, 0, s>>>(P.ntot, b.pid, vs, ks1);
    CG_LAUNCH_CHECK();
    int pbits = 8;
    while (pbits < 32 && (static_cast<int64_t>(1) << pbits) < P.num) pbits += 8;
    unsigned* perm = nullptr;
    sort_pairs_stable(ks1, vs, kother, vother, P.ntot, pbits, b.scounts, s, &perm);
    if (d <= kSweepMaxD) {
        const bool one_cta = btune_grid_ == bsms_;
        CG_CUDA(cudaMemsetAsync(status_ptr(), 0, sizeof(int), s));
        switch (sweep_dp(d)) {
            case 4: launch_tiles<4>(b, perm, s); launch_sweeps<4>(b, one_cta, status_ptr(), s); break;
            case 8: launch_tiles<8>(b, perm, s); launch_sweeps<8>(b, one_cta, status_ptr(), s); break;
            case 12: launch_tiles<12>(b, perm, s); launch_sweeps<12>(b, one_cta, status_ptr(), s); break;
            default: launch_tiles<16>(b, perm, s); launch_sweeps<16>(b, one_cta, status_ptr(), s); break;
        }
    } else {
        bm_gather_kernel<<<grid_cap(P.ntot * d), 256, 0, s>>>(b.xc, P.ntot, d, perm, b.pid, b.off, b.xs, b.lidx);
        CG_LAUNCH_CHECK();
        CG_CUDA(cudaMemsetAsync(b.counter, 0, sizeof(unsigned), s));
        if (dp_for(d) == 32) launch_knn<32>(btune_grid_, b, s);
        else launch_knn<64>(btune_grid_, b, s);
    }
    bl_lrd_kernel<<<static_cast<unsigned>(ceil_div(P.ntot, 256)), 256, 0, s>>>(P.ntot, b.pid, b.off, b.ks, b.nkoff,
                                                                               b.nbr, b.d2, b.kd, b.lrd);
    CG_LAUNCH_CHECK();
    bl_score_kernel<<<static_cast<unsigned>(ceil_div(P.ntot, 256)), 256, 0, s>>>(P.ntot, b.pid, b.off, b.ks,
                                                                                 b.nkoff, b.nbr, b.lrd, d_scores);
    CG_LAUNCH_CHECK();
}

// Time the k-NN kernel's variants on this batch (once per layout).
void Engine::batch_autotune(const float* d_x, float* d_scores) {
    int sms = 152;
    CG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device_));
    const size_t smem = dp_for(bplan_.d) == 32 ? sizeof(BatchSmem<32>) : sizeof(BatchSmem<64>);
    int max_per_sm = static_cast<int>(227 * 1024 / (smem + 1024));
    if (max_per_sm < 1) max_per_sm = 1;
    if (max_per_sm > 2) max_per_sm = 2;
    const bool sweep = bplan_.d <= kSweepMaxD;  // one CTA per SM, or (2) as many as fit
    if (sweep) max_per_sm = 2;
    bsms_ = sms;
    cudaEvent_t e0, e1;
    CG_CUDA(cudaEventCreate(&e0));
    CG_CUDA(cudaEventCreate(&e1));
    float best = 1e30f;
    for (float& t : btune_ms_) t = -1.0f;
    for (int per = 1; per <= max_per_sm; ++per) {
        btune_grid_ = per * sms;
        batch_launch(d_x, d_scores);  // warm (first use configures the kernel)
        CG_CUDA(cudaEventRecord(e0, stream_));
        batch_launch(d_x, d_scores);
        CG_CUDA(cudaEventRecord(e1, stream_));
        CG_CUDA(cudaEventSynchronize(e1));
        float ms = 0.0f;
        CG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        btune_ms_[2 * (per - 1)] = ms;
        if (ms < best) {
            best = ms;
            bbest_grid_ = btune_grid_;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    btune_grid_ = bbest_grid_;
    btuned_ = true;
}

bool Engine::batch_same_plan(int num, const int64_t* offsets, const int* ks, int d, bool normalize) const {
    const BatchPlan& P = bplan_;
    if (P.num != num || P.d != d || P.normalize != normalize) return false;
    if (std::memcmp(P.off.data(), offsets, sizeof(int64_t) * (num + 1)) != 0) return false;
    return std::memcmp(P.ks.data(), ks, sizeof(int) * num) == 0;
}

void Engine::lof_batched_device(int num, const int64_t* offsets, const int* ks, const float* d_x, int d,
                                bool normalize, float* d_scores) {
    if (!d_x || !d_scores) throw Error(kInvalidArgument, "device pointers must not be null");
    if (!offsets || !ks) throw Error(kInvalidArgument, "offsets and ks must not be null");
    CG_CUDA(cudaSetDevice(device_));
    if (!(bplan_.num > 0 && batch_same_plan(num, offsets, ks, d, normalize))) batch_plan(num, offsets, ks, d, normalize);
    if (!btuned_) batch_autotune(d_x, d_scores);
    if (!use_graphs_) {
        batch_launch(d_x, d_scores);
        return;
    }
    if (!bgraph_valid_ || bgraph_x_ != d_x || bgraph_scores_ != d_scores || bgraph_stream_ != stream_) {
        if (bgraph_exec_) {
            cudaGraphExecDestroy(bgraph_exec_);
            bgraph_exec_ = nullptr;
        }
        bgraph_valid_ = false;
        cudaGraph_t g = nullptr;
        const unsigned long long before = launch_count();
        CG_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
        try {
            batch_launch(d_x, d_scores);
        } catch (...) {
            cudaStreamEndCapture(stream_, &g);
            if (g) cudaGraphDestroy(g);
            throw;
        }
        CG_CUDA(cudaStreamEndCapture(stream_, &g));
        bgraph_kernels_ = launch_count() - before;  // captured, not launched
        uncount_launches(bgraph_kernels_);
        const cudaError_t ie = cudaGraphInstantiate(&bgraph_exec_, g, 0);
        cudaGraphDestroy(g);
        CG_CUDA(ie);
        bgraph_valid_ = true;
        bgraph_x_ = d_x;
        bgraph_scores_ = d_scores;
        bgraph_stream_ = stream_;
    }
    CG_CUDA(cudaGraphLaunch(bgraph_exec_, stream_));
    count_launches(bgraph_kernels_);
}

void Engine::lof_batched_host(int num, const int64_t* offsets, const int* ks, const float* x, int d, bool normalize,
                              float* scores) {
    if (!x || !scores) throw Error(kInvalidArgument, "points and scores must not be null");
    if (num < 1 || !offsets) throw Error(kInvalidArgument, "num_problems must be >= 1");
    CG_CUDA(cudaSetDevice(device_));
    const int64_t ntot = offsets[num];
    if (ntot < 0) throw Error(kInvalidArgument, "offsets must be non-decreasing");
    float* dx = x_.as<float>(static_cast<size_t>(ntot) * (d > 0 ? d : 1));
    float* ds = scores_.as<float>(static_cast<size_t>(ntot > 0 ? ntot : 1));
    CG_CUDA(cudaMemcpyAsync(dx, x, sizeof(float) * ntot * d, cudaMemcpyHostToDevice, stream_));
    lof_batched_device(num, offsets, ks, dx, d, normalize, ds);
    CG_CUDA(cudaMemcpyAsync(scores, ds, sizeof(float) * ntot, cudaMemcpyDeviceToHost, stream_));
    check_status();
}

}  // namespace culof_gb300

namespace culof_gb300 {
void Engine::batched_tuning(float* ms4, int* per_sm, int* pairs_per_lane) const {
    for (int i = 0; i < 4; ++i) ms4[i] = btuned_ ? btune_ms_[i] : -1.0f;
    const int sms = bbest_grid_ > 0 ? bbest_grid_ : 1;
    int dev_sms = 152;
    cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, device_);
    *per_sm = btuned_ ? sms / (dev_sms > 0 ? dev_sms : 1) : 0;
    *pairs_per_lane = btuned_ ? 1 : 0;
}
}  // namespace culof_gb300
