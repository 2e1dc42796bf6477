// The fast exact k-NN path: fused distance + filtered exact select.
//
// Replaces the reference's hot loop (pipeline.cu:175-195: cuBLAS SGEMM of a
// rows x n Gram tile to HBM, then knn_select_kernel's four sweeps of it,
// knn.cu:119-232, ~24 B of HBM traffic per pair) with one evaluation per
// pair that never leaves the SM:
//
//  1. spatial order: a 32-bit Morton key of the centred coordinates, sorted
//     with a stable LSD radix sort; tiles of 128 consecutive sorted points
//     are spatially compact.
//  2. d <= 8: one kernel per row tile (small.cu) with per-row pruning.
//     Wider points: a sweep over the column tiles on the tensor cores
//     (tc_sweep.cu) or in FP32 (wide.cu, started from a seed: per row, the
//     exact k best over its own tile): a filter value per pair is compared
//     with a per-row threshold, a rigorous error bound over the row's current
//     k-th key, so every column that can still enter the k best passes and is
//     rescored exactly.
//  3. the tensor path's final kernel, or the FP32 path's merge of its seed and
//     S column-split lists, gives the k best keys; slots are written in the
//     reference's order (keys below the k-th by ascending index, then the
//     ties, knn.cu:190-224).
//
// Exactness: the selection key is (exact float32 distance bits, original
// index), identical to the general path and the oracle; the filter only
// decides which pairs get an exact evaluation, and its bound is proven
// conservative (sweep_common.cuh: tau_from; tc_sweep.cu: row_bounds).
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <utility>

#include "common.cuh"
#include "block.cuh"
#include "engine.cuh"
#include "fast.cuh"
#include "prep.cuh"
#include "small.cuh"
#include "sweep_common.cuh"
#include "tc_scale.cuh"
#include "warp_sort.cuh"

namespace culof_gb300 {

namespace {

using namespace small;

constexpr int kSeedWindow = 5;  // tiles of the seed: T, T+1, T-1, T+2, T-2
constexpr int kMaxWideD = 128;
constexpr int kMortonDims = 8;  // Morton key over (up to) the 8 widest dimensions

// ---------------------------------------------------------------- spatial order

// 32-bit Morton key: 32/m bits for each of the (up to) kMortonDims features of
// the widest range, widest first (ties by index), interleaved from the most
// significant bit, over the bounding box of the centred data (mm, see
// center()). Every block picks the features itself, with one warp. With tc, a
// warp of the last block also writes what the tensor path starts from (in a
// launch of its own it took 3.3 us).
__global__ void morton_kernel(const float* __restrict__ xc, int64_t n, int d, const unsigned* __restrict__ mm,
                              unsigned* __restrict__ keys, unsigned* __restrict__ vals,
                              const unsigned* __restrict__ max_norm_bits, TcStart* __restrict__ tc) {
    __shared__ int dims[kMortonDims];
    __shared__ float dlo[kMortonDims], dspan[kMortonDims];
    const int md = d < kMortonDims ? d : kMortonDims;
    const int bits = (32 / md) < 30 ? (32 / md) : 30;
    if (tc != nullptr && blockIdx.x == gridDim.x - 1 && threadIdx.x / 32 == 1) tc_start(mm, d, max_norm_bits, tc);
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        float span[kMaxTensorD / 32];
#pragma unroll
        for (int j = 0; j < kMaxTensorD / 32; ++j) {
            const int f = 32 * j + lane;
            span[j] = f < d ? range_hi(mm, f) - range_lo(mm, f) : -1.0f;
        }
        for (int q = 0; q < md; ++q) {
            float best = -1.0f;
            int at = d;
#pragma unroll
            for (int j = 0; j < kMaxTensorD / 32; ++j)
                if (span[j] > best) {
                    best = span[j];
                    at = 32 * j + lane;
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int oa = __shfl_xor_sync(0xffffffffu, at, o);
                if (ob > best || (ob == best && oa < at)) {
                    best = ob;
                    at = oa;
                }
            }
            if (at >= d) at = q;  // (ranges that are not numbers: any feature)
#pragma unroll
            for (int j = 0; j < kMaxTensorD / 32; ++j)
                if (32 * j + lane == at) span[j] = -2.0f;
            if (lane == 0) {
                dims[q] = at;
                dlo[q] = range_lo(mm, at);
                dspan[q] = range_hi(mm, at) - range_lo(mm, at);
            }
        }
    }
    __syncthreads();
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        unsigned q[kMortonDims];
        for (int j = 0; j < md; ++j) {
            const float span = dspan[j];
            float t = span > 0.0f ? (xc[i * d + dims[j]] - dlo[j]) / span : 0.0f;
            t = fminf(fmaxf(t, 0.0f), 1.0f);
            const float scale = static_cast<float>((1u << bits) - 1u);
            q[j] = static_cast<unsigned>(t * scale + 0.5f);
        }
        unsigned key = 0u;
        for (int b = bits - 1; b >= 0; --b)
            for (int j = 0; j < md; ++j) key = (key << 1) | ((q[j] >> b) & 1u);
        keys[i] = key;
        vals[i] = static_cast<unsigned>(i);
    }
}

// ---- stable LSD radix sort, 8-bit digits, 2048 items per block -------------
constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;

__global__ void sort_upsweep_kernel(const unsigned* __restrict__ keys, int64_t n, int shift,
                                    unsigned* __restrict__ counts, int nblocks) {
    __shared__ unsigned hist[256];
    hist[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kSortTile;
    for (int it = 0; it < kSortItems; ++it) {
        const int64_t i = base + static_cast<int64_t>(it) * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&hist[(keys[i] >> shift) & 0xFF], 1u);
    }
    __syncthreads();
    counts[static_cast<int64_t>(threadIdx.x) * nblocks + blockIdx.x] = hist[threadIdx.x];
}

// Exclusive scan of each digit's row counts[digit][0 .. nblocks) and the row's
// total, one block per digit (the downsweep adds the lower digits' totals; one
// block scanning all rows took 14 us at n = 200,000 and 38 us at a million).
constexpr int kRowScanThreads = 256;
__global__ void __launch_bounds__(kRowScanThreads) sort_rowscan_kernel(unsigned* __restrict__ counts, int nblocks,
                                                                       unsigned* __restrict__ totals) {
    __shared__ int warp_sums[kRowScanThreads / 32];
    unsigned* row = counts + static_cast<int64_t>(blockIdx.x) * nblocks;
    unsigned carry = 0;
    for (int b0 = 0; b0 < nblocks; b0 += kRowScanThreads) {
        const int b = b0 + static_cast<int>(threadIdx.x);
        const int v = b < nblocks ? static_cast<int>(row[b]) : 0;
        int total;
        const int excl = block_exclusive_scan(v, warp_sums, total);
        if (b < nblocks) row[b] = carry + static_cast<unsigned>(excl);
        carry += static_cast<unsigned>(total);
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

__global__ void sort_downsweep_kernel(const unsigned* __restrict__ keys_in, const unsigned* __restrict__ vals_in,
                                      unsigned* __restrict__ keys_out, unsigned* __restrict__ vals_out, int64_t n,
                                      int shift, const unsigned* __restrict__ offsets,
                                      const unsigned* __restrict__ totals, int nblocks) {
    __shared__ unsigned wcount[kWarps][256];
    __shared__ unsigned first[256];  // first place of each digit
    __shared__ int warp_sums[kWarps];
    {
        int all;
        first[threadIdx.x] = static_cast<unsigned>(block_exclusive_scan(static_cast<int>(totals[threadIdx.x]), warp_sums, all));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int d = lane; d < 256; d += 32) wcount[warp][d] = 0;
    __syncwarp();
    // warp w owns elements [w*256, (w+1)*256) of the block tile, 32 at a time
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kSortTile + warp * (kSortTile / kWarps);
    unsigned key[kSortItems], val[kSortItems], rank[kSortItems];
    const unsigned lt = (1u << lane) - 1u;
    for (int it = 0; it < kSortItems; ++it) {
        const int64_t i = base + it * 32 + lane;
        const bool valid = i < n;
        key[it] = valid ? keys_in[i] : 0u;
        val[it] = valid ? vals_in[i] : 0u;
        const unsigned dg = valid ? ((key[it] >> shift) & 0xFF) : 256u;
        const unsigned peers = __match_any_sync(0xffffffffu, dg);
        const unsigned r = __popc(peers & lt);
        unsigned prior = 0;
        if (valid) prior = wcount[warp][dg];
        rank[it] = prior + r;
        __syncwarp();
        if (valid && r == 0) wcount[warp][dg] = prior + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // per digit: exclusive prefix over warps
    {
        const int dg = threadIdx.x;  // 256 threads = 256 digits
        unsigned run = 0;
        for (int w = 0; w < kWarps; ++w) {
            const unsigned t = wcount[w][dg];
            wcount[w][dg] = run;
            run += t;
        }
    }
    __syncthreads();
    for (int it = 0; it < kSortItems; ++it) {
        const int64_t i = base + it * 32 + lane;
        if (i < n) {
            const unsigned dg = (key[it] >> shift) & 0xFF;
            const unsigned pos =
                first[dg] + offsets[static_cast<int64_t>(dg) * nblocks + blockIdx.x] + wcount[warp][dg] + rank[it];
            keys_out[pos] = key[it];
            vals_out[pos] = val[it];
        }
    }
}

// ---------------------------------------------------------------- seed

// Exact distances (the oracle's formula: t = a - b, s = fma(t, t, s) over the
// dimensions in order) from row a (each coordinate duplicated into both
// halves) to the two columns of pair p of a tile, with packed f32x2
// instructions: per element the same IEEE operations as the scalar chain.
template <int DP>
__device__ __forceinline__ void pair_dist2(const float* tile, int p, const uint64_t (&a2)[DP], float& d0, float& d1) {
    uint64_t s = 0;  // (+0, +0)
#pragma unroll
    for (int f = 0; f < DP; ++f) {
        const uint64_t t = sub2(a2[f], *reinterpret_cast<const uint64_t*>(tile + f * kCT + 2 * p));
        s = fma2(t, t, s);
    }
    d0 = lo_f(s);
    d1 = hi_f(s);
}

// Per row tile T (one block): the column tiles that can hold a candidate for
// any of its rows under the seed's k-th distances, in visiting order (the
// tensor sweep over d <= 8 points visits only those), each with its
// rounded-down box gap.
template <int DP>
__global__ void __launch_bounds__(256) prune_list_kernel(const float* __restrict__ boxes, int nt, int t0, int qs,
                                                         const unsigned long long* __restrict__ kth_seed,
                                                         uint2* __restrict__ plist, int* __restrict__ pcount) {
    __shared__ float tbox[2][DP];
    __shared__ float kmax_s;
    __shared__ int wtot[8];
    __shared__ int base_s;
    const int T = t0 + static_cast<int>(blockIdx.x);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 2 * DP)
        tbox[threadIdx.x / DP][threadIdx.x % DP] = boxes[static_cast<int64_t>(T) * 2 * DP + threadIdx.x];
    if (warp == 0) {
        float v = __int_as_float(0xff800000);
        for (int r = lane; r < kRT; r += 32) {
            const unsigned long long kk = kth_seed[static_cast<int64_t>(T) * kRT + r];
            v = fmaxf(v, kk == kKeyMax ? __int_as_float(0x7f800000) : __uint_as_float(key_bits(kk)));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) {
            kmax_s = v;
            base_s = 0;
        }
    }
    __syncthreads();
    const float kmax = kmax_s;
    uint2* out = plist + static_cast<int64_t>(T) * nt;
    for (int q0 = qs; q0 < nt; q0 += 256) {
        const int q = q0 + static_cast<int>(threadIdx.x);
        bool pass = false;
        unsigned t = 0;
        float g2 = 0.0f;
        if (q < nt) {
            t = static_cast<unsigned>(spiral_tile(T, q, nt));
            const float* b = boxes + static_cast<int64_t>(t) * 2 * DP;
#pragma unroll
            for (int f = 0; f < DP; ++f) {
                const float gap = fmaxf(0.0f, fmaxf(__fsub_rd(b[f], tbox[1][f]), __fsub_rd(tbox[0][f], b[DP + f])));
                g2 = __fadd_rd(g2, __fmul_rd(gap, gap));
            }
            pass = !(__fmul_rd(g2, prune_shrink<DP>()) > kmax);
        }
        const unsigned m = __ballot_sync(0xffffffffu, pass);
        if (lane == 0) wtot[warp] = __popc(m);
        __syncthreads();
        int before = base_s;
        for (int w = 0; w < warp; ++w) before += wtot[w];
        if (pass) out[before + __popc(m & ((1u << lane) - 1u))] = make_uint2(t, __float_as_uint(g2));
        __syncthreads();
        if (threadIdx.x == 0) {
            int tot = 0;
            for (int w = 0; w < 8; ++w) tot += wtot[w];
            base_s += tot;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) pcount[T] = base_s;
}

// (The tensor path over d <= 8 points.) Per row of tile T: the exact k best keys
// over the seed window (sorted, kKeyMax padded) and its k-th key, from which the
// sweep's thresholds start (kth_shared). The window is the first qs spiral
// positions: tile T itself and its Morton neighbours T+1, T-1, T+2 and T-2, whose
// points start the k-th distances much closer to their final values than tile T
// alone (fewer candidates reach the sweep's lists); the sweep covers the spiral
// from position qs on.
template <int DP>
__global__ void __launch_bounds__(kThreads) seed_kernel(const float* __restrict__ tiles, int nt, int t0, int64_t n,
                                                        int k, int qs, uint64_t* __restrict__ seed_keys,
                                                        unsigned long long* __restrict__ kth_shared) {
    __shared__ __align__(16) float tile[kSeedWindow][tile_floats(DP)];
    __shared__ uint64_t wl[kWarps][96];  // per warp: the row's sorted k best (k <= 64), then up to 32 new keys
    const int T = t0 + static_cast<int>(blockIdx.x);
    for (int q = 0; q < qs; ++q) {
        const float* src = tiles + static_cast<int64_t>(spiral_tile(T, q, nt)) * tile_floats(DP);
        for (int i = threadIdx.x; i < tile_floats(DP); i += kThreads) tile[q][i] = src[i];
    }
    __syncthreads();
    const unsigned* idx = reinterpret_cast<const unsigned*>(tile[0] + tile_index_off(DP));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t* lst = wl[warp];
    const auto exact = [](uint64_t key) { return key; };
    for (int r = warp; r < kRT; r += kWarps) {
        const int64_t pos = static_cast<int64_t>(T) * kRT + r;
        const bool row_valid = idx[r] != kNoIndex;
        uint64_t ra2[DP];  // the row's coordinates, duplicated for the packed chains
#pragma unroll
        for (int f = 0; f < DP; ++f) ra2[f] = dup2(tile_coord<DP>(tile[0], r, f));
        // own tile: its 128 keys (the k best of them sorted below); lane l
        // takes the columns of pairs l and l + 32
        uint64_t v[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int p = h * 32 + lane;
            float d0, d1;
            pair_dist2<DP>(tile[0], p, ra2, d0, d1);
            const int c0 = 2 * p, c1 = 2 * p + 1;
            v[2 * h] = (row_valid && c0 != r && idx[c0] != kNoIndex) ? make_key(__float_as_uint(d0), idx[c0]) : kKeyMax;
            v[2 * h + 1] =
                (row_valid && c1 != r && idx[c1] != kNoIndex) ? make_key(__float_as_uint(d1), idx[c1]) : kKeyMax;
        }
        uint64_t kk = kKeyMax;
        uint64_t best = kKeyMax;  // k <= 32: the 32 best so far, sorted across the warp
        if (k <= 32) {
            // the first 32 keys sorted, the other three registers merged in
            // (those with a key below the current k-th key)
            uint64_t w[1] = {v[0]};
            warp_bitonic_sort<1>(w);
            best = w[0];
            kk = __shfl_sync(0xffffffffu, best, k - 1);
#pragma unroll
            for (int j = 1; j < 4; ++j) {
                if (!__any_sync(0xffffffffu, v[j] < kk)) continue;
                uint64_t x[1] = {v[j] < kk ? v[j] : kKeyMax};
                warp_bitonic_sort<1>(x);
                best = warp_merge_lowest32(best, x[0]);
                kk = __shfl_sync(0xffffffffu, best, k - 1);
            }
        } else {
            warp_bitonic_sort<4>(v);
            const int owner = (k - 1) & 31, oreg = (k - 1) >> 5;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint64_t t = __shfl_sync(0xffffffffu, v[j], owner);
                if (j == oreg) kk = t;
            }
        }
        if (row_valid && qs > 1 && k <= 32) {
            // neighbour tiles, k <= 32: the 32 best so far stay in one
            // register across the warp (sorted); keys below the current k-th
            // key gather in shared memory, 32 at most, and join by a bitonic
            // merge in registers
            int cnt = 0;
            const auto merge_pending = [&]() {
                uint64_t w[1] = {lane < cnt ? lst[lane] : kKeyMax};
                warp_bitonic_sort<1>(w);
                best = warp_merge_lowest32(best, w[0]);
                kk = __shfl_sync(0xffffffffu, best, k - 1);
                cnt = 0;
            };
            for (int q = 1; q < qs; ++q) {
                const unsigned* idq = reinterpret_cast<const unsigned*>(tile[q] + tile_index_off(DP));
                float dd[4];  // columns 2p and 2p + 1 of pairs p = l and l + 32
                pair_dist2<DP>(tile[q], lane, ra2, dd[0], dd[1]);
                pair_dist2<DP>(tile[q], lane + 32, ra2, dd[2], dd[3]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = 2 * ((j >> 1) * 32 + lane) + (j & 1);
                    const uint64_t key = idq[c] != kNoIndex ? make_key(__float_as_uint(dd[j]), idq[c]) : kKeyMax;
                    unsigned m = __ballot_sync(0xffffffffu, key < kk);
                    if (m && cnt + __popc(m) > 32) {
                        __syncwarp();
                        merge_pending();
                        __syncwarp();
                        m = __ballot_sync(0xffffffffu, key < kk);
                    }
                    if (m) {
                        if (key < kk) lst[cnt + __popc(m & ((1u << lane) - 1u))] = key;
                        cnt += __popc(m);
                    }
                }
            }
            __syncwarp();
            if (cnt > 0) merge_pending();
            if (lane < k) seed_keys[pos * k + lane] = best;
            __syncwarp();
        } else if (row_valid && qs > 1) {
            // neighbour tiles: append the keys below the current k-th key and
            // merge them into the sorted k best (at most 32 at a time)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int e = j * 32 + lane;
                if (e < k) lst[e] = v[j];
            }
            int cnt = k;
            for (int q = 1; q < qs; ++q) {
                const unsigned* idq = reinterpret_cast<const unsigned*>(tile[q] + tile_index_off(DP));
                float dd[4];  // columns 2p and 2p + 1 of pairs p = l and l + 32
                pair_dist2<DP>(tile[q], lane, ra2, dd[0], dd[1]);
                pair_dist2<DP>(tile[q], lane + 32, ra2, dd[2], dd[3]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = 2 * ((j >> 1) * 32 + lane) + (j & 1);
                    const uint64_t key = idq[c] != kNoIndex ? make_key(__float_as_uint(dd[j]), idq[c]) : kKeyMax;
                    unsigned m = __ballot_sync(0xffffffffu, key < kk);
                    if (m && cnt + __popc(m) > k + 32) {
                        __syncwarp();
                        cnt = merge_sorted_prefix<1>(lst, k, cnt, k, k - 1, exact, &kk);
                        m = __ballot_sync(0xffffffffu, key < kk);
                    }
                    if (m) {
                        __syncwarp();
                        if (key < kk) lst[cnt + __popc(m & ((1u << lane) - 1u))] = key;
                        cnt += __popc(m);
                    }
                }
            }
            __syncwarp();
            if (cnt > k) cnt = merge_sorted_prefix<1>(lst, k, cnt, k, k - 1, exact, &kk);
            for (int e = lane; e < k; e += 32) seed_keys[pos * k + e] = lst[e];
            __syncwarp();
        } else if (k <= 32) {
            if (lane < k) seed_keys[pos * k + lane] = best;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int e = j * 32 + lane;
                if (e < k) seed_keys[pos * k + e] = v[j];
            }
        }
        if (lane == 0) kth_shared[pos] = row_valid ? kk : kKeyMax;
    }
}

// ---------------------------------------------------------------- merge

// Per row (one warp): the k smallest of the seed list and the S split lists,
// written in the reference's slot order. The lists are sorted, disjoint
// (different columns) and kKeyMax padded, so an element's final rank is its
// position in its own list plus, for every other list, the count of keys
// below it (a binary search in shared memory); no sort is needed. In the
// result the ties with the k-th key already sit at the end in index order;
// the keys below it are placed by counting smaller indices among them.
constexpr int kMergeWarps = 8;

__global__ void __launch_bounds__(32 * kMergeWarps)
merge_kernel(const uint64_t* __restrict__ seed_keys, const uint64_t* __restrict__ partial,
             const unsigned* __restrict__ perm, int64_t n, int nt, int64_t pos0, int64_t pos1, int nsplit, int k,
             int32_t* __restrict__ nbr_idx, float* __restrict__ nbr_d2, float* __restrict__ kdist2) {
    extern __shared__ uint64_t msh[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nl = nsplit + 1, total = nl * k;
    uint64_t* lists = msh + static_cast<int64_t>(warp) * (total + k);
    uint64_t* out = lists + total;
    const int64_t pos = pos0 + static_cast<int64_t>(blockIdx.x) * kMergeWarps + warp;
    if (pos >= pos1) return;
    // element e of the concatenated lists is key t of list l, e = l k + t
    // (found by subtraction: e < (S + 1) k, and division by a run-time k is slow)
    const auto split_index = [k](int e, int& t) {
        int l = 0;
        t = e;
        while (t >= k) {
            t -= k;
            ++l;
        }
        return l;
    };
    for (int e = lane; e < total; e += 32) {
        int t;
        const int l = split_index(e, t);
        lists[e] = (l == 0) ? seed_keys[pos * k + t]
                            : partial[(static_cast<int64_t>(l - 1) * nt * kRT + pos) * k + t];
    }
    for (int e = lane; e < k; e += 32) out[e] = kKeyMax;
    __syncwarp();
    for (int e = lane; e < total; e += 32) {
        const uint64_t x = lists[e];
        if (x == kKeyMax) continue;
        int rank;
        const int l = split_index(e, rank);
        for (int o = 0; o < nl && rank < k; ++o) {
            if (o == l) continue;
            const uint64_t* lo = lists + o * k;
            int a = 0, b = k;  // count of keys < x in list o
            while (a < b) {
                const int mid = (a + b) >> 1;
                if (lo[mid] < x) a = mid + 1;
                else b = mid;
            }
            rank += a;
        }
        if (rank < k) out[rank] = x;
    }
    __syncwarp();
    const uint64_t kth = out[k - 1];
    const uint32_t kbits = key_bits(kth);
    // keys strictly below the k-th occupy out[0, below); the ties follow
    int below = 0;
    for (int e = lane; e < k; e += 32) below += key_bits(out[e]) < kbits ? 1 : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) below += __shfl_xor_sync(0xffffffffu, below, o);
    const unsigned self = perm[pos];
    for (int e = lane; e < k; e += 32) {
        const uint64_t y = out[e];
        int slot = e;  // ties: already in index order after the keys below
        if (e < below) {
            const uint32_t yi = key_index(y);
            slot = 0;
            for (int q = 0; q < below; ++q) slot += key_index(out[q]) < yi ? 1 : 0;
        }
        nbr_idx[static_cast<int64_t>(slot) * n + self] = static_cast<int32_t>(key_index(y) & 0x7FFFFFFFu);
        nbr_d2[static_cast<int64_t>(slot) * n + self] = __uint_as_float(key_bits(y));
    }
    if (lane == 0) kdist2[self] = __uint_as_float(kbits);
}

// The whole sort of a small input in one launch: a cluster of eight CTAs, each
// with a contiguous eighth of the pairs, runs all passes with its digit counts
// in (distributed) shared memory; the pairs go through global memory (L2)
// between passes, ordered by the cluster barriers: bound by their latency and
// the eight SMs' issue rate. Three launches per pass spent most of their time
// starting and in the gaps; the order (keys, sort, refinement) of 8,000 points
// at d=200 takes 45 us for 96, of 20,000 at d=8 87 for 125 (31 of it this
// kernel), of 30,000 at d=100 68 for 105, of 50,000 at d=3 112 for 121 (66 of
// it this kernel). At 65,536 pairs the two meet: that is the limit.
constexpr int kCsThreads = 1024;
constexpr int kCsWarps = kCsThreads / 32;
constexpr int kCsCtas = 8;
constexpr int kCsItems = 8;  // most pairs per thread
constexpr int64_t kCsMax = static_cast<int64_t>(kCsCtas) * kCsThreads * kCsItems;

struct ClusterSortSmem {
    unsigned wcount[kCsWarps][256];
    unsigned totals[2][256];  // this CTA's digit counts, by pass parity (other CTAs read them)
    unsigned first[256];      // first place of the CTA's pairs of each digit
    int warp_sums[8];
};

template <int IPT>
__global__ void __launch_bounds__(kCsThreads)
cluster_sort_kernel(unsigned* __restrict__ keys, unsigned* __restrict__ vals, unsigned* __restrict__ keys_tmp,
                    unsigned* __restrict__ vals_tmp, int n, int key_bits) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char cs_raw[];
    ClusterSortSmem& sh = *reinterpret_cast<ClusterSortSmem*>(cs_raw);
    cg::cluster_group cl = cg::this_cluster();
    const int rank = static_cast<int>(cl.block_rank());
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    // warp w of CTA r owns pairs [(r kCsWarps + w) 32 IPT, ...), 32 at a time
    const int base = (rank * kCsWarps + warp) * 32 * IPT + lane;
    unsigned *kin = keys, *vin = vals, *kout = keys_tmp, *vout = vals_tmp;
    for (int shift = 0, pass = 0; shift < key_bits; shift += 8, ++pass) {
        for (int i = tid; i < kCsWarps * 256; i += kCsThreads) (&sh.wcount[0][0])[i] = 0;
        unsigned key[IPT], val[IPT], place[IPT];
#pragma unroll
        for (int it = 0; it < IPT; ++it) {
            const int i = base + it * 32;
            key[it] = i < n ? __ldcg(kin + i) : 0u;
            val[it] = i < n ? __ldcg(vin + i) : 0u;
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < IPT; ++it) {
            const bool valid = base + it * 32 < n;
            const unsigned dg = valid ? (key[it] >> shift) & 0xFFu : 256u;
            const unsigned peers = __match_any_sync(0xffffffffu, dg);
            const unsigned r = __popc(peers & lt);
            const unsigned prior = valid ? sh.wcount[warp][dg] : 0u;
            place[it] = prior + r;
            __syncwarp();
            if (valid && r == 0) sh.wcount[warp][dg] = prior + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        if (tid < 256) {  // exclusive prefix over the warps
            unsigned run = 0;
#pragma unroll 8
            for (int w = 0; w < kCsWarps; ++w) {
                const unsigned t = sh.wcount[w][tid];
                sh.wcount[w][tid] = run;
                run += t;
            }
            sh.totals[pass & 1][tid] = run;
        }
        cl.sync();
        // places of the lower digits' pairs and of the same digit's in lower CTAs
        unsigned all = 0, lower = 0;
        if (tid < 256) {
            for (int c = 0; c < kCsCtas; ++c) {
                const unsigned t = *cl.map_shared_rank(&sh.totals[pass & 1][tid], c);
                all += t;
                lower += c < rank ? t : 0u;
            }
            const int incl = warp_inclusive_scan(static_cast<int>(all));
            if (lane == 31) sh.warp_sums[warp] = incl;
            sh.first[tid] = static_cast<unsigned>(incl) - all + lower;
        }
        __syncthreads();
        if (tid < 256) {
            unsigned before = 0;
            for (int w = 0; w < warp; ++w) before += static_cast<unsigned>(sh.warp_sums[w]);
            sh.first[tid] += before;
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < IPT; ++it) {
            if (base + it * 32 < n) {
                const unsigned dg = (key[it] >> shift) & 0xFFu;
                const unsigned pos = sh.first[dg] + sh.wcount[warp][dg] + place[it];
                __stcg(kout + pos, key[it]);
                __stcg(vout + pos, val[it]);
            }
        }
        cl.sync();  // the next pass reads what every CTA wrote
        unsigned* t = kin;
        kin = kout;
        kout = t;
        t = vin;
        vin = vout;
        vout = t;
    }
}

template <int IPT>
void launch_cluster_sort(unsigned* keys, unsigned* vals, unsigned* keys_tmp, unsigned* vals_tmp, int n, int key_bits,
                         cudaStream_t s) {
    set_max_dynamic_smem(reinterpret_cast<const void*>(cluster_sort_kernel<IPT>), sizeof(ClusterSortSmem));
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    cfg.gridDim = dim3(kCsCtas);
    cfg.blockDim = dim3(kCsThreads);
    cfg.dynamicSmemBytes = sizeof(ClusterSortSmem);
    cfg.stream = s;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kCsCtas;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    CG_CUDA(cudaLaunchKernelEx(&cfg, cluster_sort_kernel<IPT>, keys, vals, keys_tmp, vals_tmp, n, key_bits));
    count_launch();
}

int grid_for(int64_t items, int block) {
    int64_t g = ceil_div(items, block);
    if (g > 152 * 8) g = 152 * 8;
    return static_cast<int>(g < 1 ? 1 : g);
}

// Whether isolated rows leave the small-d sweep for a pass of their own: from
// 16,384 points on; CULOF_ISO_ROWS=0 or 1 forces the choice (the results are
// the same either way).
constexpr int64_t kIsoMinPoints = 16384;
bool iso_rows_enabled(int64_t n) {
    if (const char* env = std::getenv("CULOF_ISO_ROWS")) return env[0] != '0';
    return n >= kIsoMinPoints;
}

}  // namespace

int choose_splits(int nt, int sms) {
    // enough CTAs (2 per SM resident) for ~16 waves, at most 7 splits
    const int want = (32 * sms + nt - 1) / nt;
    int s = want < 1 ? 1 : want;
    if (s > 7) s = 7;
    if (s > nt - 1) s = nt - 1 > 0 ? nt - 1 : 1;
    return s;
}

void launch_merge(const uint64_t* seed_keys, const uint64_t* partial, const unsigned* perm, int64_t n, int nt,
                  int64_t pos0, int64_t pos1, int nsplit, int k, int32_t* idx, float* d2, float* kd, cudaStream_t s) {
    const size_t smem = sizeof(uint64_t) * kMergeWarps * static_cast<size_t>((nsplit + 1) * k + k);
    if (smem > 48 * 1024)
        CG_CUDA(cudaFuncSetAttribute(merge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    if (pos1 <= pos0) return;
    merge_kernel<<<static_cast<unsigned>(ceil_div(pos1 - pos0, kMergeWarps)), 32 * kMergeWarps, smem, s>>>(
        seed_keys, partial, perm, n, nt, pos0, pos1, nsplit, k, idx, d2, kd);
    CG_LAUNCH_CHECK();
}

size_t sort_pairs_counts(int64_t n) {
    return static_cast<size_t>(256) * (static_cast<size_t>(ceil_div(n, kSortTile)) + 1);  // the rows, then their totals
}

unsigned* sort_pairs_stable(unsigned* keys, unsigned* vals, unsigned* keys_tmp, unsigned* vals_tmp, int64_t n,
                            int key_bits, unsigned* counts, cudaStream_t s, unsigned** vals_out) {
    const int nblocks = static_cast<int>(ceil_div(n, kSortTile));
    unsigned* totals = counts + static_cast<int64_t>(256) * nblocks;
    if (n <= kCsMax) {
        const int ni = static_cast<int>(n), per = static_cast<int>(ceil_div(n, kCsCtas * kCsThreads));
        if (per <= 1) launch_cluster_sort<1>(keys, vals, keys_tmp, vals_tmp, ni, key_bits, s);
        else if (per <= 2) launch_cluster_sort<2>(keys, vals, keys_tmp, vals_tmp, ni, key_bits, s);
        else if (per <= 4) launch_cluster_sort<4>(keys, vals, keys_tmp, vals_tmp, ni, key_bits, s);
        else launch_cluster_sort<kCsItems>(keys, vals, keys_tmp, vals_tmp, ni, key_bits, s);
        const bool back = (key_bits + 7) / 8 % 2 == 0;  // an even number of passes: in the first buffers
        *vals_out = back ? vals : vals_tmp;
        return back ? keys : keys_tmp;
    }
    unsigned *kin = keys, *vin = vals, *kout = keys_tmp, *vout = vals_tmp;
    for (int shift = 0; shift < key_bits; shift += 8) {
        sort_upsweep_kernel<<<nblocks, kSortThreads, 0, s>>>(kin, n, shift, counts, nblocks);
        CG_LAUNCH_CHECK();
        sort_rowscan_kernel<<<256, kRowScanThreads, 0, s>>>(counts, nblocks, totals);
        CG_LAUNCH_CHECK();
        sort_downsweep_kernel<<<nblocks, kSortThreads, 0, s>>>(kin, vin, kout, vout, n, shift, counts, totals, nblocks);
        CG_LAUNCH_CHECK();
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    *vals_out = vin;
    return kin;
}

bool fast_path_supported(int64_t n, int d, int k) {
    return d >= 1 && d <= kMaxWideD && k >= 1 && k <= kMaxK && n >= 2 && static_cast<int64_t>(k) < n &&
           n <= (static_cast<int64_t>(1) << 30);
}

bool tensor_supported(int64_t n, int d, int k) {
    return d >= 1 && d <= kMaxTensorD && fast_path_supported(n, 1, k);
}

// Host orchestration of the fast path.
void Engine::knn_fast(const float* xc, const float* norms, int64_t n, int d, int k, bool tensor, int32_t* nbr_idx,
                      float* nbr_d2, float* kdist2, int shard, int num_shards, int32_t* shard_rows) {
    cudaStream_t s = stream_;
    const bool wide = !tensor && d > kMaxDP;
    // the tensor sweep for d <= 8 starts from the small-d seed window and
    // visits only the column tiles of the small-d prune lists
    const bool small_tc = tensor && d <= kMaxDP;
    const bool small_fp32 = !wide && !tensor;  // small.cu
    const int dp = padded_dims(d);
    const int nt = static_cast<int>(ceil_div(n, kCT));
    const int64_t padded = static_cast<int64_t>(nt) * kCT;
    // the rows of this call: row tiles [t0, t0 + mt) of the spatial order
    // (all of them unless the call is one shard of a row-sharded run)
    const int t0 = static_cast<int>(static_cast<int64_t>(nt) * shard / num_shards);
    const int mt = static_cast<int>(static_cast<int64_t>(nt) * (shard + 1) / num_shards) - t0;
    int sms = 152;
    CG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device_));
    // The tensor sweep: every split of a row tile scans for its own bounds and
    // keeps its own lists, so it takes the split that needs the least rounds of
    // CTAs times their length. Up to 128 features two CTAs share an SM and a
    // split costs about 64 tile visits (n = 30,011, d = 100, k = 30: 1.42 ms per
    // fit_predict with one split, 1.50 with two, 1.53 with three, when a pass
    // took twice what it does now; n = 50,000, d = 32, k = 20, forward and
    // backward: 4.18, 4.06, 4.08 ms). Above, one CTA takes an SM and 30 fit
    // (scores, factor model, d = 200, k = 20, splits 1 to 4: n = 5,000 309, 259,
    // 245, 283 us; 8,000 381, 305, 357, 332; 12,000 472, 505, 436, 479; 20,000
    // 993, 915, 889, 888; 30,000 1275, 1528, 1404, 1506). Past k = 56 there one
    // split: a list of a share starts from a looser bound, and clusters fill it
    // (d = 200, k = 64, n = 4,100, one split against the three of that rule: 1,227
    // for 1,500 us, factor model 688 for 601; n = 8,000 2,726 for 2,948 and 822
    // for 788; the general path takes 767 and 2,412).
    int nsplit = 1;
    if (nt > 1) {
        if (wide) {
            nsplit = choose_splits(mt, sms);
            if (nsplit > nt - 1) nsplit = nt - 1;
        } else if (tensor) {
            const bool one = d > kMaxWideD;            // CTA per SM
            const int64_t slots = one ? sms : 2 * sms;  // CTAs at a time
            // (k > 56 leaves a list little room for the filter's margin: most
            // rows rescore candidates exactly, and every split pays that anew)
            const int64_t own = one ? 30 : k > 56 ? 256 : 64;
            int64_t best = -1;
            // (past two rounds the list entries that every split repeats cost
            // more than the last round's idle SMs: n = 200,000, d = 128, k = 50,
            // 24.2 ms with one split, 31.0 with two)
            const int most = mt >= 2 * slots || (one && k > 56) ? 1 : tc_max_splits();
            for (int v = 1; v <= most && v < nt; ++v) {
                const int64_t cost = ceil_div(static_cast<int64_t>(mt) * v, slots) * (nt / v + own);
                if (best < 0 || cost < best) {
                    best = cost;
                    nsplit = v;
                }
            }
        }
    }
    if (const char* env = std::getenv("CULOF_SPLITS")) {  // tuning override (1..nt-1)
        const long v = std::atol(env);
        if (v >= 1 && nt > 1) nsplit = static_cast<int>(v < nt - 1 ? v : nt - 1);
        if (tensor && nsplit > tc_max_splits()) nsplit = tc_max_splits();
    }
    // the small-d seed of the tensor path covers the first qs spiral positions
    // of every row tile, the sweep the rest (the other seeds cover tile T alone)
    const int qs = small_tc ? (nt < kSeedWindow ? nt : kSeedWindow) : tensor ? 0 : 1;
    const bool sweep = nt > qs;
    if (sweep && nsplit > nt - qs) nsplit = nt - qs;  // no split without a column tile

    // 1. Morton keys of the centred coordinates, then a stable radix sort.
    const unsigned* mm = range_words();  // from the centring
    unsigned* keys = morton_.as<unsigned>(2 * static_cast<size_t>(n));
    unsigned* vals = perm_.as<unsigned>(2 * static_cast<size_t>(n));
    TcStart* start = tensor ? static_cast<TcStart*>(lost_.get(sizeof(TcStart) + sizeof(int32_t) * static_cast<size_t>(mt) * kRT))
                            : nullptr;
    morton_kernel<<<grid_for(n, 256), 256, 0, s>>>(xc, n, d, mm, keys, vals, max_norm_word(), start);
    CG_LAUNCH_CHECK();
    unsigned* vin = nullptr;  // after 4 passes: back in the first half
    sort_pairs_stable(keys, vals, keys + n, vals + n, n, 32, sort_tmp_.as<unsigned>(sort_pairs_counts(n)), s, &vin);
    const unsigned* perm = vin;
    if (small_fp32 || small_tc) small_refine_order(xc, n, d, vin, s);
    const int64_t pos0 = static_cast<int64_t>(t0) * kCT;
    const int64_t pos1 = std::min<int64_t>(n, static_cast<int64_t>(t0 + mt) * kCT);
    if (shard_rows && pos1 > pos0)  // original indices of the shard's rows
        CG_CUDA(cudaMemcpyAsync(shard_rows, perm + pos0, sizeof(unsigned) * (pos1 - pos0), cudaMemcpyDeviceToDevice,
                                s));

    // 2. column tiles
    float* tiles = nullptr;
    TcBuffers tcb{};
    float* boxes = nullptr;
    if (tensor) tcb = tc_prepare(cols_.get(tc_buffer_bytes(padded, d)), xc, norms, n, d, perm, nt, &start->scale, s);
    if (wide) {
        tiles = cols_.as<float>(wide_tiles_floats(d, nt));
        wide_build_tiles(xc, norms, n, d, perm, nt, tiles, s);
    } else if (small_fp32 || small_tc) {
        // tiles, then the quarter records (32 bytes each)
        tiles = tiles_.as<float>(small_tiles_floats(dp, nt) + static_cast<size_t>(nt) * kQuarters * 8);
        boxes = boxes_.as<float>(static_cast<size_t>(nt) * 2 * dp);
        void* qbox = tiles + small_tiles_floats(dp, nt);
        small_build_tiles(xc, n, d, perm, nt, tiles, boxes, qbox, s);
        if (small_fp32) {
            mark(2);
            mark(3);
            unsigned long long* ev = evaluated_word();
            // pairs past the window (tile T and its four Morton neighbours)
            const int window = nt < kSeedWindow ? nt : kSeedWindow;
            stat_total_pairs_ = static_cast<double>(mt) * (nt - window) * kRT * kCT;
            // CULOF_PRUNE_LISTS=0 lists the column tiles in short segments, as
            // inputs of many segments do (the same results)
            const char* env = std::getenv("CULOF_PRUNE_LISTS");
            const bool defer = small_defers(iso_rows_enabled(n), nt, mt);
            small_knn(tiles, boxes, qbox, perm, n, d, nt, t0, mt, k, sms, defer, env && env[0] == '0' ? 8 : kSegTiles,
                      iso_.get(small_iso_bytes(mt, k, defer)), iso_count_word(), nbr_idx, nbr_d2, kdist2, status_ptr(), ev, s);
            mark(4);
            return;
        }
    }

    // 3. seed lists and the shared k-th keys (the tensor sweep past 8 features
    // has no seed)
    uint64_t* seed_keys = nullptr;
    unsigned long long* kth_shared = nullptr;
    uint64_t* partial = nullptr;
    if (wide || small_tc) {
        seed_keys = rows_.as<uint64_t>(static_cast<size_t>(padded) * (k + 1) +
                                       (wide ? static_cast<size_t>(nsplit) * padded * k : 0));
        kth_shared = reinterpret_cast<unsigned long long*>(seed_keys + padded * k);
        partial = reinterpret_cast<uint64_t*>(kth_shared + padded);
    }
    int* status = status_ptr();
    const unsigned* maxn = max_norm_word();
    mark(2);
    if (tensor && !small_tc) {  // no seed: the sweep covers every tile
    } else if (wide) wide_seed(tiles, nt, t0, mt, d, k, seed_keys, kth_shared, s);
    else switch (dp) {
        case 2: seed_kernel<2><<<mt, kThreads, 0, s>>>(tiles, nt, t0, n, k, qs, seed_keys, kth_shared); break;
        case 4: seed_kernel<4><<<mt, kThreads, 0, s>>>(tiles, nt, t0, n, k, qs, seed_keys, kth_shared); break;
        case 6: seed_kernel<6><<<mt, kThreads, 0, s>>>(tiles, nt, t0, n, k, qs, seed_keys, kth_shared); break;
        default: seed_kernel<8><<<mt, kThreads, 0, s>>>(tiles, nt, t0, n, k, qs, seed_keys, kth_shared); break;
    }
    if (small_tc) CG_LAUNCH_CHECK();
    mark(3);

    // per row tile: the column tiles the seed's k-th distances leave
    uint2* plist = nullptr;
    int* pcount = nullptr;
    constexpr int kMaxListTiles = 16384;  // lists take nt^2 x 8 bytes: up to 2 GiB
    // CULOF_PRUNE_LISTS=0 walks the whole spiral as inputs above the list
    // limit do (the same results; it puts that path within reach of tests)
    const char* lists_env = std::getenv("CULOF_PRUNE_LISTS");
    const bool lists_on = !(lists_env && lists_env[0] == '0');
    if (small_tc && sweep && nt <= kMaxListTiles && lists_on) {
        plist = plist_.as<uint2>(static_cast<size_t>(nt) * nt);
        pcount = pcount_.as<int>(nt);
        switch (dp) {
            case 2: prune_list_kernel<2><<<mt, 256, 0, s>>>(boxes, nt, t0, qs, kth_shared, plist, pcount); break;
            case 4: prune_list_kernel<4><<<mt, 256, 0, s>>>(boxes, nt, t0, qs, kth_shared, plist, pcount); break;
            case 6: prune_list_kernel<6><<<mt, 256, 0, s>>>(boxes, nt, t0, qs, kth_shared, plist, pcount); break;
            default: prune_list_kernel<8><<<mt, 256, 0, s>>>(boxes, nt, t0, qs, kth_shared, plist, pcount); break;
        }
        CG_LAUNCH_CHECK();
    }
    // 4. sweep over the other tiles, split S ways
    if (sweep && mt > 0 && tensor) {
        uint64_t* lists = static_cast<uint64_t*>(tc_lists_.get(tc_list_bytes(mt, nsplit)));
        int32_t* lost = reinterpret_cast<int32_t*>(start + 1);
        tc_sweep(tcb, n, nt, t0, mt, nsplit, d, k, maxn, kth_shared, seed_keys, lists, status, nbr_idx, nbr_d2, kdist2, s,
                 qs, lost, lost_count_word(), plist, pcount);
        lost_rows(xc, n, d, k, lost, lost_count_word(), lost_keys_.get(lost_rows_bytes(n, pos1 - pos0, k, sms)),
                  start->arrived, sms, nbr_idx, nbr_d2, kdist2, s);
        mark(4);
        return;
    } else if (nt > 1 && mt > 0 && wide) {
        wide_sweep(tiles, nt, t0, mt, nsplit, d, k, maxn, kth_shared, partial, s);
    }
    const int ns = sweep ? nsplit : 0;
    mark(4);

    // 5. merge into the reference slot order
    launch_merge(seed_keys, partial, perm, n, nt, pos0, pos1, ns, k, nbr_idx, nbr_d2, kdist2, s);
}

}  // namespace culof_gb300
