// The small-d exact k-NN (d <= 8): one kernel that finds every row's k best
// over all column tiles, pruning per row, and a pass of its own for isolated
// rows.
//
// A CTA owns 64 or 128 consecutive rows of the spatial order (8 warps of 8 or
// 16 rows) and streams column tiles of 128 points into shared memory (TMA bulk
// copies, the last warp done with a stage refills it):
//   1. the window: its own tile T and the neighbours T+-1, T+-2, which start
//      every row's list and k-th distance;
//   2. rows whose k-th distance stays far above the CTA's median (isolated
//      points) are handed to the pass of their own: they would make the CTA
//      visit tiles that none of its other rows needs;
//   3. the other tiles that can hold a candidate under the k-th distances so
//      far (bounding boxes), nearest centres first, so that the k-th
//      distances shrink early.
// Per tile and warp, one test per lane compares the boxes of the tile's two
// 64-column halves with every row's own k-th distance (16 rows x 2 halves).
// Only the (row, half) pairs that pass are evaluated, lane = column pair, with the exact direct-difference distance; keys within the row's
// k-th distance are inserted into the row's sorted list (32 or 64 keys, one or
// two registers per lane while it is worked on, in shared memory between).
//
// What bounds it, and why per row: at n = 200,000, d = 8, k = 20 (five
// clusters and 1% outliers) 20% of the (128 rows, tile) blocks hold a candidate
// for some row of the block, but only 4.7% of the (row, half) pairs hold one
// for their row (145 halves per row). Evaluating whole blocks with packed FMAs,
// as an earlier form did, took 5.94 ms (and 0.52 ms for its seeds, 0.16 ms to
// merge its lists); this kernel takes 3.64 ms with lists and output included
// (ncu, same input). It is bound by issue: 2.6e9 warp instructions, 62% of the
// issue slots while an SM is busy, about 40% of them distances, 20% box tests,
// the rest list insertions and the window.
#include <cuda_bf16.h>

#include <algorithm>

#include "engine.cuh"
#include "row_list.cuh"
#include "small.cuh"
#include "sweep_rows.cuh"
#include "tile_order.cuh"
#include "warp_sort.cuh"

namespace culof_gb300 {

namespace {

using namespace small;

constexpr float kSparseRatio = 4.0f;  // a tile is sparse when its squared diagonal exceeds 4x the median tile's
// Sparse tiles leave whole up to 4 row tiles per SM; with more only those a
// thousand times as wide as the median tile (heavy tails: 1-d Cauchy data, n =
// 100,000 and 200,000, 0.77 and 0.80 ms for 1.21 and 1.58; with kSparseRatio at
// any size, clusters with uniform outliers, d = 1, n = 200,000, 0.93 for 0.78).
constexpr int kSparseWaves = 4;
constexpr float kVerySparseRatio = 1e6f;

// ---------------------------------------------------------------- tiles

// One CTA of 128 threads per tile, one thread per column: coordinates,
// indices, half boxes, the quarter boxes of the isolated rows' pass (bf16
// rounded outward: 16 values per quarter, lower bounds then upper bounds) and
// the tile's box.
template <int DP>
__global__ void __launch_bounds__(kCT) small_tile_kernel(const float* __restrict__ xc, int64_t n, int d,
                                                         const unsigned* __restrict__ perm, float* __restrict__ tiles,
                                                         float* __restrict__ boxes, __nv_bfloat16* __restrict__ qbox) {
    __shared__ float wb[kQuarters][2][DP];
    const int64_t t = blockIdx.x;
    const int c = threadIdx.x, lane = c & 31, q = c >> 5;
    float* tile = tiles + t * tile_floats(DP);
    const int64_t p = t * kCT + c;
    const bool valid = p < n;
    const unsigned orig = valid ? perm[p] : kNoIndex;
    float mine = 0.0f;  // lane f: lower bound of dimension f of this quarter; lane 8 + f: upper bound
#pragma unroll
    for (int f = 0; f < DP; ++f) {
        const float v = (valid && f < d) ? xc[static_cast<int64_t>(orig) * d + f] : 0.0f;
        tile[f * kCT + c] = (!valid && f == 0) ? __int_as_float(0x7fc00000) : v;
        float lo = valid ? v : inf_f(), hi = valid ? v : -inf_f();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(kFullMask, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(kFullMask, hi, o));
        }
        if (lane == f) mine = lo;
        if (lane == 8 + f) mine = hi;
        if (lane == 0) {
            wb[q][0][f] = lo;
            wb[q][1][f] = hi;
        }
    }
    reinterpret_cast<unsigned*>(tile)[tile_index_off(DP) + c] = orig;
    if (lane < 16)
        qbox[16 * (t * kQuarters + q) + lane] = lane < 8 ? __float2bfloat16_rd(mine) : __float2bfloat16_ru(mine);
    __syncthreads();
    if (c < kHalves * DP) {
        const int h = c / DP, f = c % DP;
        tile[tile_box_off(DP) + (h * DP + f) * 2] = fminf(wb[2 * h][0][f], wb[2 * h + 1][0][f]);
        tile[tile_box_off(DP) + (h * DP + f) * 2 + 1] = -fmaxf(wb[2 * h][1][f], wb[2 * h + 1][1][f]);
    }
    if (c < DP) {
        boxes[t * 2 * DP + c] = fminf(fminf(wb[0][0][c], wb[1][0][c]), fminf(wb[2][0][c], wb[3][0][c]));
        boxes[t * 2 * DP + DP + c] = fmaxf(fmaxf(wb[0][1][c], wb[1][1][c]), fmaxf(wb[2][1][c], wb[3][1][c]));
    }
}

// ---------------------------------------------------------------- spatial order

// Refines the Morton order: every chunk of 1024 sorted points becomes a
// balanced k-d order (halved along the dimension of largest variance down to
// 16 points), which makes tiles, halves and the 16-row groups more compact:
// the sweep evaluates 145 instead of 192 halves per row (n = 200,000, d = 8,
// k = 20; larger chunks gain little more). One CTA per chunk, one thread per
// point; a point's sort key is its coordinate's order-preserving bits with
// the low 10 replaced by its place in the chunk (the order is a heuristic, no
// result depends on it).
// Bound by the instructions and barriers of the sorts. Chunks of 512 take half
// the time (18 us for 34 at n = 20,000, d = 8) and cost the sweep more (277 us
// for 253; 3,759 for 3,599 at n = 200,000). The V sums of a level by V
// reductions of their own took 40 and 66 us, together 34 and 59.
constexpr int kChunk = 1024;
template <int DP>
__global__ void __launch_bounds__(kChunk) refine_order_kernel(const float* __restrict__ xc, int64_t n, int d,
                                                              unsigned* __restrict__ perm) {
    constexpr int V = DP <= 2 ? 4 : DP <= 4 ? 8 : 16;  // sums and sums of squares, padded
    __shared__ float xs[DP][kChunk];
    __shared__ unsigned key_s[kChunk];
    __shared__ float stat[kChunk / 32][V];
    __shared__ float cnt[kChunk / 32];
    __shared__ unsigned orig[kChunk];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t pos = static_cast<int64_t>(blockIdx.x) * kChunk + tid;
    const bool valid = pos < n;
    const unsigned o = valid ? perm[pos] : 0u;
    orig[tid] = o;
    for (int f = 0; f < d; ++f) xs[f][tid] = valid ? xc[static_cast<int64_t>(o) * d + f] : 0.0f;
    __syncthreads();
    // slot: which of the chunk's points is at this place; places >= m hold none
    const int m = static_cast<int>(n - static_cast<int64_t>(blockIdx.x) * kChunk < kChunk
                                       ? n - static_cast<int64_t>(blockIdx.x) * kChunk
                                       : kChunk);
    unsigned slot = tid;
    for (int size = kChunk; size >= 32; size >>= 1) {
        // the segment's dimension of largest variance
        const bool in = static_cast<int>(slot) < m;
        float v[V];
#pragma unroll
        for (int f = 0; f < V / 2; ++f) {
            const float x = in && f < d ? xs[f < DP ? f : 0][slot] : 0.0f;
            v[2 * f] = x;
            v[2 * f + 1] = x * x;
        }
        // the warp's V sums, halving the number of values with each exchange:
        // sum lane / (32 / V) ends up in every lane
#pragma unroll
        for (int h = V / 2, st = 16; h > 0; h >>= 1, st >>= 1) {
            const bool up = (lane & st) != 0;
#pragma unroll
            for (int j = 0; j < h; ++j) {
                const float give = up ? v[j] : v[j + h], keep = up ? v[j + h] : v[j];
                v[j] = keep + __shfl_xor_sync(kFullMask, give, st);
            }
        }
#pragma unroll
        for (int st = 16 / V; st > 0; st >>= 1) v[0] += __shfl_xor_sync(kFullMask, v[0], st);
        if (lane % (32 / V) == 0) stat[warp][lane / (32 / V)] = v[0];
        const unsigned here = __ballot_sync(kFullMask, in);
        if (lane == 0) cnt[warp] = static_cast<float>(__popc(here));
        __syncthreads();
        const int w0 = tid / size * (size / 32), nw = size / 32;
        float var = -1.0f;
        if (lane < d) {  // (d <= DP <= V / 2)
            float s1 = 0.0f, s2 = 0.0f, c = 0.0f;
            for (int w = 0; w < nw; ++w) {
                s1 += stat[w0 + w][2 * lane];
                s2 += stat[w0 + w][2 * lane + 1];
                c += cnt[w0 + w];
            }
            var = c > 0.0f ? s2 - s1 * s1 / c : 0.0f;
        }
        int dim = lane;
#pragma unroll
        for (int st = 4; st > 0; st >>= 1) {
            const float ov = __shfl_xor_sync(kFullMask, var, st);
            const int od = __shfl_xor_sync(kFullMask, dim, st);
            if (ov > var || (ov == var && od < dim)) {
                var = ov;
                dim = od;
            }
        }
        dim = __shfl_sync(kFullMask, dim, 0);
        if (dim >= d) dim = 0;
        // bitonic sort of the segment by that coordinate
        const unsigned u = __float_as_uint(xs[dim][slot]);
        unsigned key = in ? ((u & 0x80000000u ? ~u : u | 0x80000000u) & ~1023u) | slot : 0xFFFFFC00u | slot;
        for (int sz = 2; sz <= size; sz <<= 1) {
            const bool asc = (tid & sz) == 0 || sz == size;
            for (int st = sz >> 1; st > 0; st >>= 1) {
                unsigned ok;
                if (st >= 32) {
                    __syncthreads();
                    key_s[tid] = key;
                    __syncthreads();
                    ok = key_s[tid ^ st];
                } else {
                    ok = __shfl_xor_sync(kFullMask, key, st);
                }
                const bool keep_min = ((tid & st) == 0) == asc;
                key = keep_min ? min(key, ok) : max(key, ok);
            }
        }
        slot = key & 1023u;
        __syncthreads();  // stat is rewritten by the next level
    }
    if (valid) perm[pos] = orig[slot];
}

// Squared diagonal of a tile's box.
__device__ __forceinline__ float box_extent(const float* __restrict__ b, int dp) {
    float e = 0.0f;
    for (int f = 0; f < dp; ++f) {
        const float w = b[dp + f] - b[f];
        e = fmaf(w, w, e);
    }
    return e;
}

// Launch order of the sweep's row tiles [t0, t0 + mt): widest boxes first
// (their rows lie in sparse regions, have far neighbours and take the
// longest), so that no long CTA starts last. The rank is counted against
// every other tile (mt^2 comparisons) in a total order (tile_order.cuh), so
// every place of order is written once, whatever the points hold.
__global__ void __launch_bounds__(256) tile_order_kernel(const float* __restrict__ boxes, int dp, int t0, int mt,
                                                         int* __restrict__ order) {
    // 32 tiles per block, eight threads per tile for an eighth of the others each
    __shared__ unsigned other[256];
    __shared__ int ranks[32];
    const auto extent = [&](int t) {
        return extent_key(__float_as_uint(box_extent(boxes + static_cast<int64_t>(t0 + t) * 2 * dp, dp)));
    };
    const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
    const int t = blockIdx.x * 32 + lane;
    const unsigned mine = t < mt ? extent(t) : 0u;
    if (part == 0) ranks[lane] = 0;
    int rank = 0;
    for (int c0 = 0; c0 < mt; c0 += 256) {
        __syncthreads();
        if (c0 + static_cast<int>(threadIdx.x) < mt) other[threadIdx.x] = extent(c0 + threadIdx.x);
        __syncthreads();
        const int c1 = min(32 * (part + 1), mt - c0);
        for (int i = 32 * part; i < c1; ++i) rank += starts_before(other[i], c0 + i, mine, t) ? 1 : 0;
    }
    __syncthreads();
    atomicAdd(&ranks[lane], rank);
    __syncthreads();
    if (part == 0 && t < mt) order[ranks[lane]] = t;
}

// ---------------------------------------------------------------- sweep

template <int DP, int KR, int G, int RW, int W>
__global__ void __launch_bounds__(32 * W, (KR == 1 ? 24 : 16) / W)
small_sweep_kernel(SweepRows P, int64_t row0, const int* __restrict__ order, int mt, int defer_rows) {
    using Smem = SmallSmem<DP, KR, RW, W>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Smem& sh = *reinterpret_cast<Smem*>(smem_raw);
    // first row position; the tiles' CTAs start in the given order
    constexpr int kPerTile = kCT / Smem::kRows;
    const int tile_i = static_cast<int>(blockIdx.x) / kPerTile;
    const int tile = order ? order[tile_i] : tile_i;
    if (static_cast<unsigned>(tile) >= static_cast<unsigned>(mt)) {  // never: order is a permutation
        if (threadIdx.x == 0) atomicExch(P.status, 2);
        return;
    }
    P.base = row0 + static_cast<int64_t>(tile) * kCT + static_cast<int>(blockIdx.x) % kPerTile * Smem::kRows;
    if (P.base >= P.n) return;
    if (defer_rows) {
        const int median = static_cast<int>(min(static_cast<unsigned>(order[mt / 2]), static_cast<unsigned>(mt - 1)));
        const float usual = box_extent(P.boxes + (row0 / kCT + median) * 2 * DP, DP);
        P.sparse = tile_i < mt / 32 && (defer_rows == 2 || usual > 0.0f) &&
                   box_extent(P.boxes + P.base / kCT * 2 * DP, DP) > (defer_rows == 2 ? kSparseRatio : kVerySparseRatio) * usual;
        sweep_rows<DP, KR, G, RW, W, true>(sh, P);
    } else {
        sweep_rows<DP, KR, G, RW, W, false>(sh, P);
    }
}

// ---------------------------------------------------------------- isolated rows

// Gaps are kept as the upper 16 bits of their float32 bit pattern
// (non-negative floats truncated: rounded down, so pruning stays
// conservative); kGapSkip marks a quarter the pass never visits.
constexpr uint16_t kGapSkip = 0xFFFFu;
constexpr int kIsoMaxTiles = 8192;  // 4 gaps of 2 bytes per column tile in shared memory
__device__ __forceinline__ uint16_t gap_bits_down(float g) { return static_cast<uint16_t>(__float_as_uint(g) >> 16); }
// the smallest 16-bit pattern not below distance b (+inf: 0x7F80)
__device__ __forceinline__ unsigned bound_bits_up(float b) { return (__float_as_uint(b) + 0xFFFFu) >> 16; }

// One CTA (kIsoWarps warps) per listed row: its k best over the column tiles
// outside the window, joined with its list from the sweep.
//  1. The rounded-down gap between the point and every quarter's box
//     (coalesced, into shared memory; the window's quarters are skipped).
//  2. Warp w owns quarter w of every tile (the quarters near the point are
//     spread over all warps) and visits its quarters in three rounds of
//     growing gap: gaps up to 1/16 of the row's current bound, then 1/4,
//     then the whole bound, so that the bound tightens on the nearest
//     quarters before the far ones are tested; quarters within the bound
//     are evaluated kIsoBatch at a time.
//  3. The warps share the bound (the smallest of the k-th distances held) in
//     shared memory and merge their lists at the end.
constexpr int kIsoWarps = 4;
constexpr int kIsoBatch = 4;
template <int DP, int KR>
__global__ void __launch_bounds__(32 * kIsoWarps, 6)
small_iso_kernel(const float* __restrict__ tiles, const __nv_bfloat16* __restrict__ qbox,
                 const unsigned* __restrict__ perm, int64_t n, int nt, int k, IsoRows iso,
                 int32_t* __restrict__ nbr_idx, float* __restrict__ nbr_d2, float* __restrict__ kdist2) {
    extern __shared__ __align__(16) uint16_t qgap_s[];  // 4 per tile
    __shared__ uint64_t fin[kIsoWarps][32 * KR];
    __shared__ unsigned bound_s;  // float bits of the row's smallest k-th distance so far
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int count = *iso.count;
    const int nb = (nt + 31) / 32;
    const int64_t nq = static_cast<int64_t>(nt) * kQuarters;
    const int wsize = nt < kWindow ? nt : kWindow;
    const int wlo = (wsize - 1) / 2, whi = wsize / 2;  // the window: offsets -wlo .. whi
    for (int h = blockIdx.x; h < count; h += gridDim.x) {
        const int64_t pos = iso.pos[h];
        const int T = static_cast<int>(pos / kCT), r = static_cast<int>(pos % kCT);
        const float* own = tiles + static_cast<int64_t>(T) * tile_floats(DP);
        float a[DP];
#pragma unroll
        for (int f = 0; f < DP; ++f) a[f] = tile_coord<DP>(own, r, f);
        uint64_t b[KR];  // warp 0 starts from the window's list
#pragma unroll
        for (int j = 0; j < KR; ++j) b[j] = iso.list[(static_cast<int64_t>(h) * KR + j) * 32 + lane];
        const float kd0 = list_kth<KR>(b, k);
        if (warp != 0) {
#pragma unroll
            for (int j = 0; j < KR; ++j) b[j] = kKeyMax;
        }
        if (threadIdx.x == 0) bound_s = __float_as_uint(kd0);
#pragma unroll 4
        for (int q = threadIdx.x; q < nq; q += 32 * kIsoWarps) {
            const int t = q / kQuarters;
            int off = t - T;  // offset from the row tile, in (-nt/2, nt/2]
            if (off > nt / 2) off -= nt;
            if (off <= -((nt + 1) / 2)) off += nt;
            const uint4 lo4 = reinterpret_cast<const uint4*>(qbox)[2 * q];
            const uint4 hi4 = reinterpret_cast<const uint4*>(qbox)[2 * q + 1];
            const unsigned lw[4] = {lo4.x, lo4.y, lo4.z, lo4.w}, hw[4] = {hi4.x, hi4.y, hi4.z, hi4.w};
            float g2 = 0.0f;
#pragma unroll
            for (int f = 0; f < DP; ++f) {  // bf16 to float is exact: the bits shifted up
                const float lo = __uint_as_float((f & 1 ? lw[f >> 1] >> 16 : lw[f >> 1] & 0xFFFFu) << 16);
                const float hi = __uint_as_float((f & 1 ? hw[f >> 1] >> 16 : hw[f >> 1] & 0xFFFFu) << 16);
                const float gap = fmaxf(0.0f, fmaxf(__fsub_rd(lo, a[f]), __fsub_rd(a[f], hi)));
                g2 = __fadd_rd(g2, __fmul_rd(gap, gap));
            }
            qgap_s[q] = (off >= -wlo && off <= whi) ? kGapSkip : gap_bits_down(__fmul_rd(g2, prune_shrink<DP>()));
        }
        __syncthreads();
        float bound = kd0;
        const auto shared_bound = [&]() {  // publish this warp's bound, take the CTA's
            unsigned sb = 0;
            if (lane == 0) sb = atomicMin(&bound_s, __float_as_uint(bound));
            sb = __shfl_sync(kFullMask, sb, 0);
            bound = fminf(bound, __uint_as_float(sb));
        };
        // up to kIsoBatch quarters against the point, all loads issued first;
        // lane l takes column l of each
        const auto eval = [&](int q0, int q1, int q2, int q3, int mq) {
            const int qs[kIsoBatch] = {q0, mq > 1 ? q1 : q0, mq > 2 ? q2 : q0, mq > 3 ? q3 : q0};
            float x[kIsoBatch][DP];
            unsigned ix[kIsoBatch];
#pragma unroll
            for (int i = 0; i < kIsoBatch; ++i) {
                const int qi = qs[i];
                const float* tl = tiles + static_cast<int64_t>(qi / kQuarters) * tile_floats(DP);
                const int c = (qi % kQuarters) * kQuarter + lane;
#pragma unroll
                for (int f = 0; f < DP; ++f) x[i][f] = tl[f * kCT + c];
                ix[i] = reinterpret_cast<const unsigned*>(tl)[tile_index_off(DP) + c];
            }
            float d2[kIsoBatch];
#pragma unroll
            for (int i = 0; i < kIsoBatch; ++i) {
                d2[i] = 0.0f;
#pragma unroll
                for (int f = 0; f < DP; ++f) {
                    const float t = __fsub_rn(a[f], x[i][f]);
                    d2[i] = __fmaf_rn(t, t, d2[i]);
                }
            }
#pragma unroll 1
            for (int i = 0; i < mq; ++i) {  // one copy of the list code
                float di = d2[0];
                unsigned ii = ix[0];
#pragma unroll
                for (int j = 1; j < kIsoBatch; ++j) {
                    di = i == j ? d2[j] : di;
                    ii = i == j ? ix[j] : ii;
                }
                const unsigned hits = __ballot_sync(kFullMask, !(di > bound) && ii != kNoIndex);
                if (hits) {
                    list_add<KR>(b, make_key(__float_as_uint(di), ii), hits);
                    bound = fminf(bound, list_kth<KR>(b, k));
                }
            }
        };
        const auto bound_up = [&]() { return isinf(bound) ? 0xFFFEu : bound_bits_up(bound); };
        // quarters waiting for evaluation, the latest first (warp-uniform)
        int w0 = 0, w1 = 0, w2 = 0, w3 = 0, nbatch = 0;
        unsigned lo_bits = 0;  // this round takes tiles whose gap lies in [lo_bits, hi_bits]
        for (int round = 0; round < 3; ++round) {
            shared_bound();
            const float frac = round == 0 ? 0.0625f : round == 1 ? 0.25f : 1.0f;
            unsigned hi_bits = bound_bits_up(bound * frac);
            if (round == 2 || hi_bits > 0xFFFEu) hi_bits = 0xFFFEu;  // the last round takes every quarter left
            if (hi_bits < lo_bits) continue;
            for (int bi = 0; bi < nb; ++bi) {
                const int t = 32 * bi + lane;
                const unsigned g = t < nt ? qgap_s[kQuarters * t + warp] : kGapSkip;
                unsigned todo = __ballot_sync(kFullMask, g >= lo_bits && g <= hi_bits && g <= bound_up());
                while (todo) {
                    const int src = __ffs(todo) - 1;
                    todo &= todo - 1;
                    if (__shfl_sync(kFullMask, g, src) > bound_up()) continue;  // a tighter bound prunes it
                    const int qn = (32 * bi + src) * kQuarters + warp;
                    w3 = w2;
                    w2 = w1;
                    w1 = w0;
                    w0 = qn;
                    if (++nbatch == kIsoBatch) {
                        eval(w0, w1, w2, w3, nbatch);
                        nbatch = 0;
                        shared_bound();
                    }
                }
            }
            lo_bits = hi_bits + 1;
        }
        if (nbatch > 0) eval(w0, w1, w2, w3, nbatch);
#pragma unroll
        for (int j = 0; j < KR; ++j) fin[warp][32 * j + lane] = b[j];
        __syncthreads();
        if (warp == 0) {
            for (int w = 1; w < kIsoWarps; ++w)
#pragma unroll
                for (int j = 0; j < KR; ++j) {
                    const uint64_t key = fin[w][32 * j + lane];
                    const unsigned have = __ballot_sync(kFullMask, key != kKeyMax);
                    if (have) list_add<KR>(b, key, have);
                }
            emit_row<KR>(b, k, n, perm[pos], nbr_idx, nbr_d2, kdist2);
        }
        __syncthreads();
    }
}

struct SmallArgs {
    const float* tiles;
    const float* boxes;
    const __nv_bfloat16* qbox;
    const unsigned* perm;
    int64_t n;
    int nt, t0, mt, k, sms, segment;
    bool defer;
    const int* order;
    IsoRows iso;
    int32_t* idx;
    float* d2;
    float* kd;
    int* status;
    unsigned long long* evaluated;
    cudaStream_t s;
};

template <int DP, int KR, int G, int RW, int W>
void launch_small(const SmallArgs& A) {
    using Smem = SmallSmem<DP, KR, RW, W>;
    set_max_dynamic_smem(reinterpret_cast<const void*>(small_sweep_kernel<DP, KR, G, RW, W>), static_cast<int>(sizeof(Smem)));
    const unsigned grid = static_cast<unsigned>(static_cast<int64_t>(A.mt) * kCT / Smem::kRows);
    const SweepRows P{A.tiles, A.boxes, A.n, 0, A.nt, A.k, A.segment, A.idx, A.d2, A.kd, A.status, A.evaluated, false, A.iso};
    small_sweep_kernel<DP, KR, G, RW, W><<<grid, 32 * W, sizeof(Smem), A.s>>>(
        P, static_cast<int64_t>(A.t0) * kCT, A.order, A.mt, !A.defer ? 0 : A.mt <= kSparseWaves * A.sms ? 2 : 1);
    CG_LAUNCH_CHECK();
    if (!A.defer) return;
    const size_t gap_bytes = sizeof(uint16_t) * kQuarters * static_cast<size_t>(A.nt);
    constexpr size_t kDefaultDynamicSmem = 40 * 1024;
    if (gap_bytes > kDefaultDynamicSmem)
        set_max_dynamic_smem(reinterpret_cast<const void*>(small_iso_kernel<DP, KR>), 72 * 1024);
    small_iso_kernel<DP, KR><<<6 * A.sms, 32 * kIsoWarps, gap_bytes, A.s>>>(A.tiles, A.qbox, A.perm, A.n, A.nt, A.k,
                                                                           A.iso, A.idx, A.d2, A.kd);
    CG_LAUNCH_CHECK();
}

template <int DP, int KR, int G>
void dispatch_rows(const SmallArgs& A) {
    // Rows per CTA: 128 (16 per warp: a test per lane, each tile staged for
    // more rows) from 6 row tiles per SM up, else 64 (n = 200,000, d = 8,
    // k = 20: 4.42 against 5.59 ms per fit_predict; n = 20,000: 0.76 against
    // 0.61 ms, the larger CTAs leave SMs idle).
    if (A.mt >= 6 * A.sms) launch_small<DP, KR, G, 16, 8>(A);
    else launch_small<DP, KR, G, 8, 8>(A);
}
template <int DP>
void dispatch_small(const SmallArgs& A) {
    // one group of window columns per lane up to k = 24, two above (the bound
    // from 32 groups takes in 43 columns at k = 24 and 110 at k = 32)
    if (A.k <= 24) dispatch_rows<DP, 1, 1>(A);
    else if (A.k <= 32) dispatch_rows<DP, 1, 2>(A);
    else dispatch_rows<DP, 2, 2>(A);
}

constexpr int kOrderMaxTiles = 16384;
// Most rows that can leave (none without the pass of their own).
int64_t iso_capacity(int mt, bool defer) {
    return defer ? static_cast<int64_t>(mt) * kCT / 4 + static_cast<int64_t>(mt / 32) * kCT : 0;
}

}  // namespace

void small_refine_order(const float* xc, int64_t n, int d, unsigned* perm, cudaStream_t s) {
    const unsigned grid = static_cast<unsigned>(ceil_div(n, kChunk));
    switch (padded_dims(d)) {
        case 2: refine_order_kernel<2><<<grid, kChunk, 0, s>>>(xc, n, d, perm); break;
        case 4: refine_order_kernel<4><<<grid, kChunk, 0, s>>>(xc, n, d, perm); break;
        case 6: refine_order_kernel<6><<<grid, kChunk, 0, s>>>(xc, n, d, perm); break;
        default: refine_order_kernel<8><<<grid, kChunk, 0, s>>>(xc, n, d, perm); break;
    }
    CG_LAUNCH_CHECK();
}

size_t small_tiles_floats(int dp, int nt) { return static_cast<size_t>(tile_floats(dp)) * nt; }

void small_build_tiles(const float* xc, int64_t n, int d, const unsigned* perm, int nt, float* tiles, float* boxes,
                       void* qbox, cudaStream_t s) {
    __nv_bfloat16* qb = static_cast<__nv_bfloat16*>(qbox);
    switch (padded_dims(d)) {
        case 2: small_tile_kernel<2><<<nt, kCT, 0, s>>>(xc, n, d, perm, tiles, boxes, qb); break;
        case 4: small_tile_kernel<4><<<nt, kCT, 0, s>>>(xc, n, d, perm, tiles, boxes, qb); break;
        case 6: small_tile_kernel<6><<<nt, kCT, 0, s>>>(xc, n, d, perm, tiles, boxes, qb); break;
        default: small_tile_kernel<8><<<nt, kCT, 0, s>>>(xc, n, d, perm, tiles, boxes, qb); break;
    }
    CG_LAUNCH_CHECK();
}

bool small_defers(bool wanted, int nt, int mt) {
    return wanted && nt > kWindow && nt <= kIsoMaxTiles && mt <= kOrderMaxTiles;
}

size_t small_iso_bytes(int mt, int k, bool defer) {
    const size_t cap = static_cast<size_t>(iso_capacity(mt, defer));
    return sizeof(uint64_t) * cap * 32 * (k <= 32 ? 1 : 2) + sizeof(int) * (cap + (mt <= kOrderMaxTiles ? mt : 0));
}

void small_knn(const float* tiles, const float* boxes, const void* qbox, const unsigned* perm, int64_t n, int d, int nt,
               int t0, int mt, int k, int sms, bool defer, int segment, void* iso, int* iso_count, int32_t* nbr_idx, float* nbr_d2,
               float* kdist2, int* status, unsigned long long* evaluated, cudaStream_t s) {
    if (mt <= 0) return;
    SmallArgs A{tiles, boxes, static_cast<const __nv_bfloat16*>(qbox), perm, n, nt, t0, mt, k, sms,
                segment, defer, nullptr, {}, nbr_idx, nbr_d2, kdist2, status, evaluated, s};
    char* w = static_cast<char*>(iso);
    A.iso.count = iso_count;
    A.iso.list = reinterpret_cast<uint64_t*>(w);
    A.iso.pos = reinterpret_cast<int*>(w + sizeof(uint64_t) * static_cast<size_t>(iso_capacity(mt, defer)) * 32 * (k <= 32 ? 1 : 2));
    if (mt <= kOrderMaxTiles) {
        int* order = A.iso.pos + iso_capacity(mt, defer);
        tile_order_kernel<<<static_cast<unsigned>(ceil_div(mt, 32)), 256, 0, s>>>(boxes, padded_dims(d), t0, mt, order);
        CG_LAUNCH_CHECK();
        A.order = order;
    }
    switch (padded_dims(d)) {
        case 2: dispatch_small<2>(A); break;
        case 4: dispatch_small<4>(A); break;
        case 6: dispatch_small<6>(A); break;
        default: dispatch_small<8>(A); break;
    }
}

}  // namespace culof_gb300
