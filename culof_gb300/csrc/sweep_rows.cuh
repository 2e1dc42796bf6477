// The row-pruned sweep over column tiles: how a CTA finds the k nearest of its
// rows among a set of points in spatial order (single problems of up to 8
// features in small.cu, where the design is described, and batches of up to 16
// in batched.cu).
#pragma once

#include <algorithm>

#include "row_list.cuh"
#include "small.cuh"

namespace culof_gb300 {
namespace small {

constexpr int kWindow = 5;          // tiles of the window: T, T+1, T-1, T+2, T-2
constexpr int kSmStages = kWindow;  // column tiles in flight (the window is staged whole)
constexpr float kDeferRatio = 4.0f;  // a row leaves when its squared k-th distance exceeds 4x the CTA's median

// Row record in shared memory (floats): coordinates, each twice (one operand
// of the packed f32x2 instructions), k-th distance, own index.
__host__ __device__ constexpr int row_stride(int dp) { return 2 * dp + 4; }

__device__ __forceinline__ uint64_t add2_rd(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

template <int DP, int KR, int RW, int W>
struct SmallSmem {
    static constexpr int kRows = W * RW;
    alignas(16) float tiles[kSmStages][tile_floats(DP)];  // also the unsorted tile list while no copy is in flight
    uint64_t list[kRows][32 * KR];
    alignas(16) float row[kRows][row_stride(DP)];
    uint64_t full_bar[kSmStages];
    alignas(8) unsigned ent[kSegTiles];  // (before: each warp's keys while it works on the window)
                                         // listed tiles in visiting order: gap bits (upper 16) and offset in the segment
    unsigned hist[32];
    float wbox[W][2][DP];
    float cbox[2][DP];
    float wkmax[8];       // largest k-th distance among each warp's rows
    float kdv[kRows];     // the rows' k-th distances at the end of the window
    float median;
    int done[kSmStages], stage_tile[kSmStages], last_fill[kSmStages];
    int next_e, count;
    int left;  // rows that asked to leave
    unsigned evaluated;
};
static_assert(kSegTiles * 4 <= kSmStages * tile_bytes(2), "the unsorted list fits in the stages");

// A row record's packed coordinates.
template <int DP>
__device__ __forceinline__ void load_row(const float* rec, uint64_t (&a)[DP]) {
#pragma unroll
    for (int f = 0; f < DP; f += 2) {
        const ulonglong2 v = reinterpret_cast<const ulonglong2*>(rec)[f / 2];
        a[f] = v.x;
        a[f + 1] = v.y;
    }
}
// This lane's two columns of a half of a tile.
template <int DP>
__device__ __forceinline__ void load_columns(const float* tl, int h, uint64_t (&x)[DP]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int f = 0; f < DP; ++f) x[f] = *reinterpret_cast<const uint64_t*>(tl + f * kCT + h * kHalf + 2 * lane);
}
// Exact distances (the oracle's chain: t = a - b, s = fma(t, t, s) over the
// dimensions in order) from a row to two columns, packed.
template <int DP>
__device__ __forceinline__ uint64_t pair_dist(const uint64_t (&a)[DP], const uint64_t (&x)[DP]) {
    uint64_t s = 0;
#pragma unroll
    for (int f = 0; f < DP; ++f) {
        const uint64_t t = sub2(a[f], x[f]);
        s = fma2(t, t, s);
    }
    return s;
}

// N floats (a multiple of 4) from a 16-byte boundary.
template <int N>
__device__ __forceinline__ void load4(const float* p, float (&v)[N]) {
    static_assert(N % 4 == 0, "whole 16-byte words");
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
        const float4 x = reinterpret_cast<const float4*>(p)[i];
        v[4 * i] = x.x;
        v[4 * i + 1] = x.y;
        v[4 * i + 2] = x.z;
        v[4 * i + 3] = x.w;
    }
}

// Rows that left the sweep: their positions, their lists and how many.
struct IsoRows {
    int* count;
    int* pos;
    uint64_t* list;  // [slot][32 KR]
};

// What a CTA's sweep works on.
struct SweepRows {
    const float* tiles;  // column tiles [nt]
    const float* boxes;  // their boxes, [nt][2 DP]
    int64_t n;           // points
    int64_t base;        // the CTA's first row position
    int nt, k, segment;
    int32_t* nbr_idx;    // outputs of the n points
    float* nbr_d2;
    float* kdist2;
    int* status;
    unsigned long long* evaluated;  // nullable
    bool sparse;                    // (kDefer) all rows leave after the window
    IsoRows iso;                    // (kDefer)
};

// One CTA: the k nearest of the rows at positions base .. base + W RW - 1 (those
// below n) among all n points. kDefer: isolated rows leave (see above).
template <int DP, int KR, int G, int RW, int W, bool kDefer>
__device__ __forceinline__ void sweep_rows(SmallSmem<DP, KR, RW, W>& sh, const SweepRows& P)
{
    constexpr int kRows = W * RW, kThreads = 32 * W;
    constexpr int kKd = 2 * DP, kSelf = 2 * DP + 1;  // fields of a row record
    constexpr unsigned kTileBytes = tile_bytes(DP);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* __restrict__ tiles = P.tiles;
    const float* __restrict__ boxes = P.boxes;
    const int64_t n = P.n, base = P.base;
    const int nt = P.nt, k = P.k, segment = P.segment;
    const int T = static_cast<int>(base / kCT);
    const int r_in_tile = static_cast<int>(base % kCT);
    const int wsize = nt < kWindow ? nt : kWindow;
    // a warp's rows are spread over (up to) 64 consecutive ones, so that the
    // CTA's warps have about the same work on every tile
    constexpr int kGroup = kRows < kHalf ? kRows : kHalf, kGroupWarps = kGroup / RW;
    const int rfirst = warp / kGroupWarps * kGroup + warp % kGroupWarps;
    const auto row_of = [&](int i) { return rfirst + i * kGroupWarps; };

    if (tid < kRows) {
        const float* own = tiles + static_cast<int64_t>(T) * tile_floats(DP);
        const unsigned self = reinterpret_cast<const unsigned*>(own)[tile_index_off(DP) + r_in_tile + tid];
#pragma unroll
        for (int f = 0; f < DP; ++f) {
            const float v = self != kNoIndex ? own[f * kCT + r_in_tile + tid] : 0.0f;
            sh.row[tid][2 * f] = v;
            sh.row[tid][2 * f + 1] = v;
        }
        sh.row[tid][kKd] = self != kNoIndex ? inf_f() : -inf_f();  // -inf: takes no candidates
        sh.row[tid][kSelf] = __uint_as_float(self);
    }
    for (int i = tid; i < kRows * 32 * KR; i += kThreads) (&sh.list[0][0])[i] = kKeyMax;
    if (tid < kSmStages) {
        sh.done[tid] = 0;
        sh.last_fill[tid] = 0;
    }
    if (tid < 8) sh.wkmax[tid] = tid < W ? inf_f() : -inf_f();
    if (tid == 0) {
        sh.evaluated = 0;
        for (int s = 0; s < kSmStages; ++s) mbar_init(&sh.full_bar[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        sh.left = 0;
    }
    __syncthreads();
    if (tid == 0) {
        // the window's tiles, one per stage (bulk copies are issued by one
        // thread: their operands live in registers uniform over the warp)
        for (int st = 0; st < kSmStages; ++st) {
            if (st < wsize) {
                const int t = spiral_tile(T, st, nt);
                mbar_expect_tx(&sh.full_bar[st], kTileBytes);
                tma_load_1d(sh.tiles[st], tiles + static_cast<int64_t>(t) * tile_floats(DP), kTileBytes,
                            &sh.full_bar[st]);
            } else {
                mbar_arrive_plain(&sh.full_bar[st]);
            }
        }
    }
    __syncwarp();
    // the tiles outside the window form a ring of `rest` tiles from first_up
    // on; entry u of the phases' concatenated segments starts half a segment
    // below the window, so that the first segment lies around it
    const int rest = nt - wsize;
    const int first_up = T + wsize / 2 + 1;
    int seg_at = 0;  // the current segment's first entry
    const auto ring_tile = [&](int u) {
        const int ring = (u + rest - min(rest, segment) / 2) % rest;
        return (first_up + ring) % nt;
    };

    // this lane's test: row tr of the warp against half th of a tile, its
    // coordinates as packed (-a, a)
    const int tr = lane & (RW - 1), th = lane / RW;
    const bool tester = th < kHalves;
    // (in registers up to 8 dimensions, read per tile above)
    constexpr int kHeld = DP <= 8 ? DP : 1;
    uint64_t na[kHeld];
    const auto negated_pair = [&](int f) {  // (-a, a)
        const float v = sh.row[row_of(tr)][2 * f];
        return static_cast<uint64_t>(__float_as_uint(-v)) | (static_cast<uint64_t>(__float_as_uint(v)) << 32);
    };
#pragma unroll
    for (int f = 0; f < kHeld; ++f) na[f] = negated_pair(f);

    // The stage loader (one warp at a time): the next listed tile whose gap is
    // within the CTA's largest k-th distance (stale values only prune less);
    // a stage with no tile left gets a sentinel.
    auto fill = [&](int stage, int fill_no) {
        float kmax = lane < 8 ? sh.wkmax[lane] : -inf_f();
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) kmax = fmaxf(kmax, __shfl_xor_sync(kFullMask, kmax, o));
        kmax = __shfl_sync(kFullMask, kmax, 0);
        int found = -1;
        int e0 = sh.next_e;
        const int count = sh.count;
        while (found < 0 && e0 < count) {
            const int e = e0 + lane;
            unsigned v = 0;
            bool pass = false;
            if (e < count) {
                v = sh.ent[e];
                pass = __uint_as_float(v & 0xFFFF0000u) <= kmax;
            }
            const unsigned mk = __ballot_sync(kFullMask, pass);
            if (mk) {
                const int o = __ffs(mk) - 1;
                found = static_cast<int>(__shfl_sync(kFullMask, v, o) & 0xFFFFu);
                e0 += o + 1;
            } else {
                e0 += 32;
            }
        }
        if (lane == 0) {
            sh.next_e = e0;
            sh.last_fill[stage] = fill_no;
            if (found >= 0) {
                const int t = ring_tile(seg_at + found);
                sh.stage_tile[stage] = t;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                mbar_expect_tx(&sh.full_bar[stage], kTileBytes);
                tma_load_1d(sh.tiles[stage], tiles + static_cast<int64_t>(t) * tile_floats(DP), kTileBytes,
                            &sh.full_bar[stage]);
            } else {
                sh.stage_tile[stage] = -1;
                mbar_arrive_plain(&sh.full_bar[stage]);
            }
        }
        __syncwarp();
    };

    bool ok = true;
    // The window: every row against all of its columns at once. The smallest
    // value of each of 32 (64) groups of columns, one or two groups per lane,
    // bounds the row's k-th distance by the k-th smallest of them; the columns
    // within that bound (about 31 of 640 at k = 20) are gathered, sorted and
    // merged. (Inserting the columns half by half into the list cost 2.5 times
    // the instructions of this form.)
    for (int st = 0; st < kSmStages; ++st) ok = ok && mbar_wait_warp(&sh.full_bar[st], 0);
    if (ok) {
#pragma unroll 1
        for (int i = 0; i < RW; ++i) {
            const int r = row_of(i);
            if (sh.row[r][kKd] < 0.0f) continue;  // padding row
            uint64_t ra[DP];
            load_row<DP>(sh.row[r], ra);
            unsigned v[4 * kWindow];  // distance bits; all ones: no candidate
#pragma unroll
            for (int q = 0; q < kWindow; ++q) {
#pragma unroll
                for (int h = 0; h < kHalves; ++h) {
                    uint64_t x[DP];
                    load_columns<DP>(sh.tiles[q], h, x);
                    const uint64_t s2 = pair_dist<DP>(ra, x);
                    v[4 * q + 2 * h] = static_cast<unsigned>(s2);
                    v[4 * q + 2 * h + 1] = static_cast<unsigned>(s2 >> 32);
                }
                const int t = q < wsize ? spiral_tile(T, q, nt) : nt;
                if (static_cast<int64_t>(t + 1) * kCT > n) {  // the last tile's padding, or no tile
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (static_cast<int64_t>(t) * kCT + (j >> 1) * kHalf + 2 * lane + (j & 1) >= n)
                            v[4 * q + j] = 0xFFFFFFFFu;
                }
            }
            const int own = r_in_tile + r;  // the row's own column
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if ((j >> 1) * kHalf + 2 * lane + (j & 1) == own) v[j] = 0xFFFFFFFFu;
            constexpr int kSpan = 4 * kWindow / G;
            unsigned g[G];
#pragma unroll
            for (int j = 0; j < G; ++j) {
                g[j] = v[j * kSpan];
#pragma unroll
                for (int e = 1; e < kSpan; ++e) g[j] = min(g[j], v[j * kSpan + e]);
            }
            unsigned bound = warp_rank_value<G>(g, k - 1);
            uint64_t b[KR];
#pragma unroll
            for (int j = 0; j < KR; ++j) b[j] = kKeyMax;
            // gather the keys within the bound (kBuf at most; the rest, if
            // any, by further rounds with the bound that the first ones give)
            constexpr int kBuf = kSegTiles / 2 / W;
            uint64_t* buf = reinterpret_cast<uint64_t*>(sh.ent) + warp * kBuf;
            for (;;) {
                int found = 0;
#pragma unroll
                for (int e = 0; e < 4 * kWindow; ++e) {
                    const bool in = v[e] <= bound && v[e] != 0xFFFFFFFFu;
                    const unsigned m = __ballot_sync(kFullMask, in);
                    const int at = found + __popc(m & ((1u << lane) - 1u));
                    if (in && at < kBuf) {
                        buf[at] = make_key(v[e], reinterpret_cast<const unsigned*>(
                                                     sh.tiles[e / 4])[tile_index_off(DP) + (e % 4 >> 1) * kHalf + 2 * lane + (e & 1)]);
                        v[e] = 0xFFFFFFFFu;  // taken
                    }
                    found += __popc(m);
                }
                __syncwarp();
                const int have = min(found, kBuf);
#pragma unroll 1
                for (int e0 = 0; e0 < have; e0 += 32)
                    list_merge<KR>(b, e0 + lane < have ? buf[e0 + lane] : kKeyMax);
                __syncwarp();
                if (found <= kBuf) break;
                const unsigned kb = list_kth_bits<KR>(b, k);
                bound = kb < bound ? kb : bound;
            }
#pragma unroll
            for (int j = 0; j < KR; ++j) sh.list[r][32 * j + lane] = b[j];
            const float kd = list_kth<KR>(b, k);  // the whole warp
            if (lane == 0) sh.row[r][kKd] = kd;
            __syncwarp();
        }
    }
    unsigned evaluated = 0;
    int m = kSmStages;  // fill number over all phases; the window was 0 .. kSmStages - 1
    // phase p > 0: segment p - 1 of the other tiles
    const int phases = 1 + (rest + segment - 1) / segment;
    if (__syncthreads_or(ok ? 0 : 1)) {
        if (tid == 0) atomicExch(P.status, 1);
        return;
    }
    for (int ph = 1; ph < phases; ++ph) {
        {
            // every row's k-th distance and the box of the rows that take part
            const int mine = row_of(lane & (RW - 1));
            const float kdr = lane < RW ? sh.row[mine][kKd] : -inf_f();
            float wk = kdr;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) wk = fmaxf(wk, __shfl_xor_sync(kFullMask, wk, o));
            if (ph == 1) {
                if constexpr (kDefer) {
                    if (lane < RW) sh.kdv[mine] = kdr;
                    __syncthreads();
                    if (tid < kRows) {
                        const float v = sh.kdv[tid];
                        int rank = 0;
                        for (int i = 0; i < kRows; ++i) {
                            const float w = sh.kdv[i];
                            rank += (w < v || (w == v && i < tid)) ? 1 : 0;
                        }
                        if (rank == kRows / 2) sh.median = v;
                    }
                    __syncthreads();
                    const float med = sh.median;
                    const bool sparse = P.sparse;  // a tile of a sparse region: all of its rows leave
                    const bool far = lane < RW && kdr >= 0.0f && kdr < inf_f() &&
                                     (sparse || (med > 0.0f && kdr > kDeferRatio * med));
                    unsigned leave = __ballot_sync(kFullMask, far);
                    // otherwise at most a quarter of the CTA's rows (the list's capacity)
                    const int most = sparse ? kRows : kRows / 4;
                    int first = 0;
                    if (lane == 0 && leave) first = atomicAdd(&sh.left, __popc(leave));
                    first = __shfl_sync(kFullMask, first, 0);
                    while (leave && first < most) {
                        const int i = row_of(__ffs(leave) - 1);
                        leave &= leave - 1;
                        ++first;
                        int slot = 0;
                        if (lane == 0) slot = atomicAdd(P.iso.count, 1);
                        slot = __shfl_sync(kFullMask, slot, 0);
                        if (lane == 0) {
                            P.iso.pos[slot] = static_cast<int>(base + i);
                            sh.row[i][kKd] = -inf_f();
                            sh.row[i][kSelf] = __uint_as_float(kNoIndex);
                        }
#pragma unroll
                        for (int j = 0; j < KR; ++j)
                            P.iso.list[(static_cast<int64_t>(slot) * KR + j) * 32 + lane] = sh.list[i][32 * j + lane];
                    }
                    __syncwarp();
                    wk = lane < RW ? sh.row[mine][kKd] : -inf_f();
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) wk = fmaxf(wk, __shfl_xor_sync(kFullMask, wk, o));
                }
                const bool in = lane < RW && sh.row[mine][kKd] >= 0.0f;
#pragma unroll
                for (int f = 0; f < DP; ++f) {
                    const float v = sh.row[mine][2 * f];
                    float lo = in ? v : inf_f(), hi = in ? v : -inf_f();
#pragma unroll
                    for (int o = RW / 2; o > 0; o >>= 1) {
                        lo = fminf(lo, __shfl_xor_sync(kFullMask, lo, o));
                        hi = fmaxf(hi, __shfl_xor_sync(kFullMask, hi, o));
                    }
                    if (lane == 0) {
                        sh.wbox[warp][0][f] = lo;
                        sh.wbox[warp][1][f] = hi;
                    }
                }
            }
            if (lane == 0) sh.wkmax[warp] = wk;
            if (tid < 32) sh.hist[tid] = 0;
            __syncthreads();
            if (ph == 1 && tid < DP) {
                float lo = inf_f(), hi = -inf_f();
                for (int w = 0; w < W; ++w) {
                    lo = fminf(lo, sh.wbox[w][0][tid]);
                    hi = fmaxf(hi, sh.wbox[w][1][tid]);
                }
                sh.cbox[0][tid] = lo;
                sh.cbox[1][tid] = hi;
            }
            seg_at = (ph - 1) * segment;
            const int len = min(segment, rest - seg_at);
            if (tid == 0) {
                sh.next_e = 0;
                sh.count = 0;
            }
            __syncthreads();
            float kmax = sh.wkmax[0];
            for (int w = 1; w < W; ++w) kmax = fmaxf(kmax, sh.wkmax[w]);
            // visiting order: the centres' squared distance in quarter octaves
            // over kmax / 8, 32 classes
            const int c0 = static_cast<int>(__float_as_uint(kmax * 0.125f) >> 21);
            unsigned* raw = reinterpret_cast<unsigned*>(&sh.tiles[0][0]);
            for (int i = tid; i < len; i += kThreads) {
                float bx[2 * DP];
                load4(boxes + static_cast<int64_t>(ring_tile(seg_at + i)) * 2 * DP, bx);
                float g2 = 0.0f, cd = 0.0f;
#pragma unroll
                for (int f = 0; f < DP; ++f) {
                    const float lo = bx[f], hi = bx[DP + f];
                    const float gap = fmaxf(0.0f, fmaxf(__fsub_rd(lo, sh.cbox[1][f]), __fsub_rd(sh.cbox[0][f], hi)));
                    g2 = __fadd_rd(g2, __fmul_rd(gap, gap));
                    const float cc = 0.5f * ((lo + hi) - (sh.cbox[0][f] + sh.cbox[1][f]));
                    cd = fmaf(cc, cc, cd);
                }
                const float g = __fmul_rd(g2, prune_shrink<DP>());
                unsigned v = 0xFFFFFFFFu;
                if (g <= kmax) {
                    int cls = static_cast<int>(__float_as_uint(cd) >> 21) - c0;
                    cls = cls < 0 ? 0 : cls > 31 ? 31 : cls;
                    atomicAdd(&sh.hist[cls], 1u);
                    // class in the low bits of the gap's 16 (rounded down further)
                    v = (__float_as_uint(g) & 0xFFFF0000u) | static_cast<unsigned>(cls);
                }
                raw[i] = v;
            }
            __syncthreads();
            if (warp == 0) {
                const unsigned c = sh.hist[lane];
                unsigned x = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned y = __shfl_up_sync(kFullMask, x, o);
                    if (lane >= o) x += y;
                }
                sh.hist[lane] = x - c;
                if (lane == 31) sh.count = static_cast<int>(x);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // before copies into the stages again
            __syncthreads();
            for (int i = tid; i < len; i += kThreads) {
                const unsigned v = raw[i];
                if (v != 0xFFFFFFFFu)
                    sh.ent[atomicAdd(&sh.hist[v & 31u], 1u)] = (v & 0xFFFF0000u) | static_cast<unsigned>(i);
            }
            __syncthreads();
        }
        if (warp == 0)
            for (int st = 0; st < kSmStages; ++st) fill((m + st) % kSmStages, m + st);

        for (;; ++m) {
            const int stage = m % kSmStages;
            if (!mbar_wait_warp(&sh.full_bar[stage], (m / kSmStages) & 1)) {
                ok = false;
                break;
            }
            if (sh.stage_tile[stage] < 0) break;  // the phase is done
            const float* tl = sh.tiles[stage];
            // which of the warp's rows can find a candidate in which half
            bool pass = false;
            if (tester) {
                float hb[2 * DP];
                load4(tl + tile_box_off(DP) + th * 2 * DP, hb);
                float g2 = 0.0f;
#pragma unroll
                for (int f = 0; f < DP; ++f) {  // (lo - a, a - hi) rounded down
                    const uint64_t lh = static_cast<uint64_t>(__float_as_uint(hb[2 * f])) |
                                        (static_cast<uint64_t>(__float_as_uint(hb[2 * f + 1])) << 32);
                    const uint64_t g = add2_rd(lh, DP <= 8 ? na[f % kHeld] : negated_pair(f));
                    const float gap = fmaxf(fmaxf(lo_f(g), hi_f(g)), 0.0f);
                    g2 = __fmaf_rd(gap, gap, g2);
                }
                pass = __fmul_rd(g2, prune_shrink<DP>()) <= sh.row[row_of(tr)][kKd];
            }
            const unsigned todo = __ballot_sync(kFullMask, pass);
            bool changed = false;
            if (todo) {
                evaluated += __popc(todo);
#pragma unroll 1
                for (int h = 0; h < kHalves; ++h) {
                    unsigned rows = (todo >> (h * RW)) & ((1u << RW) - 1u);
                    if (!rows) continue;
                    uint64_t x[DP];
                    load_columns<DP>(tl, h, x);
                    const uint2 ix = *reinterpret_cast<const uint2*>(tl + tile_index_off(DP) + h * kHalf + 2 * lane);
                    do {  // two rows at a time: two independent distance chains
                        const int r0 = row_of(__ffs(rows) - 1);
                        rows &= rows - 1;
                        const int r1 = rows ? row_of(__ffs(rows) - 1) : r0;
                        rows &= rows - 1;
                        uint64_t a0[DP], a1[DP];
                        load_row<DP>(sh.row[r0], a0);
                        load_row<DP>(sh.row[r1], a1);
                        const uint64_t s0 = pair_dist<DP>(a0, x), s1 = pair_dist<DP>(a1, x);
                        const float k0 = sh.row[r0][kKd], k1 = sh.row[r1][kKd];
                        // not farther than the k-th distance (NaN distances
                        // count as candidates, as their keys order last)
                        if (!__any_sync(kFullMask, !(lo_f(s0) > k0) || !(hi_f(s0) > k0) || !(lo_f(s1) > k1) ||
                                                       !(hi_f(s1) > k1)))
                            continue;
#pragma unroll 1
                        for (int w = 0; w < 2; ++w) {
                            if (w && r1 == r0) break;
                            const int r = w ? r1 : r0;
                            const uint64_t s2 = w ? s1 : s0;
                            float kd = w ? k1 : k0;
                            if (!__any_sync(kFullMask, !(lo_f(s2) > kd) || !(hi_f(s2) > kd))) continue;
                            // nothing but ties (duplicates): only a lower
                            // index enters (20,000 equal points: 1.5 ms for
                            // 8.3; testing every candidate by key cost 2.6%
                            // at n = 200,000, d = 8)
                            if (!__any_sync(kFullMask, lo_f(s2) < kd || hi_f(s2) < kd)) {
                                const uint64_t kk = sh.list[r][k - 1];
                                if (!__any_sync(kFullMask, (ix.x != kNoIndex && make_key(__float_as_uint(lo_f(s2)), ix.x) < kk) ||
                                                               (ix.y != kNoIndex && make_key(__float_as_uint(hi_f(s2)), ix.y) < kk)))
                                    continue;
                            }
                            uint64_t b[KR];
#pragma unroll
                            for (int j = 0; j < KR; ++j) b[j] = sh.list[r][32 * j + lane];
#pragma unroll 1
                            for (int e = 0; e < 2; ++e) {
                                const float d2 = e ? hi_f(s2) : lo_f(s2);
                                const unsigned i = e ? ix.y : ix.x;
                                const unsigned hits = __ballot_sync(kFullMask, !(d2 > kd) && i != kNoIndex);
                                if (hits) {
                                    list_add<KR>(b, make_key(__float_as_uint(d2), i), hits);
                                    kd = list_kth<KR>(b, k);
                                    changed = true;
                                }
                            }
#pragma unroll
                            for (int j = 0; j < KR; ++j) sh.list[r][32 * j + lane] = b[j];
                            if (lane == 0) sh.row[r][kKd] = kd;
                            __syncwarp();
                        }
                    } while (rows);
                }
            }
            if (changed) {
                float wk = lane < RW ? sh.row[row_of(lane & (RW - 1))][kKd] : -inf_f();
#pragma unroll
                for (int o = RW / 2; o > 0; o >>= 1) wk = fmaxf(wk, __shfl_xor_sync(kFullMask, wk, o));
                if (lane == 0) sh.wkmax[warp] = wk;
            }
            // done with this stage; the last warp out refills it
            __syncwarp();
            int prev = 0;
            if (lane == 0) {
                __threadfence_block();
                prev = atomicAdd(&sh.done[stage], 1);
            }
            prev = __shfl_sync(kFullMask, prev, 0);
            if (prev == W - 1) {
                if (lane == 0) sh.done[stage] = 0;
                fill(stage, m + kSmStages);
            }
        }
        if (__syncthreads_or(ok ? 0 : 1)) {
            if (tid == 0) atomicExch(P.status, 1);
            // wait (bounded) for this CTA's copies still in flight before exiting
            if (tid < kSmStages && sh.last_fill[tid] >= 0)
                mbar_wait(&sh.full_bar[tid], (sh.last_fill[tid] / kSmStages) & 1);
            __syncthreads();
            return;
        }
        m += kSmStages;  // every stage holds a sentinel: the next phase fills them anew
    }
    if (lane == 0 && evaluated) atomicAdd(&sh.evaluated, evaluated);
    for (int i = 0; i < RW; ++i) {
        const int r = row_of(i);
        const unsigned self = __float_as_uint(sh.row[r][kSelf]);
        if (self == kNoIndex) continue;  // padding, or the row's own pass writes it
        uint64_t b[KR];
#pragma unroll
        for (int j = 0; j < KR; ++j) b[j] = sh.list[r][32 * j + lane];
        emit_row<KR>(b, k, n, self, P.nbr_idx, P.nbr_d2, P.kdist2);
    }
    __syncthreads();
    if (tid == 0 && P.evaluated) atomicAdd(P.evaluated, static_cast<unsigned long long>(sh.evaluated));
}

}  // namespace small
}  // namespace culof_gb300
