// The fused distance + filtered exact select on the tensor cores
// (8 < d <= 256): the same algorithm as the FP32 sweeps (fast.cu, wide.cu),
// with the per-pair filter value taken from an FP16 Gram tile computed by
// tcgen05.mma instead of an FP32 FMA chain.
//
//   * operands: the centred points in Morton order, scaled by a power of two
//     2^S (so the largest coordinate lands in [2^14, 2^15)) and rounded to
//     f16, row-major [padded][Kp] (Kp = 64, 128, 192 or 256, zero padded);
//   * a CTA owns a 128-row tile (its A operand stays in shared memory) and
//     streams 128-column tiles of the same array by TMA (two stages);
//   * one warp issues the TMA loads, one issues tcgen05.mma (M = N = 128,
//     K = 16 per instruction) into one of two TMEM accumulators, and four
//     epilogue warps read the accumulator back (thread = row) and evaluate
//     f = |b|^2 - 2 a.b with packed fma.rn.f32x2;
//   * first the rows' bounds: part of the column tiles only feed 64 group
//     minima of f per row, whose k-th smallest bounds the row's k-th f. A list
//     of k that starts empty takes about k ln(columns / k) entries before it
//     has its final threshold (375 per row for n = 200,000, k = 50); started
//     from the bound it takes a fraction of that;
//   * then every tile: if a chunk's smallest f reaches the row's threshold tau,
//     the passing pairs' (f, column) enter the row's list (the row's own
//     thread appends them; no coordinates are read). Lists are compacted by
//     f: with fk the k-th smallest f in the list, every entry above a proven
//     margin over fk (approx_thr) is strictly farther than k listed columns
//     and is dropped, and the filter threshold tightens to that margin;
//   * a second kernel rescores each row's surviving entries (about k) exactly
//     from FP32 row-major coordinates (the oracle's direct-difference chain)
//     and writes the k best in the reference's slot order. A row whose list
//     would overflow with entries inside the margin (a wide margin, duplicates)
//     switches to an exact list: its candidates are then rescored as they pass.
//     A row that rescores more than a pass over all points would cost leaves
//     this path for that pass (lost_rows.cu).
//
// What bounds it: the MMAs and their operand copies alone take 7.6 ms at
// n = 200,000, d = 128 (72% of the measured f16 rate); reading the
// accumulators back and testing them 10.2 ms, a quarter of that again for the
// bounds, and the list entries of about one chunk in six the rest of 20.2 ms
// (34.7 ms without the bounds and with the rescoring as the sweep's last
// phase). n = 30,011, d = 100, k = 30: 2.61 -> 0.68 ms; n = 50,000, d = 32,
// k = 20: 3.10 -> 1.43 ms.
//
// Exactness: the thresholds (row_bounds below) cover the f16 rounding of
// both operands (relative 2^-11, absolute 2^-14 in scaled units for values
// that fall below the f16 normal range or are flushed), the f32 accumulation
// of the tensor core (taken as K * 2^-20 relative), the float32 norms and
// the float32 evaluation of f, so no column that belongs to a row's k
// nearest is ever dropped. Data whose scale cannot be brought into the f16
// range (|S| > 62, or non-finite values) or whose squared norms come near the
// largest float (above 2^124: f would overflow) disable the filter: every row
// then leaves.
#include <cuda_fp16.h>

#include <cmath>
#include <cstdlib>

#include "common.cuh"
#include "engine.cuh"
#include "fast.cuh"
#include "prep.cuh"
#include "row_list.cuh"
#include "sweep_common.cuh"
#include "tc.cuh"
#include "tc_scale.cuh"

namespace culof_gb300 {

namespace {

using namespace sweep;

constexpr int kStages = 2;                        // column tiles in flight (two CTAs share an SM)
constexpr int kEpiWarps = 4;
constexpr int kTcThreads = 32 * (2 + kEpiWarps);  // producer, MMA, epilogue warps
constexpr int kTmemCols = 256;                    // two 128-column f32 accumulators
constexpr int kTcM = 128;                         // list capacity per row (k <= 64)
constexpr int kBox = 128 * 128;                   // bytes of one TMA box: 128 rows x 64 f16

// Sorted position p: f16 operand row (scaled), FP32 coordinates (row-major,
// dr = d rounded up to 4, zero padded), norm (+inf for padding) and original
// index (kNoIndex for padding). With split, element f < 3d of the row
// operand xh is [hi, lo, hi][f / d] of coordinate f % d and of the column
// operand xb [hi, hi, lo][f / d]; hi = f16(x), lo = f16(x - hi) (x - hi is
// exact in float32).
__global__ void tc_build_kernel(const float* __restrict__ xc, const float* __restrict__ norms, int64_t n, int d,
                                int Kp, int dr, int split, const unsigned* __restrict__ perm, int64_t padded,
                                const TcScale* __restrict__ scale, __half* __restrict__ xh, __half* __restrict__ xb,
                                float* __restrict__ xr, float* __restrict__ cn, unsigned* __restrict__ ix) {
    const float sc = scale->sc;
    const int64_t total = padded * Kp;
    for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total;
         e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t p = e / Kp;
        const int f = static_cast<int>(e % Kp);
        const bool valid = p < n;
        const unsigned orig = valid ? perm[p] : kNoIndex;
        const int seg = split ? f / d : 0, j = split ? f % d : f;
        const float x = (valid && j < d && seg < 3) ? xc[static_cast<int64_t>(orig) * d + j] : 0.0f;
        const float xs = x * sc;
        const __half hi = __float2half_rn(xs);
        if (split) {
            const __half lo = __float2half_rn(__fsub_rn(xs, __half2float(hi)));
            xh[e] = seg == 1 ? lo : hi;
            xb[e] = seg == 2 ? lo : hi;
        } else {
            xh[e] = hi;
        }
        if (f < dr) xr[p * dr + f] = f < d && valid ? xc[static_cast<int64_t>(orig) * d + f] : 0.0f;
        if (f == 0) {
            cn[p] = valid ? norms[orig] : __int_as_float(0x7f800000);
            ix[p] = orig;
        }
    }
}

// Residual norms of the single f16 operands: rn[p] >= |a - f16(a)| (unscaled;
// an operand below the f16 normal range may be flushed, so its residual is the
// larger of the value and its rounding error), and the largest of them. A
// warp per row; every rounding upwards. Bound by reading the coordinates. The
// worst case over all values, 2^-11 |a|, is about two and a half times the
// measured norm, and the filter's margin follows it (row_bounds): with it
// clusters of d = 64, n = 20,000, k = 20 take 3.1 ms for 6.7.
__global__ void __launch_bounds__(256) tc_resid_kernel(const float* __restrict__ xr, int64_t padded, int d, int dr,
                                                       TcScale* __restrict__ scale, float* __restrict__ rn) {
    const int lane = threadIdx.x & 31;
    const float sc = scale->sc;
    float most = 0.0f;
    const int64_t step = static_cast<int64_t>(gridDim.x) * 8;
    for (int64_t p = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5); p < padded; p += step) {
        float s = 0.0f;
        for (int f = lane; f < d; f += 32) {
            const float xs = xr[p * dr + f] * sc;
            const float hi = __half2float(__float2half_rn(xs));
            float r = fabsf(__fsub_rn(xs, hi));
            if (fabsf(hi) < 6.103515625e-05f) r = fmaxf(r, fabsf(xs));  // 2^-14
            s = __fmaf_ru(r, r, s);
        }
#pragma unroll
        for (int st = 16; st > 0; st >>= 1) s = __fadd_ru(s, __shfl_xor_sync(0xffffffffu, s, st));
        const float v = __fdiv_ru(__fsqrt_ru(s), sc);
        if (lane == 0) rn[p] = v;
        most = fmaxf(most, v);
    }
    __shared__ unsigned top;
    if (threadIdx.x == 0) top = 0u;
    __syncthreads();
    if (lane == 0) atomicMax(&top, __float_as_uint(most));
    __syncthreads();
    if (threadIdx.x == 0 && __ldcg(&scale->resmax) < top) atomicMax(&scale->resmax, top);
}

// ---- thresholds ---------------------------------------------------------------
// Per row a (float32 norm na, K = Kp terms, u = 2^-24, g the relative error of
// the float32 norms, A >= |a|, B >= |b| for every column b, ra >= |a - f16(a)|,
// rb >= |b - f16(b)| for every column b), the f16 Gram value G of a column b
// and its filter value f = fl(Nb - 2 G) satisfy
//   |G - a.b| <= E = ra B + (A + ra) rb + K ua (A + ra) (B + rb)
//   |f - (|b|^2 - 2 a.b)| <= m0 = g / (1 - g) Nmax + 2 E + u (Nmax + 2 (A B + E))
// (ua = 2^-20 per accumulated term of the tensor core). Two consequences, each evaluated with
// upward rounding:
//  * exact threshold: a column whose exact float32 distance is <= D has
//    f <= D c1 + c0 (c1 = (1 + 8u) / (1 - (K + 2) u),
//    c0 = -na / (1 + g) + m0 + 8u (na + Nmax + 2 A B));
//  * approximate threshold: with T the real squared distance and
//    D in T [1 - dl, 1 + dl] (dl = (K + 3) u / (1 - (K + 3) u)), a column b with
//    f_b > thr(fk) = fk + 2 m0 + 2 dl / (1 - dl) max(0, fk + na / (1 - g) + m0)
//    (+ slack) is strictly farther than every column c with f_c <= fk, so once
//    k columns with f <= fk are known, b can never be among the k nearest.
// With split operands (x = hi + r exactly, lo = f16(r), |r| <= uh |x|,
// |lo - r| <= uh |r| + eta, uh = 2^-11 the f16 rounding, eta the absolute f16
// error) the summed products hi.hi + lo.hi + hi.lo miss
// a.b by at most
//   E = (3 uh^2 + 3 uh^3) A B + eta (1 + uh) sqrt(d) (A + B) + 2 d eta^2
//       + Ka ua (1 + 3 uh) ((1 + uh) A + sqrt(Ka) eta) ((1 + uh) B + sqrt(Ka) eta)
// (Ka = the accumulated K, 16 per MMA step), in place of the first line of E.
struct RowBounds {
    float c0, c3, c4;  // per row: exact offset; approximate offset and shift
};
constexpr double kU = 5.9604644775390625e-08;  // 2^-24

__device__ RowBounds row_bounds(float na_f, float nmax_f, int K, float ra_f, float rb_f, float eta_f, int split_d,
                                int kacc) {
    const double uh = 4.8828125e-04;        // 2^-11
    const double ua = 9.5367431640625e-07;  // 2^-20
    const double g = (K + 1) * kU / (1.0 - (K + 1) * kU);
    const double a = static_cast<double>(na_f), m = static_cast<double>(nmax_f), eta = static_cast<double>(eta_f);
    const double A = sqrt(a / (1.0 - g)), B = sqrt(m / (1.0 - g));
    double E;
    if (split_d > 0) {
        const double sd = sqrt(static_cast<double>(split_d)), sa = sqrt(static_cast<double>(kacc));
        E = (3.0 * uh * uh + 3.0 * uh * uh * uh) * A * B + eta * (1.0 + uh) * sd * (A + B) +
            2.0 * split_d * eta * eta +
            kacc * ua * (1.0 + 3.0 * uh) * ((1.0 + uh) * A + sa * eta) * ((1.0 + uh) * B + sa * eta);
    } else {
        const double ra = static_cast<double>(ra_f), rb = static_cast<double>(rb_f);
        E = ra * B + (A + ra) * rb + K * ua * (A + ra) * (B + rb);
    }
    const double m0 = g / (1.0 - g) * m + 2.0 * E + kU * (m + 2.0 * (A * B + E));
    const double slack = 8.0 * kU * (a + m + 2.0 * A * B) + 1e-30;
    RowBounds r;
    r.c0 = __double2float_ru(-a / (1.0 + g) + m0 + slack);
    r.c3 = __double2float_ru(2.0 * m0 + slack);
    r.c4 = __double2float_ru(a / (1.0 - g) + m0);
    return r;
}
// (host) a double rounded up to float, and the two constants of the thresholds
float up_float(double x) {
    const float f = static_cast<float>(x);
    return static_cast<double>(f) < x ? std::nextafter(f, INFINITY) : f;
}
float exact_c1(int K) { return up_float((1.0 + 8.0 * kU) / (1.0 - (K + 2) * kU)); }
float approx_c2(int K) {
    const double dl = (K + 3) * kU / (1.0 - (K + 3) * kU);
    return up_float(2.0 * dl / (1.0 - dl) * (1.0 + 8.0 * kU));
}
// Filter threshold of a row from its exact k-th key.
__device__ __forceinline__ float exact_tau(uint64_t kth, float c1, float c0) {
    if (kth == kKeyMax) return __int_as_float(0x7f800000);
    return __fmaf_ru(__uint_as_float(key_bits(kth)), c1, c0);
}
// The approximate threshold over a k-th filter value fk.
__device__ __forceinline__ float approx_thr(float fk, float c2, float c3, float c4) {
    return __fadd_ru(fk, __fmaf_ru(fmaxf(0.0f, __fadd_ru(fk, c4)), c2, c3));
}

__device__ __forceinline__ uint64_t tau_pair(float tau) {
    // f <= tau  <=>  f - next_up(tau) < 0 (the sign of a rounded difference
    // is exact), so a packed subtract's sign bits decide two columns at once.
    const float t = isinf(tau) ? tau : nextafterf(tau, __int_as_float(0x7f800000));
    return dup2(t);
}

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    return static_cast<uint64_t>(__float_as_uint(lo)) | (static_cast<uint64_t>(__float_as_uint(hi)) << 32);
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Row modes: approximate lists hold (order_bits(f) << 32 | sorted column position);
// exact lists hold the usual (distance bits << 32 | original index).
constexpr int kModeApprox = 0;
constexpr int kModeExact = 1;
// Rows that lost_rows() takes afterwards. Rescoring a pair reads two rows of
// coordinates and costs 10 to 18 times a pair there (92 against 5.2 ps, d = 32,
// n = 20,000 equal points; 273 against 25, d = 128). So an exact row leaves once
// it has rescored kExactPerTile pairs per column tile of its share: with 8, a
// few rows of clusters (d = 128, n = 50,000, k = 50) left that are cheaper to
// keep (12.6 ms for 10.7), with 16 Cauchy data (d = 32, n = 20,000) take 7.4 ms
// for 5.2 (36.4 when no row left). Rows leave as soon as their list overflows
// (kLose) where a CTA's share of the columns is short, so that the budget would
// not cover the rescoring of the list itself (kShortShare tiles: 5,000 clustered
// points of 64 features 414 us for 726, 8,000 were slower that way, 959 for 739),
// and past 128 features, where a pair costs the most.
constexpr int kModeLost = 2;
constexpr int kExactPerTile = 16;
constexpr int kShortShare = 12;

// Per-row lists live in global memory (L2-resident while their CTA runs):
// kTcM keys per row, 128 rows per CTA. Keeping them out of shared memory
// lets two CTAs share an SM, so two epilogue warps per SM sub-partition
// hide each other's latencies.
constexpr int kTcListRow = kTcM;
constexpr size_t kTcListTile = static_cast<size_t>(kRT) * kTcListRow;  // keys per row tile
constexpr int kTcMaxTilesPerLaunch = 4096;                             // bounds the list workspace (512 MiB)

struct TcRows {
    uint64_t kth[kRT];            // exact k-th key known for the row (only decreases)
    float athr[kRT];              // approximate threshold of the row's list (+inf until k entries)
    float c0[kRT], c3[kRT], c4[kRT];  // RowBounds
    int cnt[kRT];
    int sorted[kRT];  // the row's list[0..sorted) is sorted (the last compaction's result)
    int mode[kRT];
    int abort;
};
// NB: operand boxes of 64 K values (2: d <= 128, two CTAs per SM; 4: d <= 256,
// one).
template <int NB>
struct TcSmem : TcRows {
    alignas(1024) uint8_t a[NB][kBox];  // row tile operand
    uint8_t b[kStages][NB][kBox];       // column tile operands
    float nb[kEpiWarps][2][kCT];  // column norms of the current and the next tile, per epilogue warp
    uint64_t full[kStages], empty[kStages], tfull[2], tempty[2], afull, fin;
    uint32_t tmem_base;
};
static_assert(2 * (sizeof(TcSmem<2>) + 1024 + 1024) <= 233472, "two tensor-sweep CTAs must fit on an SM");

// What a row leaves to the final kernel, beside its list.
struct TcRow {
    int cnt, mode;
    float c3, c4;
};

__device__ void tc_abort(TcRows& sh, int* status) {
    *reinterpret_cast<volatile int*>(&sh.abort) = 1;
    atomicExch(status, 1);
}
__device__ __forceinline__ bool tc_aborted(TcRows& sh) { return *reinterpret_cast<volatile int*>(&sh.abort) != 0; }

// g[b] for a lane-dependent b, without local memory: a 5-level select tree.
__device__ __forceinline__ uint32_t select32(const uint32_t (&g)[32], int b) {
    uint32_t v16[16], v8[8], v4[4], v2[2];
#pragma unroll
    for (int i = 0; i < 16; ++i) v16[i] = (b & 16) ? g[16 + i] : g[i];
#pragma unroll
    for (int i = 0; i < 8; ++i) v8[i] = (b & 8) ? v16[8 + i] : v16[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) v4[i] = (b & 4) ? v8[4 + i] : v8[i];
#pragma unroll
    for (int i = 0; i < 2; ++i) v2[i] = (b & 2) ? v4[2 + i] : v4[i];
    return (b & 1) ? v2[1] : v2[0];
}

// Exact key of (row position pa, column position pb), one lane: the oracle's
// direct-difference chain over row-major FP32 coordinates.
__device__ __forceinline__ uint64_t exact_key_lane(const float* __restrict__ xr, const unsigned* __restrict__ ix,
                                                   int64_t pa, int64_t pb, int dr) {
    const unsigned ib = __ldg(ix + pb);
    if (ib == kNoIndex) return kKeyMax;
    const float4* va = reinterpret_cast<const float4*>(xr + pa * dr);
    const float4* vb = reinterpret_cast<const float4*>(xr + pb * dr);
    float s = 0.0f;
#pragma unroll 4
    for (int f4 = 0; 4 * f4 < dr; ++f4) {  // (the zero padding past d adds fma(0, 0, s) = s)
        const float4 x = __ldg(va + f4), y = __ldg(vb + f4);
        const float xa[4] = {x.x, x.y, x.z, x.w}, yb[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float t = __fsub_rn(xa[q], yb[q]);
            s = __fmaf_rn(t, t, s);
        }
    }
    return make_key(__float_as_uint(s), ib);
}

constexpr int kListE = kTcListRow / 32;  // list keys per lane in a compaction
static_assert(kListE == 4, "the compaction sorts 4 keys per lane");

// Exact list of row r (whole warp): sort, drop duplicates, keep the k
// smallest; tighten the row's exact k-th key.
__noinline__ __device__ void compact_exact(TcRows& sh, uint64_t* __restrict__ lst, int r, int k) {
    const int lane = threadIdx.x & 31;
    const int c = min(sh.cnt[r], kTcListRow);
    {
        const int s = sh.sorted[r];
        if (s <= c && c - s <= 64) {  // merge the new entries into the sorted prefix
            uint64_t kk;
            const int kept = merge_sorted_prefix(lst, s, c, k, k - 1, [](uint64_t) { return kKeyMax; }, &kk);
            if (lane == 0) {
                sh.cnt[r] = kept;
                sh.sorted[r] = kept;
                if (kk != kKeyMax && kk < sh.kth[r]) sh.kth[r] = kk;
            }
            __syncwarp();
            return;
        }
    }
    uint64_t v[kListE];
#pragma unroll
    for (int j = 0; j < kListE; ++j) {
        const int e = j * 32 + lane;
        v[j] = e < c ? lst[e] : kKeyMax;
    }
    warp_bitonic_sort<kListE>(v);
    int rank[kListE];
    const int uniq = warp_unique_ranks<kListE>(v, kKeyMax, rank);
    __syncwarp();
    uint64_t kth_new = kKeyMax;
#pragma unroll
    for (int j = 0; j < kListE; ++j) {
        if (rank[j] >= 0 && rank[j] < k) lst[rank[j]] = v[j];
        if (rank[j] == k - 1) kth_new = v[j];
    }
    const unsigned m = __ballot_sync(0xffffffffu, kth_new != kKeyMax);
    const uint64_t kk = __shfl_sync(0xffffffffu, kth_new, m ? __ffs(m) - 1 : 0);
    if (lane == 0) {
        sh.cnt[r] = min(uniq, k);
        sh.sorted[r] = min(uniq, k);
        if (m && kk < sh.kth[r]) sh.kth[r] = kk;
    }
    __syncwarp();
}

// Sort row r's approximate list (whole warp), find its k-th filter value fk
// and keep the entries with f <= approx_thr(fk) (all of them while fewer than
// k are known). Returns the number kept; if that exceeds `cap`, the list is
// left untrimmed and the caller decides.
__noinline__ __device__ int approx_compact(TcRows& sh, uint64_t* __restrict__ lst, int r, int k, float c2, float c3,
                                           float c4, int cap) {
    const int lane = threadIdx.x & 31;
    const int c = min(sh.cnt[r], kTcListRow);
    {
        const int s = sh.sorted[r];
        if (s <= c && c - s <= 64) {  // merge the new entries into the sorted prefix
            float thr = __int_as_float(0x7f800000);
            uint64_t fk;
            // entries above the margin over the k-th value are dropped (fewer
            // than k entries: all are kept)
            const int keep = merge_sorted_prefix(
                lst, s, c, kTcListRow, k - 1,
                [&](uint64_t key) -> uint64_t {
                    if (key == kKeyMax) return kKeyMax;
                    thr = approx_thr(order_value(key_bits(key)), c2, c3, c4);
                    return (static_cast<uint64_t>(order_bits(thr)) << 32) | 0xFFFFFFFFull;
                },
                &fk);
            if (lane == 0) {
                sh.cnt[r] = keep;
                sh.sorted[r] = keep;
                if (keep <= cap) sh.athr[r] = fminf(sh.athr[r], thr);
            }
            __syncwarp();
            return keep;
        }
    }
    uint64_t v[kListE];
#pragma unroll
    for (int j = 0; j < kListE; ++j) {
        const int e = j * 32 + lane;
        v[j] = e < c ? lst[e] : kKeyMax;
    }
    warp_bitonic_sort<kListE>(v);
    float thr = __int_as_float(0x7f800000);
    if (c >= k) {
        const int owner = (k - 1) & 31, oreg = (k - 1) >> 5;
        uint64_t kk = kKeyMax;
#pragma unroll
        for (int j = 0; j < kListE; ++j) {
            const uint64_t t = __shfl_sync(0xffffffffu, v[j], owner);
            if (j == oreg) kk = t;
        }
        thr = approx_thr(order_value(key_bits(kk)), c2, c3, c4);
    }
    int keep = 0;
#pragma unroll
    for (int j = 0; j < kListE; ++j) {
        const bool in = v[j] != kKeyMax && order_value(key_bits(v[j])) <= thr;
        keep += __popc(__ballot_sync(0xffffffffu, in));
    }
    if (keep <= cap) {
#pragma unroll
        for (int j = 0; j < kListE; ++j) {
            const int e = j * 32 + lane;
            if (e < keep) lst[e] = v[j];
        }
        if (lane == 0) {
            sh.cnt[r] = keep;
            sh.sorted[r] = keep;
            sh.athr[r] = fminf(sh.athr[r], thr);
        }
    }
    __syncwarp();
    return keep;
}

// Row r leaves approximate mode (its list would overflow with entries within
// the approximate margin, e.g. many duplicates): every entry is rescored
// exactly (one lane per entry) and the list becomes an exact k-best list.
__noinline__ __device__ void to_exact_mode(TcRows& sh, uint64_t* __restrict__ lst, int r, int64_t pa,
                                           const float* __restrict__ xr, const unsigned* __restrict__ ix, int dr,
                                           int k) {
    const int lane = threadIdx.x & 31;
    const int c = min(sh.cnt[r], kTcListRow);
    for (int e = lane; e < c; e += 32) {
        const int64_t pb = static_cast<int64_t>(key_index(lst[e]));
        lst[e] = pb != pa ? exact_key_lane(xr, ix, pa, pb, dr) : kKeyMax;  // not the row itself
    }
    __syncwarp();
    if (lane == 0) {
        sh.mode[r] = kModeExact;
        sh.sorted[r] = 0;  // exact keys: the approximate order no longer holds
    }
    __syncwarp();
    compact_exact(sh, lst, r, k);
}

// Candidates of exact-mode rows waiting to be rescored: one per lane, the
// first `n` lanes (n the same in all).
struct ExactPending {
    int n = 0;
    int row = 0;      // row of the tile
    int64_t col = 0;  // column position
};

// Rescores the pending pairs (whole warp, a lane per pair) and appends the keys
// that beat their row's k-th key. True if a list was compacted.
__noinline__ __device__ bool exact_flush(TcRows& sh, uint64_t* __restrict__ glist, const ExactPending& p, int64_t rbase,
                                         const float* __restrict__ xr, const unsigned* __restrict__ ix, int dr, int k) {
    const int lane = threadIdx.x & 31;
    uint64_t key = kKeyMax;
    if (lane < p.n) key = exact_key_lane(xr, ix, rbase + p.row, p.col, dr);
    const bool in = lane < p.n && key < sh.kth[p.row];
    const unsigned peers = __match_any_sync(0xffffffffu, in ? p.row : -1 - lane);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    int cnt = 0;
    if (in) {
        cnt = sh.cnt[p.row];
        glist[static_cast<size_t>(p.row) * kTcListRow + cnt + rank] = key;
    }
    __syncwarp();
    if (in && rank == 0) sh.cnt[p.row] = cnt + __popc(peers);
    __syncwarp();
    // room for the next 32 of a row
    unsigned full = __ballot_sync(0xffffffffu, in && rank == 0 && cnt + __popc(peers) > kTcListRow - 32);
    const bool compacted = full != 0;
    while (full) {
        const int r = __shfl_sync(0xffffffffu, p.row, __ffs(full) - 1);
        full &= full - 1;
        compact_exact(sh, glist + static_cast<size_t>(r) * kTcListRow, r, k);
    }
    return compacted;
}

// Exact-mode rows of a chunk (whole warp; pass: this lane's row's candidate
// columns, 0 for rows in approximate mode): the chunk's pairs join the pending
// ones, 32 at a time are rescored. A row at a time, its candidates over the
// lanes, leaves most lanes idle where the filter's margin is wide but passes a
// few columns per chunk (clusters, d = 64, n = 20,000, k = 20: 9.3 ms, this
// way 6.7).
// True if a list was compacted.
__noinline__ __device__ bool exact_chunk(TcRows& sh, uint64_t* __restrict__ glist, int row0, unsigned pass,
                                         ExactPending& p, int64_t rbase, int64_t cbase, const float* __restrict__ xr,
                                         const unsigned* __restrict__ ix, int dr, int k) {
    const int lane = threadIdx.x & 31;
    bool compacted = false;
    const int64_t own = rbase + row0 + lane - cbase;  // not the row itself
    if (own >= 0 && own < 32) pass &= ~(1u << static_cast<int>(own));
    // a row that most columns pass: the lanes are its columns, consecutive in
    // memory (20,000 equal points of 32 features: 38 ms for 42)
    unsigned dense = __ballot_sync(0xffffffffu, __popc(pass) >= 16);
    while (dense) {
        const int src = __ffs(dense) - 1;
        dense &= dense - 1;
        const unsigned cols = __shfl_sync(0xffffffffu, pass, src);
        ExactPending q;
        q.row = row0 + src;
        q.col = cbase + __fns(cols, 0, lane + 1);
        q.n = __popc(cols);
        compacted |= exact_flush(sh, glist, q, rbase, xr, ix, dr, k);
        if (lane == src) pass = 0u;
    }
    while (__any_sync(0xffffffffu, pass != 0u)) {
        // every row with candidates left gives one to the next free lanes
        const unsigned rows = __ballot_sync(0xffffffffu, pass != 0u);
        const int give = __popc(rows), room = 32 - p.n, take = give < room ? give : room;
        const int mine = __popc(rows & ((1u << lane) - 1u));  // my place among the givers
        const int b = pass != 0u ? __ffs(pass) - 1 : 0;
        const int want = lane - p.n;  // which giver this lane takes
        const int src = want < 0 || want >= take ? 0 : give == 32 ? want : static_cast<int>(__fns(rows, 0, want + 1));
        const int gb = __shfl_sync(0xffffffffu, b, src);
        if (want >= 0 && want < take) {
            p.row = row0 + src;
            p.col = cbase + gb;
        }
        if (pass != 0u && mine < take) pass &= pass - 1;
        p.n += take;
        if (p.n == 32) {
            compacted |= exact_flush(sh, glist, p, rbase, xr, ix, dr, k);
            p.n = 0;
        }
    }
    return compacted;
}

// Column tiles of a CTA's share that are scanned for the rows' bounds: 128, or
// a quarter if that is more. A longer scan costs more than the list entries it
// saves, a shorter one less (fit_predict with a scan of 1/8, 1/4, 1/2 and all:
// 1563 tiles, d = 128, k = 50: 24.2, 24.0, 25.0, 28.1 ms; 235 tiles, d = 100,
// k = 30: 1.60, 1.51, 1.42, 1.43 ms; 157 tiles, d = 32, k = 20: 1.48, 1.38,
// 1.29, 1.22 ms).
// (k = 64, d = 24, n = 20,000: 2.8 ms in two halves, 3.2 without a scan; the
// lists of k = 50 are as fast either way, 0.9 ms)
constexpr int kHalvesK = 56;
__device__ __forceinline__ int bound_tiles(int count) { return min(count, max(128, count / 4)); }

template <int NB, bool kLose>
__global__ void __launch_bounds__(kTcThreads, NB == 2 ? 2 : 1)
tc_sweep_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap tmapb,
                const float* __restrict__ xr,
                const float* __restrict__ cn, const float* __restrict__ rn, const unsigned* __restrict__ ix,
                const TcScale* __restrict__ scale, int nt, int T0, int ntb, int nsplit, int d, int dr, int Kp, int split_ops, int ksteps, int k, float c1,
                float c2, const unsigned* __restrict__ max_norm_bits, const unsigned long long* __restrict__ kth_seed,
                uint64_t* __restrict__ lists, TcRow* __restrict__ row_info, int* __restrict__ status, int qs,
                const uint2* __restrict__ plist, const int* __restrict__ pcount) {
    extern __shared__ uint8_t tc_raw[];
    TcSmem<NB>& sh = *reinterpret_cast<TcSmem<NB>*>((reinterpret_cast<uintptr_t>(tc_raw) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int T = T0 + static_cast<int>(blockIdx.x) % ntb;
    const int split = static_cast<int>(blockIdx.x) / ntb;
    // the split's column tiles: entries split + nsplit j of the row tile's
    // prune list (visiting order, tiles that the seed's k-th distances cannot
    // rule out), or its contiguous share of the spiral past the seed window
    const int per = (nt - qs + nsplit - 1) / nsplit;
    const int q0 = qs + split * per;
    const int q1 = min(nt, q0 + per);
    const int lcount = plist ? pcount[T] : 0;
    const bool off = scale->all != 0.0f;  // the f values carry no information: every row leaves
    const int count = off ? 0 : plist ? (lcount > split ? (lcount - split + nsplit - 1) / nsplit : 0) : (q1 > q0 ? q1 - q0 : 0);
    const uint2* tlist = plist ? plist + static_cast<int64_t>(T) * nt : nullptr;
    // without a seed window the row itself is among the columns: its list holds
    // one entry more
    const int kx = qs == 0 ? k + 1 : k;
    // tiles 0 .. scan - 1 are read twice: first for the rows' bounds (below)
    const int scan = bound_tiles(count);
    const int total = scan + count;
    const int halves = kx > kHalvesK && scan > 1 ? 2 : 1;
    auto col_tile = [&](int jj) -> int {
        // (two halves: the even tiles, then the odd)
        const int even = (scan + 1) / 2;
        const int j = jj >= scan ? jj - scan : halves == 1 ? jj : jj < even ? 2 * jj : 2 * (jj - even) + 1;
        return tlist ? static_cast<int>(tlist[split + nsplit * j].x) : spiral_tile(T, q0 + j, nt);
    };
    const int nkb = Kp / 64;
    const float nmax = __uint_as_float(*max_norm_bits);
    const int64_t rbase = static_cast<int64_t>(T) * kRT;
    uint64_t* glist = lists + static_cast<size_t>(blockIdx.x) * kTcListTile;

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&sh.full[s], 1);
            mbar_init(&sh.empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&sh.tfull[a], 1);
            mbar_init(&sh.tempty[a], kEpiWarps);
        }
        mbar_init(&sh.afull, 1);
        mbar_init(&sh.fin, 1);
        sh.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tc::tmem_alloc(&sh.tmem_base, kTmemCols);
    if (warp >= 2) {
        const int r = 32 * (warp & 3) + lane;
        sh.kth[r] = kth_seed ? kth_seed[rbase + r] : kKeyMax;
        sh.cnt[r] = 0;
        sh.sorted[r] = 0;
        sh.athr[r] = __int_as_float(0x7f800000);
        sh.mode[r] = off ? kModeLost : kModeApprox;
        const RowBounds rb = row_bounds(cn[rbase + r], nmax, Kp, split_ops ? 0.0f : rn[rbase + r],
                                        __uint_as_float(scale->resmax), scale->eta, split_ops ? d : 0, 16 * ksteps);
        sh.c0[r] = rb.c0;
        sh.c3[r] = rb.c3;
        sh.c4[r] = rb.c4;
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = sh.tmem_base;

    if (warp == 0) {
        // ---- TMA producer
        if (lane == 0) {
            int issued = 0;
            mbar_expect_tx(&sh.afull, nkb * kBox);
            for (int kb = 0; kb < nkb; ++kb) tc::tma_load_2d(sh.a[kb], &tmap, 64 * kb, static_cast<int>(rbase), &sh.afull);
            for (int j = 0; j < total; ++j) {
                const int s = j % kStages;
                if (j >= kStages && !mbar_wait(&sh.empty[s], (j / kStages - 1) & 1)) {
                    tc_abort(sh, status);
                    break;
                }
                if (tc_aborted(sh)) break;
                const int col0 = col_tile(j) * kCT;
                mbar_expect_tx(&sh.full[s], nkb * kBox);
                for (int kb = 0; kb < nkb; ++kb) tc::tma_load_2d(sh.b[s][kb], &tmapb, 64 * kb, col0, &sh.full[s]);
                issued = j + 1;
            }
            // no copy may still be landing in shared memory when the CTA exits
            if (!mbar_wait(&sh.afull, 0)) atomicExch(status, 1);
            for (int j = issued - kStages; j < issued; ++j)
                if (j >= 0 && !mbar_wait(&sh.full[j % kStages], (j / kStages) & 1)) atomicExch(status, 1);
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---- MMA issuer
        if (lane == 0) {
            constexpr uint32_t idesc = tc::f16_idesc(128, 128);
            bool ok = mbar_wait(&sh.afull, 0);
            if (!ok) tc_abort(sh, status);
            for (int j = 0; ok && j < total; ++j) {
                const int s = j % kStages, acc = j & 1;
                if (tc_aborted(sh) || !mbar_wait(&sh.full[s], (j / kStages) & 1) ||
                    (j >= 2 && !mbar_wait(&sh.tempty[acc], ((j >> 1) - 1) & 1))) {
                    tc_abort(sh, status);
                    break;
                }
                tc::tc_fence_after();
                const uint32_t dt = tmem + static_cast<uint32_t>(acc * 128);
                for (int kk = 0; kk < ksteps; ++kk) {
                    const int kb = kk >> 2, sub = kk & 3;
                    const uint64_t ad = tc::sw128_desc(smem_u32(sh.a[kb]) + 32 * sub);
                    const uint64_t bd = tc::sw128_desc(smem_u32(sh.b[s][kb]) + 32 * sub);
                    tc::mma_f16kind(dt, ad, bd, idesc, kk > 0);
                }
                tc::mma_commit(&sh.tfull[acc]);
                tc::mma_commit(&sh.empty[s]);
            }
            // every MMA issued has completed before TMEM is released
            tc::mma_commit(&sh.fin);
            if (!mbar_wait(&sh.fin, 0)) atomicExch(status, 1);
        }
        __syncwarp();
    } else {
        // ---- epilogue: thread = row
        const int wq = warp - 2;
        const int row0 = 32 * (warp & 3);  // the TMEM lanes this warp may read
        const int r = row0 + lane;
        uint64_t* const mylist = glist + static_cast<size_t>(r) * kTcListRow;
        const TcScale sc = *scale;
        const bool row_valid = __ldg(ix + rbase + r) != kNoIndex;
        bool exact_any = false;  // some list of the warp is exact
        bool exact_row = false;
        bool lost = off;
        int exact_left = kExactPerTile * count;  // pairs that this row may rescore
        // (from k = 48 on, a list that keeps much more than k by the wide margin of
        // single operands is compacted again every few entries: clusters of d = 140,
        // n = 4,100, k = 64 1.31 ms for 1.73; of d = 100 1.47 for 1.85)
        const int most_kept = kLose && !split_ops && kx > 48 ? min(kx + 12, kTcListRow - 32) : kTcListRow - 32;
        ExactPending pending;
        int cnt = 0;  // entries of this thread's list while it is approximate (sh.cnt while compacting)
        float tau = 0.0f;  // the list's threshold, and as a packed pair
        uint64_t tq = 0;
        auto set_tau = [&]() {
            tau = __int_as_float(0xff800000);
            if (row_valid && !lost) {
                tau = exact_tau(sh.kth[r], c1, sh.c0[r]);
                if (!exact_row) tau = fminf(tau, sh.athr[r]);
            }
            tq = tau_pair(tau);
        };
        set_tau();
        const uint64_t k2 = dup2(sc.k2);
        const uint32_t lane_addr = tmem + (static_cast<uint32_t>(row0) << 16);
        // This tile's column norms are staged in a per-warp shared ring one
        // tile ahead (one coalesced 512-byte load per warp), so the filter
        // never waits on global memory.
        auto tile_base = [&](int jj) -> int64_t {
            return static_cast<int64_t>(col_tile(jj)) * kCT;
        };
        auto tile_norms = [&](int jj) {
            return __ldg(reinterpret_cast<const float4*>(cn + tile_base(jj)) + lane);
        };
        float4 npre = make_float4(0.f, 0.f, 0.f, 0.f);
        if (total > 0) npre = tile_norms(0);
        int64_t cbase = 0;  // position of the tile's first column
        const float* nbj = nullptr;
        // The accumulator of tile j: its column norms staged (and the next
        // tile's requested), its MMA waited for. False if a wait expired.
        auto begin_tile = [&](int j) -> bool {
            cbase = tile_base(j);
            float* nbw = sh.nb[wq][j & 1];
            reinterpret_cast<float4*>(nbw)[lane] = npre;
            if (j + 1 < total) npre = tile_norms(j + 1);
            nbj = nbw;
            __syncwarp();
            if (!mbar_wait_warp(&sh.tfull[j & 1], (j >> 1) & 1)) {
                if (lane == 0) tc_abort(sh, status);
                return false;
            }
            tc::tc_fence_after();
            return true;
        };
        auto end_tile = [&](int j) {  // the accumulator is free for the next tile but one
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.tempty[j & 1]);
        };
        // filter one 32-column chunk held in registers; list its candidates
        auto process_chunk = [&](const uint32_t (&gr)[32], int ch) {
            // the chunk's smallest f decides whether anything passes
            uint64_t f[16];
            const float4* nb4 = reinterpret_cast<const float4*>(nbj + 32 * ch);
            float lo[2] = {__int_as_float(0x7f800000), __int_as_float(0x7f800000)};
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float4 nb = nb4[q];
                f[2 * q] = fma2(pack2(__uint_as_float(gr[4 * q]), __uint_as_float(gr[4 * q + 1])), k2, pack2(nb.x, nb.y));
                f[2 * q + 1] =
                    fma2(pack2(__uint_as_float(gr[4 * q + 2]), __uint_as_float(gr[4 * q + 3])), k2, pack2(nb.z, nb.w));
                lo[0] = fminf(fminf(lo[0], lo_f(f[2 * q])), hi_f(f[2 * q]));
                lo[1] = fminf(fminf(lo[1], lo_f(f[2 * q + 1])), hi_f(f[2 * q + 1]));
            }
            if (!__any_sync(0xffffffffu, fminf(lo[0], lo[1]) <= tau)) return;
            // the signs of f - tq (tq the next float above the threshold), in
            // four independent chains of shifts
            unsigned part[4] = {0, 0, 0, 0};
#pragma unroll
            for (int q = 3; q >= 0; --q) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint64_t dl = sub2(f[4 * c + q], tq);
                    part[c] = __funnelshift_l(static_cast<unsigned>(dl >> 32), part[c], 1);
                    part[c] = __funnelshift_l(static_cast<unsigned>(dl), part[c], 1);
                }
            }
            const unsigned pass = part[0] | part[1] << 8 | part[2] << 16 | part[3] << 24;
            if (!exact_row) {
                // approximate keys straight into the thread's own list (f
                // recomputed exactly as the packed filter did)
                unsigned pp = pass;
                while (pp) {
                    const int b = __ffs(pp) - 1;
                    pp &= pp - 1;
                    const float fb = __fmaf_rn(__uint_as_float(select32(gr, b)), sc.k2, nbj[32 * ch + b]);
                    mylist[cnt++] = make_key(order_bits(fb), static_cast<uint32_t>(cbase + 32 * ch + b));
                }
            }
            bool changed = false;
            __syncwarp();
            if (!kLose && exact_any) {
                changed = exact_chunk(sh, glist, row0, exact_row ? pass : 0u, pending, rbase, cbase + 32 * ch, xr, ix,
                                      dr, k);
                if (exact_row) exact_left -= __popc(pass);
                if (__any_sync(0xffffffffu, exact_row && exact_left < 0)) {
                    if (exact_row && exact_left < 0) {
                        sh.mode[r] = kModeLost;
                        lost = true;
                        exact_row = false;
                        cnt = 0;
                    }
                    exact_any = __any_sync(0xffffffffu, exact_row);
                    changed = true;
                }
            }
            // keep room for the next chunk: compact approximate lists with
            // less than 32 free slots
            unsigned full = __ballot_sync(0xffffffffu, !exact_row && cnt > kTcListRow - 32);
            if (full) {
                changed = true;
                if (!exact_row) sh.cnt[r] = cnt;
                __syncwarp();
                while (full) {
                    const int src = __ffs(full) - 1;
                    full &= full - 1;
                    uint64_t* lst = glist + static_cast<size_t>(row0 + src) * kTcListRow;
                    const int kept = approx_compact(sh, lst, row0 + src, kx, c2, sh.c3[row0 + src], sh.c4[row0 + src],
                                                    kTcListRow - 32);
                    if (kept <= most_kept) continue;
                    if (kLose) {
                        if (lane == src) lost = true;
                    } else {
                        to_exact_mode(sh, lst, row0 + src, rbase + row0 + src, xr, ix, dr, k);
                        exact_any = true;
                    }
                }
                exact_row = sh.mode[r] == kModeExact;
                cnt = lost ? 0 : sh.cnt[r];
            }
            if (changed) set_tau();
        };
        bool alive = true;
        if (scan > 0) {
            // Bounds first: the row's smallest f in each of 64 groups of the
            // scanned columns. k groups with a value <= B are k columns with
            // f <= B, so the k-th smallest of the minima bounds the row's k-th
            // f, and the threshold over it (approx_thr) starts the lists.
            // Above kHalvesK in two halves of the scan, half of the k from
            // each: the k-th smallest of 64 minima has about -64 ln(1 - k / 64)
            // scanned columns below it (102 at k = 51, all at 64), the halves
            // together -128 ln(1 - k / 128) (65 and 89).
            float gm[64];
            float B = __int_as_float(0xff800000), top = B;
#pragma unroll 1
            for (int part = 0; part < halves && alive; ++part) {
                const int need = halves == 1 ? kx : part == 0 ? (kx + 1) / 2 : kx / 2;
#pragma unroll
                for (int q = 0; q < 64; ++q) gm[q] = __int_as_float(0x7f800000);
                const int j1 = part == halves - 1 ? scan : (scan + 1) / 2;
                for (int j = part == 0 ? 0 : (scan + 1) / 2; j < j1; ++j) {
                    if (!begin_tile(j)) {
                        alive = false;
                        break;
                    }
                    const uint32_t taddr = lane_addr + static_cast<uint32_t>((j & 1) * 128);
#pragma unroll
                    for (int ch = 0; ch < 4; ++ch) {
                        uint32_t ga[32];
                        tc::tmem_ld32_bits(taddr + static_cast<uint32_t>(32 * ch), ga);
                        if (ch == 3) end_tile(j);
                        const float4* nb4 = reinterpret_cast<const float4*>(nbj + 32 * ch);
#pragma unroll
                        for (int q = 0; q < 8; q += 2) {
                            // columns c and c + 4 share a group: one three-way minimum
                            uint64_t f[4];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const float4 nb = nb4[q + e];
                                const uint32_t* g4 = ga + 4 * (q + e);
                                f[2 * e] = fma2(pack2(__uint_as_float(g4[0]), __uint_as_float(g4[1])), k2, pack2(nb.x, nb.y));
                                f[2 * e + 1] =
                                    fma2(pack2(__uint_as_float(g4[2]), __uint_as_float(g4[3])), k2, pack2(nb.z, nb.w));
                            }
                            float* g = gm + 16 * ch + 2 * q;
                            g[0] = fminf(fminf(g[0], lo_f(f[0])), lo_f(f[2]));
                            g[1] = fminf(fminf(g[1], hi_f(f[0])), hi_f(f[2]));
                            g[2] = fminf(fminf(g[2], lo_f(f[1])), lo_f(f[3]));
                            g[3] = fminf(fminf(g[3], hi_f(f[1])), hi_f(f[3]));
                        }
                    }
                }
                if (kLose) {
#pragma unroll
                    for (int q = 0; q < 64; ++q) top = fmaxf(top, gm[q]);
                }
                // the need-th smallest of the 64, by bisection over the ordered bits
                uint32_t at = 0;
#pragma unroll 1
                for (int bit = 31; bit >= 0; --bit) {
                    const float probe = order_value(at | ((1u << bit) - 1u));  // every value with this bit clear
                    int below = 0;
#pragma unroll
                    for (int q = 0; q < 64; ++q) below += gm[q] <= probe ? 1 : 0;
                    // (a probe that is not a number lies outside the floats: all
                    // values are below a positive one, none below a negative one)
                    if (probe != probe) below = bit == 31 || (at >> 31) ? 64 : 0;
                    if (below < need) at |= 1u << bit;
                }
                const float bound = need <= 64 ? order_value(at) : __int_as_float(0x7f800000);
                B = bound == bound ? fmaxf(B, bound) : __int_as_float(0x7f800000);
            }
            if (row_valid && B < __int_as_float(0x7f800000)) {
                const float athr = approx_thr(B, c2, sh.c3[r], sh.c4[r]);
                sh.athr[r] = athr;
                // a threshold over every group's minimum takes in more columns
                // than the list holds (for k up to 31 the bound it starts from
                // is close to the row's k-th f)
                if (kLose) lost = kx <= 32 && top <= athr;
            }
            set_tau();
        }
        for (int j = scan; alive && j < total; ++j) {
            if (!begin_tile(j)) break;
            const uint32_t taddr = lane_addr + static_cast<uint32_t>((j & 1) * 128);
            uint32_t ga[32];
#pragma unroll 1
            for (int ch = 0; ch < 4; ++ch) {
                tc::tmem_ld32_bits(taddr + static_cast<uint32_t>(32 * ch), ga);
                if (ch == 3) end_tile(j);  // released before its last columns are filtered
                process_chunk(ga, ch);
            }
        }
        if (!kLose && pending.n > 0) exact_flush(sh, glist, pending, rbase, xr, ix, dr, k);
        TcRow info;
        info.cnt = exact_row ? sh.cnt[r] : cnt;
        info.mode = lost ? kModeLost : exact_row ? kModeExact : kModeApprox;
        info.c3 = sh.c3[r];
        info.c4 = sh.c4[r];
        row_info[static_cast<size_t>(blockIdx.x) * kRT + r] = info;
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, kTmemCols);
    }
}

// ---- final: the rows' k best from their lists -------------------------------
//
// One warp per row. With fk the k-th smallest f (the row itself aside) over the lists of all splits,
// the entries within approx_thr(fk) (about k + 2) are rescored exactly, lane =
// candidate, and join the seed's list (if there is one), which is then written
// in the reference's slot order. It is bound by its gathers (4 dr bytes per candidate from L2).
// As the last phase of the sweep's four epilogue warps the same rescoring took
// 1.2 million cycles per CTA (n = 200,000, d = 128, k = 50: 6 ms of 27, and
// half of the sweep at n = 30,011); here a row's gathers hide behind those of
// 31 other warps per SM.
constexpr int kFinWarps = 8;
constexpr int kMaxTcSplits = 4;

template <int KR>
__global__ void __launch_bounds__(32 * kFinWarps)
tc_final_kernel(const float* __restrict__ xr, const unsigned* __restrict__ ix, int64_t n, int T0, int ntb, int nsplit,
                int dr, int k, int kx, float c2, const uint64_t* __restrict__ lists, const TcRow* __restrict__ row_info,
                const uint64_t* __restrict__ seed_keys, int32_t* __restrict__ nbr_idx, float* __restrict__ nbr_d2,
                float* __restrict__ kdist2, int32_t* __restrict__ lost_rows, int* __restrict__ lost_count) {
    __shared__ __align__(16) float row[kFinWarps][kMaxTensorD];
    __shared__ unsigned cand[kFinWarps][kMaxTcSplits * kTcListRow];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int local = blockIdx.x * kFinWarps + warp;  // row of the launch batch
    const int64_t pos = static_cast<int64_t>(T0) * kRT + local;
    if (local >= ntb * kRT || pos >= n) return;
    for (int f = lane; f < dr; f += 32) row[warp][f] = xr[pos * dr + f];
    uint64_t b[KR];
#pragma unroll
    for (int j = 0; j < KR; ++j) b[j] = seed_keys && 32 * j + lane < k ? seed_keys[pos * k + 32 * j + lane] : kKeyMax;
    // the approximate entries of all splits, 4 per lane and split
    uint64_t v[kMaxTcSplits * 4];
    int have = 0;
    float c3 = 0.0f, c4 = 0.0f;
#pragma unroll
    for (int s = 0; s < kMaxTcSplits; ++s) {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[4 * s + j] = kKeyMax;
        if (s >= nsplit) continue;
        const size_t at = static_cast<size_t>(s) * ntb * kRT + local;
        const TcRow info = row_info[at];
        if (info.mode == kModeLost) {
            if (lane == 0) lost_rows[atomicAdd(lost_count, 1)] = static_cast<int32_t>(__ldg(ix + pos));
            return;
        }
        c3 = info.c3;
        c4 = info.c4;
        const uint64_t* lst = lists + at * kTcListRow;
        if (info.mode == kModeExact) {  // exact keys already
            for (int e0 = 0; e0 < info.cnt; e0 += 32) list_merge<KR>(b, e0 + lane < info.cnt ? lst[e0 + lane] : kKeyMax);
            continue;
        }
        have += info.cnt;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (32 * j + lane < info.cnt) v[4 * s + j] = lst[32 * j + lane];
    }
    uint32_t keep = 0xFFFFFFFFu;  // ordered bits of the largest f that is kept
    if (have > kx) {
        uint32_t at = 0;
#pragma unroll 1
        for (int bit = 31; bit >= 0; --bit) {
            const uint32_t probe = at | ((1u << bit) - 1u);
            int below = 0;
#pragma unroll
            for (int j = 0; j < 4 * kMaxTcSplits; ++j) below += key_bits(v[j]) <= probe ? 1 : 0;
            if (__reduce_add_sync(0xffffffffu, below) < kx) at |= 1u << bit;
        }
        keep = order_bits(approx_thr(order_value(at), c2, c3, c4));
    }
    __syncwarp();
    int P = 0;
#pragma unroll
    for (int j = 0; j < 4 * kMaxTcSplits; ++j) {
        const bool in = v[j] != kKeyMax && key_bits(v[j]) <= keep && key_index(v[j]) != static_cast<uint32_t>(pos);
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) cand[warp][P + __popc(m & ((1u << lane) - 1u))] = key_index(v[j]);
        P += __popc(m);
    }
    __syncwarp();
    const float4* ra = reinterpret_cast<const float4*>(row[warp]);
    for (int e0 = 0; e0 < P; e0 += 32) {
        uint64_t key = kKeyMax;
        if (e0 + lane < P) {
            const int64_t pb = cand[warp][e0 + lane];
            const float4* rb = reinterpret_cast<const float4*>(xr + pb * dr);
            // the oracle's chain (padded dimensions are zero in both: fma(0, 0, s) = s)
            float s = 0.0f;
#pragma unroll 8
            for (int f = 0; f < dr / 4; ++f) {
                const float4 x = ra[f], y = __ldg(rb + f);
                float t = __fsub_rn(x.x, y.x);
                s = __fmaf_rn(t, t, s);
                t = __fsub_rn(x.y, y.y);
                s = __fmaf_rn(t, t, s);
                t = __fsub_rn(x.z, y.z);
                s = __fmaf_rn(t, t, s);
                t = __fsub_rn(x.w, y.w);
                s = __fmaf_rn(t, t, s);
            }
            const unsigned ib = __ldg(ix + pb);
            if (ib != kNoIndex) key = make_key(__float_as_uint(s), ib);
        }
        list_merge<KR>(b, key);
    }
    emit_row<KR>(b, k, n, __ldg(ix + pos), nbr_idx, nbr_d2, kdist2);
}

}  // namespace

// Split operands when the three d-wide segments fit one or two 64-wide
// boxes (d <= 42). CULOF_TC_SPLIT=0 keeps single f16 operands (measurement).
static bool tc_use_split(int d) {
    const char* env = std::getenv("CULOF_TC_SPLIT");
    if (env && env[0] == '0') return false;
    return d <= kTcSplitD;
}
static int tc_kp(int d, bool split) {
    const int w = split ? 3 * d : d;
    return (w + 63) / 64 * 64;
}

size_t tc_buffer_bytes(int64_t padded, int d) {
    const bool split = tc_use_split(d);
    const int Kp = tc_kp(d, split);
    const int dr = (d + 3) & ~3;
    const auto up = [](size_t x) { return (x + 255) & ~static_cast<size_t>(255); };
    return up(sizeof(__half) * padded * Kp) * (split ? 2 : 1) + up(sizeof(float) * padded * dr) +
           2 * up(sizeof(float) * padded) + up(sizeof(unsigned) * padded);
}

int tc_max_splits() { return kMaxTcSplits; }

static int64_t tc_list_tiles(int nt, int nsplit) {
    const int64_t tiles = static_cast<int64_t>(nt) * nsplit;
    return tiles > kTcMaxTilesPerLaunch ? kTcMaxTilesPerLaunch : tiles;
}
size_t tc_list_bytes(int nt, int nsplit) {
    return (sizeof(uint64_t) * kTcListTile + sizeof(TcRow) * kRT) * static_cast<size_t>(tc_list_tiles(nt, nsplit));
}

TcBuffers tc_prepare(void* buf, const float* xc, const float* norms, int64_t n, int d, const unsigned* perm, int nt,
                     void* scale, cudaStream_t s) {
    const int64_t padded = static_cast<int64_t>(nt) * kCT;
    const auto up = [](size_t x) { return (x + 255) & ~static_cast<size_t>(255); };
    TcBuffers b;
    const bool split = tc_use_split(d);
    b.split = split ? 1 : 0;
    b.Kp = tc_kp(d, split);
    b.ksteps = ((split ? 3 * d : d) + 15) / 16;
    b.dr = (d + 3) & ~3;
    char* p = static_cast<char*>(buf);
    b.xh = p;
    p += up(sizeof(__half) * padded * b.Kp);
    b.xb = b.xh;
    if (split) {
        b.xb = p;
        p += up(sizeof(__half) * padded * b.Kp);
    }
    b.xr = reinterpret_cast<float*>(p);
    p += up(sizeof(float) * padded * b.dr);
    b.cn = reinterpret_cast<float*>(p);
    p += up(sizeof(float) * padded);
    b.rn = reinterpret_cast<float*>(p);
    p += up(sizeof(float) * padded);
    b.ix = reinterpret_cast<unsigned*>(p);
    b.scale = scale;
    int64_t g = ceil_div(padded * b.Kp, 256);
    if (g > 152 * 16) g = 152 * 16;
    tc_build_kernel<<<static_cast<unsigned>(g), 256, 0, s>>>(xc, norms, n, d, b.Kp, b.dr, b.split, perm, padded,
                                                             reinterpret_cast<const TcScale*>(b.scale),
                                                             static_cast<__half*>(b.xh), static_cast<__half*>(b.xb),
                                                             b.xr, b.cn, b.ix);
    CG_LAUNCH_CHECK();
    if (!split) {
        g = ceil_div(padded, 8);
        if (g > 152 * 8) g = 152 * 8;
        tc_resid_kernel<<<static_cast<unsigned>(g), 256, 0, s>>>(b.xr, padded, d, b.dr, reinterpret_cast<TcScale*>(b.scale),
                                                                 b.rn);
        CG_LAUNCH_CHECK();
    }
    return b;
}

void tc_sweep(const TcBuffers& b, int64_t n, int nt, int t0, int mt, int nsplit, int d, int k, const unsigned* maxn,
              const unsigned long long* kth_seed, const uint64_t* seed_keys, uint64_t* lists, int* status,
              int32_t* nbr_idx, float* nbr_d2, float* kdist2, cudaStream_t s, int qs, int32_t* lost_rows,
              int* lost_count, const uint2* plist, const int* pcount) {
    const bool wide = b.Kp > 128;
    const size_t smem = (wide ? sizeof(TcSmem<4>) : sizeof(TcSmem<2>)) + 1024;
    const bool lose = wide || (nt - qs + nsplit - 1) / nsplit <= kShortShare;
    const auto kernel = wide ? tc_sweep_kernel<4, true> : lose ? tc_sweep_kernel<2, true> : tc_sweep_kernel<2, false>;
    set_max_dynamic_smem(reinterpret_cast<const void*>(kernel), static_cast<int>(smem));
    const CUtensorMap map = tc::make_kmajor_map(b.xh, static_cast<int64_t>(nt) * kCT, b.Kp, true);
    const CUtensorMap mapb = tc::make_kmajor_map(b.xb, static_cast<int64_t>(nt) * kCT, b.Kp, true);
    TcRow* info = reinterpret_cast<TcRow*>(lists + kTcListTile * static_cast<size_t>(tc_list_tiles(mt, nsplit)));
    const float c1 = exact_c1(b.Kp), c2 = approx_c2(b.Kp);
    const int kx = qs == 0 ? k + 1 : k;
    // row tiles in batches, so that the list workspace stays bounded
    const int ntb_max = kTcMaxTilesPerLaunch / nsplit;
    for (int T0 = t0; T0 < t0 + mt; T0 += ntb_max) {
        const int ntb = t0 + mt - T0 < ntb_max ? t0 + mt - T0 : ntb_max;
        kernel<<<ntb * nsplit, kTcThreads, smem, s>>>(
            map, mapb, b.xr, b.cn, b.rn, b.ix, reinterpret_cast<const TcScale*>(b.scale), nt, T0, ntb, nsplit, d, b.dr, b.Kp,
            b.split, b.ksteps, k, c1, c2, maxn, kth_seed, lists, info, status, qs, plist, pcount);
        CG_LAUNCH_CHECK();
        const unsigned grid = static_cast<unsigned>(ntb) * kRT / kFinWarps;
        if (k <= 32)
            tc_final_kernel<1><<<grid, 32 * kFinWarps, 0, s>>>(b.xr, b.ix, n, T0, ntb, nsplit, b.dr, k, kx, c2, lists, info,
                                                               seed_keys, nbr_idx, nbr_d2, kdist2, lost_rows, lost_count);
        else
            tc_final_kernel<2><<<grid, 32 * kFinWarps, 0, s>>>(b.xr, b.ix, n, T0, ntb, nsplit, b.dr, k, kx, c2, lists, info,
                                                               seed_keys, nbr_idx, nbr_d2, kdist2, lost_rows, lost_count);
        CG_LAUNCH_CHECK();
    }
}

}  // namespace culof_gb300
