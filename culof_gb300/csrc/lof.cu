// Local reachability density, LOF scores, the contamination offset and the
// labels.
//
// lrd / score follow src/cuda/lof.cu:32-62 term for term: FP64 sums in slot
// order, sqrt of the max of squared distances, the 1e-10 guard, float results.
// The offset replaces the host-side np.percentile of src/culof/__init__.py:183
// with a GPU order-statistic select plus numpy's 'linear' interpolation; the
// labels are predict()'s `nof < offset_` (__init__.py:208-210).
#include <cooperative_groups.h>

#include <cmath>

#include "block.cuh"
#include "common.cuh"
#include "fp64.cuh"
#include "prep.cuh"

namespace culof_gb300 {

namespace {

constexpr int kBlock = 256;

// A CTA of 8 warps takes 32 points (lane = point): the warps compute the
// points' slot terms side by side, 32 slots at a time, and warp 0 adds them in
// slot order. One thread per point, its k terms one after another, was bound
// by the latency of that chain (a gather, an FP64 square root or division and
// an addition per slot: 32 + 21 us at n = 500, k = 20, and still 33 + 24 us at
// n = 20,000). From about 100,000 points on both forms are bound by the FP64
// units.
// `rows` (nullable) lists the m points of a row block (a shard of a
// row-sharded run), otherwise every point.
constexpr int kTermSlots = 32;
constexpr int kTermWarps = kBlock / 32;

__device__ __forceinline__ int64_t block_row(const int32_t* rows, int64_t m, int64_t n, int* status) {
    const int64_t r = static_cast<int64_t>(blockIdx.x) * 32 + (threadIdx.x & 31);
    if (r >= m) return -1;
    const int64_t i = rows ? static_cast<int64_t>(rows[r]) : r;
    if (i < 0 || i >= n) {
        if (status != nullptr) atomicExch(status, 2);
        return -1;
    }
    return i;
}

__global__ void __launch_bounds__(kBlock) lrd_kernel(const int32_t* __restrict__ nbr_idx,
                                                     const float* __restrict__ nbr_d2,
                                                     const float* __restrict__ kdist2, int64_t n, int k,
                                                     const int32_t* __restrict__ rows, int64_t m,
                                                     float* __restrict__ lrd, int* status) {
    __shared__ double term[kTermSlots][32];
    __shared__ int bad[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t i = block_row(rows, m, n, status);
    if (warp == 0) bad[lane] = status != nullptr && *status != 0 ? 1 : 0;
    __syncthreads();
    double sum = 0.0;
    for (int c0 = 0; c0 < k; c0 += kTermSlots) {
        const int c1 = k - c0 < kTermSlots ? k - c0 : kTermSlots;
        for (int t = warp; t < c1; t += kTermWarps) {
            double v = 0.0;
            if (i >= 0) {
                const int64_t o = static_cast<int64_t>(c0 + t) * n + i;
                const int32_t j = nbr_idx[o];
                if (j < 0 || j >= n) bad[lane] = 2;  // never for a valid k-NN graph; do not read out of range
                else v = __dsqrt_rn(static_cast<double>(fmaxf(kdist2[j], nbr_d2[o])));
            }
            term[t][lane] = v;
        }
        __syncthreads();
        if (warp == 0)
            for (int t = 0; t < c1; ++t) sum = __dadd_rn(sum, term[t][lane]);
        __syncthreads();
    }
    if (warp != 0 || i < 0) return;
    if (bad[lane]) {
        if (bad[lane] == 2 && status != nullptr) atomicExch(status, 2);
        lrd[i] = __int_as_float(0x7fc00000);
        return;
    }
    lrd[i] = __double2float_rn(__ddiv_rn(1.0, __dadd_rn(__ddiv_rn(sum, static_cast<double>(k)), 1e-10)));
}

// The slot terms are the correctly rounded quotients lrd_j / lrd_i, from one
// reciprocal per point (quotient(), fp64.cuh).
__global__ void __launch_bounds__(kBlock) score_kernel(const int32_t* __restrict__ nbr_idx,
                                                       const float* __restrict__ lrd, int64_t n, int k,
                                                       const int32_t* __restrict__ rows, int64_t m,
                                                       float* __restrict__ scores, float* __restrict__ nof,
                                                       int* status) {
    __shared__ double term[kTermSlots][32];
    __shared__ double recip[32];
    __shared__ int bad[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t i = block_row(rows, m, n, status);
    const double self = i >= 0 ? static_cast<double>(lrd[i]) : 1.0;
    if (warp == 0) {
        recip[lane] = __ddiv_rn(1.0, self);
        bad[lane] = 0;
    }
    __syncthreads();
    const double y = recip[lane];
    const bool quick = quotient_quick(y);
    double sum = 0.0;
    for (int c0 = 0; c0 < k; c0 += kTermSlots) {
        const int c1 = k - c0 < kTermSlots ? k - c0 : kTermSlots;
        for (int t = warp; t < c1; t += kTermWarps) {
            double v = 0.0;
            if (i >= 0) {
                const int32_t j = nbr_idx[static_cast<int64_t>(c0 + t) * n + i];
                if (j < 0 || j >= n) {
                    bad[lane] = 1;
                } else {
                    v = quotient(lrd[j], self, y, quick);
                }
            }
            term[t][lane] = v;
        }
        __syncthreads();
        if (warp == 0)
            for (int t = 0; t < c1; ++t) sum = __dadd_rn(sum, term[t][lane]);
        __syncthreads();
    }
    if (warp != 0 || i < 0) return;
    if (bad[lane]) {
        if (status != nullptr) atomicExch(status, 2);
        sum = __longlong_as_double(0x7ff8000000000000ll);
    }
    const float s = __double2float_rn(__ddiv_rn(sum, static_cast<double>(k)));
    scores[i] = s;
    if (nof != nullptr) nof[i] = -s;
}

// ---- contamination offset --------------------------------------------------

__global__ void offset_init_kernel(int* __restrict__ hist, OffsetState* __restrict__ st) {
    for (int b = threadIdx.x; b < kOffsetHistBins; b += blockDim.x) hist[b] = 0;
    if (threadIdx.x == 0) {
        st->prefix = 0u;
        st->below = 0;
        st->a_key = 0u;
        st->min_gt = 0xFFFFFFFFu;
        st->count_le = 0;
        st->offset = 0.0;
        st->offset_f = 0.0f;
    }
}

// Histogram of the digit (shift, width) of every key whose bits above the
// digit equal the prefix found so far.
__global__ void offset_hist_kernel(const float* __restrict__ nof, int64_t n, int shift, int width,
                                   int* __restrict__ hist, const OffsetState* __restrict__ st) {
    __shared__ int sh[kOffsetHistBins];
    const int bins = 1 << width;
    for (int b = threadIdx.x; b < bins; b += blockDim.x) sh[b] = 0;
    __syncthreads();
    const unsigned int hi_mask = (shift + width >= 32) ? 0u : (0xFFFFFFFFu << (shift + width));
    const unsigned int prefix = st->prefix;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const unsigned int key = order_bits(nof[i]);
        if ((key & hi_mask) == (prefix & hi_mask)) atomicAdd(&sh[(key >> shift) & (bins - 1)], 1);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < bins; b += blockDim.x)
        if (sh[b]) atomicAdd(&hist[b], sh[b]);
}

// Single block: locate the bin of the need-th key, extend the prefix, and
// clear the histogram for the next pass.
__global__ void offset_pick_kernel(int* __restrict__ hist, int shift, int width, int64_t rank,
                                   OffsetState* __restrict__ st) {
    __shared__ int warp_sums[kBlock / 32];
    __shared__ int found_bin, found_acc;
    const int bins = 1 << width;
    const int per = bins / kBlock;
    const int need = static_cast<int>(rank + 1) - st->below;
    int local = 0;
    for (int b = threadIdx.x * per; b < (threadIdx.x + 1) * per; ++b) local += hist[b];
    int total;
    const int excl = block_exclusive_scan(local, warp_sums, total);
    if (excl < need && excl + local >= need) {
        int acc = excl, bin = threadIdx.x * per;
        for (int b = threadIdx.x * per; b < (threadIdx.x + 1) * per; ++b) {
            if (acc + hist[b] >= need) {
                bin = b;
                break;
            }
            acc += hist[b];
        }
        found_bin = bin;
        found_acc = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        st->prefix |= static_cast<unsigned int>(found_bin) << shift;
        st->below += found_acc;
    }
    for (int b = threadIdx.x; b < kOffsetHistBins; b += blockDim.x) hist[b] = 0;
}

// count of keys <= a, and the smallest key > a.
__global__ void offset_next_kernel(const float* __restrict__ nof, int64_t n, OffsetState* __restrict__ st) {
    const unsigned int a = st->prefix;
    int cnt = 0;
    unsigned int mn = 0xFFFFFFFFu;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const unsigned int key = order_bits(nof[i]);
        if (key <= a) ++cnt;
        else mn = min(mn, key);
    }
    for (int o = 16; o > 0; o >>= 1) {
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&st->count_le, cnt);
        atomicMin(&st->min_gt, mn);
    }
}

__global__ void offset_finalize_kernel(int64_t n, int64_t lo, int use_upper, float w, OffsetState* __restrict__ st,
                                       double* __restrict__ out) {
    const float a = order_value(st->prefix);
    const float b = (static_cast<int64_t>(st->count_le) >= lo + 2 || lo >= n - 1) ? a : order_value(st->min_gt);
    const float diff = __fsub_rn(b, a);
    const float r = use_upper ? __fsub_rn(b, __fmul_rn(diff, w)) : __fadd_rn(a, __fmul_rn(diff, w));
    st->a_key = st->prefix;
    st->offset_f = r;
    st->offset = static_cast<double>(r);
    *out = static_cast<double>(r);
}

__global__ void labels_kernel(const float* __restrict__ nof, int64_t n, const double* __restrict__ offset,
                              int64_t* __restrict__ labels) {
    const float off = __double2float_rn(*offset);
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        labels[i] = nof[i] < off ? -1 : 1;
}

// The whole offset in one launch: a cluster of CTAs takes the radix passes
// over the scores with its histograms in (distributed) shared memory, then
// the smallest score above the order statistic, and writes the offset and,
// if asked for, the labels. Every CTA adds up the cluster's histograms and
// finds the bin itself, so a pass costs one cluster barrier. The separate
// kernels (an initialisation, three histograms, three bin searches, the next
// score, the result, the labels) are bound by their ten launches: 39 us of
// kernel time at n = 20,000 against 19.5 us here; they remain for inputs
// past kOffsetClusterMax scores, where eight CTAs are too few.
constexpr int kOffThreads = 1024;
constexpr int kOffCtas = 8;
constexpr int64_t kOffOneCta = 8192;  // up to here one CTA is as fast
constexpr int64_t kOffsetClusterMax = 1 << 20;

__global__ void __launch_bounds__(kOffThreads)
offset_cluster_kernel(const float* __restrict__ nof, int64_t n, int64_t lo, int use_upper, float w,
                      double* __restrict__ out, int64_t* __restrict__ labels) {
    namespace cg = cooperative_groups;
    __shared__ __align__(8) int hist[3][kOffsetHistBins];  // read two bins at a time
    __shared__ int warp_sums[kOffThreads / 32];
    __shared__ int found_bin, found_acc, found_eq;
    __shared__ unsigned mn_s;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = static_cast<int>(cl.block_rank()), nctas = static_cast<int>(cl.num_blocks());
    const int tid = threadIdx.x, lane = tid & 31;
    for (int b = tid; b < 3 * kOffsetHistBins; b += kOffThreads) (&hist[0][0])[b] = 0;
    if (tid == 0) mn_s = 0xFFFFFFFFu;
    __syncthreads();
    const int64_t stride = static_cast<int64_t>(nctas) * kOffThreads;
    const int64_t base = static_cast<int64_t>(rank) * kOffThreads;
    unsigned prefix = 0;
    int below = 0, eq = 0;
#pragma unroll 1
    for (int p = 0; p < 3; ++p) {
        const int shift = p == 0 ? 21 : p == 1 ? 10 : 0, width = p == 2 ? 10 : 11;
        const unsigned hi_mask = p == 0 ? 0u : 0xFFFFFFFFu << (shift + width);
        for (int64_t i0 = base; i0 < n; i0 += stride) {
            const int64_t i = i0 + tid;
            const unsigned key = i < n ? order_bits(nof[i]) : 0u;
            const bool in = i < n && ((key ^ prefix) & hi_mask) == 0u;
            // lanes of the same bin elect one adder (scores share few bins)
            const unsigned active = __ballot_sync(0xffffffffu, in);
            if (in) {
                const unsigned bin = (key >> shift) & ((1u << width) - 1u);
                const unsigned peers = __match_any_sync(active, bin);
                if (lane == __ffs(peers) - 1) atomicAdd(&hist[p][bin], __popc(peers));
            }
        }
        cl.sync();
        int c[2] = {0, 0};
        for (int r = 0; r < nctas; ++r) {
            const int2 v = *reinterpret_cast<const int2*>(cl.map_shared_rank(&hist[p][2 * tid], r));
            c[0] += v.x;
            c[1] += v.y;
        }
        int total;
        const int excl = block_exclusive_scan(c[0] + c[1], warp_sums, total);
        const int need = static_cast<int>(lo + 1) - below;
        if (excl < need && excl + c[0] + c[1] >= need) {
            const int second = excl + c[0] < need ? 1 : 0;
            found_bin = 2 * tid + second;
            found_acc = excl + (second ? c[0] : 0);
            found_eq = c[second];
        }
        __syncthreads();
        prefix |= static_cast<unsigned>(found_bin) << shift;
        below += found_acc;
        eq = found_eq;
        __syncthreads();
    }
    // the smallest key above the order statistic
    unsigned mn = 0xFFFFFFFFu;
    for (int64_t i = base + tid; i < n; i += stride) {
        const unsigned key = order_bits(nof[i]);
        if (key > prefix) mn = min(mn, key);
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    if (lane == 0) atomicMin(&mn_s, mn);
    cl.sync();
    mn = 0xFFFFFFFFu;
    for (int r = 0; r < nctas; ++r) mn = min(mn, *cl.map_shared_rank(&mn_s, r));
    const float a = order_value(prefix);
    const float b = (static_cast<int64_t>(below) + eq >= lo + 2 || lo >= n - 1) ? a : order_value(mn);
    const float diff = __fsub_rn(b, a);
    const float res = use_upper ? __fsub_rn(b, __fmul_rn(diff, w)) : __fadd_rn(a, __fmul_rn(diff, w));
    if (rank == 0 && tid == 0) *out = static_cast<double>(res);
    if (labels != nullptr)
        for (int64_t i = base + tid; i < n; i += stride) labels[i] = nof[i] < res ? -1 : 1;
    cl.sync();  // no CTA leaves while another reads its shared memory
}

// contamination 'auto': the offset is a constant.
__global__ void auto_labels_kernel(const float* __restrict__ nof, int64_t n, double* __restrict__ out,
                                   int64_t* __restrict__ labels) {
    const float off = -1.5f;
    if (blockIdx.x == 0 && threadIdx.x == 0) *out = static_cast<double>(off);
    if (labels == nullptr) return;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        labels[i] = nof[i] < off ? -1 : 1;
}

int small_grid(int64_t n) {
    int64_t g = ceil_div(n, kBlock);
    if (g > 152 * 4) g = 152 * 4;
    return static_cast<int>(g < 1 ? 1 : g);
}

}  // namespace

void compute_lrd(const int32_t* nbr_idx, const float* nbr_d2, const float* kdist2, int64_t n, int k,
                 float* lrd, int* status, cudaStream_t s, const int32_t* rows, int64_t m) {
    if (!rows) m = n;
    if (m <= 0) return;
    lrd_kernel<<<static_cast<unsigned>(ceil_div(m, 32)), kBlock, 0, s>>>(nbr_idx, nbr_d2, kdist2, n, k, rows, m,
                                                                             lrd, status);
    CG_LAUNCH_CHECK();
}

void compute_scores(const int32_t* nbr_idx, const float* lrd, int64_t n, int k, float* scores,
                    float* nof, int* status, cudaStream_t s, const int32_t* rows, int64_t m) {
    if (!rows) m = n;
    if (m <= 0) return;
    score_kernel<<<static_cast<unsigned>(ceil_div(m, 32)), kBlock, 0, s>>>(nbr_idx, lrd, n, k, rows, m, scores,
                                                                               nof, status);
    CG_LAUNCH_CHECK();
}

// numpy 'linear' percentile of a float32 array with a Python-float q as the
// reference's LOF.fit passes it (np.percentile(nof, 100.0 * c)):
// q = (100 c) / 100, v = (n - 1) q, lo = floor(v), gamma = v - lo; the
// interpolation itself runs in float32 (offset_finalize_kernel).
OffsetPlan plan_offset(int64_t n, double contamination) {
    OffsetPlan p{};
    if (contamination <= 0.0) {
        p.is_auto = 1;
        return p;
    }
    const double q = (100.0 * contamination) / 100.0;
    const double v = static_cast<double>(n - 1) * q;
    double lo = std::floor(v);
    if (v >= static_cast<double>(n - 1)) lo = static_cast<double>(n - 1);
    if (lo < 0) lo = 0;
    const double gamma = v - lo;
    p.lo = static_cast<int64_t>(lo);
    p.use_upper = gamma >= 0.5 ? 1 : 0;
    p.w = p.use_upper ? static_cast<float>(1.0 - gamma) : static_cast<float>(gamma);
    if (p.lo >= n - 1) {  // no upper neighbour: the largest value itself
        p.lo = n - 1;
        p.use_upper = 0;
        p.w = 0.0f;
    }
    return p;
}

size_t offset_scratch_bytes() { return kOffsetHistBins * sizeof(int) + sizeof(OffsetState); }

void contamination_offset(const float* nof, int64_t n, const OffsetPlan& plan, void* scratch,
                          double* offset_out_dev, int64_t* labels, cudaStream_t s) {
    if (plan.is_auto) {
        auto_labels_kernel<<<labels ? small_grid(n) : 1, kBlock, 0, s>>>(nof, n, offset_out_dev, labels);
        CG_LAUNCH_CHECK();
        return;
    }
    if (n <= kOffsetClusterMax) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr{};
        const unsigned ctas = n <= kOffOneCta ? 1u : kOffCtas;
        cfg.gridDim = dim3(ctas);
        cfg.blockDim = dim3(kOffThreads);
        cfg.stream = s;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = ctas;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        CG_CUDA(cudaLaunchKernelEx(&cfg, offset_cluster_kernel, nof, n, plan.lo, plan.use_upper, plan.w, offset_out_dev,
                                   labels));
        count_launch();
        return;
    }
    int* hist = static_cast<int*>(scratch);
    OffsetState* st = reinterpret_cast<OffsetState*>(hist + kOffsetHistBins);
    offset_init_kernel<<<1, kBlock, 0, s>>>(hist, st);
    CG_LAUNCH_CHECK();
    const int g = small_grid(n);
    const int shifts[3] = {21, 10, 0}, widths[3] = {11, 11, 10};
    for (int p = 0; p < 3; ++p) {
        offset_hist_kernel<<<g, kBlock, 0, s>>>(nof, n, shifts[p], widths[p], hist, st);
        CG_LAUNCH_CHECK();
        offset_pick_kernel<<<1, kBlock, 0, s>>>(hist, shifts[p], widths[p], plan.lo, st);
        CG_LAUNCH_CHECK();
    }
    offset_next_kernel<<<g, kBlock, 0, s>>>(nof, n, st);
    CG_LAUNCH_CHECK();
    offset_finalize_kernel<<<1, 1, 0, s>>>(n, plan.lo, plan.use_upper, plan.w, st, offset_out_dev);
    CG_LAUNCH_CHECK();
    if (labels == nullptr) return;
    labels_kernel<<<small_grid(n), kBlock, 0, s>>>(nof, n, offset_out_dev, labels);
    CG_LAUNCH_CHECK();
}

}  // namespace culof_gb300
