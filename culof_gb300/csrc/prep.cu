// Preprocessing: centring / z-scoring and squared row norms.
//
// Reference: src/cuda/preprocess.cu:31-72 (standardize_kernel: FP64 mean and
// population std per feature, zero-variance features keep scale 1, x written
// back as float((x - mean) * inv_std)) and :75-84 (squared_norms_kernel: FP64
// sum of squares cast to float).
//
// The reference reduces each feature with one block (tree order). Here the
// reduction is split into partial sums over chunks of kCenterChunk rows, each
// summed sequentially in row order, and the partials are then summed in chunk
// order. That order is fixed and is the one the CPU oracle uses, so the FP64
// means (and the centred floats) agree with it bit for bit; the partials give
// n/kCenterChunk x d parallel work instead of d blocks.
#include "common.cuh"
#include "fp64.cuh"
#include "prep.cuh"

namespace culof_gb300 {

namespace {

constexpr int kApplyThreads = 1024;  // at most (center_apply_kernel)

__device__ __forceinline__ double center_term(double s, float x, double m, bool square) {
    if (!square) return __dadd_rn(s, widen(x));
    const double v = __dsub_rn(widen(x), m);
    return __dadd_rn(s, __dmul_rn(v, v));
}

// One thread per (chunk, feature). mean == nullptr: sums x; otherwise sums
// (x - mean)^2. Consecutive threads are consecutive features of the same
// rows, so each row read is coalesced across the feature threads.
__global__ void center_partials_kernel(const float* __restrict__ x, int64_t n, int d,
                                       const double* __restrict__ mean,
                                       double* __restrict__ partial) {
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t chunks = ceil_div(n, kCenterChunk);
    if (t >= chunks * d) return;
    const int64_t c = t / d;
    const int f = static_cast<int>(t % d);
    const int64_t begin = c * kCenterChunk;
    const int64_t end = begin + kCenterChunk < n ? begin + kCenterChunk : n;
    const double m = mean != nullptr ? mean[f] : 0.0;
    double s = 0.0;
    // 32 loads in flight under the previous 32 values' chain of additions
    float v[32];
    int64_t i = begin;
    const float* p = x + begin * d + f;
    if (i + 32 <= end) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = p[static_cast<int64_t>(j) * d];
        for (; i + 32 <= end; i += 32) {
            float u[32];
            p += static_cast<int64_t>(32) * d;
            if (i + 64 <= end) {
#pragma unroll
                for (int j = 0; j < 32; ++j) u[j] = p[static_cast<int64_t>(j) * d];
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) s = center_term(s, v[j], m, mean != nullptr);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = u[j];
        }
    }
    for (; i < end; ++i) s = center_term(s, x[i * d + f], m, mean != nullptr);
    partial[t] = s;
}

// One block per feature: the feature's partials are staged in shared memory
// (the whole block loads, many loads in flight), then one thread sums them in
// chunk order. mode 0 -> mean[f]; mode 1 -> inv_std[f] (population std; 1 for
// sd <= 1e-12).
constexpr int kFinalizeBuf = 4096;
__global__ void center_finalize_kernel(const double* __restrict__ partial, int64_t chunks,
                                       int d, int64_t n, int mode, double* __restrict__ mean,
                                       double* __restrict__ inv_std) {
    __shared__ double buf[kFinalizeBuf];
    const int f = blockIdx.x;
    double total = 0.0;
    for (int64_t c0 = 0; c0 < chunks; c0 += kFinalizeBuf) {
        const int m = static_cast<int>(chunks - c0 < kFinalizeBuf ? chunks - c0 : kFinalizeBuf);
        for (int i = threadIdx.x; i < m; i += blockDim.x) buf[i] = partial[(c0 + i) * d + f];
        __syncthreads();
        if (threadIdx.x == 0) {
            int i = 0;
            for (; i + 16 <= m; i += 16) {
                double v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = buf[i + j];
#pragma unroll
                for (int j = 0; j < 16; ++j) total = __dadd_rn(total, v[j]);
            }
            for (; i < m; ++i) total = __dadd_rn(total, buf[i]);
        }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    const double dn = static_cast<double>(n);
    if (mode == 0) {
        mean[f] = __ddiv_rn(total, dn);
        inv_std[f] = 1.0;
    } else {
        const double sd = __dsqrt_rn(__ddiv_rn(total, dn));
        inv_std[f] = (sd > 1e-12) ? __ddiv_rn(1.0, sd) : 1.0;
    }
}

// One pass over the n x d values: each thread stays on one feature (the
// block's active threads and its stride are multiples of d) and has
// kApplyLoads loads in flight. With mm, also the features' ranges for the
// spatial order (range_put), reduced in shared memory first. One load at a
// time, a comparison and a product per value that does not need them (an FP64
// instruction each) and 256-thread blocks with two global atomics per feature
// each took 158 us at n = 200,000, d = 128 (now 91, where the one FP64
// instruction per value takes 44), 39 at n = 30,011, d = 100 (16) and 32 at
// n = 8,000, d = 200 (13). Blocks of 1,024 threads mean fewer atomics; below
// d = 32, where those are few, the 341 threads of a feature in one block's
// shared atomics cost more (8 us for 5 at n = 50,021, d = 3): 256 threads.
constexpr int kApplyLoads = 4;
template <bool kScale>  // normalising (otherwise the scale is 1 and the product the value itself)
__global__ void __launch_bounds__(kApplyThreads)
center_apply_kernel(const float* __restrict__ x, int64_t n, int d, const double* __restrict__ mean,
                    const double* __restrict__ inv_std, float* __restrict__ xc, unsigned* __restrict__ mm) {
    __shared__ unsigned slo[kMaxRangeDims], shi[kMaxRangeDims];
    if (mm != nullptr) {
        for (int f = threadIdx.x; f < d; f += blockDim.x) slo[f] = shi[f] = 0u;
        __syncthreads();
    }
    const int64_t total = n * d;
    if (d <= static_cast<int>(blockDim.x)) {
        const int per = static_cast<int>(blockDim.x) / d * d;  // active threads
        if (static_cast<int>(threadIdx.x) < per) {
            const int f = static_cast<int>(threadIdx.x) % d;
            const double m = mean[f], inv = inv_std[f];
            unsigned lo = 0u, hi = 0u;
            const int64_t stride = static_cast<int64_t>(gridDim.x) * per;
            for (int64_t t = static_cast<int64_t>(blockIdx.x) * per + threadIdx.x; t < total;
                 t += stride * kApplyLoads) {
                float v[kApplyLoads];
#pragma unroll
                for (int j = 0; j < kApplyLoads; ++j)
                    if (t + j * stride < total) v[j] = x[t + j * stride];
#pragma unroll
                for (int j = 0; j < kApplyLoads; ++j) {
                    if (t + j * stride >= total) break;
                    double w = __dsub_rn(widen(v[j]), m);
                    if (kScale) w = __dmul_rn(w, inv);
                    const float c = narrow(w);
                    xc[t + j * stride] = c;
                    lo = max(lo, ~order_bits(c));
                    hi = max(hi, order_bits(c));
                }
            }
            if (mm != nullptr) {
                atomicMax(&slo[f], lo);
                atomicMax(&shi[f], hi);
            }
        }
    } else {
        for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
             t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
            const int f = static_cast<int>(t % d);
            double w = __dsub_rn(widen(x[t]), mean[f]);
            if (kScale) w = __dmul_rn(w, inv_std[f]);
            xc[t] = narrow(w);
        }
    }
    if (mm != nullptr) {
        __syncthreads();
        for (int f = threadIdx.x; f < d; f += blockDim.x) {
            // (ranges only grow: most blocks find theirs covered and write nothing)
            if (__ldcg(&mm[2 * f]) < slo[f]) atomicMax(&mm[2 * f], slo[f]);
            if (__ldcg(&mm[2 * f + 1]) < shi[f]) atomicMax(&mm[2 * f + 1], shi[f]);
        }
    }
}

// The whole centring of a small input in one launch: a CTA per feature keeps
// its column in shared memory (one float of padding per chunk, so that the
// threads' chunks lie in different banks), one thread per chunk sums it in
// row order, one thread adds the chunks, and the CTA writes the column back:
// the same operations in the same order as the kernels above. Those take
// three launches (five when normalising) of a few CTAs each, 55 us of kernel
// time at n = 500, d = 8 and 115 us normalising at n = 3,001, d = 5.
constexpr int kSmallRows = 8192;
constexpr int kSmallThreads = 256;
__global__ void __launch_bounds__(kSmallThreads)
center_small_kernel(const float* __restrict__ x, int n, int d, int normalize, double* __restrict__ partial,
                    double* __restrict__ mean, double* __restrict__ inv_std, float* __restrict__ xc,
                    unsigned* __restrict__ mm) {
    extern __shared__ double sq[];  // squares (when normalising), padded as the column
    float* col = reinterpret_cast<float*>(sq + (normalize ? n + n / kCenterChunk + 1 : 0));
    __shared__ double part[kSmallRows / kCenterChunk];
    __shared__ double stat[2];
    const int f = blockIdx.x, tid = threadIdx.x;
    for (int i = tid; i < n; i += kSmallThreads) col[i + i / kCenterChunk] = x[static_cast<int64_t>(i) * d + f];
    __syncthreads();
    const int chunks = (n + kCenterChunk - 1) / kCenterChunk;
    const double dn = static_cast<double>(n);
    for (int pass = 0; pass <= normalize; ++pass) {
        if (pass) {  // every thread: the squares, so that the chains below only add
            for (int i = tid; i < n; i += kSmallThreads) {
                const int at = i + i / kCenterChunk;
                const double v = __dsub_rn(widen(col[at]), stat[0]);
                sq[at] = __dmul_rn(v, v);
            }
            __syncthreads();
        }
        if (tid < chunks) {
            const int begin = tid * kCenterChunk, len = min(kCenterChunk, n - begin);
            const float* c = col + begin + tid;
            const double* q = sq + begin + tid;
            double s = 0.0;
            int i = 0;
            for (; i + 16 <= len; i += 16) {
                double v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = pass ? q[i + j] : widen(c[i + j]);
#pragma unroll
                for (int j = 0; j < 16; ++j) s = __dadd_rn(s, v[j]);
            }
            for (; i < len; ++i) s = __dadd_rn(s, pass ? q[i] : widen(c[i]));
            part[tid] = s;
            partial[static_cast<int64_t>(tid) * d + f] = s;
        }
        __syncthreads();
        if (tid == 0) {
            double total = 0.0;
            for (int c = 0; c < chunks; ++c) total = __dadd_rn(total, part[c]);
            if (pass == 0) {
                stat[0] = __ddiv_rn(total, dn);
                stat[1] = 1.0;
                mean[f] = stat[0];
            } else {
                const double sd = __dsqrt_rn(__ddiv_rn(total, dn));
                stat[1] = (sd > 1e-12) ? __ddiv_rn(1.0, sd) : 1.0;
            }
            inv_std[f] = stat[1];
        }
        __syncthreads();
    }
    if (xc == nullptr) return;
    const double m = stat[0], v = stat[1];
    unsigned lo = 0u, hi = 0u;
    for (int i = tid; i < n; i += kSmallThreads) {
        double w = __dsub_rn(widen(col[i + i / kCenterChunk]), m);
        if (normalize) w = __dmul_rn(w, v);
        const float c = narrow(w);
        xc[static_cast<int64_t>(i) * d + f] = c;
        lo = max(lo, ~order_bits(c));
        hi = max(hi, order_bits(c));
    }
    if (mm != nullptr) {
        lo = __reduce_max_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if ((tid & 31) == 0) {
            atomicMax(&mm[2 * f], lo);
            atomicMax(&mm[2 * f + 1], hi);
        }
    }
}

// norms[i] = (float) sum_f (double) xc[i,f]^2 (feature order), and the
// maximum norm (non-negative float bits order like the values). Bound by the
// chain of d multiply-adds per row: blocks of 64 rows reach every SM from
// 10,000 rows on, and a row's loads are 16 bytes wide (d a multiple of 4),
// because each touches 32 lines: 47 us at n = 200,000, d = 128 and 20 at
// n = 8,000, d = 200, where blocks of 256 rows and single loads took 101 and 29.
__global__ void norms_kernel(const float* __restrict__ xc, int64_t n, int d,
                             float* __restrict__ norms, unsigned int* __restrict__ max_norm_bits) {
    unsigned int local_max = 0u;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const float* row = xc + i * d;
        double s = 0.0;
        int f = 0;
        if ((d & 3) == 0) {
            const float4* r4 = reinterpret_cast<const float4*>(row);
            for (; f + 16 <= d; f += 16) {
                float4 u[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) u[j] = r4[f / 4 + j];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const double v = widen(reinterpret_cast<const float*>(u)[j]);
                    s = __fma_rn(v, v, s);  // (the square of a float is exact in double)
                }
            }
        }
        for (; f < d; ++f) {
            const double v = widen(row[f]);
            s = __fma_rn(v, v, s);
        }
        const float nf = __double2float_rn(s);
        norms[i] = nf;
        local_max = max(local_max, __float_as_uint(nf));
    }
    if (max_norm_bits != nullptr) {
        for (int o = 16; o > 0; o >>= 1) local_max = max(local_max, __shfl_xor_sync(0xffffffffu, local_max, o));
        if ((threadIdx.x & 31) == 0) atomicMax(max_norm_bits, local_max);
    }
}

int grid_for(int64_t items, int block, int max_blocks = 152 * 16) {
    int64_t g = ceil_div(items, block);
    if (g < 1) g = 1;
    if (g > max_blocks) g = max_blocks;
    return static_cast<int>(g);
}

}  // namespace

void center(const float* x, int64_t n, int d, bool normalize, float* xc, double* partial,
            double* mean, double* inv_std, cudaStream_t s, unsigned* mm) {
    if (d > kMaxRangeDims) mm = nullptr;
    const int64_t chunks = ceil_div(n, kCenterChunk);
    const int64_t items = chunks * d;
    // up to 8,192 rows (the column's shared memory) and 131,072 values (a
    // column's strided reads cost whole sectors)
    if (n <= kSmallRows && n * d <= (1 << 17)) {
        const size_t places = static_cast<size_t>(n) + n / kCenterChunk + 1;
        const size_t smem = places * (sizeof(float) + (normalize ? sizeof(double) : 0));
        set_max_dynamic_smem(reinterpret_cast<const void*>(center_small_kernel),
                             static_cast<int>((kSmallRows + kSmallRows / kCenterChunk + 1) * (sizeof(float) + sizeof(double))));
        center_small_kernel<<<d, kSmallThreads, smem, s>>>(
            x, static_cast<int>(n), d, normalize ? 1 : 0, partial, mean, inv_std, xc, mm);
        CG_LAUNCH_CHECK();
        return;
    }
    const int block = 64;  // a chain of 256 additions per thread: spread them over the SMs
    const int pgrid = static_cast<int>(ceil_div(items, block));
    center_partials_kernel<<<pgrid, block, 0, s>>>(x, n, d, nullptr, partial);
    CG_LAUNCH_CHECK();
    center_finalize_kernel<<<d, 256, 0, s>>>(partial, chunks, d, n, 0, mean, inv_std);
    CG_LAUNCH_CHECK();
    if (normalize) {
        center_partials_kernel<<<pgrid, block, 0, s>>>(x, n, d, mean, partial);
        CG_LAUNCH_CHECK();
        center_finalize_kernel<<<d, 256, 0, s>>>(partial, chunks, d, n, 1, mean, inv_std);
        CG_LAUNCH_CHECK();
    }
    if (xc == nullptr) return;
    const int ablock = d < 32 ? 256 : kApplyThreads;
    const int agrid = grid_for(n * d, ablock * kApplyLoads, 152 * 2048 / ablock);
    if (normalize) center_apply_kernel<true><<<agrid, ablock, 0, s>>>(x, n, d, mean, inv_std, xc, mm);
    else center_apply_kernel<false><<<agrid, ablock, 0, s>>>(x, n, d, mean, inv_std, xc, mm);
    CG_LAUNCH_CHECK();
}

void squared_norms(const float* xc, int64_t n, int d, float* norms, unsigned int* max_norm_bits,
                   cudaStream_t s) {
    norms_kernel<<<grid_for(n, 64, 152 * 32), 64, 0, s>>>(xc, n, d, norms, max_norm_bits);
    CG_LAUNCH_CHECK();
}

size_t center_partial_count(int64_t n, int d) { return static_cast<size_t>(ceil_div(n, kCenterChunk)) * d; }

}  // namespace culof_gb300
