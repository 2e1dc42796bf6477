// Sparse backward of the LOF scores with respect to the points (no reference
// counterpart: the reference computes scores only).
//
// With the neighbour sets N(i) held fixed (the k slots of a forward k-NN
// result, slot k-1 designating a k-th neighbour), the forward chain is
//   d2_ij   = |xc_i - xc_j|^2                         j in N(i)
//   kd2_j   = d2_{j, slot k-1}                         (squared k-distance)
//   reach_ij = sqrt(max(kd2_j, d2_ij))
//   lrd_i   = 1 / (sum_j reach_ij / k + 1e-10)         (lof.cu:32-46 of the reference)
//   score_i = sum_j lrd_j / (k lrd_i)                   (lof.cu:49-62)
// and xc = (x - mean) (* inv_std when normalising, population std, scale 1
// for zero-variance features). Given g = dL/dscore, the backward is evaluated
// in FP64 and is bit-reproducible: every sum over a point's reverse
// neighbours (the pairs (i, t) whose slot t names it) runs in a fixed order,
// taken from a stable radix sort of the slots by neighbour index (a
// transposed k-NN list), so no floating-point atomics are used.
//
// Subgradient conventions: max(kd2_j, d2_ij) sends the gradient to d2_ij when
// d2_ij > kd2_j and to kd2_j otherwise (ties go to the k-distance); a zero
// reach distance contributes no gradient (sqrt is not differentiable at 0).
#include "common.cuh"
#include "engine.cuh"
#include "fast.cuh"
#include "fp64.cuh"
#include "prep.cuh"

namespace culof_gb300 {

namespace {

__device__ __forceinline__ void flag_bad(int* status) { atomicExch(status, 2); }
// Indices used for addressing are clamped into [0, n): an invalid neighbour
// index (reported through the status word by bw_pair_kernel) gives a wrong
// gradient, never an out-of-range access.
__device__ __forceinline__ int64_t clampj(int32_t j, int64_t n) { return j < 0 ? 0 : (j >= n ? n - 1 : j); }

// The per-point sums below run one warp per point: lanes take the terms
// lane, lane + 32, ... in order and a fixed xor-shuffle tree adds the lanes'
// partials, so every sum has one fixed order and the gradient is
// bit-reproducible.
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ int64_t warp_id() { return (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; }
__device__ __forceinline__ int64_t warp_count() { return (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5; }

// d2[e] (e = t * n + i, the layout of the k-NN slots) in FP64 from the raw
// points: (x_i - x_j) * inv_std, the mean cancels. A thread per slot, features
// in order (blockIdx.y = t, neighbouring threads neighbouring points): two FP64
// instructions per feature and 32 slots (three when normalising). A warp per
// point with its lanes over the features needed ten per slot for its shuffle
// sum, and FP64 issues once per 64 cycles and scheduler: 626 us at n = 50,000,
// d = 32, k = 20.
__global__ void __launch_bounds__(256) bw_pair_kernel(const float* __restrict__ x, int64_t n, int d,
                                                      const int32_t* __restrict__ nbr, const double* __restrict__ inv,
                                                      int normalize, int aligned, double* __restrict__ d2,
                                                      int* __restrict__ status) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t e = static_cast<int64_t>(blockIdx.y) * n + i;
    const int32_t j = nbr[e];
    double s = 0.0;
    if (j < 0 || j >= n) {
        flag_bad(status);
    } else {
        const float* xi = x + i * d;
        const float* xj = x + static_cast<int64_t>(j) * d;
        if (aligned) {  // rows on 16-byte boundaries
            for (int f = 0; f < d; f += 4) {
                const float4 p = *reinterpret_cast<const float4*>(xi + f), q = *reinterpret_cast<const float4*>(xj + f);
                const float pv[4] = {p.x, p.y, p.z, p.w}, qv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    double u = __dsub_rn(widen(pv[c]), widen(qv[c]));
                    if (normalize) u = __dmul_rn(u, inv[f + c]);
                    s = __fma_rn(u, u, s);
                }
            }
        } else {
            for (int f = 0; f < d; ++f) {
                double u = __dsub_rn(widen(xi[f]), widen(xj[f]));
                if (normalize) u = __dmul_rn(u, inv[f]);
                s = __fma_rn(u, u, s);
            }
        }
    }
    d2[e] = s;
}

// Per point: reach distances of its slots, lrd. A CTA of 8 warps takes 32
// points (lane = point), the warps compute the slots side by side, 32 at a
// time, and warp 0 adds them in slot order.
__global__ void __launch_bounds__(256) bw_lrd_kernel(int64_t n, int k, const int32_t* __restrict__ nbr,
                                                     const double* __restrict__ d2, double* __restrict__ reach,
                                                     double* __restrict__ lrd) {
    __shared__ double term[32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t i = static_cast<int64_t>(blockIdx.x) * 32 + lane;
    double R = 0.0;
    for (int c0 = 0; c0 < k; c0 += 32) {
        const int c1 = k - c0 < 32 ? k - c0 : 32;
        for (int t = warp; t < c1; t += 8) {
            double r = 0.0;
            if (i < n) {
                const int64_t e = static_cast<int64_t>(c0 + t) * n + i;
                const int64_t j = clampj(nbr[e], n);
                r = __dsqrt_rn(fmax(d2[static_cast<int64_t>(k - 1) * n + j], d2[e]));
                reach[e] = r;
            }
            term[t][lane] = r;
        }
        __syncthreads();
        if (warp == 0)
            for (int t = 0; t < c1; ++t) R = __dadd_rn(R, term[t][lane]);
        __syncthreads();
    }
    if (warp == 0 && i < n) lrd[i] = __ddiv_rn(1.0, __dadd_rn(__ddiv_rn(R, static_cast<double>(k)), 1e-10));
}

// Per point (a thread): S_i = sum_j lrd_j, the score, and w_i = g_i / (k lrd_i),
// what the point adds to dL/dlrd of each of its neighbours.
__global__ void bw_score_kernel(int64_t n, int k, const int32_t* __restrict__ nbr, const double* __restrict__ lrd,
                                const double* __restrict__ g, double* __restrict__ S, double* __restrict__ w,
                                double* __restrict__ score) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = 0.0;
    for (int t0 = 0; t0 < k; t0 += 8) {  // eight gathers in flight
        double v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            v[j] = t0 + j < k ? lrd[clampj(nbr[static_cast<int64_t>(t0 + j) * n + i], n)] : 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (t0 + j < k) s = __dadd_rn(s, v[j]);
    }
    S[i] = s;
    const double kl = __dmul_rn(static_cast<double>(k), lrd[i]);
    w[i] = __ddiv_rn(g[i], kl);
    if (score) score[i] = __ddiv_rn(s, kl);
}

// Transposed slot list: keys and values for the stable sort, then each
// index's first place in the sorted keys (off[n] = total).
__global__ void bw_rev_init_kernel(int64_t n, int64_t total, const int32_t* __restrict__ nbr, unsigned* __restrict__ keys,
                                   unsigned* __restrict__ vals) {
    for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total;
         e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        keys[e] = static_cast<unsigned>(clampj(nbr[e], n));
        vals[e] = static_cast<unsigned>(e);
    }
}
__global__ void bw_rev_offsets_kernel(int64_t n, int64_t total, const unsigned* __restrict__ keys,
                                      unsigned* __restrict__ off) {
    for (int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p <= total;
         p += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        // indices past the previous key, up to this one (the end: up to n)
        int64_t j = p > 0 ? static_cast<int64_t>(keys[p - 1]) + 1 : 0;
        const int64_t last = p < total ? static_cast<int64_t>(keys[p]) : n;
        for (; j <= last; ++j) off[j] = static_cast<unsigned>(p);
    }
}

// Per point, over its reverse slots (i, t): the sum of w_i. (A warp per point,
// lanes over the reverse slots.)
__global__ void bw_gather_kernel(int64_t n, const double* __restrict__ w, const unsigned* __restrict__ off,
                                 const unsigned* __restrict__ rev, double* __restrict__ acc_out) {
    const int lane = threadIdx.x & 31;
    const unsigned n32 = static_cast<unsigned>(n);
    for (int64_t m = warp_id(); m < n; m += warp_count()) {
        double acc = 0.0;
        for (unsigned p = off[m] + lane; p < off[m + 1]; p += 32) acc = __dadd_rn(acc, w[rev[p] % n32]);
        acc = warp_sum(acc);
        if (lane == 0) acc_out[m] = acc;
    }
}

// Per point (a thread): dL/dlrd_m = -g_m S_m / (k lrd_m^2) + the reverse sum,
// and gR_m = -dL/dlrd_m lrd_m^2 / k, the gradient of its reach distances' sum.
__global__ void bw_point_kernel(int64_t n, int k, const double* __restrict__ g, const double* __restrict__ lrd,
                                const double* __restrict__ S, const double* __restrict__ acc, double* __restrict__ gR) {
    const int64_t m = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (m >= n) return;
    const double dk = static_cast<double>(k), lm = lrd[m], l2 = __dmul_rn(lm, lm);
    const double glrd = __dadd_rn(-__ddiv_rn(__dmul_rn(g[m], S[m]), __dmul_rn(dk, l2)), acc[m]);
    gR[m] = -__ddiv_rn(__dmul_rn(glrd, l2), dk);
}

// Per slot: the reach-distance gradient c = dL/dR_i / (2 reach), routed to
// d2_ij (gd2) or to kd2_j (gkd).
__global__ void bw_route_kernel(int64_t n, const int32_t* __restrict__ nbr, const double* __restrict__ d2,
                                const double* __restrict__ kd2, const double* __restrict__ reach, const double* __restrict__ gR,
                                double* __restrict__ gd2, double* __restrict__ gkd) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t e = static_cast<int64_t>(blockIdx.y) * n + i;
    const int64_t j = clampj(nbr[e], n);
    const double r = reach[e];
    const double c = r > 0.0 ? __ddiv_rn(gR[i], __dmul_rn(2.0, r)) : 0.0;
    const bool via_d2 = d2[e] > kd2[j];
    gd2[e] = via_d2 ? c : 0.0;
    gkd[e] = via_d2 ? 0.0 : c;
}

// Per point j: the k-distance gradient (sum over its reverse slots, fixed
// order) joins the gradient of its own slot k-1.
// (A warp per point.)
__global__ void bw_kd_kernel(int64_t n, int k, const unsigned* __restrict__ off, const unsigned* __restrict__ rev,
                             const double* __restrict__ gkd, double* __restrict__ gd2) {
    const int lane = threadIdx.x & 31;
    for (int64_t j = warp_id(); j < n; j += warp_count()) {
        double s = 0.0;
        for (unsigned p = off[j] + lane; p < off[j + 1]; p += 32) s = __dadd_rn(s, gkd[rev[p]]);
        s = warp_sum(s);
        if (lane == 0) {
            const int64_t e = static_cast<int64_t>(k - 1) * n + j;
            gd2[e] = __dadd_rn(gd2[e], s);
        }
    }
}

// Gradient with respect to the normalised coordinates, one warp per point:
// over its own and its reverse slots, the sum of gd2 (x_i - x_other), times
// 2 inv at the end. Lanes take the features; with d <= 16 the warp works on 32
// / DL slots side by side (DL = d rounded up to a power of two, at most 32) and
// adds the groups' sums in a fixed order. Two FP64 instructions per slot and
// lane, with the slot's scaling left to the end and the floats widened by
// integers (six before, 723 us at n = 50,000, d = 32, k = 20).
template <int DL>
__global__ void bw_gx_kernel(const float* __restrict__ x, int64_t n, int d, int k, const int32_t* __restrict__ nbr,
                             const double* __restrict__ inv, const double* __restrict__ gd2,
                             const unsigned* __restrict__ off, const unsigned* __restrict__ rev,
                             double* __restrict__ gxc) {
    constexpr int kGroups = 32 / DL;
    const int lane = threadIdx.x & 31, fl = lane % DL, grp = lane / DL;
    const unsigned n32 = static_cast<unsigned>(n);
    for (int64_t i = warp_id(); i < n; i += warp_count()) {
        const unsigned r0 = off[i], r1 = off[i + 1];
        for (int f0 = 0; f0 < d; f0 += DL) {
            const int f = f0 + fl;
            const bool on = f < d;
            const double xif = on ? widen(x[i * d + f]) : 0.0;
            double acc = 0.0;
#pragma unroll 4
            for (int t = grp; t < k; t += kGroups) {
                const int64_t e = static_cast<int64_t>(t) * n + i;
                const double g = gd2[e];
                if (on) acc = __fma_rn(g, __dsub_rn(xif, widen(x[clampj(nbr[e], n) * d + f])), acc);
            }
#pragma unroll 4
            for (unsigned p = r0 + grp; p < r1; p += kGroups) {
                const unsigned e = rev[p];
                const double g = gd2[e];
                if (on) acc = __fma_rn(g, __dsub_rn(xif, widen(x[static_cast<int64_t>(e % n32) * d + f])), acc);
            }
#pragma unroll
            for (int o = DL; o < 32; o <<= 1) acc = __dadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, o));
            if (on && grp == 0) gxc[i * d + f] = __dmul_rn(acc, __dmul_rn(2.0, inv[f]));
        }
    }
}

// Per (chunk of kCenterChunk rows, feature): partial sums of gxc and of
// gxc * xc; then per feature over the chunks. One block per chunk: warp w
// sums rows w, w + 8, ... of the chunk in order (lanes over features), and
// the 8 warps' partials are added in warp order.
constexpr int kColMaxD = 128;
__global__ void __launch_bounds__(256) bw_col_partials_kernel(const float* __restrict__ x, int64_t n, int d,
                                                              const double* __restrict__ mean,
                                                              const double* __restrict__ inv,
                                                              const double* __restrict__ gxc,
                                                              double* __restrict__ pa, double* __restrict__ pb) {
    __shared__ double sa[8][kColMaxD], sb[8][kColMaxD];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t chunks = ceil_div(n, kCenterChunk);
    for (int64_t c = blockIdx.x; c < chunks; c += gridDim.x) {
        const int64_t r1 = (c + 1) * kCenterChunk < n ? (c + 1) * kCenterChunk : n;
        for (int fb = 0; fb < d; fb += kColMaxD) {  // blocks of features that fit the shared arrays
            const int fe = d - fb < kColMaxD ? d - fb : kColMaxD;
            for (int f0 = 0; f0 < fe; f0 += 32) {
                const int fl = f0 + lane, f = fb + fl;
                if (fl < fe) {
                    double a = 0.0, b = 0.0;
                    const double mf = mean[f], vf = inv[f];
                    for (int64_t r = c * kCenterChunk + warp; r < r1; r += 8) {
                        const double g = gxc[r * d + f];
                        const double xc = __dmul_rn(__dsub_rn(static_cast<double>(x[r * d + f]), mf), vf);
                        a = __dadd_rn(a, g);
                        b = __fma_rn(g, xc, b);
                    }
                    sa[warp][fl] = a;
                    sb[warp][fl] = b;
                }
            }
            __syncthreads();
            for (int fl = threadIdx.x; fl < fe; fl += blockDim.x) {
                double a = 0.0, b = 0.0;
                for (int w = 0; w < 8; ++w) {
                    a = __dadd_rn(a, sa[w][fl]);
                    b = __dadd_rn(b, sb[w][fl]);
                }
                pa[c * d + fb + fl] = a;
                pb[c * d + fb + fl] = b;
            }
            __syncthreads();
        }
    }
}

// Per feature: column means A_f = mean(gxc), B_f = mean(gxc * xc) and whether
// the feature was scaled (normalising and std > 1e-12, the rule of the
// forward centring).
// (A warp per feature, lanes over the chunks; the variance partials are
// summed in chunk order, as the forward centring sums them.)
__global__ void bw_col_finalize_kernel(int64_t n, int d, int normalize, const double* __restrict__ pa,
                                       const double* __restrict__ pb, const double* __restrict__ var_partial,
                                       double* __restrict__ A, double* __restrict__ B, int* __restrict__ scaled) {
    const int lane = threadIdx.x & 31;
    const int64_t chunks = ceil_div(n, kCenterChunk);
    const double dn = static_cast<double>(n);
    for (int64_t f = warp_id(); f < d; f += warp_count()) {
        double a = 0.0, b = 0.0;
        for (int64_t c = lane; c < chunks; c += 32) {
            a = __dadd_rn(a, pa[c * d + f]);
            b = __dadd_rn(b, pb[c * d + f]);
        }
        a = warp_sum(a);
        b = warp_sum(b);
        if (lane == 0) {
            double v = 0.0;
            if (normalize)
                for (int64_t c = 0; c < chunks; ++c) v = __dadd_rn(v, var_partial[c * d + f]);
            A[f] = __ddiv_rn(a, dn);
            B[f] = __ddiv_rn(b, dn);
            scaled[f] = normalize && __dsqrt_rn(__ddiv_rn(v, dn)) > 1e-12;
        }
    }
}

// dL/dx: centring (and scaling) backward of the normalised-coordinate gradient.
__global__ void bw_apply_kernel(const float* __restrict__ x, int64_t n, int d, const double* __restrict__ mean,
                                const double* __restrict__ inv, const double* __restrict__ gxc,
                                const double* __restrict__ A, const double* __restrict__ B,
                                const int* __restrict__ scaled, double* __restrict__ gx) {
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < n * d;
         t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int f = static_cast<int>(t % d);
        const double g = __dsub_rn(gxc[t], A[f]);
        if (scaled[f]) {
            const double xc = __dmul_rn(__dsub_rn(static_cast<double>(x[t]), mean[f]), inv[f]);
            gx[t] = __dmul_rn(inv[f], __fma_rn(-xc, B[f], g));
        } else {
            gx[t] = g;
        }
    }
}

int grid_of(int64_t items) {
    int64_t g = ceil_div(items, 256);
    if (g > 152 * 16) g = 152 * 16;
    return static_cast<int>(g < 1 ? 1 : g);
}

}  // namespace

void Engine::lof_backward_device(const float* d_x, int64_t n, int d, int k, bool normalize, const int32_t* nbr_idx,
                                 const double* grad_scores, double* grad_x, double* scores_out) {
    validate_lof_args(d_x, n, d, k);
    if (!nbr_idx || !grad_scores || !grad_x) throw Error(kInvalidArgument, "device pointers must not be null");
    if (n * static_cast<int64_t>(k) > 0x7FFFFFFFll)
        throw Error(kInvalidArgument, "the backward takes n_points * k < 2^31 neighbour slots");
    CG_CUDA(cudaSetDevice(device_));
    cudaStream_t s = stream_;
    const int64_t total = n * k;
    const size_t nk = static_cast<size_t>(total);
    // statistics of the forward centring (same kernels, same order; no points)
    double* partial = partial_.as<double>(center_partial_count(n, d));
    double* mean = mean_.as<double>(d);
    double* inv = inv_std_.as<double>(d);
    CG_CUDA(cudaMemsetAsync(status_ptr(), 0, sizeof(int), s));
    center(d_x, n, d, normalize, nullptr, partial, mean, inv, s);

    // workspace: FP64 slot arrays, per-point arrays, the transposed slot list
    const size_t chunks_d = center_partial_count(n, d);
    char* w = static_cast<char*>(bw_.get(sizeof(double) * (4 * nk + 5 * static_cast<size_t>(n) +
                                                          2 * chunks_d + 2 * static_cast<size_t>(d) +
                                                          static_cast<size_t>(n) * d) +
                                         sizeof(unsigned) * (4 * nk + static_cast<size_t>(n) + 1 +
                                                             sort_pairs_counts(total)) +
                                         sizeof(int) * static_cast<size_t>(d) + 32 * 256));
    auto take = [&](size_t bytes) {
        char* p = w;
        w += (bytes + 255) & ~static_cast<size_t>(255);
        return p;
    };
    double* d2 = reinterpret_cast<double*>(take(sizeof(double) * nk));
    double* reach = reinterpret_cast<double*>(take(sizeof(double) * nk));
    double* gd2 = reinterpret_cast<double*>(take(sizeof(double) * nk));
    double* gkd = reinterpret_cast<double*>(take(sizeof(double) * nk));
    double* lrd = reinterpret_cast<double*>(take(sizeof(double) * n));
    double* S = reinterpret_cast<double*>(take(sizeof(double) * n));
    double* w_pt = reinterpret_cast<double*>(take(sizeof(double) * n));
    double* gR = reinterpret_cast<double*>(take(sizeof(double) * n));
    double* gxc = reinterpret_cast<double*>(take(sizeof(double) * n * d));
    double* pa = reinterpret_cast<double*>(take(sizeof(double) * chunks_d));
    double* pb = reinterpret_cast<double*>(take(sizeof(double) * chunks_d));
    double* A = reinterpret_cast<double*>(take(sizeof(double) * d));
    double* B = reinterpret_cast<double*>(take(sizeof(double) * d));
    int* scaled = reinterpret_cast<int*>(take(sizeof(int) * d));
    unsigned* keys = reinterpret_cast<unsigned*>(take(sizeof(unsigned) * nk));
    unsigned* vals = reinterpret_cast<unsigned*>(take(sizeof(unsigned) * nk));
    unsigned* keys2 = reinterpret_cast<unsigned*>(take(sizeof(unsigned) * nk));
    unsigned* vals2 = reinterpret_cast<unsigned*>(take(sizeof(unsigned) * nk));
    unsigned* off = reinterpret_cast<unsigned*>(take(sizeof(unsigned) * (n + 1)));
    unsigned* counts = reinterpret_cast<unsigned*>(take(sizeof(unsigned) * sort_pairs_counts(total)));
    int* status = status_ptr();
    double* score = scores_out;
    const int aligned = (d & 3) == 0 && (reinterpret_cast<uintptr_t>(d_x) & 15) == 0 ? 1 : 0;

    const dim3 slots(static_cast<unsigned>(ceil_div(n, 256)), static_cast<unsigned>(k));
    const unsigned points = static_cast<unsigned>(ceil_div(n, 256));
    // (blockIdx.y takes at most 65535 slots)
    for (int t0 = 0; t0 < k; t0 += 65535) {
        const dim3 g(slots.x, static_cast<unsigned>(k - t0 < 65535 ? k - t0 : 65535));
        bw_pair_kernel<<<g, 256, 0, s>>>(d_x, n, d, nbr_idx + static_cast<int64_t>(t0) * n, inv, normalize ? 1 : 0,
                                         aligned, d2 + static_cast<int64_t>(t0) * n, status);
        CG_LAUNCH_CHECK();
    }
    bw_lrd_kernel<<<static_cast<unsigned>(ceil_div(n, 32)), 256, 0, s>>>(n, k, nbr_idx, d2, reach, lrd);
    CG_LAUNCH_CHECK();
    bw_score_kernel<<<points, 256, 0, s>>>(n, k, nbr_idx, lrd, grad_scores, S, w_pt, score);
    CG_LAUNCH_CHECK();
    // transposed slots: in (t, i) enumeration order within each index (stable
    // sort)
    bw_rev_init_kernel<<<grid_of(total), 256, 0, s>>>(n, total, nbr_idx, keys, vals);
    CG_LAUNCH_CHECK();
    int bits = 8;
    while (bits < 32 && (static_cast<int64_t>(1) << bits) < n) bits += 8;
    unsigned* rev = nullptr;
    const unsigned* sorted = sort_pairs_stable(keys, vals, keys2, vals2, total, bits, counts, s, &rev);
    bw_rev_offsets_kernel<<<grid_of(total + 1), 256, 0, s>>>(n, total, sorted, off);
    CG_LAUNCH_CHECK();

    bw_gather_kernel<<<grid_of(n * 32), 256, 0, s>>>(n, w_pt, off, rev, gR);
    CG_LAUNCH_CHECK();
    bw_point_kernel<<<points, 256, 0, s>>>(n, k, grad_scores, lrd, S, gR, gR);
    CG_LAUNCH_CHECK();
    for (int t0 = 0; t0 < k; t0 += 65535) {
        const dim3 g(slots.x, static_cast<unsigned>(k - t0 < 65535 ? k - t0 : 65535));
        const int64_t at = static_cast<int64_t>(t0) * n;
        bw_route_kernel<<<g, 256, 0, s>>>(n, nbr_idx + at, d2 + at, d2 + static_cast<int64_t>(k - 1) * n, reach + at, gR,
                                          gd2 + at, gkd + at);
        CG_LAUNCH_CHECK();
    }
    bw_kd_kernel<<<grid_of(n * 32), 256, 0, s>>>(n, k, off, rev, gkd, gd2);
    CG_LAUNCH_CHECK();
    const auto gx = d <= 1 ? bw_gx_kernel<1> : d <= 2 ? bw_gx_kernel<2> : d <= 4 ? bw_gx_kernel<4> : d <= 8
                        ? bw_gx_kernel<8> : d <= 16 ? bw_gx_kernel<16> : bw_gx_kernel<32>;
    gx<<<grid_of(n * 32), 256, 0, s>>>(d_x, n, d, k, nbr_idx, inv, gd2, off, rev, gxc);
    CG_LAUNCH_CHECK();
    // the centring statistics' partials of (x - mean)^2 are still in `partial`
    // when normalising (the second pass of center())
    const int64_t col_chunks = ceil_div(n, kCenterChunk);
    bw_col_partials_kernel<<<static_cast<int>(col_chunks < 152 * 8 ? col_chunks : 152 * 8), 256, 0, s>>>(
        d_x, n, d, mean, inv, gxc, pa, pb);
    CG_LAUNCH_CHECK();
    bw_col_finalize_kernel<<<static_cast<int>(ceil_div(static_cast<int64_t>(d) * 32, 256)), 256, 0, s>>>(
        n, d, normalize ? 1 : 0, pa, pb, partial, A, B, scaled);
    CG_LAUNCH_CHECK();
    bw_apply_kernel<<<grid_of(n * d), 256, 0, s>>>(d_x, n, d, mean, inv, gxc, A, B, scaled, grad_x);
    CG_LAUNCH_CHECK();
}

}  // namespace culof_gb300
