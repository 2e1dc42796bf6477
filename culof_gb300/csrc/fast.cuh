// Fused distance + filtered exact select (the fast k-NN path).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace culof_gb300 {

// True when the fast path handles (n, d, k).
bool fast_path_supported(int64_t n, int d, int k);

// Small inputs (direct.cu): the k nearest of rows [row_begin, row_end) among
// all n points by two passes over the columns.
bool direct_supported(int64_t n, int d, int k);
void direct_knn(const float* xc, int64_t n, int d, int64_t row_begin, int64_t row_end, int k, int32_t* idx, float* d2,
                float* kd, cudaStream_t s);

// The wide-point variant (8 < d <= 128), wide.cu.
int wide_dims_padded(int d);
size_t wide_tiles_floats(int d, int nt);
void wide_build_tiles(const float* xc, const float* norms, int64_t n, int d, const unsigned* perm, int nt,
                      float* tiles, cudaStream_t s);
// Row tiles [t0, t0 + mt) of the nt (every call covers a block of row tiles;
// the whole problem is t0 = 0, mt = nt).
void wide_seed(const float* tiles, int nt, int t0, int mt, int d, int k, uint64_t* seed_keys,
               unsigned long long* kth_shared, cudaStream_t s);
void wide_sweep(const float* tiles, int nt, int t0, int mt, int nsplit, int d, int k, const unsigned* maxn,
                unsigned long long* kth_shared, uint64_t* partial, cudaStream_t s);

// Stable LSD radix sort of (key, value) pairs on the low key_bits bits of the
// keys (8 bits per pass); keys_tmp / vals_tmp are scratch of n entries and
// counts holds sort_pairs_counts(n) entries. Returns the buffer holding the
// sorted keys (keys or keys_tmp) and sets *vals_out to the sorted values.
size_t sort_pairs_counts(int64_t n);
unsigned* sort_pairs_stable(unsigned* keys, unsigned* vals, unsigned* keys_tmp, unsigned* vals_tmp, int64_t n,
                            int key_bits, unsigned* counts, cudaStream_t s, unsigned** vals_out);

// Shared by the FP32 and tensor-core sweeps (fast.cu).
int choose_splits(int nt, int sms);
// Merges the rows at sorted positions [pos0, pos1).
void launch_merge(const uint64_t* seed_keys, const uint64_t* partial, const unsigned* perm, int64_t n, int nt,
                  int64_t pos0, int64_t pos1, int nsplit, int k, int32_t* idx, float* d2, float* kd, cudaStream_t s);

// The tensor-core variant (tc_sweep.cu). Sorted-order arrays of one call:
// xh f16 operand rows [padded][Kp], xr FP32 coordinates [padded][dr], cn
// norms, ix original indices, scale a device record of the f16 scaling.
// split: each coordinate x (scaled) is carried as two f16 values, hi =
// f16(x) and lo = f16(x - hi); the row operand holds [hi, lo, hi] and the
// column operand [hi, hi, lo] (d values each), so their product sums
// hi.hi + lo.hi + hi.lo, the Gram value to about 2^-22 relative instead of
// 2^-11 (used when 3d <= 128); xb is then the column-arrangement array
// (otherwise xb == xh). ksteps: the K steps of 16 the MMA issues.
struct TcBuffers {
    void* xh;
    void* xb;
    float* xr;
    float* cn;
    unsigned* ix;
    void* scale;
    float* rn;  // residual norms of the operand rows (single operands)
    int Kp;
    int dr;
    int split;
    int ksteps;
};
size_t tc_buffer_bytes(int64_t padded, int d);
// scale: the call's scale record (tc_scale.cuh).
TcBuffers tc_prepare(void* buf, const float* xc, const float* norms, int64_t n, int d, const unsigned* perm, int nt,
                     void* scale, cudaStream_t s);
int tc_max_splits();
constexpr int kMaxTensorD = 256;
constexpr int kTcSplitD = 42;  // split operands up to here (3d <= 128)
// True when the tensor path handles (n, d, k) (AUTO only above d = 128).
bool tensor_supported(int64_t n, int d, int k);
// Workspace of the per-row lists of one sweep launch batch.
size_t tc_list_bytes(int nt, int nsplit);
// The sweep and the rows' final results (k best of the seed's lists and the
// sweep's, in the reference's slot order). qs: the seed window (spiral
// positions 0..qs-1 are the seed's; 0: no seed, kth_seed and seed_keys null);
// plist / pcount (nullable): per row tile,
// the column tiles to visit in order (the small-d prune lists); without them
// every tile past the window is visited. lost_rows / lost_count: the original
// indices of the rows that it leaves to lost_rows().
void tc_sweep(const TcBuffers& b, int64_t n, int nt, int t0, int mt, int nsplit, int d, int k, const unsigned* maxn,
              const unsigned long long* kth_seed, const uint64_t* seed_keys, uint64_t* lists, int* status,
              int32_t* nbr_idx, float* nbr_d2, float* kdist2, cudaStream_t s, int qs, int32_t* lost_rows, int* lost_count,
              const uint2* plist = nullptr, const int* pcount = nullptr);

// The exact k nearest of the points rows[0 .. *count) (lost_rows.cu; both on the
// device, at most max_rows) among all n points, d <= kMaxTensorD. scratch:
// lost_rows_bytes() bytes; arrived: kLostGroups words, zero.
constexpr int kLostGroups = 512;
size_t lost_rows_bytes(int64_t n, int64_t max_rows, int k, int sms);
void lost_rows(const float* xc, int64_t n, int d, int k, const int32_t* rows, const int* count, void* scratch,
               int* arrived, int sms, int32_t* idx, float* d2, float* kd, cudaStream_t s);

}  // namespace culof_gb300
