// Column tiles of the small-d path (d <= 8) and the pieces its kernels share.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "sweep_common.cuh"

namespace culof_gb300 {
namespace small {

using namespace sweep;

constexpr int kMaxDP = 8;
constexpr int kHalf = 64;     // columns the sweep tests and evaluates together (two per lane)
constexpr int kHalves = kCT / kHalf;
constexpr int kQuarter = 32;  // columns the isolated rows' pass tests and evaluates together
constexpr int kQuarters = kCT / kQuarter;

// Column tile t (kCT consecutive sorted points), in global memory and, when
// staged, in shared memory (floats):
//   coords: dimension-major, [f][c] = coordinate f of column c (NaN in
//           dimension 0 of padding columns), so that 32 columns, or 32 column
//           pairs, are DP coalesced (bank-conflict-free) warp reads
//   index : kCT uint32 original indices (kNoIndex for padding)
//   boxes : per half, [f][2] = lower bound and negated upper bound of
//           dimension f over its valid columns (both +inf when it has none)
__host__ __device__ constexpr int tile_index_off(int dp) { return dp * kCT; }
__host__ __device__ constexpr int tile_box_off(int dp) { return tile_index_off(dp) + kCT; }
__host__ __device__ constexpr int tile_floats(int dp) { return tile_box_off(dp) + kHalves * 2 * dp; }
__host__ __device__ constexpr int tile_bytes(int dp) { return tile_floats(dp) * 4; }

// Coordinate f of column c within a tile.
template <int DP>
__device__ __forceinline__ float tile_coord(const float* tile, int c, int f) {
    return tile[f * kCT + c];
}

// Pruning margin: the float32 direct-difference distance D of two points at
// real squared distance T >= LB satisfies D >= T (1 - (d + 2) 2^-24), so a box
// whose rounded-down gap times the factor exceeds a row's k-th distance holds
// no candidate for it: 1 - 2^-20 for d <= 8, 1 - 2^-17 for d <= 64.
template <int DP>
__device__ __forceinline__ constexpr float prune_shrink() {
    return DP <= 8 ? 0.99999904632568359375f : 0.9999923706054688f;
}

constexpr int kSegTiles = 1024;  // column tiles a CTA lists at a time

// DP (padded dimensions) of d <= 8 points.
inline int padded_dims(int d) { return d <= 2 ? 2 : d <= 4 ? 4 : d <= 6 ? 6 : 8; }

}  // namespace small

// Refines the Morton order perm of the points (n, d <= 8) in place.
void small_refine_order(const float* xc, int64_t n, int d, unsigned* perm, cudaStream_t s);

// Tiles [nt], their boxes ([nt][2 dp] floats: lower bounds, upper bounds) and
// the 32-byte bf16 quarter records that the isolated rows' pass tests.
size_t small_tiles_floats(int dp, int nt);
void small_build_tiles(const float* xc, int64_t n, int d, const unsigned* perm, int nt, float* tiles, float* boxes,
                       void* qbox, cudaStream_t s);

// Whether rows may leave the sweep for a pass of their own, if that is wanted.
bool small_defers(bool wanted, int nt, int mt);
// Workspace of the row tiles' order and, with defer, of the rows that leave.
size_t small_iso_bytes(int mt, int k, bool defer);
// Exact k-NN of the rows of row tiles [t0, t0 + mt), written in the
// reference's slot order. evaluated (nullable) counts (row, half) pairs
// past the seed window; defer as small_defers() has it, iso small_iso_bytes(mt,
// k, defer) bytes, *iso_count zero; segment (at most
// kSegTiles) column tiles are listed at a time.
void small_knn(const float* tiles, const float* boxes, const void* qbox, const unsigned* perm, int64_t n, int d, int nt,
               int t0, int mt, int k, int sms, bool defer, int segment, void* iso, int* iso_count, int32_t* nbr_idx, float* nbr_d2,
               float* kdist2, int* status, unsigned long long* evaluated, cudaStream_t s);

}  // namespace culof_gb300
