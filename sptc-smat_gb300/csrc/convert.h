// convert.h — B operand packing (convert.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace smat {

// 128-column tiles per k-block of the packed layout (padded to an even count
// when there is more than one).
int64_t packed_b_tiles(int64_t N);

// Bytes of one packed copy of a K x N operand.
size_t packed_b_bytes(int64_t K, int64_t N);

// B is packed in units of kPackUnitBlocks k-blocks of one 64-column half tile;
// each unit has a byte that says whether it holds an infinite or NaN value, and
// a word per 32 columns with a bit for each column that does. The bytes of a half
// (pack_flag_stride of them, zeros after the last unit) lie one after the other,
// behind those of all halves the words (two per unit, half by half).
constexpr int kPackUnitBlocks = 8;
__host__ __device__ constexpr int64_t pack_units_k(int64_t K) {
  return ((K + 15) / 16 + kPackUnitBlocks - 1) / kPackUnitBlocks;
}
__host__ __device__ constexpr int64_t pack_halves(int64_t N) { return (N + 63) / 64; }
__host__ __device__ constexpr int64_t pack_flag_stride(int64_t K) { return (pack_units_k(K) + 15) / 16 * 16; }
__host__ __device__ constexpr int64_t pack_cols_offset(int64_t K, int64_t N) {
  return pack_halves(N) * pack_flag_stride(K);
}
size_t pack_flag_bytes(int64_t K, int64_t N);  // the bytes and the words

// Packs B into 4 KB tiles of 16 rows x 128 columns ordered [128-column
// tile][k-block] (layout: convert.cu), so that the tiles of consecutive
// k-blocks of one column tile are contiguous.
// in_dtype: 0 F32, 1 F16, 2 BF16; layout: 0 row-major (k*ldi + n), 1
// column-major (k + n*ldi); out_mode: 0 FP16, 1 BF16, 2 hi+lo BF16 (8 KB per
// tile, twice packed_b_bytes).
// kperm (device, optional): row kperm[k] of `in` feeds packed row k (a
// column permutation of A; gathered with scalar loads).
// flags: pack_flag_bytes() bytes; the units' bytes and words are written.
// counters (optional): kLaunchCounters integers set to zero, for the SpMM
// launched behind.
constexpr int kLaunchCounters = 4;
cudaError_t pack_b(const void* in, int in_dtype, int layout, int64_t ldi, int out_mode, uint8_t* out,
                   int64_t K, int64_t N, const int32_t* kperm, uint8_t* flags, int32_t* counters, cudaStream_t s);

// The 2:4 path's copy of B: 8 KB tiles ordered [128-column tile][window],
// window w = k-blocks 2w and 2w+1 (32 k-values; the second half zero past
// K), 128 rows of 64 bytes in the 64-byte swizzle, made from the packed
// FP16/BF16 tiles of pack_b.
size_t packed_b64_bytes(int64_t K, int64_t N);
cudaError_t pack_b_sw64(const uint8_t* packed, int64_t K, int64_t N, uint8_t* out, cudaStream_t s);

// One B operand of a grouped pack: `in` (in_dtype, layout, ldi, K x N) into
// `out` (out_mode as pack_b), covering the global units [begin, begin +
// pack_halves(N) * pack_units_k(K)).
struct PackJob {
  const void* in;
  uint8_t* out;
  const int32_t* kperm;  // column permutation of A (device), or null
  uint8_t* flags;
  uint32_t* cols;        // flags + pack_cols_offset
  int64_t ldi, K, N, begin;
  int32_t in_dtype, layout, out_mode, pad;
};

// Packs every job in one launch (jobs sorted by begin, in device memory).
// any_col / any_split: whether a job is column-major / of the split form.
// counters: n_counters integers set to zero, for the SpMMs launched behind.
cudaError_t pack_b_grouped(const PackJob* d_jobs, int njobs, int64_t total_units, bool any_col, bool any_split,
                           int num_sms, int32_t* counters, int n_counters, cudaStream_t s);

}  // namespace smat
