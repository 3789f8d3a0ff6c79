// convert.cu — packs the dense operand B for the tensor-core SpMM.
//
// B arrives as FP32, FP16 or BF16, row-major (k*ld + n) or column-major
// (k + n*ld, the reference's layout, src/cuda_hgemm/src/mma/mmaOBT.cu:75).
// Packed tile (t, kb) holds rows k = 16*kb .. 16*kb+15 and columns
// n = 128*t .. 128*t+127 as two halves of 64 columns, each 16 rows (one per k)
// of 64 16-bit values (128 bytes): the MMA reads its 128 x 16 operand with N
// contiguous (MN-major, 128-byte swizzle: 16-byte chunk c of row k lies at
// chunk c ^ (k & 7)). Tiles are ordered [t][kb]. So an aligned tile is one
// 4 KB copy, and a single row of B is two 128-byte pieces that a gathered tile
// can bring to any row of its own by undoing one swizzle and applying the
// other. The split form writes hi = bf16(b) and lo = bf16(b - hi), [hi | lo]
// inside each half.
//
// K is zero-padded to 16 and N to 64 columns; a half without a column below N
// is neither written nor read.
//
// A block packs one UNIT: 8 k-blocks of one half. It also says, in the unit's
// byte of `flags`, whether any packed value is infinite or NaN, and in the unit's
// two words of `cols` in which columns: the SpMM then restores what a block's
// stored zeros make of such a value (spmm_tc.cu).
//
// What bounds it: DRAM and L2 traffic of a copy (268 MB of FP32 in and 134 MB out
// in 62 us, 6.5 TB/s of the 6.7 a copy reaches; six blocks an SM, 64^3 stencil
// 183 -> 180 us against four). Row-major B needs no
// transposition in this layout (a thread moves eight neighbouring columns);
// column-major B goes through shared memory, 128 x 64 values at a time.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "convert.h"
#include "spmm_tc.h"
#include "tc_ptx.cuh"

namespace smat {
namespace dev {

enum : int { OUT_F16 = 0, OUT_BF16 = 1, OUT_SPLIT = 2 };
constexpr int kPackThreads = 256;
constexpr int kUnitK = 16 * kPackUnitBlocks;  // rows of B per unit
constexpr int kStride = 33;                   // words per k of the transposition buffer (64 values and one word)

template <typename T>
__device__ __forceinline__ float load_f(const T* p);
template <>
__device__ __forceinline__ float load_f<float>(const float* p) {
  return __ldg(p);
}
template <>
__device__ __forceinline__ float load_f<__half>(const __half* p) {
  return __half2float(__ldg(p));
}
template <>
__device__ __forceinline__ float load_f<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(__ldg(p));
}

// Element i of a 16-byte vector of T, as float.
template <typename T>
__device__ __forceinline__ float vec_elem(const uint4& v, int i);
template <>
__device__ __forceinline__ float vec_elem<float>(const uint4& v, int i) {
  return __uint_as_float(reinterpret_cast<const uint32_t*>(&v)[i]);
}
template <>
__device__ __forceinline__ float vec_elem<__half>(const uint4& v, int i) {
  return __half2float(__ushort_as_half(reinterpret_cast<const uint16_t*>(&v)[i]));
}
template <>
__device__ __forceinline__ float vec_elem<__nv_bfloat16>(const uint4& v, int i) {
  return __bfloat162float(__ushort_as_bfloat16(reinterpret_cast<const uint16_t*>(&v)[i]));
}

// The packed hi (and, split form, lo) bits of x.
template <int OUT>
__device__ __forceinline__ uint32_t hi_bits(float x) {
  return OUT == OUT_F16 ? __half_as_ushort(__float2half_rn(x)) : __bfloat16_as_ushort(__float2bfloat16_rn(x));
}
__device__ __forceinline__ uint32_t lo_bits(float x, uint32_t hi) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(x - __bfloat162float(__ushort_as_bfloat16((uint16_t)hi))));
}
// Nonzero when either 16-bit half of w is infinite or NaN.
template <int OUT>
__device__ __forceinline__ uint32_t nonfinite2(uint32_t w) {
  constexpr uint32_t E = OUT == OUT_F16 ? 0x7c00u : 0x7f80u;
  return ((w & E) == E || ((w >> 16) & E) == E) ? 1u : 0u;
}

// Eight columns n .. n + 7 of row ks (n a multiple of 8) as packed pairs.
template <typename T, int OUT>
__device__ __forceinline__ void row_chunk(const T* __restrict__ in, int64_t ldi, int64_t N, int64_t ks, int64_t n,
                                          bool vec, bool inside, uint32_t hi[4], uint32_t lo[4]) {
  float x[8];
  if (inside && vec && n + 8 <= N) {
    constexpr int V = 16 / sizeof(T);
    const uint4* p = reinterpret_cast<const uint4*>(in + ks * ldi + n);
    uint4 v[8 / V];
#pragma unroll
    for (int q = 0; q < 8 / V; q++) v[q] = __ldg(p + q);
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = vec_elem<T>(v[i / V], i % V);
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = (inside && n + i < N) ? load_f<T>(in + ks * ldi + n + i) : 0.0f;
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t a = hi_bits<OUT>(x[2 * i]), b = hi_bits<OUT>(x[2 * i + 1]);
    hi[i] = a | (b << 16);
    if (OUT == OUT_SPLIT) lo[i] = lo_bits(x[2 * i], a) | (lo_bits(x[2 * i + 1], b) << 16);
  }
}

// One unit: k-blocks 8 * kc .. 8 * kc + 7 of half hx (columns 64 * hx ..).
// `tr`: kUnitK * kStride words of shared memory per operand (column-major).
// Returns, to every thread, whether the unit holds infinite or NaN values.
template <typename T, int OUT>
__device__ __forceinline__ bool pack_unit(const T* __restrict__ in, int layout, int64_t ldi, uint8_t* __restrict__ out,
                                          int64_t K, int64_t N, int64_t kc, int64_t hx,
                                          const int32_t* __restrict__ kperm, uint8_t* __restrict__ flags,
                                          uint32_t* tr) {
  constexpr int NOPS = OUT == OUT_SPLIT ? 2 : 1;
  const int tid = threadIdx.x;
  const int64_t kbs = (K + 15) / 16, n0 = hx * 64, k0 = kc * kUnitK;
  uint8_t* const half = out + ((hx >> 1) * kbs + kc * kPackUnitBlocks) * (4096 * NOPS) + (hx & 1) * (2048 * NOPS);
  uint32_t bad = 0;
  if (layout == 0) {
    // row-major: chunk q of the unit = row q / 8, columns 8 * (q % 8)
    const bool vec = ((reinterpret_cast<uintptr_t>(in) | (uint64_t)ldi * sizeof(T)) & 15) == 0;
#pragma unroll
    for (int it = 0; it < kUnitK * 8 / kPackThreads; it++) {
      const int q = tid + it * kPackThreads, kr = q >> 3, c = q & 7;
      const int64_t k = k0 + kr;
      if ((k >> 4) < kbs) {
        const bool inside = k < K;
        const int64_t ks = (inside && kperm) ? (int64_t)kperm[k] : k;  // row of B feeding permuted column k
        uint32_t hi[4], lo[4];
        row_chunk<T, OUT>(in, ldi, N, ks, n0 + 8 * c, vec, inside, hi, lo);
        uint8_t* dst = half + (kr >> 4) * (4096 * NOPS) + (kr & 15) * 128 + ((c ^ (kr & 7)) << 4);
        *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        if (OUT == OUT_SPLIT) *reinterpret_cast<uint4*>(dst + 2048) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
#pragma unroll
        for (int i = 0; i < 4; i++) bad |= nonfinite2<OUT>(hi[i]);
      }
    }
  } else {
    // column-major: a thread reads V consecutive k of columns n and n + 1 and
    // leaves them as column pairs in tr[k][pair]; then the chunks are written
    // as above
    constexpr int V = 16 / sizeof(T), KV = kUnitK / V;
    const bool vec = !kperm && ((reinterpret_cast<uintptr_t>(in) | (uint64_t)ldi * sizeof(T)) & 15) == 0;
#pragma unroll 2
    for (int q = tid; q < KV * 32; q += kPackThreads) {
      // 8 vectors along k (128 contiguous bytes) x 4 column pairs per warp
      const int w = q >> 5, l = q & 31;
      const int kv = (w % (KV / 8)) * 8 + (l & 7), np = (w / (KV / 8)) * 4 + (l >> 3);
      const int64_t k = k0 + kv * V, n = n0 + 2 * np;
      float x[2][V];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const T* p = in + (n + e) * ldi;
        if (vec && n + e < N && k + V <= K) {
          const uint4 v = __ldg(reinterpret_cast<const uint4*>(p + k));
#pragma unroll
          for (int i = 0; i < V; i++) x[e][i] = vec_elem<T>(v, i);
        } else {
#pragma unroll
          for (int i = 0; i < V; i++)
            x[e][i] = (n + e < N && k + i < K) ? load_f<T>(p + (kperm ? (int64_t)kperm[k + i] : k + i)) : 0.0f;
        }
      }
#pragma unroll
      for (int i = 0; i < V; i++) {
        const uint32_t a = hi_bits<OUT>(x[0][i]), b = hi_bits<OUT>(x[1][i]);
        tr[(kv * V + i) * kStride + np] = a | (b << 16);
        bad |= nonfinite2<OUT>(a | (b << 16));
        if (OUT == OUT_SPLIT)
          tr[(kUnitK + kv * V + i) * kStride + np] = lo_bits(x[0][i], a) | (lo_bits(x[1][i], b) << 16);
      }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kUnitK * 8 / kPackThreads; it++) {
      const int q = tid + it * kPackThreads, kr = q >> 3, c = q & 7;
      if (((k0 + kr) >> 4) >= kbs) continue;
      uint8_t* dst = half + (kr >> 4) * (4096 * NOPS) + (kr & 15) * 128 + ((c ^ (kr & 7)) << 4);
#pragma unroll
      for (int o = 0; o < NOPS; o++) {
        const uint32_t* s = tr + (o * kUnitK + kr) * kStride + 4 * c;
        *reinterpret_cast<uint4*>(dst + o * 2048) = make_uint4(s[0], s[1], s[2], s[3]);
      }
    }
  }
  const int any = __syncthreads_or((int)bad);
  const int64_t fs = pack_flag_stride(K);
  if (tid == 0) flags[hx * fs + kc] = any ? 1 : 0;
  if (kc == pack_units_k(K) - 1 && tid > 0 && kc + tid < fs) flags[hx * fs + kc + tid] = 0;  // the unused bytes
  return any != 0;
}

// The unit's words of `cols`: the columns in which it holds such values. A thread
// looks at the chunks it wrote, all of columns 8 * (tid % 8) .. (A call of its own:
// packing keeps its registers.)
__device__ __noinline__ void unit_columns(const uint8_t* out, int out_mode, int64_t K, int64_t kc, int64_t hx,
                                             uint32_t* cols) {
  __shared__ uint32_t bits[2];
  const int tid = threadIdx.x;
  const uint32_t E = out_mode == OUT_F16 ? 0x7c00u : 0x7f80u;
  const int nops = out_mode == OUT_SPLIT ? 2 : 1;
  const int64_t kbs = (K + 15) / 16;
  const uint8_t* const half = out + ((hx >> 1) * kbs + kc * kPackUnitBlocks) * (4096 * nops) + (hx & 1) * (2048 * nops);
  if (tid < 2) bits[tid] = 0;
  __syncthreads();
  uint32_t m = 0;
#pragma unroll 1
  for (int kr = tid >> 3; kr < kUnitK && kc * kPackUnitBlocks + (kr >> 4) < kbs; kr += kPackThreads / 8) {
    const uint32_t* const w = reinterpret_cast<const uint32_t*>(half + (kr >> 4) * (4096 * nops) + (kr & 15) * 128 +
                                                                (((tid & 7) ^ (kr & 7)) << 4));
#pragma unroll
    for (int i = 0; i < 4; i++)
      m |= ((w[i] & E) == E ? 1u : 0u) << (2 * i) | (((w[i] >> 16) & E) == E ? 2u : 0u) << (2 * i);
  }
  if (m) atomicOr(&bits[(tid & 7) >> 2], m << (8 * (tid & 3)));
  __syncthreads();
  if (tid < 2) cols[(hx * pack_units_k(K) + kc) * 2 + tid] = bits[tid];
}

template <typename T, int OUT>
__global__ void __launch_bounds__(kPackThreads, 6)
    pack_b_kernel(const T* __restrict__ in, int layout, int64_t ldi, uint8_t* __restrict__ out, int64_t K, int64_t N,
                  const int32_t* __restrict__ kperm, uint8_t* __restrict__ flags, uint32_t* __restrict__ cols,
                  int32_t* __restrict__ counters) {
  extern __shared__ uint32_t tr[];
  grid_release();  // the SpMM launched behind may be set up
  if (counters && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < kLaunchCounters) counters[threadIdx.x] = 0;
  const bool any = pack_unit<T, OUT>(in, layout, ldi, out, K, N, blockIdx.x, blockIdx.y, kperm, flags, tr);
  if (threadIdx.x < 2) cols[((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * 2 + threadIdx.x] = 0;
  if (any) unit_columns(out, OUT, K, blockIdx.x, blockIdx.y, cols);
}

// Many B operands in one launch: block g packs unit g of the list of all
// jobs' units (jobs sorted by their first unit).
__global__ void __launch_bounds__(kPackThreads, 6)
    pack_b_grouped_kernel(const PackJob* __restrict__ jobs, int njobs, int64_t total, int32_t* __restrict__ counters,
                          int n_counters) {
  extern __shared__ uint32_t tr[];
  grid_release();
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < n_counters; i += kPackThreads) counters[i] = 0;
  for (int64_t g = blockIdx.x; g < total; g += gridDim.x) {
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (jobs[mid].begin <= g) lo = mid; else hi = mid - 1;
    }
    const PackJob& j = jobs[lo];
    const int64_t nkc = pack_units_k(j.K), kc = (g - j.begin) % nkc, hx = (g - j.begin) / nkc;
    bool any = false;
#define SMAT_GPACK(T)                                                                                        \
  switch (j.out_mode) {                                                                                      \
    case OUT_F16: any = pack_unit<T, OUT_F16>((const T*)j.in, j.layout, j.ldi, j.out, j.K, j.N, kc, hx, j.kperm, j.flags, tr); break; \
    case OUT_BF16: any = pack_unit<T, OUT_BF16>((const T*)j.in, j.layout, j.ldi, j.out, j.K, j.N, kc, hx, j.kperm, j.flags, tr); break; \
    default: any = pack_unit<T, OUT_SPLIT>((const T*)j.in, j.layout, j.ldi, j.out, j.K, j.N, kc, hx, j.kperm, j.flags, tr); break; \
  }
    switch (j.in_dtype) {
      case 0: SMAT_GPACK(float) break;
      case 1: SMAT_GPACK(__half) break;
      default: SMAT_GPACK(__nv_bfloat16) break;
    }
#undef SMAT_GPACK
    // every column or none: the exact words, of whichever form, cost the 24 jobs of
    // 512..8192 rows 0.6-3 us of their 8.7 here (registers), and are a filter only
    if (threadIdx.x < 2) j.cols[(g - j.begin) * 2 + threadIdx.x] = any ? 0xffffffffu : 0u;
  }
}

// Shared memory of a block: the transposition buffer, column-major only.
static size_t pack_smem(int layout, bool split) {
  return layout == 1 ? (size_t)kUnitK * kStride * 4 * (split ? 2 : 1) : 0;
}

template <typename T, int OUT>
static cudaError_t run_pack(const void* in, int layout, int64_t ldi, uint8_t* out, int64_t K, int64_t N,
                            const int32_t* kperm, uint8_t* flags, int32_t* counters, cudaStream_t s) {
  const int64_t nkc = pack_units_k(K), halves = pack_halves(N);
  if (nkc == 0 || halves == 0) return cudaSuccess;
  uint32_t* const cols = reinterpret_cast<uint32_t*>(flags + pack_cols_offset(K, N));
  // grid.y is limited to 65,535 halves: wider B goes in several launches
  for (int64_t h0 = 0; h0 < halves; h0 += 65534) {
    const int64_t hn = halves - h0 < 65534 ? halves - h0 : 65534;
    const T* src = (const T*)in + (layout == 1 ? h0 * 64 * ldi : h0 * 64);
    uint8_t* dst = out + (h0 >> 1) * ((K + 15) / 16) * (OUT == OUT_SPLIT ? 8192 : 4096);
    pack_b_kernel<T, OUT><<<dim3((unsigned)nkc, (unsigned)hn), kPackThreads, pack_smem(layout, OUT == OUT_SPLIT), s>>>(
        src, layout, ldi, dst, K, N - h0 * 64, kperm, flags + h0 * pack_flag_stride(K), cols + h0 * nkc * 2, counters);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// The 2:4 path's B operand from the packed tiles: tile (t, w) holds k-blocks
// 2w and 2w+1 of column tile t side by side, 128 rows (n) of 64 bytes (32
// k-values) in the 64-byte swizzle (inside every 8-row group, 16-byte chunk
// c of row n sits at chunk c ^ ((n >> 1) & 3)). One thread per row n; the
// lanes of a warp read neighbouring columns of one row k. Zeros for a half
// without a column below N, which is not packed.
__global__ void pack_b_sw64_kernel(const uint8_t* __restrict__ p, uint8_t* __restrict__ out, int64_t kbs,
                                   int64_t kw, int64_t N) {
  grid_release();  // the kernels launched behind may be set up
  grid_wait();     // the packed tiles
  const int64_t w = blockIdx.x;
  const int64_t t = blockIdx.y;
  const int n = threadIdx.x;
  const bool packed = t * 128 + (n & 64) < N;
  uint4 c[4];
  uint16_t* const v = reinterpret_cast<uint16_t*>(c);
#pragma unroll
  for (int hb = 0; hb < 2; ++hb) {
    const int64_t kb = 2 * w + hb;
    const uint8_t* src = p + (t * kbs + kb) * 4096 + (n >> 6) * 2048 + (n & 7) * 2;
#pragma unroll
    for (int k = 0; k < 16; ++k)
      v[hb * 16 + k] = packed && kb < kbs
                           ? *reinterpret_cast<const uint16_t*>(src + k * 128 + ((((n >> 3) & 7) ^ (k & 7)) << 4))
                           : (uint16_t)0;
  }
  uint4* dst = reinterpret_cast<uint4*>(out + (t * kw + w) * 8192 + n * 64);
  const int sw = (n >> 1) & 3;
#pragma unroll
  for (int q = 0; q < 4; ++q) dst[q ^ sw] = c[q];
}

}  // namespace dev

size_t packed_b64_bytes(int64_t K, int64_t N) {
  const int64_t kw = ((K + 15) / 16 + 1) / 2;
  return (size_t)kw * (size_t)packed_b_tiles(N) * 8192;
}

cudaError_t pack_b_sw64(const uint8_t* packed, int64_t K, int64_t N, uint8_t* out, cudaStream_t s) {
  const int64_t kbs = (K + 15) / 16, kw = (kbs + 1) / 2, nt = (N + 127) / 128;
  if (kw == 0 || nt == 0) return cudaSuccess;
  dim3 grid((unsigned)kw, (unsigned)nt);
  void* params[] = {&packed, &out, const_cast<int64_t*>(&kbs), const_cast<int64_t*>(&kw), &N};
  return launch_kernel(reinterpret_cast<const void*>(dev::pack_b_sw64_kernel), grid, dim3(128), 0, s, true, params);
}

int64_t packed_b_tiles(int64_t N) {
  const int64_t t = (N + 127) / 128;
  return t > 1 ? (t + 1) / 2 * 2 : t;
}

size_t packed_b_bytes(int64_t K, int64_t N) {
  return (size_t)((K + 15) / 16) * (size_t)packed_b_tiles(N) * 4096;
}

size_t pack_flag_bytes(int64_t K, int64_t N) {
  return (size_t)pack_cols_offset(K, N) + (size_t)pack_halves(N) * (size_t)pack_units_k(K) * 8;
}

cudaError_t pack_b(const void* in, int in_dtype, int layout, int64_t ldi, int out_mode, uint8_t* out,
                   int64_t K, int64_t N, const int32_t* kperm, uint8_t* flags, int32_t* counters, cudaStream_t s) {
  using namespace dev;
#define SMAT_PACK(T)                                                                             \
  switch (out_mode) {                                                                            \
    case OUT_F16: return run_pack<T, OUT_F16>(in, layout, ldi, out, K, N, kperm, flags, counters, s);     \
    case OUT_BF16: return run_pack<T, OUT_BF16>(in, layout, ldi, out, K, N, kperm, flags, counters, s);   \
    case OUT_SPLIT: return run_pack<T, OUT_SPLIT>(in, layout, ldi, out, K, N, kperm, flags, counters, s); \
    default: return cudaErrorInvalidValue;                                                       \
  }
  switch (in_dtype) {
    case 0: SMAT_PACK(float)
    case 1: SMAT_PACK(__half)
    case 2: SMAT_PACK(__nv_bfloat16)
    default: return cudaErrorInvalidValue;
  }
#undef SMAT_PACK
}

cudaError_t pack_b_grouped(const PackJob* d_jobs, int njobs, int64_t total_units, bool any_col, bool any_split,
                           int num_sms, int32_t* counters, int n_counters, cudaStream_t s) {
  const int64_t want = (int64_t)num_sms * 8;
  const int grid = (int)(total_units < 1 ? 1 : (total_units < want ? total_units : want));
  dev::pack_b_grouped_kernel<<<grid, dev::kPackThreads, dev::pack_smem(any_col ? 1 : 0, any_split), s>>>(
      d_jobs, njobs, total_units, counters, n_counters);
  return cudaGetLastError();
}

}  // namespace smat
