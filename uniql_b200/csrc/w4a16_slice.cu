// Load-time slicing primitives for packed W4A16 layers on sm_100a.
//
// UniQL re-slices its packed weights at every load of an elastic checkpoint
// (modeling/modeling_helpers.py:235-867: slice_w4a16_{up_gate,down,qk,v,o,in,out}_proj) by unpacking to one int per
// weight on the CPU, slicing and packing again (quantize/quantize_helpers.py:279-328, :67-84).  The two kernels here do
// the same work directly on the packed buffers:
//   * w4a16_gather_columns_kernel: new layer = chosen output columns of an old one (q/k/v/in_proj slicing).  An output
//     word holds 4 k-values x 2 columns; the 4 nibbles of one column sit in ONE source word (same packed row, same k
//     sub-position), so an output word is assembled from two source words and a few shifts.  Scales are gathered
//     through the 64-column scale permutation.
//   * w4a16_dequantize_rows_kernel: fp16 (q - 8) * s of chosen input rows, written in the nn.Linear layout
//     [column][kept row] that uniql_w4a16_quantize reads (o_proj / out_proj slicing re-quantises, :632-650).
// Memory-bound gathers (4-byte words of the columns, 16-byte pieces of the rows), run once per layer at load time.
#include "common.cuh"

namespace uniql {

namespace {

// position of column r (0..63) of a 64-column block inside a packed row, and its scale slot
struct ColPos {
  int j, g, hi;       // register index, fragment row, +8 half
};
__device__ __forceinline__ ColPos col_pos(int r) {
  ColPos p;
  p.j = r >> 4;
  p.g = r & 7;
  p.hi = (r >> 3) & 1;
  return p;
}
__device__ __forceinline__ int scale_slot(int r) { return 8 * (r & 7) + (r >> 3); }   // stored[8 i + j] = natural[i + 8 j]

// One CTA per 64 output columns and scale group: a thread looks its two source columns up once and assembles the same word
// of eight packed rows, sixteen independent loads in flight (one row per CTA: 12.9 us for 3584 of 4096 columns x 4096).
__global__ void __launch_bounds__(128)
w4a16_gather_columns_kernel(const uint32_t* __restrict__ packed_in, const __half* __restrict__ scales_in, int n_src_pad,
                            const int* __restrict__ col_index, int n_new, int zero_rows_from,
                            uint32_t* __restrict__ packed_out, __half* __restrict__ scales_out, int n_out_pad,
                            int* __restrict__ status_word) {
  const int w = threadIdx.x;                     // output word of this 64-column block
  const int b = blockIdx.x, grp = blockIdx.y;
  const int i = w >> 2, j = w & 3, g = i >> 2, c = i & 3;
  uint32_t word[2][8];
  int shift[2];                                  // 8 * the source column's half of its word
#pragma unroll
  for (int hi = 0; hi < 2; ++hi) {
    const int n_out = 64 * b + 16 * j + g + 8 * hi;
    int src = n_out < n_new ? col_index[n_out] : -1;
    if (src >= n_src_pad) {                      // not a column of the source: zero column, and say so
      if (status_word) atomicOr(status_word, UNIQL_STATUS_BAD_INDEX);
      src = -1;
    }
    const ColPos sp = col_pos(src & 63);
    shift[hi] = 8 * sp.hi;
    const uint32_t* from = packed_in + (size_t)grp * 8 * (2 * (size_t)n_src_pad) + (size_t)((src < 0 ? 0 : src) >> 6) * 128 +
                           (sp.g * 4 + c) * 4 + sp.j;
#pragma unroll
    for (int u = 0; u < 8; ++u) word[hi][u] = src < 0 ? 0u : from[(size_t)u * 2 * n_src_pad];
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int kt = grp * 8 + u;
    // nibbles of k = 2c, 2c + 8 (bits 0-7 of a column's half) and 2c + 1, 2c + 9 (bits 16-23); rows from zero_rows_from on
    // get code 0
    uint32_t keep = 0;
#pragma unroll
    for (int bit1 = 0; bit1 < 2; ++bit1)
#pragma unroll
      for (int bit8 = 0; bit8 < 2; ++bit8)
        if (16 * kt + 2 * c + bit1 + 8 * bit8 < zero_rows_from) keep |= 0xfu << (4 * bit8 + 16 * bit1);
    const uint32_t out = ((word[0][u] >> shift[0]) & keep) | (((word[1][u] >> shift[1]) & keep) << 8);
    packed_out[(size_t)kt * (2 * (size_t)n_out_pad) + (size_t)b * 128 + w] = out;
  }
  if (w < 64) {
    const int r = (w >> 3) + 8 * (w & 7);        // natural column stored at slot w
    const int n_out = 64 * b + r;
    const int src = n_out < n_new ? col_index[n_out] : -1;
    __half s = __float2half(0.f);
    if (src >= 0 && src < n_src_pad) s = scales_in[(size_t)grp * n_src_pad + (size_t)(src >> 6) * 64 + scale_slot(src & 63)];
    scales_out[(size_t)grp * n_out_pad + 64 * b + w] = s;
  }
}

// One CTA per 64 columns x 128 kept rows.  A thread takes the 16 bytes that hold all columns g, g + 8, ... of one source
// row (the permuted scales of those columns are 16 bytes too), writes its values to a shared tile and the CTA stores the
// tile in 16-byte pieces of 256 contiguous bytes per column.  One 4-byte load and one 2-byte store per weight, as before,
// moved 4096 x 3584 in 50 us; the traffic needs 6.
constexpr int kRowTile = 128, kRowPad = 8;
__global__ void __launch_bounds__(256)
w4a16_dequantize_rows_kernel(const uint32_t* __restrict__ packed, const __half* __restrict__ scales, int size_k,
                             int n_src_pad, const int* __restrict__ row_index, int k_new, int n_real,
                             __half* __restrict__ out, int64_t ld, int vec_in, int* __restrict__ status_word) {
  __shared__ __align__(16) __half tile[64][kRowTile + kRowPad];
  const int kk0 = blockIdx.x * kRowTile, b = blockIdx.y;
  const int kk = threadIdx.x & (kRowTile - 1);
  const int src = kk0 + kk < k_new ? row_index[kk0 + kk] : 0;
  const bool bad = src < 0 || src >= size_k;     // not a row of the source: zero, and say so
  if (bad && status_word) atomicOr(status_word, UNIQL_STATUS_BAD_INDEX);
  const int k = bad ? 0 : src;
  const int c = (k & 7) >> 1, sh = 4 * ((k >> 3) & 1) + 16 * (k & 1);
  const uint32_t* prow = packed + (size_t)(k >> 4) * (2 * (size_t)n_src_pad) + (size_t)b * 128 + c * 4;
  const __half* srow = scales + (size_t)(k >> 7) * n_src_pad + (size_t)b * 64;
  uint4 w4[4], s4[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int g = (threadIdx.x >> 7) * 4 + i;
    if (vec_in) {
      w4[i] = *reinterpret_cast<const uint4*>(prow + g * 16);
      s4[i] = *reinterpret_cast<const uint4*>(srow + g * 8);
    } else {                                     // buffers that are not 16-byte aligned
      const uint32_t* pw = prow + g * 16;
      w4[i] = make_uint4(pw[0], pw[1], pw[2], pw[3]);
      uint32_t v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        v[e] = __half_as_ushort(srow[g * 8 + 2 * e]) | ((uint32_t)__half_as_ushort(srow[g * 8 + 2 * e + 1]) << 16);
      s4[i] = make_uint4(v[0], v[1], v[2], v[3]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int g = (threadIdx.x >> 7) * 4 + i;
    const uint32_t w[4] = {w4[i].x, w4[i].y, w4[i].z, w4[i].w}, sc[4] = {s4[i].x, s4[i].y, s4[i].z, s4[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      // columns 16 j + g (nibble sh / 4) and 16 j + g + 8 (two nibbles up), exact q - 8, one rounding of the product
      const uint32_t q = w[j] >> sh;
      const uint32_t m8 = nib_pair_to_half2_m8((q & 0xfu) | ((q & 0xf00u) << 8));
      const __half2 y = __hmul2(*reinterpret_cast<const __half2*>(&m8), *reinterpret_cast<const __half2*>(&sc[j]));
      tile[16 * j + g][kk] = bad ? __float2half(0.f) : __low2half(y);
      tile[16 * j + g + 8][kk] = bad ? __float2half(0.f) : __high2half(y);
    }
  }
  __syncthreads();
  const int rows = min(kRowTile, k_new - kk0);
  const bool vec = rows == kRowTile && (ld & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  for (int v = threadIdx.x; v < 64 * (kRowTile / 8); v += 256) {
    const int r = v / (kRowTile / 8), x = (v % (kRowTile / 8)) * 8, n = b * 64 + r;
    if (n >= n_real) continue;
    __half* d = out + (size_t)n * ld + kk0 + x;
    if (vec) *reinterpret_cast<uint4*>(d) = *reinterpret_cast<const uint4*>(&tile[r][x]);
    else
      for (int e = 0; e < 8 && x + e < rows; ++e) d[e] = tile[r][x + e];
  }
}

}  // namespace

}  // namespace uniql

extern "C" int uniql_w4a16_gather_columns(const void* packed_in, const void* scales_in, int64_t size_k, int64_t n_src_pad,
                                          const int32_t* col_index, int64_t n_new, int64_t zero_rows_from,
                                          void* packed_out, void* scales_out, int64_t n_out_pad, int* status_word,
                                          void* stream) {
  using namespace uniql;
  if (size_k <= 0 || size_k % 128 != 0 || n_src_pad <= 0 || n_src_pad % 64 != 0) return UNIQL_ESHAPE;
  if (n_out_pad <= 0 || n_out_pad % 64 != 0 || n_new < 0 || n_new > n_out_pad) return UNIQL_ESHAPE;
  if (size_k / 16 > 65535) return UNIQL_ESHAPE;
  if (!packed_in || !scales_in || !packed_out || !scales_out || (n_new > 0 && !col_index)) return UNIQL_EINVAL;
  if (zero_rows_from < 0 || zero_rows_from > size_k) zero_rows_from = size_k;
  dim3 grid((unsigned)(n_out_pad / 64), (unsigned)(size_k / 128));
  w4a16_gather_columns_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>(
      (const uint32_t*)packed_in, (const __half*)scales_in, (int)n_src_pad, col_index, (int)n_new, (int)zero_rows_from,
      (uint32_t*)packed_out, (__half*)scales_out, (int)n_out_pad, status_word);
  return launch_status();
}

extern "C" int uniql_w4a16_dequantize_rows(const void* packed, const void* scales, int64_t size_k, int64_t n_src_pad,
                                           const int32_t* row_index, int64_t k_new, int64_t n_real, void* out, int64_t ld,
                                           int* status_word, void* stream) {
  using namespace uniql;
  if (size_k <= 0 || size_k % 128 != 0 || n_src_pad <= 0 || n_src_pad % 64 != 0) return UNIQL_ESHAPE;
  if (k_new < 0 || n_real < 0 || n_real > n_src_pad || n_real > 65535 || ld < k_new) return UNIQL_ESHAPE;
  if (k_new == 0 || n_real == 0) return UNIQL_OK;
  if (!packed || !scales || !row_index || !out) return UNIQL_EINVAL;
  dim3 grid((unsigned)((k_new + kRowTile - 1) / kRowTile), (unsigned)((n_real + 63) / 64));
  w4a16_dequantize_rows_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(
      (const uint32_t*)packed, (const __half*)scales, (int)size_k, (int)n_src_pad, row_index, (int)k_new, (int)n_real,
      (__half*)out, ld, aligned16(packed) && aligned16(scales) ? 1 : 0, status_word);
  return launch_status();
}
