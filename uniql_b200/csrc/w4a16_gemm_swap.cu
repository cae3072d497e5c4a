// Operand-swapped W4A16 linear for sm_100a (small and middle row counts): tcgen05 tensor cores with the dequantised
// weights as the 128-row operand, fed from tensor memory.
//
// Replaces the same launches of UniQL's Marlin kernel (csrc/linear/marlin_gemm_kernel.cuh:176-740) on the same packed
// buffers (quantize/quantize_helpers.py:145-165 weight order, :54-62 scale order).
//
// The weight tile [128 columns x 128 k] of a stage is the 128-row MMA operand (tensor-memory lane = output column), the
// activation tile [Mb x 128 k] (Mb = rows of the tile rounded up to 16, at most 256) the N operand, so the MMA is
// 128 x Mb x 16 and no tensor work is spent on padding rows.  The weight operand never enters shared memory: a lane of
// the packed layout holds exactly the register fragment of tcgen05.st.16x128b, so the dequantise warps write it to
// tensor memory and the MMA reads it from there.  One stage = one scale group (128 k, eight MMAs), because every
// hand-off between the warp roles is paid once per stage.
//   warp 0       TMA producer of the packed words (two 4 KB boxes per stage, one per 64-column block)
//   warps 1, 3   one elected lane each issues the MMAs of every other stage, the commit that releases the stage and a poll
//                of its next stage's barrier (warp 1 also owns the tensor-memory allocation).  Two issuers on two SM
//                sub-partitions, each with an accumulator of its own: next to the dequantise warps one issuing thread
//                needs ~420 cycles per stage (~120 alone), more than the 128 to 256 the MMAs take up to 64 rows.
//   warp 2       TMA producer of the activation tile (two swizzled [Mb x 64 k] sub-tiles in one 3-D box)
//   warps 4-7    epilogue (GS: they also apply the group scales, see below)
//   warps 8-23   dequantise, four sets of four (one warp per 32-lane quarter of tensor memory); set t converts every
//                fourth k-block.  The ring of stages is deeper than the number of sets where tensor memory allows (six
//                for Mb <= 64), so that a set can convert its next k-block while the MMAs of the last one are in flight.
// GS (at most 16 rows): the operand is the exact code (q - 8), the MMAs of a stage write a fresh accumulator of 16
// columns, and the epilogue warps add it to the running fp32 sums times the group scale -- the arithmetic of the decode
// kernel of w4a16_gemv.cu.  Otherwise the scale is multiplied into the weight with one fp16 rounding, bit-identical to
// the reference's dequantised weight.
//
// Up to four projections that read the same activations share a launch: their 128-column tiles form one list.  A SwiGLU
// pair has tiles of 64 gate columns and the 64 up columns beside them, so that the epilogue forms silu(gate) * up.
// With few tiles a cluster of up to 8 CTAs shares each tile, every CTA reducing a slice of k; the partial accumulators
// are parked in shared memory and summed in rank order through distributed shared memory (deterministic).
//
// TP (at most 16 rows): the launch is a step of a tensor-parallel layer.  The sums are those of the plain launch; the
// epilogue works on four columns of a row at a time and carries the exchanges of tp_exchange.cuh: the sum of a row-parallel
// shard over the ranks, or the columns of a column shard stored into every rank's feature area.  A CTA pushes all its words
// of a tile before it waits for any, and every rank takes its tiles in ascending order (the tiled kernel too, which a rank
// with another k may run), so the lowest unfinished tile never waits for a higher one; waits are bounded.
//
// Bound: weight stream (HBM) below ~128 rows, tensor pipe above; in practice the per-stage chain of the dequantise warps
// (13 instructions per packed word, 9 with GS, and ~110 per warp and stage: ~320 or ~250) and the fixed cost of a launch.
// All 24 warps together issue 1961 warp instructions per stage at 64 rows, 1631 at 16 (14336 x 4096, counters); the SMs that
// work issue on 84 % and 79 % of their cycles.
// Every mbarrier wait is bounded; a wait that gives up sets UNIQL_STATUS_WAIT_TIMEOUT and the kernel drains.
#include "common.cuh"
#include "linear_internal.cuh"
#include "tc.cuh"
#include "tp_exchange.cuh"

#include <cuda.h>
#include <stdlib.h>
#include <string.h>

namespace uniql {

namespace sw {
constexpr int BNW = 128, BK = 128;
constexpr int P_BLK = 4096;                     // 8 packed rows of one 64-column block
constexpr int P_BYTES = 2 * P_BLK;
constexpr int MAX_STAGES = 6, MAX_PSTAGES = 16;
constexpr int NSETS = 4, DEQ_WARPS = 4;
constexpr int FIRST_EPI_WARP = 4, FIRST_DEQ_WARP = 8;
constexpr int THREADS = (FIRST_DEQ_WARP + NSETS * DEQ_WARPS) * 32;
constexpr int FINISH_THREADS = THREADS - FIRST_EPI_WARP * 32;
constexpr int NUM_BARS = 3 * MAX_STAGES + 2 * MAX_PSTAGES + 4;
constexpr int MB_MAX = 256;                     // rows of a tile
constexpr int RC = 16;                          // batch rows per epilogue chunk
constexpr int ROW_BYTES = BNW * 4;              // one batch row of a parked fp32 tile
constexpr int OFF_BAR = 0, OFF_PART = 1024, OFF_P = OFF_PART + 2 * RC * ROW_BYTES;
constexpr int TMEM_COLS = 512;
constexpr int SMEM_MAX = 227 * 1024;
static_assert(NUM_BARS * 8 + 16 <= 1024, "barrier block");
static_assert(THREADS <= 1024, "block size");
}  // namespace sw

struct SwapProj {
  const __half* S;                              // permuted scales [K/128][N]
  const __half* bias;
  __half* D;
  int64_t ldd;
  int N, n_out;
};
struct SwapParams {
  SwapProj proj[kMaxProj];
  int tile_start[kMaxProj + 1];                 // first column tile of each projection
  int nproj, pair;                              // pair: projections 0 and 1 are gate and up of a SwiGLU
  const __half* residual;                       // fp16 [M, n_out] added to the rounded result, or nullptr
  int64_t ldr;
  int M, Mb, K;
  int rtiles, ntiles;                           // row tiles of Mb rows; ntiles = column tiles * rtiles
  int split;                                    // CTAs of a cluster that share one tile, each a slice of k
  int one_tile;                                 // no CTA has more than one tile
  int nst, pst, nsets;                          // stages of the tensor-memory / activation ring, of the packed ring; sets of
                                                // dequantise warps in use (nst >= nsets, pst a multiple of nsets)
  int nissue;                                   // issuing threads (1 or 2; with 2, nst is even: a stage has one issuer)
  int nbuf;                                     // tiles whose accumulators are kept (1 or 2)
  int off_x;                                    // activation ring in shared memory
  const unsigned char* pf_ptr[4];               // byte ranges to pull into L2 when this CTA's weight stream ends, in
  long long pf_lines[4];                        // 128-byte lines
  int npf;
  int early_weights;                            // 0: weights and scales may have been written by the preceding kernel
  int* status_word;
  CommView cv;                                  // tensor-parallel launches only
};
struct SwapMaps {
  CUtensorMap w[kMaxProj];                      // packed weights, boxes of 128 words x 8 packed rows
};

// column tile -> (projection, tile inside it)
__device__ __forceinline__ void sw_tile_of(const SwapParams& p, int ct, int& pi, int& lt) {
  pi = 0;
  if (!p.pair) {
#pragma unroll
    for (int i = 1; i < kMaxProj; ++i)
      if (i < p.nproj && ct >= p.tile_start[i]) pi = i;
  }
  lt = ct - p.tile_start[pi];
}

__device__ __forceinline__ void sw_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void sw_tma_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void sw_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void sw_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// The eight MMAs of one 128-k stage, the commit that releases the stage, and one poll of the NEXT stage's barrier, in
// one block: the poll is issued first and its result read last, so its latency hides behind the issue of the MMAs.
// ("Next": the issuer's next stage.)
// The weight operand comes from tensor memory (8 columns per K=16 step), the activation operand from two swizzled
// [Mb x 64 k] sub-tiles in shared memory.  Returns whether the next stage was already full.
__device__ __forceinline__ uint32_t sw_issue_stage(uint32_t tmem_d, uint32_t tmem_w, uint32_t xlo0, uint32_t xlo1,
                                                   uint32_t xhi, uint32_t idesc, uint32_t accumulate, uint32_t bar_release,
                                                   uint32_t bar_next, uint32_t par_next) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q, t;\n\t.reg .b32 a1, a2, a3, a4, a5, a6, a7, l1, l2, l3, m1, m2, m3;\n\t"
      ".reg .b64 b0, b1, b2, b3, c0, c1, c2, c3;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%9], %10;\n\t"
      "setp.ne.b32 p, %7, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "add.u32 a1, %2, 8;\n\tadd.u32 a2, %2, 16;\n\tadd.u32 a3, %2, 24;\n\tadd.u32 a4, %2, 32;\n\t"
      "add.u32 a5, %2, 40;\n\tadd.u32 a6, %2, 48;\n\tadd.u32 a7, %2, 56;\n\t"
      "add.u32 l1, %3, 2;\n\tadd.u32 l2, %3, 4;\n\tadd.u32 l3, %3, 6;\n\t"
      "add.u32 m1, %4, 2;\n\tadd.u32 m2, %4, 4;\n\tadd.u32 m3, %4, 6;\n\t"
      "mov.b64 b0, {%3, %5};\n\tmov.b64 b1, {l1, %5};\n\tmov.b64 b2, {l2, %5};\n\tmov.b64 b3, {l3, %5};\n\t"
      "mov.b64 c0, {%4, %5};\n\tmov.b64 c1, {m1, %5};\n\tmov.b64 c2, {m2, %5};\n\tmov.b64 c3, {m3, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [%2], b0, %6, p;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [a1], b1, %6, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [a2], b2, %6, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [a3], b3, %6, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [a4], c0, %6, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [a5], c1, %6, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [a6], c2, %6, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [a7], c3, %6, t;\n\t"
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%8];\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(ok)
      : "r"(tmem_d), "r"(tmem_w), "r"(xlo0), "r"(xlo1), "r"(xhi), "r"(idesc), "r"(accumulate), "r"(bar_release),
        "r"(bar_next), "r"(par_next)
      : "memory");
  return ok;
}

// Where the columns of a tile go; looked up once per tile (the projection index is dynamic), not once per value.
struct SwOut {
  const __half* bias;
  const __half* ubias;                          // bias of the up projection of a pair
  const __half* residual;
  __half* D;
  int64_t ldd, ldr;
  int n0, n_out, row0, row_end;                 // first column, real columns, first row, end of the real rows
};
__device__ __forceinline__ SwOut sw_out_of(const SwapParams& p, int T) {
  int pi, lt;
  sw_tile_of(p, T / p.rtiles, pi, lt);
  const SwapProj& pr = p.proj[pi];
  SwOut o;
  o.bias = pr.bias; o.ubias = p.pair ? p.proj[1].bias : nullptr; o.residual = p.residual;
  o.D = pr.D; o.ldd = pr.ldd; o.ldr = p.ldr;
  o.n0 = lt * (p.pair ? 64 : sw::BNW); o.n_out = pr.n_out;
  o.row0 = (T % p.rtiles) * p.Mb; o.row_end = p.M;
  return o;
}
// One value: bias, SwiGLU product, residual, with the roundings of the separate modules (fp16 result, fp16 SiLU, fp16
// product, fp16 sum).  Everything optional sits behind a uniform branch: this code runs once per launch, so the
// instructions it does not fetch are what it saves.
template <bool PAIR, bool RES>
__device__ __forceinline__ __half sw_value(const SwOut& o, int row, int n, float a, float u) {
  if (o.bias) a += __half2float(o.bias[n]);
  __half h = __float2half_rn(a);
  if (PAIR) {
    if (o.ubias) u += __half2float(o.ubias[n]);
    const __half uh = __float2half_rn(u);
    const float gf = __half2float(h);
    const __half ah = __float2half_rn(gf / (1.0f + expf(-gf)));
    h = __float2half_rn(__half2float(ah) * __half2float(uh));
  }
  if (RES && o.residual) h = __float2half_rn(__half2float(h) + __half2float(o.residual[(size_t)row * o.ldr + n]));
  return h;
}
// Four adjacent columns of one batch row of a plain launch.  c4: column inside the tile.
template <bool RES>
__device__ __forceinline__ void sw_finish4(const SwOut& o, int row, int c4, float4 v) {
  const int n = o.n0 + c4;
  if (n >= o.n_out || row >= o.row_end) return;
  __half* d = o.D + (size_t)row * o.ldd + n;
  const float a[4] = {v.x, v.y, v.z, v.w};
  if (n + 3 < o.n_out && !o.bias && !(RES && o.residual) && (reinterpret_cast<uintptr_t>(d) & 7u) == 0) {
    const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(d) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (n + e < o.n_out) d[e] = sw_value<false, RES>(o, row, n + e, a[e], 0.f);
  }
}

// The same quad of a tensor-parallel launch (u: the up columns of a pair): like sw_value, and a column shard's columns
// travel to every rank's feature area.
template <bool PAIR>
__device__ __forceinline__ void sw_finish4_tp(const SwOut& o, const CommView& cv, uint32_t gather_ep, int row, int c4,
                                              float4 v, float4 u) {
  const int n = o.n0 + c4;
  if (n >= o.n_out || row >= o.row_end) return;
  __half* d = o.D + (size_t)row * o.ldd + n;
  const float a[4] = {v.x, v.y, v.z, v.w}, b[4] = {u.x, u.y, u.z, u.w};
  __half h[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    h[e] = __float2half_rn(0.f);
    if (n + e < o.n_out) d[e] = h[e] = sw_value<PAIR, true>(o, row, n + e, a[e], b[e]);
  }
  if (cv.gather_out) tp_feature4(cv, gather_ep, row, n, o.n_out, h);
}

__device__ __forceinline__ float4 sw_lds_f4(uint32_t addr) {
  const uint4 v = tc_lds128(addr);
  return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ float sw_lds_f(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

template <bool GS, bool PAIR, bool TP>
__global__ void __launch_bounds__(sw::THREADS, 1)
w4a16_gemm_swap_kernel(const __grid_constant__ SwapParams p, const __grid_constant__ CUtensorMap xmap,
                       const __grid_constant__ SwapMaps wmaps) {
  using namespace sw;
  static_assert(GS || (!PAIR && !TP), "above 16 rows: plain outputs only");
  extern __shared__ uint8_t smem_unaligned[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = tc_smem_addr(smem);
  // full[s]: the activation tile has landed (TMA bytes) AND a set's warps have written the stage's weight tile;
  // empty[s]: the MMAs that read stage s have completed; acc_empty[s] (GS): its accumulator has been read
  const uint32_t bar_full = sbase + OFF_BAR, bar_empty = bar_full + 8 * MAX_STAGES;
  const uint32_t bar_acc_empty = bar_empty + 8 * MAX_STAGES;
  const uint32_t bar_full_p = bar_acc_empty + 8 * MAX_STAGES, bar_empty_p = bar_full_p + 8 * MAX_PSTAGES;
  const uint32_t bar_tmem_full = bar_empty_p + 8 * MAX_PSTAGES, bar_tmem_empty = bar_tmem_full + 16;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + OFF_BAR + NUM_BARS * 8);
  const uint32_t xbase = sbase + p.off_x;
  const uint32_t x_half = (uint32_t)p.Mb * 128, x_bytes = 2 * x_half;   // one [Mb x 64 k] sub-tile; a stage

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // a cluster of p.split CTAs owns one tile at a time; CTA `rank` of it reduces k-blocks [kb0, kb0 + KB)
  const int rank = (int)blockIdx.x % p.split;
  const int tile0 = (int)blockIdx.x / p.split, tile_step = (int)gridDim.x / p.split;
  const int groups = p.K / BK;
  const int kb0 = (int)((long long)groups * rank / p.split);
  const int KB = (int)((long long)groups * (rank + 1) / p.split) - kb0;
  const int my_tiles = (tile0 < p.ntiles) ? (p.ntiles - 1 - tile0) / tile_step + 1 : 0;
  const int total_it = my_tiles * KB;
  const int tmem_w0 = TMEM_COLS - p.nst * (BK / 2);   // weight tile of stage s: columns tmem_w0 + 64 s

  // Packed words of k-block kb of column tile (pi, lt): two boxes, one barrier.
  auto load_packed = [&](int pi, int lt, int kb, int sp) {
    const int x0 = PAIR ? lt * 128 : lt * 256;
    const uint32_t dst = sbase + OFF_P + sp * P_BYTES, bar = bar_full_p + 8 * sp;
    tc_mbar_expect_tx(bar, P_BYTES);
    tc_tma_2d(dst, &wmaps.w[pi], x0, (kb0 + kb) * (BK / 16), bar);
    tc_tma_2d(dst + P_BLK, PAIR ? &wmaps.w[1] : &wmaps.w[pi], PAIR ? x0 : x0 + 128, (kb0 + kb) * (BK / 16), bar);   // past the width: zeros
  };
  // The first packed stages (of the first tile) are requested before anything else is set up: from here to the first MMA
  // a CTA needs the latency of these loads plus a conversion.
  const int early = tile0 < p.ntiles ? min(p.nsets, KB) : 0;
  if (warp == 0 && tc_elect()) {
    for (int s = 0; s < p.pst; ++s) {
      tc_mbar_init(bar_full_p + 8 * s, 1);
      tc_mbar_init(bar_empty_p + 8 * s, DEQ_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    int pi, lt;
    sw_tile_of(p, tile0 / p.rtiles, pi, lt);
    if (!p.early_weights) pdl_wait();
    for (int kb = 0; kb < early; ++kb) load_packed(pi, lt, kb, kb);
  }
  if (warp == 2 && tc_elect()) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
    for (int s = 0; s < p.nst; ++s) {
      tc_mbar_init(bar_full + 8 * s, 1 + DEQ_WARPS);
      tc_mbar_init(bar_empty + 8 * s, 1);
      tc_mbar_init(bar_acc_empty + 8 * s, 4);
    }
    for (int b = 0; b < 2; ++b) {
      tc_mbar_init(bar_tmem_full + 8 * b, p.nissue);
      tc_mbar_init(bar_tmem_empty + 8 * b, 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_addr((const void*)tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  bool timed_out = false;
  if (!p.early_weights) pdl_wait();              // before the first scale is read

  // TP: finishes rows [r0, r1) of a tile with `nthreads` threads, four columns of a row per thread and step; `quad` delivers
  // the sums of four adjacent columns of the tile.  kQuads divides every nthreads, so a thread stays in one 64-column block.
  auto finish_tp = [&](const SwOut& o, int r0, int r1, int tid, int nthreads, uint32_t reduce_ep, uint32_t gather_ep, auto&& quad) {
    constexpr int kQuads = PAIR ? 16 : 32;
    const int c4 = (tid % kQuads) * 4, block = (o.n0 + c4) >> 6, c = c4 & 63;
    const bool push = !PAIR && p.cv.reduce;
    if (o.n0 + c4 >= p.proj[0].N && push) return;   // past the packed width: nothing travels (a reduce launch has one projection)
    if (push) {
#pragma unroll 1
      for (int r = r0 + tid / kQuads; r < r1; r += nthreads / kQuads) tp_push4(p.cv, reduce_ep, block, o.row0 + r, c, quad(r, c4));
    }
#pragma unroll 1
    for (int r = r0 + tid / kQuads; r < r1; r += nthreads / kQuads) {
      const float4 v = push ? tp_gather4<4>(p.cv, reduce_ep, block, o.row0 + r, c, timed_out) : quad(r, c4);
      const float4 u = PAIR ? quad(r, c4 + 64) : make_float4(0.f, 0.f, 0.f, 0.f);
      sw_finish4_tp<PAIR>(o, p.cv, gather_ep, o.row0 + r, c4, v, u);
    }
  };
  // Epochs of this thread's words (see finish_tp).  The wait keeps every exchange of this launch behind the preceding ones:
  // they advance the counters, and a peer that runs one exchange ahead relies on this rank having finished the one before.
  auto tp_epochs = [&](const SwOut& o, int tid, uint32_t& reduce_ep, uint32_t& gather_ep) {
    pdl_wait();
    const int n = o.n0 + (tid % (PAIR ? 16 : 32)) * 4;
    reduce_ep = (p.cv.reduce && n < p.proj[0].N) ? *tp_reduce_counter(p.cv, n >> 6) + 1 : 0;
    gather_ep = p.cv.gather_out ? tp_gather_epoch(p.cv) : 0;
  };
  // once every thread has finished its part of the tile: one thread per 64-column block
  auto tp_advance = [&](const SwOut& o, int tid) {
    if (p.cv.reduce && tid < 2 && o.n0 + tid * 64 < p.proj[0].N) {
      volatile uint32_t* ctr = tp_reduce_counter(p.cv, (o.n0 >> 6) + tid);
      *ctr = *ctr + 1;
    }
  };

  // Finishes 16 rows of a tile, held by four warps (one per quarter of the columns; `v`: this lane's column).  A cluster
  // parks them in the activation ring (idle once the last MMA has completed) for the sum over the ranks, below.
  // Otherwise the values of a plain launch are stored straight from the registers (64 bytes per warp and row); a pair
  // (and a tensor-parallel launch) goes through `park`, 16 rows of shared memory, and a barrier of the four epilogue
  // warps, which bring gate and up together.
  auto emit = [&](const SwOut& o, int c0, const float (&v)[16], uint32_t park, int gtid) {
    const int col = (warp & 3) * 32 + lane;
    if (p.split > 1) {
#pragma unroll
      for (int e = 0; e < RC; ++e) tc_sts32(xbase + (c0 + e) * ROW_BYTES + col * 4, __float_as_uint(v[e]));
    } else if (TP) {
      uint32_t reduce_ep, gather_ep;
      tp_epochs(o, gtid, reduce_ep, gather_ep);
#pragma unroll
      for (int e = 0; e < RC; ++e) tc_sts32(park + e * ROW_BYTES + col * 4, __float_as_uint(v[e]));
      asm volatile("bar.sync 1, 128;" ::: "memory");
      finish_tp(o, 0, min(RC, o.row_end - o.row0), gtid, 128, reduce_ep, gather_ep,
                [&](int r, int c) { return sw_lds_f4(park + r * ROW_BYTES + c * 4); });
      asm volatile("bar.sync 1, 128;" ::: "memory");
      tp_advance(o, gtid);
    } else if (!PAIR) {
      const int n = o.n0 + col, rows = o.row_end - o.row0 - c0;
      if (n < o.n_out) {
        __half* d = o.D + (size_t)(o.row0 + c0) * o.ldd + n;
        const float bv = o.bias ? __half2float(o.bias[n]) : 0.f;
        if (GS && o.residual) {
          const __half* res = o.residual + (size_t)(o.row0 + c0) * o.ldr + n;
#pragma unroll
          for (int e = 0; e < RC; ++e)
            if (e < rows)
              d[(size_t)e * o.ldd] = __float2half_rn(__half2float(__float2half_rn(v[e] + bv)) + __half2float(res[(size_t)e * o.ldr]));
        } else {
#pragma unroll
          for (int e = 0; e < RC; ++e)
            if (e < rows) d[(size_t)e * o.ldd] = __float2half_rn(v[e] + bv);
        }
      }
    } else {
#pragma unroll
      for (int e = 0; e < RC; ++e) tc_sts32(park + e * ROW_BYTES + col * 4, __float_as_uint(v[e]));
      asm volatile("bar.sync 1, 128;" ::: "memory");
      // one value per thread and step: a small loop, because instructions that run once per tile are fetched cold
      const int c = gtid & 63, n = o.n0 + c, rows = min(RC, o.row_end - o.row0 - c0);
      if (n < o.n_out) {
#pragma unroll 1
        for (int r = gtid >> 6; r < rows; r += 2) {
          const uint32_t a = park + r * ROW_BYTES + c * 4;
          const int row = o.row0 + c0 + r;
          o.D[(size_t)row * o.ldd + n] = sw_value<true, true>(o, row, n, sw_lds_f(a), sw_lds_f(a + 256));
        }
      }
    }
  };
  // reads the accumulators of 16 rows (both issuers') of tensor-memory tile `acc` and finishes them
  auto drain = [&](const SwOut& o, uint32_t acc, int c0) {
    uint32_t r0[16], r1[16];
    sw_ld16(acc + c0, r0);
    if (p.nissue == 2) sw_ld16(acc + p.Mb + c0, r1);
    sw_wait_ld();
    float v[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(r0[e]);
    if (p.nissue == 2) {
#pragma unroll
      for (int e = 0; e < 16; ++e) v[e] += __uint_as_float(r1[e]);
    }
    emit(o, c0, v, 0, 0);                        // plain outputs: nothing is parked
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ packed-weight producer (the HBM stream)
    if (tc_elect()) {
      int sp = early == p.pst ? 0 : early;
      uint32_t ph = early == p.pst ? 1 : 0;
      int kb = early;
      for (int T = tile0; T < p.ntiles && !timed_out; T += tile_step, kb = 0) {   // no copy is issued after a wait gave up
        int pi, lt;
        sw_tile_of(p, T / p.rtiles, pi, lt);
        for (; kb < KB; ++kb) {
          if (!tc_mbar_wait(bar_empty_p + 8 * sp, ph ^ 1)) { timed_out = true; break; }
          load_packed(pi, lt, kb, sp);
          if (++sp == p.pst) { sp = 0; ph ^= 1; }
        }
      }
    }
    // The last packed words are on their way: ask L2 for this CTA's share of the weights that the following launches will
    // stream, so that HBM keeps working while this launch converts, reduces and drains (plain per-line hints).
    __syncwarp();
    for (int r = 0; r < p.npf; ++r)
      for (long long l = (long long)blockIdx.x * 32 + lane; l < p.pf_lines[r]; l += (long long)gridDim.x * 32)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p.pf_ptr[r] + l * 128));
  } else if (warp == 2) {
    // ------------------------------------------------------------------ activation producer (re-reads, L2 hits)
    if (tc_elect()) {
      // Programmatic dependent launch: everything up to here (barriers, tensor memory, the first weight tiles and their
      // conversion) ran while the producer of the activations was still finishing; the activation tiles are the only
      // thing that has to wait for it.  Results (and the residual) are touched after MMAs that consumed those tiles.
      // The next kernel in the stream may start its own set-up and weights from here on: behind the wait, so that it may
      // rely on everything in front of this launch having ended.
      pdl_wait();
      pdl_launch_dependents();
      int s = 0;
      uint32_t ph = 0;
      for (int T = tile0; T < p.ntiles && !timed_out; T += tile_step) {
        const int y = (T % p.rtiles) * p.Mb;
        for (int kb = 0; kb < KB; ++kb) {
          if (!tc_mbar_wait(bar_empty + 8 * s, ph ^ 1)) { timed_out = true; break; }
          tc_mbar_expect_tx(bar_full + 8 * s, x_bytes);
          sw_tma_3d(xbase + s * x_bytes, &xmap, 0, y, (kb0 + kb) * 2, bar_full + 8 * s);
          if (++s == p.nst) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp < FIRST_EPI_WARP) {
    // ------------------------------------------------------------------ MMA issuers: warp 1 (and 3) take every nissue-th stage
    const int issuer = warp >> 1;
    if (issuer < p.nissue && tc_elect()) {
      // D fp32, A/B fp16, both K-major, M = 128 (weight columns), N = Mb (batch rows)
      const uint32_t idesc = (1u << 4) | ((uint32_t)(p.Mb >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
      const uint64_t xdesc = tc_smem_desc(xbase);
      const uint32_t xlo = (uint32_t)xdesc, xhi = (uint32_t)(xdesc >> 32);
      const uint32_t x_step = x_bytes >> 4, x_half_step = x_half >> 4;
      const int step = p.nissue;
      int it = issuer, it_tile = 0, s = issuer, kb = issuer;
      uint32_t ph = 0;
      uint32_t ready = 0;                        // the current stage's full barrier was seen complete by the last poll
      for (int T = tile0; T < p.ntiles && !timed_out; T += tile_step, ++it_tile) {
        const int buf = p.nbuf == 2 ? (it_tile & 1) : 0;
        const int use = p.nbuf == 2 ? it_tile >> 1 : it_tile;
        if (!GS && !tc_mbar_wait(bar_tmem_empty + 8 * buf, (use & 1) ^ 1)) timed_out = true;
        const uint32_t tmem_d = tmem_base + (uint32_t)((buf * step + issuer) * p.Mb);
        const int kb_first = kb;
        for (; kb < KB; kb += step, it += step) {
          if (GS && !tc_mbar_wait(bar_acc_empty + 8 * s, ph ^ 1)) timed_out = true;
          if (!ready && !timed_out && !tc_mbar_wait(bar_full + 8 * s, ph)) timed_out = true;
          if (timed_out) break;
          tc_fence_after();
          int s1 = s + step;
          uint32_t ph1 = ph;
          if (s1 >= p.nst) { s1 -= p.nst; ph1 ^= 1; }
          ready = sw_issue_stage(GS ? tmem_base + s * 16 : tmem_d, tmem_base + tmem_w0 + s * (BK / 2), xlo + s * x_step,
                                 xlo + s * x_step + x_half_step, xhi, idesc, (GS || kb == kb_first) ? 0u : 1u,
                                 bar_empty + 8 * s, bar_full + 8 * s1, ph1);
          if (it + step >= total_it) ready = 0;   // that poll looked at a phase nobody will complete
          s = s1;
          ph = ph1;
        }
        kb -= KB;
        if (!GS) tc_commit(bar_tmem_full + 8 * buf);
      }
    }
  } else if (warp < FIRST_DEQ_WARP) {
    // ------------------------------------------------------------------ epilogue (lane = column, TMEM column = batch row)
    const int q = warp & 3;
    const int etid = (int)threadIdx.x - FIRST_EPI_WARP * 32;
    const int col = q * 32 + lane;
    int pbuf = 0;                                // two buffers, so one barrier per chunk: a buffer is written again only
                                                 // after every thread has passed the barrier behind its last read
    auto park = [&]() {
      const uint32_t a = sbase + OFF_PART + pbuf * (RC * ROW_BYTES);
      pbuf ^= 1;
      return a;
    };
    const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16);
    int it_tile = 0, s = 0;
    uint32_t ph = 0;
    for (int T = tile0; T < p.ntiles && (GS || !p.one_tile); T += tile_step, ++it_tile) {
      const SwOut o = sw_out_of(p, T);
      if (GS) {
        int pi, lt;
        sw_tile_of(p, T / p.rtiles, pi, lt);
        // this lane's column: its projection, its place in the permuted scale rows
        const int r64 = col & 63, sp_i = PAIR ? col >> 6 : pi;
        const int blk = PAIR ? lt : lt * 2 + (col >> 6);
        const int N = p.proj[sp_i].N;
        const bool valid = blk * 64 < N;
        const __half* sc = p.proj[sp_i].S + (size_t)kb0 * N + (valid ? blk * 64 : 0) + 8 * (r64 & 7) + (r64 >> 3);
        float acc[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[e] = 0.f;
        __half nxt[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) nxt[j] = j < KB ? __ldg(sc + (size_t)j * N) : __float2half(0.f);
        for (int kb = 0; kb < KB; kb += 4) {
          float cur[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            cur[j] = __half2float(nxt[j]);
            if (kb + 4 + j < KB) nxt[j] = __ldg(sc + (size_t)(kb + 4 + j) * N);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (kb + j < KB) {
              if (!timed_out && !tc_mbar_wait(bar_empty + 8 * s, ph)) timed_out = true;
              tc_fence_after();
              uint32_t r[16];
              sw_ld16(lane_base + s * 16, r);
              sw_wait_ld();
              tc_fence_before();
              __syncwarp();
              if (lane == 0) tc_mbar_arrive(bar_acc_empty + 8 * s);
              if (++s == p.nst) { s = 0; ph ^= 1; }
#pragma unroll
              for (int e = 0; e < 16; ++e) acc[e] = fmaf(__uint_as_float(r[e]), cur[j], acc[e]);
            }
        }
        emit(o, 0, acc, park(), etid);
      } else {
        const int buf = p.nbuf == 2 ? (it_tile & 1) : 0;
        const int use = p.nbuf == 2 ? it_tile >> 1 : it_tile;
        if (!timed_out && !tc_mbar_wait(bar_tmem_full + 8 * buf, use & 1)) timed_out = true;
        tc_fence_after();
        const int rows = min(p.Mb, p.M - o.row0);
        for (int c0 = 0; c0 < rows; c0 += RC)
          drain(o, lane_base + buf * p.nissue * p.Mb, c0);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(bar_tmem_empty + 8 * buf);
      }
    }
  } else {
    // ------------------------------------------------------------------ dequantise into tensor memory
    // A lane of the packed layout holds, per word j, the half2 pairs (n = 16j+g | 16j+g+8) x (k = 2c.. | 2c+8..):
    // exactly the register fragment of tcgen05.st.16x128b (register 2i -> lane g, column 4i+c; 2i+1 -> lane g+8).  Warp
    // quarter q owns tensor-memory lanes 32q..32q+31 = columns 32q.. of the tile = 64-column block q/2, words 2(q%2) + {0, 1}.
    const int dw = warp - FIRST_DEQ_WARP;
    const int set = dw / DEQ_WARPS;
    const int q = warp & 3;
    const int blk_local = q >> 1;
    const int g = lane >> 2;
    // Where this warp's scales of tile T start (null for a 64-column block past the projection's width), and the distance
    // between the k-blocks it converts; looked up when the tile changes, not per stage: this loop is issue-bound.
    int64_t s_step = 0;
    auto scales_of = [&](int T) -> const uint2* {
      int pi, lt;
      sw_tile_of(p, T / p.rtiles, pi, lt);
      const SwapProj& pr = p.proj[PAIR ? blk_local : pi];
      const int blk = PAIR ? lt : lt * 2 + blk_local;
      s_step = (int64_t)p.nsets * (pr.N >> 2);
      if (blk >= (pr.N >> 6)) return nullptr;
      return reinterpret_cast<const uint2*>(pr.S + (size_t)kb0 * pr.N + blk * 64 + g * 8) + (q & 1);
    };
    const uint2 kNoScale = make_uint2(0, 0);
    int s = set, sp = set;
    uint32_t ph = 0, pph = 0;
    int kb = set;                               // k-block inside the current tile
    int T = tile0;
    const uint2* sptr = nullptr;                // scales of k-block kb of tile T
    uint2 snext = kNoScale;
    auto seek = [&]() {                         // first tile in which the set has a k-block left, and that k-block's scales
      while (kb >= KB && T < p.ntiles) { kb -= KB; T += tile_step; }
      if (GS || T >= p.ntiles) return;
      sptr = scales_of(T);
      if (sptr) sptr += (size_t)kb * (s_step / p.nsets);
      snext = sptr ? __ldg(sptr) : kNoScale;
    };
    if (set < p.nsets) seek();
    // A barrier's parity tells a phase from the one before it only, so a set may never wait for a phase while the phase
    // two before it is the last one known to be complete.  Stages: the set's previous wait saw the MMAs of k-block
    // it - nsets - nst complete, in order, which covers it - 2 nst because nst >= nsets.  Packed slots fill out of order, so
    // each slot belongs to one set: pst is a multiple of nsets.
    while (T < p.ntiles && set < p.nsets) {
      uint32_t sdup[4];
      kb += p.nsets;
      if (!GS) {
        sdup[0] = __byte_perm(snext.x, 0, 0x1010);   // word j0:   columns 16 j0 + g
        sdup[1] = __byte_perm(snext.x, 0, 0x3232);   //            columns 16 j0 + g + 8
        sdup[2] = __byte_perm(snext.y, 0, 0x1010);   // word j0+1
        sdup[3] = __byte_perm(snext.y, 0, 0x3232);
      }
      if (kb >= KB) {
        seek();
      } else if (!GS && sptr) {
        sptr += s_step;
        snext = __ldg(sptr);
      }
      if (!timed_out && !tc_mbar_wait(bar_full_p + 8 * sp, pph)) timed_out = true;
      const uint32_t pk = sbase + OFF_P + sp * P_BYTES + blk_local * P_BLK + lane * 16 + (q & 1) * 8;
      uint32_t wq[8][2];
#pragma unroll
      for (int kt = 0; kt < 8; ++kt)
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(wq[kt][0]), "=r"(wq[kt][1]) : "r"(pk + kt * 512) : "memory");
      if (!timed_out && !tc_mbar_wait(bar_empty + 8 * s, ph ^ 1)) timed_out = true;
      tc_fence_after();
#pragma unroll
      for (int hk = 0; hk < 2; ++hk) {            // the two 64-k halves of the stage: packed rows 4 hk .. 4 hk + 3
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
          uint32_t r[16];
#pragma unroll
          for (int kt = 0; kt < 4; ++kt) {
            const uint32_t qw = wq[4 * hk + kt][jj], qs = qw >> 8;
            r[4 * kt + 0] = nib_pair_to_half2_m8(qw);                   // n = 16j+g,   k = 16kt + 2c, 2c+1
            r[4 * kt + 1] = nib_pair_to_half2_m8(qs);                   // n = 16j+g+8, k = 16kt + 2c, 2c+1
            r[4 * kt + 2] = nib_pair_hi_to_half2_m8(qw);                // n = 16j+g,   k = 16kt + 2c+8, 2c+9
            r[4 * kt + 3] = nib_pair_hi_to_half2_m8(qs);                // n = 16j+g+8, k = 16kt + 2c+8, 2c+9
            if (!GS) {
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const __half2 h = __hmul2(*reinterpret_cast<const __half2*>(&r[4 * kt + e]),
                                          *reinterpret_cast<const __half2*>(&sdup[2 * jj + (e & 1)]));
                r[4 * kt + e] = *reinterpret_cast<const uint32_t*>(&h);
              }
            }
          }
          const uint32_t taddr = tmem_base + ((uint32_t)(q * 32 + jj * 16) << 16) + tmem_w0 + s * (BK / 2) + hk * 32;
          asm volatile(
              "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], "
              "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
              ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
              : "memory");
        }
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      // One warp barrier in front of both arrives.  The packed slot goes back here, where the stores above have consumed
      // every lane's words, and not right behind its loads: there the arrive overtook loads still in flight, with a warp
      // barrier in between too (256 rows, 19008 x 5120: wrong values where TMA refilled the slot under a reader).
      __syncwarp();
      if (lane == 0) {
        tc_mbar_arrive(bar_full + 8 * s);
        tc_mbar_arrive(bar_empty_p + 8 * sp);
      }
      s += p.nsets;
      if (s >= p.nst) { s -= p.nst; ph ^= 1; }
      sp += p.nsets;
      if (sp >= p.pst) { sp -= p.pst; pph ^= 1; }
    }
  }

  if (!GS && p.one_tile && warp >= FIRST_EPI_WARP && tile0 < p.ntiles) {
    // A CTA with a single tile has no next main loop to hide its epilogue behind, and its dequantise warps are idle by
    // now: all twenty warps past the producers drain the accumulator, five groups of four taking 16 rows in turn.
    const int grp = (warp - FIRST_EPI_WARP) >> 2;
    const SwOut o = sw_out_of(p, tile0);
    const int rows = min(p.Mb, p.M - o.row0);
    if (!timed_out && !tc_mbar_wait(bar_tmem_full, 0)) timed_out = true;
    tc_fence_after();
    for (int c0 = grp * RC; c0 < rows; c0 += (FINISH_THREADS / 128) * RC)
      drain(o, tmem_base + ((uint32_t)((warp & 3) * 32) << 16), c0);
  }
  if (p.split > 1) {
    // The parked tile is finished by all twenty warps past the producers (the dequantise warps are idle by now), four
    // columns of one row per thread and step.  Rank r finishes its slice of the rows: it fetches the quad from every
    // rank's shared memory, the loads in flight together, and adds in rank order, so that the sum does not depend on
    // timing.
    const bool have = warp >= FIRST_EPI_WARP && tile0 < p.ntiles;
    SwOut o;
    if (have) o = sw_out_of(p, tile0);
    uint32_t reduce_ep = 0, gather_ep = 0;
    if (TP && have) tp_epochs(o, (int)threadIdx.x - FIRST_EPI_WARP * 32, reduce_ep, gather_ep);
    __syncwarp();
    sw_cluster_sync();                          // every rank's partial tile is in its shared memory
    if (have) {
      const int ftid = (int)threadIdx.x - FIRST_EPI_WARP * 32;
      const int rows = min(p.Mb, p.M - o.row0);
      const int row0 = rows * rank / p.split, row1 = rows * (rank + 1) / p.split;
      // the sums of four adjacent columns: the quads of every rank, added in rank order
      auto sum4 = [&](int r, int c4) {
        const uint32_t off = (uint32_t)r * ROW_BYTES + c4 * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int r0 = 0; r0 < p.split; r0 += 4) {
          float4 t[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (r0 + i < p.split) {
              uint32_t remote;
              asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(xbase + off), "r"(r0 + i));
              asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
                           : "=f"(t[i].x), "=f"(t[i].y), "=f"(t[i].z), "=f"(t[i].w) : "r"(remote) : "memory");
            }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (r0 + i < p.split) { v.x += t[i].x; v.y += t[i].y; v.z += t[i].z; v.w += t[i].w; }
        }
        return v;
      };
      if (TP) {
        finish_tp(o, row0, row1, ftid, FINISH_THREADS, reduce_ep, gather_ep, sum4);
      } else if (PAIR) {
        auto sum_ranks = [&](uint32_t off) {
          float t[8], v = 0.f;
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (i < p.split) {
              uint32_t remote;
              asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(xbase + off), "r"(i));
              asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(t[i]) : "r"(remote) : "memory");
            }
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (i < p.split) v += t[i];
          return v;
        };
        const int c = ftid & 63, n = o.n0 + c;
        if (n < o.n_out) {
#pragma unroll 1
          for (int r = row0 + (ftid >> 6); r < row1; r += FINISH_THREADS / 64) {
            const uint32_t off = (uint32_t)r * ROW_BYTES + c * 4;
            const int row = o.row0 + r;
            const float v = sum_ranks(off);
            o.D[(size_t)row * o.ldd + n] = sw_value<true, true>(o, row, n, v, sum_ranks(off + 256));
          }
        }
      } else {
#pragma unroll 1
        for (int idx = ftid; idx < (row1 - row0) * 32; idx += FINISH_THREADS) {
          const int r = row0 + (idx >> 5), c4 = (idx & 31) * 4;
          sw_finish4<GS>(o, o.row0 + r, c4, sum4(r, c4));
        }
      }
    }
    __syncwarp();
    sw_cluster_sync();                          // no rank leaves while its shared memory may still be read
    if (TP && have && rank == 0) tp_advance(o, (int)threadIdx.x - FIRST_EPI_WARP * 32);
  }
  if (timed_out && p.status_word) atomicOr(p.status_word, UNIQL_STATUS_WAIT_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ------------------------------------------------------------------ host side
static int swap_env(const char* name, int dflt) {
  const char* e = getenv(name);
  return (e && *e) ? atoi(e) : dflt;
}

typedef void (*SwapKernel)(const SwapParams, const CUtensorMap, const SwapMaps);
static SwapKernel swap_kernel(bool gs, bool pair, bool tp) {
  if (tp) return pair ? w4a16_gemm_swap_kernel<true, true, true> : w4a16_gemm_swap_kernel<true, false, true>;
  if (gs) return pair ? w4a16_gemm_swap_kernel<true, true, false> : w4a16_gemm_swap_kernel<true, false, false>;
  return w4a16_gemm_swap_kernel<false, false, false>;
}

// Clusters of `split` CTAs that can be resident together (0 if the query fails).
static int swap_max_clusters(bool gs, int split, int smem) {
  static thread_local int cache[64][2][9][2];   // [device][kernel][split] -> {smem the answer is for, answer}
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || split < 1 || split > 8) return 0;
  int* slot = cache[dev][gs ? 1 : 0][split];
  if (slot[0] == smem) return slot[1];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(split * 64));
  cfg.blockDim = dim3(sw::THREADS);
  cfg.dynamicSmemBytes = (size_t)smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, swap_kernel(gs, false, false), &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    n = 0;
  }
  slot[0] = smem;
  slot[1] = n;
  return n;
}

// Stages, accumulators and shared memory of a launch whose row tile has Mb rows.
struct SwapPlan {
  int nst, pst, nsets, nissue, nbuf, off_x, smem;
};
// min_kb: the fewest k-blocks a CTA has per tile.
static SwapPlan swap_plan(int Mb, bool gs, bool one_tile, int min_kb) {
  using namespace sw;
  SwapPlan pl;
  pl.nbuf = (!gs && !one_tile && Mb <= 128) ? 2 : 1;
  // two issuers up to 64 rows (above, the MMAs of a stage take longer than one thread needs to issue them)
  pl.nissue = (Mb <= 64 && min_kb >= 2) ? 2 : 1;
  const int acc_cols = gs ? MAX_STAGES * 16 : pl.nbuf * pl.nissue * Mb;
  pl.nst = (TMEM_COLS - acc_cols) / (BK / 2);
  if (pl.nst > MAX_STAGES) pl.nst = MAX_STAGES;
  if (pl.nissue == 2) pl.nst &= ~1;
  const int x_bytes = Mb * BK * 2;
  // the packed ring keeps the HBM stream in flight: at least four stages
  while (pl.nst > 2 && OFF_P + 4 * P_BYTES + pl.nst * x_bytes + 1024 > SMEM_MAX) --pl.nst;
  pl.nsets = pl.nst < NSETS ? pl.nst : NSETS;
  pl.pst = (SMEM_MAX - 1024 - OFF_P - pl.nst * x_bytes) / P_BYTES;
  if (pl.pst > MAX_PSTAGES) pl.pst = MAX_PSTAGES;
  pl.pst = pl.pst / pl.nsets * pl.nsets;
  pl.off_x = OFF_P + pl.pst * P_BYTES;
  pl.smem = pl.off_x + pl.nst * x_bytes + 1024;
  // two CTAs (each allocates all of tensor memory) must never share an SM
  if (pl.smem < 120 * 1024) pl.smem = 120 * 1024;
  return pl;
}

// What the kernel's barriers, tensor-memory columns and shared memory rely on.
static bool swap_plan_ok(const SwapPlan& pl, int Mb, bool gs) {
  using namespace sw;
  const int acc_cols = gs ? pl.nst * 16 : pl.nbuf * pl.nissue * Mb;
  return Mb >= 16 && Mb <= MB_MAX && Mb % 16 == 0 && pl.nst >= 2 && pl.nst <= MAX_STAGES && pl.nsets >= 1 && pl.nsets <= NSETS &&
         pl.nst >= pl.nsets && pl.nst % pl.nissue == 0 && pl.pst >= pl.nsets && pl.pst <= MAX_PSTAGES && pl.pst % pl.nsets == 0 &&
         acc_cols + pl.nst * (BK / 2) <= TMEM_COLS && pl.off_x % 1024 == 0 && pl.off_x >= OFF_P + pl.pst * P_BYTES &&
         pl.off_x + pl.nst * Mb * BK * 2 + 1024 <= pl.smem && pl.smem <= SMEM_MAX &&
         Mb * ROW_BYTES <= pl.nst * Mb * BK * 2;
}

// Row tiles and k-split of a launch: the cheapest of a few by a model of its cycles.  A stage (128 columns x Mb rows x
// 128 k) takes 4 Mb cycles of the tensor pipe, but no less than ~430 of the dequantise warps; a wave of tiles whose
// epilogue has no second accumulator to hide behind adds ~20 cycles a row; a cluster sum ~3000.  14336 x 4096, 160 rows:
// 628 cycles a stage measured (640 by the pipe), 224 rows 865 (896); above 224 rows the activation ring has room for two
// stages only: 256 rows 1153 (1024).
static int swap_forced_split() {
  static const int forced = swap_env("UNIQL_B200_TC_SPLIT", 0);
  return forced;
}
struct SwapShape {
  int rtiles, Mb, split;
  double cycles;
};
// forced > 0: that k-split instead (the largest possible one where it is too large), for tests and profiling.
static SwapShape swap_shape(int64_t m, int64_t k, int ctiles, bool gs, int forced) {
  using namespace sw;
  const int sms = device_info().sm_count;
  const int groups = (int)(k / 128);
  forced = min(forced, min(8, groups));
  SwapShape best{};
  best.cycles = 1e30;
  const int rt0 = (int)((m + MB_MAX - 1) / MB_MAX), rt1 = m <= 128 ? 1 : rt0 + 2;
  for (int rt = rt0; rt <= rt1; ++rt) {
    const int Mb = (int)(((m + rt - 1) / rt + 15) / 16 * 16);
    if ((int64_t)(rt - 1) * Mb >= m) continue;
    const int64_t tiles = (int64_t)ctiles * rt;
    const double stage = Mb > 224 ? 4.5 * Mb : Mb > 107 ? 4.0 * Mb : 430.0;
    for (int split = 1; split <= 8; ++split) {
      if (forced > 0 ? split != forced : (split > 1 && (tiles * split > sms || groups / split < 4)))
        continue;
      // every cluster must be resident at once (a second wave would cost more than the split gains): clusters are placed
      // inside one GPC, so fewer fit than SMs / split suggests
      if (split > 1 && forced <= 0 &&
          swap_max_clusters(gs, split, swap_plan(Mb, gs, true, groups / split).smem) < tiles)
        continue;
      const int64_t waves = split > 1 ? 1 : (tiles + sms - 1) / sms;
      const double epi = (Mb > 128 || waves == 1) ? 20.0 * Mb : 0.0;
      const double cycles = waves * (((groups + split - 1) / split) * stage + epi) + (split > 1 ? 3000.0 : 0.0);
      if (cycles < best.cycles) { best.cycles = cycles; best.rtiles = rt; best.Mb = Mb; best.split = split; }
    }
  }
  return best;
}

// The model's figure for a launch of `ctiles` 128-column tiles (the kernel's attributes must have been set: see there).
static int swap_set_attributes(bool gs, bool pair, bool tp);
double gemm_swap_cycles(int64_t m, int64_t k, int ctiles) {
  if (swap_set_attributes(m <= 16, false, false) != UNIQL_OK) return 1e30;
  return swap_shape(m, k, ctiles, m <= 16, swap_forced_split()).cycles;
}

SwapGrid gemm_swap_grid(int64_t m, int64_t k, int ctiles) {
  const bool gs = m <= 16;
  if (swap_set_attributes(gs, false, false) != UNIQL_OK) return SwapGrid{0, 0, 0};
  const SwapShape s = swap_shape(m, k, ctiles, gs, swap_forced_split());
  if (s.split < 1) return SwapGrid{0, 0, 0};
  const int sms = device_info().sm_count, groups = (int)(k / 128);
  return SwapGrid{s.split > 1 ? 1 : (ctiles * s.rtiles + sms - 1) / sms, s.split, (groups + s.split - 1) / s.split};
}

bool gemm_swap_supported(int64_t m, int64_t k, const int64_t* n, int nproj) {
  if (m < 1 || k % 128 || nproj < 1 || nproj > kMaxProj) return false;
  for (int i = 0; i < nproj; ++i)
    if (n[i] < 128 || n[i] % 64) return false;
  return true;
}

// Function attributes are per device; the occupancy query behind the k-split needs them too (always on the plain kernel).
static int swap_set_attributes(bool gs, bool pair, bool tp) {
  static thread_local bool set[64][8] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  for (int own = 0; own < 2; ++own) {
    const bool pr = own && pair, t = own && tp;
    bool& done = set[dev][(gs ? 4 : 0) + (pr ? 2 : 0) + (t ? 1 : 0)];
    if (done) continue;
    UNIQL_CUDA_TRY(cudaFuncSetAttribute(swap_kernel(gs, pr, t), cudaFuncAttributeMaxDynamicSharedMemorySize, sw::SMEM_MAX));
    done = true;
  }
  return UNIQL_OK;
}

int launch_gemm_swap(const SwapArgs& a, cudaStream_t stream) {
  using namespace sw;
  if (a.nproj < 1 || a.nproj > kMaxProj) return UNIQL_EINVAL;
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return cuda_fail(cudaErrorNotSupported);
  const int64_t m = a.m, k = a.projs[0].k;
  SwapParams p;
  memset(&p, 0, sizeof(p));
  SwapMaps wmaps;
  p.pair = a.pair ? 1 : 0;
  int ctiles = 0;
  for (int i = 0; i < a.nproj; ++i) {
    const LinearArgs& q = a.projs[i];
    if (q.k != k || q.n < 64 || q.n % 64) return UNIQL_ESHAPE;
    const int st = cached_weight_map(&wmaps.w[i], q.B, q.n, k / 16);
    if (st != UNIQL_OK) return st;
    p.proj[i].S = (const __half*)q.s; p.proj[i].bias = (const __half*)q.bias; p.proj[i].D = (__half*)a.Ds[i];
    p.proj[i].ldd = q.ldd; p.proj[i].N = (int)q.n; p.proj[i].n_out = (int)q.n_out;
    p.tile_start[i] = ctiles;
    if (a.pair) ctiles = (int)(q.n / 64);
    else ctiles += (int)((q.n + BNW - 1) / BNW);
  }
  if (a.pair) p.tile_start[0] = p.tile_start[1] = 0;
  for (int i = a.nproj; i <= kMaxProj; ++i) p.tile_start[i] = ctiles;
  for (int i = a.nproj; i < kMaxProj; ++i) { wmaps.w[i] = wmaps.w[0]; p.proj[i] = p.proj[0]; }
  p.nproj = a.nproj;
  p.residual = (const __half*)a.residual; p.ldr = a.ldr;
  const bool gs = m <= 16;
  if (!gs && (a.pair || a.residual || a.comm)) return UNIQL_ESHAPE;   // plain outputs only
  if (a.comm) {
    if (a.comm->reduce && (a.nproj != 1 || a.pair)) return UNIQL_EINVAL;
    p.cv = *a.comm;
  }
  {
    const int st = swap_set_attributes(gs, a.pair, a.comm != nullptr);
    if (st != UNIQL_OK) return st;
  }
  const SwapShape shape = swap_shape(m, k, ctiles, gs, swap_forced_split());
  if (shape.split < 1) return UNIQL_ESHAPE;
  const int Mb = shape.Mb, split = shape.split, sms = device_info().sm_count;
  p.M = (int)m; p.Mb = Mb; p.K = (int)k;
  p.rtiles = shape.rtiles;
  p.ntiles = ctiles * p.rtiles;
  p.status_word = a.projs[0].status_word;
  p.early_weights = a.early_weights ? 1 : 0;
  for (int i = 0; i < a.nprefetch && i < 4; ++i)
    if (a.prefetch_ptr[i] && a.prefetch_bytes[i] >= 128) {
      p.pf_ptr[p.npf] = (const unsigned char*)a.prefetch_ptr[i];
      p.pf_lines[p.npf] = (long long)(a.prefetch_bytes[i] / 128);
      ++p.npf;
    }
  CUtensorMap xmap;
  {
    // [k / 64][rows][64 k]: one box brings both swizzled 64-k sub-tiles of a stage
    cuuint64_t dims[3] = {64, (cuuint64_t)m, (cuuint64_t)(k / 64)};
    cuuint64_t strides[2] = {(cuuint64_t)a.lda * 2, 128};
    cuuint32_t box[3] = {64, (cuuint32_t)Mb, 2};
    cuuint32_t estr[3] = {1, 1, 1};
    if (enc(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<__half*>(a.A), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return cuda_fail(cudaErrorInvalidValue);
  }
  p.split = split;
  p.one_tile = split > 1 || p.ntiles <= sms;
  const SwapPlan pl = swap_plan(Mb, gs, p.one_tile != 0, (int)(k / 128) / split);
  if (!swap_plan_ok(pl, Mb, gs)) return UNIQL_ESHAPE;
  p.nst = pl.nst; p.pst = pl.pst; p.nsets = pl.nsets; p.nissue = pl.nissue; p.nbuf = pl.nbuf; p.off_x = pl.off_x;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = split == 1 ? dim3((unsigned)(p.ntiles < sms ? p.ntiles : sms)) : dim3((unsigned)(p.ntiles * split));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = (size_t)pl.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int nattr = 0;
  // May start behind its predecessor; the kernel waits (griddepcontrol.wait) before it reads the activations, and before it
  // reads weights and scales too unless the caller rules out that the predecessor wrote them.
  static const int pdl_on = swap_env("UNIQL_B200_PDL", 1);
  if (pdl_on && m <= 128) {
    attr[nattr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[nattr].val.programmaticStreamSerializationAllowed = 1;
    ++nattr;
  }
  if (split > 1) {
    attr[nattr].id = cudaLaunchAttributeClusterDimension;
    attr[nattr].val.clusterDim.x = (unsigned)split;
    attr[nattr].val.clusterDim.y = 1;
    attr[nattr].val.clusterDim.z = 1;
    ++nattr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = nattr;
  UNIQL_CUDA_TRY(cudaLaunchKernelEx(&cfg, swap_kernel(gs, a.pair, a.comm != nullptr), p, xmap, wmaps));
  return launch_status();
}

}  // namespace uniql

// Host-only check (no device work): every row tile this kernel can be launched with gets a plan that its barriers, tensor
// memory and shared memory can hold, and every launch gets row tiles that cover its rows and a k-split, whatever split is
// asked for.  0, or the row-tile size whose plan fails, or 1000 + the scale groups of a launch without a shape.
extern "C" int uniql_w4a16_swap_plan_check(void) {
  for (int Mb = 16; Mb <= uniql::sw::MB_MAX; Mb += 16)
    for (int one = 0; one < 2; ++one)
      for (int gs = 0; gs <= (Mb == 16 ? 1 : 0); ++gs)
        for (int kb = 1; kb <= 2; ++kb)
          if (!uniql::swap_plan_ok(uniql::swap_plan(Mb, gs != 0, one != 0, kb), Mb, gs != 0)) return Mb;
  for (int groups : {1, 2, 3, 8, 9, 112})
    for (int m : {5, 64, 256, 257, 4096})
      for (int forced : {0, 1, 3, 8, 9, 64}) {
        const uniql::SwapShape sh = uniql::swap_shape(m, (int64_t)groups * 128, 8, m <= 16, forced);
        const bool covers = sh.Mb >= 16 && sh.Mb <= uniql::sw::MB_MAX && sh.Mb % 16 == 0 &&
                            (int64_t)sh.rtiles * sh.Mb >= m && (int64_t)(sh.rtiles - 1) * sh.Mb < m;
        if (!covers || sh.split < 1 || sh.split > 8 || sh.split > groups) return 1000 + groups;
      }
  return 0;
}
