// Prefill-regime W4A16 linear for sm_100a: tcgen05 tensor cores with the accumulator in TMEM and the int4 -> fp16
// dequantisation done on the SM in front of the MMA, on 256 x 256 tiles.  Also the dispatch between this kernel and the
// operand-swapped one (w4a16_gemm_swap.cu) for more than 16 rows.
//
// Replaces the large-batch instantiations of UniQL's Marlin kernel (csrc/linear/marlin_gemm_kernel.cuh:176-740,
// tile table :802-810), which run mma.sync with dequantisation on the same warps, while consuming the same
// packed buffers (quantize/quantize_helpers.py:145-165 weight order, :54-62 scale order).
//
// w4a16_gemm_tc_kernel.  Tile: 256 batch rows x 256 output columns x 64 k per pipeline stage, one persistent CTA per SM.
// The two 128-row halves are separate M=128 MMAs that read the same dequantised weight tile, which halves the
// dequantisation work and the shared-memory writes per tensor-core cycle; their accumulators are the two 256-column
// halves of TMEM.
//   warp 0      TMA producer: activation tile(s) [128 x 64] fp16 (128B-swizzled, K-major); no multicast.
//   warp 1      allocates TMEM (2 x 256 fp32 columns); one elected lane issues, per stage, one block of
//               tcgen05.mma kind::f16 (M=128, N=256, K=16) + the commit that releases the stage + a poll of the next
//               stage's barrier whose latency hides behind the MMA issue.
//   warps 2..9  epilogue (4 per 128-row half): tcgen05.ld (32 lanes x 32 columns), + bias, fp32 -> fp16, row-major
//               stores.
//   16 warps    dequantise, as two sets of eight that convert alternate stages so two stages are always in
//               conversion: packed words straight from global memory into registers (requested two stages ahead,
//               no hop through shared memory), exact (q - 8) in fp16 via LOP3 + HSUB2/HFMA2, one HMUL2 by the group
//               scale (bit-identical to the reference's dequantised weight), 32-bit stores into the K-major
//               128B-swizzled B tile (bank-conflict free), fence.proxy.async, arrive.
// One barrier per stage collects both the TMA bytes of the activation tile and the arrivals of the dequantise warps, so
// the issuing thread pays one wait per stage.
// Roofline: tensor pipe (2*m*n*k flops); algorithmic bytes k*n/2 + (k/128)*n*2 + m*k*2 + m*n*2.
// Every mbarrier wait is bounded; a wait that gives up sets UNIQL_STATUS_WAIT_TIMEOUT and the kernel drains.
#include "common.cuh"
#include "linear_internal.cuh"
#include "tc.cuh"

#include <cuda.h>
#include <stdlib.h>
#include <string.h>

namespace uniql {

namespace tc {
constexpr int BMH = 128, BN = 256, BK = 64;   // BMH: rows of one MMA (one "half")
constexpr int A_BYTES = BMH * BK * 2;         // 16 KB per half
constexpr int B_BYTES = BN * BK * 2;          // 32 KB
constexpr int DEQ_SETS = 2;                   // dequantise warp sets; set t converts k-blocks t, t + 2, ...
constexpr int DEQ_SET_WARPS = 8;              // per set: 4 column blocks x 2 pairs of packed rows
constexpr int DEQ_WARPS = DEQ_SETS * DEQ_SET_WARPS;
constexpr int TMEM_COLS = 512;
constexpr int H = 2;                          // 128-row halves of a tile
constexpr int AB_STAGES = 3;
constexpr int STAGE_A = H * A_BYTES;
constexpr int OFF_A = 0;
constexpr int OFF_B = OFF_A + AB_STAGES * STAGE_A;
constexpr int OFF_BAR = OFF_B + AB_STAGES * B_BYTES;
constexpr int NUM_BARS = 2 * AB_STAGES + 4;
constexpr int SMEM_BYTES = OFF_BAR + NUM_BARS * 8 + 16 + 1024;   // + slack to align the base to 1 KB
constexpr int FIRST_EPI_WARP = 2;
constexpr int EPI_WARPS = 4 * H;
constexpr int FIRST_DEQ_WARP = FIRST_EPI_WARP + EPI_WARPS;
constexpr int THREADS = (FIRST_DEQ_WARP + DEQ_WARPS) * 32;
// instruction descriptor: D fp32, A/B fp16, both K-major, N = 256, M = 128
constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BMH >> 4) << 24);
}  // namespace tc

struct TcParams {
  const uint4* B;        // packed weights [K/16][2N] words
  const uint4* S;        // permuted scales, row g has n/8 uint4
  const __half* bias;
  __half* D;
  int64_t ldd;
  int M, N, n_out, K;
  int mtiles, ntiles;
  int* status_word;
};

// All MMAs of one 64-k stage (four K=16 steps for each 128-row half), the commit that releases the stage, and one poll
// of the NEXT stage's barrier, in one block: the poll is issued first and its result read last, so its latency hides
// behind the issue of the MMAs instead of adding to the single issuing thread's serial time per stage.  Returns
// whether the next stage was already full.
__device__ __forceinline__ uint32_t tc_issue_stage(uint32_t tmem_d, uint64_t adesc0, uint64_t adesc1, uint64_t bdesc,
                                                   uint32_t accumulate, uint32_t bar_release, uint32_t bar_next,
                                                   uint32_t par_next) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q, t;\n\t.reg .b64 a1, a2, a3, c1, c2, c3, b1, b2, b3;\n\t.reg .b32 d1;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%8], %9;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "add.u32 d1, %1, 256;\n\t"
      "add.u64 a1, %2, 2;\n\tadd.u64 a2, %2, 4;\n\tadd.u64 a3, %2, 6;\n\t"
      "add.u64 c1, %3, 2;\n\tadd.u64 c2, %3, 4;\n\tadd.u64 c3, %3, 6;\n\t"
      "add.u64 b1, %4, 2;\n\tadd.u64 b2, %4, 4;\n\tadd.u64 b3, %4, 6;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], %2, %4, %5, p;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], a1, b1, %5, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], a2, b2, %5, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], a3, b3, %5, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [d1], %3, %4, %5, p;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [d1], c1, b1, %5, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [d1], c2, b2, %5, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [d1], c3, b3, %5, t;\n\t"
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(ok)
      : "r"(tmem_d), "l"(adesc0), "l"(adesc1), "l"(bdesc), "r"(tc::IDESC), "r"(accumulate), "r"(bar_release),
        "r"(bar_next), "r"(par_next)
      : "memory");
  return ok;
}

__global__ void __launch_bounds__(tc::THREADS, 1)
w4a16_gemm_tc_kernel(const TcParams p, const __grid_constant__ CUtensorMap amap) {
  using namespace tc;
  static_assert(BN == 256, "the second accumulator sits 256 tensor-memory columns after the first");
  extern __shared__ uint8_t smem_unaligned[];
  // 1 KB alignment: the 128B-swizzled tiles must start on a swizzle-atom boundary
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = tc_smem_addr(smem);
  const uint32_t bars = sbase + OFF_BAR;
  // full[s]: the activation tile has landed (TMA bytes) AND one set's warps have written the weight tile;
  // empty[s]: the MMAs that read stage s have completed
  const uint32_t bar_full = bars, bar_empty_ab = bars + 8 * AB_STAGES;
  const uint32_t bar_tmem_full = bars + 16 * AB_STAGES, bar_tmem_empty = bar_tmem_full + 16;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + OFF_BAR + NUM_BARS * 8);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KB = p.K / BK;
  const int total_tiles = p.mtiles * p.ntiles;
  const int my_tiles = ((int)blockIdx.x < total_tiles) ? (total_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const int total_it = my_tiles * KB;

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&amap) : "memory");
    for (int s = 0; s < AB_STAGES; ++s) {
      tc_mbar_init(bar_full + 8 * s, 1 + DEQ_SET_WARPS);
      tc_mbar_init(bar_empty_ab + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc_mbar_init(bar_tmem_full + 8 * b, 1);
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

  if (warp == 0) {
    // ------------------------------------------------------------------ activation producer
    if (tc_elect()) {
      int it_ab = 0;
      for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
        const int mt = tile % p.mtiles;
        for (int kb = 0; kb < KB; ++kb, ++it_ab) {
          const int s = it_ab % AB_STAGES;
          if (!timed_out && !tc_mbar_wait(bar_empty_ab + 8 * s, ((it_ab / AB_STAGES) & 1) ^ 1)) timed_out = true;
          tc_mbar_expect_tx(bar_full + 8 * s, STAGE_A);
#pragma unroll
          for (int h = 0; h < H; ++h)
            tc_tma_2d(sbase + OFF_A + s * STAGE_A + h * A_BYTES, &amap, kb * BK, (mt * H + h) * BMH, bar_full + 8 * s);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (tc_elect()) {
      int it_ab = 0, it_tile = 0;
      uint32_t ready = 0;                        // the current stage's full barrier was seen complete by the last poll
      for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++it_tile) {
        const uint32_t empty_parity = (it_tile & 1) ^ 1;
#pragma unroll
        for (int h = 0; h < H; ++h)
          if (!timed_out && !tc_mbar_wait(bar_tmem_empty + 8 * h, empty_parity)) timed_out = true;
        tc_fence_after();
        for (int kb = 0; kb < KB; ++kb, ++it_ab) {
          const int s = it_ab % AB_STAGES;
          if (!ready && !timed_out && !tc_mbar_wait(bar_full + 8 * s, (it_ab / AB_STAGES) & 1)) timed_out = true;
          tc_fence_after();
          const int s1 = (s + 1 == AB_STAGES) ? 0 : s + 1;
          const uint64_t adesc0 = tc_smem_desc(sbase + OFF_A + s * STAGE_A);
          ready = tc_issue_stage(tmem_base, adesc0, adesc0 + (A_BYTES >> 4),
                                    tc_smem_desc(sbase + OFF_B + s * B_BYTES), kb != 0 ? 1u : 0u, bar_empty_ab + 8 * s,
                                    bar_full + 8 * s1, ((it_ab + 1) / AB_STAGES) & 1);
          if (it_ab + 1 >= total_it) ready = 0;   // that poll looked at a phase nobody will complete
        }
#pragma unroll
        for (int h = 0; h < H; ++h) tc_commit(bar_tmem_full + 8 * h);   // accumulators complete
      }
    }
  } else if (warp < FIRST_DEQ_WARP) {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;                     // TMEM lane quadrant this warp may access
    const int half = (warp - FIRST_EPI_WARP) >> 2;   // which 128-row half of the tile 
    int it_tile = 0;
    const bool vec_ok = ((p.ldd & 7) == 0) && ((reinterpret_cast<uintptr_t>(p.D) & 15u) == 0);
    for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++it_tile) {
      const int mt = tile % p.mtiles, nt = tile / p.mtiles;
      const int buf = half;
      const uint32_t full_parity = it_tile & 1;
      if (!timed_out && !tc_mbar_wait(bar_tmem_full + 8 * buf, full_parity)) timed_out = true;
      tc_fence_after();
      const int m = (mt * H + half) * BMH + q * 32 + lane;
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * BN;
      __half* drow = p.D + (size_t)m * p.ldd;
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += 32) {
        uint32_t r[32];
        tc_ld32(taddr + c0, r);
        const int n0 = nt * BN + c0;
        if (m < p.M && n0 < p.n_out) {
          if (vec_ok && n0 + 32 <= p.n_out) {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint32_t pk[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                float f0 = __uint_as_float(r[8 * v + 2 * e]), f1 = __uint_as_float(r[8 * v + 2 * e + 1]);
                if (p.bias) {
                  f0 += __half2float(p.bias[n0 + 8 * v + 2 * e]);
                  f1 += __half2float(p.bias[n0 + 8 * v + 2 * e + 1]);
                }
                __half2 h = __floats2half2_rn(f0, f1);
                pk[e] = *reinterpret_cast<uint32_t*>(&h);
              }
              *reinterpret_cast<uint4*>(drow + n0 + 8 * v) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            }
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (n0 + e < p.n_out) {
                float f = __uint_as_float(r[e]);
                if (p.bias) f += __half2float(p.bias[n0 + e]);
                drow[n0 + e] = __float2half_rn(f);
              }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(bar_tmem_empty + 8 * buf);
    }
  } else {
    // ------------------------------------------------------------------ dequantise
    // Two sets of eight warps convert alternate k-blocks, so that two stages are in conversion at any time: what
    // bounds this path is the latency of one warp's chain per stage (barrier polls, packed-word read, convert, store,
    // proxy fence, arrive), not its instruction count.
    const int dw = warp - FIRST_DEQ_WARP;
    const int set = dw / DEQ_SET_WARPS;
    const int blk_local = dw & 3;               // 64-column block of the 256-column tile
    const int kt0 = ((dw >> 2) & 1) * 2;        // this warp's two packed rows of the stage: k = 16 kt0 .. 16 kt0 + 31
    const int g = lane >> 2, c = lane & 3;
    const int nblk = p.N >> 6;
    const uint32_t srow_u4 = (uint32_t)(p.N >> 3);
    const uint4* sbase_g = p.S + g;
    // position of the k-block this warp converts next, and of the one after it (whose scales are requested early)
    int ti = 0, kb = set;
    while (kb >= KB && ti < my_tiles) { kb -= KB; ++ti; }
    int ti2 = ti, kb2 = kb + DEQ_SETS;
    while (kb2 >= KB && ti2 < my_tiles) { kb2 -= KB; ++ti2; }
    // The packed words come straight from global memory into registers (512 contiguous bytes per warp and packed
    // row), requested one iteration = two k-blocks ahead like the scales: a hop through shared memory would add a
    // barrier wait and a read to the chain that bounds this path, and 16 KB per stage to the shared-memory traffic.
    const uint32_t prow_u4 = (uint32_t)(p.N >> 1);            // one packed row: 2N words = N/2 uint4
    const uint4* pbase = p.B + (size_t)kt0 * prow_u4 + lane;
    const uint4 kZero = make_uint4(0x88888888u, 0x88888888u, 0x88888888u, 0x88888888u);   // (8 - 8) * scale = 0
    uint4 snext = make_uint4(0, 0, 0, 0), wnext[2] = {kZero, kZero};
    if (set < total_it) {
      const int blk = (((int)blockIdx.x + ti * (int)gridDim.x) / p.mtiles) * 4 + blk_local;
      if (blk < nblk) {
        snext = ld_nc16(sbase_g + (size_t)blk * 8 + (size_t)(kb >> 1) * srow_u4);
        const uint4* src = pbase + (size_t)kb * 4 * prow_u4 + (size_t)blk * 32;
        wnext[0] = ld_nc16(src);
        wnext[1] = ld_nc16(src + prow_u4);
      }
    }
    for (int it = set; it < total_it; it += DEQ_SETS) {
      uint32_t sdup[8];                         // the lane's 8 group scales, each duplicated into a half2
      const uint4 w4[2] = {wnext[0], wnext[1]};
      {
        const uint32_t s4[4] = {snext.x, snext.y, snext.z, snext.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          sdup[2 * j] = __byte_perm(s4[j], 0, 0x1010);       // low half  -> columns 16j+g
          sdup[2 * j + 1] = __byte_perm(s4[j], 0, 0x3232);   // high half -> columns 16j+g+8
        }
        if (it + DEQ_SETS < total_it) {
          const int blk2 = (((int)blockIdx.x + ti2 * (int)gridDim.x) / p.mtiles) * 4 + blk_local;
          wnext[0] = wnext[1] = kZero;
          if (blk2 < nblk) {
            snext = ld_nc16(sbase_g + (size_t)blk2 * 8 + (size_t)(kb2 >> 1) * srow_u4);
            const uint4* src = pbase + (size_t)kb2 * 4 * prow_u4 + (size_t)blk2 * 32;
            wnext[0] = ld_nc16(src);
            wnext[1] = ld_nc16(src + prow_u4);
          }
        }
        ti = ti2; kb = kb2;
        kb2 += DEQ_SETS;
        while (kb2 >= KB && ti2 < my_tiles) { kb2 -= KB; ++ti2; }
      }
      const int s = it % AB_STAGES;
      if (!timed_out && !tc_mbar_wait(bar_empty_ab + 8 * s, ((it / AB_STAGES) & 1) ^ 1)) timed_out = true;
      const uint32_t btile = sbase + OFF_B + s * B_BYTES + (uint32_t)(blk_local * 64 + g) * 128 + 4 * c;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int kt = kt0 + u;
        const uint32_t wq[4] = {w4[u].x, w4[u].y, w4[u].z, w4[u].w};
        const uint32_t a_lo = btile + ((uint32_t)((2 * kt) ^ g) << 4), a_hi = btile + ((uint32_t)((2 * kt + 1) ^ g) << 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t qw = wq[j], qs = wq[j] >> 8;
          uint32_t v;
          __half2 r;
          v = nib_pair_to_half2_m8(qw);                               // n = 16j+g,   k = 2c, 2c+1
          r = __hmul2(*reinterpret_cast<__half2*>(&v), *reinterpret_cast<const __half2*>(&sdup[2 * j]));
          tc_sts32(a_lo + (16 * j) * 128, *reinterpret_cast<uint32_t*>(&r));
          v = nib_pair_hi_to_half2_m8(qw);                            // n = 16j+g,   k = 2c+8, 2c+9
          r = __hmul2(*reinterpret_cast<__half2*>(&v), *reinterpret_cast<const __half2*>(&sdup[2 * j]));
          tc_sts32(a_hi + (16 * j) * 128, *reinterpret_cast<uint32_t*>(&r));
          v = nib_pair_to_half2_m8(qs);                               // n = 16j+g+8, k = 2c, 2c+1
          r = __hmul2(*reinterpret_cast<__half2*>(&v), *reinterpret_cast<const __half2*>(&sdup[2 * j + 1]));
          tc_sts32(a_lo + (16 * j + 8) * 128, *reinterpret_cast<uint32_t*>(&r));
          v = nib_pair_hi_to_half2_m8(qs);                            // n = 16j+g+8, k = 2c+8, 2c+9
          r = __hmul2(*reinterpret_cast<__half2*>(&v), *reinterpret_cast<const __half2*>(&sdup[2 * j + 1]));
          tc_sts32(a_hi + (16 * j + 8) * 128, *reinterpret_cast<uint32_t*>(&r));
        }
      }
      // make the generic-proxy stores visible to the tensor core's async-proxy reads, then signal
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(bar_full + 8 * s);
    }
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
bool gemm_tc_supported(int64_t m, int64_t n, int64_t k) {
  return m > 16 && n >= 128 && n % 64 == 0 && k % 128 == 0;
}

// Which kernel runs m > 16 rows.  The 256 x 256 tiles of the kernel above reuse activations and weights twice as often as
// the 128-column tiles of the operand-swapped kernel, whose finer tiles, k-split and shared launches waste less of the
// last wave: the modelled cycles decide (a 64-k stage of a tile ~1200 cycles and ~4000 for its epilogue, against the
// other kernel's model times the 1.12 it falls short of it by).  Measured, tiles / swapped, us: 14336 x 4096 at 301 rows
// 72 (its 128-row form, since removed) / 38, 1024 rows 98 / 115, 4096 rows 363 / 421; 4096 x 14336 at 1024 rows
// 120 / 95, 4096 rows 346 / 384.
static bool prefill_tiles_win(int64_t m, int64_t n, int64_t k) {
  static const int forced = [] { const char* e = getenv("UNIQL_B200_TC_SWAP"); return (e && *e) ? atoi(e) : -1; }();
  if (forced >= 0) return forced == 0;
  if (m <= 128) return false;
  const int sms = device_info().sm_count;
  const int64_t tiles = ((m + 255) / 256) * ((n + 255) / 256);
  const double cycles = (double)((tiles + sms - 1) / sms) * (k / 64 * 1200.0 + 4000.0);
  return cycles < 1.12 * gemm_swap_cycles(m, k, (int)((n + 127) / 128));
}

int launch_gemm_tc(const LinearArgs& a, const __half* A, int64_t lda, __half* D, int64_t m, bool early_weights, cudaStream_t stream) {
  using namespace tc;
  if (!prefill_tiles_win(m, a.n, a.k)) {
    void* d1[1] = {D};
    SwapArgs sa{};
    sa.projs = &a; sa.Ds = d1; sa.nproj = 1; sa.A = A; sa.lda = lda; sa.m = m;
    sa.early_weights = early_weights;
    return launch_gemm_swap(sa, stream);
  }
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return cuda_fail(cudaErrorNotSupported);
  CUtensorMap amap;
  {
    cuuint64_t dims[2] = {(cuuint64_t)a.k, (cuuint64_t)m};
    cuuint64_t strides[1] = {(cuuint64_t)lda * 2};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)BMH};
    cuuint32_t estr[2] = {1, 1};
    if (enc(&amap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(A), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return cuda_fail(cudaErrorInvalidValue);
  }
  TcParams p;
  p.B = (const uint4*)a.B; p.S = (const uint4*)a.s; p.bias = (const __half*)a.bias; p.D = D; p.ldd = a.ldd;
  p.M = (int)m; p.N = (int)a.n; p.n_out = (int)a.n_out; p.K = (int)a.k;
  p.ntiles = (int)((a.n + BN - 1) / BN);
  p.mtiles = (int)((m + H * BMH - 1) / (H * BMH));
  p.status_word = a.status_word;
  {
    static thread_local bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!attr_set[dev]) {
      UNIQL_CUDA_TRY(cudaFuncSetAttribute(w4a16_gemm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
      attr_set[dev] = true;
    }
  }
  const int64_t tiles = (int64_t)p.mtiles * p.ntiles;
  const int sms = device_info().sm_count;
  const int grid = (int)(tiles < sms ? tiles : sms);
  w4a16_gemm_tc_kernel<<<grid, THREADS, SMEM_BYTES, stream>>>(p, amap);
  return launch_status();
}

}  // namespace uniql
