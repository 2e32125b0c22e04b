// Dense GEMM for multi-token (prefill) passes on the 5th-generation tensor cores:
// C[M,N] = A[M,K] . W[N,K]^T with fp32 accumulation in tensor memory (TMEM), A and W in FP16, W in Q8_0, or
// both in bfloat16 with the epilogues of the layer-list decoders (rows.cuh) and tiles grouped by expert.
//
// Replaces, for many rows, the reference's matmul_b0_tb_fp16_v2.comp and matmul_b0_fp16_x_q8_0.comp
// (src/ops/mat_mul.cpp:71-103), which re-read the whole weight matrix for every input row.
//
// Q8_0 weights are dequantised on the way into shared memory: sixteen extra warps, in two groups that take
// alternating K steps, fetch the codes and scales of their stage's W tile (tiled planes, common.cuh) with
// ordered asynchronous copies, turn every code into the fp16 value fp16(q * d) and store it where a
// 128-byte-swizzled tensor copy would have put it, so the MMA loop is the same as for FP16 weights.
// q * d has up to 19 significant bits: this path rounds every weight once to fp16 (relative 2^-12), where
// the reference multiplies in fp32; the mma.sync kernels (skinny_gemm.cuh, matvec.cu) keep the exact form and run
// below GEMM_Q8_MIN_ROWS rows.
//
// Long prompts of 16-bit weights go to pairs of CTAs where pick_tile finds them faster (gemm_pair.cu). Here one CTA computes
// a 128 x BN output tile (BN = 32 ... 256, picked per launch) with these kinds of warps:
//   warp 0    producer: one lane issues TMA tensor copies (cp.async.bulk.tensor.2d, 128-byte
//             swizzle) of the A and W tiles of each 64-wide K block into a ring of shared-
//             memory stages; the copies complete on the stage's "full" mbarrier.
//   warp 1    MMA: allocates the TMEM accumulator (BN columns); one lane waits for a full
//             stage and issues four tcgen05.mma (M128 N{BN} K16, kind::f16) on shared-memory
//             descriptors; tcgen05.commit arrives on the stage's "empty" mbarrier when the
//             tensor core has read the stage, and on "acc_ready" after the last K block.
//   warps 2-5, or more with 16-bit weights, epilogue: each reads its 32 TMEM lanes (= 32 output rows) with tcgen05.ld,
//             applies the op's rounding (scale, bias, SiLU, residual add) and stores fp16 or
//             raw fp32 rows with 128-bit stores.
// Every mbarrier wait is bounded; on a time-out the kernel raises the error word, lets
// copies in flight land, frees its TMEM and returns.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "rows.cuh"
#include "tcgen05.cuh"

namespace vkl {
namespace {

// 16-bit weights: TMA producer, MMA, and one, two or four epilogue warps per 32 rows, each with its share of the columns (why:
// gemm_pair.cu). Experts of 777 tokens, us per gate/up launch with 1 / 2 / 4: 72.6 / 60.7 / 55.0.
__host__ __device__ constexpr int epilogue_parts(bool rows, bool swiglu) { return rows ? 4 : swiglu ? 2 : 1; }
__host__ __device__ constexpr int gemm_threads(bool rows, bool swiglu) { return 64 + 128 * epilogue_parts(rows, swiglu); }
#ifndef VKL_GEMM_NDW
#define VKL_GEMM_NDW 16
#endif
constexpr int NDW = VKL_GEMM_NDW;               // warps dequantising the W tile: one warp issues an instruction every five cycles or so
                                                // (a dependent chain of permutes, multiplies and stores), so it takes several per SM
                                                // sub-partition to keep up with the weight stream
#ifndef VKL_GEMM_NG
#define VKL_GEMM_NG 2
#endif
constexpr int NG = VKL_GEMM_NG;                 // the dequantising warps work in NG groups on alternating K steps: a warp's pass over
                                                // one K step is a serial chain of waits, loads, conversion, stores and a proxy fence
                                                // (about half a microsecond), so several K steps have to be in work at a time
// The MMA lane (warp 1) issues some sixty instructions per K step and the whole CTA waits on it. A warp's scheduler
// is warp % 4: the dequantising warps that would share warp 1's scheduler (every fourth) are left idle, or that
// lane gets an issue slot every twenty-odd cycles and a K step takes 0.58 us instead of 0.3.
__host__ __device__ constexpr int skipped_below(int w) { return w < 9 ? 0 : (w - 9) / 4 + 1; }  // warps 9, 13, 17, ... below warp w
constexpr int NDW_ACTIVE = NDW - skipped_below(6 + NDW);                      // the launched warps 6 .. 5 + NDW, less those
constexpr int NDWG = NDW_ACTIVE / NG;           // warps per group = arrivals per stage
static_assert(NDW_ACTIVE % NG == 0, "whole groups");
constexpr int GEMM_THREADS_Q8 = 192 + 32 * NDW;

// Q8_0 weights: what a dequantising warp keeps in flight from DRAM, in shared memory (asynchronous 16-byte
// copies, waited for in order): Q8_UNITS_AHEAD units of 512 bytes of codes + 128 bytes of scales per warp.
constexpr uint32_t Q8_UNIT_STAGING = 512 + 128, Q8_UNITS_AHEAD = NDW_ACTIVE >= 16 ? 4 : 6;
constexpr uint32_t Q8_STAGING_BYTES = NDW_ACTIVE * Q8_UNITS_AHEAD * Q8_UNIT_STAGING;  // 45 KB

template <int BN, bool Q8 = false> struct Cfg {
  static constexpr uint32_t B_TILE_BYTES = BN * BK * 2;
  static constexpr uint32_t STAGE_BYTES = A_TILE_BYTES + B_TILE_BYTES;
  static constexpr int RING_BYTES = 192 * 1024 - (Q8 ? (int)Q8_STAGING_BYTES : 0);  // up to 192 KB of stages (and staging)
  static constexpr int STAGES = (RING_BYTES / (int)STAGE_BYTES) < 8 ? (RING_BYTES / (int)STAGE_BYTES) : 8;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + (Q8 ? Q8_STAGING_BYTES : 0) + 1024;
};

// One Q8_0 unit (16 rows x 32 columns, 512 bytes of codes) -> fp16 values q * d in the swizzled W tile.
// Lane (g, t) holds 8 codes of row g and 8 codes of row g + 8 at columns 8 t .. 8 t + 7 (common.cuh). 128-byte
// swizzle of a K-major tile with 128-byte rows: 16-byte chunk c of row r sits at chunk c ^ (r % 8); the two store
// offsets depend on the warp's unit, not on the K step, and are worked out beforehand.
__device__ __forceinline__ void dequant_unit_at(unsigned char *wtile, uint32_t off_a, uint32_t off_b, uint4 w, uint32_t d_lo, uint32_t d_hi) {
  const __half2 dl = __half2half2(__ushort_as_half((unsigned short)d_lo)), dh = __half2half2(__ushort_as_half((unsigned short)d_hi));
  uint32_t a[4], b[4];
  a[0] = codes_to_h2(w.x, false); a[1] = codes_to_h2(w.x, true); a[2] = codes_to_h2(w.y, false); a[3] = codes_to_h2(w.y, true);
  b[0] = codes_to_h2(w.z, false); b[1] = codes_to_h2(w.z, true); b[2] = codes_to_h2(w.w, false); b[3] = codes_to_h2(w.w, true);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    __half2 x = __hmul2(*reinterpret_cast<__half2 *>(&a[i]), dl), y = __hmul2(*reinterpret_cast<__half2 *>(&b[i]), dh);
    a[i] = *reinterpret_cast<uint32_t *>(&x);
    b[i] = *reinterpret_cast<uint32_t *>(&y);
  }
  *reinterpret_cast<uint4 *>(wtile + off_a) = make_uint4(a[0], a[1], a[2], a[3]);
  *reinterpret_cast<uint4 *>(wtile + off_b) = make_uint4(b[0], b[1], b[2], b[3]);
}

// The kernel's operands: FP16 weights, Q8_0 weights, or bfloat16 with GemmRows' epilogues.
enum GemmKind { GK_F16, GK_Q8, GK_ROWS };
template <int KIND> struct GemmArgs { using Type = GemmParams; };
template <> struct GemmArgs<GK_ROWS> { using Type = GemmRows; };

template <int BN, int KIND>
__global__ void __launch_bounds__(KIND == GK_Q8 ? GEMM_THREADS_Q8 : gemm_threads(KIND == GK_ROWS, true), 1)
    gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ WeightMaps maps, const typename GemmArgs<KIND>::Type p) {
  constexpr bool Q8 = KIND == GK_Q8;
  using C = Cfg<BN, Q8>;
  extern __shared__ unsigned char smem_raw[];
  // swizzle atoms are 1024 bytes: align the stage ring
  unsigned char *stages = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[C::STAGES];   // TMA bytes of the stage have landed
  __shared__ __align__(8) uint64_t empty[C::STAGES];  // the MMAs have read the stage
  __shared__ __align__(8) uint64_t acc_ready;
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile uint32_t failed_s;

  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // grid y: one matrix's column tiles behind the other's. SwiGLU: the first half of a W tile is gate rows, the second
  // the up rows of the same outputs.
  uint32_t mat = 0, ny = blockIdx.y;
  bool swiglu = false;
  if constexpr (KIND != GK_ROWS) {
    swiglu = p.swiglu;
    const uint32_t per = (p.N + BN - 1) / BN;
    if (!swiglu) {
      mat = ny / per;
      ny -= mat * per;
    }
  }
  const uint32_t m0 = blockIdx.x * BM, n0 = ny * (swiglu ? BN / 2 : BN);
  const uint32_t nkb = p.K / BK;
  uint32_t w_row = n0, a_row = m0;  // first weight and input row of the tile
  if constexpr (KIND == GK_ROWS) {
    if (p.n2 && n0 >= p.n2) a_row += p.M;  // rows beyond an input's M are read (the next one's, or zeros) and dropped by the epilogue
    if (p.tile_expert) {
      const int32_t e = p.tile_expert[blockIdx.x];
      if (e < 0) return;  // uniform over the CTA
      w_row += (uint32_t)e * p.N;
    }
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sa(&full[s])), "r"(Q8 ? 1u + NDWG : 1u) : "memory");  // the TMA lane (+ one lane per dequantising warp)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sa(&empty[s])) : "memory");
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sa(&acc_ready)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    failed_s = 0;
  }
  // Tiles of up to 128 columns accumulate the even and the odd 16-wide K slices in two TMEM accumulators, added in
  // the epilogue: a tcgen05.mma of so few columns takes about 110 cycles however narrow it is when it has to
  // follow the one before it on the same accumulator; two independent chains hide half of that.
  constexpr uint32_t NACC = BN <= 128 ? 2 : 1;
  if (warp == 1) tmem_alloc<NACC * BN>(sa(&tmem_base_s));
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_acc = tmem_base_s;

  if (warp == 0) {
    // ---------------------------------------------------------------- producer
    if (elect_one()) {
      RingPos<C::STAGES> pos;
      for (uint32_t kb = 0; kb < nkb; ++kb, pos.next()) {
        if (kb >= C::STAGES && !mbar_wait_bounded(sa(&empty[pos.s]), pos.phase ^ 1u)) {
          failed_s = 1;
          break;
        }
        const uint32_t bar = sa(&full[pos.s]), st = sa(stages) + pos.s * C::STAGE_BYTES;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(Q8 ? A_TILE_BYTES : C::STAGE_BYTES) : "memory");
        tma_load_2d(st, &map_a, kb * BK, a_row, bar);
        if (!Q8) tma_load_2d(st + A_TILE_BYTES, &maps.w[mat], kb * BK, w_row, bar);
        if (!Q8 && swiglu) tma_load_2d(st + A_TILE_BYTES + C::B_TILE_BYTES / 2, &maps.w[1], kb * BK, w_row, bar);
      }
    }
  } else if (Q8 && warp >= 6 && (warp & 3u) != 1u) {
    if constexpr (Q8) {
    // ------------------------------------------- W tile: Q8_0 -> fp16 in shared memory
    // BN rows x 64 columns = (BN / 16) row tiles x 2 blocks: units of 512 bytes of codes, dealt round robin to
    // the dequantising warps. The scales of a row tile and 4-block group are 8 x 16 bytes: row g's four blocks, then row g + 8's.
    const uint32_t dw = (warp - 6) - (uint32_t)skipped_below((int)warp), g = lane >> 2, t = lane & 3;  // index among the active dequantising warps
    const uint32_t grp = dw % NG, wi = dw / NG;  // this warp's group (its K steps: grp, grp + NG, ...) and place in it
    const uint32_t tiles16 = (p.N + 15) / 16, groups = ((p.K + 31) / 32 + 3) / 4;
    constexpr uint32_t UNITS = (BN / 16) * 2, UPQ = (UNITS + NDWG - 1) / NDWG;  // units per stage, and of those at most this warp's
    constexpr uint32_t PF = Q8_UNITS_AHEAD / UPQ;                              // of its own K steps, how many are requested ahead
    static_assert(UPQ <= Q8_UNITS_AHEAD && PF >= 1, "staging holds at least one stage of a warp's units");
    // The codes of a stage come from DRAM (a microsecond away), so the warp's next PF stages' units are kept in
    // flight. They travel as asynchronous copies into this warp's own staging area, which complete in order
    // (cp.async groups): loads into registers would share the warp's few scoreboards, and the wait for the oldest
    // would also wait for the youngest.
    unsigned char *stg = stages + (size_t)C::STAGES * C::STAGE_BYTES + (size_t)dw * Q8_UNITS_AHEAD * Q8_UNIT_STAGING;
    // What does not change from K step to K step is worked out once per unit of this warp: where its codes and its
    // scales start in the planes (they advance by 1024 bytes per K step and by 128 bytes per two K steps), where
    // its two stores go in the W tile (128-byte swizzle), which half of the block pair it is.
    const unsigned char *cbase[UPQ], *sbase[UPQ];
    uint32_t off_a[UPQ], off_b[UPQ], bl[UPQ];
    bool valid[UPQ];
#pragma unroll
    for (uint32_t j = 0; j < UPQ; ++j) {
      const uint32_t u = wi + NDWG * j, up = swiglu && (u >> 1) >= BN / 32 ? 1u : 0u, tile = n0 / 16 + (u >> 1) - up * (BN / 32);
      bl[j] = u & 1u;
      valid[j] = u < UNITS && tile < tiles16;
      cbase[j] = p.w_codes[mat + up] + (((size_t)tile * groups * 4 + bl[j]) * 32 + lane) * 16;
      sbase[j] = p.w_scales[mat + up] + ((size_t)tile * groups * 8 + g) * 16;
      const uint32_t ra = (u >> 1) * 16 + g, rb = ra + 8, c = bl[j] * 4 + t;
      off_a[j] = ra * 128 + ((c ^ (ra & 7)) << 4);
      off_b[j] = rb * 128 + ((c ^ (rb & 7)) << 4);
    }
    auto request = [&](uint32_t kb, uint32_t slot) {
#pragma unroll
      for (uint32_t j = 0; j < UPQ; ++j) {
        if (valid[j] && kb < nkb) {
          const uint32_t dst = sa(stg + (slot * UPQ + j) * Q8_UNIT_STAGING);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + lane * 16), "l"(cbase[j] + (size_t)kb * 1024) : "memory");
          if (t == 0)  // the 4-block group's scales of rows g and g + 8: 16 bytes
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 512 + g * 16), "l"(sbase[j] + (size_t)(kb >> 1) * 128) : "memory");
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");  // one group per stage, also when it is empty
    };
#pragma unroll
    for (uint32_t i = 0; i < PF; ++i) request(grp + NG * i, i);
    for (uint32_t kb0 = grp; kb0 < nkb; kb0 += NG * PF) {
      bool stop = false;
#pragma unroll
      for (uint32_t i = 0; i < PF; ++i) {  // staging slots are indexed by compile-time constants
        const uint32_t kb = kb0 + NG * i;
        if (kb >= nkb || stop) continue;
        const uint32_t s = kb % C::STAGES, use = kb / C::STAGES;
        uint32_t ok = 1;
        if (lane == 0 && use > 0) ok = mbar_wait_bounded(sa(&empty[s]), (use - 1) & 1u, 100) ? 1u : 0u;
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) {
          if (lane == 0) failed_s = 4;
          stop = true;
          continue;
        }
        if (failed_s) {
          stop = true;
          continue;
        }
        asm volatile("cp.async.wait_group %0;" ::"n"(PF - 1) : "memory");  // this stage's copies (the oldest group) have landed
        __syncwarp();
        unsigned char *wt = stages + (size_t)s * C::STAGE_BYTES + A_TILE_BYTES;
#pragma unroll
        for (uint32_t j = 0; j < UPQ; ++j) {
          if (wi + NDWG * j >= UNITS) continue;
          uint4 w = make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u);  // code 0 (stored biased by 128): rows beyond the matrix
          uint32_t lo = 0, hi = 0;
          if (valid[j]) {
            const unsigned char *src = stg + (i * UPQ + j) * Q8_UNIT_STAGING;
            w = *reinterpret_cast<const uint4 *>(src + lane * 16);
            // row g's four block scales, then row g + 8's: this unit's block of the four is ((kb & 1) << 1) | bl
            const unsigned short *d = reinterpret_cast<const unsigned short *>(src + 512 + g * 16) + (((kb & 1u) << 1) | bl[j]);
            lo = d[0];
            hi = d[4];
          }
          dequant_unit_at(wt, off_a[j], off_b[j], w, lo, hi);
        }
        // the tensor core reads shared memory through the async proxy: order this warp's stores before its arrival.
        // (The fence waits for the thread's memory operations in flight: the refill below comes after it.)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();          // every lane has fenced, and has read the staging slot
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sa(&full[s])) : "memory");
        request(kb + NG * PF, i);   // refill the slot for this warp's stage PF steps ahead
      }
      if (stop) break;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");  // nothing of this warp may still be landing when the CTA exits
    }
  } else if (warp == 1) {
    // --------------------------------------------------------------------- MMA
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc(BM, BN, KIND == GK_ROWS);
      const uint32_t a0 = desc_lo(sa(stages)), b0 = desc_lo(sa(stages) + A_TILE_BYTES);
      RingPos<C::STAGES> pos;
      bool ok = true;
      for (uint32_t kb = 0; kb < nkb; ++kb, pos.next()) {
        if (!mbar_wait_bounded(sa(&full[pos.s]), pos.phase)) {
          failed_s = 2;
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t off = pos.s * (C::STAGE_BYTES >> 4);
#pragma unroll
        for (uint32_t k = 0; k < BK / 16; ++k)
          mma_f16<1>(tmem_acc + (NACC == 2 ? (k & 1u) * BN : 0u), a0 + off + 2 * k, b0 + off + 2 * k, idesc, k >= NACC || kb);
        mma_commit(sa(&empty[pos.s]));
      }
      if (ok) mma_commit(sa(&acc_ready));
    }
  } else if (!Q8 || warp < 6) {
    // ---------------------------------------------------------------- epilogue
    // a warp may only touch TMEM lanes 32*(warp % 4) .. +31
    const uint32_t quad = warp & 3u;
    const uint32_t row = m0 + quad * 32 + lane;
    uint32_t ok = 1;
    if (lane == 0) ok = mbar_wait_bounded(sa(&acc_ready), 0, 1000) ? 1u : 0u;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (!ok) {
      if (lane == 0) failed_s = 3;
    } else if (!failed_s) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // 32 fp32 results of this thread's row, from column `col` of the accumulators on
      auto take = [&](uint32_t col, float (&v)[32]) {
        uint32_t r[32];
        tmem_ld32(tmem_acc + ((quad * 32u) << 16) + col, r);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
        if (NACC == 2) {
          tmem_ld32(tmem_acc + ((quad * 32u) << 16) + BN + col, r);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] += __uint_as_float(r[j]);
        }
      };
      const uint32_t cols = swiglu ? BN / 2 : BN;
#pragma unroll 1
      for (uint32_t cc = Q8 ? 0 : (warp - 2) / 4 * 32; cc < cols; cc += Q8 ? 32 : (blockDim.x - 64) / 4) {
        if (n0 + cc >= p.N) break;  // uniform over the warp
        float acc[32];
        take(cc, acc);
        if constexpr (KIND != GK_ROWS && BN >= 64) {
          if (swiglu) {
            float up[32];
            take(BN / 2 + cc, up);
            if (row < p.M) swiglu_chunk(acc, up, p.c[0] + (size_t)row * p.N + n0 + cc, p.N - n0 - cc);
            continue;
          }
        }
        if constexpr (KIND == GK_ROWS) {
          if (row < p.M) {
            rows_chunk<bf16>(p.out, row, n0 + cc, acc);
          }
        } else if (row < p.M) {
          f16_chunk(p, mat, row, n0 + cc, acc);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (failed_s) {
    if (threadIdx.x == 0 && p.error) atomicExch(p.error, failed_s);
    // let tensor copies that are still in flight land before the shared memory is given back
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
    __syncthreads();
  }
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"((uint32_t)(NACC * BN)) : "memory");
}

template <int BN, int KIND> cudaError_t launch_bn(const typename GemmArgs<KIND>::Type &p, cudaStream_t s, uint32_t w_rows) {
  constexpr bool Q8 = KIND == GK_Q8;
  CUtensorMap ma;
  WeightMaps mw = {};  // unused with Q8_0: the W tile is written by the dequantising warps
  uint32_t a_rows = p.M, ny = (p.N + BN - 1) / BN;
  int threads = Q8 ? GEMM_THREADS_Q8 : gemm_threads(KIND == GK_ROWS, false);
  if constexpr (KIND == GK_ROWS) {
    a_rows *= p.n2 ? 2 : 1;
    if (!make_map(&mw.w[0], p.w, w_rows, p.K, BN, true)) return cudaErrorInvalidValue;
  } else {
    for (uint32_t i = 0; i < p.nmat && !Q8; ++i)
      if (!make_map(&mw.w[i], p.w[i], w_rows, p.K, p.swiglu ? BN / 2 : BN)) return cudaErrorInvalidValue;
    ny = p.swiglu ? (p.N + BN / 2 - 1) / (BN / 2) : ny * p.nmat;
    if (!Q8) threads = gemm_threads(false, p.swiglu);
  }
  if (!make_map(&ma, p.a, a_rows, p.K, BM, KIND == GK_ROWS)) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_kernel<BN, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg<BN, Q8>::SMEM);
  if (e != cudaSuccess) return e;
  // x = row tile, so that the CTAs sharing one tile of W run together and W crosses HBM once
  gemm_tcgen05_kernel<BN, KIND><<<dim3((p.M + BM - 1) / BM, ny), threads, Cfg<BN, Q8>::SMEM, s>>>(ma, mw, p);
  return cudaGetLastError();
}

}  // namespace

bool gemm_tcgen05_supported(uint32_t M, uint32_t N, uint32_t K) { return M >= 1 && K % BK == 0 && K >= BK && (N % 8) == 0; }

// Tile shape. A grid runs in waves of one CTA (or pair) per SM (two SMs), and a last wave that fills a fraction of the
// SMs takes as long as a full one: pick the shape with the smallest waves x (time of one tile). A tile's time is a K step's
// times their number, plus what a wave does not overlap (its first copies and, without the pairs' second accumulator, its epilogue).
struct Tile {
  bool pair;
  int bn;
};
static int forced_bn() {
  static const int forced = [] { const char *e = getenv("VKLLAMA_GEMM_BN"); return e ? atoi(e) : 0; }();  // experiments
  return forced == 256 || forced == 128 || forced == 64 || forced == 32 ? forced : 0;
}
static Tile pick_tile(uint32_t M, uint32_t N, uint32_t K, uint32_t nmat, bool swiglu, bool pairs) {
  if (int f = forced_bn()) return {false, std::max(f, 128)};
  // measured, us, fp16, K = 4096 and 11008 (a step: from the difference): 512 rows x 4096 columns 20.4 / 47.7 for 128 columns of one
  // CTA, 29.2 / 67.8 for 256, 18.5 / 43.8 and 25.4 / 65.1 for a pair's 128 and 256; 2048 rows 73.9 / 183, 59.5 / 149, 61.0 / 156, 53.2 / 139;
  // 777 x 17152, K = 2048: 97.6, 79.3, 69.3, 55.8
  static const struct {
    Tile tile;
    double step, wave;
  } shapes[] = {{{true, 256}, 0.38, 0.5}, {{false, 256}, 0.42, 4.0}, {{true, 128}, 0.235, 0.5}, {{false, 128}, 0.25, 4.0}};
  Tile best = {false, 0};
  double best_cost = 0.0;
  for (const auto &sh : shapes) {
    if (sh.tile.pair && !pairs) continue;
    const size_t rows = sh.tile.pair ? 2 * BM : BM, bn = (size_t)sh.tile.bn, slots = sm_count() / (sh.tile.pair ? 2 : 1);
    const size_t tiles = (M + rows - 1) / rows * (swiglu ? (2 * (size_t)N + bn - 1) / bn : nmat * ((N + bn - 1) / bn));
    const double cost = (double)((tiles + slots - 1) / slots) * (K / BK * sh.step + sh.wave);
    if (!best.bn || cost < best_cost) {
      best = sh.tile;
      best_cost = cost;
    }
  }
  return best;
}
// Q8_0: the dequantising warps set the pace, one wave at K = 4096 takes 21.5 / 31.4 / 44.5 / 76.5 us for 32 / 64 / 128 / 256 columns.
static int pick_bn_q8(uint32_t M, uint32_t N, uint32_t nmat, bool swiglu) {
  if (int f = forced_bn()) return std::max(f, swiglu ? 64 : 32);
  const size_t mt = (M + BM - 1) / BM, sms = sm_count();
  int best = 0;
  double best_cost = 0.0;
  for (int bn : {256, 128, 64, 32}) {
    if (swiglu && bn < 64) break;
    const size_t ctas = mt * (swiglu ? (2 * N + bn - 1) / bn : nmat * ((N + bn - 1) / bn)), waves = (ctas + sms - 1) / sms;
    const double cost = (double)waves * (bn == 32 ? 21.5 : bn == 64 ? 31.4 : bn == 128 ? 44.5 : 76.5);
    if (!best || cost < best_cost) {
      best = bn;
      best_cost = cost;
    }
  }
  return best;
}

static bool gemm_params_ok(const GemmParams &p, bool q8) {
  if (!gemm_tcgen05_supported(p.M, p.N, p.K) || !p.nmat || p.nmat > 3 || (p.swiglu && p.nmat != 2) || (p.c_f32 && (p.swiglu || p.nmat != 1))) return false;
  for (uint32_t i = 0; i < p.nmat; ++i)
    if (q8 ? !p.w_codes[i] || !p.w_scales[i] : !p.w[i]) return false;
  return true;
}

cudaError_t launch_gemm_f16_tcgen05(const GemmParams &p, cudaStream_t s) {
  if (!gemm_params_ok(p, false)) return cudaErrorInvalidValue;
  for (uint32_t i = 0; i < p.nmat; ++i)
    if ((reinterpret_cast<uintptr_t>(p.a) | reinterpret_cast<uintptr_t>(p.w[i])) & 15) return cudaErrorMisalignedAddress;
  const Tile t = pick_tile(p.M, p.N, p.K, p.nmat, p.swiglu, true);
  if (t.pair) return launch_gemm_pair_f16(p, t.bn, s);
  return t.bn == 256 ? launch_bn<256, GK_F16>(p, s, p.N) : launch_bn<128, GK_F16>(p, s, p.N);
}

namespace {
struct WidenArgs {
  const uint8_t *codes[3], *scales[3];
  __half *out;
};
// Tiled planes -> row-major fp16(q * d), the values that the dequantising warps write. A thread turns eight codes each of two
// rows; bound by memory (4096 x 11008: 24 us, 138 MB).
__device__ __forceinline__ void widen_rows(const uint8_t *__restrict__ codes, const uint8_t *__restrict__ scales, __half *__restrict__ out, const Q8Layout &L) {
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;  // (row tile, block, lane)
  const uint32_t lane = i & 31, g = lane >> 2, t = lane & 3, per = L.groups * 4;
  const uint32_t unit = (uint32_t)(i >> 5), tile = unit / per, b = unit - tile * per, k = b * 32 + t * 8, row = tile * 16 + g;
  if (tile >= L.tiles || k >= L.K) return;
  const uint4 w = ldg_stream(codes + i * 16);
  const __half *d = reinterpret_cast<const __half *>(scales) + (((size_t)tile * L.groups + (b >> 2)) * 8 + g) * 8 + (b & 3);
  const __half sc[2] = {d[0], d[4]};
  const uint32_t c[2][4] = {{codes_to_h2(w.x, false), codes_to_h2(w.x, true), codes_to_h2(w.y, false), codes_to_h2(w.y, true)},
                            {codes_to_h2(w.z, false), codes_to_h2(w.z, true), codes_to_h2(w.w, false), codes_to_h2(w.w, true)}};
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    if (row + 8 * r >= L.N) break;
    const __half2 s = __half2half2(sc[r]);
    uint32_t v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __half2 x = __hmul2(*reinterpret_cast<const __half2 *>(&c[r][j]), s);
      v[j] = *reinterpret_cast<const uint32_t *>(&x);
    }
    *reinterpret_cast<uint4 *>(out + (size_t)(row + 8 * r) * L.K + k) = make_uint4(v[0], v[1], v[2], v[3]);
  }
}
// Grid y: the matrices of one GEMM. A prompt of 509 rows through four 7B blocks took 1321 us with a launch per matrix and 64-bit
// divisions, 1277 this way (and 1476 where the compiler could not see that stores and scales do not alias).
__global__ void __launch_bounds__(256) widen_kernel(const WidenArgs a, Q8Layout L) {
  const uint32_t m = blockIdx.y;
  widen_rows(m == 0 ? a.codes[0] : m == 1 ? a.codes[1] : a.codes[2], m == 0 ? a.scales[0] : m == 1 ? a.scales[1] : a.scales[2], a.out + (size_t)m * L.N * L.K, L);
}
}  // namespace

// A 128-row tile dequantises the whole matrix for itself, at the pace of its dequantising warps (0.67 us per K step of 128
// columns); widened once, the matrix runs on the fp16 GEMM's tiles. A prompt through four 7B blocks, us, dequantised in the tiles /
// widened: 100 rows 937 / -, 128 rows 989 / 1077, 129 1361 / 1077, 256 1387 / 1117, 509 2046 / 1277, 900 3386 / 1716, 2048 6639 / 3015.
// Only vkl_model keeps the room (GemmParams::wide); the operator classes dequantise in the tiles at any number of rows.
constexpr uint32_t kWideRows = 129;
bool gemm_q8_wide(uint32_t M) {
  static const uint32_t rows = [] { const char *e = getenv("VKLLAMA_Q8_WIDE"); return e ? (uint32_t)atoi(e) : kWideRows; }();  // experiments
  return M >= rows;
}

cudaError_t launch_gemm_q8_tcgen05(const GemmParams &p, cudaStream_t s) {
  if (!gemm_params_ok(p, true)) return cudaErrorInvalidValue;
  if (reinterpret_cast<uintptr_t>(p.a) & 15) return cudaErrorMisalignedAddress;
  if (p.wide && gemm_q8_wide(p.M)) {
    const Q8Layout L = q8_layout(p.N, p.K);
    const size_t threads = (size_t)L.tiles * L.groups * 4 * 32;
    GemmParams h = p;
    WidenArgs a = {{}, {}, p.wide};
    for (uint32_t i = 0; i < p.nmat; ++i) {
      a.codes[i] = p.w_codes[i];
      a.scales[i] = p.w_scales[i];
      h.w[i] = p.wide + (size_t)i * p.N * p.K;
    }
    widen_kernel<<<dim3((unsigned)((threads + 255) / 256), p.nmat), 256, 0, s>>>(a, L);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_gemm_f16_tcgen05(h, s);
  }
  switch (pick_bn_q8(p.M, p.N, p.nmat, p.swiglu)) {
    case 256: return launch_bn<256, GK_Q8>(p, s, p.N);
    case 128: return launch_bn<128, GK_Q8>(p, s, p.N);
    case 64: return launch_bn<64, GK_Q8>(p, s, p.N);
    default: return launch_bn<32, GK_Q8>(p, s, p.N);
  }
}

cudaError_t launch_gemm_rows_bf16(const GemmRows &p, cudaStream_t s) {
  if (!gemm_tcgen05_supported(p.M, p.N, p.K) || p.N % 32 || (p.tile_expert && (p.M % BM || p.n2)) || p.n2 % kInputAlign) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(p.a) | reinterpret_cast<uintptr_t>(p.w)) & 15) return cudaErrorMisalignedAddress;
  const Tile t = pick_tile(p.M, p.N, p.K, 1, false, !p.tile_expert);  // the two row tiles of a pair share their weights: not grouped
  if (t.pair) return launch_gemm_pair_bf16(p, t.bn, s);
  // grouped: a tile's weight rows beyond its expert's N are read (the next expert's, or zeros) and dropped by the epilogue
  const uint32_t w_rows = p.tile_expert ? p.w_rows : p.N;
  return t.bn == 256 ? launch_bn<256, GK_ROWS>(p, s, w_rows) : launch_bn<128, GK_ROWS>(p, s, w_rows);
}

}  // namespace vkl
