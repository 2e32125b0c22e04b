// Many tokens in true 32-bit: Y[M,N] = A[M,K] . W[N,K]^T, A fp32, W bf16 (exact in the 32-bit mode), on the bfloat16
// tensor cores. The layer-list decoders' 32-bit mode runs its prompts through it; segments, grouping by expert and
// epilogues are those of the bfloat16 GEMM.
//
// Nothing is rounded on the way in: a float's 24 significant bits are cut into three bfloat16 numbers of 8 bits each
// (high + middle + low = a, exactly from 2^-110 on; what lies below 2^-133, bfloat16's smallest step, is cut off), each product of one of
// them with a bfloat16 weight has 16 bits, and the three products go into the same fp32 sum. What can lose precision is
// the sum: the tensor core cuts off where an FMA rounds. So the accumulator in TMEM holds 64 products per output
// only (one stage, the small parts first) and every stage's sum is added to a register in fp32. Against 64 bits (300 tokens,
// K = 2048 ... 7680) the result is closer than the serial FMA sum that this replaced. Infinities and NaN, of A or of W, come out as
// in that sum (but for numbers below 2^-80 times an infinite weight: NaN).
//
// Measured: the 10 GEMMs of a 300-token prompt at width 2048, feed-forward 5632, four layers: 8.26 ms with the FMA kernel
// (64 x 64 tiles, 15 TFLOP/s), the whole call of 9.31 ms now takes 2.14; error of the logits against 64 bits 7.5e-7 -> 4.7e-7.
//
// Bound: tensor cores at three MMAs per product, or L2 -> shared memory traffic (three A tiles and one W tile,
// 64 KB per 64-wide K step and CTA). One CTA computes 128 x BN with the warps of gemm_tcgen05.cu: TMA producer, MMA
// lane, eight epilogue warps, here working through the whole K loop: while the tensor core fills one
// of two accumulators, they add the other one to their 32 x BN / 2 sums (BN / 2 registers per thread; with four warps
// and BN sums each a launch of 128 columns took 86 us on average in the 300-token prompt, with eight 71).
#include "rows.cuh"
#include "tcgen05.cuh"

namespace vkl {
namespace {

constexpr int kParts = 3, kBuffers = 2;
constexpr int kHalves = 2;  // epilogue warps per 32 rows, each with half of the columns
constexpr int kThreads = 64 + 128 * kHalves;

template <int BN> struct SplitCfg {
  static constexpr uint32_t W_TILE_BYTES = BN * BK * 2;
  static constexpr uint32_t STAGE_BYTES = kParts * A_TILE_BYTES + W_TILE_BYTES;
  static constexpr int STAGES = 3;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + 1024;
};

// [rows, K] floats -> their three parts, one [rows, K] matrix behind the other. Eight values per thread.
__global__ void __launch_bounds__(256) split_kernel(const float *__restrict__ a, bf16 *__restrict__ out, size_t n) {
  const size_t i = ((size_t)blockIdx.x * 256 + threadIdx.x) * 8;
  if (i >= n) return;
  float v[8];
  load8(a + i, v);
  uint32_t part[kParts][8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t u = __float_as_uint(v[j]), sign = u >> 16 & 0x8000u;
    const bool finite = (u & 0x7f800000u) != 0x7f800000u;
    // cut, not rounded: no overflow at the top of the range, and every remainder is exact
    const float r = finite ? v[j] - __uint_as_float(u & 0xffff0000u) : 0.f;
    const uint32_t ur = __float_as_uint(r);
    part[0][j] = (u >> 16) | (!finite && (u & 0x007fffffu) ? 0x40u : 0u);  // a NaN stays one
    part[1][j] = ur >> 16;
    part[2][j] = __float_as_uint(r - __uint_as_float(ur & 0xffff0000u)) >> 16;
    // Times an infinite weight a zero part would give NaN where a * w is infinite, so a part of a number from 2^-80 on is never
    // zero: 2^-126 with its sign takes the place, 2^-46 of the number at most.
    if ((u & 0x7fffffffu) >= 0x17800000u) {
#pragma unroll
      for (int s = 1; s < kParts; ++s)
        if (!(part[s][j] & 0x7fffu)) part[s][j] = sign | 0x0080u;
    }
  }
#pragma unroll
  for (int s = 0; s < kParts; ++s) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = part[s][2 * j] | (part[s][2 * j + 1] << 16);
    *reinterpret_cast<uint4 *>(out + s * n + i) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
    gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const GemmRows p) {
  using C = SplitCfg<BN>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *stages = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[C::STAGES];       // TMA bytes of the stage have landed
  __shared__ __align__(8) uint64_t empty[C::STAGES];      // the MMAs have read the stage
  __shared__ __align__(8) uint64_t acc_full[kBuffers];    // a stage's sums are in the accumulator
  __shared__ __align__(8) uint64_t acc_empty[kBuffers];   // the epilogue warps have taken them
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile uint32_t failed_s;

  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t m0 = blockIdx.x * BM, n0 = blockIdx.y * BN, nkb = p.K / BK;
  const uint32_t rows = p.n2 ? 2 * p.M : p.M;  // of one part
  uint32_t w_row = n0, a_row = m0;
  if (p.n2 && n0 >= p.n2) a_row += p.M;
  if (p.tile_expert) {
    const int32_t e = p.tile_expert[blockIdx.x];
    if (e < 0) return;  // uniform over the CTA
    w_row += (uint32_t)e * p.N;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sa(&full[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sa(&empty[s])) : "memory");
    }
    for (int b = 0; b < kBuffers; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sa(&acc_full[b])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sa(&acc_empty[b])), "n"(4 * kHalves) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    failed_s = 0;
  }
  if (warp == 1) tmem_alloc<kBuffers * BN>(sa(&tmem_base_s));
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_acc = tmem_base_s;

  if (warp == 0) {
    if (elect_one()) {
      RingPos<C::STAGES> pos;
      for (uint32_t kb = 0; kb < nkb; ++kb, pos.next()) {
        if (kb >= C::STAGES && !mbar_wait_bounded(sa(&empty[pos.s]), pos.phase ^ 1u)) {
          failed_s = 1;
          break;
        }
        const uint32_t bar = sa(&full[pos.s]), st = sa(stages) + pos.s * C::STAGE_BYTES;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(C::STAGE_BYTES) : "memory");
        // rows beyond a part's end are the next part's (or zeros): they make rows that the epilogue drops
#pragma unroll
        for (uint32_t i = 0; i < kParts; ++i) tma_load_2d(st + i * A_TILE_BYTES, &map_a, kb * BK, i * rows + a_row, bar);
        tma_load_2d(st + kParts * A_TILE_BYTES, &map_w, kb * BK, w_row, bar);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc(BM, BN, true);
      const uint32_t a0 = desc_lo(sa(stages)), w0 = desc_lo(sa(stages) + kParts * A_TILE_BYTES);
      RingPos<C::STAGES> pos;
      RingPos<kBuffers> buf;
      for (uint32_t kb = 0; kb < nkb; ++kb, pos.next(), buf.next()) {
        if ((kb >= kBuffers && !mbar_wait_bounded(sa(&acc_empty[buf.s]), buf.phase ^ 1u)) || !mbar_wait_bounded(sa(&full[pos.s]), pos.phase)) {
          failed_s = 2;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t off = pos.s * (C::STAGE_BYTES >> 4), acc = tmem_acc + buf.s * BN;
#pragma unroll
        for (int i = kParts - 1; i >= 0; --i)  // small parts first: little is cut off from their sums
#pragma unroll
          for (uint32_t k = 0; k < BK / 16; ++k) mma_f16<1>(acc, a0 + off + i * (A_TILE_BYTES >> 4) + 2 * k, w0 + off + 2 * k, idesc, i < kParts - 1 || k);
        mma_commit(sa(&empty[pos.s]));
        mma_commit(sa(&acc_full[buf.s]));
      }
    }
  } else {
    const uint32_t quad = warp & 3u, row = m0 + quad * 32 + lane;
    constexpr int COLS = BN / kHalves;
    const uint32_t c0 = (warp - 2) / 4 * COLS;
    float sum[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
    bool done = true;
    for (uint32_t kb = 0; kb < nkb; ++kb) {
      const uint32_t b = kb % kBuffers, buse = kb / kBuffers;
      uint32_t ok = 1;
      if (lane == 0) ok = mbar_wait_bounded(sa(&acc_full[b]), buse & 1u) ? 1u : 0u;
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok && lane == 0) failed_s = 3;
      // one lane's view of the flag: the warp leaves together
      if (__shfl_sync(0xffffffffu, failed_s, 0)) {
        done = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int cc = 0; cc < COLS; cc += 32) {
        uint32_t r[32];
        tmem_ld32(tmem_acc + ((quad * 32u) << 16) + b * BN + c0 + cc, r);
#pragma unroll
        for (int j = 0; j < 32; ++j) sum[cc + j] += __uint_as_float(r[j]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sa(&acc_empty[b])) : "memory");
    }
    if (done && row < p.M) {
#pragma unroll
      for (int cc = 0; cc < COLS; cc += 32) {
        if (n0 + c0 + cc >= p.N) break;  // N is a multiple of 32
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = sum[cc + j];
        rows_chunk<float>(p.out, row, n0 + c0 + cc, v);
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
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"((uint32_t)(kBuffers * BN)) : "memory");
}

template <int BN> cudaError_t launch_split(const GemmRows &p, cudaStream_t s) {
  const uint32_t rows = p.n2 ? 2 * p.M : p.M, w_rows = p.tile_expert ? p.w_rows : p.N;
  CUtensorMap ma, mw;
  if (!make_map(&ma, p.split, kParts * rows, p.K, BM, true) || !make_map(&mw, p.w, w_rows, p.K, BN, true)) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SplitCfg<BN>::SMEM);
  if (e != cudaSuccess) return e;
  const size_t n = (size_t)rows * p.K;
  split_kernel<<<(unsigned)((n + 2047) / 2048), 256, 0, s>>>(static_cast<const float *>(p.a), p.split, n);
  // x = row tile, so that the CTAs sharing one tile of W run together and W crosses HBM once
  gemm_split_kernel<BN><<<dim3((p.M + BM - 1) / BM, (p.N + BN - 1) / BN), kThreads, SplitCfg<BN>::SMEM, s>>>(ma, mw, p);
  return cudaGetLastError();
}

}  // namespace

// Tile width: 128 columns share an A tile's three parts among most; 64 where 128 would leave half of the SMs idle (a
// K step of 64 columns takes about 0.9 of the time of one of 128, both are bound by the A parts' copies).
cudaError_t launch_gemm_rows_f32(const GemmRows &p, cudaStream_t s) {
  if (!p.M || !p.N || p.N % 32 || p.K % BK || !p.K || p.n2 % kInputAlign || !p.split || (p.tile_expert && (p.M % BM || p.n2))) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(p.a) | reinterpret_cast<uintptr_t>(p.w) | reinterpret_cast<uintptr_t>(p.split)) & 15) return cudaErrorMisalignedAddress;
  const size_t ctas = (size_t)((p.M + BM - 1) / BM) * ((p.N + 127) / 128);
  return ctas * 2 <= sm_count() ? launch_split<64>(p, s) : launch_split<128>(p, s);
}

}  // namespace vkl
