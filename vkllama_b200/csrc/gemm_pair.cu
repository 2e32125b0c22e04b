// Dense GEMM for long prompts: C[M,N] = A[M,K] . W[N,K]^T by pairs of CTAs (tcgen05.mma.cta_group::2), fp16 or
// bfloat16 operands, fp32 accumulation in tensor memory; results and rounding are those of gemm_tcgen05.cu.
//
// A CTA alone reads 16 + 32 KB from L2 for the 128 x 256 x 64 products of a K step, 96 bytes per clock and SM at the full
// tensor rate. A pair computes a 256 x BN tile, each CTA holding its own 128 rows of A and HALF of the W tile, which the
// tensor cores of both read: 64 bytes per clock. The kernel is persistent, one pair per two SMs: tile after tile through
// the same ring of stages, and of two accumulators in TMEM one is stored while the next tile fills the other.
//   warp 0    producer (both CTAs): TMA copies of its A rows and its half of W; both complete on the leader's barrier.
//   warp 1    MMA (leader): four tcgen05.mma (M256 N{BN} K16) per stage; commits give the stage back in both CTAs.
//   the others epilogue (both CTAs): their 128 rows of the tile, one, two or four warps per 32 rows, then they give the accumulator back to the leader.
// With SwiGLU the leader's half of a W tile is gate rows and the other CTA's the up rows of the same outputs.
// 2048 rows, 4096 x 11008: 167 us with one CTA per tile and a slow MMA lane, 149 with the present one, 139 in pairs (1330
// TFLOP/s, 0.84 of the cuBLAS burst rate); 777 x 17152 x 2048 79 -> 56. What is left is the last wave and the power limit.
// Every wait is bounded; after a time-out both CTAs run out of work, raise the error word and leave together.
#include "kernels.h"
#include "rows.cuh"
#include "tcgen05.cuh"

namespace vkl {
namespace {

// Epilogue warps per 32 rows, each with its share of the columns. A warp executes some thousand dependent instructions per 32 x 32
// chunk of an epilogue with activations in it: with one warp per 32 rows a 777 x 13856 tile grid of K = 2048 waited for its
// epilogues (27 us per tile, the products of a tile take 9). us per launch with 1 / 2 / 4: layer-list in-projection of 777 rows 81.7 /
// 56.6 / 45.9, 2048 rows 142.8 / 108.7 / 103.5, SwiGLU of 509 rows 81.3 / 77.8 / -; a plain rounding: 2048 x 4096 gained nothing.
__host__ __device__ constexpr uint32_t epilogue_parts(bool rows, bool swiglu) { return rows ? 4 : swiglu ? 2 : 1; }
__host__ __device__ constexpr int pair_threads(bool rows, bool swiglu) { return 64 + 128 * (int)epilogue_parts(rows, swiglu); }
constexpr uint32_t kTmemColumns = 512;  // all of them: the two CTAs' accumulators lie at the same address

template <int BN> struct PairCfg {
  static constexpr uint32_t STAGE_BYTES = A_TILE_BYTES + BN / 2 * BK * 2;
  static constexpr int STAGES = 192 * 1024 / STAGE_BYTES;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + 1024;
};

struct PairGrid {
  uint32_t mtiles, ntiles, per;  // tiles of 256 rows; column tiles of all matrices, of one
};

template <bool ROWS> struct PairArgs { using Type = GemmParams; };
template <> struct PairArgs<true> { using Type = GemmRows; };

__device__ __forceinline__ uint32_t leader_address(uint32_t addr) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void commit_both(uint32_t bar) {  // arrives on this barrier of both CTAs once all MMAs so far have completed
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t leader_bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(leader_bar)
               : "memory");
}

template <int BN, bool ROWS, bool SWIGLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pair_threads(ROWS, SWIGLU), 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ WeightMaps maps, const typename PairArgs<ROWS>::Type p, const PairGrid g) {
  using C = PairCfg<BN>;
  constexpr uint32_t OUT = SWIGLU ? BN / 2 : BN;  // output columns of a tile
  constexpr uint32_t kParts = epilogue_parts(ROWS, SWIGLU);
  extern __shared__ unsigned char smem_raw[];
  unsigned char *stages = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[C::STAGES];   // leader: the TMA bytes of both CTAs have landed
  __shared__ __align__(8) uint64_t empty[C::STAGES];  // the MMAs have read the stage
  __shared__ __align__(8) uint64_t acc_full[2];       // a tile's sums are in the accumulator
  __shared__ __align__(8) uint64_t acc_empty[2];      // leader: the epilogue warps of both CTAs have taken them
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile uint32_t failed_s;

  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const uint32_t nkb = p.K / BK, tiles = g.mtiles * g.ntiles, step = gridDim.x / 2;
  // tile t: rows fastest, so that the pairs that share a W tile run together and W crosses HBM once
  uint32_t m0, n0, mat;
  auto locate = [&](uint32_t t) {
    const uint32_t nt = t / g.mtiles;
    m0 = (t - nt * g.mtiles) * 2 * BM + rank * BM;
    mat = nt / g.per;
    n0 = (nt - mat * g.per) * OUT;
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sa(&full[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sa(&empty[s])) : "memory");
    }
    for (int b = 0; b < 2; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sa(&acc_full[b])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sa(&acc_empty[b])), "n"(8 * kParts) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    failed_s = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sa(&tmem_base_s)), "r"(kTmemColumns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();  // the other CTA's barriers are there
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;

  if (warp == 0) {
    if (elect_one()) {
      RingPos<C::STAGES> pos;
      bool first = true, ok = true;  // first: the ring's first round, no stage to wait for
      const uint32_t leader_full = leader_address(sa(&full[0]));
      for (uint32_t t = blockIdx.x / 2; t < tiles && ok; t += step) {
        locate(t);
        uint32_t a_row = m0;  // rows beyond an input's M are read (the next one's, or zeros) and dropped by the epilogue
        if constexpr (ROWS) {
          if (p.n2 && n0 >= p.n2) a_row += p.M;
        }
        const CUtensorMap *mw = SWIGLU ? &maps.w[rank] : &maps.w[mat];
        const uint32_t w_row = SWIGLU ? n0 : n0 + rank * (BN / 2);
        for (uint32_t k = 0; k < p.K; k += BK) {
          if (!first && !mbar_wait_bounded(sa(&empty[pos.s]), pos.phase ^ 1u)) {
            failed_s = 1;
            ok = false;
            break;
          }
          if (rank == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sa(&full[pos.s])), "r"(2 * C::STAGE_BYTES) : "memory");
          const uint32_t bar = leader_full + pos.s * 8, st = sa(stages) + pos.s * C::STAGE_BYTES;
          tma_load_pair(st, &map_a, k, a_row, bar);
          tma_load_pair(st + A_TILE_BYTES, mw, k, w_row, bar);
          pos.next();
          if (pos.s == 0) first = false;
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = instr_desc(2 * BM, BN, ROWS);
      const uint32_t a0 = desc_lo(sa(stages)), b0 = desc_lo(sa(stages) + A_TILE_BYTES);
      RingPos<C::STAGES> pos;
      uint32_t done = 0;
      bool ok = true;
      for (uint32_t t = blockIdx.x / 2; t < tiles && ok; t += step, ++done) {
        const uint32_t b = done & 1u, acc = tmem + b * BN;
        if (done >= 2 && !mbar_wait_bounded(sa(&acc_empty[b]), ((done >> 1) - 1) & 1u)) {
          failed_s = 4;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (uint32_t kb = 0; kb < nkb; ++kb, pos.next()) {
          if (!mbar_wait_bounded(sa(&full[pos.s]), pos.phase)) {
            failed_s = 2;
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t off = pos.s * (C::STAGE_BYTES >> 4);
#pragma unroll
          for (uint32_t k = 0; k < BK / 16; ++k) mma_f16<2>(acc, a0 + off + 2 * k, b0 + off + 2 * k, idesc, k || kb);
          commit_both(sa(&empty[pos.s]));
        }
        if (ok) commit_both(sa(&acc_full[b]));
      }
    }
  } else {
    // a warp may only touch TMEM lanes 32*(warp % 4) .. +31
    const uint32_t quad = warp & 3u;
    uint32_t done = 0;
    for (uint32_t t = blockIdx.x / 2; t < tiles; t += step, ++done) {
      locate(t);
      const uint32_t b = done & 1u, row = m0 + quad * 32 + lane, acc = tmem + ((quad * 32u) << 16) + b * BN;
      uint32_t ok = 1;
      if (lane == 0) ok = mbar_wait_bounded(sa(&acc_full[b]), (done >> 1) & 1u, 200) ? 1u : 0u;
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) {
        if (lane == 0) failed_s = 3;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
      for (uint32_t cc = (warp - 2) / 4 * 32; cc < OUT; cc += 32 * kParts) {
        if (n0 + cc >= p.N) break;  // uniform over the warp
        uint32_t r[32];
        float v[32];
        tmem_ld32(acc + cc, r);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
        if constexpr (SWIGLU) {
          float up[32];
          tmem_ld32(acc + BN / 2 + cc, r);
#pragma unroll
          for (int j = 0; j < 32; ++j) up[j] = __uint_as_float(r[j]);
          if (row < p.M) swiglu_chunk(v, up, p.c[0] + (size_t)row * p.N + n0 + cc, p.N - n0 - cc);
        } else if constexpr (ROWS) {
          if (row < p.M) rows_chunk<bf16>(p.out, row, n0 + cc, v);
        } else {
          if (row < p.M) f16_chunk(p, mat, row, n0 + cc, v);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_address(sa(&acc_empty[b]))) : "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (failed_s) {
    if (threadIdx.x == 0 && p.error) atomicExch(p.error, failed_s);
    // let tensor copies that are still in flight land before the shared memory is given back
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
  }
  __syncwarp();
  cluster_sync();  // nothing arrives here or writes to the other CTA any more
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemColumns) : "memory");
}

template <int BN, bool ROWS, bool SWIGLU> cudaError_t launch_pair(const typename PairArgs<ROWS>::Type &p, cudaStream_t s) {
  constexpr uint32_t OUT = SWIGLU ? BN / 2 : BN;
  CUtensorMap ma;
  WeightMaps mw = {};
  uint32_t a_rows = p.M;
  PairGrid g;
  g.mtiles = (p.M + 2 * BM - 1) / (2 * BM);
  g.per = g.ntiles = (p.N + OUT - 1) / OUT;
  if constexpr (ROWS) {
    a_rows *= p.n2 ? 2 : 1;
    if (!make_map(&mw.w[0], p.w, p.N, p.K, BN / 2, true)) return cudaErrorInvalidValue;
  } else {
    for (uint32_t i = 0; i < p.nmat; ++i)
      if (!make_map(&mw.w[i], p.w[i], p.N, p.K, BN / 2)) return cudaErrorInvalidValue;
    if (!SWIGLU) g.ntiles *= p.nmat;
  }
  if (!make_map(&ma, p.a, a_rows, p.K, BM, ROWS)) return cudaErrorInvalidValue;
  auto kern = gemm_pair_kernel<BN, ROWS, SWIGLU>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PairCfg<BN>::SMEM);
  if (e != cudaSuccess) return e;
  const size_t tiles = (size_t)g.mtiles * g.ntiles, pairs = sm_count() / 2;
  kern<<<(unsigned)(2 * (tiles < pairs ? tiles : pairs)), pair_threads(ROWS, SWIGLU), PairCfg<BN>::SMEM, s>>>(ma, mw, p, g);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_gemm_pair_f16(const GemmParams &p, int bn, cudaStream_t s) {
  if (p.swiglu) return bn == 256 ? launch_pair<256, false, true>(p, s) : launch_pair<128, false, true>(p, s);
  return bn == 256 ? launch_pair<256, false, false>(p, s) : launch_pair<128, false, false>(p, s);
}
cudaError_t launch_gemm_pair_bf16(const GemmRows &p, int bn, cudaStream_t s) {
  return bn == 256 ? launch_pair<256, true, false>(p, s) : launch_pair<128, true, false>(p, s);
}

}  // namespace vkl
