// A few rows (9 to 64) times a weight matrix: Y[M,N] = epilogue(X[M,K] . W[N,K]^T), Q8_0 or FP16 weights, with the exact
// arithmetic and the epilogues of the mat-vec kernel (matvec.cu): products of codes and inputs on mma.sync with fp32
// accumulators, the block scale applied in fp32 per 32 columns.
//
// The roofs are the weights' bytes up to some 24 rows and the mma.sync pipe beyond (a scale per 32 columns and row keeps Q8_0 off
// tcgen05, whose accumulators cannot be scaled on the way without rounding the weights); at 45 rows the pipe is a third busy, the
// rest is what one CTA per SM does not overlap: its first copies and its reduction. What held the mat-vec kernel back at a
// fifth of that was X: every 16-row tile fetched all of it from L2, 0.8 GB for 45 rows of the 13B gate/up. Here a
// CTA takes 64 weight rows (or 32), and both operands arrive K chunk by K chunk in a ring of shared-memory stages: X (and FP16
// weights) by TMA tensor copies, Q8_0 planes by bulk copies, a few large ones per chunk, since issuing a copy takes a
// warp some 60 cycles (a copy per row of X was twice as slow as the mat-vec kernel). Sixteen warps: each takes a pair of 16-row
// tiles (with SwiGLU a gate and an up tile) and one 32-column block of the chunk, so that an X fragment serves two
// tiles. The warps' K shares are added in a fixed order at the end. 62 to 128 registers; at the cap of 128 (one CTA per SM) some of those of 33 rows and more
// spill 4 to 16 bytes (12 to 52 with 64-bit shared addresses). MMAs whose order the scheduler may choose and 32-bit shared addresses, us per call of
// four 13B blocks before / now: FP16 17 rows 916 / 848, 45 858 / 836, Q8_0 17 rows 848 / 823, 45 977 / 955 (about 10 of each are the call's).
//
// Included by skinny_gemm.cu (Q8_0, and the rule) and skinny_gemm_f16.cu. In one file the 48 kernels with their line tables were 10 MB, from which
// size on nvcc compresses device code: a process's first launch took 9.3 ms to unpack and load them, 3.2 (Q8_0) and 3.6 ms (FP16) now.
#pragma once
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "tcgen05.cuh"

namespace vkl {
namespace {

constexpr int kWarps = 16, kThreads = 32 * kWarps;
constexpr uint32_t kFewRows = 16;  // two fragments of 8 rows: the least this kernel takes
constexpr int kMaxStages = 8;
constexpr size_t kRing = 220 * 1024;

// PAIRS: pairs of row tiles per CTA. A chunk is KQ blocks of 32 columns, one per warp of a pair, SUB tensor copies of 64.
template <int MT, bool Q8, int PAIRS> struct SkinnyCfg {
  static constexpr int KQ = kWarps / PAIRS, TILES = 2 * PAIRS, CHUNK = 32 * KQ, SUB = CHUNK / 64;
  static constexpr uint32_t X_BYTES = MT * 8 * CHUNK * 2;
  static constexpr uint32_t CODES = KQ * 512, SCALES = KQ / 4 * 128, ROWS16 = 16 * CHUNK * 2;  // of one tile
  static constexpr uint32_t TILE = Q8 ? CODES + SCALES : ROWS16, STAGE = X_BYTES + TILES * TILE;
  static constexpr uint32_t RED = kWarps * 2 * MT * 4 * 32 * 4;
  static_assert(STAGE % 1024 == 0, "swizzle atoms");
};

// Stages hold 128-byte rows in the 128-byte swizzle (16-byte piece c of row r at c ^ (r % 8)). A fragment load of eight lanes reads
// four pieces of two rows; for rows r and r + 1 they share their banks, for r and r + 4 they do not: row g of a fragment is row
// swap3(g) of memory.
__device__ __forceinline__ uint32_t swap3(uint32_t g) { return (g & 1u) << 2 | g >> 1; }
__device__ __forceinline__ uint32_t unswap3(uint32_t r) { return (r & 3u) << 1 | r >> 2; }

__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ __half lds_half(uint32_t a) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
  return __ushort_as_half(v);
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// (Not volatile, the order is the scheduler's to choose.)
__device__ __forceinline__ void mma16816_zero(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

__device__ __forceinline__ void mma16816_onto(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int MT, int EPI, bool Q8, int PAIRS>
__global__ void __launch_bounds__(kThreads, 1)
    skinny_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ WeightMaps maps, const MvParams p, const uint32_t nst) {
  using C = SkinnyCfg<MT, Q8, PAIRS>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages];
  __shared__ volatile uint32_t failed_s;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t ntiles = (p.N + 15) / 16, blocks = (p.K + 31) / 32, groups = (blocks + 3) / 4, chunks = (blocks + C::KQ - 1) / C::KQ;
  const uint32_t mat = EPI == EPI_SWIGLU ? 0u : blockIdx.y;
  constexpr uint32_t OUT_TILES = EPI == EPI_SWIGLU ? PAIRS : C::TILES;
  const uint32_t tile0 = blockIdx.x * OUT_TILES;
  // tile i of the CTA: SwiGLU: gate and up tiles in turn
  auto tile_of = [&](uint32_t i) { return tile0 + (EPI == EPI_SWIGLU ? i >> 1 : i); };
  auto matrix_of = [&](uint32_t i) { return EPI == EPI_SWIGLU ? i & 1u : mat; };
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < nst; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sa(&full[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sa(&empty[s])), "r"((uint32_t)kWarps) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    failed_s = 0;
  }
  __syncthreads();

  float acc[2][MT][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) acc[i][mt][0] = acc[i][mt][1] = acc[i][mt][2] = acc[i][mt][3] = 0.f;
  const uint32_t pair = warp / C::KQ, kq = warp % C::KQ, sub = kq >> 1;
  const uint32_t row = swap3(g), piece = ((((kq & 1u) << 2) + t) ^ row) * 16;
  // this lane's pieces of a stage: inputs, weights (of the pair's first tile), scales
  const uint32_t x_at = sa(smem) + sub * (MT * 1024) + row * 128 + piece;
  const uint32_t w_at = sa(smem) + C::X_BYTES + pair * 2 * C::TILE + (Q8 ? kq * 512 + lane * 16 : sub * 2048 + row * 128 + piece);
  const uint32_t d_at = sa(smem) + C::X_BYTES + pair * 2 * C::TILE + C::CODES + (kq >> 2) * 128 + g * 16 + (kq & 3) * 2;
  uint32_t tiles_here = 0;
  for (uint32_t i = 0; i < C::TILES; ++i) tiles_here += tile_of(i) < ntiles ? 1u : 0u;

  // Chunk c's copies, shared out over warps 0 (X) and 1 ... TILES (a tile each); rows and columns beyond a matrix read as zero
  uint32_t is = 0, iphase = 0;
  auto issue = [&](uint32_t c) {
    if (warp <= C::TILES && elect_one()) {
      if (c >= nst && !mbar_wait_bounded(sa(&empty[is]), iphase ^ 1u)) {
        failed_s = 1;
      } else {
        const uint32_t bar = sa(&full[is]), st = sa(smem) + is * C::STAGE;
        const uint32_t ng = min((uint32_t)C::KQ / 4, groups - c * (C::KQ / 4)), cb = ng * 2048, sb = ng * 128;
        if (warp == 0) {
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                       "r"(C::X_BYTES + (Q8 ? tiles_here * (cb + sb) : (uint32_t)C::TILES * C::ROWS16))
                       : "memory");
#pragma unroll
          for (uint32_t i = 0; i < C::SUB; ++i) tma_load_2d(st + i * (MT * 1024), &map_x, c * C::CHUNK + i * 64, 0, bar);
        } else {
          const uint32_t i = warp - 1, w = st + C::X_BYTES + i * C::TILE, mi = matrix_of(i);
          if constexpr (Q8) {
            if (tile_of(i) < ntiles) {
              const size_t grp = (size_t)tile_of(i) * groups + c * (C::KQ / 4);
              bulk_load(w, p.codes[mi] + grp * 2048, cb, bar);
              bulk_load(w + C::CODES, p.scales[mi] + grp * 128, sb, bar);
            }
          } else {
#pragma unroll
            for (uint32_t j = 0; j < C::SUB; ++j) tma_load_2d(w + j * 2048, &maps.w[mi], c * C::CHUNK + j * 64, tile_of(i) * 16, bar);
          }
        }
      }
    }
    __syncwarp();
    if (++is == nst) {
      is = 0;
      iphase ^= 1u;
    }
  };
  for (uint32_t c = 0; c + 1 < nst && c < chunks; ++c) issue(c);
  uint32_t s = 0, phase = 0;
  for (uint32_t c = 0; c < chunks; ++c) {
    if (c + nst - 1 < chunks) issue(c + nst - 1);
    if (!mbar_wait_bounded(sa(&full[s]), phase)) {
      failed_s = 2;
      break;
    }
    if (c * C::KQ + kq < blocks) {  // uniform over the warp; the last chunk may be short. Rows beyond N hold anything and are not stored
      const uint32_t xs = x_at + s * C::STAGE, ws = w_at + s * C::STAGE;
      uint32_t A0[2][4], A1[2][4];
      float d_lo[2], d_hi[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if constexpr (Q8) {
          const uint4 cw = lds128(ws + i * C::TILE);
          A0[i][0] = codes_to_h2(cw.x, false);
          A0[i][1] = codes_to_h2(cw.z, false);
          A0[i][2] = codes_to_h2(cw.x, true);
          A0[i][3] = codes_to_h2(cw.z, true);
          A1[i][0] = codes_to_h2(cw.y, false);
          A1[i][1] = codes_to_h2(cw.w, false);
          A1[i][2] = codes_to_h2(cw.y, true);
          A1[i][3] = codes_to_h2(cw.w, true);
          const uint32_t d = d_at + s * C::STAGE + i * C::TILE;
          d_lo[i] = __half2float(lds_half(d));
          d_hi[i] = __half2float(lds_half(d + 8));
        } else {
          const uint4 r0 = lds128(ws + i * C::TILE), r8 = lds128(ws + i * C::TILE + 1024);
          A0[i][0] = r0.x; A0[i][1] = r8.x; A0[i][2] = r0.y; A0[i][3] = r8.y;
          A1[i][0] = r0.z; A1[i][1] = r8.z; A1[i][2] = r0.w; A1[i][3] = r8.w;
          d_lo[i] = d_hi[i] = 1.f;
        }
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const uint4 X = lds128(xs + mt * 1024);
        if constexpr (Q8) {
          float v[2][4];
#pragma unroll
          for (int i = 0; i < 2; ++i) mma16816_zero(v[i], A0[i][0], A0[i][1], A0[i][2], A0[i][3], X.x, X.y);
#pragma unroll
          for (int i = 0; i < 2; ++i) mma16816_onto(v[i], A1[i][0], A1[i][1], A1[i][2], A1[i][3], X.z, X.w);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            acc[i][mt][0] = fmaf(v[i][0], d_lo[i], acc[i][mt][0]);
            acc[i][mt][1] = fmaf(v[i][1], d_lo[i], acc[i][mt][1]);
            acc[i][mt][2] = fmaf(v[i][2], d_hi[i], acc[i][mt][2]);
            acc[i][mt][3] = fmaf(v[i][3], d_hi[i], acc[i][mt][3]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 2; ++i) mma16816_onto(acc[i][mt], A0[i][0], A0[i][1], A0[i][2], A0[i][3], X.x, X.y);
#pragma unroll
          for (int i = 0; i < 2; ++i) mma16816_onto(acc[i][mt], A1[i][0], A1[i][1], A1[i][2], A1[i][3], X.z, X.w);
        }
      }
    }
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sa(&empty[s])) : "memory");
    if (++s == nst) {
      s = 0;
      phase ^= 1u;
    }
  }
  __syncthreads();
  if (failed_s) {  // uniform: written before the barrier
    if (threadIdx.x == 0 && p.error) atomicExch(p.error, 8u);
    for (int i = 0; i < 2000; ++i) __nanosleep(100);  // copies that are still in flight land
    return;
  }
  // ---- the warps' K shares, added in order; the ring is done with
  float *red = reinterpret_cast<float *>(smem);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int j = 0; j < 4; ++j) red[(((warp * 2 + i) * MT + mt) * 4 + j) * 32 + lane] = acc[i][mt][j];
  __syncthreads();
  auto total = [&](uint32_t tile, uint32_t mt, uint32_t j, uint32_t ln) {
    float v = 0.f;
#pragma unroll
    for (uint32_t q = 0; q < C::KQ; ++q) v += red[(((((tile >> 1) * C::KQ + q) * 2 + (tile & 1)) * MT + mt) * 4 + j) * 32 + ln];
    return v;
  };
  // idx: row of the tile fastest, so that neighbouring threads store neighbouring columns
  for (uint32_t idx = threadIdx.x; idx < OUT_TILES * MT * 128u; idx += kThreads) {
    const uint32_t ot = (idx >> 4) % OUT_TILES, r = idx & 15, m = (idx >> 4) / OUT_TILES, mt = m >> 3, col = unswap3(m & 7), n = (tile0 + ot) * 16 + r;
    if (m >= p.M || n >= p.N) continue;
    const uint32_t ln = (Q8 ? r & 7 : unswap3(r & 7)) * 4 + (col >> 1), j = (r >> 3) * 2 + (col & 1);
    const size_t o = (size_t)m * p.out_ld + n;
    if (EPI == EPI_SWIGLU) {
      const float gate = total(2 * ot, mt, j, ln), up = total(2 * ot + 1, mt, j, ln);
      p.out[0][o] = __float2half_rn(gate / (1.0f + expf(-gate)) * up);
    } else if (EPI == EPI_ADD) {
      const float y = round_h(total(ot, mt, j, ln) * p.scale + p.bias);
      p.out[0][o] = __float2half_rn(y + __half2float(p.residual[o]));
    } else {
      float y = total(ot, mt, j, ln) * p.scale + p.bias;
      if (p.act == 1) y = y / (1.0f + expf(-y));
      const __half hy = __float2half_rn(y);
      p.out[mat][o] = hy;
      if (p.out_f32) p.out_f32[o] = __half2float(hy);
    }
  }
}

template <int MT, int EPI, bool Q8, int PAIRS> cudaError_t launch_t(const MvParams &p, cudaStream_t s) {
  using C = SkinnyCfg<MT, Q8, PAIRS>;
  const uint32_t out_tiles = EPI == EPI_SWIGLU ? PAIRS : C::TILES, gx = ((p.N + 15) / 16 + out_tiles - 1) / out_tiles, gy = EPI == EPI_SWIGLU ? 1u : p.nmat;
  const uint32_t nst = (uint32_t)std::min<size_t>(kMaxStages, kRing / C::STAGE);
  static_assert(kRing / C::STAGE >= 2, "a ring");
  const size_t smem = std::max<size_t>((size_t)nst * C::STAGE, C::RED) + 1024;
  CUtensorMap mx;
  WeightMaps mw = {};
  if (!make_map(&mx, p.x, p.M, p.K, MT * 8)) return cudaErrorInvalidValue;
  for (uint32_t i = 0; !Q8 && i < (EPI == EPI_SWIGLU ? 2u : p.nmat); ++i)
    if (!make_map(&mw.w[i], p.codes[i], p.N, p.K, 16)) return cudaErrorInvalidValue;
  auto kern = skinny_kernel<MT, EPI, Q8, PAIRS>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<dim3(gx, gy), kThreads, smem, s>>>(mx, mw, p, nst);
  return cudaGetLastError();
}
template <int MT, int EPI, bool Q8> cudaError_t launch_p(const MvParams &p, cudaStream_t s) {
  const size_t tiles = EPI == EPI_SWIGLU ? 2 * ((p.N + 15) / 16) : (size_t)p.nmat * ((p.N + 15) / 16);
  return tiles / 4 >= sm_count() ? launch_t<MT, EPI, Q8, 2>(p, s) : launch_t<MT, EPI, Q8, 1>(p, s);
}
template <int EPI, bool Q8> cudaError_t launch_m(const MvParams &p, cudaStream_t s) {
  if (p.M <= kFewRows) {
    if constexpr (!Q8) return launch_p<2, EPI, false>(p, s);
    else if constexpr (EPI != EPI_SWIGLU) return launch_t<2, EPI, true, 1>(p, s);  // the others are not taken (skinny_gemm_takes)
    else return cudaErrorInvalidValue;
  }
  if (p.M <= 32) return launch_p<4, EPI, Q8>(p, s);
  if (p.M <= 48) return launch_p<6, EPI, Q8>(p, s);
  return launch_p<8, EPI, Q8>(p, s);
}
template <bool Q8> cudaError_t launch_kind(const MvParams &p, int epi, cudaStream_t s) {
  switch (epi) {
    case EPI_PLAIN: return launch_m<EPI_PLAIN, Q8>(p, s);
    case EPI_ADD: return launch_m<EPI_ADD, Q8>(p, s);
    case EPI_SWIGLU: return launch_m<EPI_SWIGLU, Q8>(p, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace
}  // namespace vkl
