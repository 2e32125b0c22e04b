// What the tcgen05 GEMM kernels share: bounded barrier waits, descriptors, TMA and TMEM access, epilogues of the Llama
// path, tensor maps.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "kernels.h"

namespace vkl {
namespace {

constexpr int BM = 128, BK = 64;  // output rows of a tile and K slice of a stage
constexpr uint32_t A_TILE_BYTES = BM * BK * 2;  // 16 KB
constexpr uint32_t GEMM_WAIT_LIMIT = 1u << 22;

__device__ __forceinline__ uint32_t sa(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Bounded wait. `sleep_ns`: pause between polls, for the waits that are long by design (the epilogue warps wait
// for the whole K loop): a warp that spins takes issue slots from the warps that work on the same sub-partition.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, uint32_t sleep_ns = 0) {
  for (uint32_t i = 0; i < GEMM_WAIT_LIMIT; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if (sleep_ns) __nanosleep(sleep_ns);
  }
  return false;
}

// The single-lane roles (TMA producer, MMA issuer) run a K step's instructions one after the other at their latencies, and
// the CTA waits on them: at some 780 cycles per step they, not the 256 ... 512 cycles of the MMAs, set the pace of every
// GEMM here. Hence: the lane is picked by elect.sync, which tells the compiler that one thread is active (under
// `lane == 0` every instruction with uniform operands, MMAs, commits and copies, became a loop over lanes); stages are
// counted, not divided; descriptors differ from stage to stage in their low word only; and the loop polls its one barrier, nothing else.
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(one));
  return one != 0;
}
template <int STAGES> struct RingPos {
  uint32_t s = 0, phase = 0;  // stage, and the parity that its barrier completes next
  __device__ __forceinline__ void next() {
    if (++s == STAGES) {
      s = 0;
      phase ^= 1u;
    }
  }
};

// Shared-memory matrix descriptor: K-major tile, 128-byte swizzle, 8-row groups 1024 B apart. Low word: start address
// in 16-byte units, leading-dimension offset 1 (unused with swizzle); the high one (mma_f16): stride between the groups,
// descriptor version of this architecture, 128-byte swizzle.
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | 1u << 16; }

// One K slice of 16: descriptors by their low words (the high one is the same for every address).
template <int CTAS> __device__ __forceinline__ void mma_f16(uint32_t acc, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, bool accumulate) {
  constexpr uint32_t hi = (1024u >> 4) | 1u << 14 | 2u << 29;
  if constexpr (CTAS == 1)
    asm volatile(
        "{\n .reg .pred p;\n .reg .b64 a, b;\n mov.b64 a, {%1, %3};\n mov.b64 b, {%2, %3};\n setp.ne.b32 p, %5, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n}" ::"r"(acc), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred p;\n .reg .b64 a, b;\n mov.b64 a, {%1, %3};\n mov.b64 b, {%2, %3};\n setp.ne.b32 p, %5, 0;\n"
        " tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, p;\n}" ::"r"(acc), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}
// arrives on this CTA's barrier once every MMA issued so far has completed (implies fence::before_thread_sync)
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// kind::f16 instruction descriptor: fp16 x fp16 or bf16 x bf16 -> fp32, both operands K-major, M x N tile.
__host__ __device__ constexpr uint32_t instr_desc(uint32_t m, uint32_t n, bool bf) {
  return (1u << 4) | (bf ? (1u << 7) | (1u << 10) : 0u) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
               : "memory");
}

template <int COLS> __device__ __forceinline__ void tmem_alloc(uint32_t dst_smem) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"((uint32_t)COLS) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

struct WeightMaps {
  CUtensorMap w[3];
};

// 32 outputs fp16(silu(gate) * up) of a row, of which n exist (n a multiple of 8).
__device__ __forceinline__ void swiglu_chunk(const float (&gate)[32], const float (&up)[32], __half *out, uint32_t n) {
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    if (j >= n) break;
    union {
      uint4 u;
      __half h[8];
    } y;
#pragma unroll
    for (int i = 0; i < 8; ++i) y.h[i] = __float2half_rn(gate[j + i] / (1.0f + expf(-gate[j + i])) * up[j + i]);
    *reinterpret_cast<uint4 *>(out + j) = y.u;
  }
}
// 32 results of matrix `mat`: this row's columns from n on, rounded as GemmParams says.
__device__ __forceinline__ void f16_chunk(const GemmParams &p, uint32_t mat, uint32_t row, uint32_t n, const float (&acc)[32]) {
  const size_t o = (size_t)row * p.N + n;
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    if (n + j >= p.N) break;  // N is a multiple of 8
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i] = acc[j + i] * p.scale + p.bias;
      if (p.act == 1) v[i] = v[i] / (1.0f + expf(-v[i]));
    }
    if (p.c_f32) {
      *reinterpret_cast<float4 *>(p.c_f32 + o + j) = make_float4(v[0], v[1], v[2], v[3]);
      *reinterpret_cast<float4 *>(p.c_f32 + o + j + 4) = make_float4(v[4], v[5], v[6], v[7]);
    } else {
      union {
        uint4 u;
        __half h[8];
      } out, res;
      if (p.residual) {
        res.u = *reinterpret_cast<const uint4 *>(p.residual + o + j);
#pragma unroll
        for (int i = 0; i < 8; ++i) out.h[i] = __float2half_rn(round_h(v[i]) + __half2float(res.h[i]));
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) out.h[i] = __float2half_rn(v[i]);
      }
      *reinterpret_cast<uint4 *>(p.c[mat] + o + j) = out.u;
    }
  }
}

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                 const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
  static EncodeTiled fn = [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
    return reinterpret_cast<EncodeTiled>(f);
  }();
  return fn;
}

// Tensor map over a row-major fp16 or bf16 matrix [rows, K]: boxes of 64 columns x box_rows rows,
// 128-byte swizzle, rows beyond the matrix read as zero.
bool make_map(CUtensorMap *map, const void *base, uint32_t rows, uint32_t K, uint32_t box_rows, bool bf = false) {
  EncodeTiled enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t dims[2] = {K, rows};
  const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {BK, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return enc(map, bf ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// SMs of the current device (the tile shape is chosen so that the grid still fills them).
inline size_t sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
  return (size_t)n;
}

}  // namespace
}  // namespace vkl
