// Attention core of the model path: RoPE(q), RoPE(k), KV-cache append, causal
// softmax(q.K^T/sqrt(d)).V over the fp16 cache, split over the KV length with a
// fixed-order combine. One kernel for decode (T = 1); for multi-token calls a
// small rotate-and-append kernel runs first.
//
// Replaces this op chain of the reference (src/ops/multiheadattention_v2.cpp:
// 236-309): Transpose x3, Rope x2 (rope_fp16.comp), UpdateKVCache x2
// (update_kvcache_fp16.comp), MatMul Q.K^T (matmul_b0_tb_fp16_v2.comp), Softmax
// (softmax_fp16.comp), MatMul P.V (matmul_broadcast0_fp16_v2.comp), Transpose.
// Rounding points kept: roped q and k are fp16, the scaled score is rounded to
// fp16 before the softmax, the head output is fp16. The probabilities are kept
// in fp32 here (the reference stores them as fp16 between two dispatches).
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "common.cuh"
#include "kernels.h"

namespace vkl {
namespace {

constexpr int kAttnThreads = 128;
constexpr uint32_t kMostSplits = 8;  // parts of a cache

__device__ __forceinline__ void rope_pair(float x0, float x1, float c, float s, __half &o0,
                                          __half &o1) {
  o0 = __float2half_rn(x0 * c - x1 * s);
  o1 = __float2half_rn(x0 * s + x1 * c);
}

// Eight consecutive dimensions d .. d + 7 of a row at position pos, rotated.
__device__ __forceinline__ uint4 rope8(uint4 raw, const AttnParams &p, size_t pos, uint32_t d) {
  union {
    uint4 u;
    __half h[8];
  } x;
  x.u = raw;
  const size_t fi = pos * (p.dim / 2) + d / 2;
  const float4 c = __ldg(reinterpret_cast<const float4 *>(p.freqc + fi)), s = __ldg(reinterpret_cast<const float4 *>(p.freqs + fi));
  const float cs[4] = {c.x, c.y, c.z, c.w}, sn[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) rope_pair(__half2float(x.h[2 * i]), __half2float(x.h[2 * i + 1]), cs[i], sn[i], x.h[2 * i], x.h[2 * i + 1]);
  return x.u;
}

// Multi-token calls: cache[h,(pos+m)%maxlen,:] = rope(k[m,h,:]) and v likewise. A thread moves eight dimensions with
// 16-byte accesses (the head width is a multiple of 8): bound by memory. 2048 rows of 32 heads x 128: 36 us with a
// thread per pair and 64 threads per block, 10 this way.
__global__ void __launch_bounds__(256) rope_append_kernel(const AttnParams p) {
  const uint32_t vecs = p.dim / 8, row = p.heads * vecs;
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= (size_t)p.T * row) return;
  const uint32_t m = (uint32_t)(i / row), c = (uint32_t)(i % row), h = c / vecs, d = c % vecs * 8;
  const uint32_t pos = *p.pos_dev + m;
  const size_t src = (size_t)m * p.heads * p.dim + (size_t)c * 8, dst = ((size_t)h * p.maxlen + pos % p.maxlen) * p.dim + d;
  const uint4 k = __ldg(reinterpret_cast<const uint4 *>(p.k + src)), v = __ldg(reinterpret_cast<const uint4 *>(p.v + src));
  *reinterpret_cast<uint4 *>(p.kcache + dst) = rope8(k, p, pos, d);
  *reinterpret_cast<uint4 *>(p.vcache + dst) = v;
}

// Columns of a part of a cache of which a row sees `vis`. A short cache is one part, since the parts' merge costs 2 us (32 heads, one row of
// 65 columns, us: one part 6.7, two 9.5; of 101 8.5, 9.7), up to 128 columns where CTAs are few and up to 512 where they fill the SMs without
// parts (31 rows of up to 231: 33.5, four parts 35.2; 40 heads x 64 24.6, 33.3). Beyond, a part has 64 columns at least (12 rows, 16 heads,
// 212 columns: four of 64 13.2, seven of 32 16.7).
__host__ __device__ __forceinline__ uint32_t whole_columns(uint32_t splits) { return splits == kMostSplits ? 128 : 512; }
__device__ __forceinline__ uint32_t part_columns(uint32_t vis, uint32_t splits) {
  const uint32_t whole = whole_columns(splits);
  if (vis <= whole) return whole;
  return max(((vis + splits - 1) / splits + 31) & ~31u, 64u);
}

// grid (heads, T, splits), 128 threads. FUSED: T == 1, the CTA whose column
// range holds the new position rotates k, uses it and writes both cache rows.
template <bool FUSED>
__global__ void __launch_bounds__(kAttnThreads) attention_kernel(const AttnParams p) {
  extern __shared__ __align__(16) float sm[];
  const uint32_t h = blockIdx.x, m = p.clip ? p.T - 1 : blockIdx.y, split = blockIdx.z;
  const uint32_t D = p.dim, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float *q_s = sm;                 // [D] roped query, fp16-rounded values
  float *kn_s = sm + D;            // [D] roped new key (FUSED)
  float *red_s = sm + 2 * D;       // [2*D + 8] reduction scratch
  float *s_s = sm + 4 * D + 8;     // [chunk] scores, then probabilities

  if (p.use_pdl) asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t pos0 = *p.pos_dev;
  const uint32_t L = min(pos0 + p.T, p.maxlen);
  const uint32_t vis = min(L, m + (L - p.T) + 1);  // causal: col <= row + (W - H)
  const uint32_t chunk = part_columns(vis, p.splits);
  if (split * chunk >= vis) {
    if (p.use_pdl) asm volatile("griddepcontrol.launch_dependents;");
    return;
  }
  const uint32_t c0 = min(split * chunk, vis), c1 = min(c0 + chunk, vis);
  const uint32_t jn = pos0 % p.maxlen;  // FUSED: physical column of the new token
  const bool owns_new = FUSED && jn >= c0 && jn < c1;

  const size_t row_in = (size_t)m * p.heads * D + (size_t)h * D;
  if (2 * tid < D) {
    const size_t fi = (size_t)(pos0 + (p.clip ? 0u : m)) * (D / 2) + tid;
    const float c = p.freqc[fi], s = p.freqs[fi];
    __half r0, r1;
    rope_pair(__half2float(p.q[row_in + 2 * tid]), __half2float(p.q[row_in + 2 * tid + 1]), c, s, r0, r1);
    q_s[2 * tid] = __half2float(r0);
    q_s[2 * tid + 1] = __half2float(r1);
    if (owns_new) {
      rope_pair(__half2float(p.k[row_in + 2 * tid]), __half2float(p.k[row_in + 2 * tid + 1]), c, s, r0, r1);
      kn_s[2 * tid] = __half2float(r0);
      kn_s[2 * tid + 1] = __half2float(r1);
      const size_t dst = ((size_t)h * p.maxlen + jn) * D + 2 * tid;
      p.kcache[dst] = r0;
      p.kcache[dst + 1] = r1;
      p.vcache[dst] = p.v[row_in + 2 * tid];
      p.vcache[dst + 1] = p.v[row_in + 2 * tid + 1];
    }
  }
  __syncthreads();

  // ---- scores: one column per lane ----------------------------------------
  const float scale = 1.0f / sqrtf((float)D);
  const __half *kc = p.kcache + (size_t)h * p.maxlen * D;
  float lmax = -INFINITY;
  for (uint32_t j = c0 + tid; j < c1; j += kAttnThreads) {
    float acc = 0.f;
    if (owns_new && j == jn) {
      for (uint32_t d = 0; d < D; ++d) acc = fmaf(q_s[d], kn_s[d], acc);
    } else {
      const uint4 *kr = reinterpret_cast<const uint4 *>(kc + (size_t)j * D);
#pragma unroll 16  // the whole row in flight: one memory round trip per column
      for (uint32_t d8 = 0; d8 < D / 8; ++d8) {
        const uint4 kv = __ldg(kr + d8);
        const float4 qa = *reinterpret_cast<const float4 *>(q_s + d8 * 8);
        const float4 qb = *reinterpret_cast<const float4 *>(q_s + d8 * 8 + 4);
        const float2 k0 = __half22float2(*reinterpret_cast<const __half2 *>(&kv.x));
        const float2 k1 = __half22float2(*reinterpret_cast<const __half2 *>(&kv.y));
        const float2 k2 = __half22float2(*reinterpret_cast<const __half2 *>(&kv.z));
        const float2 k3 = __half22float2(*reinterpret_cast<const __half2 *>(&kv.w));
        acc = fmaf(qa.x, k0.x, acc);
        acc = fmaf(qa.y, k0.y, acc);
        acc = fmaf(qa.z, k1.x, acc);
        acc = fmaf(qa.w, k1.y, acc);
        acc = fmaf(qb.x, k2.x, acc);
        acc = fmaf(qb.y, k2.y, acc);
        acc = fmaf(qb.z, k3.x, acc);
        acc = fmaf(qb.w, k3.y, acc);
      }
    }
    const float sc = round_h(acc * scale);
    s_s[j - c0] = sc;
    lmax = fmaxf(lmax, sc);
  }
  lmax = warp_max(lmax);
  if (lane == 0) red_s[warp] = lmax;
  __syncthreads();
  const float mloc = fmaxf(fmaxf(red_s[0], red_s[1]), fmaxf(red_s[2], red_s[3]));
  __syncthreads();
  float lsum = 0.f;
  for (uint32_t j = c0 + tid; j < c1; j += kAttnThreads) {
    const float pj = expf(s_s[j - c0] - mloc);
    s_s[j - c0] = pj;
    lsum += pj;
  }
  lsum = warp_sum(lsum);
  if (lane == 0) red_s[4 + warp] = lsum;
  __syncthreads();
  const float lloc = red_s[4] + red_s[5] + red_s[6] + red_s[7];

  // ---- P.V: thread = (column parity group, dim pair) ----------------------
  const uint32_t npair = D / 2;  // <= 64
  const uint32_t grp = tid / 64, dp = tid % 64;
  float2 acc = make_float2(0.f, 0.f);
  if (dp < npair) {
    const __half *vc = p.vcache + (size_t)h * p.maxlen * D + 2 * dp;
    constexpr uint32_t UN = 8;  // cache rows in flight per thread
    for (uint32_t jb = c0 + grp; jb < c1; jb += 2 * UN) {
      uint32_t raw[UN];
#pragma unroll
      for (uint32_t u = 0; u < UN; ++u) {
        const uint32_t j = jb + 2 * u;
        raw[u] = 0;
        if (j < c1)
          raw[u] = (owns_new && j == jn) ? *reinterpret_cast<const uint32_t *>(p.v + row_in + 2 * dp)
                                         : __ldg(reinterpret_cast<const uint32_t *>(vc + (size_t)j * D));
      }
#pragma unroll
      for (uint32_t u = 0; u < UN; ++u) {
        const uint32_t j = jb + 2 * u;
        if (j < c1) {
          const float2 vv = __half22float2(*reinterpret_cast<const __half2 *>(&raw[u]));
          const float pj = s_s[j - c0];
          acc.x = fmaf(pj, vv.x, acc.x);
          acc.y = fmaf(pj, vv.y, acc.y);
        }
      }
    }
  }
  __syncthreads();
  if (grp == 1 && dp < npair) {
    red_s[8 + 2 * dp] = acc.x;
    red_s[8 + 2 * dp + 1] = acc.y;
  }
  __syncthreads();
  if (grp == 0 && dp < npair) {
    acc.x += red_s[8 + 2 * dp];
    acc.y += red_s[8 + 2 * dp + 1];
  }
  if (p.use_pdl) asm volatile("griddepcontrol.launch_dependents;");

  __half *orow = p.out + (p.clip ? (size_t)h * D : row_in);
  if (chunk >= vis) {
    if (grp == 0 && dp < npair) {
      orow[2 * dp] = __float2half_rn(acc.x / lloc);
      orow[2 * dp + 1] = __float2half_rn(acc.y / lloc);
    }
    return;
  }
  // ---- split combine: last CTA to arrive sums the partials in split order --
  const size_t unit = (size_t)blockIdx.y * p.heads + h;
  float *part = p.scratch + (unit * p.splits + split) * (D + 2);
  if (grp == 0 && dp < npair) {
    part[2 * dp] = acc.x;
    part[2 * dp + 1] = acc.y;
  }
  if (tid == 0) {
    part[D] = mloc;
    part[D + 1] = lloc;
  }
  const uint32_t parts = (vis + chunk - 1) / chunk;
  __threadfence();
  __syncthreads();
  __shared__ uint32_t s_last;
  if (tid == 0) s_last = atomicAdd(&p.counters[unit], 1u) == parts - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const float *base = p.scratch + unit * p.splits * (D + 2);
  for (uint32_t d = tid; d < D; d += kAttnThreads) {
    float M = -INFINITY, den = 0.f, num = 0.f;
#pragma unroll 1
    for (uint32_t s0 = 0; s0 < parts; s0 += 4) {  // four parts' loads in flight together
      float ms[4], ls[4], v[4], m = M;
#pragma unroll
      for (uint32_t s = 0; s < 4; ++s) {
        const float *part = base + (s0 + s) * (D + 2);
        const bool here = s0 + s < parts;
        ms[s] = here ? __ldcg(part + D) : -INFINITY;
        ls[s] = here ? __ldcg(part + D + 1) : 0.f;
        v[s] = here ? __ldcg(part + d) : 0.f;
      }
#pragma unroll
      for (uint32_t s = 0; s < 4; ++s) m = fmaxf(m, ms[s]);
      const float keep = M == m ? 1.f : expf(M - m);
      den *= keep;
      num *= keep;
      M = m;
#pragma unroll
      for (uint32_t s = 0; s < 4; ++s) {
        if (ls[s] > 0.f) {
          const float w = expf(ms[s] - M);
          den += ls[s] * w;
          num += v[s] * w;
        }
      }
    }
    orow[d] = __float2half_rn(num / den);
  }
  if (tid == 0) p.counters[unit] = 0;
}

size_t attn_smem(const AttnParams &p) {  // scores of the longest part
  const uint32_t chunk = std::max(((p.maxlen + p.splits - 1) / p.splits + 31) & ~31u, std::min(whole_columns(p.splits), p.maxlen));
  return (size_t)(4 * p.dim + 8 + chunk) * sizeof(float);
}

// ---- multi-token calls with many rows: 64 query rows of one head per CTA ----------------------
// The per-row kernel above re-reads the head's K and V rows for every query row. This one stages
// a 64-position K/V tile in shared memory once for 64 query rows and runs both products on the
// tensor cores (mma.sync m16n8k16, fp32 accumulate): S = Q.K^T per warp of 16 rows, the scaled
// score rounded to fp16 as the reference's softmax input is, a running (max, sum) per row, the
// probabilities as fp16 MMA operands (the reference stores them as fp16 between two dispatches),
// O += P.V with V fragments transposed by ldmatrix. Columns are physical cache rows 0..L-1 with
// the reference's mask col <= row + (L - T) (softmax_fp16.comp:52-60), so a wrapped ring behaves
// as in the per-row kernel.
//
// Bound: the mma.sync pipe (a quarter of the tcgen05 rate) beside the softmax's instructions. So all fragments
// come by ldmatrix, the V tile is on its way (cp.async) during Q.K^T and the next K tile during P.V, only
// tiles at the causal edge are masked, and one tile of each (52 KB) leaves room for three CTAs per SM that hide each
// other's softmax. Few query tiles behind a long cache do not fill the SMs: the cache is then split
// (grid z, at least kSplitTiles tiles each) and the CTA of a query tile that finishes last merges the parts in order.
// 32 heads x 128, 2048 rows: 255 us with scalar fragment loads and no overlap, 140 now (244 TFLOP/s of the causal half);
// 40 heads, 45 rows behind 700: 66 -> 19 us, mostly by the splits.
__device__ __forceinline__ void mma16816_h(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
  const __half2 v = __halves2half2(__float2half_rn(lo), __float2half_rn(hi));
  return *reinterpret_cast<const uint32_t *>(&v);
}

__device__ __forceinline__ void ldm4(uint32_t (&r)[4], const __half *p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], const __half *p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

constexpr uint32_t kSplitTiles = 2;   // a split of the tile kernel holds at least this many 64-row cache tiles
constexpr float kLog2e = 1.4426950408889634f;

template <int D>
__global__ void __launch_bounds__(128, 3) attention_tile_kernel(const AttnParams p) {
  constexpr int QT = 64, KT = 64, LD = D + 8;  // padded rows: conflict-free fragment loads
  extern __shared__ __align__(16) __half smh[];
  __half *q_s = smh;             // [QT][LD] roped queries
  __half *k_s = q_s + QT * LD;   // [KT][LD]
  __half *v_s = k_s + KT * LD;   // [KT][LD]
  __shared__ uint32_t last_s;
  const uint32_t h = blockIdx.x, qt = gridDim.y - 1 - blockIdx.y, m0 = qt * QT;  // longest rows first
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const uint32_t T = p.T, pos0 = *p.pos_dev;
  const uint32_t L = min(pos0 + T, p.maxlen), shift = L - T;
  const uint32_t jmax = min(L, min(m0 + QT, T) + shift);  // columns any row of this tile can see
  const uint32_t tiles = (jmax + KT - 1) / KT;
  const uint32_t most = min(gridDim.z, (tiles + kSplitTiles - 1) / kSplitTiles), per = (tiles + most - 1) / most, splits = (tiles + per - 1) / per;
  const uint32_t split = blockIdx.z;
  if (split >= splits) return;
  const uint32_t j_begin = split * per * KT, j_end = min(jmax, j_begin + per * KT);
  const __half *kc = p.kcache + (size_t)h * p.maxlen * D, *vc = p.vcache + (size_t)h * p.maxlen * D;
  auto fetch = [&](__half *dst, const __half *src, uint32_t j0) {  // 64 cache rows; those beyond L become zero
#pragma unroll
    for (uint32_t i = tid; i < KT * (D / 8); i += 128) {
      const uint32_t r = i / (D / 8), c8 = i % (D / 8), j = j0 + r;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + r * LD + c8 * 8)),
                   "l"(src + (j < L ? (size_t)j * D + c8 * 8 : 0)), "r"(j < L ? 16u : 0u)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(k_s, kc, j_begin);
  for (uint32_t i = tid; i < QT * (D / 8); i += 128) {  // rotate the query tile at positions pos0 + row
    const uint32_t r = i / (D / 8), d = i % (D / 8) * 8, m = m0 + r;
    uint4 q = make_uint4(0, 0, 0, 0);
    if (m < T) q = rope8(__ldg(reinterpret_cast<const uint4 *>(p.q + (size_t)m * p.heads * D + (size_t)h * D + d)), p, (size_t)pos0 + m, d);
    *reinterpret_cast<uint4 *>(q_s + r * LD + d) = q;
  }
  const uint32_t r_lo = m0 + warp * 16 + g, r_hi = r_lo + 8;
  const uint32_t vis_lo = r_lo < T ? min(L, r_lo + shift + 1) : 0u, vis_hi = r_hi < T ? min(L, r_hi + shift + 1) : 0u;
  const uint32_t vis_all = m0 + warp * 16 + 15 < T ? min(L, m0 + warp * 16 + shift + 1) : 0u;  // columns that all of the warp's rows see
  const float scale = 1.0f / sqrtf((float)D);
  float o[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m_lo = -INFINITY, m_hi = -INFINITY, l_lo = 0.f, l_hi = 0.f;  // l: this thread's columns, summed over the row's four threads at the end
  const __half *qf = q_s + (warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LD + (lane >> 4) * 8;
  const __half *kf = k_s + ((lane & 7) + (lane >> 4) * 8) * LD + ((lane >> 3) & 1) * 8;
  const __half *vf = v_s + ((lane & 7) + ((lane >> 3) & 1) * 8) * LD + (lane >> 4) * 8;
  for (uint32_t j0 = j_begin; j0 < j_end; j0 += KT) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the K tile is here for everyone (first time: the query tile too), the last V tile is consumed
    fetch(v_s, vc, j0);
    // ---- S = Q.K^T: 16 rows x 64 columns per warp
    float sc[KT / 8][4];
#pragma unroll
    for (int nt = 0; nt < KT / 8; ++nt) sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      uint32_t a[4], b[4];
      ldm4(a, qf + kk * 16);
#pragma unroll
      for (int nt = 0; nt < KT / 8; nt += 2) {
        ldm4(b, kf + nt * 8 * LD + kk * 16);
        mma16816_h(sc[nt], a[0], a[1], a[2], a[3], b[0], b[1]);
        mma16816_h(sc[nt + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
      }
    }
    // ---- scaled fp16 scores, mask, running max and sum
    float tmax_lo = -INFINITY, tmax_hi = -INFINITY;
#pragma unroll
    for (int nt = 0; nt < KT / 8; ++nt) {
#pragma unroll
      for (int i = 0; i < 4; ++i) sc[nt][i] = round_h(sc[nt][i] * scale);
    }
    if (j0 + KT > vis_all) {  // uniform over the warp
#pragma unroll
      for (int nt = 0; nt < KT / 8; ++nt) {
        const uint32_t c = j0 + nt * 8 + 2 * t;
        if (c >= vis_lo) sc[nt][0] = -INFINITY;
        if (c + 1 >= vis_lo) sc[nt][1] = -INFINITY;
        if (c >= vis_hi) sc[nt][2] = -INFINITY;
        if (c + 1 >= vis_hi) sc[nt][3] = -INFINITY;
      }
    }
#pragma unroll
    for (int nt = 0; nt < KT / 8; ++nt) {
      tmax_lo = fmaxf(tmax_lo, fmaxf(sc[nt][0], sc[nt][1]));
      tmax_hi = fmaxf(tmax_hi, fmaxf(sc[nt][2], sc[nt][3]));
    }
#pragma unroll
    for (int w = 1; w < 4; w <<= 1) {
      tmax_lo = fmaxf(tmax_lo, __shfl_xor_sync(0xffffffffu, tmax_lo, w));
      tmax_hi = fmaxf(tmax_hi, __shfl_xor_sync(0xffffffffu, tmax_hi, w));
    }
    const float mn_lo = fmaxf(m_lo, tmax_lo), mn_hi = fmaxf(m_hi, tmax_hi);
    const float ref_lo = mn_lo == -INFINITY ? 0.f : mn_lo, ref_hi = mn_hi == -INFINITY ? 0.f : mn_hi;
    const float corr_lo = exp2f((m_lo - ref_lo) * kLog2e), corr_hi = exp2f((m_hi - ref_hi) * kLog2e);
    m_lo = mn_lo;
    m_hi = mn_hi;
    float rs_lo = 0.f, rs_hi = 0.f;
#pragma unroll
    for (int nt = 0; nt < KT / 8; ++nt) {
      sc[nt][0] = exp2f((sc[nt][0] - ref_lo) * kLog2e);
      sc[nt][1] = exp2f((sc[nt][1] - ref_lo) * kLog2e);
      sc[nt][2] = exp2f((sc[nt][2] - ref_hi) * kLog2e);
      sc[nt][3] = exp2f((sc[nt][3] - ref_hi) * kLog2e);
      rs_lo += sc[nt][0] + sc[nt][1];
      rs_hi += sc[nt][2] + sc[nt][3];
    }
    l_lo = l_lo * corr_lo + rs_lo;
    l_hi = l_hi * corr_hi + rs_hi;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      o[i][0] *= corr_lo;
      o[i][1] *= corr_lo;
      o[i][2] *= corr_hi;
      o[i][3] *= corr_hi;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the V tile is here for everyone, the K tile is consumed
    if (j0 + KT < j_end) fetch(k_s, kc, j0 + KT);
    // ---- O += P.V: 16 cache rows per step, V fragments transposed by ldmatrix
#pragma unroll
    for (int j16 = 0; j16 < KT / 16; ++j16) {
      const uint32_t a0 = pack_h2(sc[2 * j16][0], sc[2 * j16][1]), a1 = pack_h2(sc[2 * j16][2], sc[2 * j16][3]);
      const uint32_t a2 = pack_h2(sc[2 * j16 + 1][0], sc[2 * j16 + 1][1]), a3 = pack_h2(sc[2 * j16 + 1][2], sc[2 * j16 + 1][3]);
#pragma unroll
      for (int dt = 0; dt < D / 16; ++dt) {
        uint32_t b[4];
        ldm4t(b, vf + j16 * 16 * LD + dt * 16);
        mma16816_h(o[2 * dt], a0, a1, a2, a3, b[0], b[1]);
        mma16816_h(o[2 * dt + 1], a0, a1, a2, a3, b[2], b[3]);
      }
    }
  }
#pragma unroll
  for (int w = 1; w < 4; w <<= 1) {
    l_lo += __shfl_xor_sync(0xffffffffu, l_lo, w);
    l_hi += __shfl_xor_sync(0xffffffffu, l_hi, w);
  }
  if (splits > 1) {
    // ---- a part per split, in this kernel's own fragment order: [D / 8 + 1][128 threads] x 16 bytes
    constexpr uint32_t kPart = (D / 8 + 1) * 128;
    const uint32_t unit = qt * p.heads + h;
    float4 *part = reinterpret_cast<float4 *>(p.scratch) + (size_t)unit * gridDim.z * kPart + tid;
    float4 *mine = part + (size_t)split * kPart;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) __stcg(mine + i * 128, make_float4(o[i][0], o[i][1], o[i][2], o[i][3]));
    __stcg(mine + D / 8 * 128, make_float4(m_lo, m_hi, l_lo, l_hi));
    __threadfence();
    __syncthreads();
    if (tid == 0) last_s = atomicAdd(&p.counters[unit], 1u) == splits - 1;
    __syncthreads();
    if (!last_s) return;
    __threadfence();
    float M_lo = -INFINITY, M_hi = -INFINITY;
    for (uint32_t s = 0; s < splits; ++s) {
      const float4 ml = __ldcg(part + (size_t)s * kPart + D / 8 * 128);
      M_lo = fmaxf(M_lo, ml.x);
      M_hi = fmaxf(M_hi, ml.y);
    }
    if (M_lo == -INFINITY) M_lo = 0.f;
    if (M_hi == -INFINITY) M_hi = 0.f;
    l_lo = l_hi = 0.f;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    for (uint32_t s = 0; s < splits; ++s) {
      const float4 ml = __ldcg(part + (size_t)s * kPart + D / 8 * 128);
      const float c_lo = exp2f((ml.x - M_lo) * kLog2e), c_hi = exp2f((ml.y - M_hi) * kLog2e);
      l_lo = fmaf(c_lo, ml.z, l_lo);
      l_hi = fmaf(c_hi, ml.w, l_hi);
#pragma unroll
      for (int i = 0; i < D / 8; ++i) {
        const float4 v = __ldcg(part + (size_t)s * kPart + i * 128);
        o[i][0] = fmaf(c_lo, v.x, o[i][0]);
        o[i][1] = fmaf(c_lo, v.y, o[i][1]);
        o[i][2] = fmaf(c_hi, v.z, o[i][2]);
        o[i][3] = fmaf(c_hi, v.w, o[i][3]);
      }
    }
    if (tid == 0) p.counters[unit] = 0;
  }
  // ---- out[m, h*D + d] = fp16(O / sum)
  const float inv_lo = l_lo > 0.f ? 1.0f / l_lo : 0.f, inv_hi = l_hi > 0.f ? 1.0f / l_hi : 0.f;
#pragma unroll
  for (int nt = 0; nt < D / 8; ++nt) {
    const uint32_t d = nt * 8 + 2 * t;
    if (r_lo < T) *reinterpret_cast<uint32_t *>(p.out + (size_t)r_lo * p.heads * D + (size_t)h * D + d) = pack_h2(o[nt][0] * inv_lo, o[nt][1] * inv_lo);
    if (r_hi < T) *reinterpret_cast<uint32_t *>(p.out + (size_t)r_hi * p.heads * D + (size_t)h * D + d) = pack_h2(o[nt][2] * inv_hi, o[nt][3] * inv_hi);
  }
}

constexpr uint32_t kTileMinRows = 32;  // below this the per-row kernel is used
constexpr uint32_t kMostUnits = 16;    // rows x heads per SM up to which a row's cache is split

bool use_tiles(uint32_t T, bool clip, uint32_t dim) {
  static const bool off = [] { const char *e = getenv("VKLLAMA_PREFILL_ATTENTION"); return e && !strcmp(e, "rows"); }();
  return !off && T >= kTileMinRows && !clip && (dim == 64 || dim == 128);
}

}  // namespace

// Parts that a cache is split into at most; a kernel uses fewer where the cache is short. Tiles: up to three CTAs per SM. Rows (128
// threads each, a serial walk over the part): eight, as in decode, while that is up to 16 CTAs per SM, else four, whose idle CTAs cost less
// on short caches. us in one / four / eight parts: 32 heads x 128, the last row of 2048 129 / 46 / 33; 3 rows behind 2000 96 / 40 / 36;
// 31 rows behind 700 97 / 83 / 83, behind nothing 7.9 / 8.1 / 8.3; 40 heads, 31 rows behind nothing 8.5 / 8.8 / 10.3.
AttnPlan attention_plan(uint32_t T, bool clip, uint32_t heads, uint32_t dim, uint32_t sms) {
  AttnPlan a = {};
  const bool tiles = use_tiles(T, clip, dim);
  const uint32_t rows = tiles ? (T + 63) / 64 : clip ? 1 : T, units = rows * heads;
  if (tiles) a.splits = std::min(std::max(3 * sms / units, 1u), kMostSplits);
  else a.splits = rows == 1 || units <= 2 * sms ? kMostSplits : units <= kMostUnits * sms ? 4 : 1;
  a.scratch_bytes = a.splits == 1 ? 0 : (size_t)units * a.splits * (tiles ? 64 * (dim + 8) : dim + 2) * sizeof(float);
  a.counters = units;
  return a;
}
AttnPlan attention_plan_most(uint32_t T, uint32_t heads, uint32_t dim, uint32_t sms) {
  AttnPlan a = {};
  a.splits = kMostSplits;
  // rows: eight parts of a single one or of up to 2 * sms, four of up to kMostUnits * sms
  const size_t row_parts = std::max({(size_t)kMostSplits * heads, (size_t)kMostSplits * 2 * sms, T > 1 ? (size_t)4 * kMostUnits * sms : 0});
  const size_t tile_units = std::min((size_t)3 * sms, (size_t)kMostSplits * heads * ((T + 63) / 64));
  a.scratch_bytes = row_parts * (dim + 2) * sizeof(float);
  if (T >= kTileMinRows && a.scratch_bytes < tile_units * 64 * (dim + 8) * sizeof(float)) a.scratch_bytes = tile_units * 64 * (dim + 8) * sizeof(float);
  a.counters = std::max(heads, kMostUnits * sms);
  return a;
}

cudaError_t launch_attention(const AttnParams &p, cudaStream_t s) {
  if (p.dim > 128 || (p.dim & 7) || p.T == 0) return cudaErrorInvalidValue;
  if (p.T > 1) {
    const size_t n = (size_t)p.T * p.heads * (p.dim / 8);
    rope_append_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(p);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (use_tiles(p.T, p.clip, p.dim)) {
    const size_t tsmem = (size_t)3 * 64 * (p.dim + 8) * sizeof(__half);
    auto tk = p.dim == 128 ? attention_tile_kernel<128> : attention_tile_kernel<64>;
    cudaError_t e = cudaFuncSetAttribute(tk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsmem);
    if (e != cudaSuccess) return e;
    tk<<<dim3(p.heads, (p.T + 63) / 64, p.splits), 128, tsmem, s>>>(p);
    return cudaGetLastError();
  }
  const size_t smem = attn_smem(p);
  auto kern = p.T == 1 ? attention_kernel<true> : attention_kernel<false>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.heads, p.clip ? 1 : p.T, p.splits);
  cfg.blockDim = dim3(kAttnThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (p.use_pdl && p.T == 1) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, p);
}

}  // namespace vkl
