// One persistent kernel per decode token (Q8_0 or FP16 weights, batch 1).
//
// The reference records 19 Vulkan dispatches per layer per token
// (models/llama2.h:160-213, src/ops/multiheadattention_v2.cpp:190-319) and stalls
// the weight stream at every one of them. Here the whole token is one
// cooperative launch of one CTA per SM:
//
//   * what a CTA reads of an op is one consecutive range of the op's packed stream, cut into equal shares, one per
//     warp. Every warp streams its share through a ring of its own in shared memory with bulk-copy TMA
//     (cp.async.bulk + mbarrier): as soon as it has used a piece (MEGA_SU units), its lane 0 requests the piece
//     that takes its place, across op boundaries. Weights never depend on activations, so HBM stays busy while
//     the warps sit in a norm, an attention op or a wait;
//   * a unit is one Q8_0 block x 32 rows (FP16: 16 columns x 32 rows, MMA operands as they are): the codes go into the tensor cores as fp16 subnormals (exact, one
//     byte permute per pair; m16n8k16, fp32 accumulate), block scales are applied in fp32, the warps' sums of
//     a tile are added in fixed order and the fused epilogue runs (RMSNorm prologue, residual add, SwiGLU, fp32
//     logits, running arg-max);
//   * activations cross CTAs as tagged words (value + sequence tag in one 32-bit word) that
//     the readers poll; only the output layer's arg-max needs a grid barrier.
//
// Tiles of op i go to CTA (tile + rot_i) mod grid; rot_i advances by the op's
// tile count so the uneven remainder rotates over the SMs.
//
// What bounds it: not HBM (7B: 1.45 ms per token against 1.07 at the measured copy rate) and not the tensor pipe (12 %), but
// what a warp executes one instruction after the other: with three warps per scheduler and dependent instructions four to six
// cycles apart, a branch costs 50 to 100 cycles of a warp's time and even an empty turn of the stream loop took 400. With no
// weight copies at all a 7B token of this form's first version took 1.49 of its 1.53 ms. Hence: no producer warp and no barrier pair
// per stage between warps (its handshake, table entry and two units per stage and warp bounded the earlier form: 1.60 ms);
// straight-line code for whole pieces; divisions, addresses and residuals worked out before the input arrives; and little code
// and no spills, because both come from memory behind the weight stream when they miss (150 KB of code 1.68 ms, 123 KB
// 1.60, 80 KB 1.53 for like loops; 16 warps of 128 registers with 200 bytes of spills 1.9 to 2.0 ms).
// Warps x units per piece, ms per token (7B) / us per call (13B shape, four blocks): 11 x 4 1.453 / 399, 11 x 5 1.482 / 399,
// 12 x 3 1.464 / 397, 12 x 4 1.497 / 386, 12 x 5 1.477 / 385, 16 x 2 1.501 / 431, 16 x 3 1.520 / 405: 11 x 4 has the deepest
// rings at 7B (four pieces, 191 KB).
// Every wait is bounded; on a time-out the kernel raises *error, stops issuing
// copies, drains the copies in flight and leaves through the normal path.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace vkl {
namespace {

constexpr int NCW = (int)MEGA_NCW;     // warps: at most 184 registers per thread (160 to 168 are used)
constexpr int CT = NCW * 32;
constexpr int THREADS = CT;
constexpr int SU = (int)MEGA_SU;       // units per piece, the step of a warp's ring
constexpr uint32_t UNIT_CODES = MEGA_UNIT_CODES, UNIT_SCALES = MEGA_UNIT_SCALES;
constexpr uint32_t UNIT_BYTES = UNIT_CODES + UNIT_SCALES;  // a unit's codes, then its 32 scales
constexpr uint32_t PIECE_BYTES = SU * UNIT_BYTES;
static_assert(PIECE_BYTES == MEGA_PIECE_BYTES, "host and device agree on the size of a piece");
template <bool F16> struct Unit {  // bytes; columns of a unit
  static constexpr uint32_t BYTES = F16 ? MEGA_UNIT_CODES : UNIT_BYTES, COLUMNS = F16 ? 16 : 32;
};
constexpr uint32_t XB_BYTES = 64;      // the input vector in shared memory: fp16, 64 bytes per block of 32 inputs
constexpr int MAX_NST = (int)MEGA_MAX_NST;  // a ring's pieces are a launch parameter (whatever fits), at most this many
// Every wait of the kernel is bounded by MegaParams::wait_limit polls (about half a microsecond each): the host
// picks the bound, the same for all waits, so that no wait gives up while another one it depends on is still
// legitimately waiting (for a slower tensor-parallel rank, say).

__device__ __forceinline__ uint32_t s32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t a, uint32_t tx) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(tx) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t a) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(a), "r"(parity)
      : "memory");
  return ok;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ void cons_sync() { asm volatile("bar.sync 1, %0;" ::"n"(CT) : "memory"); }
__device__ __forceinline__ uint32_t ld_acq_sys_u32(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_rel_sys_u32(uint32_t *p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Eight halves as floats.
__device__ __forceinline__ void unpack8(const uint4 &v, float *f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&w[e]));
    f[2 * e] = a.x;
    f[2 * e + 1] = a.y;
  }
}
// ---- tagged activation words: fp16 value | (low 16 bits of the producing op's sequence number) << 16
__device__ __forceinline__ uint32_t ll_pack(__half v, uint32_t tag) { return (uint32_t)__half_as_ushort(v) | (tag << 16); }
__device__ __forceinline__ __half ll_half(uint32_t w) { return __ushort_as_half((unsigned short)(w & 0xffffu)); }
__device__ __forceinline__ uint32_t ld_vol_u32(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.volatile.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint2 ld_vol_v2(const uint32_t *p) {
  uint2 v;
  asm volatile("ld.volatile.global.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_vol_v4(const uint32_t *p) {
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

// Read-only 128-bit load that keeps its place among the volatile polls around it (a plain
// __ldg may be scheduled after them, behind a spin).
__device__ __forceinline__ float4 ldg_f4_ordered(const float4 *p) {
  float4 v;
  asm volatile("ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ uint64_t ld_acq_u64(const unsigned long long *p) {
  uint64_t v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ bool getenv_prologue(const MegaParams &p) { return (p.timing_mode & 1u) != 0; }
__device__ __forceinline__ unsigned long long gtime() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Trace mode (timing_mode bit 256, TIMED instances): thread 0 of EVERY CTA stamps the global
// timer at fixed points of every op: [0] op entered, [1] input vector complete (after the
// norm), [2] this warp's stream done, [3] all warps' streams done, [4] results stored,
// [5] end-of-op synchronisation passed. Layout: trace[(op * grid + cta) * 8 + k].
#define VKL_TRACE(k)                                                   \
  do {                                                                 \
    if (TIMED && trace) trace[k] = gtime();                            \
  } while (0)

// The spin loops of the bounded waits. They are inlined like everything else in this kernel: kept out
// of line (to make the code smaller) they cost 10 % of the token time, the calls forcing the polled
// words through local memory and registers to be saved around every wait.
struct Ctx;
#define VKL_SLOW __forceinline__
__device__ VKL_SLOW bool slow_mbar_wait(volatile uint32_t *abort_s, uint32_t *error, uint32_t limit, uint32_t bar, uint32_t parity, uint32_t code) {
#pragma unroll 1
  for (uint32_t i = 0; i < limit; ++i) {
    if (mbar_try(bar, parity)) return true;
    if ((i & 255u) == 255u && (*(volatile uint32_t *)error != 0u || *abort_s != 0)) {
      *abort_s = 1;
      return false;
    }
  }
  *abort_s = 1;
  atomicCAS(error, 0u, code);
  return false;
}
__device__ VKL_SLOW uint32_t slow_ll_wait1(volatile uint32_t *abort_s, uint32_t *error, uint32_t limit, const uint32_t *src, uint32_t tag) {
  uint32_t w = 0;
#pragma unroll 1
  for (uint32_t i = 0; i < limit; ++i) {
    w = ld_vol_u32(src);
    if ((w >> 16) == tag) return w;
    if ((i & 255u) == 255u && (*(volatile uint32_t *)error != 0u || *abort_s != 0)) {
      *abort_s = 1;
      return w;
    }
  }
  *abort_s = 1;
  atomicCAS(error, 0u, 6u);
  return w;
}
__device__ __forceinline__ bool ll_ready8(const uint4 &a, const uint4 &b, uint32_t tag) {
  const uint32_t t = tag << 16;
  return (((a.x ^ t) | (a.y ^ t) | (a.z ^ t) | (a.w ^ t) | (b.x ^ t) | (b.y ^ t) | (b.z ^ t) | (b.w ^ t)) & 0xffff0000u) == 0;
}
__device__ __forceinline__ uint4 ll_pack8(const uint4 &a, const uint4 &b) {
  return make_uint4(__byte_perm(a.x, a.y, 0x5410), __byte_perm(a.z, a.w, 0x5410), __byte_perm(b.x, b.y, 0x5410), __byte_perm(b.z, b.w, 0x5410));
}
// polls eight consecutive tagged words until all carry `tag`; the words come back through a, b
__device__ VKL_SLOW void slow_ll_wait8(volatile uint32_t *abort_s, uint32_t *error, uint32_t limit, const uint32_t *src, uint32_t tag, uint4 &a, uint4 &b) {
#pragma unroll 1
  for (uint32_t i = 0; i < limit; ++i) {
    a = ld_vol_v4(src);
    b = ld_vol_v4(src + 4);
    if (ll_ready8(a, b, tag)) return;
    if ((i & 255u) == 255u && (*(volatile uint32_t *)error != 0u || *abort_s != 0)) {
      *abort_s = 1;  // give up quietly: another wait has already raised the error
      return;
    }
  }
  *abort_s = 1;
  atomicCAS(error, 0u, 6u);
}

struct Ctx {
  const MegaParams &p;
  volatile uint32_t *abort_s;  // shared flag: some wait of this CTA timed out or *error was seen
  __device__ __forceinline__ bool aborted() const { return *abort_s != 0; }
  // Under tensor parallelism an input may sit behind an all-reduce that is itself waiting for a slow
  // rank: the input's wait must outlast that one (four times its polls), so that the error names the wait that really failed.
  __device__ __forceinline__ uint32_t ll_limit() const { return p.tp_size > 1 ? (p.wait_limit < 0x40000000u ? 4u * p.wait_limit : 0xffffffffu) : p.wait_limit; }
  __device__ __forceinline__ void raise(uint32_t code) const {
    *abort_s = 1;
    atomicCAS(p.error, 0u, code);
  }
  // One tagged word, polled (bounded) until its tag is `tag`. Returns the word; on a time-out
  // or an abort returns what it last read (the caller's results are discarded on abort).
  __device__ __forceinline__ uint32_t ll_wait1(const uint32_t *src, uint32_t tag) const {
    const uint32_t w = ld_vol_u32(src);
    if ((w >> 16) == tag) return w;
    return slow_ll_wait1(abort_s, p.error, ll_limit(), src, tag);
  }
  // Eight consecutive tagged words (32-byte aligned), already requested once -> eight packed halves, polled the same way.
  __device__ __forceinline__ uint4 ll_wait8(const uint32_t *src, uint4 a, uint4 b, uint32_t tag) const {
    if (!ll_ready8(a, b, tag)) slow_ll_wait8(abort_s, p.error, ll_limit(), src, tag, a, b);
    return ll_pack8(a, b);
  }
  // Up to N vectors of eight tagged words, `stride` words apart: all requested together, then those that were not there.
  template <int N> __device__ __forceinline__ void ll_gather(const uint32_t *src, uint32_t stride, uint32_t n, uint32_t tag, uint4 (&a)[N], uint4 (&b)[N]) const {
    uint32_t missing = n >= N ? (1u << N) - 1u : (1u << n) - 1u;
    const uint32_t limit = ll_limit();
#pragma unroll 1
    for (uint32_t i = 0;; ++i) {
#pragma unroll
      for (int j = 0; j < N; ++j)
        if (missing & (1u << j)) {
          a[j] = ld_vol_v4(src + j * stride);
          b[j] = ld_vol_v4(src + j * stride + 4);
        }
#pragma unroll
      for (int j = 0; j < N; ++j)
        if ((missing & (1u << j)) && ll_ready8(a[j], b[j], tag)) missing &= ~(1u << j);
      if (!missing) return;
      if (i >= limit) break;
      if ((i & 255u) == 255u && (*(volatile uint32_t *)p.error != 0u || *abort_s != 0)) {
        *abort_s = 1;  // give up quietly: another wait has already raised the error
        return;
      }
    }
    *abort_s = 1;
    atomicCAS(p.error, 0u, 6u);
  }
};

// ------------------------------------------------------------------ weight and cache streams
// A warp's ring: nst pieces of PIECE_BYTES, each with an mbarrier. Lane 0 walks the CTA's table of runs (MegaRun: what the CTA
// reads of one op) and requests this warp's share of each, piece by piece; the warp takes them in the same order. A piece is
// requested into the place of the one that the warp has just taken, so nothing but the copy's own barrier is needed: the
// reads of the old bytes come before the request in program order (__syncwarp between them). The requests sit between a
// warp's loads and its arithmetic, so what they need is worked out beforehand: no divisions, nothing from global memory.
// The cached rows that a warp takes of every attention op of the token.
struct alignas(16) KvShare {
  unsigned long long off;  // bytes from the start of a cache to the first of them
  uint32_t r0, rows;       // the first row's position in the cache, and their number
};
struct KvPlan {            // in shared memory, the same for every attention op of the token
  KvShare share[NCW];
  uint32_t L, S;           // cached rows, splits per head
  uint32_t head, split;    // this CTA's; head >= heads: none
  uint32_t per_piece;      // rows of a piece: at most 16, those of one m16n8k16
};
// 4, 8 or 16 lanes hold a cache row's 16-byte parts: log2 of that.
__device__ __forceinline__ uint32_t kv_lanes_log(uint32_t head_dim) { return head_dim > 64 ? 4u : head_dim > 32 ? 3u : 2u; }
__device__ __forceinline__ void kv_plan(const MegaParams &p, KvPlan &k, uint32_t pos0, uint32_t warp) {  // one thread per warp
  const uint32_t L = min(pos0 + 1, p.maxlen), S = mega_splits(L, p.splits, p.split_rows), head = blockIdx.x / S, split = blockIdx.x % S;
  const uint32_t rowb = p.head_dim * 2u;
  KvShare sh = {0, 0, 0};
  if (head < p.heads) {
    uint32_t c0, c1;
    mega_kv_range(L, S, split, c0, c1);
    mega_kv_share(c0, c1, warp, sh.r0, sh.rows);
    sh.off = ((unsigned long long)head * p.maxlen + sh.r0) * rowb;
  }
  k.share[warp] = sh;
  if (warp == 0) {
    k.L = L;
    k.S = S;
    k.head = head;
    k.split = split;
    k.per_piece = min(PIECE_BYTES / rowb, 16u);
  }
}
struct RunTable {  // in shared memory
  const MegaRun *runs;
  uint32_t n;
  const KvPlan *kv;
};
struct Ring {
  uint32_t piece, bar;  // shared addresses of the next piece and of its barrier
  uint32_t ph;          // the barrier's parity
  uint32_t last;        // the last barrier of the ring
  bool lead;            // lane 0, until a wait fails: requests
  // requesting side, lane 0 only
  const uint8_t *src;
  uint32_t whole;       // whole pieces of weights that follow at src
  uint32_t rest;        // bytes of the run behind them (cache run: of one of the caches, all of it)
  uint32_t next;        // runs of the table that have been begun
  uint32_t asked;       // pieces requested so far
  int32_t to_v;         // cache run: V cache minus K cache, / 256; a run of weights: 0
  bool second;          // cache run: the K piece has been requested, its V piece comes next
};
// Lane 0: requests the next piece into the place `piece`.
template <bool DBG, bool F16>
__device__ __forceinline__ void ring_request(const MegaParams &p, const RunTable &tab, Ring &r, uint32_t piece, uint32_t bar, uint32_t warp) {
  constexpr uint32_t UB = Unit<F16>::BYTES;
  uint32_t bytes = SU * UB;
  const uint8_t *src = r.src;
  if (r.whole) {  // most requests
    --r.whole;
    r.src += SU * UB;
  } else {
#pragma unroll 1
    while (r.rest == 0) {  // on to the next run that has something for this warp
      if (r.next == tab.n) return;
      const MegaRun e = tab.runs[r.next++];
      r.to_v = e.to_v;
      if (e.units == MEGA_KV_MARK) {
        const KvShare &sh = tab.kv->share[warp];
        r.src = e.src + sh.off;
        r.rest = sh.rows * p.head_dim * 2u;
      } else {
        const uint32_t u0 = mega_share_begin(e.units, warp), n = mega_share_begin(e.units, warp + 1) - u0;
        r.src = e.src + (size_t)u0 * UB;
        r.whole = n / SU;
        r.rest = n % SU * UB;
        if (r.whole) break;
      }
    }
    src = r.src;
    if (r.to_v != 0) {
      bytes = min(tab.kv->per_piece * p.head_dim * 2u, r.rest);
      if (r.second) {
        src += (long long)r.to_v * 256;
        r.src += bytes;
        r.rest -= bytes;
      }
      r.second = !r.second;
    } else if (r.whole) {
      --r.whole;
      r.src += SU * UB;
    } else {
      bytes = r.rest;
      r.rest = 0;
    }
  }
  ++r.asked;
  if (DBG && (p.timing_mode & 2u)) {  // diagnostic: no copies
    mbar_arrive(bar);
  } else {
    mbar_expect(bar, bytes);
    bulk_g2s(piece, src, bytes, bar);
  }
}
// Waits for the next piece, or until the wait has run out: the warp then goes on with whatever lies there and requests nothing more.
template <bool DBG>
__device__ __forceinline__ void ring_take(const Ctx &c, Ring &r) {
  if (DBG && (c.p.timing_mode & 128u)) return;
  if (mbar_try(r.bar, r.ph)) return;
  if (c.aborted() || !slow_mbar_wait(c.abort_s, c.p.error, c.p.wait_limit, r.bar, r.ph, 1)) r.lead = false;
}
// The warp has read what it needs of the piece: request the one that takes its place, and on to the next.
template <bool DBG, bool F16>
__device__ __forceinline__ void ring_give(const Ctx &c, const RunTable &tab, Ring &r, uint32_t warp) {
  __syncwarp();
  if (r.lead) ring_request<DBG, F16>(c.p, tab, r, r.piece, r.bar, warp);
  r.piece += PIECE_BYTES;
  r.bar += 8;
  if (r.bar > r.last) {
    const uint32_t nst = c.p.nst;
    r.bar -= nst * 8;
    r.piece -= nst * PIECE_BYTES;
    r.ph ^= 1u;
  }
}
// After a wait that ran out: nothing may still be landing in this CTA's shared memory when it exits.
__device__ __forceinline__ void ring_drain(const MegaParams &p, const Ring &r) {
  const uint32_t n = min(r.asked, p.nst), bar0 = r.last - (p.nst - 1) * 8;
#pragma unroll 1
  for (uint32_t j = r.asked - n; j < r.asked; ++j) {
    const uint32_t bar = bar0 + j % p.nst * 8, ph = j / p.nst & 1u;
    // (not the caller's bound, which a test may have made very short: a copy in flight lands within microseconds)
#pragma unroll 1
    for (uint32_t i = 0; i < max(p.wait_limit, 1u << 20) && !mbar_try(bar, ph); ++i) {
    }
  }
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float ldsf(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts128(uint32_t a, const uint4 &v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void stsf(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }

// ------------------------------------------------------------ grid barrier
__device__ VKL_SLOW bool grid_barrier(const Ctx &c, uint64_t target, uint32_t round, volatile uint32_t *seen_s) {
  cons_sync();  // every consumer store of this op is issued
  // Lane 0 of the first POLLERS warps poll the counter, each a fraction of a memory round trip
  // after the previous one, so that the last arrival is seen a fraction of a round trip after it
  // lands instead of half a round trip on average. `seen_s` holds the last round (1, 2, ... within
  // this launch) that one of them has seen complete.
  const uint32_t POLLERS = c.p.barrier_pollers;
  const uint32_t w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0 && w < POLLERS && !c.aborted()) {
    if (w == 0) {
      // release-add without a return value: orders this CTA's stores (made visible to
      // thread 0 by the bar.sync above) before the arrival, one L2 trip instead of two
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(c.p.bar), "l"(1ull) : "memory");
    } else {
      __nanosleep(160 * w);
    }
    const uint32_t tgt = round;
    bool ok = false;
    // (under tensor parallelism a CTA without a tile of the projections runs ahead to this barrier while others
    // wait for another rank's partial sums: the barrier's wait outlasts theirs, so that the error names theirs)
    const uint32_t limit = c.p.tp_size > 1 ? (c.p.wait_limit < 0x10000000u ? 16u * c.p.wait_limit : 0xffffffffu) : c.p.wait_limit;
#pragma unroll 1
    for (uint32_t i = 0; i < limit; ++i) {
      if (*seen_s == tgt || ld_acq_u64(c.p.bar) >= target) {
        ok = true;
        break;
      }
      if (i > 100000u) __nanosleep(64);
      if ((i & 1023u) == 1023u && *(volatile uint32_t *)c.p.error != 0u) break;
    }
    if (ok)
      *seen_s = tgt;
    else
      c.raise(3);
    __threadfence();
  }
  cons_sync();
  return !c.aborted();
}

// ------------------------------------------------------------------ mat-vec
struct Best {
  float v;
  uint32_t i;
};
__device__ __forceinline__ bool better(float v, uint32_t i, const Best &b) {
  return b.i == 0xffffffffu || v > b.v || (v == b.v && i < b.i);
}

// Two stored codes (bytes 0 and 2, or 1 and 3, of a plane word) as a pair of fp16 subnormals u * 2^-24.
__device__ __forceinline__ uint32_t codes_sub_h2(uint32_t w, bool hi) { return __byte_perm(w, 0u, hi ? 0x4341u : 0x4240u); }

// m16n8k16 from a zero accumulator and onto one. (Not volatile: the order is the scheduler's to choose.)
__device__ __forceinline__ void mma_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mma_next(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void lds_if(uint4 &v, uint32_t addr, bool take) {  // other lanes keep what they have
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n @p ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n}"
               : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
               : "r"(addr), "r"((uint32_t)take)
               : "memory");
}

__device__ __forceinline__ void lds64_if(uint32_t &x, uint32_t &y, uint32_t addr, bool take) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p ld.shared.v2.u32 {%0,%1}, [%2];\n}" : "+r"(x), "+r"(y) : "r"(addr), "r"((uint32_t)take) : "memory");
}

// One mat-vec op of the token: y = W . x for the op's packed weight stream (MegaOp).
//
// Arithmetic. The stored codes u = q + 128 go into the tensor core as fp16 subnormals u * 2^-24
// (one byte permute per pair, no arithmetic): products and their fp32 sums are exact up to the
// accumulator's rounding, and sum_k u_k x_k = sum_k q_k x_k + 128 * sum_k x_k, so a block's
// result is 2^24 * acc - 128 * sum(x of the block), scaled by the block's fp16 scale in fp32 as
// the reference does (matmul_b0_fp16_x_q8_0.comp:99-133). The input is column 0 of the B operand,
// the other columns read zeros. (An integer path, dp4a on three byte planes of the input, was
// measured 30 % slower: dp4a issues at about 16 lanes per clock and SM on this GPU.)
template <bool TIMED, bool DBG, bool TP, bool F16>
__device__ __forceinline__ void matvec_op(const Ctx &c, const MegaOp &op_global, const RunTable &tab, Ring &ring, __half *xs, float *xbias,
                                          float *red, float *ssum, Best &best, unsigned long long *tw, uint32_t ar_seq,
                                          uint32_t tag_in, uint32_t tag_out, uint32_t tag_res, unsigned long long *trace) {
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const uint32_t G = gridDim.x, cta = blockIdx.x;
  // The op's entry sits in shared memory: fields are read where they are used (the prologue, then again
  // in the epilogue) instead of being carried in registers through the streaming loop, which needs them all.
  const MegaOp &op = op_global;
  const uint32_t K = op.K, tiles = op.tiles, blocks = op.blocks;
  const uint32_t tile0 = (cta + G - (op.rot % G)) % G;
  const uint32_t tl = tile0 < tiles ? (tiles - tile0 + G - 1) / G : 0u;  // this CTA's tiles
  // No tile here: nothing to read either. (It must not wait for the input: nobody waits for this
  // CTA's results, so by the time it looked the producers of a later op may have re-tagged the words.)
  if (tl == 0) return;
  // This warp's share of the CTA's units, and, for the reduction, the warps whose shares touch this thread's tile.
  const uint32_t units = tl * blocks, rspan = c.p.red_slots;
  uint32_t u = mega_share_begin(units, warp), b = u % blocks;
  const uint32_t u1 = mega_share_begin(units, warp + 1);
  auto touching = [&](uint32_t lt, uint32_t &at, uint32_t &n) {
    const MegaTileShares ts = mega_tile_shares(units, blocks, lt);
    at = (ts.first * rspan + ts.place) * 32;
    n = ts.more | ts.first << 16;
  };
  // row r of tile lt: which matrix and which of its rows
  auto row_of = [&](uint32_t lt, uint32_t r, uint32_t &m, uint32_t &n) {
    const uint32_t gt = tile0 + lt * G;
    m = 0;
    if (op.epi == EPI_SWIGLU) {
      n = gt * 16 + r;
    } else if (op.nmat == 3) {
      const uint32_t tpm = (op.N + 31) / 32;
      m = (gt >= tpm) + (gt >= 2 * tpm);
      n = (gt - m * tpm) * 32 + r;
    } else {
      n = gt * 32 + r;
    }
  };
  // worked out here, not between the end of the stream and the publication of the results
  uint32_t t_at = 0, t_n = 0, t_m = 0, t_row = 0xffffffffu;
  if (tid < tl * 32) {
    touching(tid >> 5, t_at, t_n);
    row_of(tid >> 5, lane, t_m, t_row);
  }
  asm volatile("" : "+r"(t_at), "+r"(t_n), "+r"(t_m), "+r"(t_row));  // (and stays worked out)
  // ---- input vector -> shared memory (RMSNorm fused, rounded to fp16 where the reference's RMSNorm op rounds:
  // rms_norm_fp16.comp:70-77). A thread's words are requested together, then only those that were not there yet.
  uint32_t rw = 0;
  {
    constexpr int NV = (11008 / 8 + CT - 1) / CT;  // vectors of eight words in one go: K <= 11008
    const uint32_t nv = K / 8;
    const bool norm = op.norm_w != nullptr;
    float4 nw[2][2];  // the norm weights depend on nothing: the first two vectors' are requested before the polls, which can spin for a while
    if (norm) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t i = tid + j * CT;
        if (i < nv) {
          nw[j][0] = ldg_f4_ordered(reinterpret_cast<const float4 *>(op.norm_w) + 2 * i);
          nw[j][1] = ldg_f4_ordered(reinterpret_cast<const float4 *>(op.norm_w) + 2 * i + 1);
        }
      }
    }
    // EPI_ADD: this thread's residual word, so that its memory round trip is not on the path to the stream or the results
    if (t_row < op.N && (op.epi == EPI_ADD || (TP && op.epi == EPI_REDUCE))) rw = ld_vol_u32(op.out_ll[0] + t_row);
    float sq = 0.f;
#pragma unroll 1
    for (uint32_t i0 = tid; i0 < nv; i0 += NV * CT) {
      uint4 a[NV], b8[NV];
      c.template ll_gather<NV>(op.in + 8 * i0, 8 * CT, (nv - i0 + CT - 1) / CT, tag_in, a, b8);
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const uint32_t i = i0 + j * CT;
        if (i >= nv) continue;
        const uint4 v = ll_pack8(a[j], b8[j]);
        *reinterpret_cast<uint4 *>(xs + 8 * i) = v;
        if (norm) {
          float f[8];
          unpack8(v, f);
#pragma unroll
          for (int e = 0; e < 8; e += 2) sq += f[e] * f[e] + f[e + 1] * f[e + 1];
        }
      }
    }
    float alpha = 1.f;
    if (norm) {
      sq = warp_sum(sq);
      if (lane == 0) ssum[warp] = sq;
      cons_sync();
      float tot = 0.f;
#pragma unroll
      for (int w = 0; w < NCW; ++w) tot += ssum[w];
      alpha = 1.0f / sqrtf(tot / (float)K + op.eps);
    }
    // this thread's vectors again: the norm, and for Q8_0 codes (biased) 128 * the sum of every block of 32 inputs = 4 consecutive lanes' vectors
#pragma unroll 1
    for (uint32_t i = tid; i - tid < nv && (norm || !F16); i += CT) {
      float bs = 0.f;
      if (i < nv) {
        uint4 v = *reinterpret_cast<const uint4 *>(xs + 8 * i);
        float f[8];
        unpack8(v, f);
        if (norm) {
          const float w[8] = {nw[0][0].x, nw[0][0].y, nw[0][0].z, nw[0][0].w, nw[0][1].x, nw[0][1].y, nw[0][1].z, nw[0][1].w};
          __half2 o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) o[e] = __halves2half2(__float2half_rn(f[2 * e] * w[2 * e] * alpha), __float2half_rn(f[2 * e + 1] * w[2 * e + 1] * alpha));
          v = *reinterpret_cast<uint4 *>(o);
          *reinterpret_cast<uint4 *>(xs + 8 * i) = v;
          unpack8(v, f);
          nw[0][0] = nw[1][0];
          nw[0][1] = nw[1][1];
          if (i + 2 * CT < nv) {
            nw[1][0] = __ldg(reinterpret_cast<const float4 *>(op.norm_w) + 2 * (i + 2 * CT));
            nw[1][1] = __ldg(reinterpret_cast<const float4 *>(op.norm_w) + 2 * (i + 2 * CT) + 1);
          }
        }
#pragma unroll
        for (int e = 0; e < 8; e += 2) bs += f[e] + f[e + 1];
      }
      if (F16) continue;
      bs += __shfl_xor_sync(0xffffffffu, bs, 1);
      bs += __shfl_xor_sync(0xffffffffu, bs, 2);
      if ((lane & 3) == 0 && i < nv) xbias[i >> 2] = 128.0f * bs;
    }
    cons_sync();
  }
  if (t_row < op.N && (op.epi == EPI_ADD || (TP && op.epi == EPI_REDUCE)) && (rw >> 16) != tag_res) rw = c.ll_wait1(op.out_ll[0] + t_row, tag_res);  // (the word may come from another CTA)
  const float resid = __half2float(ll_half(rw));
  if (TIMED && tw) tw[1] = clock64();
  VKL_TRACE(1);

  // ---- stream this warp's share of the CTA's tiles: consecutive units, piece by piece. A unit is one block (32 columns) of
  // a 32-row tile: two 16-row halves, each the A operand of two m16n8k16 MMAs. The sums of a tile go to a place of this warp's
  // own in shared memory when its units move on to the next tile, and nothing synchronises until the op's single reduction.
  {
    uint32_t slotp = s32(red) + (warp * rspan * 32 + g) * 4;  // the warp's first tile, then its second, ...
    float acc[4] = {0.f, 0.f, 0.f, 0.f};                      // lanes t == 0: rows g, g + 8, 16 + g, 24 + g of the tile
    float even_a[4] = {0.f, 0.f, 0.f, 0.f}, even_b[4] = {0.f, 0.f, 0.f, 0.f}, odd_a[4] = {0.f, 0.f, 0.f, 0.f}, odd_b[4] = {0.f, 0.f, 0.f, 0.f};  // FP16
    auto flush = [&]() {
      if (F16) {
        acc[0] = even_a[0] + odd_a[0];
        acc[1] = even_a[2] + odd_a[2];
        acc[2] = even_b[0] + odd_b[0];
        acc[3] = even_b[2] + odd_b[2];
#pragma unroll
        for (int i = 0; i < 4; ++i) even_a[i] = even_b[i] = odd_a[i] = odd_b[i] = 0.f;
      }
      if (t == 0) {
        stsf(slotp, acc[0]);
        stsf(slotp + 32, acc[1]);
        stsf(slotp + 64, acc[2]);
        stsf(slotp + 96, acc[3]);
      }
    };
    constexpr uint32_t UB = Unit<F16>::BYTES, XB = Unit<F16>::COLUMNS * 2;  // of the weights, of the input
    const uint32_t wofs = lane * 16, dofs = UNIT_CODES + g * 8, xaddr = s32(xs) + t * (F16 ? 8 : 16), baddr = s32(xbias);
    uint4 X[SU];  // column 0 of B = the input (lanes g == 0); the other columns' lanes are never loaded and stay zero
#pragma unroll
    for (int q = 0; q < SU; ++q) X[q] = make_uint4(0, 0, 0, 0);
    auto scale = [&](const float (&ca)[4], const float (&cb)[4], const uint2 &dsc, float xb) {
      const float2 d0 = __half22float2(*reinterpret_cast<const __half2 *>(&dsc.x));  // rows g, g + 8
      const float2 d1 = __half22float2(*reinterpret_cast<const __half2 *>(&dsc.y));  // rows 16 + g, 24 + g
      acc[0] = fmaf(fmaf(ca[0], 16777216.f, -xb), d0.x, acc[0]);
      acc[1] = fmaf(fmaf(ca[2], 16777216.f, -xb), d0.y, acc[1]);
      acc[2] = fmaf(fmaf(cb[0], 16777216.f, -xb), d1.x, acc[2]);
      acc[3] = fmaf(fmaf(cb[2], 16777216.f, -xb), d1.y, acc[3]);
    };
    auto next_tile = [&]() {
      flush();
      slotp += 128;
      b = 0;
      acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
    };
    // (after a wait that ran out the warp multiplies whatever lies in the ring: the results are discarded)
#pragma unroll 1
    while (u < u1) {
      if (b == blocks) next_tile();
      // whole pieces within the tile: straight-line code, the units' chains run side by side
      uint32_t whole = min(u1 - u, blocks - b) / SU;
      u += whole * SU;
#pragma unroll 1
      for (; whole; --whole) {
        unsigned long long w0 = 0;
        if (TIMED && tw) w0 = clock64();
        ring_take<DBG>(c, ring);
        if (TIMED && tw) tw[0] += (clock64() - w0) * 1000ull / c.p.sm_mhz;  // SM cycles -> ns at the SM clock the host measured
        const uint32_t st = ring.piece;
        if (DBG && (c.p.timing_mode & (4u | 64u))) {  // diagnostic: handshake only, or ring traffic without arithmetic
          if (c.p.timing_mode & 4u) acc[0] += ldsf(st + wofs);
          b += SU;
          ring_give<DBG, F16>(c, tab, ring, warp);
          continue;
        }
        if constexpr (F16) {
          uint4 wa[SU], wb[SU];
#pragma unroll
          for (int q = 0; q < SU; ++q) {
            wa[q] = lds128(st + wofs + q * UB);        // rows g, g + 8 of the tile: columns 4 t, 4 t + 1, then the next two
            wb[q] = lds128(st + wofs + q * UB + 512);  // rows 16 + g, 24 + g
            lds64_if(X[q].x, X[q].y, xaddr + b * XB + q * XB, g == 0);
          }
#pragma unroll
          for (int q = 0; q < SU; ++q) {  // two chains per half tile
            mma_next(q & 1 ? odd_a : even_a, wa[q].x, wa[q].y, wa[q].z, wa[q].w, X[q].x, X[q].y);
            mma_next(q & 1 ? odd_b : even_b, wb[q].x, wb[q].y, wb[q].z, wb[q].w, X[q].x, X[q].y);
          }
        } else {
        uint4 wa[SU], wb[SU];
        uint2 dsc[SU];
        float xb[SU], ca[SU][4], cb[SU][4];
#pragma unroll
        for (int q = 0; q < SU; ++q) {
          wa[q] = lds128(st + wofs + q * UB);        // rows g, g + 8 of the tile
          wb[q] = lds128(st + wofs + q * UB + 512);  // rows 16 + g, 24 + g
          dsc[q] = lds64(st + dofs + q * UB);        // their four block scales
          lds_if(X[q], xaddr + b * XB + q * XB, g == 0);
          xb[q] = ldsf(baddr + b * 4 + q * 4);
        }
#pragma unroll
        for (int q = 0; q < SU; ++q) {
          mma_first(ca[q], codes_sub_h2(wa[q].x, false), codes_sub_h2(wa[q].z, false), codes_sub_h2(wa[q].x, true), codes_sub_h2(wa[q].z, true), X[q].x, X[q].y);
          mma_first(cb[q], codes_sub_h2(wb[q].x, false), codes_sub_h2(wb[q].z, false), codes_sub_h2(wb[q].x, true), codes_sub_h2(wb[q].z, true), X[q].x, X[q].y);
        }
#pragma unroll
        for (int q = 0; q < SU; ++q) {
          mma_next(ca[q], codes_sub_h2(wa[q].y, false), codes_sub_h2(wa[q].w, false), codes_sub_h2(wa[q].y, true), codes_sub_h2(wa[q].w, true), X[q].z, X[q].w);
          mma_next(cb[q], codes_sub_h2(wb[q].y, false), codes_sub_h2(wb[q].w, false), codes_sub_h2(wb[q].y, true), codes_sub_h2(wb[q].w, true), X[q].z, X[q].w);
        }
#pragma unroll
        for (int q = 0; q < SU; ++q) scale(ca[q], cb[q], dsc[q], xb[q]);
        }
        b += SU;
        ring_give<DBG, F16>(c, tab, ring, warp);
      }
      if (u == u1 || b == blocks) continue;
      // a piece that a tile or the share ends in
      const uint32_t n = min((uint32_t)SU, u1 - u);
      u += n;
      ring_take<DBG>(c, ring);
#pragma unroll 1
      for (uint32_t q = 0; q < n; ++q) {
        if (b == blocks) next_tile();
        const uint32_t su = ring.piece + q * UB;
        const uint4 wa = lds128(su + wofs), wb = lds128(su + 512 + wofs);
        if constexpr (F16) {
          lds64_if(X[0].x, X[0].y, xaddr + b * XB, g == 0);
          mma_next(even_a, wa.x, wa.y, wa.z, wa.w, X[0].x, X[0].y);
          mma_next(even_b, wb.x, wb.y, wb.z, wb.w, X[0].x, X[0].y);
        } else {
          lds_if(X[0], xaddr + b * XB, g == 0);
          float ca[4], cb[4];
          mma_first(ca, codes_sub_h2(wa.x, false), codes_sub_h2(wa.z, false), codes_sub_h2(wa.x, true), codes_sub_h2(wa.z, true), X[0].x, X[0].y);
          mma_first(cb, codes_sub_h2(wb.x, false), codes_sub_h2(wb.z, false), codes_sub_h2(wb.x, true), codes_sub_h2(wb.z, true), X[0].x, X[0].y);
          mma_next(ca, codes_sub_h2(wa.y, false), codes_sub_h2(wa.w, false), codes_sub_h2(wa.y, true), codes_sub_h2(wa.w, true), X[0].z, X[0].w);
          mma_next(cb, codes_sub_h2(wb.y, false), codes_sub_h2(wb.w, false), codes_sub_h2(wb.y, true), codes_sub_h2(wb.w, true), X[0].z, X[0].w);
          scale(ca, cb, lds64(su + dofs), ldsf(baddr + b * 4));
        }
        ++b;
      }
      ring_give<DBG, F16>(c, tab, ring, warp);
    }
    flush();  // (an empty share: zeros)
  }
  // ---- one fixed-order reduction over the warps and the epilogue for all tiles
  VKL_TRACE(2);
  if (TIMED && tw) {
    tw[2] = clock64();
    if (c.p.timing_mode & 32u) tw[0] = (((tw[2] - tw[1]) * 1000ull / c.p.sm_mhz) << 16) | (uint64_t)min((units / NCW + SU - 1) / SU, 65535u);
  }
  uint32_t *const out0 = t_m == 0 ? op.out_ll[0] : t_m == 1 ? op.out_ll[1] : op.out_ll[2];
  cons_sync();
  VKL_TRACE(3);
#pragma unroll 1
  for (uint32_t idx = tid; idx < tl * 32; idx += CT) {  // tl * 32 is a multiple of the warp size: whole warps
    const uint32_t r = idx & 31;
    if (idx != tid) {  // a CTA with more tiles than warps
      touching(idx >> 5, t_at, t_n);
      row_of(idx >> 5, r, t_m, t_row);
    }
    const uint32_t n = t_row, m = t_m;
    float part[NCW];
    const float *sp = red + (size_t)((t_n >> 16) + 1) * rspan * 32 + r;
    float sum = red[t_at + r];
#pragma unroll
    for (int w = 0; w < NCW - 1; ++w) part[w] = w < (t_n & 0xffffu) ? sp[w * rspan * 32] : 0.f;
#pragma unroll
    for (int w = 0; w < NCW - 1; ++w) sum += part[w];
    if (op.epi == EPI_SWIGLU) {
      // rows 0..15 of the tile are gate rows, rows 16..31 the up rows of the same outputs
      const float up = __shfl_down_sync(0xffffffffu, sum, 16);
      if (r < 16 && n < op.N) out0[n] = ll_pack(__float2half_rn(sum / (1.0f + expf(-sum)) * up), tag_out);
      continue;
    }
    // (After an abort what is published is not looked at any more; another rank must not get it, though.)
    if (n < op.N && !(TP && c.aborted())) {
      if (op.epi == EPI_ADD) {
        const float res = idx == tid ? resid : __half2float(ll_half(c.ll_wait1(op.out_ll[0] + n, tag_res)));
        out0[n] = ll_pack(__float2half_rn(round_h(sum) + res), tag_out);
      } else if (TP && op.epi == EPI_REDUCE) {
        // this rank's share of a row-split projection, reduced in place: the row's raw fp32 sum and the all-reduce's
        // sequence number go as one 8-byte word into slot [parity][my rank] of every OTHER rank's exchange buffer
        // (plain peer stores over NVLink; the word is its own arrival flag); then this thread polls (bounded, all
        // missing words per round) the same row's words of the other ranks in its own buffer, adds in rank order (the
        // same order on every rank: bit-identical residual streams) and publishes x = fp16(fp16(sum) + x).
        const MegaParams &pp = c.p;
        const uint32_t tp = pp.tp_size, me = pp.tp_rank;
        const size_t par = (size_t)(ar_seq & 1u) * tp;
        for (uint32_t rk = 0; rk < tp; ++rk) {
          if (rk == me) continue;
          uint32_t *dst = static_cast<uint32_t *>(pp.tp_peer[rk]) + 2 * ((par + me) * pp.dim + n);
          asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(dst), "r"(__float_as_uint(sum)), "r"(ar_seq) : "memory");
        }
        const float res = idx == tid ? resid : __half2float(ll_half(c.ll_wait1(op.out_ll[0] + n, tag_res)));
        const uint32_t *mine = static_cast<const uint32_t *>(pp.tp_peer[me]) + 2 * (par * pp.dim + n);
        float part[8];
        uint32_t missing = ((1u << tp) - 1u) & ~(1u << me);
        part[me & 7u] = sum;
        const uint32_t limit = pp.wait_limit;
      #pragma unroll 1
        for (uint32_t itw = 0; missing && itw < limit; ++itw) {
#pragma unroll
          for (uint32_t r = 0; r < 8; ++r) {
            if (missing & (1u << r)) {
              const uint2 w = ld_vol_v2(mine + 2 * (size_t)r * pp.dim);
              if (w.y == ar_seq) {
                part[r] = __uint_as_float(w.x);
                missing &= ~(1u << r);
              }
            }
          }
          if (itw > 100000u) __nanosleep(64);
          if ((itw & 1023u) == 1023u && (*(volatile uint32_t *)pp.error != 0u || c.aborted())) break;
        }
        if (missing) {
          c.raise(4);
        } else {
          float s = 0.f;
#pragma unroll
          for (uint32_t r = 0; r < 8; ++r)
            if (r < tp) s += part[r];
          op.out_ll[0][n] = ll_pack(__float2half_rn(round_h(s) + res), tag_out);
        }
      } else if (TP && op.epi == EPI_PARTIAL) {
        // this rank's share of a row-split projection: the raw fp32 sum and the all-reduce's
        // sequence number go, as one 8-byte word, into slot [parity][my rank] of every rank's
        // exchange buffer (plain peer stores over NVLink; the word is its own arrival flag)
        const MegaParams &pp = c.p;
        for (uint32_t rk = 0; rk < pp.tp_size; ++rk) {
          uint32_t *dst = static_cast<uint32_t *>(pp.tp_peer[rk]) + 2 * (((size_t)(ar_seq & 1u) * pp.tp_size + pp.tp_rank) * pp.dim + n);
          asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(dst), "r"(__float_as_uint(sum)), "r"(ar_seq) : "memory");
        }
      } else {
        const __half h0 = __float2half_rn(sum);
        uint32_t *o = idx == tid ? out0 : m == 0 ? op.out_ll[0] : m == 1 ? op.out_ll[1] : op.out_ll[2];
        if (o) {
          o[n] = ll_pack(h0, tag_out);
        } else {
          op.out[0][n] = h0;
        }
        if (op.out_f32) {
          op.out_f32[n] = __half2float(h0);
          if (c.p.host_logits) c.p.host_logits[n] = __half2float(h0);
        }
        if (op.track_argmax && better(__half2float(h0), n, best)) {
          best.v = __half2float(h0);
          best.i = n;
        }
      }
    }
  }
}

// ---------------------------------------------------------------- attention
__device__ __forceinline__ void rope_pair(float x0, float x1, float cs, float sn, __half &o0, __half &o1) {
  o0 = __float2half_rn(x0 * cs - x1 * sn);
  o1 = __float2half_rn(x0 * sn + x1 * cs);
}

// RoPE of four pairs of neighbours (eight packed halves), rounded to fp16.
__device__ __forceinline__ uint4 rope8(const uint4 &v, const float4 &cs, const float4 &sn) {
  float f[8];
  unpack8(v, f);
  const float cc[4] = {cs.x, cs.y, cs.z, cs.w}, ss[4] = {sn.x, sn.y, sn.z, sn.w};
  uint32_t o[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    __half a, b;
    rope_pair(f[2 * e], f[2 * e + 1], cc[e], ss[e], a, b);
    o[e] = (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// One (head, split) per CTA: RoPE(q), RoPE(k) + cache append, scores over the split's rows, partial softmax and P.V (the
// arithmetic of attention_kernel, attention.cu, with a running maximum). Every warp takes its share of the rows through its
// ring, a piece of K rows and the piece of the same V rows behind it: cached rows do not depend on this token, only the row of
// the new position does; the warp whose share it is in takes it from the fresh projections, puts it into the pieces and into
// the caches. Up to 16 rows' scores come from the tensor cores (rows x dims, the query as column 0; fp16 products, fp32 sums),
// P.V stays in fp32: 4, 8 or 16 lanes hold a V row's 16-byte parts. Warps meet once, to add their results in order.
// The kernel's time depends on its code size (beyond the instruction caches a phase's code comes from memory behind the
// weight stream), hence loops where a few registers more would have allowed straight-line code.
template <bool DBG, bool F16>
__device__ __forceinline__ void attn_part_op(const Ctx &c, const MegaOp &op, float *sm, uint32_t pos0, const KvPlan &kv, uint32_t tag_in,
                                             uint32_t tag_out, const RunTable &tab, Ring &ring) {
  const MegaParams &p = c.p;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const uint32_t h = kv.head, split = kv.split, S = kv.S, D = p.head_dim;
  if (h >= p.heads) return;
  const uint32_t lanes_log = kv_lanes_log(D), per_step = 32u >> lanes_log, per_piece = kv.per_piece;
  const uint32_t r0 = kv.share[warp].r0, r1 = r0 + kv.share[warp].rows;
  const uint32_t jn = pos0 < p.maxlen ? pos0 : pos0 % p.maxlen;
  const size_t row = (size_t)h * D;
  const uint32_t sub = lane & ((1u << lanes_log) - 1u), hi = lane >> lanes_log;
  const bool act = sub * 8 < D, owns = jn >= r0 && jn < r1;
  float m = -INFINITY, l = 0.f, acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  // (A split without rows waits for its queries too, with warp 0: it must not arrive at the merge of a later layer first.)
  if (r0 < r1 || warp == 0) {
    // The query lands where this warp's sums will lie; the new K and V rows behind all of them. The upper lanes fetch the
    // key while the lower ones fetch the query (from buffers that follow each other), then the lower ones the value.
    const uint32_t q_s = s32(sm + warp * D), n_s = s32(sm + NCW * D), part = lane & 15u, upper = lane >> 4;
    const size_t fi = (size_t)pos0 * (D / 2) + part * 4, cell = ((size_t)h * p.maxlen + jn) * D + part * 8;
#pragma unroll 1
    for (uint32_t pass = 0; pass < (owns ? 2u : 1u); ++pass) {
      if (part * 8 >= D || (upper && (pass || !owns))) continue;
      const uint32_t *src = (pass ? p.v : upper ? p.k : p.q) + row + part * 8;
      float4 cs, sn;
      if (!pass) {
        cs = ldg_f4_ordered(reinterpret_cast<const float4 *>(p.freqc + fi));
        sn = ldg_f4_ordered(reinterpret_cast<const float4 *>(p.freqs + fi));
      }
      uint4 v = c.ll_wait8(src, ld_vol_v4(src), ld_vol_v4(src + 4), tag_in);
      if (!pass) v = rope8(v, cs, sn);
      if (pass || upper) *reinterpret_cast<uint4 *>((pass ? op.vcache : op.kcache) + cell) = v;
      sts128((pass ? n_s + D * 2 : upper ? n_s : q_s) + part * 16, v);
    }
    __syncwarp();
    uint4 Q[4];  // B fragments: of every 32 dims lane t has 8 t .. 8 t + 7, for the A fragments the same; column 0 only
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      Q[i] = make_uint4(0, 0, 0, 0);
      lds_if(Q[i], q_s + (i * 4 + t) * 16, g == 0 && (i * 4 + t) * 8 < D);
    }
    float s0 = 0.f, s1 = 0.f;  // scores, then probabilities, of rows g and g + 8 of the piece
    bool values = false;
#pragma unroll 1
    for (uint32_t r = r0; r < r1;) {
      const uint32_t nr = min(per_piece, r1 - r);
      const uint32_t piece = ring.piece;
      ring_take<DBG>(c, ring);
      if (owns && jn - r < nr) {  // the new row
        if (part * 8 < D && !upper) sts128(piece + (jn - r) * D * 2 + part * 16, lds128(n_s + (values ? D * 2 : 0) + part * 16));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // before the copy that will take the piece's place
        __syncwarp();
      }
      if (!values) {
        float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};  // lanes t == 0: rows g, g + 8 in [0], [2]
        const uint32_t ra = piece + (min(g, nr - 1) * D + t * 8) * 2, rb = piece + (min(g + 8, nr - 1) * D + t * 8) * 2;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (i * 32 >= D) break;
          uint4 A = make_uint4(0, 0, 0, 0), B = A;
          if ((i * 4 + t) * 8 < D) {
            A = lds128(ra + i * 64);
            B = lds128(rb + i * 64);
          }
          mma_next(c0, A.x, B.x, A.y, B.y, Q[i].x, Q[i].y);
          mma_next(c1, A.z, B.z, A.w, B.w, Q[i].z, Q[i].w);
        }
        s0 = __shfl_sync(0xffffffffu, c0[0] + c1[0], lane & 28);
        s1 = __shfl_sync(0xffffffffu, c0[2] + c1[2], lane & 28);
        s0 = g < nr ? round_h(s0 * p.attn_scale) : -INFINITY;
        s1 = g + 8 < nr ? round_h(s1 * p.attn_scale) : -INFINITY;
        float mx = fmaxf(m, fmaxf(s0, s1));
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float base = mx == -INFINITY ? 0.f : mx;  // (rows of minus infinity so far: weights of 0, not NaN)
        const float keep = expf(m - base);
        s0 = expf(s0 - base);
        s1 = expf(s1 - base);
        m = mx;
        l = l * keep + (s0 + s1);  // this quad's rows
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] *= keep;
      } else {
#pragma unroll 1
        for (uint32_t a0 = 0; a0 < nr; a0 += 4 * per_step) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t first = a0 + i * per_step, at = first + hi;  // (a step's rows are all among the first eight or among the others)
            const float pj = __shfl_sync(0xffffffffu, first < 8 ? s0 : s1, (at & 7u) * 4);
            uint4 vv = make_uint4(0, 0, 0, 0);
            if (act && at < nr) vv = lds128(piece + (at * D + sub * 8) * 2);
            float f[8];
            unpack8(vv, f);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] = fmaf(pj, f[e], acc[e]);
          }
        }
        r += nr;
      }
      values = !values;
      ring_give<DBG, F16>(c, tab, ring, warp);
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll 1
    for (uint32_t o = 1u << lanes_log; o < 32; o <<= 1) {
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    }
    __syncwarp();  // the query has been read
  }
  // [warp][D] sums, the new rows, then [warp] maxima, then [warp] denominators
  float *wm = sm + (NCW + 1) * D, *wl = wm + NCW;
  if (act && hi == 0) {
#pragma unroll
    for (int e = 0; e < 8; e += 4) *reinterpret_cast<float4 *>(sm + warp * D + sub * 8 + e) = make_float4(acc[e], acc[e + 1], acc[e + 2], acc[e + 3]);
  }
  if (lane == 0) {
    wm[warp] = m;
    wl[warp] = l;
  }
  cons_sync();
  float *part = p.attn_scratch + ((size_t)h * p.splits + split) * (D + 4);
  if ((tid & ~31u) < D) {
    // lane w < NCW: warp w's weight
    const float mw = lane < NCW ? wm[lane] : -INFINITY, lw = lane < NCW ? wl[lane] : 0.f;
    const float mloc = warp_max(mw);
    const float e = lw != 0.f ? expf(mw - mloc) : 0.f;  // (NaN counts)
    const float lloc = warp_sum(lw * e);
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < NCW; ++w) {
      const float ew = __shfl_sync(0xffffffffu, e, w);
      if (ew != 0.f) s = fmaf(sm[w * D + min(tid, D - 1)], ew, s);
    }
    if (tid < D) {
      if (S == 1)
        p.ao[row + tid] = ll_pack(__float2half_rn(s / lloc), tag_out);  // whole row in this CTA: no combine phase
      else
        part[tid] = s;
    }
    if (tid == 0) {
      part[D] = mloc;
      part[D + 1] = lloc;
    }
  }
  if (S > 1 && p.attn_counters) {
    // The split that finishes last merges the head's partials (in split order, so the result
    // does not depend on who is last): no separate combine op and no grid barrier before it.
    __threadfence();  // this thread's partial results before the CTA's arrival below
    cons_sync();
    volatile uint32_t *last_s = reinterpret_cast<volatile uint32_t *>(wl + NCW);
    if (tid == 0) {
      uint32_t old;
      asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(p.attn_counters + h) : "memory");
      const bool last = old == S - 1;
      if (last) p.attn_counters[h] = 0;  // all splits of the head have arrived; its next use is a grid barrier away
      *last_s = last ? 1u : 0u;
    }
    cons_sync();
    if (*last_s && tid < D) {
      const float *base = p.attn_scratch + (size_t)h * p.splits * (D + 4);
      float M = -INFINITY;
#pragma unroll 1
      for (uint32_t sp = 0; sp < S; ++sp) M = fmaxf(M, __ldcg(base + sp * (D + 4) + D));
      float den = 0.f, num = 0.f;
#pragma unroll 1
      for (uint32_t sp = 0; sp < S; ++sp) {
        const float ms = __ldcg(base + sp * (D + 4) + D), ls = __ldcg(base + sp * (D + 4) + D + 1);
        if (ls > 0.f) {
          const float w = expf(ms - M);
          den += ls * w;
          num += __ldcg(base + sp * (D + 4) + tid) * w;
        }
      }
      p.ao[row + tid] = ll_pack(__float2half_rn(num / den), tag_out);
    }
  }
}

// One head per CTA: merge the partials of the token's S splits in split order (the places of further splits hold an earlier token's).
__device__ VKL_SLOW void attn_combine_op(const Ctx &c, uint32_t S, uint32_t tag_out) {
  const MegaParams &p = c.p;
  const uint32_t h = blockIdx.x, tid = threadIdx.x, D = p.head_dim;
  if (h >= p.heads || tid >= D) return;
  const float *base = p.attn_scratch + (size_t)h * p.splits * (D + 4);
  float M = -INFINITY;
#pragma unroll 1
  for (uint32_t s = 0; s < S; ++s) M = fmaxf(M, __ldcg(base + s * (D + 4) + D));
  float den = 0.f, num = 0.f;
#pragma unroll 1
  for (uint32_t s = 0; s < S; ++s) {
    const float ms = __ldcg(base + s * (D + 4) + D), ls = __ldcg(base + s * (D + 4) + D + 1);
    if (ls > 0.f) {
      const float w = expf(ms - M);
      den += ls * w;
      num += __ldcg(base + s * (D + 4) + tid) * w;
    }
  }
  p.ao[(size_t)h * D + tid] = ll_pack(__float2half_rn(num / den), tag_out);
}

// Embedding gather + dequantisation of the current token (embedding_q8_0.comp:39-85).
template <bool F16>
__device__ VKL_SLOW void embed_op(const Ctx &c, uint32_t tok, uint32_t tag_out) {
  const MegaParams &p = c.p;
  const uint32_t per = (p.dim + gridDim.x - 1) / gridDim.x;
  const uint32_t k = blockIdx.x * per + threadIdx.x;
  if (threadIdx.x >= per || k >= p.dim) return;
  if (tok >= p.embd_rows) tok = 0;  // UNK = 0 (models/llama2.h:455-458)
  if (F16) {
    p.x[k] = ll_pack(reinterpret_cast<const __half *>(p.embd)[(size_t)tok * p.dim + k], tag_out);
    return;
  }
  const Q8Layout L = q8_layout(p.embd_rows, p.dim);
  const uint32_t tile = tok >> 4, r = tok & 15, g = r & 7, half = r >> 3;
  const uint32_t b = k >> 5, t = (k >> 3) & 3, i = k & 7;
  const uint8_t cb = p.embd[(((size_t)tile * L.groups * 4 + b) * 32 + g * 4 + t) * 16 + half * 8 + q8_byte_pos(i)];
  const uint16_t *sc = reinterpret_cast<const uint16_t *>(p.embd + L.codes_bytes());
  const uint16_t d = sc[(((size_t)tile * L.groups + (b >> 2)) * 8 + g) * 8 + half * 4 + (b & 3)];
  p.x[k] = ll_pack(__float2half_rn((float)((int)cb - 128) * __half2float(__ushort_as_half(d))), tag_out);
}

// CTA 0: best of the per-CTA candidates (lowest index on ties), then publish the id,
// feed it back and advance position, step and launch epoch.
template <bool TP>
__device__ VKL_SLOW void argmax_final_op(const Ctx &c, float *sm, uint32_t pos0, uint64_t rounds_done, uint32_t ar_done,
                                                uint32_t next_ebase) {
  const MegaParams &p = c.p;
  if (blockIdx.x != 0) return;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  Best b = {0.f, 0xffffffffu};
#pragma unroll 1
  for (uint32_t i = tid; i < gridDim.x; i += CT) {
    const float v = __ldcg(p.arg_scratch + 2 * i);
    const uint32_t ix = __float_as_uint(__ldcg(p.arg_scratch + 2 * i + 1));
    if (ix != 0xffffffffu && better(v, ix, b)) {
      b.v = v;
      b.i = ix;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, b.v, o);
    const uint32_t oi = __shfl_xor_sync(0xffffffffu, b.i, o);
    if (oi != 0xffffffffu && better(ov, oi, b)) {
      b.v = ov;
      b.i = oi;
    }
  }
  uint32_t *si = reinterpret_cast<uint32_t *>(sm);
  if (lane == 0) {
    sm[32 + warp] = b.v;
    si[warp] = b.i;
  }
  cons_sync();
  if (tid == 0) {
#pragma unroll 1
    for (int w = 1; w < NCW; ++w)
      if (si[w] != 0xffffffffu && better(sm[32 + w], si[w], b)) {
        b.v = sm[32 + w];
        b.i = si[w];
      }
    if (TP && p.tp_size > 1 && !c.aborted()) {
      // vocabulary-split lm head: exchange (value, global index) candidates with all ranks
      const uint32_t tp = p.tp_size, aseq = p.state[4] + 1;
      b.i += p.tp_rank * p.vocab;
      for (uint32_t r = 0; r < tp; ++r) {
        float *cand = static_cast<float *>(p.tp_peer[r]) + p.tp_flag_off + 32 + 2 * p.tp_rank;
        cand[0] = b.v;
        cand[1] = __uint_as_float(b.i);
      }
      __threadfence_system();
      for (uint32_t r = 0; r < tp; ++r) st_rel_sys_u32(static_cast<uint32_t *>(p.tp_peer[r]) + p.tp_flag_off + 16 + p.tp_rank, aseq);
      const uint32_t *mine = static_cast<const uint32_t *>(p.tp_peer[p.tp_rank]) + p.tp_flag_off;
      for (uint32_t r = 0; r < tp && !c.aborted(); ++r) {
        bool ok = false;
      #pragma unroll 1
        for (uint32_t i = 0; i < c.p.wait_limit; ++i) {
          if ((int32_t)(ld_acq_sys_u32(mine + 16 + r) - aseq) >= 0) {
            ok = true;
            break;
          }
          if (i > 100000u) __nanosleep(64);
        }
        if (!ok) c.raise(5);
      }
      Best gb = {0.f, 0xffffffffu};
      for (uint32_t r = 0; r < tp; ++r) {
        const float *cand = static_cast<const float *>(p.tp_peer[p.tp_rank]) + p.tp_flag_off + 32 + 2 * r;
        const float v = __ldcg(cand);
        const uint32_t ix = __float_as_uint(__ldcg(cand + 1));
        if (better(v, ix, gb)) {
          gb.v = v;
          gb.i = ix;
        }
      }
      b = gb;
      p.state[4] = aseq;
    }
    if (!c.aborted()) {
      const uint32_t step = p.with_token ? 0u : p.state[1], n_forced = p.with_token ? 0u : p.state[5];
      if (p.with_token) p.state[5] = 0;
      p.state[2] = b.i;
      if (pos0 + 1 < n_forced) {
        p.tok[0] = p.forced[pos0 + 1];  // still inside the prompt: feed the next prompt token
      } else {
        p.tok[0] = b.i;
        if (step < p.out_cap) p.out_ids[step] = b.i;
        p.state[1] = step + 1;
      }
      p.state[0] = pos0 + 1;
      p.state[3] = ar_done;
      p.state[7] = next_ebase;
      p.bar[1] = rounds_done;
      if (p.host_logits) reinterpret_cast<uint32_t *>(p.host_logits)[p.vocab] = 0u;
    }
  }
}

// Tensor-parallel all-reduce, second half. The partial sums were pushed to every rank by the
// preceding row-split projection as 8-byte words {fp32 sum, all-reduce sequence number}.
// Every CTA reduces its slice of rows in rank order as soon as the words of all ranks carry
// this all-reduce's number: x <- fp16( fp16(sum_r partial_r) + x ), the same rounding as
// o_proj/down + residual add. No grid barrier and no separate flags: two parities of slots
// keep a fast rank's next push from overwriting what a slow rank still reads.
__device__ VKL_SLOW void allreduce_op(const Ctx &c, const MegaOp &op, uint32_t seq, uint32_t tag_out, uint32_t tag_res) {
  const MegaParams &p = c.p;
  const uint32_t tid = threadIdx.x, tp = p.tp_size;
  if (c.aborted()) return;
  const uint32_t per = (p.dim + gridDim.x - 1) / gridDim.x;
  const uint32_t i = blockIdx.x * per + tid;
  if (tid < per && i < p.dim) {
    // every rank pushed {partial sum, sequence number} words into this rank's buffer: poll this
    // row's word of every rank (bounded), add in rank order
    const uint32_t *part = static_cast<const uint32_t *>(p.tp_peer[p.tp_rank]) + 2 * ((size_t)(seq & 1u) * tp * p.dim);
    float s = 0.f;
    for (uint32_t r = 0; r < tp; ++r) {
      const uint32_t *src = part + 2 * ((size_t)r * p.dim + i);
      uint2 w = ld_vol_v2(src);
      if (w.y != seq) {
        bool ok = false;
      #pragma unroll 1
        for (uint32_t it = 0; it < p.wait_limit; ++it) {
          w = ld_vol_v2(src);
          if (w.y == seq) {
            ok = true;
            break;
          }
          if (it > 100000u) __nanosleep(64);
          if ((it & 1023u) == 1023u && (*(volatile uint32_t *)p.error != 0u || c.aborted())) break;
        }
        if (!ok) {
          c.raise(4);
          return;
        }
      }
      s += __uint_as_float(w.x);
    }
    const float res = __half2float(ll_half(c.ll_wait1(op.out_ll[0] + i, tag_res)));  // the residual, under the tag of the op that wrote it
    op.out_ll[0][i] = ll_pack(__float2half_rn(round_h(s) + res), tag_out);
  }
}

template <bool TIMED, bool DBG, bool TP, bool F16>
__global__ void __launch_bounds__(THREADS, 1) decode_mega_kernel(const __grid_constant__ MegaParams p) {
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t NST = p.nst;
  unsigned char *rings = smem;
  unsigned char *xq = smem + (size_t)NCW * NST * PIECE_BYTES;  // input vector; attention scratch
  float *red = reinterpret_cast<float *>(xq + p.xs_bytes);
  float *ssum = red + (size_t)p.red_slots * NCW * 32;  // [64]
  MegaRun *runs = reinterpret_cast<MegaRun *>(ssum + 64);  // [run_stride], 16-byte aligned
  KvPlan *kvp = reinterpret_cast<KvPlan *>(runs + p.run_stride);
  uint64_t *full = reinterpret_cast<uint64_t *>(kvp + 1);
  volatile uint32_t *abort_s = reinterpret_cast<volatile uint32_t *>(full + NCW * MAX_NST);
  // The op table lives in global memory; reading an entry there costs a chain of L2 round trips
  // (kind, then the fields, then what they point to) at the start of every op. Three entries are
  // kept in shared memory instead: the running op, the next one (looked at when this one ends)
  // and the one after, which is copied in asynchronously while this op runs.
  MegaOp *opbuf = reinterpret_cast<MegaOp *>(reinterpret_cast<unsigned char *>(full + NCW * MAX_NST) + 16);
  constexpr uint32_t OPV = sizeof(MegaOp) / 16;
  static_assert(sizeof(MegaOp) % 16 == 0, "MegaOp is copied in 16-byte pieces");
  if (threadIdx.x < 2 * OPV && threadIdx.x / OPV < p.nops)
    reinterpret_cast<uint4 *>(opbuf)[threadIdx.x] = reinterpret_cast<const uint4 *>(p.ops)[threadIdx.x];

  const uint32_t nruns = p.run_count[blockIdx.x];
#pragma unroll 1
  for (uint32_t i = threadIdx.x; i < nruns; i += CT) runs[i] = p.runs[(size_t)blockIdx.x * p.run_stride + i];
  const uint32_t pos0 = p.with_token ? p.call_pos : p.state[0], tok = p.with_token ? p.call_tok : p.tok[0];
  if ((threadIdx.x & 31) == 0) {
    const uint32_t warp = threadIdx.x >> 5;
#pragma unroll 1
    for (uint32_t i = 0; i < NST; ++i) mbar_init(s32(&full[warp * NST + i]), 1);
    kv_plan(p, *kvp, pos0, warp);
  }
  if (threadIdx.x == 0) {
    abort_s[0] = 0;
    abort_s[1] = 0;
  }
  if ((threadIdx.x & 31) == 0) {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  const Ctx c{p, abort_s};
  const RunTable tab{runs, nruns, kvp};
  Ring ring;
  {
    const uint32_t warp = threadIdx.x >> 5;
    ring.piece = s32(rings + (size_t)warp * NST * PIECE_BYTES);
    ring.bar = s32(full + warp * NST);
    ring.last = ring.bar + (NST - 1) * 8;
    ring.ph = ring.whole = ring.rest = ring.next = ring.asked = 0;
    ring.lead = (threadIdx.x & 31) == 0 && (!DBG || !(p.timing_mode & 128u));
    ring.second = false;
    ring.src = nullptr;
    ring.to_v = 0;
    if (ring.lead)
#pragma unroll 1
      for (uint32_t i = 0; i < NST; ++i) ring_request<DBG, F16>(p, tab, ring, ring.piece + i * PIECE_BYTES, ring.bar + i * 8, warp);
    __syncwarp();
  }
  const uint32_t S_eff = kvp->S;

  const uint32_t G = gridDim.x;
  const uint64_t base_rounds = p.bar[1];  // barrier rounds completed by earlier launches
  uint64_t rounds = 0;
  const uint32_t seq0 = p.state[3];  // all-reduces completed by earlier launches
  uint32_t ar_i = 0;
  const uint32_t ebase = p.state[7];  // sequence number of this launch's first op; op oi tags its results with ebase + oi
  auto tag = [&](uint32_t op_index) { return (ebase + op_index) & 0xffffu; };
  Best best = {0.f, 0xffffffffu};
  const bool tracing = TIMED && p.timing != nullptr && (p.timing_mode & 256u) != 0;
  const bool timed = TIMED && p.timing != nullptr && !tracing && blockIdx.x == 0 && threadIdx.x == 0;
  unsigned long long t0 = 0, twait[3] = {0, 0, 0}, c0 = 0;
  if (timed) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (uint32_t oi = 0; oi < p.nops; ++oi) {
    const MegaOp &op = opbuf[oi % 3];
    if (oi + 2 < p.nops && threadIdx.x < OPV) {  // entry oi + 2 replaces entry oi - 1, which every thread has left
      const uint32_t dst = s32(reinterpret_cast<uint4 *>(opbuf + (oi + 2) % 3) + threadIdx.x);
      const uint4 *src = reinterpret_cast<const uint4 *>(p.ops + oi + 2) + threadIdx.x;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(__cvta_generic_to_global(src)) : "memory");
    }
    if (op.kind == MK_ATTN_COMBINE && S_eff == 1) {  // nothing to merge, no grid barrier either
      cons_sync();  // every thread has read this entry before the next op's copy may replace it
      continue;
    }
    if (timed) c0 = clock64();
    unsigned long long *trace = (tracing && threadIdx.x == 0) ? p.timing + ((size_t)oi * gridDim.x + blockIdx.x) * 8 : nullptr;
    VKL_TRACE(0);
    switch (op.kind) {
      case MK_EMBED: embed_op<F16>(c, tok, tag(oi)); break;
      case MK_MATVEC: matvec_op<TIMED, DBG, TP, F16>(c, op, tab, ring, reinterpret_cast<__half *>(xq), reinterpret_cast<float *>(xq + (size_t)p.xmax_blocks * XB_BYTES), red, ssum, best, (TIMED && timed) ? twait : nullptr, seq0 + ar_i + 1,
                         tag(op.src_op), tag(oi), tag(op.res_op), trace);
        if (op.epi == EPI_REDUCE) ++ar_i;  // (every CTA counts it, with or without a tile of the op)
        break;
      case MK_ATTN_PART:
        attn_part_op<DBG, F16>(c, op, reinterpret_cast<float *>(xq), pos0, *kvp, tag(op.src_op), tag(op.tag_op), tab, ring);
        break;
      case MK_ATTN_COMBINE: attn_combine_op(c, S_eff, tag(oi)); break;
      case MK_ALLREDUCE:
        if (!TP) break;
        ++ar_i;
        allreduce_op(c, op, seq0 + ar_i, tag(oi), tag(op.res_op));
        break;
      case MK_ARGMAX:
        argmax_final_op<TP>(c, reinterpret_cast<float *>(xq), pos0, base_rounds + rounds, seq0 + ar_i, ebase + p.nops);
        break;
    }
    if (op.kind == MK_MATVEC && op.track_argmax) {
      // per-CTA arg-max candidate: every epilogue thread holds the best of its rows
      Best bb = best;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bb.v, o);
        const uint32_t oi2 = __shfl_xor_sync(0xffffffffu, bb.i, o);
        if (oi2 != 0xffffffffu && better(ov, oi2, bb)) {
          bb.v = ov;
          bb.i = oi2;
        }
      }
      float *cand = ssum;  // [NCW] values, then [NCW] indices
      cons_sync();
      if ((threadIdx.x & 31) == 0) {
        cand[threadIdx.x >> 5] = bb.v;
        cand[NCW + (threadIdx.x >> 5)] = __uint_as_float(bb.i);
      }
      cons_sync();
      if (threadIdx.x == 0) {
#pragma unroll 1
        for (int w = 1; w < NCW; ++w) {
          const uint32_t wi = __float_as_uint(cand[NCW + w]);
          if (wi != 0xffffffffu && better(cand[w], wi, bb)) {
            bb.v = cand[w];
            bb.i = wi;
          }
        }
        p.arg_scratch[2 * blockIdx.x] = bb.v;
        p.arg_scratch[2 * blockIdx.x + 1] = __uint_as_float(bb.i);
      }
    }
    unsigned long long t1 = 0, t2 = 0;
    VKL_TRACE(4);
    if (timed) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
    if (oi + 1 < p.nops) {
      // While waiting for the other CTAs: start what the next op will need from DRAM and does not depend
      // on this op's results. The 7 GB weight stream of a token flushes everything else out of L2 between
      // two uses, so the norm weights would otherwise sit, with a DRAM round trip, at the start of the next
      // op: this prefetch is worth 7 % of the token time.
      const MegaOp &nx = opbuf[(oi + 1) % 3];
      if (nx.kind == MK_MATVEC) {
        if (nx.norm_w)
#pragma unroll 1
          for (uint32_t i = threadIdx.x * 32; i < nx.K; i += CT * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(nx.norm_w + i));
      }
      asm volatile("cp.async.wait_all;" ::: "memory");  // entry oi + 2 has landed; the barrier below publishes it
      if (op.barrier_after) {
        ++rounds;
        grid_barrier(c, (base_rounds + rounds) * G, (uint32_t)rounds, abort_s + 1);
      } else {
        cons_sync();  // the next op reuses this one's shared memory; its input words carry their own arrival tags
      }
    }
    VKL_TRACE(5);
    if (timed) {
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t2));
      p.timing[2 * oi] = t1 - t0;
      p.timing[2 * oi + 1] = t2 - t1;
      const unsigned long long cend = clock64();
      p.timing[2 * p.nops + oi] = (p.timing_mode & 8u) ? (twait[2] ? (cend - twait[2]) * 1000ull / p.sm_mhz - (t2 - t1) : 0ull)
                                  : getenv_prologue(p) ? (twait[1] > c0 ? (twait[1] - c0) * 1000ull / p.sm_mhz : 0ull)
                                                        : twait[0];
      twait[2] = 0;
      twait[0] = 0;
      twait[1] = 0;
      t0 = t2;
    }
  }
  if ((threadIdx.x & 31) == 0 && !ring.lead && (!DBG || !(p.timing_mode & 128u))) ring_drain(p, ring);
  // A CTA that gave up has published words computed from whatever it had, and CTA 0 may have ended the launch with them all the
  // same. (Its threads have met since it gave up, in the last op's barrier; CTA 0's own late waits are this thread's.)
  if (threadIdx.x == 0 && p.host_logits && c.aborted()) reinterpret_cast<uint32_t *>(p.host_logits)[p.vocab + 1] = 1u;
}

}  // namespace

size_t decode_mega_xs_bytes(uint32_t max_blocks, uint32_t head_dim) {
  const size_t x = (size_t)max_blocks * (XB_BYTES + 4);  // fp16 input + one fp32 bias term per block of 32 inputs
  const size_t a = (size_t)(NCW * (head_dim + 2) + 4 + head_dim) * 4;  // attention: every warp's sums, maximum and denominator; the new K and V rows
  return (std::max(x, a) + 127) / 128 * 128;
}
size_t decode_mega_smem(size_t xs_bytes, uint32_t nst, uint32_t red_slots, uint32_t runs) {
  return (size_t)NCW * nst * PIECE_BYTES + xs_bytes + ((size_t)red_slots * NCW * 32 + 64) * 4 + runs * sizeof(MegaRun) + sizeof(KvPlan) + NCW * MAX_NST * 8 + 16 + 3 * sizeof(MegaOp) + 64;
}
int decode_mega_max_k() { return 16384; }
int decode_mega_max_stages() { return MAX_NST; }

// Packs the op's matrices from the library's tiled planes (common.cuh) into the stream layout of
// MegaOp: one CTA per (block, tile), one thread per 16-byte piece. A 32-row tile's unit is the two
// 512-byte (16 rows x 32 columns) units of the planes that hold its rows, unchanged (codes stay
// biased by +128 in MMA fragment order), followed by the 32 scales in the order the consumer lanes
// read them. Tiles are stored in the order the decode kernel's CTAs take them (mega_stream_tile), so
// that every CTA reads one consecutive range of the op.
namespace {
constexpr uint32_t kGridY = 65535;  // tiles of a launch: a vocabulary of 2.1 million rows has more
__global__ void __launch_bounds__(64) mega_pack_kernel(const uint8_t *p0, const uint8_t *p1, const uint8_t *p2, uint32_t nmat, int swiglu, uint32_t N,
                                                       uint32_t K, uint32_t tile0, uint32_t tiles, uint32_t grid, uint8_t *stream) {
  const uint32_t b = blockIdx.x, t = tile0 + blockIdx.y, blocks = K / 32;
  const uint32_t half = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tpm = (N + 31) / 32;
  // the 16-row plane tile behind this half of the 32-row tile
  uint32_t m, tile16;
  if (swiglu) {
    m = half;  // gate rows 16 t .., then up rows 16 t ..
    tile16 = t;
  } else if (nmat == 3) {
    m = t / tpm;
    tile16 = (t % tpm) * 2 + half;
  } else {
    m = 0;
    tile16 = t * 2 + half;
  }
  const uint8_t *src = m == 0 ? p0 : m == 1 ? p1 : p2;
  const Q8Layout L = q8_layout(N, K);
  const bool in = tile16 < L.tiles;
  uint4 w = make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u);  // code 0, biased
  if (in) w = *reinterpret_cast<const uint4 *>(src + (((size_t)tile16 * L.groups * 4 + b) * 32 + lane) * 16);
  const size_t unit = (size_t)mega_stream_tile(t, tiles, grid) * blocks + b;
  uint8_t *dst = stream + unit * (MEGA_UNIT_CODES + MEGA_UNIT_SCALES);
  reinterpret_cast<uint4 *>(dst)[half * 32 + lane] = w;
  if (lane < 16) {
    // scales of the unit: [g][row g | g + 8 of half 0, row g | g + 8 of half 1] as fp16
    const uint32_t g = lane & 7, up8 = lane >> 3;
    unsigned short d = 0;
    if (in) {
      const unsigned short *sc = reinterpret_cast<const unsigned short *>(src + L.codes_bytes());
      d = sc[(((size_t)tile16 * L.groups + (b >> 2)) * 8 + g) * 8 + up8 * 4 + (b & 3)];
    }
    reinterpret_cast<unsigned short *>(dst + MEGA_UNIT_CODES)[g * 4 + half * 2 + up8] = d;
  }
}
}  // namespace

cudaError_t launch_mega_pack(const uint8_t *const planes[3], uint32_t nmat, int swiglu, uint32_t N, uint32_t K, uint32_t tiles, uint32_t grid,
                             uint8_t *stream, cudaStream_t s) {
  if (K % 32 || tiles == 0 || grid == 0) return cudaErrorInvalidValue;
  for (uint32_t t = 0; t < tiles; t += kGridY)
    mega_pack_kernel<<<dim3(K / 32, std::min(tiles - t, kGridY)), 64, 0, s>>>(planes[0], planes[1], planes[2], nmat, swiglu, N, K, t, tiles, grid, stream);
  return cudaGetLastError();
}

// The same for FP16 matrices [N, K]: a unit is 32 rows x 16 columns, 512 bytes per 16 rows: lane (g, t) has columns 4 t and 4 t + 1 of
// rows g and g + 8, then columns 4 t + 2 and 4 t + 3 of both, the A fragment of one m16n8k16 whose k runs through the columns
// in this order (for the input the same).
namespace {
// A CTA packs eight blocks of a tile, a warp each, so that it reads whole lines.
__global__ void __launch_bounds__(256) mega_pack_f16_kernel(const __half *p0, const __half *p1, const __half *p2, uint32_t nmat, int swiglu, uint32_t N, uint32_t K, uint32_t tile0,
                                                            uint32_t tiles, uint32_t grid, uint8_t *stream) {
  const uint32_t b = blockIdx.x * 8 + (threadIdx.x >> 5), t = tile0 + blockIdx.y, blocks = K / 16, lane = threadIdx.x & 31, g = lane >> 2, c = b * 16 + (lane & 3) * 4;
  if (b >= blocks) return;
  const uint32_t tpm = (N + 31) / 32;
  uint4 *dst = reinterpret_cast<uint4 *>(stream + ((size_t)mega_stream_tile(t, tiles, grid) * blocks + b) * MEGA_UNIT_CODES) + lane;
#pragma unroll
  for (uint32_t half = 0; half < 2; ++half) {
    const uint32_t m = swiglu ? half : nmat == 3 ? t / tpm : 0u, row = swiglu ? t * 16 + g : (nmat == 3 ? t % tpm : t) * 32 + half * 16 + g;
    const __half *src = m == 0 ? p0 : m == 1 ? p1 : p2;
    uint2 lo = make_uint2(0, 0), hi = lo;
    if (row < N) lo = __ldcs(reinterpret_cast<const uint2 *>(src + (size_t)row * K + c));
    if (row + 8 < N) hi = __ldcs(reinterpret_cast<const uint2 *>(src + (size_t)(row + 8) * K + c));
    dst[half * 32] = make_uint4(lo.x, hi.x, lo.y, hi.y);
  }
}
}  // namespace
cudaError_t launch_mega_pack_f16(const __half *const w[3], uint32_t nmat, int swiglu, uint32_t N, uint32_t K, uint32_t tiles, uint32_t grid, uint8_t *stream, cudaStream_t s) {
  if (K % 16 || tiles == 0 || grid == 0) return cudaErrorInvalidValue;
  for (uint32_t t = 0; t < tiles; t += kGridY)
    mega_pack_f16_kernel<<<dim3((K / 16 + 7) / 8, std::min(tiles - t, kGridY)), 256, 0, s>>>(w[0], w[1], w[2], nmat, swiglu, N, K, t, tiles, grid, stream);
  return cudaGetLastError();
}

cudaError_t launch_decode_mega(const MegaParams &p, int grid, cudaStream_t s) {
  if (p.nst < 2 || p.nst > (uint32_t)MAX_NST) return cudaErrorInvalidValue;
  const size_t smem = decode_mega_smem(p.xs_bytes, p.nst, p.red_slots, p.run_stride);
  // the diagnostic switches (no weight copies, no arithmetic) are compiled into separate instances, for Q8_0 weights only
  const bool dbg = (p.timing_mode & (2u | 4u | 16u | 64u | 128u)) != 0;  // (16: the diagnostic instance with nothing switched off, its own baseline)
  auto kern = p.f16 ? (p.timing ? decode_mega_kernel<true, false, false, true> : decode_mega_kernel<false, false, false, true>)
              : p.timing ? (dbg || p.tp_size > 1 ? decode_mega_kernel<true, true, true, false> : decode_mega_kernel<true, false, false, false>)
              : dbg      ? decode_mega_kernel<false, true, true, false>
              : p.tp_size > 1 ? decode_mega_kernel<false, false, true, false> : decode_mega_kernel<false, false, false, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  void *args[] = {(void *)&p};
  return cudaLaunchCooperativeKernel((void *)kern, dim3(grid), dim3(THREADS), args, smem, s);
}

cudaError_t decode_mega_occupancy(size_t smem, bool f16, bool tp, int *blocks_per_sm) {
  auto kern = f16 ? decode_mega_kernel<false, false, false, true> : tp ? decode_mega_kernel<false, false, true, false> : decode_mega_kernel<false, false, false, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kern, THREADS, smem);
}

}  // namespace vkl
