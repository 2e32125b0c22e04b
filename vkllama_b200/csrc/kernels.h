// Host-callable launchers of every CUDA kernel in the library. All pointers are
// device pointers; every launcher enqueues on `stream` and returns the CUDA
// error of the launch (no synchronisation).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace vkl {

// EPI_PARTIAL (persistent decode kernel only): raw fp32 partial sums of a row-split
// projection, pushed into every tensor-parallel rank's exchange buffer.
// EPI_REDUCE (persistent decode kernel only): the same, and the thread that pushed a row's partial sum also
// waits for the other ranks' sums of that row, adds them in rank order with the residual and publishes the row:
// the all-reduce needs no op of its own.
enum MvEpilogue { EPI_PLAIN = 0, EPI_ADD = 1, EPI_SWIGLU = 2, EPI_PARTIAL = 3, EPI_REDUCE = 4 };

// Y = epilogue(X . W^T) for up to three Q8_0 (tiled planes) or FP16 (row-major)
// weight matrices [N,K] sharing one input X [M,K].
struct MvParams {
  const uint8_t *codes[3];   // Q8_0: codes plane; FP16: row-major weights
  const uint8_t *scales[3];  // Q8_0: scales plane; FP16: unused
  __half *out[3];            // fp16 [M, out_ld] per matrix (SWIGLU: out[0] only)
  float *out_f32;            // optional fp32 copy of out[0] (cast of the fp16 value)
  const __half *x;           // [M, x_ld]
  const __half *residual;    // EPI_ADD: [M, out_ld], may alias out[0]
  const float *norm_w;       // fused RMSNorm weight [K] (decode path), or null
  float eps;
  uint32_t nmat;             // 1..3 matrices (SWIGLU: codes[0]=gate, codes[1]=up, nmat=1)
  uint32_t N, K, M;
  uint32_t x_ld, out_ld;
  float scale, bias;
  int act;                   // 1 = SiLU on the PLAIN epilogue
  int fp16_weights;          // 0 = Q8_0 tiled planes, 1 = FP16 row-major
  int use_pdl;               // programmatic dependent launch: prefetch weights before waiting
  uint32_t *error;           // device word raised when a bounded wait ran out (where matvec_waits), or null
};
cudaError_t launch_matvec(const MvParams &p, int epilogue, bool fuse_norm_smem, cudaStream_t s);
// 9 to 64 rows (skinny_gemm.cu); launch_matvec sends what it takes there
bool skinny_gemm_takes(const MvParams &p, int epilogue);
cudaError_t launch_skinny_gemm(const MvParams &p, int epilogue, cudaStream_t s);
bool matvec_waits(const MvParams &p, int epilogue);  // whether launch_matvec runs a kernel with bounded waits (p.error)

// 34-byte GGUF blocks <-> tiled planes (codes at dst, scales at dst + codes_bytes).
cudaError_t launch_q8_repack(const uint8_t *blocks34, uint8_t *planes, uint32_t N, uint32_t K,
                             cudaStream_t s);
cudaError_t launch_q8_unpack(const uint8_t *planes, uint8_t *blocks34, uint32_t N, uint32_t K,
                             cudaStream_t s);
// fp32 [N,K] -> 34-byte blocks on the device (same arithmetic as the host quantizer).
cudaError_t launch_q8_quantize(const float *src, uint8_t *blocks34, uint32_t N, uint32_t K,
                               cudaStream_t s);
// Seeded synthetic data, bit-identical to the host generator.
cudaError_t launch_synth_f32(float *dst, uint64_t seed, uint64_t tensor, uint64_t first,
                             uint64_t n, float mean, float stdv, cudaStream_t s);
cudaError_t launch_synth_f16(__half *dst, uint64_t seed, uint64_t tensor, uint64_t first,
                             uint64_t n, float mean, float stdv, cudaStream_t s);
// Synthetic N(mean,std) matrix quantised straight into 34-byte blocks. The [N,K]
// result is the window at (row0, col0) of a full matrix with `ld_full` columns
// (element index = (row0+r)*ld_full + col0 + k), so a shard equals a slice.
cudaError_t launch_synth_q8(uint8_t *blocks34, uint64_t seed, uint64_t tensor, uint32_t N,
                            uint32_t K, float mean, float stdv, uint32_t row0, uint32_t col0,
                            uint32_t ld_full, cudaStream_t s);

cudaError_t launch_rms_norm(const __half *x, const float *w, __half *y, uint32_t rows,
                            uint32_t W, float eps, cudaStream_t s);
cudaError_t launch_add(const __half *x, __half *y, uint64_t n, int op, cudaStream_t s);
// x <- fp16(x op alpha), op 0 add, 1 sub, 2 mul, 3 div.
cudaError_t launch_scalar_op(__half *x, uint64_t n, int op, float alpha, cudaStream_t s);
// Copies a dense [C,H,W] input to out[c * ocs + h * ohs + w + offset] (element strides).
cudaError_t launch_concat_copy(const __half *in, __half *out, uint32_t C, uint32_t H, uint32_t W, uint64_t ocs, uint64_t ohs, uint64_t offset,
                               cudaStream_t s);
// Row reduction over W: op 0 sum, 1 max, 2 min; the result is scaled by mean_scale.
cudaError_t launch_reduce(const __half *in, __half *out, uint32_t rows, uint32_t W, int op, float mean_scale, cudaStream_t s);
// out[c, y, :] = cache[c, (y + offset) % H, :] for y < len.
cudaError_t launch_read_kvcache(const __half *cache, __half *out, uint32_t C, uint32_t H, uint32_t W, uint32_t offset, uint32_t len,
                                cudaStream_t s);
// All-reduce of fp32 partial sums [n] over tensor-parallel ranks with the residual add of the K-split
// projections: x = fp16(fp16(sum over ranks, in rank order) + x). part[r] / flags[r] are rank r's partial
// sums and flag words [tp] (peer mappings; [rank] is this GPU's). A wait that runs out of `wait_limit`
// polls stores 16 into *error and leaves x as it was.
struct TpRowsParams {
  const float *part[8];
  uint32_t *flags[8];
  __half *x;
  size_t n;
  uint32_t rank, tp, seq, wait_limit;
  uint32_t *error;
};
cudaError_t launch_tp_reduce_rows(const TpRowsParams &p, int sms, cudaStream_t s);
cudaError_t launch_embedding(const uint8_t *vocab, int vocab_is_q8, const uint32_t *ids,
                             __half *out, uint32_t T, uint32_t VH, uint32_t VW, uint32_t unk,
                             cudaStream_t s);
// Two-stage arg-max/min over rows of width W; partials needs rows*ceil(W/1024)*8 bytes.
cudaError_t launch_argop(const __half *x, uint32_t *out, void *partials, uint32_t rows,
                         uint32_t W, int op_type, cudaStream_t s);
cudaError_t launch_argmax_f32(const float *x, uint32_t *out, void *partials, uint32_t rows, uint32_t W, cudaStream_t s);
size_t argop_partials_bytes(uint32_t rows, uint32_t W);
// The k largest of n fp32 values and their indices, descending (equal values: lowest index first).
cudaError_t launch_topk_f32(const float *x, uint32_t n, uint32_t k, float *vals, uint32_t *ids, cudaStream_t s);
cudaError_t launch_softmax(const __half *in, __half *out, uint32_t C, uint32_t H, uint32_t W,
                           int seq_mask, uint32_t offset, cudaStream_t s);
cudaError_t launch_rope(__half *x, uint32_t C, uint32_t H, uint32_t W, uint64_t cs, uint64_t hs,
                        const uint32_t *pos_dev, uint32_t offset, const float *freqc,
                        const float *freqs, cudaStream_t s);
cudaError_t launch_update_kvcache(__half *cache, const __half *kv, uint32_t C, uint32_t H,
                                  uint32_t W, uint32_t HO, uint32_t WO, uint32_t offset,
                                  cudaStream_t s);
cudaError_t launch_transpose(const __half *in, __half *out, uint32_t C, uint32_t H, uint32_t W,
                             cudaStream_t s);
cudaError_t launch_slice(const __half *in, __half *out, uint32_t C, uint32_t H, uint32_t W,
                         uint32_t c0, uint32_t h0, uint32_t w0, uint32_t EC, uint32_t EH,
                         uint32_t EW, cudaStream_t s);
cudaError_t launch_cast_f16_f32(const __half *in, float *out, uint64_t n, cudaStream_t s);
cudaError_t launch_cast_f32_f16(const float *in, __half *out, uint64_t n, cudaStream_t s);
// Batched fp16 x fp16 matmul with element strides; transpose_b selects A.B^T.
cudaError_t launch_bmm_f16(const __half *a, const __half *b, __half *c, uint32_t C, uint32_t M,
                           uint32_t N, uint32_t K, uint64_t a_cs, uint64_t a_hs, uint64_t b_cs,
                           uint64_t b_hs, uint64_t c_cs, uint64_t c_hs, int transpose_b,
                           float scale, float bias, int act, cudaStream_t s);

// Fused attention core for the model path. q,k,v: [T, heads*dim] fresh projections.
// Rotates q and k at positions pos+row, appends k,v to the caches [heads,maxlen,dim]
// at (pos+row) % maxlen, then softmax(q.K^T/sqrt(dim)).V over the first
// min(pos+T, maxlen) cache rows with the causal mask; out: [T, heads*dim].
struct AttnParams {
  __half *q;
  const __half *k, *v;
  __half *kcache, *vcache;
  __half *out;
  const float *freqc, *freqs;
  const uint32_t *pos_dev;  // position of row 0, read on the device
  float *scratch;           // of attention_plan's size
  uint32_t *counters;       // attention_plan's number, zero before first use (left zero after)
  uint32_t T, heads, dim, maxlen, splits;  // splits: attention_plan's, or fewer
  // clip: only the last row is computed and written to row 0 of `out`; its query is
  // rotated at position pos (row 0), as the reference does after clipping Q
  // (src/ops/multiheadattention_v2.cpp:223-253).
  int clip;
  int use_pdl;
};
cudaError_t launch_attention(const AttnParams &p, cudaStream_t s);
struct AttnPlan {
  uint32_t splits;
  size_t scratch_bytes;
  uint32_t counters;
};
AttnPlan attention_plan(uint32_t T, bool clip, uint32_t heads, uint32_t dim, uint32_t sms);
AttnPlan attention_plan_most(uint32_t T, uint32_t heads, uint32_t dim, uint32_t sms);  // what calls of up to T rows need

// ---- persistent decode step (decode_mega.cu) --------------------------------
enum MegaKind { MK_EMBED = 0, MK_MATVEC = 1, MK_ATTN_PART = 2, MK_ATTN_COMBINE = 3, MK_ARGMAX = 4, MK_ALLREDUCE = 5 };
// One entry of the token's op table. The kernel keeps the current and the next entry in shared
// memory (copied there with 16-byte asynchronous copies while the op before runs), so the size
// is a multiple of 16 bytes.
struct alignas(16) MegaOp {
  uint32_t kind, epi, nmat, rot;
  uint32_t N, K;          // rows of one matrix, columns
  uint32_t tiles, blocks; // 32-row tiles of the op's packed weight stream, units per tile (K / 32; FP16 weights K / 16)
  // The op's weights, packed for the kernel (mega_pack): per 32-row tile and block one unit of
  // MEGA_UNIT_CODES + MEGA_UNIT_SCALES bytes. Codes: the two 512-byte (16 rows x 32 columns) units of the
  // library's tiled planes (common.cuh) that hold the tile's rows, as they are: MMA A-fragment order, biased
  // by +128. Then the unit's scales: [g 0..7][rows g, g + 8, 16 + g, 24 + g] fp16. (FP16 weights: mega_pack_f16.) Units of a tile follow each
  // other block by block, tiles in the order of mega_stream_tile: everything one CTA reads of the op is one
  // consecutive range. Which matrix row a tile row is:
  //   one matrix         tile t, row r = matrix row 32 t + r
  //   nmat = 3 (K, Q, V) tile t = matrix t / tpm, rows 32 (t % tpm) + r, tpm = ceil(N / 32)
  //   SwiGLU (gate, up)  tile t: rows 0..15 = gate rows 16 t + r, rows 16..31 = up rows 16 t + r - 16
  const uint8_t *codes;
  const float *norm_w;  // fused RMSNorm of the input, or null
  float eps;
  uint32_t track_argmax;  // lm head: keep a per-CTA (max, index) candidate
  // Activations that cross CTAs inside a token live in "tagged" buffers: one 32-bit word per
  // element, fp16 value in the low half and the low 16 bits of the producing op's sequence
  // number in the high half. A reader that knows which op produced its input polls the words
  // until every tag matches: the data is its own arrival flag, so most ops need no grid barrier.
  const uint32_t *in;     // input vector [K], tagged words
  uint32_t src_op;        // index of the op that produced `in` (MK_ATTN_PART: of the op that produced q, k, v)
  uint32_t tag_op;        // index of the op whose tag this op's tagged results carry (its own, unless a skipped op is expected)
  uint32_t res_op;        // residual add (and all-reduce): index of the op that last wrote out_ll[0], whose tag the residual words carry
  uint32_t barrier_after; // a grid barrier follows this op (its results are not tagged, or the next op needs one)
  uint32_t *out_ll[3];    // tagged outputs; EPI_ADD: out_ll[0] is also the residual
  __half *out[3];         // plain fp16 outputs (lm head)
  float *out_f32;
  __half *kcache, *vcache;  // MK_ATTN_PART
};
// What one CTA reads of one op, in the order of the ops: its tiles' units, one range of memory, which the CTA's warps share
// out evenly. Or, with units == MEGA_KV_MARK, the K and V rows of an attention op: src is the layer's K cache, the V cache
// lies to_v * 256 bytes behind it, and the rows follow from the token's position.
struct alignas(16) MegaRun {
  const uint8_t *src;
  uint32_t units;
  int32_t to_v;
};
constexpr uint32_t MEGA_KV_MARK = 0xffffffffu;
// Where tile t of an op (of `tiles` tiles, dealt to a grid of `grid` CTAs as tile0 + lt * grid) sits in the
// op's weight stream: the tiles of one CTA are consecutive, CTAs in the order of their first tile.
__host__ __device__ inline uint32_t mega_stream_tile(uint32_t t, uint32_t tiles, uint32_t grid) {
  const uint32_t tile0 = t % grid, lt = t / grid, q = tiles / grid, r = tiles % grid;
  return tile0 * q + (tile0 < r ? tile0 : r) + lt;
}
constexpr uint32_t MEGA_UNIT_CODES = 1024, MEGA_UNIT_SCALES = 64;  // 32 rows x 32 codes, 32 fp16 scales
#ifndef VKL_MEGA_SU
#define VKL_MEGA_SU 4
#endif
#ifndef VKL_MEGA_NCW
#define VKL_MEGA_NCW 11
#endif
constexpr uint32_t MEGA_NCW = VKL_MEGA_NCW;  // warps of the kernel
constexpr uint32_t MEGA_SU = VKL_MEGA_SU;    // units per piece, the step of a warp's ring
constexpr uint32_t MEGA_MAX_NST = 8;         // pieces of a ring, at most
constexpr uint32_t MEGA_PIECE_BYTES = MEGA_SU * (MEGA_UNIT_CODES + MEGA_UNIT_SCALES);
// Splits per head at KV length L: as few as keep a split within `split_rows` cache rows. With one
// split a head needs no merge step between CTAs; more splits only pay when the rows of a head no
// longer stream through one SM fast enough.
__host__ __device__ inline uint32_t mega_splits(uint32_t L, uint32_t splits, uint32_t split_rows) {
  if (!split_rows) return splits;
  const uint32_t want = (L + split_rows - 1) / split_rows;
  return want < 1 ? 1u : (want < splits ? want : splits);
}
// The cached rows [c0, c1) that split `split` of `S` reads at KV length L.
__host__ __device__ inline void mega_kv_range(uint32_t L, uint32_t S, uint32_t split, uint32_t &c0, uint32_t &c1) {
  uint32_t chunk = (L + S - 1) / S;
  chunk = (chunk + 31) & ~31u;
  c0 = split * chunk < L ? split * chunk : L;
  c1 = c0 + chunk < L ? c0 + chunk : L;
}
// Shares. The `units` units that a CTA reads of an op (its tiles of `blocks` blocks, one behind the other) go to the warps in equal
// consecutive parts: warp w has those from mega_share_begin(units, w) to mega_share_begin(units, w + 1).
__host__ __device__ inline uint32_t mega_share_begin(uint32_t units, uint32_t w) { return units * w / MEGA_NCW; }
// A warp adds up each tile of its share by itself, in a place of its own per tile. The warps whose shares touch tile lt are first ..
// first + more (warps with an empty share among them count: their first place holds zeros), and the tile is the place-th that warp `first`
// touches and the first that the others do.
struct MegaTileShares {
  uint32_t first, more, place;
};
__host__ __device__ inline MegaTileShares mega_tile_shares(uint32_t units, uint32_t blocks, uint32_t lt) {
  const uint32_t ub = lt * blocks, first = (MEGA_NCW * (ub + 1) - 1) / units;
  return {first, (MEGA_NCW * (ub + blocks) - 1) / units - first, lt - mega_share_begin(units, first) / blocks};
}
// The most places that a warp needs of an op of `tiles` tiles.
__host__ __device__ inline uint32_t mega_red_slots(uint32_t tiles, uint32_t blocks, uint32_t grid) {
  const uint32_t tl = (tiles + grid - 1) / grid, share = (tl * blocks + MEGA_NCW - 1) / MEGA_NCW, most = (share + blocks - 2) / blocks + 1;
  return tl < most ? tl : most;
}
// The cached rows [r0, r0 + rows) of a split's [c0, c1) that warp w takes.
__host__ __device__ inline void mega_kv_share(uint32_t c0, uint32_t c1, uint32_t w, uint32_t &r0, uint32_t &rows) {
  const uint32_t each = (c1 - c0 + MEGA_NCW - 1) / MEGA_NCW, at = c0 + w * each;
  r0 = at < c1 ? at : c1;
  rows = each < c1 - r0 ? each : c1 - r0;
}
struct MegaParams {
  const MegaOp *ops;
  const MegaRun *runs;           // [grid][run_stride]: what every CTA reads, op by op
  const uint32_t *run_count;     // [grid]
  uint32_t run_stride;
  uint32_t nops, nbarriers;
  uint32_t *state;    // [0] position, [1] step, [2] picked id, [3] all-reduces done, [4] arg-max exchanges done,
                      // [5] number of forced (prompt) tokens, [6] prefill GEMM error, [7] sequence number of the next launch's first op
  const uint32_t *forced;  // prompt ids: while position+1 < state[5] the next input is forced[position+1]
  uint32_t *tok;      // current token id
  // A one-token call of a host-driven loop: position and token come with the launch (instead of state[0] and tok), and the output
  // layer writes its fp32 logits to page-locked host memory as well. Of the two words behind them CTA 0 sets the first to 0 when it
  // ends the launch, and any CTA with a wait that ran out sets the second to 1.
  uint32_t with_token, call_pos, call_tok;
  float *host_logits;
  uint32_t *out_ids;
  uint32_t out_cap;
  uint32_t f16;         // FP16 weights: units of 32 rows x 16 columns without scales (mega_pack_f16), embedding rows of halves
  const uint8_t *embd;  // token embedding, Q8_0 tiled planes (or rows of halves)
  uint32_t embd_rows;
  uint32_t *x, *q, *k, *v, *ao;  // tagged words (see MegaOp)
  const float *freqc, *freqs;
  float attn_scale;         // 1 / sqrt(head_dim)
  float *attn_scratch;      // heads*splits*(head_dim+4): per (head, split) the un-normalised P.V row, its max and its sum
  uint32_t attn_merge;      // how a head's split partials are merged: 0 combine op, 1 last-arriving split
  uint32_t *attn_counters;  // [heads] arrivals of a head's splits (the last one merges them), or null: separate combine op
  float *arg_scratch;       // grid*2
  unsigned long long *bar;  // [0] arrivals, [1] completed launches
  uint32_t *error;          // 0, or the code of the wait that timed out
  uint32_t dim, heads, head_dim, maxlen, splits, vocab;
  uint32_t xs_bytes;
  uint32_t xmax_blocks;  // largest K of any op, in blocks of 32 inputs: the input area holds that many blocks of digits
  // Tensor parallelism: every rank's exchange buffer (peer pointers, own included).
  // Layout of one buffer, in 4-byte words: partial sums [2 parities][tp][dim] x {fp32 sum, sequence number}, then
  // at word tp_flag_off: flags[16] (all-reduce sequence per source rank), arg flags[16],
  // arg candidates [16][2].
  uint32_t tp_rank, tp_size, tp_flag_off;
  void *tp_peer[8];
  uint32_t nst;               // pieces of a warp's ring (as many as fit beside the input and reduction areas)
  uint32_t red_slots;         // the most tiles that one warp's share of any op touches
  uint32_t split_rows;        // cache rows one attention split should hold: a token at KV length L uses min(splits, ceil(L / split_rows)) splits per head (0: always `splits`)
  uint32_t barrier_pollers;   // warps whose lane 0 polls the grid barrier counter, staggered in time
  // Optional timeline of CTA 0: per op, nanoseconds of work and of barrier wait.
  unsigned long long *timing;
  uint32_t timing_mode;  // third column of the timeline: 0 = ring wait, 1 = op prologue
  uint32_t sm_mhz;       // SM clock for the timeline's cycle counts (measured by the host before a profiled launch)
  uint32_t wait_limit;   // polls after which any wait of the kernel gives up and raises *error
};
size_t decode_mega_xs_bytes(uint32_t max_blocks, uint32_t head_dim);
// Packs up to three Q8_0 matrices (tiled planes) that share an input into one op's weight stream
// (layout and row rules at MegaOp). tiles = the stream's 32-row tiles.
cudaError_t launch_mega_pack(const uint8_t *const planes[3], uint32_t nmat, int swiglu, uint32_t N, uint32_t K, uint32_t tiles,
                             uint32_t grid, uint8_t *stream, cudaStream_t s);
cudaError_t launch_mega_pack_f16(const __half *const w[3], uint32_t nmat, int swiglu, uint32_t N, uint32_t K, uint32_t tiles, uint32_t grid, uint8_t *stream, cudaStream_t s);
size_t decode_mega_smem(size_t xs_bytes, uint32_t nst, uint32_t red_slots, uint32_t runs);
int decode_mega_max_k();
int decode_mega_max_stages();
cudaError_t decode_mega_occupancy(size_t smem_bytes, bool f16, bool tp, int *blocks_per_sm);  // of the instance that a launch takes
cudaError_t launch_decode_mega(const MegaParams &p, int grid, cudaStream_t s);

// ---- dense FP16 GEMM on tcgen05 tensor cores: C[M,N] = A[M,K] . W[N,K]^T (gemm_tcgen05.cu) ----
// One to three weight matrices of the same shape that share the input (queries, keys, values), each with an output of its
// own, or a gate and an up matrix whose results meet in the epilogue.
struct GemmParams {
  const __half *a;            // [M,K] row-major
  const __half *w[3];         // [N,K] row-major (a transposed-weight matrix of the reference); FP16 weights
  const uint8_t *w_codes[3];  // Q8_0 weights [N,K] as tiled planes (common.cuh): codes ...
  const uint8_t *w_scales[3]; // ... and scales
  __half *wide;               // Q8_0: room for the nmat matrices in fp16 (gemm_q8_wide), or null (operators; a device without room)
  __half *c[3];               // [M,N] fp16 output, or nullptr when c_f32 is set
  uint32_t nmat;
  int swiglu;                 // c[0] = fp16(silu(gate) * up) of the fp32 products with w[0] (gate) and w[1] (up): the
                              // rounding of ffn_up_and_gate_fp16.comp; scale, bias, act and residual are not used
  float *c_f32;               // raw fp32 output of w[0] (partial sums of a sharded projection)
  const __half *residual;     // optional [M,N]: c = fp16(fp16(acc) + residual)
  uint32_t *error;            // device word raised when a bounded wait ran out
  uint32_t M, N, K;
  float scale, bias;          // MatMul's scale and bias (mat_mul.cpp:39-41)
  int act;                    // 0 none, 1 SiLU
};
// The same by pairs of CTAs (gemm_pair.cu); bn: columns of W per tile, 128 or 256. Operands as checked by the caller.
cudaError_t launch_gemm_pair_f16(const GemmParams &p, int bn, cudaStream_t s);
constexpr uint32_t GEMM_MIN_ROWS = 32;  // below this launch_matvec (skinny_gemm.cuh or the mat-vec kernel)
bool gemm_tcgen05_supported(uint32_t M, uint32_t N, uint32_t K);
cudaError_t launch_gemm_f16_tcgen05(const GemmParams &p, cudaStream_t s);
// The same GEMM with Q8_0 weights (w_codes / w_scales), dequantised into the shared-memory tiles.
constexpr uint32_t GEMM_Q8_MIN_ROWS = 64;  // below this launch_matvec, whose kernels keep the exact fp32 scaling
cudaError_t launch_gemm_q8_tcgen05(const GemmParams &p, cudaStream_t s);
// Whether the Q8_0 matrices are turned into fp16 once, in GemmParams::wide, and multiplied as such.
bool gemm_q8_wide(uint32_t M);
inline uint32_t gemm_launches(const GemmParams &p) { return !p.w[0] && p.wide && gemm_q8_wide(p.M) ? 2 : 1; }
// Rows from which a weight of this kind goes to the tensor-core GEMM.
inline uint32_t gemm_min_rows(bool q8) { return q8 ? GEMM_Q8_MIN_ROWS : GEMM_MIN_ROWS; }
// Dispatch on the weight kind: w[0] set = FP16 weights, else w_codes / w_scales = Q8_0.
inline cudaError_t launch_gemm_tcgen05(const GemmParams &p, cudaStream_t s) { return p.w[0] ? launch_gemm_f16_tcgen05(p, s) : launch_gemm_q8_tcgen05(p, s); }

}  // namespace vkl
