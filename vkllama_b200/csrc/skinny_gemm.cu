// Q8_0 kernels of skinny_gemm.cuh, and which launches it takes.
#include "skinny_gemm.cuh"

namespace vkl {

cudaError_t launch_skinny_gemm_f16(const MvParams &p, int epilogue, cudaStream_t s);  // skinny_gemm_f16.cu

// Tensor copies want rows of X (and of FP16 weights) that follow each other on 16-byte boundaries; whole 32-column blocks, so
// that no fragment reaches beyond K.
//
// Where it pays: the mat-vec kernel fetches X per 16-row tile, which costs little while the launch is small; here a CTA alone on
// its SM starts and reduces bare. us, mat-vec / here, weights from HBM, 17 rows of Q8_0 unless said (q: three D x D matrices, o: D x D,
// g: gate and up 2.7 D x D):
//   o   D = 512 3.4 / 4.3   1024 3.7 / 5.4   2048 5.6 / 6.9    2304 7.8 / 7.5    4096 11.6 / 10.5;  33 rows: 1024 5.6 / 6.7, 1408 8.5 / 7.4
//   q   D = 1024 4.2 / 5.5  2048 11.0 / 12.5  2304 14.9 / 13.7  5120 47.9 / 38.0;  33 rows: 704 5.3 / 6.4, 1024 9.7 / 6.9;  FP16: 1024 4.9 / 5.7, 1408 7.0 / 6.7
//   g   D = 704 4.9 / 5.2, 1024 8.3 / 9.3, any other 0.70 ... 0.95 of the time, 33 rows 0.44 ... 0.85;  up to 16 rows: Q8_0 up to 1.27, FP16 1664 9.5 / 11.5, 2048 16.8 / 14.9
// Gate and up of less than 6 million weights gain 1 us here (2 from 33 rows on, to 1.6 million), and the error word, which only this kernel needs, costs
// a call 4 us.
// So a launch needs as many weights as the lines below say. Over the four launches of a block, widths 128 to 5120, 9 to 63 rows, that is
// 0.38 to 1.00 of the mat-vec kernel's time (a rule by rows alone: up to 1.29 at widths 512 to 1024).
bool skinny_gemm_takes(const MvParams &p, int epilogue) {
  uintptr_t a = reinterpret_cast<uintptr_t>(p.x);
  if (p.fp16_weights)
    for (uint32_t i = 0; i < 3; ++i) a |= reinterpret_cast<uintptr_t>(p.codes[i]);
  if (p.M <= 8 || p.M > 64 || p.K % 32 || p.x_ld != p.K || (a & 15) || p.norm_w) return false;
  const bool swiglu = epilogue == EPI_SWIGLU, few = p.M <= kFewRows, half = p.M <= 32;
  const size_t tiles = (swiglu ? 2 : p.nmat) * (size_t)((p.N + 15) / 16), weights = tiles * 16 * p.K;
  // 16 rows of Q8_0: a second wave of CTAs that is a third full is too much already (us: 402 tiles of K = 2304 9.4 / 10.2, 320 of 5120 20.9 / 16.9)
  if (!p.fp16_weights && few && (swiglu || p.nmat > 1 || 2 * tiles > 5 * sm_count())) return false;
  if (swiglu) return weights >= (few ? 20000000u : half ? 6000000u : 1600000u);
  if (p.nmat > 1) return weights >= (!half ? 2000000u : !p.fp16_weights ? 15000000u : few ? 25000000u : 5000000u);
  return weights >= (half ? 5000000u : 1600000u);
}
cudaError_t launch_skinny_gemm(const MvParams &p, int epilogue, cudaStream_t s) {
  return p.fp16_weights ? launch_skinny_gemm_f16(p, epilogue, s) : launch_kind<true>(p, epilogue, s);
}

}  // namespace vkl
