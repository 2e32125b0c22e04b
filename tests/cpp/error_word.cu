// Reaches private parts of the library's objects for tests: the error words that kernels raise when a bounded wait runs out, so
// that one can be raised from the host, the bound of the decode kernel's waits, a layer's cache.
#include "model.h"

extern "C" int raise_model_word(vkl_model *m) {
  const uint32_t one = 1;
  return (int)cudaMemcpy((uint32_t *)m->state->data() + 6, &one, 4, cudaMemcpyHostToDevice);
}
extern "C" int command_is_watched(vkl_command *cmd) { return cmd->err_used; }
extern "C" int raise_command_word(vkl_command *cmd) {
  const uint32_t one = 1;
  return (int)cudaMemcpy(cmd->err_word, &one, 4, cudaMemcpyHostToDevice);
}
// The decode kernel's waits give up after so many polls from now on; the word that they raise then.
extern "C" void set_polls(vkl_model *m, uint32_t polls) { m->mp.wait_limit = polls; }
extern "C" uint32_t decode_word(vkl_model *m) {
  uint32_t w = 0;
  return cudaMemcpy(&w, m->mp.error, 4, cudaMemcpyDeviceToHost) == cudaSuccess ? w : ~0u;
}
// The layer's V cache 128 bytes into a new allocation. (The old one and the new allocation are left to the process's end.)
extern "C" int shift_v_cache(vkl_model *m, uint32_t layer) {
  vkl_tensor *old = m->L[layer].vcache, *t = new vkl_tensor();
  const size_t bytes = old->c * old->cs;
  void *p = nullptr;
  const cudaError_t e = cudaMalloc(&p, bytes + 256);
  if (e != cudaSuccess) return (int)e;
  t->dev = old->dev;
  t->dtype = old->dtype;
  t->c = old->c, t->h = old->h, t->w = old->w;
  t->cs = old->cs, t->hs = old->hs, t->ws = old->ws;
  t->buf = std::shared_ptr<vkl::Buffer>(new vkl::Buffer(old->dev, (uint8_t *)p + 128, bytes), [](vkl::Buffer *) {});
  m->L[layer].vcache = t;
  return (int)cudaMemset(t->data(), 0, bytes);
}
