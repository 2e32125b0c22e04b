// Reaches the private error words that kernels raise when a bounded wait runs out, so that a test can raise one from the host, and their bound.
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
