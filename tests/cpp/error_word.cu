// Reaches the private error words that kernels raise when a bounded wait runs out, so that a test can raise one from the host.
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
