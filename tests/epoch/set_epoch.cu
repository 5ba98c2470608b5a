// The library with a way to move the epoch base of the halo words, which counts
// up over all solves and starts over after some 3e9 exchanges.
#include "noalloc.cu"

#include "ctx.h"

using namespace cupic;

extern "C" int set_epoch(cupic_ctx *c, unsigned v) {
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) return 1;
  return cudaMemcpy(&c->ctl->jepoch, &v, sizeof(v), cudaMemcpyHostToDevice) != cudaSuccess;
}

extern "C" int get_epoch(cupic_ctx *c, unsigned *v) {
  return cudaMemcpy(v, &c->ctl->jepoch, sizeof(*v), cudaMemcpyDeviceToHost) != cudaSuccess;
}

static Ctl *static_ctl() {
  void *p = nullptr;
  return cudaGetSymbolAddress(&p, g_solver_scratch) == cudaSuccess ? static_cast<Ctl *>(p) : nullptr;
}

extern "C" int set_static_epoch(unsigned v) {
  return cudaMemcpy(&static_ctl()->jepoch, &v, sizeof(v), cudaMemcpyHostToDevice) != cudaSuccess;
}

extern "C" int get_static_epoch(unsigned *v) {
  return cudaMemcpy(v, &static_ctl()->jepoch, sizeof(*v), cudaMemcpyDeviceToHost) != cudaSuccess;
}
