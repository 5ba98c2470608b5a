// A CUDA runtime for the host side of the library alone: memory is host
// memory, copies happen at once, and a launch is looked at instead of run.
// Linked with the library's objects in place of the runtime, it lets the host
// code (layouts, tuners, scratch, order of calls) be tested without a GPU.
//
// Looked at, for every launch: shared memory against the kernel's limit (48 KB
// of static and dynamic memory together, unless the limit was raised), and for
// the solves the scratch that the layout reaches.  A solve also leaves its
// number where it would write: in its potential and field, and in the report.
#include <cuda_runtime.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "cupic_internal.cuh"
#include "kernels.h"

using namespace cupic;

namespace {

constexpr size_t kDefaultSmem = 48 * 1024;
constexpr size_t kStaticSmem = 720;  // of every kernel
constexpr int kSms = 152, kMaxSmem = 232448;

struct Kernel {
  std::string name;
  size_t dyn = kDefaultSmem - kStaticSmem;  // largest dynamic shared memory
};

std::recursive_mutex mu;
std::map<const char *, size_t> blocks;  // allocations: start, bytes
std::map<const void *, Kernel> kernels;
std::map<const void *, std::pair<void *, size_t>> symbols;
std::vector<std::string> faults;
std::vector<std::string> launches;  // names, in order, with those captured
bool capturing = false;
int give_up_ctas = -1, give_up_depth = -1, batch_give_up = -1;
float last_ms = 1.0f;
int solves = 0;
// while watched: where exchange words and where counters of any launch lay
bool watching = false;
std::vector<std::pair<const char *, size_t>> words, counters;
size_t allocated = 0;

void fault(const std::string &s) { faults.push_back(s); }

// bytes from p to the end of its allocation; 0 outside of any
size_t room(const void *p) {
  const char *q = static_cast<const char *>(p);
  auto it = blocks.upper_bound(q);
  if (it == blocks.begin()) return 0;
  --it;
  return q < it->first + it->second ? (size_t)(it->first + it->second - q) : 0;
}

void *take(size_t n) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  char *p = static_cast<char *>(aligned_alloc(256, (n + 511) / 256 * 256));
  memset(p, 0x5a, n);
  blocks[p] = n;
  allocated += n;
  return p;
}

void give(void *p) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (!p) return;
  if (!blocks.count(static_cast<char *>(p))) return fault("free of no allocation");
  blocks.erase(static_cast<char *>(p));
  free(p);
}

void need(const char *what, const void *p, size_t bytes, const std::string &who) {
  if (room(p) < bytes)
    fault(who + ": " + what + " needs " + std::to_string(bytes) + " bytes, has " + std::to_string(room(p)));
}

void apart(std::vector<std::pair<const char *, size_t>> *mine, const std::vector<std::pair<const char *, size_t>> &others,
           const void *p, size_t n, const std::string &who) {
  const char *q = static_cast<const char *>(p);
  mine->push_back({q, n});
  for (const auto &o : others)
    if (q < o.first + o.second && o.first < q + n) return fault(who + ": exchange words and counters in one place");
}

void solve(const std::string &name, const SimArgs &a, const JacobiArgs &J, dim3 grid, size_t smem) {
  const std::string who = name + " " + std::to_string(a.nnx - 1) + "x" + std::to_string(a.nny - 1) + " G=" +
                          std::to_string(J.G) + " K=" + std::to_string(J.depth);
  const bool tile = name.find("k_tile") != std::string::npos;
  const int M = a.nny - 2;
  const size_t G = J.G, K = J.depth;
  if ((int)grid.x != J.G) fault(who + ": grid");
  if (tile) {
    if (J.G > 1 && !J.near) need("halo", J.halo, 2 * (size_t)J.pwords * 8, who);
    need("gmax", J.gmax, 128 * 8, who);
    need("tbar", J.tbar, 4 * 4, who);
  } else if (J.G > 1) {
    need("flags", J.flags, (G + 1) * 4, who);
    need("bar", J.bar, 4, who);
    need("res", J.res_cta, 2 * G * 4, who);
    need("halo", J.halo, 4 * G * K * J.pitch * 8, who);
    if (K < 1 || (int)K > M / J.G) fault(who + ": blocks own fewer rows than the depth");
  }
  if (!tile) {
    if (J.rows_per_cta < (M + J.G - 1) / J.G) fault(who + ": rows of a block");
    if (smem < jacobi_smem_bytes(J.rows_per_cta, J.G > 1 ? J.depth : 1, J.pitch)) fault(who + ": shared memory");
  }
  if (watching) {
    if (J.G > 1 && !(tile && J.near))
      apart(&words, counters, J.halo, tile ? 2 * (size_t)J.pwords * 8 : 4 * G * K * J.pitch * 8, who);
    if (J.G > 1 && !tile) {
      apart(&counters, words, J.flags, (G + 1) * 4, who);
      apart(&counters, words, J.res_cta, 2 * G * 4, who);
    }
    if (tile) apart(&counters, words, J.gmax, 130 * 8, who);
  }
  if (capturing) return;
  const size_t nodes = (size_t)a.nnx * a.nny;
  const float mark = (float)++solves;
  float *phi = J.phi ? J.phi : a.phi;
  need("phi", phi, nodes * 4, who);
  if (room(phi) >= nodes * 4) std::fill(phi, phi + nodes, mark);
  if (J.do_field) {
    need("E", a.E, nodes * 8, who);
    if (room(a.E) >= nodes * 8) std::fill(a.E, a.E + nodes, make_float2(mark, mark));
  }
  if (J.r64_phi) {
    need("phi64", J.r64_phi, nodes * 8, who);
    if (room(J.r64_phi) >= nodes * 8) std::fill(J.r64_phi, J.r64_phi + nodes, (double)mark);
  }
  if (J.write_stats || J.r64_stats) a.ctl->sweeps = solves;
  const bool gives_up = J.G == give_up_ctas && J.depth == give_up_depth;
  if (a.ctl->abort && !gives_up) fault(who + ": begins with the flag of another that gave up");
  last_ms = a.ctl->abort || gives_up ? 1e-3f : 1.0f;
  if (gives_up) {
    a.ctl->abort = 1;
    a.ctl->step_flags |= CUPIC_FLAG_TIMEOUT;
  }
}

cudaError_t launch(const void *fn, dim3 grid, dim3 block, void **args, size_t smem) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  const Kernel &k = kernels[fn];
  launches.push_back(k.name);
  if (block.x * block.y * block.z > 1024 || grid.x < 1) return cudaErrorInvalidConfiguration;
  if (smem > k.dyn) {
    fault(k.name + ": " + std::to_string(smem) + " bytes of shared memory refused");
    return cudaErrorInvalidValue;
  }
  if (k.name.find("k_tile") != std::string::npos ||
      (k.name.find("k_jacobi") != std::string::npos && k.name.find("batch") == std::string::npos))
    solve(k.name, *static_cast<const SimArgs *>(args[0]), *static_cast<const JacobiArgs *>(args[1]), grid, smem);
  if (k.name.find("k_jacobi_batch") != std::string::npos && !capturing) {
    const SimArgs *inst = *static_cast<const SimArgs *const *>(args[0]);
    const int n = (int)(room(inst) / sizeof(SimArgs));
    last_ms = 1.0f;
    for (int i = 0; i < n; ++i)
      if (inst[i].ctl->abort) last_ms = 1e-3f;
    if (batch_give_up >= 0 && batch_give_up-- == 0) inst[n - 1].ctl->abort = 1;
  }
  return cudaSuccess;
}

}  // namespace

extern "C" {

// ---- what the tests ask for -----------------------------------------------
int fake_faults(char *text, int n) {
  std::string all;
  for (const std::string &s : faults) all += s + "\n";
  if (n > 0) {
    strncpy(text, all.c_str(), n - 1);
    text[n - 1] = 0;
  }
  return (int)faults.size();
}
int fake_launches(const char *name) {
  int n = 0;
  for (const std::string &s : launches) n += s.find(name) != std::string::npos;
  return n;
}
unsigned long long fake_allocated() { return allocated; }
// the solves of this layout give up, fast
void fake_give_up(int ctas, int depth) {
  give_up_ctas = ctas;
  give_up_depth = depth;
}
// the n-th batched solve from now gives up, in its last member
void fake_batch_give_up(int n) { batch_give_up = n; }
void fake_watch() {
  watching = true;
  words.clear();
  counters.clear();
}
void fake_reset() {
  watching = false;
  faults.clear();
  launches.clear();
  give_up_ctas = give_up_depth = batch_give_up = -1;
  allocated = 0;
}
void *fake_alloc(unsigned long long n) { return take(n); }
// raise_dyn_smem of some kernel; the dynamic shared memory it may have then
unsigned long long fake_raise(unsigned long long bytes) {
  static const char any = 0;
  kernels[&any] = Kernel{};
  return raise_dyn_smem(&any, bytes) == cudaSuccess ? kernels[&any].dyn : 0;
}

// ---- the runtime ------------------------------------------------------------
void **__cudaRegisterFatBinary(void *) {
  static void *h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *fn, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
  kernels[fn].name = name;
}
void __cudaRegisterVar(void **, char *var, char *, const char *, int, size_t n, int, int) { symbols[var] = {nullptr, n}; }
static dim3 g_grid, g_block;
static size_t g_smem;
// (declared for device code too under its own name)
unsigned fake_push(dim3 grid, dim3 block, size_t smem, CUstream_st *) __asm__("__cudaPushCallConfiguration");
unsigned fake_push(dim3 grid, dim3 block, size_t smem, CUstream_st *) {
  g_grid = grid;
  g_block = block;
  g_smem = smem;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *st) {
  *grid = g_grid;
  *block = g_block;
  *smem = g_smem;
  *static_cast<void **>(st) = nullptr;
  return cudaSuccess;
}
static cudaError_t g_last = cudaSuccess;
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fn) {
  *k = (cudaKernel_t)fn;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t) {
  return g_last = launch((const void *)k, grid, block, args, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *fn, void **args) {
  return g_last = launch(fn, c->gridDim, c->blockDim, args, c->dynamicSmemBytes);
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaFuncSetAttribute(const void *fn, cudaFuncAttribute at, int v) {
  if (at != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
  if (v + kStaticSmem > (size_t)kMaxSmem) return cudaErrorInvalidValue;
  kernels[fn].dyn = v;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *at, const void *fn) {
  memset(at, 0, sizeof(*at));
  at->sharedSizeBytes = kStaticSmem;
  at->maxDynamicSharedSizeBytes = (int)kernels[fn].dyn;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *fn, int, size_t smem) {
  *n = smem <= kernels[fn].dyn ? 1 : 0;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *fn, int b, size_t smem, unsigned) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, fn, b, smem);
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *fn, const cudaLaunchConfig_t *c) {
  *n = c->dynamicSmemBytes <= kernels[fn].dyn ? 1 : 0;
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) {
  *p = take(n);
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { return cudaMallocAsync(p, n, nullptr); }
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaMallocAsync(p, n, nullptr); }
cudaError_t cudaFree(void *p) {
  give(p);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaGetSymbolAddress(void **p, const void *var) {
  auto &s = symbols[var];
  if (!s.first) {
    s.first = take(s.second);
    memset(s.first, 0, s.second);
  }
  *p = s.first;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
  if (capturing) return cudaSuccess;
  if (room(p) < n) {
    fault("memset of " + std::to_string(n) + " bytes, has " + std::to_string(room(p)));
    return cudaErrorInvalidValue;
  }
  memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) { return cudaMemsetAsync(p, v, n, nullptr); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind kind, cudaStream_t) {
  if (capturing) return cudaSuccess;
  if ((kind != cudaMemcpyDeviceToHost && room(d) < n) || (kind != cudaMemcpyHostToDevice && room(s) < n)) {
    fault("copy of " + std::to_string(n) + " bytes past an allocation");
    return cudaErrorInvalidValue;
  }
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind kind) {
  return cudaMemcpyAsync(d, s, n, kind, nullptr);
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *at, const void *) {
  memset(at, 0, sizeof(*at));
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int *n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr at, int) {
  *v = at == cudaDevAttrMultiProcessorCount ? kSms : at == cudaDevAttrMaxSharedMemoryPerBlockOptin ? kMaxSmem : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int) {
  *p = nullptr;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *v) {
  *static_cast<uint64_t *>(v) = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t)take(1);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return cudaFree(s); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = (cudaEvent_t)take(1);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return cudaFree(e); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = last_ms;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  capturing = true;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  capturing = false;
  *g = (cudaGraph_t)take(1);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
  *e = (cudaGraphExec_t)take(1);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return cudaFree(g); }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { return cudaFree(g); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }

}  // extern "C"
