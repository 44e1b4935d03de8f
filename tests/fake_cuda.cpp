// A CUDA runtime without a device, for tests of libswave's host code on the
// CPU: device memory is host memory (small numbers when allocated), copies and
// sets are done at once, kernels are recorded and do nothing, and the test
// decides what fails.  Linked with libswave's own objects in place of cudart.
//
// k_onchip2d is checked as it is launched: its CTAs take a border packet when
// it carries the epoch of the step, so no packet that is in the inbox before
// the launch may carry an epoch of the launch.  The fake then leaves the
// launch's own epochs in half of it (a launch does not use every slot).
#include <cuda_runtime.h>
#include <cuda.h>

#include <unistd.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "../seismic_gb300/csrc/engine.h"

namespace {

struct Launch {
  std::string name;
  dim3 grid, block;
  bool coop;
};
// As OcArgs of onchip2d.cuh.
struct OcArgsView {
  const void *shots, *oc, *tiles;
  uint32_t *inbox;   // 64-bit halves {value, epoch}
  int cap, s0, s1;
  unsigned epoch0;
};

// Kernels by their host stub (filled while the library's objects start up).
std::map<const void *, std::string> &names() {
  static std::map<const void *, std::string> m;
  return m;
}
std::map<void *, size_t> mem;
std::vector<Launch> launches;
std::string report;
struct Call { dim3 g, b; size_t smem; cudaStream_t s; };
std::vector<Call> calls;
cudaError_t last = cudaSuccess;
size_t limit = size_t(8) << 30, used = 0;
int fail_alloc = -1;      // that many more allocations succeed, then one fails
int blocks_per_sm = 2, coop_error = 0, stale = 0;
bool capturing = false;

cudaError_t ret(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}

cudaError_t launch(const void *f, dim3 g, dim3 b, void **args, bool coop) {
  if (g.x < 1 || g.y < 1 || g.z < 1 || g.x > 0x7fffffffu || g.y > 65535 || g.z > 65535 ||
      b.x * b.y * b.z < 1 || b.x * b.y * b.z > 1024)
    return ret(cudaErrorInvalidConfiguration);
  const std::string n = names().count(f) ? names()[f] : "?";
  if (coop) {
    if (coop_error) return ret((cudaError_t)coop_error);
    if ((int)g.x > 152 * blocks_per_sm) return ret(cudaErrorCooperativeLaunchTooLarge);
    const OcArgsView &A = *(const OcArgsView *)args[0];
    const uint64_t first = (uint64_t)A.epoch0 + 1, end = (uint64_t)A.epoch0 + (A.s1 - A.s0);
    const size_t words = (size_t)g.x * 8 * A.cap * 4;
    for (size_t q = 1; q < words; q += 2) {
      const uint64_t e = A.inbox[q];
      if ((e >= first && e <= end) || (end >> 32 && e <= (end & 0xffffffffu))) ++stale;
    }
    for (size_t q = 1; q < words; q += 4) A.inbox[q] = (uint32_t)(end - (q / 4) % 2);
  }
  launches.push_back({n, g, b, coop});
  return cudaSuccess;
}

CUresult encode(CUtensorMap *m, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  std::memset(m, 0, sizeof(*m));
  return CUDA_SUCCESS;
}

}  // namespace

extern "C" {

// ---- what the test sets and reads ----
void fake_reset(size_t mem_limit) {
  launches.clear();
  limit = mem_limit;
  fail_alloc = -1;
  blocks_per_sm = 2;
  coop_error = stale = 0;
  last = cudaSuccess;
}
void fake_fail_alloc(int after) { fail_alloc = after; }
void fake_blocks_per_sm(int n) { blocks_per_sm = n; }
void fake_coop_error(int e) { coop_error = e; }
int fake_stale() { return stale; }
size_t fake_used() { return used; }
void fake_set_epoch(sw_ctx *c, unsigned e) { c->oc_epoch = e; }
unsigned fake_epoch(const sw_ctx *c) { return c->oc_epoch; }
// Every launch as "name grid.x grid.y grid.z coop" lines.
const char *fake_launches() {
  report.clear();
  for (auto &l : launches)
    report += l.name + " " + std::to_string(l.grid.x) + " " + std::to_string(l.grid.y) + " " +
              std::to_string(l.grid.z) + " " + std::to_string(l.coop) + "\n";
  return report.c_str();
}

// ---- what nvcc's host code calls ----
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *,
                            uint3 *, dim3 *, dim3 *, int *) {
  names()[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
  calls.push_back({g, b, smem, s});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
  *g = calls.back().g;
  *b = calls.back().b;
  *smem = calls.back().smem;
  *(cudaStream_t *)s = calls.back().s;
  calls.pop_back();
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void **args, size_t, cudaStream_t) {
  return launch((const void *)k, g, b, args, false);
}

// ---- the runtime ----
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
  return launch(f, c->gridDim, c->blockDim, args, false);
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **args, size_t,
                                        cudaStream_t) {
  return launch(f, g, b, args, true);
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
  *n = blocks_per_sm;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
  const bool refuse = fail_alloc == 0;
  if (fail_alloc >= 0) --fail_alloc;
  if (refuse || used + n > limit) return ret(cudaErrorMemoryAllocation);
  *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
  for (size_t q = 0; q < n / 4; ++q) ((uint32_t *)*p)[q] = q % 1021;
  mem[*p] = n;
  used += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (!p) return cudaSuccess;
  used -= mem[p];
  mem.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  *f = limit > used ? limit - used : 0;
  *t = limit;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h,
                              cudaMemcpyKind, cudaStream_t) {
  for (size_t q = 0; q < h; ++q) std::memcpy((char *)d + q * dp, (const char *)s + q * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) {
  *p = const_cast<void *>(s);
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **p, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *r) {
  usleep(200000);   // a slow lookup: a second thread asks meanwhile
  *p = (void *)encode;
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t)std::malloc(1);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = true; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  capturing = false;
  *g = (cudaGraph_t)std::malloc(1);
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
  *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
  *x = (cudaGraphExec_t)std::malloc(1);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
  launches.push_back({"graph", dim3(1), dim3(1), false});
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { std::free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { std::free(x); return cudaSuccess; }

}  // extern "C"
