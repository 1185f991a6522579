// A CUDA runtime on host memory for the CPU tests of the library's host code: "device" memory is host
// memory, kernels do nothing, and what a stream was given runs when the stream is waited for, as late as
// CUDA allows. It records what the host code does wrong on the way ("faults"): a source of an
// asynchronous copy that changed or was freed before the copy ran, and batch pair launches whose work
// tables do not fit the members' buffers. Any call can be made to fail.
#include <malloc.h>
#include <stdlib.h>
#include <string.h>
#include <functional>
#include <map>
#include <set>
#include <string>
#include <vector>
#include "od_internal.h"

namespace {
using op = std::function<void()>;
struct graph_t { std::vector<op> ops; std::string kernels; };
struct stream_t { std::vector<op> ops; graph_t* capture = nullptr; };
struct call_t { dim3 grid, block; size_t smem; cudaStream_t s; };

stream_t g_legacy;
std::set<stream_t*> g_streams = {&g_legacy};
std::map<char*, size_t> g_blocks;            // device allocations
std::vector<std::string> g_faults;
std::string g_log;                           // the calls made and, indented, the kernels launched
std::map<std::string, int> g_fail;           // call -> successful calls left before it fails once
std::vector<call_t> g_calls;
cudaError_t g_last = cudaSuccess;
std::string g_poke;                          // kernel whose pointer argument g_poke_arg gets g_poke_bits
int g_poke_arg = 0;
uint32_t g_poke_bits = 0, g_member_bits = 0;  // g_member_bits: error word of a batch's first member

// function-local: the kernels register themselves before this file's globals are built
std::map<const void*, std::string>& kernels() {
  static std::map<const void*, std::string> m;
  return m;
}
stream_t& st(cudaStream_t s) { return s ? *reinterpret_cast<stream_t*>(s) : g_legacy; }
void put(cudaStream_t s, op f) {
  stream_t& q = st(s);
  (q.capture ? q.capture->ops : q.ops).push_back(std::move(f));
}
void run(stream_t& q) {
  std::vector<op> ops;
  ops.swap(q.ops);
  for (op& f : ops) f();
}
cudaError_t call(const char* name, cudaError_t what = cudaErrorUnknown) {
  g_log += std::string(name) + "\n";
  auto it = g_fail.find(name);
  if (it == g_fail.end() || it->second-- > 0) return cudaSuccess;
  g_fail.erase(it);
  return g_last = what;
}
// device bytes from p to the end of its allocation
size_t room(const void* p) {
  auto it = g_blocks.upper_bound((char*)p);
  if (it == g_blocks.begin()) return 0;
  --it;
  const char* end = it->first + it->second;
  return (char*)p < end ? end - (char*)p : 0;
}
void fault(const std::string& s) { g_faults.push_back(s); }

void check_directed(const od_simdesc* sims, const int4* items, int n) {
  for (int k = 0; k < n; k++) {
    const od_simdesc& d = sims[items[k].x];
    const size_t need = sizeof(float4) * (size_t)d.jsplit * d.Npad;
    if (room(d.b.part_hi) < need || room(d.b.part_lo) < need) {
      fault("directed batch launch past the partial-sum slabs");
      return;
    }
  }
}
void check_once(const od_simdesc* sims, const int2* items, int n, int targets) {
  const int sources = targets == 8 ? 2 : targets;
  for (int k = 0; k < n; k++) {
    const od_simdesc& d = sims[items[k].x];
    const long long NG = d.Npad / (32 * targets), NS = d.Npad / (32 * sources), R = targets / sources;
    if (d.n3.pairs != NG * NS - R * (NG * (NG - 1) / 2)) {
      fault("each-pair-once batch launch with the group pairs of another shape");
      return;
    }
  }
}

cudaError_t launch(const std::string& name, dim3 grid, void** args, cudaStream_t s) {
  const cudaError_t e = call("launch", cudaErrorLaunchFailure);
  if (e != cudaSuccess) return e;
  (st(s).capture ? st(s).capture->kernels : g_log) += "  " + name + "\n";
  if (!g_poke.empty() && name.find(g_poke) != std::string::npos) {
    uint32_t* p = *(uint32_t**)args[g_poke_arg];
    const uint32_t bits = g_poke_bits;
    put(s, [p, bits] { *p |= bits; });
  }
  const size_t once = name.find("12k_b_pairs_n3ILi");
  if (name.find("11k_kick_flagE") != std::string::npos) {  // K3 reads part_hi, part_lo
    const float4 *ph = *(const float4**)args[4], *pl = *(const float4**)args[5];
    const size_t need = sizeof(float4) * *(int*)args[6];
    put(s, [=] { if (room(ph) < need || room(pl) < need) fault("no partial sums to take"); });
  }
  if (name.find("9k_b_pairsE") != std::string::npos) {
    const od_simdesc* sims = *(const od_simdesc**)args[0];
    const int4* items = *(const int4**)args[1];
    const int n = *(int*)args[2];
    put(s, [=] { check_directed(sims, items, n); });
  } else if (once != std::string::npos) {
    const od_simdesc* sims = *(const od_simdesc**)args[0];
    const int2* items = *(const int2**)args[1];
    const int n = (int)grid.x, targets = atoi(name.c_str() + once + 17);
    put(s, [=] { check_once(sims, items, n, targets); });
  } else if (name.find("10k_b_errors") != std::string::npos) {
    const od_simdesc* sims = *(const od_simdesc**)args[0];
    const int n = *(int*)args[1];
    uint32_t* err = *(uint32_t**)args[2];
    put(s, [=] {
      if (n > 0) sims[0].ds->err |= g_member_bits;
      g_member_bits = 0;
      err[1] = 0u;
      for (int m = 0; m < n; m++) err[1] |= sims[m].ds->err;
    });
  }
  return cudaSuccess;
}
}  // namespace

extern "C" {
// ------------------------------------------------------------------ controls of the tests
void fake_reset() {
  g_faults.clear();
  g_log.clear();
  g_fail.clear();
  g_poke.clear();
  g_member_bits = 0;
  g_last = cudaSuccess;
  mallopt(M_PERTURB, 0x5a);  // freed memory is overwritten at once
}
void fake_fail(const char* name, int after) { g_fail[name] = after; }
void fake_poke(const char* kernel, int arg, uint32_t bits) {
  g_poke = kernel; g_poke_arg = arg; g_poke_bits = bits;
}
void fake_member_error(uint32_t bits) { g_member_bits = bits; }
const char* fake_log() { return g_log.c_str(); }
const char* fake_faults() {
  static std::string all;
  all.clear();
  for (const std::string& f : g_faults) all += f + "\n";
  return all.c_str();
}

// ------------------------------------------------------------------ registration and launches
void** CUDARTAPI __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void CUDARTAPI __cudaRegisterFatBinaryEnd(void**) {}
void CUDARTAPI __cudaUnregisterFatBinary(void**) {}
void CUDARTAPI __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void CUDARTAPI __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*,
                                      uint3*, dim3*, dim3*, int*) {
  kernels()[host] = name;
}
unsigned CUDARTAPI __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, CUstream_st* s) {
#ifndef __CUDA_ARCH__  // nvcc declares this one for both sides
  g_calls.push_back({g, b, m, s});
#endif
  return 0;
}
cudaError_t CUDARTAPI __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
  const call_t c = g_calls.back();
  g_calls.pop_back();
  *g = c.grid; *b = c.block; *m = c.smem; *(cudaStream_t*)s = c.s;
  return cudaSuccess;
}
cudaError_t CUDARTAPI __cudaGetKernel(cudaKernel_t* k, const void* host) {
  *k = (cudaKernel_t)host;
  return cudaSuccess;
}
cudaError_t CUDARTAPI __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3, void** args, size_t,
                                         cudaStream_t s) {
  return launch(kernels()[(const void*)k], g, args, s);
}
cudaError_t CUDARTAPI cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* host, void** args) {
  return launch(kernels()[host], c->gridDim, args, c->stream);
}

// ------------------------------------------------------------------ memory
cudaError_t CUDARTAPI cudaMalloc(void** p, size_t n) {
  const cudaError_t e = call("cudaMalloc", cudaErrorMemoryAllocation);
  if (e != cudaSuccess) return e;
  *p = aligned_alloc(256, (n + 255) & ~(size_t)255);
  memset(*p, 0, n);
  g_blocks[(char*)*p] = n;
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFree(void* p) {
  if (!p) return cudaSuccess;
  for (stream_t* s : g_streams) run(*s);  // cudaFree waits for the device
  if (!g_blocks.erase((char*)p)) fault("cudaFree of something else");
  else free(p);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind,
                                      cudaStream_t q) {
  const cudaError_t e = call("cudaMemcpyAsync");
  if (e != cudaSuccess) return e;
  if (kind == cudaMemcpyHostToDevice) {
    const std::string was((const char*)s, n);
    put(q, [=] {
      if (memcmp(s, was.data(), n)) fault("the source of a copy changed before it ran");
      memcpy(d, s, n);
    });
  } else {
    put(q, [=] { memcpy(d, s, n); });
  }
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w,
                                        size_t h, cudaMemcpyKind, cudaStream_t q) {
  put(q, [=] { for (size_t k = 0; k < h; k++) memcpy((char*)d + k * dp, (const char*)s + k * sp, w); });
  return call("cudaMemcpy2DAsync");
}
cudaError_t CUDARTAPI cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  memcpy(d, s, n);
  return call("cudaMemcpy");
}
cudaError_t CUDARTAPI cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t q) {
  put(q, [=] { memset(p, v, n); });
  return call("cudaMemsetAsync");
}
cudaError_t CUDARTAPI cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return call("cudaMemset"); }
cudaError_t CUDARTAPI cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)1 << 38; return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetSymbolAddress(void**, const void*) { return cudaErrorInvalidSymbol; }

// ------------------------------------------------------------------ streams, events, graphs
cudaError_t CUDARTAPI cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  stream_t* q = new stream_t;
  g_streams.insert(q);
  *s = reinterpret_cast<cudaStream_t>(q);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamDestroy(cudaStream_t s) {
  run(st(s));
  g_streams.erase(&st(s));
  delete &st(s);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t s) {
  run(st(s));
  return call("cudaStreamSynchronize");
}
cudaError_t CUDARTAPI cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventDestroy(cudaEvent_t e) { free((void*)e); return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventRecord(cudaEvent_t, cudaStream_t) { return call("cudaEventRecord"); }
cudaError_t CUDARTAPI cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  st(s).capture = new graph_t;
  return call("cudaStreamBeginCapture");
}
cudaError_t CUDARTAPI cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  *g = reinterpret_cast<cudaGraph_t>(st(s).capture);
  st(s).capture = nullptr;
  return call("cudaStreamEndCapture");
}
cudaError_t CUDARTAPI cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
  const cudaError_t e = call("cudaGraphInstantiate");
  if (e == cudaSuccess) *x = reinterpret_cast<cudaGraphExec_t>(new graph_t(*reinterpret_cast<graph_t*>(g)));
  return e;
}
cudaError_t CUDARTAPI cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<graph_t*>(g); return cudaSuccess; }
cudaError_t CUDARTAPI cudaGraphExecDestroy(cudaGraphExec_t x) {
  delete reinterpret_cast<graph_t*>(x);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
  const cudaError_t e = call("cudaGraphLaunch");
  if (e != cudaSuccess) return e;
  const graph_t& g = *reinterpret_cast<graph_t*>(x);
  g_log += g.kernels;
  for (const op& f : g.ops) put(s, f);
  return e;
}

// ------------------------------------------------------------------ the device
cudaError_t CUDARTAPI cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t CUDARTAPI cudaSetDevice(int) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t CUDARTAPI cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int,
                                                                            size_t, unsigned) {
  *n = 4;
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
const char* CUDARTAPI cudaGetErrorString(cudaError_t) { return "made to fail"; }
const char* CUDARTAPI cudaGetErrorName(cudaError_t) { return "fake"; }
}
