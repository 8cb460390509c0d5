// A stand-in for the CUDA runtime that runs nothing: libbgp.so's host code on a machine
// without a GPU. "Device" memory is host memory, copies happen at once, a kernel launch
// is only noted. What it models beyond that:
//   * the legacy default stream: a memset on it waits in a queue until something the
//     host or that stream does orders it; a launch on another stream while the queue is
//     not empty is noted as unordered;
//   * errors on request: the n-th next cudaMalloc fails, no cluster fits, and the n-th
//     Thomas-Fermi step's barrier times out;
//   * the solver passes: a step's last pass finishes its instances, and descriptors with
//     null line tables are noted.
// Loaded in place of libcudart.so.12 (same soname and symbol version). Compiled twice: by
// nvcc the part that reads the launches' parameter blocks, by g++ the runtime.
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <string>

#if defined(__CUDACC__)
#include "bgp_solve.cuh"
#include "bgp_tf.cuh"
using namespace bgp;

void fake_note(const char* what);
int fake_tf_step_times_out();

// a launch of kernel n (mangled name) with its parameters
void fake_read_launch(const std::string& n, void** args) {
  if (n.find("k_sv_") != std::string::npos) {
    const SvLaunch& L = *(const SvLaunch*)args[0];
    for (int a = 0; a < L.nact; ++a) {
      const SvInst& I = L.insts[L.act[a]];
      for (int v = 0; v < kLVariants; ++v)
        if (!I.tabN[v] || !I.tabF[v] || (I.M && !I.tabM[v])) fake_note("null_table");
      if (n.find("k_sv_px") != std::string::npos) *I.hstate = ST_DONE;
    }
  } else if (n.find("k_tf_iter") != std::string::npos) {
    const TfArgs& A = *(const TfArgs*)args[0];
    // a CTA other than the first gives up at the step's last barrier: the status word is
    // set, the state (written by the first CTA) looks like any other step's
    if (fake_tf_step_times_out()) A.abort_flag[0] = 1;
    A.state[4] += 1.0;
  }
}

#else

#include <functional>
#include <map>
#include <mutex>
#include <vector>

void fake_read_launch(const std::string& n, void** args);

namespace {
std::recursive_mutex mu;
std::map<const void*, std::string> names;            // kernel entries
std::vector<std::function<void()>> legacy;           // memsets the default stream still owes
std::map<std::string, long long> count;              // what happened, by name
std::vector<size_t> mallocs;
cudaError_t last = cudaSuccess;
int fail_malloc = 0, fail_host = 0, clusters = 1, tf_timeout = 0, tf_steps = 0;
long long next_handle = 1;

cudaError_t err(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
void drain() {
  for (auto& f : legacy) f();
  legacy.clear();
}
bool is_legacy(cudaStream_t s) { return s == nullptr || s == cudaStreamLegacy; }

cudaError_t launched(const void* fn, void** args, cudaStream_t st) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  const std::string& n = names[fn];
  if (is_legacy(st)) drain();
  else if (!legacy.empty()) count["unordered"]++;
  count["launch"]++;
  const size_t k = n.find("k_");                       // the kernel's plain name
  if (k != std::string::npos) count[n.substr(k, n.find_first_of("ABCDEFGHIJKLMNOPQRSTUVWXYZ", k) - k)]++;
  fake_read_launch(n, args);
  return err(cudaSuccess);
}
}  // namespace

void fake_note(const char* what) { count[what]++; }
int fake_tf_step_times_out() { return ++tf_steps == tf_timeout; }

extern "C" {
// ---------------------------------------------------------------- test controls
long long fake_count(const char* what) { std::lock_guard<std::recursive_mutex> lk(mu); return count[what]; }
int fake_mallocs(size_t* out, int cap) {
  for (int k = 0; k < cap && k < (int)mallocs.size(); ++k) out[k] = mallocs[k];
  return (int)mallocs.size();
}
void fake_fail_malloc(int nth) { fail_malloc = nth; }
void fake_fail_host_alloc(int nth) { fail_host = nth; }
void fake_clusters(int n) { clusters = n; }
void fake_tf_timeout(int step) { tf_timeout = step; tf_steps = 0; }
void* fake_stream() { return (void*)(next_handle++ << 16); }

// ---------------------------------------------------------------- registration
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 1; }
void __cudaRegisterFunction(void**, const char* fn, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names[fn] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
static struct { dim3 g, b; size_t sm; cudaStream_t st; } cfg;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sm, cudaStream_t st) { cfg = {g, b, sm, st}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* sm, void* st) {
  *g = cfg.g; *b = cfg.b; *sm = cfg.sm; *(cudaStream_t*)st = cfg.st;
  return cudaSuccess;
}

// ---------------------------------------------------------------- device
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  memset(p, 0, sizeof *p);
  p->multiProcessorCount = 148;
  p->sharedMemPerBlockOptin = 232448;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaDeviceSynchronize() { std::lock_guard<std::recursive_mutex> lk(mu); drain(); return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 4; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { *n = clusters; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static char v[1 << 16]; *p = v; return cudaSuccess; }

// ---------------------------------------------------------------- memory
cudaError_t cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  mallocs.push_back(n);
  if (fail_malloc > 0 && --fail_malloc == 0) return err(cudaErrorMemoryAllocation);
  *p = malloc(n);
  memset(*p, 0xA5, n);
  count["live"]++;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  drain();
  if (p) count["live"]--;
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  if (fail_host > 0 && --fail_host == 0) return err(cudaErrorMemoryAllocation);
  *p = calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  drain();
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (is_legacy(st)) drain();
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  legacy.push_back([=] { memset(p, v, n); });
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (is_legacy(st)) drain();
  memset(p, v, n);
  return cudaSuccess;
}

// ---------------------------------------------------------------- streams, events, launches
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)fake_stream(); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (is_legacy(s)) drain();
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)fake_stream(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** a, size_t, cudaStream_t s) { return launched(f, a, s); }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3, dim3, void** a, size_t, cudaStream_t s) { return launched(f, a, s); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) { return launched(f, a, c->stream); }
}

#endif
