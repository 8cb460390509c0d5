// Host side of libbgp.so: plans, twiddle and kernel tables, team scheduling,
// cooperative launches and the C ABI declared in include/bgp.h.
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/bgp.h"
#include "bgp_programs.cuh"
#include "bgp_sizes_gen.h"
#include "bgp_table.cuh"
#include "bgp_tf.cuh"
#include "bgp_stream.cuh"
#include "bgp_solve.cuh"

using namespace bgp;

namespace {

constexpr int kProfSlots = 20 * 5;   // phase profiler: 20 phase kinds x 5 counters
constexpr int kYieldDiv = 4;         // a solve launch yields once 1/kYieldDiv of it has finished
constexpr int kTuneYield[3] = {2, 4, 8};  // relaunch schedules the autotuner tries
constexpr int kMaxSegments = 256;    // relaunch limit of one solve
constexpr int kTfAhead = 8;          // Thomas-Fermi steps enqueued between looks at their state
constexpr int kResidBlocks = 592;    // blocks of the residual's sum: 4 per SM

thread_local std::string g_err;
int fail(int code, const std::string& msg) {
  g_err = msg;
  return code;
}
// An error that a call returned and that is reported is not left behind as the runtime's
// last error as well, where the next launch's check (ours or another library's) would find it.
#define CK(call)                                                                      \
  do {                                                                                \
    cudaError_t e_ = (call);                                                          \
    if (e_ != cudaSuccess) {                                                          \
      cudaGetLastError();                                                             \
      return fail(e_ == cudaErrorMemoryAllocation ? BGP_ERR_OOM : BGP_ERR_CUDA,       \
                  std::string(#call) + ": " + cudaGetErrorString(e_));                \
    }                                                                                 \
  } while (0)

bool size_ok(int N, int M) {
#define X(n, m) if (N == n && M == m) return true;
  BGP_FOR_SIZES(X)
#undef X
  return false;
}

// persistent kernel of a size pair, or of two pairs; null if not compiled
void* kernel_for(int N, int M, int ndim) {
#define X(n, m) if (N == n && M == m) return ndim == 3 ? bgp_kptr_##n##_##m##_d3() : bgp_kptr_##n##_##m##_d2();
  BGP_FOR_SIZES(X)
#undef X
  return nullptr;
}
// two-size kernels (2D only)
void* kernel_for2(int N1, int M1, int N2, int M2, int ndim) {
  if (ndim != 2) return nullptr;
#define X(a, b, c, d)                                                                      \
  if ((N1 == a && M1 == b && N2 == c && M2 == d) ||                                      \
      (N1 == c && M1 == d && N2 == a && M2 == b))                                        \
    return bgp_kptr2_##a##_##b##_##c##_##d##_d2();
  BGP_FOR_COMBOS(X)
#undef X
  return nullptr;
}

}  // namespace

// Forward FFT of every line along axis `ax` of an L^d complex cube (table build).
template <int L>
struct OpCube {
  static constexpr bool kStore = true;
  BGP_NO_OUT(64)
  const Inst& I;
  int ax;
  double2* A;
  BGP_D Pre fetch(int t, int r, int c) {
    int i, j, k;
    Pre P;
    P.a = A[nline_elem(I, ax, t, r, c, i, j, k)];
    return P;
  }
  BGP_D double2 enter(const Pre& P, int, int, int) { return P.a; }
  BGP_D void line(double2* b, int lane, int, int) { warp_fft<L, false>(b, I.twN, lane); }
  BGP_D void leave(const Pre&, int t, int r, int c, double2 v) {
    int i, j, k;
    A[nline_elem(I, ax, t, r, c, i, j, k)] = v;
  }
};

template <int L>
__global__ void __launch_bounds__(kThreads) k_cube_fft(Inst I, int ax, double2* A) {
  extern __shared__ double2 dyn_sm[];
  OpCube<L> op{I, ax, A};
  const int nt = ntiles_axis(I);
  for (int t = blockIdx.x; t < nt; t += gridDim.x) {
    if (ax == I.ndim - 1) tile_run<L, true>(op, dyn_sm, t);
    else tile_run<L, false>(op, dyn_sm, t);
  }
}

// ---------------------------------------------------------------- host state
namespace {

struct DevCtx {
  int device = -1, sms = 0, max_grid = 0;
  size_t max_smem_optin = 0;
  std::map<int, double2*> tw;   // twiddle tables by length
  std::map<int, double2*> lf[kLVariants];   // line-transform tables of the stream passes
  std::map<int, float2*> lf32[kLVariants];  // the same rounded to FP32
  std::atomic<signed char> tf_fits[kTfClMax + 1] = {};   // clusters by size: 0 not asked, 1 fits, -1 does not
};
std::mutex g_mu;
std::map<int, DevCtx> g_dev;

// Host memory that the device writes (mapped, pinned): one block of kPinSlots slots per
// device for the process, because pinning takes 3 ms and creating a small plan 0.07 ms.
// A plan takes a slot and gives it back when it is destroyed; when all slots are taken,
// and for more than kPinBytes, the memory is the caller's own.
constexpr int kPinSlots = 256, kPinBytes = 512;
struct Pinned {
  char *host = nullptr, *dev = nullptr;
  int device = -1, slot = -1;             // slot -1: an allocation of its own
};
struct PinBlock {
  char *host = nullptr, *dev = nullptr;
  std::vector<int> free;
};
std::mutex g_pin_mu;
std::map<int, PinBlock> g_pin;

bool pin_alloc(size_t bytes, char** host, char** dev) {
  if (cudaHostAlloc((void**)host, bytes, cudaHostAllocMapped) != cudaSuccess) {
    cudaGetLastError();
    *host = nullptr;
    return false;
  }
  if (cudaHostGetDevicePointer((void**)dev, *host, 0) == cudaSuccess) return true;
  cudaGetLastError();
  cudaFreeHost(*host);
  *host = nullptr;
  return false;
}
// memory on the current device `device`
bool pin_take(int device, size_t bytes, Pinned* P) {
  if (bytes <= kPinBytes) {
    std::lock_guard<std::mutex> lk(g_pin_mu);
    PinBlock& B = g_pin[device];
    if (!B.host && pin_alloc((size_t)kPinSlots * kPinBytes, &B.host, &B.dev))
      for (int k = kPinSlots - 1; k >= 0; --k) B.free.push_back(k);
    if (!B.free.empty()) {
      P->slot = B.free.back();
      B.free.pop_back();
      P->device = device;
      P->host = B.host + (size_t)P->slot * kPinBytes;
      P->dev = B.dev + (size_t)P->slot * kPinBytes;
      return true;
    }
  }
  P->slot = -1;
  return pin_alloc(bytes, &P->host, &P->dev);
}
// once no work that writes it is left
void pin_give(Pinned* P) {
  if (!P->host) return;
  if (P->slot >= 0) {
    std::lock_guard<std::mutex> lk(g_pin_mu);
    g_pin[P->device].free.push_back(P->slot);
  } else {
    cudaFreeHost(P->host);
  }
  *P = Pinned();
}

int ensure_device(DevCtx** out) {
  int dev = 0;
  CK(cudaGetDevice(&dev));
  DevCtx& d = g_dev[dev];
  if (d.device < 0) {
    cudaDeviceProp p;
    CK(cudaGetDeviceProperties(&p, dev));
    d.device = dev;
    d.sms = p.multiProcessorCount;
    d.max_smem_optin = p.sharedMemPerBlockOptin;
  }
  *out = &d;
  return BGP_OK;
}

// A table uploaded to device memory of its own.
template <class T>
int upload(const std::vector<T>& h, T** out) {
  T* dp = nullptr;
  CK(cudaMalloc(&dp, sizeof(T) * h.size()));
  const cudaError_t e = cudaMemcpy(dp, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) cudaFree(dp);
  CK(e);
  *out = dp;
  return BGP_OK;
}

// exp(-2 pi i t / L), t = 0..L-1, from long-double sin/cos of the reduced angle
int twiddles(DevCtx* d, int L, const double2** out) {
  auto it = d->tw.find(L);
  if (it != d->tw.end()) { *out = it->second; return BGP_OK; }
  std::vector<double2> h(L);
  const long double pi = 3.141592653589793238462643383279502884L;
  for (int t = 0; t < L; ++t) {
    // reduce to the first octant by symmetry so the table is exactly symmetric
    const long double ang = 2.0L * pi * (long double)t / (long double)L;
    long double c = cosl(ang), s = sinl(ang);
    if (8LL * t % L == 0) {
      const int oct = (int)(8LL * t / L);
      const double cs[8] = {1, M_SQRT1_2, 0, -M_SQRT1_2, -1, -M_SQRT1_2, 0, M_SQRT1_2};
      const double sn[8] = {0, M_SQRT1_2, 1, M_SQRT1_2, 0, -M_SQRT1_2, -1, -M_SQRT1_2};
      c = cs[oct]; s = sn[oct];
    }
    h[t] = cmk((double)c, -(double)s);
  }
  double2* dp = nullptr;
  int rc = upload(h, &dp);
  if (rc) return rc;
  d->tw[L] = dp;
  *out = dp;
  return BGP_OK;
}

// stage twiddles of the stream passes' line transform of length L, variant V, in FP64 and
// rounded to FP32: both or neither
template <int L, int V>
int lf_table(DevCtx* d) {
  if (d->lf[V].count(L)) return BGP_OK;
  constexpr int len = lf_tab_len(L, V);
  std::vector<double2> w(L), tab(len);
  const double2* dw = nullptr;
  int rc = twiddles(d, L, &dw);
  if (rc) return rc;
  CK(cudaMemcpy(w.data(), dw, sizeof(double2) * L, cudaMemcpyDeviceToHost));
  lf_fill_table<L, V>(w.data(), tab.data());
  std::vector<float2> tf(len);
  for (int q = 0; q < len; ++q) tf[q] = cmake<float2>((float)tab[q].x, (float)tab[q].y);
  double2* dp = nullptr;
  float2* fp = nullptr;
  if ((rc = upload(tab, &dp))) return rc;
  if ((rc = upload(tf, &fp))) { cudaFree(dp); return rc; }
  d->lf[V][L] = dp;
  d->lf32[V][L] = fp;
  return BGP_OK;
}
int lf_tables(DevCtx* d, int L) {
  switch (L) {
#define X(l) case l: { int rc = lf_table<l, 0>(d); if (!rc) rc = lf_table<l, 1>(d); return rc ? rc : lf_table<l, 2>(d); }
    BGP_FOR_LINE_LENGTHS(X)
#undef X
    default: return fail(BGP_ERR_UNSUPPORTED, "line length not compiled in");
  }
}

}  // namespace

// An instance's line-transform tables by factorization. The plan holds them from its
// creation on: the maps of DevCtx are shared by all plans of a device and grow under g_mu
// while other threads apply and solve.
struct LineTables {
  const double2 *N[kLVariants] = {}, *M[kLVariants] = {};   // of its N- and M-lines
  const float2* F[kLVariants] = {};                         // N in FP32
};

struct bgp_plan {
  DevCtx* dev = nullptr;
  std::vector<bgp_instance_desc> desc;
  std::vector<Inst> inst;                 // host copies with device pointers
  std::vector<LineTables> lines;
  std::vector<void*> allocs;
  long long bytes = 0;
  Inst* d_inst = nullptr;
  int* d_cta_inst = nullptr;
  double* d_tf = nullptr;                  // Thomas-Fermi state (kTfState values), then
  int* d_abort = nullptr;                  // the status words: one copy brings both to the host
  int* d_finished = nullptr;               // finished-instance counter of a solve launch
  long long launches = 0;                  // kernel launches issued by this plan
  SolveOut* d_out = nullptr;
  double* d_res = nullptr;                // n_inst x (kNRec + 1)
  double* d_part = nullptr;               // partial sums of the operators' stream passes
  size_t part_energy = 0, part_conv = 0;  // its sections: energy sums; one convolution's sums
  // stream solver
  SvInst* d_sv = nullptr;
  SvCtl* d_ctl = nullptr;
  SvSync* d_svsync = nullptr;
  unsigned* d_svhist = nullptr;           // kSvBins per instance
  unsigned long long* d_svcand = nullptr; // kSvCap per instance
  std::vector<double*> svpart;            // partial sums per instance
  int* d_act = nullptr;                   // active instances, group by group
  int *h_state = nullptr, *d_state = nullptr; // instances' solver states (mapped host memory)
  std::vector<cudaEvent_t> sv_ev;         // two per size group
  Pinned pin_sums, pin_state;
  double* h_sums = nullptr;               // totals on the host (mapped: the device writes them)
  double* d_sums = nullptr;               // the same memory as the device sees it
  int max_team = 0;
  int lmax = 0;
  size_t smem = 0;
  int grid_cap = 0;
  std::vector<int> cta_inst;
  // relaunch schedule and its autotuner: 0 off, 1 trying candidates, 2 done
  int yield_div = kYieldDiv;
  int tune = 0, tune_next = 0;
  float tune_ms[3] = {0.f, 0.f, 0.f};
  // stream-pass schedules by line length N (autotuned on first use unless fixed)
  struct StreamSched {
    int ln = 0, v = 0;            // H psi lines per tile, radix order
    int cln = 8, csln = 8, cv = 0;   // convolution: lines of contiguous / strided tiles, radix order
    int tuned = 0;                // 0: tune on first use, 1: tuned, 2: fixed by the caller
    std::vector<std::array<float, 4>> cand;   // (ln, v, strided ln, ms) of every timed candidate
  };
  std::map<int, StreamSched> ssched;
  // batched apply: one stream per further size group (forked from and joined to the
  // caller's stream by events), so groups of different sizes overlap on the GPU
  std::vector<cudaStream_t> side_st;
  std::vector<cudaEvent_t> side_ev;   // [0] the fork, [1 + g] the join of side group g
  // per size group: the stream of the H psi passes that run beside its convolution,
  // and that overlap's fork and join events
  std::vector<cudaStream_t> ovl_st;
  std::vector<cudaEvent_t> ovl_ev;
};

namespace {

int palloc(bgp_plan* p, size_t bytes, void** out) {
  void* q = nullptr;
  if (bytes == 0) { *out = nullptr; return BGP_OK; }
  cudaError_t e = cudaMalloc(&q, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(BGP_ERR_OOM, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  }
  p->allocs.push_back(q);
  p->bytes += (long long)bytes;
  CK(cudaMemset(q, 0, bytes));
  *out = q;
  return BGP_OK;
}

// Waits until what palloc allocated is zero: it is cleared on the default stream, which
// non-blocking streams do not wait for (a memset does not hold the host).
int zeroed() {
  CK(cudaStreamSynchronize(cudaStreamLegacy));
  return BGP_OK;
}

template <class T>
int palloc_t(bgp_plan* p, size_t count, T** out) {
  void* q = nullptr;
  int rc = palloc(p, count * sizeof(T), &q);
  *out = (T*)q;
  return rc;
}

template <int L>
int cube_fft_len(const Inst& I, double2* A, int ax) {
  const size_t smem = tile_smem_bytes(L);
  CK(cudaFuncSetAttribute(k_cube_fft<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int nt = ntiles_axis(I);
  k_cube_fft<L><<<nt < 4096 ? nt : 4096, kThreads, smem>>>(I, ax, A);
  CK(cudaGetLastError());
  return BGP_OK;
}

int cube_fft(const Inst& I, double2* A, int ax) {
  switch (I.N) {
#define X(l) case l: return cube_fft_len<l>(I, A, ax);
    BGP_FOR_TABLE_LENGTHS(X)
#undef X
    default: return fail(BGP_ERR_UNSUPPORTED, "kernel table length not compiled in");
  }
}

// Build the real quadrant of the transformed cell-averaged kernel table.
int build_table(bgp_plan* p, const bgp_instance_desc& d, const Inst& I, int which, double** out) {
  const int M = I.M, ndim = I.ndim;
  const size_t tot = (ndim == 2) ? (size_t)M * M : (size_t)M * M * M;
  double2* F = nullptr;
  CK(cudaMalloc(&F, tot * sizeof(double2)));
  k_table_fill<<<1184, 256>>>(F, ndim, M, I.dx, I.kind, which, d.l_z);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { cudaFree(F); return fail(BGP_ERR_CUDA, cudaGetErrorString(e)); }
  // exact self cell at the origin (interactions.py:128-135, 146)
  double self;
  if (which == 1) self = polar_self_cell_2d(I.kind, 1, d.l_z, I.dx);
  else if (ndim == 3) self = kSelfNewton3D / I.dx;
  else if (I.kind == kNewton) self = 4.0 * asinh(1.0) / I.dx;
  else if (I.kind == kLog) self = -log(I.dx) + (1.5 + 0.5 * log(2.0) - 0.25 * M_PI);
  else self = polar_self_cell_2d(I.kind, 0, d.l_z, I.dx);
  const double2 sc = cmk(self, 0.0);
  CK(cudaMemcpy(F, &sc, sizeof(double2), cudaMemcpyHostToDevice));
  Inst C = I;
  C.N = M;  // transform the M-cube with the M twiddles
  C.twN = I.twM;
  for (int ax = 0; ax < ndim; ++ax) {
    int rc = cube_fft(C, F, ax);
    if (rc) { cudaFree(F); return rc; }
  }
  const int Mh = M / 2 + 1;
  const size_t qn = (ndim == 2) ? (size_t)Mh * Mh : (size_t)Mh * Mh * Mh;
  double* Kq = nullptr;
  int rc = palloc_t(p, qn, &Kq);
  if (rc) { cudaFree(F); return rc; }
  k_table_quadrant<<<1184, 256>>>(F, Kq, ndim, M);
  e = cudaDeviceSynchronize();
  cudaFree(F);
  if (e != cudaSuccess) return fail(BGP_ERR_CUDA, std::string("kernel table: ") + cudaGetErrorString(e));
  *out = Kq;
  return BGP_OK;
}

int grid_cap_for(bgp_plan* p, void* kern, int* cap) {
  int nb = 0;
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem));
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, kThreads, p->smem));
  if (nb < 1) return fail(BGP_ERR_CUDA, "solver kernel does not fit on an SM");
  *cap = nb * p->dev->sms;
  return BGP_OK;
}

int max_grid(bgp_plan* p) {
  int cap = 1 << 30;
  for (const Inst& I : p->inst) {
    void* k = kernel_for(I.N, I.M, I.ndim);
    if (!k) return fail(BGP_ERR_UNSUPPORTED, "grid size not compiled in");
    int c = 0;
    int rc = grid_cap_for(p, k, &c);
    if (rc) return rc;
    cap = c < cap ? c : cap;
  }
  p->grid_cap = cap;
  return BGP_OK;
}

// CTAs an instance can keep busy in its widest phase
int useful_ctas(const Inst& I) {
  const int nt = ntiles_axis(I);
  if (I.kind == kNone || I.M == 0) return nt;
  const int tpl = (I.Mh + kLines - 1) / kLines;
  return nt + (I.ndim == 2 ? tpl : I.M * tpl);
}

int launch_group(bgp_plan* p, const std::vector<int>& active, void* kern, cudaStream_t st);

// Launch the active instances: one kernel when they share a size (or form a
// compiled two-size combination), otherwise one launch per size group.
int launch(bgp_plan* p, const std::vector<int>& active, cudaStream_t st) {
  // kinds of kernel: (ndim, N, M)
  std::vector<std::array<int, 3>> kinds;
  auto kind_of = [&](int a) {
    const Inst& I = p->inst[a];
    return std::array<int, 3>{I.ndim, I.N, I.M};
  };
  for (int a : active) {
    const auto k = kind_of(a);
    bool seen = false;
    for (auto& q : kinds) seen = seen || q == k;
    if (!seen) kinds.push_back(k);
  }
  if (kinds.size() == 1)
    return launch_group(p, active, kernel_for(kinds[0][1], kinds[0][2], kinds[0][0]), st);
  if (kinds.size() == 2 && kinds[0][0] == kinds[1][0]) {
    void* k2 = kernel_for2(kinds[0][1], kinds[0][2], kinds[1][1], kinds[1][2], kinds[0][0]);
    if (k2) return launch_group(p, active, k2, st);
  }
  for (auto& k : kinds) {
    std::vector<int> grp;
    for (int a : active) if (kind_of(a) == k) grp.push_back(a);
    int rc = launch_group(p, grp, kernel_for(k[1], k[2], k[0]), st);
    if (rc) return rc;
  }
  return BGP_OK;
}

// Assign teams to the active instances and launch the persistent kernel.
int launch_group(bgp_plan* p, const std::vector<int>& active, void* kern, cudaStream_t st) {
  if (!kern) return fail(BGP_ERR_UNSUPPORTED, "grid size not compiled in");
  const int na = (int)active.size();
  std::vector<int> team(na, 1);
  std::vector<double> w(na);
  double wsum = 0.0;
  for (int a = 0; a < na; ++a) { w[a] = (double)p->inst[active[a]].n; wsum += w[a]; }
  if (na > p->grid_cap) return fail(BGP_ERR_ARG, "more instances than resident CTAs in one batch");
  int cap = p->grid_cap;
  int used = 0;
  for (int a = 0; a < na; ++a) {
    const int want = useful_ctas(p->inst[active[a]]);
    int t = (int)floor(cap * w[a] / wsum);
    t = t < 1 ? 1 : t;
    t = t > want ? want : t;
    t = t > p->max_team ? p->max_team : t;
    team[a] = t;
    used += t;
  }
  // hand out what is left, largest instances first
  for (bool grew = true; used < cap && grew;) {
    grew = false;
    for (int a = 0; a < na && used < cap; ++a) {
      const int want = useful_ctas(p->inst[active[a]]);
      if (team[a] < want && team[a] < p->max_team) { team[a]++; used++; grew = true; }
    }
  }
  while (used > cap) {  // only if the floor-1 clamps overflowed
    int big = 0;
    for (int a = 1; a < na; ++a) if (team[a] > team[big]) big = a;
    if (team[big] <= 1) return fail(BGP_ERR_ARG, "batch too large for one launch");
    team[big]--; used--;
  }
  std::vector<Inst> hi(na);
  p->cta_inst.assign(used, 0);
  int first = 0;
  for (int a = 0; a < na; ++a) {
    hi[a] = p->inst[active[a]];
    hi[a].team_first = first;
    hi[a].team_size = team[a];
    for (int q = 0; q < team[a]; ++q) p->cta_inst[first + q] = a;
    first += team[a];
  }
  CK(cudaMemcpyAsync(p->d_inst, hi.data(), sizeof(Inst) * na, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(p->d_cta_inst, p->cta_inst.data(), sizeof(int) * used, cudaMemcpyHostToDevice, st));
  CK(cudaMemsetAsync(p->d_abort, 0, (4 + (size_t)used) * sizeof(int), st));
  for (int a = 0; a < na; ++a) CK(cudaMemsetAsync(hi[a].bar, 0, sizeof(unsigned long long), st));
  Launch L{p->d_inst, p->d_cta_inst, p->d_abort};
  void* args[] = {&L};
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem));
  CK(cudaLaunchCooperativeKernel(kern, dim3(used), dim3(kThreads), args, p->smem, st));
  p->launches++;
  CK(cudaGetLastError());
  int ab[4] = {0, 0, 0, 0};
  CK(cudaMemcpyAsync(ab, p->d_abort, sizeof(ab), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if (ab[0] != 0) {
    // last barrier arrival of every CTA of the team that timed out
    std::vector<int> arr(used);
    CK(cudaMemcpy(arr.data(), p->d_abort + 4, sizeof(int) * used, cudaMemcpyDeviceToHost));
    std::string team;
    const int a0 = ab[1] >= 0 && ab[1] < used ? p->cta_inst[ab[1]] : -1;
    for (int b = 0; b < used; ++b)
      if (p->cta_inst[b] == a0) team += std::to_string(b) + ":" + std::to_string(arr[b]) + " ";
    char buf[200];
    snprintf(buf, sizeof buf,
             "device status %d (1 = team barrier timeout, 2 = size not compiled); block %d waited "
             "for barrier count %d and saw %d; last arrivals (block:count) ", ab[0], ab[1], ab[2], ab[3]);
    return fail(BGP_ERR_DEVICE, std::string(buf) + team);
  }
  return BGP_OK;
}

int check_inst(const bgp_plan* p, int i) {
  if (!p) return fail(BGP_ERR_ARG, "null plan");
  if (i < 0 || i >= (int)p->inst.size()) return fail(BGP_ERR_ARG, "instance index out of range");
  return BGP_OK;
}

}  // namespace

// error reporting for the other translation units of the library
int bgp_report_error(int code, const char* msg) { return fail(code, msg); }

// ======================================================================= C ABI
extern "C" {

int bgp_version(void) { return 100; }
const char* bgp_last_error(void) { return g_err.c_str(); }

double bgp_k0e(double x) { double a, b; k01e(x, a, b); return a; }
double bgp_k1e(double x) { double a, b; k01e(x, a, b); return b; }

int bgp_size_supported(int ndim, int N, int pad, int kernel) {
  if (ndim != 2 && ndim != 3) return 0;
  if (kernel != BGP_KERNEL_NONE && pad != 2) return 0;
  return size_ok(N, kernel == BGP_KERNEL_NONE ? 0 : 2 * N) ? 1 : 0;
}

int bgp_plan_create(const bgp_instance_desc* desc, int n_inst, bgp_plan** plan) {
  if (!desc || n_inst < 1 || !plan) return fail(BGP_ERR_ARG, "bad arguments");
  std::lock_guard<std::mutex> lk(g_mu);
  DevCtx* dev = nullptr;
  int rc = ensure_device(&dev);
  if (rc) return rc;
  bgp_plan* p = new bgp_plan();
  p->dev = dev;
  p->desc.assign(desc, desc + n_inst);
  p->inst.resize(n_inst);
  p->lines.resize(n_inst);
  auto bail = [&](int code) { bgp_plan_destroy(p); return code; };
  // first pass: sizes
  for (int i = 0; i < n_inst; ++i) {
    const bgp_instance_desc& d = desc[i];
    if (d.ndim != 2 && d.ndim != 3) return bail(fail(BGP_ERR_ARG, "ndim must be 2 or 3"));
    if (d.kernel < 0 || d.kernel > 3) return bail(fail(BGP_ERR_ARG, "unknown kernel"));
    if (d.kernel == BGP_KERNEL_LOG && d.ndim != 2) return bail(fail(BGP_ERR_ARG, "kernel 'log' is 2D only"));
    if (d.kernel == BGP_KERNEL_Q2D && (d.ndim != 2 || !(d.l_z > 0))) return bail(fail(BGP_ERR_ARG, "kernel 'q2d' needs 2D and l_z > 0"));
    if (d.kernel == BGP_KERNEL_NEWTON && false) {}
    if (!(d.L > 0)) return bail(fail(BGP_ERR_ARG, "L must be positive"));
    if (d.kernel != BGP_KERNEL_NONE && d.pad != 2)
      return bail(fail(BGP_ERR_UNSUPPORTED, "only pad = 2 is compiled in for the long-range term"));
    const int M = d.kernel == BGP_KERNEL_NONE ? 0 : 2 * d.N;
    if (!size_ok(d.N, M)) {
      char buf[160];
      snprintf(buf, sizeof buf, "grid N=%d%s is not compiled in (supported: 16 24 32 48 64 96 128 192 256 384 512; "
               "up to 384 with a long-range kernel)", d.N, M ? " with a long-range kernel" : "");
      return bail(fail(BGP_ERR_UNSUPPORTED, buf));
    }
    Inst& I = p->inst[i];
    memset(&I, 0, sizeof(Inst));
    I.ndim = d.ndim; I.N = d.N; I.M = M; I.kind = d.kernel;
    I.n = d.ndim == 2 ? d.N * d.N : d.N * d.N * d.N;
    I.Mh = M ? M / 2 + 1 : 0;
    I.i0 = M ? (M - d.N) / 2 : 0;
    I.dx = 2.0 * d.L / d.N;
    I.dv = d.ndim == 2 ? I.dx * I.dx : I.dx * I.dx * I.dx;
    I.kfac = 1.0 / (d.N * I.dx);
    I.s = d.s; I.tc = d.trap_coeff;
    I.beta2 = d.beta2; I.beta3 = d.beta3; I.Omega = d.Omega; I.G_C = d.G_C;
    I.inv_n = 1.0 / (double)I.n;
    const double Md = M ? (d.ndim == 2 ? (double)M * M : (double)M * M * M) : 1.0;
    I.conv_scale = M ? -d.G_C * I.dv / Md : 0.0;
    p->lmax = std::max(p->lmax, std::max(d.N, M));
  }
  // the tile buffer; the median's rank selection reuses it for kSelCap keys
  p->smem = std::max(tile_smem_bytes(p->lmax), (size_t)kSelCap * sizeof(unsigned long long));
  if (p->smem > dev->max_smem_optin) return bail(fail(BGP_ERR_UNSUPPORTED, "tile does not fit in shared memory"));
  rc = max_grid(p);
  if (rc) return bail(rc);
  p->max_team = p->grid_cap;
  for (int i = 0; i < n_inst; ++i) {
    Inst& I = p->inst[i];
    const bgp_instance_desc& d = desc[i];
    const size_t n = (size_t)I.n;
    if ((rc = twiddles(dev, I.N, &I.twN))) return bail(rc);
    if (I.M && (rc = twiddles(dev, I.M, &I.twM))) return bail(rc);
    if ((rc = lf_tables(dev, I.N))) return bail(rc);
    if (I.M && (rc = lf_tables(dev, I.M))) return bail(rc);
    for (int V = 0; V < kLVariants; ++V) {
      p->lines[i].N[V] = dev->lf[V][I.N];
      p->lines[i].F[V] = dev->lf32[V][I.N];
      if (I.M) p->lines[i].M[V] = dev->lf[V][I.M];
    }
    if ((rc = palloc_t(p, (size_t)kNB * n, &I.pool))) return bail(rc);
    // potentials: current and trial; 3D with a kernel also the potentials of the
    // density's linear and quadratic parts in the step (the line search's quartic)
    if ((rc = palloc_t(p, (I.M && I.ndim == 3 ? 4 : 2) * n, &I.phi2))) return bail(rc);
    if ((rc = palloc_t(p, n, &I.keys))) return bail(rc);
    if ((rc = palloc_t(p, (size_t)8 * 256 + 2, &I.hist))) return bail(rc);
    if ((rc = palloc_t(p, (size_t)kSelCap, &I.cand))) return bail(rc);
    if ((rc = palloc_t(p, (size_t)kSelCap, &I.wcand))) return bail(rc);
    // reduction partials: the solver's (2 x kNRec per team CTA) and the stream H psi
    // passes' (one per tile of the last pass: up to N^(d-1) with one-line tiles)
    const size_t stream_tiles = I.ndim == 2 ? (size_t)I.N : (size_t)I.N * I.N;
    if ((rc = palloc_t(p, std::max((size_t)2 * kNRec * p->max_team, stream_tiles), &I.part))) return bail(rc);
    if ((rc = palloc_t(p, (size_t)1, &I.bar))) return bail(rc);
    if ((rc = palloc(p, sizeof(Ctl), &I.save))) return bail(rc);
    if (I.M) {
      // rows of conv_pitch(N) >= Mh columns (the stream passes' pitch; the persistent
      // programs pack theirs Mh apart)
      const size_t pitch = (size_t)conv_pitch(I.N);
      const size_t c1 = I.ndim == 2 ? I.N * pitch : (size_t)I.N * I.N * pitch;
      if ((rc = palloc_t(p, c1, &I.cb1))) return bail(rc);
      if (I.ndim == 3 && (rc = palloc_t(p, (size_t)I.N * I.M * pitch, &I.cb2))) return bail(rc);
      double* Kq = nullptr;
      if ((rc = build_table(p, d, I, 0, &Kq))) return bail(rc);
      I.Kq = Kq;
      if (I.kind == kQ2d) {
        double* Wq = nullptr;
        if ((rc = build_table(p, d, I, 1, &Wq))) return bail(rc);
        I.Wq = Wq;
      }
    }
  }
  if ((rc = palloc_t(p, (size_t)n_inst, &p->d_inst))) return bail(rc);
  if ((rc = palloc_t(p, (size_t)p->grid_cap, &p->d_cta_inst))) return bail(rc);
  if ((rc = palloc(p, sizeof(double) * kTfState + sizeof(int) * ((size_t)4 + p->grid_cap), (void**)&p->d_tf))) return bail(rc);
  p->d_abort = (int*)(p->d_tf + kTfState);
  if ((rc = palloc_t(p, (size_t)1, &p->d_finished))) return bail(rc);
  if ((rc = palloc_t(p, (size_t)n_inst, &p->d_out))) return bail(rc);
  if ((rc = palloc_t(p, (size_t)n_inst * (kNRec + 1), &p->d_res))) return bail(rc);
  // tiles of at least 4 lines in the energy passes, 2 in the convolution's last pass
  for (const Inst& I : p->inst) {
    const size_t lines = I.ndim == 2 ? (size_t)I.N : (size_t)I.N * I.N;
    p->part_energy = std::max(p->part_energy, (kESums + 1) * I.ndim * (lines / 4));
    p->part_conv = std::max(p->part_conv, std::max(lines / 2, (size_t)kResidBlocks));
  }
  if ((rc = palloc_t(p, p->part_energy + 2 * p->part_conv, &p->d_part))) return bail(rc);
  if (!pin_take(dev->device, sizeof(double) * SumArgs::kMax, &p->pin_sums))
    return bail(fail(BGP_ERR_OOM, "pinned host memory for the operators' sums"));
  p->h_sums = (double*)p->pin_sums.host;
  p->d_sums = (double*)p->pin_sums.dev;
  for (int i = 0; i < n_inst; ++i) {
    p->inst[i].out = p->d_out + i;
    p->inst[i].res = p->d_res + (size_t)i * (kNRec + 1);
  }
#if defined(BGP_PROF)
  unsigned long long* prof = nullptr;
  if ((rc = palloc_t(p, (size_t)n_inst * kProfSlots, &prof))) return bail(rc);
  for (int i = 0; i < n_inst; ++i) p->inst[i].prof = prof + (size_t)i * kProfSlots;
#endif
  if ((rc = zeroed())) return bail(rc);
  *plan = p;
  return BGP_OK;
}

int bgp_plan_destroy(bgp_plan* p) {
  if (!p) return BGP_OK;
  for (cudaStream_t q : p->side_st) cudaStreamDestroy(q);
  for (cudaStream_t q : p->ovl_st) cudaStreamDestroy(q);
  for (cudaEvent_t q : p->ovl_ev) cudaEventDestroy(q);
  for (cudaEvent_t q : p->side_ev) cudaEventDestroy(q);
  for (void* q : p->allocs) cudaFree(q);
  pin_give(&p->pin_sums);                 // (the frees above have waited for the plan's work)
  pin_give(&p->pin_state);
  for (cudaEvent_t q : p->sv_ev) cudaEventDestroy(q);
  delete p;
  return BGP_OK;
}

long long bgp_plan_bytes(const bgp_plan* p) { return p ? p->bytes : 0; }

int bgp_plan_autotune(bgp_plan* p, int enable) {
  if (!p) return fail(BGP_ERR_ARG, "null plan");
  if (enable) { p->tune = 1; p->tune_next = 0; }
  else if (p->tune == 1) { p->tune = 0; }
  return BGP_OK;
}

int bgp_plan_schedule(const bgp_plan* p, int* yield_div, int* tuned, float* ms3) {
  if (!p) return fail(BGP_ERR_ARG, "null plan");
  if (yield_div) *yield_div = p->yield_div;
  if (tuned) *tuned = p->tune == 2;
  if (ms3) for (int c = 0; c < 3; ++c) ms3[c] = p->tune_ms[c];
  return BGP_OK;
}

#if defined(BGP_PROF)
// Phase profiler counters of instance i (kProfSlots values), profiling builds only.
int bgp_prof_read(bgp_plan* p, int i, unsigned long long* out, int reset) {
  int rc = check_inst(p, i);
  if (rc) return rc;
  CK(cudaDeviceSynchronize());
  CK(cudaMemcpy(out, p->inst[i].prof, sizeof(unsigned long long) * kProfSlots, cudaMemcpyDeviceToHost));
  if (reset) CK(cudaMemset(p->inst[i].prof, 0, sizeof(unsigned long long) * kProfSlots));
  return BGP_OK;
}
#endif
long long bgp_plan_launches(const bgp_plan* p) { return p ? p->launches : 0; }

namespace {
void op_terms(const Inst& I, const double* res, bgp_energy_terms* terms) {
  double comp[8];
  energy_assemble(I, res, 1.0, comp);
  terms->E = comp[0]; terms->Ekin = comp[1]; terms->Etrap = comp[2]; terms->Econtact = comp[3];
  terms->Ethree = comp[4]; terms->Erot = comp[5]; terms->Egrav = comp[6]; terms->Lz = comp[7];
  terms->mass = res[S_N0] * I.dv;
  terms->r2mean = res[S_R2] * I.dv;
  terms->peak = res[kNSum];
  terms->rperp2 = res[S_PERP] * I.dv;
  terms->z2 = res[S_Z2] * I.dv;
}

int run_api(bgp_plan* p, int i, Inst& I, cudaStream_t st, double* res_host) {
  Inst save = p->inst[i];
  p->inst[i] = I;
  std::vector<int> act{i};
  int rc = launch(p, act, st);
  p->inst[i] = save;
  if (rc) return rc;
  CK(cudaMemcpyAsync(res_host, p->d_res + (size_t)i * (kNRec + 1), sizeof(double) * (kNRec + 1),
                     cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if (res_host[kNRec] != 0.0) return fail(BGP_ERR_DEVICE, "device program failed");
  return BGP_OK;
}
}  // namespace

int bgp_energy_observables(bgp_plan* p, int i, const void* psi, bgp_energy_terms* terms, void* stream) {
  int rc = check_inst(p, i);
  if (rc) return rc;
  if (!psi || !terms) return fail(BGP_ERR_ARG, "null pointer");
  Inst I = p->inst[i];
  I.prog = kProgEnergy;
  I.in_psi = (const double2*)psi;
  double res[kNRec + 1] = {0};
  CK(cudaMemsetAsync(p->d_res + (size_t)i * (kNRec + 1), 0, sizeof(double) * (kNRec + 1), (cudaStream_t)stream));
  rc = run_api(p, i, I, (cudaStream_t)stream, res);
  if (rc) return rc;
  op_terms(I, res, terms);
  return BGP_OK;
}

int bgp_precondition(bgp_plan* p, int i, const void* grad, const void* psi, const double* phi,
                     double shift_min, void* z, double* sigma_out, void* stream) {
  int rc = check_inst(p, i);
  if (rc) return rc;
  if (!grad || !psi || !z) return fail(BGP_ERR_ARG, "null pointer");
  Inst I = p->inst[i];
  I.prog = kProgPrecond;
  I.in_grad = (const double2*)grad;
  I.in_psi = (const double2*)psi;
  I.in_phi = phi;
  I.use_phi = phi ? 1 : 0;
  I.out_c = (double2*)z;
  I.sp.shift_min = shift_min;
  double res[kNRec + 1] = {0};
  CK(cudaMemsetAsync(p->d_res + (size_t)i * (kNRec + 1), 0, sizeof(double) * (kNRec + 1), (cudaStream_t)stream));
  rc = run_api(p, i, I, (cudaStream_t)stream, res);
  if (rc) return rc;
  if (sigma_out) *sigma_out = res[0];
  return BGP_OK;
}

}  // extern "C"

namespace {
// ------------------------------------------------------------ stream passes
// compiled passes by tile width C, factorization V, kind and parameter block (one
// instance or a batch); null where not compiled
const SKernel* stream_h_kernel(int N, int C, int V, int stage, bool batch) {
  switch (N) {
#define X(n) case n: return bgp_sptr_##n(C, V, stage, batch);
    BGP_FOR_STREAM_N(X)
#undef X
    default: return nullptr;
  }
}
const SKernel* stream_real_kernel(int N, int C, int V, int inv, bool batch) {
  switch (2 * N) {
#define X(m) case m: return bgp_srptr_##m(C, V, inv, batch);
    BGP_FOR_STREAM_M(X)
#undef X
    default: return nullptr;
  }
}
const SKernel* stream_pad_kernel(int M, int C, int V, int mode, bool batch) {
  switch (M) {
#define X(m) case m: return bgp_spptr_##m(C, V, mode, batch);
    BGP_FOR_STREAM_M(X)
#undef X
    default: return nullptr;
  }
}

const SKernel* stream_energy_kernel(int N, int C, int V) {
  switch (N) {
#define X(n) case n: return bgp_septr_##n(C, V, 0, 0);
    BGP_FOR_STREAM_N(X)
#undef X
    default: return nullptr;
  }
}

bool has_kernel(const Inst& I) { return I.kind != kNone && I.M > 0; }

// A pass schedule in compiled terms: tile widths and factorization variants.
struct Sched {
  int c, v;          // H psi passes
  int cr, cs, cv;    // convolution: real (contiguous) and padded (strided) passes, variant
};
// The public codes name 1 to 16 lines and radix orders 0 to 7 (0 and 3 for the
// convolution); tiles of 2, 4 and 8 lines in two factorizations are compiled, and a
// code runs as the nearest of them.
Sched sched_of(const bgp_plan::StreamSched& sc) {
  auto w = [](int ln, int lo) { return ln < lo ? lo : (ln > 8 ? 8 : ln); };
  return Sched{w(sc.ln, 2), sc.v & 1, w(sc.cln, 2), w(sc.csln, 4), sc.cv ? 1 : 0};
}

// The schedule of the single-instance operators, by size. A grid of half a million
// points or more fills the GPU with 8-line tiles (128-byte rows) and takes the
// factorization with the fewest exchanges; a smaller one is a few microseconds of
// latency: narrower tiles spread it over more SMs, and lengths 2^a take the
// factorization with more threads per line. 128^3: 8 lines, 4 lines 3 % slower; 256^2: H psi
// 4 or 8 lines within 2 %, the quasi-2D convolution 2 and 4 lines 17.5 us, 8 and 8 lines
// 19 us. Padded lines of 384 and 768 have three stages in the second factorization and
// four in the first (us of a volume's apply with its potential, second / first: 192^3
// 704 / 764, 384^3 7240 / 7398); lines of 192 have three in either (96^3 95 / 93), and of
// 2^a points no fewer in the second (128^3 211 / 178, 256^3 1819 / 1561).
Sched sched_rule(const Inst& I) {
  const int v = (I.N & (I.N - 1)) == 0;
  if (I.n >= (1 << 19)) return Sched{8, 0, 8, 8, I.ndim == 3 && !v && I.M >= 384};
  return Sched{4, v, 2, 4, v};
}

// per-instance total of the tiles' partial sums, in tile order: mu = sum dV
template <int NB>
__global__ void k_stream_mu(const __grid_constant__ SLaunchT<NB> SL, int tiles, double* mu, int offset) {
  const int a = blockIdx.x;
  if (a >= SL.ninst) return;
  const SInst& I = SL.insts[a];
  double s = 0.0;
  for (int t = threadIdx.x; t < tiles; t += blockDim.x) s += I.part[t];
  __shared__ double red[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) tot += red[q];
    mu[offset + a] = tot * I.dv;
  }
}

// One pass; chained: it may start while the launch before it on the stream still runs
// (the pass itself waits, griddepcontrol, before it reads what that one writes).
template <int NB>
int stream_launch(const SKernel* kern, int tiles, SLaunchT<NB>& SL, cudaStream_t st, bool chained, int axes = 1) {
  if (!kern) return fail(BGP_ERR_UNSUPPORTED, "stream pass not compiled for this size / schedule");
  SL.tiles = tiles;
  if (kern->smem > 48 * 1024)
    CK(cudaFuncSetAttribute(kern->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kern->smem));
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(tiles * SL.ninst * axes);
  cfg.blockDim = dim3(kern->threads);
  cfg.dynamicSmemBytes = kern->smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = chained ? 1 : 0;
  void* args[] = {&SL};
  CK(cudaLaunchKernelExC(&cfg, kern->fn, args));
  return BGP_OK;
}

// The convolution passes of a group: phi from |psi|^2. The first is a plain launch
// (it reads psi and writes the scratch, so it waits for all earlier work).
template <int NB>
int stream_conv(SLaunchT<NB>& SL, const Sched& S, cudaStream_t st) {
  const SInst& I0 = SL.insts[0];
  const int N = I0.N, ndim = I0.ndim, M = I0.M, tpl = (N + 1 + S.cs - 1) / S.cs;
  const int lines = ndim == 2 ? N : N * N;
  int rc = stream_launch(stream_real_kernel(N, S.cr, S.cv, 0, NB > 1), lines / S.cr, SL, st, false);
  if (!rc && ndim == 3)
    rc = stream_launch(stream_pad_kernel(M, S.cs, S.cv, 0, NB > 1), N * tpl, SL, st, true);
  if (!rc)
    rc = stream_launch(stream_pad_kernel(M, S.cs, S.cv, 1, NB > 1), (ndim == 2 ? 1 : M) * tpl, SL, st, true);
  if (!rc && ndim == 3)
    rc = stream_launch(stream_pad_kernel(M, S.cs, S.cv, 2, NB > 1), N * tpl, SL, st, true);
  if (!rc) rc = stream_launch(stream_real_kernel(N, S.cr, S.cv, 1, NB > 1), lines / S.cr, SL, st, true);
  return rc;
}

// The passes of one group (same N, ndim, kernel): optional convolution (phi from
// |psi|^2), then the H psi axis passes, then mu.
template <int NB>
int stream_run(SLaunchT<NB>& SL, const Sched& S, bool conv, double* mu_dev, int mu_off, cudaStream_t st,
               cudaStream_t side = nullptr, cudaEvent_t ev_fork = nullptr, cudaEvent_t ev_join = nullptr) {
  const SInst& I0 = SL.insts[0];
  const int N = I0.N, ndim = I0.ndim, n = I0.n;
  const int tiles = n / (N * S.c);
  // the first axis pass is a plain launch, the later ones are chained to it; the last
  // one is plain where another stream's work comes in between
  auto hstage = [&](int st_, cudaStream_t q, bool chained) -> int {
    const int stage = (st_ == 0) ? 0 : (st_ == ndim - 1 ? 2 : 1);
    return stream_launch(stream_h_kernel(N, S.c, S.v, stage, NB > 1), tiles, SL, q, chained);
  };
  // with the potential computed and a side stream given, the H psi passes before the
  // last (which reads phi) run on the side stream beside the convolution: they write
  // only the accumulator, the convolution only its scratch and phi
  const bool overlap = conv && side && ev_fork && ev_join;
  if (overlap) {
    CK(cudaEventRecord(ev_fork, st));
    CK(cudaStreamWaitEvent(side, ev_fork, 0));
    for (int st_ = 0; st_ < ndim - 1; ++st_) {
      int rc = hstage(st_, side, st_ > 0);
      if (rc) return rc;
    }
    CK(cudaEventRecord(ev_join, side));
  }
  if (conv) {
    int rc = stream_conv(SL, S, st);
    if (rc) return rc;
  }
  if (overlap) CK(cudaStreamWaitEvent(st, ev_join, 0));
  for (int st_ = overlap ? ndim - 1 : 0; st_ < ndim; ++st_) {
    int rc = hstage(st_, st, !overlap && st_ > 0);
    if (rc) return rc;
  }
  if (mu_dev) {
    k_stream_mu<NB><<<SL.ninst, 256, 0, st>>>(SL, tiles, mu_dev, mu_off);
  }
  CK(cudaGetLastError());
  return BGP_OK;
}

// Time every compiled (lines, factorization) candidate of line length N on this
// group, then the convolution's; keep the fastest (median of 3).
template <int NB>
int stream_autotune(bgp_plan::StreamSched& sc, SLaunchT<NB>& SL, bool conv, cudaStream_t st) {
  const int N = SL.insts[0].N;
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  auto timed = [&](const bgp_plan::StreamSched& s, bool with_conv, float* ms) -> int {
    float t[3];
    int rc = stream_run(SL, sched_of(s), with_conv, nullptr, 0, st);   // warm-up
    if (rc) return rc;
    for (int r = 0; r < 3; ++r) {
      CK(cudaEventRecord(e0, st));
      if ((rc = stream_run(SL, sched_of(s), with_conv, nullptr, 0, st))) return rc;
      CK(cudaEventRecord(e1, st));
      CK(cudaEventSynchronize(e1));
      CK(cudaEventElapsedTime(&t[r], e0, e1));
    }
    std::sort(t, t + 3);
    *ms = t[1];
    return BGP_OK;
  };
  int rc = BGP_OK;
  float best = 1e30f;
  sc.cand.clear();
  bgp_plan::StreamSched s = sc;
  for (int ln : {2, 4, 8}) {
    for (int v = 0; v < 2 && !rc; ++v) {
      float ms = 0.f;
      s.ln = ln; s.v = v;
      if ((rc = timed(s, false, &ms))) break;
      sc.cand.push_back({(float)ln, (float)v, 0.f, ms});
      if (ms < best) { best = ms; sc.ln = ln; sc.v = v; }
    }
  }
  if (conv && !rc) {
    float bc = 1e30f;
    s.ln = sc.ln; s.v = sc.v;
    for (int cln : {2, 4, 8}) {
      for (int csln : {4, 8}) {
        for (int cv : {0, 3}) {
          float ms = 0.f;
          s.cln = cln; s.csln = csln; s.cv = cv;
          if (cv == 3 && (2 * N) % 32 != 0) continue;
          if (rc || (rc = timed(s, true, &ms))) break;
          // negative lines: a convolution candidate
          sc.cand.push_back({(float)(-cln), (float)cv, (float)csln, ms});
          if (ms < bc) { bc = ms; sc.cln = cln; sc.csln = csln; sc.cv = cv; }
        }
      }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (!rc) sc.tuned = 1;
  return rc;
}

// the plan's side stream of size group g >= 1 (and its join event side_ev[g])
int side_stream(bgp_plan* p, int g, cudaStream_t* out) {
  while ((int)p->side_st.size() < g) {
    cudaStream_t q;
    CK(cudaStreamCreateWithFlags(&q, cudaStreamNonBlocking));
    p->side_st.push_back(q);
    cudaEvent_t e;
    CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    p->side_ev.push_back(e);
  }
  *out = p->side_st[g - 1];
  return BGP_OK;
}

// stream descriptor of instance i (the caller sets psi, H and phi)
void stream_inst(const bgp_plan* p, int i, SInst& S) {
  const Inst& I = p->inst[i];
  S = SInst{};                  // no given density, no partial sums (launch blocks start undefined)
  S.ndim = I.ndim; S.N = I.N; S.n = I.n; S.M = I.M;
  S.dx = I.dx; S.kfac = I.kfac; S.s = I.s; S.tc = I.tc; S.beta2 = I.beta2; S.beta3 = I.beta3;
  S.Omega = I.Omega; S.dv = I.dv;
  S.A = I.pool;                 // pool field 0 of the instance as the accumulator
  S.part = I.part;
  S.cb1 = I.cb1; S.cb2 = I.cb2; S.Kq = I.Kq; S.conv_scale = I.conv_scale;
  S.phi_out = I.phi2;           // computed potential: the instance's first potential field
  S.hscale = 1.0;
  S.twM = I.twM;
  for (int V = 0; V < kLVariants; ++V) {
    S.tabN[V] = p->lines[i].N[V];
    S.tabM[V] = p->lines[i].M[V];
  }
}
}  // namespace

namespace {
// ---------------------------------------------- single-instance operators
// One instance's launch block for the operators: psi as the state (and the density of
// a convolution).
void op_init(const bgp_plan* p, int i, const void* psi, SLaunchT<1>& SL) {
  SL.ninst = 1;
  stream_inst(p, i, SL.insts[0]);
  SL.insts[0].psi = (const double2*)psi;
}

// The same for the plain convolution out = dV (K * rho) of a given density.
void op_density(const bgp_plan* p, int i, const double* rho, double* out, int which_w, SLaunchT<1>& SL) {
  const Inst& I = p->inst[i];
  op_init(p, i, nullptr, SL);
  SInst& S = SL.insts[0];
  const double Md = (double)I.M;
  S.rho = rho;
  S.phi_out = out;
  S.Kq = which_w ? I.Wq : I.Kq;
  S.conv_scale = I.dv / (I.ndim == 2 ? Md * Md : Md * Md * Md);
}

// the list of totals one k_stream_sum launch forms
struct Sums {
  SumArgs A{};
  int n = 0;
  int add(const double* part, int cnt, double scale = 1.0, bool is_max = false) {
    A.part[n] = part; A.cnt[n] = cnt; A.scale[n] = scale; A.is_max[n] = is_max;
    return n++;
  }
  // totals on the host once the stream's work is done
  int run(bgp_plan* p, cudaStream_t st) {
    if (n) {
      A.out = p->d_sums;
      k_stream_sum<<<n, 256, 0, st>>>(A);
      CK(cudaGetLastError());
      p->launches++;
    }
    CK(cudaStreamSynchronize(st));
    return BGP_OK;
  }
};

// potential of the instance's state by the table Kq, and its sum against the density
// into the gpart section `sec`
int op_conv(bgp_plan* p, SLaunchT<1>& SL, const Sched& S, int sec, Sums* sums, int* slot, cudaStream_t st) {
  SInst& I = SL.insts[0];
  I.gpart = sums ? p->d_part + p->part_energy + sec * p->part_conv : nullptr;
  int rc = stream_conv(SL, S, st);
  if (rc) return rc;
  p->launches += I.ndim == 2 ? 3 : 5;
  if (sums) *slot = sums->add(I.gpart, (I.ndim == 2 ? I.N : I.N * I.N) / S.cr);
  return BGP_OK;
}

// H psi of the launch block (SL.insts[0].H, phi, part set)
int op_hpsi(bgp_plan* p, SLaunchT<1>& SL, const Sched& S, cudaStream_t st) {
  int rc = stream_run(SL, S, false, nullptr, 0, st);
  p->launches += SL.insts[0].ndim;
  return rc;
}

// the energy sums: total q of slot0 + q (kESums sums of every axis slot, then the peak)
struct EnergySlots { int first[3][kESums], peak; };
int op_energy(bgp_plan* p, SLaunchT<1>& SL, const Sched& S, Sums& sums, EnergySlots& es, cudaStream_t st) {
  SInst& I = SL.insts[0];
  const int C = S.c, tiles = I.n / (I.N * C), grid = tiles * I.ndim;
  double* keep = I.part;
  I.part = p->d_part;
  int rc = stream_launch(stream_energy_kernel(I.N, C, S.v), tiles, SL, st, false, I.ndim);
  I.part = keep;
  if (rc) return rc;
  p->launches++;
  for (int a = 0; a < I.ndim; ++a)
    for (int q = 0; q < kESums; ++q) {
      const bool spectral = q == E_K || q == E_L;
      es.first[a][q] = (a == 0 || spectral) ? sums.add(p->d_part + (size_t)q * grid + (size_t)a * tiles, tiles) : -1;
    }
  es.peak = sums.add(p->d_part + (size_t)kESums * grid, grid, 1.0, true);
  return BGP_OK;
}

// the record of energy_assemble from the totals
void op_energy_record(const bgp_plan* p, const Inst& I, const EnergySlots& es, double grav, double* rec) {
  const double* h = p->h_sums;
  for (int q = 0; q <= kNSum; ++q) rec[q] = 0.0;
  auto at = [&](int a, int q) { return h[es.first[a][q]]; };
  rec[S_N0] = at(0, E_N0); rec[S_V] = at(0, E_V); rec[S_2] = at(0, E_2); rec[S_3] = at(0, E_3);
  rec[S_R2] = at(0, E_R2); rec[S_PERP] = at(0, E_PERP); rec[S_Z2] = at(0, E_Z2);
  rec[S_KX] = at(1, E_K); rec[S_LX] = at(1, E_L);
  const int y = I.ndim == 2 ? 0 : 2;            // axis slot of the y lines
  rec[S_KY] = at(y, E_K); rec[S_LY] = at(y, E_L);
  if (I.ndim == 3) rec[S_KZ] = at(0, E_K);
  rec[S_G] = grav;
  rec[kNSum] = h[es.peak];
}

}  // namespace

extern "C" {

int bgp_apply_H(bgp_plan* p, int i, const void* psi, void* hpsi, const double* phi, int phi_mode,
                double* mu_out, void* stream) {
  int rc = check_inst(p, i);
  if (rc) return rc;
  if (!psi || !hpsi) return fail(BGP_ERR_ARG, "null field pointer");
  if (phi_mode == 1 && !phi) return fail(BGP_ERR_ARG, "phi_mode 1 needs phi");
  const Inst& I = p->inst[i];
  cudaStream_t st = (cudaStream_t)stream;
  const Sched S = sched_rule(I);
  SLaunchT<1> SL{};
  op_init(p, i, psi, SL);
  if (phi_mode == 2 && has_kernel(I)) {
    if ((rc = op_conv(p, SL, S, 0, nullptr, nullptr, st))) return rc;
    SL.insts[0].phi = I.phi2;
  } else {
    SL.insts[0].phi = phi_mode == 1 ? phi : nullptr;
  }
  SL.insts[0].H = (double2*)hpsi;
  if ((rc = op_hpsi(p, SL, S, st))) return rc;
  Sums sums;
  const int mu = sums.add(I.part, I.n / (I.N * S.c), I.dv);
  if ((rc = sums.run(p, st))) return rc;
  if (mu_out) *mu_out = p->h_sums[mu];
  return BGP_OK;
}

int bgp_energy(bgp_plan* p, int i, const void* psi, double* phi_out, bgp_energy_terms* terms,
               void* stream) {
  int rc = check_inst(p, i);
  if (rc) return rc;
  if (!psi || !terms) return fail(BGP_ERR_ARG, "null pointer");
  const Inst& I = p->inst[i];
  cudaStream_t st = (cudaStream_t)stream;
  const Sched S = sched_rule(I);
  SLaunchT<1> SL{};
  op_init(p, i, psi, SL);
  Sums sums;
  EnergySlots es;
  int grav = -1;
  if ((rc = op_energy(p, SL, S, sums, es, st))) return rc;
  if (has_kernel(I)) {
    if (phi_out) SL.insts[0].phi_out = phi_out;
    if ((rc = op_conv(p, SL, S, 0, &sums, &grav, st))) return rc;
  }
  if ((rc = sums.run(p, st))) return rc;
  double res[kNRec];
  op_energy_record(p, I, es, grav >= 0 ? p->h_sums[grav] : 0.0, res);
  op_terms(I, res, terms);
  return BGP_OK;
}

int bgp_energy_grad(bgp_plan* p, int i, const void* psi, bgp_energy_terms* terms, void* dE_dpsi,
                    double* dparams, void* stream) {
  int rc = check_inst(p, i);
  if (rc) return rc;
  if (!psi || !terms || !dparams) return fail(BGP_ERR_ARG, "null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  const Inst& I = p->inst[i];
  const Sched S = sched_rule(I);
  const bool kern = has_kernel(I), width = kern && I.kind == kQ2d && I.Wq;
  SLaunchT<1> SL{};
  op_init(p, i, psi, SL);
  Sums sums;
  EnergySlots es;
  int grav = -1, gravW = -1;
  if ((rc = op_energy(p, SL, S, sums, es, st))) return rc;
  if (width) {
    // dK/dl_z = -(K + W)/l_z, so dE/dl_z = -(Egrav + E_W)/l_z with E_W the energy of
    // the virial kernel's potential, of which only the sum is wanted
    SInst& Q = SL.insts[0];
    Q.Kq = I.Wq;
    Q.phi_out = nullptr;
    if ((rc = op_conv(p, SL, S, 1, &sums, &gravW, st))) return rc;
    Q.Kq = I.Kq;
    Q.phi_out = I.phi2;
  }
  if (kern && (rc = op_conv(p, SL, S, 0, &sums, &grav, st))) return rc;
  if (dE_dpsi) {
    // dE/dpsi* = H psi dV, with the potential of this psi
    SInst& Q = SL.insts[0];
    Q.phi = kern ? I.phi2 : nullptr;
    Q.H = (double2*)dE_dpsi;
    Q.hscale = I.dv;
    Q.part = nullptr;
    if ((rc = op_hpsi(p, SL, S, st))) return rc;
  }
  if ((rc = sums.run(p, st))) return rc;
  double res[kNRec];
  op_energy_record(p, I, es, grav >= 0 ? p->h_sums[grav] : 0.0, res);
  op_terms(I, res, terms);
  dparams[0] = 0.5 * res[S_2] * I.dv;                                       // dE/dbeta2
  dparams[1] = res[S_3] * I.dv / 3.0;                                       // dE/dbeta3
  dparams[2] = (kern && I.G_C != 0.0) ? terms->Egrav / I.G_C : 0.0;         // dE/dG_C
  dparams[3] = -terms->Lz;                                                  // dE/dOmega
  dparams[4] = 0.0;                                                         // dE/dl_z
  if (width) dparams[4] = -(terms->Egrav + 0.5 * p->h_sums[gravW] * I.dv) / p->desc[i].l_z;
  return BGP_OK;
}

int bgp_residual(bgp_plan* p, int i, const void* psi, double* out3, void* stream) {
  int rc = check_inst(p, i);
  if (rc) return rc;
  if (!psi || !out3) return fail(BGP_ERR_ARG, "null pointer");
  const Inst& I = p->inst[i];
  cudaStream_t st = (cudaStream_t)stream;
  const Sched S = sched_rule(I);
  SLaunchT<1> SL{};
  op_init(p, i, psi, SL);
  if (has_kernel(I)) {
    if ((rc = op_conv(p, SL, S, 0, nullptr, nullptr, st))) return rc;
    SL.insts[0].phi = I.phi2;
  }
  double2* H = I.pool + I.n;                     // pool field 1 (field 0 is the accumulator)
  SL.insts[0].H = H;
  if ((rc = op_hpsi(p, SL, S, st))) return rc;
  double* mu = p->d_res + (size_t)i * (kNRec + 1);
  k_stream_mu<1><<<1, 256, 0, st>>>(SL, I.n / (I.N * S.c), mu, 0);
  const int blocks = std::min(kResidBlocks, (I.n + kResidThreads - 1) / kResidThreads);
  k_stream_resid<<<blocks, kResidThreads, 0, st>>>((const double2*)psi, H, I.n, mu, p->d_part);
  CK(cudaGetLastError());
  p->launches += 2;
  Sums sums;
  const int s_mu = sums.add(mu, 1), s_r = sums.add(p->d_part, blocks);
  if ((rc = sums.run(p, st))) return rc;
  const double m = p->h_sums[s_mu], r = sqrt(p->h_sums[s_r] * I.dv);
  out3[0] = r;
  out3[1] = m;
  out3[2] = r / fmax(1.0, fabs(m));
  return BGP_OK;
}

int bgp_convolve(bgp_plan* p, int i, const double* rho, double* out, int which, void* stream) {
  int rc = check_inst(p, i);
  if (rc) return rc;
  const Inst& I = p->inst[i];
  if (I.M == 0) return fail(BGP_ERR_ARG, "instance has no long-range kernel");
  if (which == 1 && !I.Wq) return fail(BGP_ERR_ARG, "virial kernel exists for q2d only");
  if (!rho || !out) return fail(BGP_ERR_ARG, "null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  SLaunchT<1> SL{};
  op_density(p, i, rho, out, which, SL);
  if ((rc = op_conv(p, SL, sched_rule(I), 0, nullptr, nullptr, st))) return rc;
  CK(cudaStreamSynchronize(st));
  return BGP_OK;
}

// H psi of several instances of a plan, enqueued without host synchronisation
int bgp_apply_H_batch(bgp_plan* p, int n, const int* idx, const void* const* psi, void* const* hpsi,
                      const double* const* phi, int phi_mode, double* mu_dev, void* stream) {
  if (!p || n < 1 || !idx || !psi || !hpsi) return fail(BGP_ERR_ARG, "bad arguments");
  if (phi_mode < 0 || phi_mode > 2) return fail(BGP_ERR_ARG, "phi_mode must be 0, 1 or 2");
  if (phi_mode == 1 && !phi) return fail(BGP_ERR_ARG, "phi_mode 1 needs phi");
  cudaStream_t st = (cudaStream_t)stream;
  std::vector<int> seen(p->inst.size(), 0);
  for (int a = 0; a < n; ++a) {
    int rc = check_inst(p, idx[a]);
    if (rc) return rc;
    if (seen[idx[a]]++) return fail(BGP_ERR_ARG, "an instance appears twice in one batched apply");
    if (!psi[a] || !hpsi[a]) return fail(BGP_ERR_ARG, "null field pointer");
    if (psi[a] == hpsi[a]) return fail(BGP_ERR_ARG, "hpsi must not alias psi");
    if (phi_mode == 1 && !phi[a]) return fail(BGP_ERR_ARG, "phi_mode 1 needs phi for every instance");
  }
  // groups of equal (ndim, N, convolution on), in call order, at most kStreamBatch each;
  // the first runs on the caller's stream, each further one on a side stream that
  // waits for the work enqueued before the call and that the caller's stream waits for
  std::vector<char> done(n, 0);
  bool forks = n > kStreamBatch;               // more than one group
  for (int a = 1; a < n && !forks; ++a) {
    const Inst &A = p->inst[idx[0]], &B = p->inst[idx[a]];
    forks = A.ndim != B.ndim || A.N != B.N || (phi_mode == 2 && has_kernel(A) != has_kernel(B));
  }
  if (forks) {
    if (p->side_ev.empty()) {
      cudaEvent_t e;
      CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
      p->side_ev.push_back(e);
    }
    CK(cudaEventRecord(p->side_ev[0], st));    // the fork: the work enqueued before this call
  }
  int ngroup = 0;
  for (int a = 0; a < n; ++a) {
    if (done[a]) continue;
    const int gi = ngroup++;
    const Inst& A0 = p->inst[idx[a]];
    const bool conv = phi_mode == 2 && A0.kind != kNone && A0.M > 0;
    std::vector<int> grp;
    for (int b = a; b < n && (int)grp.size() < kStreamBatch; ++b) {
      const Inst& B = p->inst[idx[b]];
      const bool cb = phi_mode == 2 && B.kind != kNone && B.M > 0;
      if (!done[b] && B.ndim == A0.ndim && B.N == A0.N && cb == conv && (!conv || B.M == A0.M)) {
        grp.push_back(b);
        done[b] = 1;
      }
    }
    cudaStream_t gs = st;
    if (gi > 0) {
      int rc = side_stream(p, gi, &gs);
      if (rc) return rc;
      CK(cudaStreamWaitEvent(gs, p->side_ev[0], 0));
    }
    cudaStream_t os = nullptr;
    cudaEvent_t oe0 = nullptr, oe1 = nullptr;
    if (conv) {
      while ((int)p->ovl_st.size() <= gi) {
        cudaStream_t q;
        CK(cudaStreamCreateWithFlags(&q, cudaStreamNonBlocking));
        p->ovl_st.push_back(q);
        for (int e = 0; e < 2; ++e) {
          cudaEvent_t ev;
          CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
          p->ovl_ev.push_back(ev);
        }
      }
      os = p->ovl_st[gi]; oe0 = p->ovl_ev[2 * gi]; oe1 = p->ovl_ev[2 * gi + 1];
    }
    auto group = [&](auto& SL) -> int {
      SL.ninst = (int)grp.size();
      for (int g = 0; g < SL.ninst; ++g) {
        const int b = grp[g];
        const Inst& I = p->inst[idx[b]];
        SInst& S = SL.insts[g];
        stream_inst(p, idx[b], S);
        S.psi = (const double2*)psi[b];
        S.H = (double2*)hpsi[b];
        S.phi = conv ? I.phi2 : (phi_mode == 1 ? phi[b] : nullptr);
        if (!mu_dev) S.part = nullptr;         // (the sums cost the last pass of 256^3 4 %)
      }
      bgp_plan::StreamSched& sc = p->ssched[A0.N];
      if (sc.tuned == 0) {
        int rc = stream_autotune(sc, SL, conv, gs);
        if (rc) return rc;
      }
      const Sched S = sched_of(sc);
      if (!mu_dev) return stream_run(SL, S, conv, nullptr, 0, gs, os, oe0, oe1);
      // the mu kernel writes SL order; the group's members are consecutive in the
      // output only when the caller passed them so: write each one at its own index
      double* tmp = nullptr;
      if (!(grp.back() - grp.front() == (int)grp.size() - 1))
        CK(cudaMallocAsync((void**)&tmp, sizeof(double) * grp.size(), gs));
      int rc = stream_run(SL, S, conv, tmp ? tmp : mu_dev, tmp ? 0 : grp.front(), gs, os, oe0, oe1);
      if (!rc && tmp) {
        for (int g = 0; g < SL.ninst; ++g)
          CK(cudaMemcpyAsync(mu_dev + grp[g], tmp + g, sizeof(double), cudaMemcpyDeviceToDevice, gs));
      }
      if (tmp) cudaFreeAsync(tmp, gs);
      return rc;
    };
    int rc;
    if (grp.size() == 1) {
      SLaunchT<1> SL{};
      rc = group(SL);
    } else {
      SLaunch SL;
      rc = group(SL);
    }
    if (rc) return rc;
    if (gi > 0) CK(cudaEventRecord(p->side_ev[gi], gs));
    p->launches += conv ? (A0.ndim == 2 ? 3 : 5) + A0.ndim : A0.ndim;
  }
  // the join: the caller's stream waits for every side group
  for (int g = 1; g < ngroup; ++g) CK(cudaStreamWaitEvent(st, p->side_ev[g], 0));
  return BGP_OK;
}

int bgp_plan_stream_schedule(bgp_plan* p, int N, int* lines, int* radix_order, int* conv_lines,
                             int* conv_strided_lines, int* conv_order, int* tuned, float* cand, int* ncand) {
  if (!p) return fail(BGP_ERR_ARG, "null plan");
  auto it = p->ssched.find(N);
  const bgp_plan::StreamSched none;
  const bgp_plan::StreamSched& sc = it == p->ssched.end() ? none : it->second;
  if (lines) *lines = sc.ln;
  if (radix_order) *radix_order = sc.v;
  if (conv_lines) *conv_lines = sc.cln;
  if (conv_strided_lines) *conv_strided_lines = sc.csln;
  if (conv_order) *conv_order = sc.cv;
  if (tuned) *tuned = sc.tuned;
  if (ncand) {
    const int cap = *ncand;
    *ncand = (int)sc.cand.size();
    if (cand)
      for (int q = 0; q < (int)sc.cand.size() && q < cap; ++q)
        for (int c = 0; c < 4; ++c) cand[4 * q + c] = sc.cand[q][c];
  }
  return BGP_OK;
}

int bgp_plan_stream_set(bgp_plan* p, int N, int lines, int radix_order, int conv_lines, int conv_strided_lines,
                        int conv_order) {
  if (!p) return fail(BGP_ERR_ARG, "null plan");
  bgp_plan::StreamSched& sc = p->ssched[N];
  if (lines == 0) { sc.tuned = 0; sc.cand.clear(); return BGP_OK; }   // tune again on next use
  const bool known = stream_h_kernel(N, 8, 0, 0, false) != nullptr;
  if (!known || (lines != 1 && lines != 2 && lines != 4 && lines != 8 && lines != 16) || N % lines != 0 ||
      radix_order < 0 || radix_order > 7 || ((radix_order & 3) == 3 && N % 32 != 0))
    return fail(BGP_ERR_UNSUPPORTED, "schedule not available for this N");
  if (conv_lines != 1 && conv_lines != 2 && conv_lines != 4 && conv_lines != 8)
    return fail(BGP_ERR_ARG, "contiguous convolution lines per tile: 1, 2, 4 or 8");
  if (conv_strided_lines != 1 && conv_strided_lines != 2 && conv_strided_lines != 4 && conv_strided_lines != 8 &&
      conv_strided_lines != 16)
    return fail(BGP_ERR_ARG, "strided convolution lines per tile: 1, 2, 4, 8 or 16");
  if (conv_order != 0 && conv_order != 3) return fail(BGP_ERR_ARG, "convolution radix order: 0 or 3");
  if (conv_order == 3 && (2 * N) % 32 != 0) return fail(BGP_ERR_UNSUPPORTED, "convolution order 3 needs 2N = 32 R");
  if (conv_strided_lines == 16 && 2 * N == 768)
    return fail(BGP_ERR_UNSUPPORTED, "convolution tile width not available for this N");
  sc.ln = lines; sc.v = radix_order; sc.cln = conv_lines; sc.csln = conv_strided_lines; sc.cv = conv_order;
  sc.tuned = 2;
  return BGP_OK;
}

namespace {
// Cooperative launch of a Thomas-Fermi kernel over `grid` CTAs (one team). The status word
// stays as earlier launches left it: the host looks at it only every few steps.
int tf_launch(void* kern, int grid, void** args, bgp_plan* p, const Inst& I, cudaStream_t st) {
  CK(cudaMemsetAsync(I.bar, 0, sizeof(unsigned long long), st));
  CK(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(kThreads), args, 0, st));
  CK(cudaGetLastError());
  p->launches++;
  return BGP_OK;
}
// CTAs of the cluster that takes a Thomas-Fermi step of n points, 0 for the grid-wide
// launch. ms of 25 steps with the convolutions, cluster / grid: without a square root in
// the root (b3 = 0) 64^2 2.3 / 3.5, 128^2 2.8 / 3.5, 192^2 3.1 / 3.8, 256^2 about equal (3.5,
// on 16 SMs instead of 128), beyond it the grid; with one 64^2 2.9 / 4.7, 128^2 4.0 / 6.5,
// 256^2 8.3 / 6.1 (the FP64 units of 16 SMs).
int tf_cluster(int n, double b3) {
  if (n > kTfClMax * kTfClThreads * (b3 > 1e-30 ? 2 : kTfClHold)) return 0;
  return std::min(kTfClMax, (n + kTfClThreads - 1) / kTfClThreads);
}
// launch configuration of a Thomas-Fermi step by one cluster
struct TfClusterLaunch {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  TfClusterLaunch(int ctas, cudaStream_t st) {
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ctas; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.gridDim = dim3(ctas); cfg.blockDim = dim3(kTfClThreads); cfg.stream = st;
    cfg.attrs = &at; cfg.numAttrs = 1;
  }
  TfClusterLaunch(const TfClusterLaunch&) = delete;
};
// Whether the device can hold such a cluster: more than 8 CTAs are beyond what every
// device (or partition of one) schedules; the grid-wide launch takes the step where not.
// Asked once per device and size: the query takes longer than a launch.
bool tf_cluster_fits(DevCtx* d, int ctas) {
  signed char known = d->tf_fits[ctas].load(std::memory_order_relaxed);
  if (known == 0) {
    const TfClusterLaunch L(ctas, nullptr);
    int n = 0;
    const bool ok = (ctas <= 8 || cudaFuncSetAttribute(k_tf_iter_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
                    cudaOccupancyMaxActiveClusters(&n, k_tf_iter_cluster, &L.cfg) == cudaSuccess;
    if (!ok) cudaGetLastError();
    known = ok && n > 0 ? 1 : -1;
    d->tf_fits[ctas].store(known, std::memory_order_relaxed);
  }
  return known > 0;
}
int tf_launch_cluster(int ctas, TfArgs A, bgp_plan* p, cudaStream_t st) {
  const TfClusterLaunch L(ctas, st);
  CK(cudaLaunchKernelEx(&L.cfg, k_tf_iter_cluster, A));
  p->launches++;
  return BGP_OK;
}
}  // namespace

int bgp_tf_density(bgp_plan* p, int i, int nonlocal, double Omega, int iters, double relax, double* n_out,
                   double* info, void* stream) {
  int rc = check_inst(p, i);
  if (rc) return rc;
  if (!n_out || !info) return fail(BGP_ERR_ARG, "null pointer");
  const Inst I = p->inst[i];
  if (nonlocal && (I.M == 0 || I.kind == kNone)) return fail(BGP_ERR_ARG, "nonlocal Thomas-Fermi needs a long-range kernel");
  if (iters < 1) return fail(BGP_ERR_ARG, "iters must be positive");
  cudaStream_t st = (cudaStream_t)stream;
  // one team over the resident CTAs, at most the plan's grid (its partial-sum and
  // status buffers are sized for it)
  int nb = 0;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_tf_iter, kThreads, 0));
  int grid = std::min(nb * p->dev->sms, p->grid_cap);
  // no more CTAs than kTfHold points a thread keep busy: a barrier's arrivals queue on one
  // address (256^2, 25 steps: 5.8 ms with 4 points a thread, 6.3 with 2, 8.0 with 1)
  grid = std::min(grid, std::max(1, (I.n + kTfHold * kThreads - 1) / (kTfHold * kThreads)));
  if (grid < 1) return fail(BGP_ERR_CUDA, "Thomas-Fermi kernel does not fit on an SM");
  int ctas = tf_cluster(I.n, I.beta3);
  if (ctas && !tf_cluster_fits(p->dev, ctas)) ctas = 0;
  double* conv = I.phi2 + I.n;   // the plan's second potential field as the convolution output
  TfArgs A;
  memset(&A, 0, sizeof(A));
  A.ndim = I.ndim; A.N = I.N; A.n = I.n; A.mode = nonlocal ? 1 : 0;
  A.dx = I.dx; A.dv = I.dv; A.tc = I.tc; A.s = I.s; A.Omega = Omega;
  A.b2 = I.beta2; A.b3 = I.beta3; A.gc = I.G_C; A.relax = relax;
  A.conv = nonlocal ? conv : nullptr;
  A.nf = n_out; A.part = I.part; A.bar = I.bar; A.abort_flag = p->d_abort; A.state = p->d_tf;
  // state and, in the last place, the first status word (a copy to pageable memory takes 9 us)
  double h[kTfState + 1] = {NAN, INFINITY, 0.0, 0.0, 0.0};
  auto read_state = [&]() -> int {
    int ab = 0;
    CK(cudaMemcpyAsync(h, p->d_tf, sizeof(double) * kTfState + sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    memcpy(&ab, h + kTfState, sizeof(int));
    if (ab != 0 || h[2] == (double)kTfBarrier) return fail(BGP_ERR_DEVICE, "Thomas-Fermi kernel: team barrier timeout");
    return BGP_OK;
  };
  auto step = [&]() -> int {
    if (ctas) return tf_launch_cluster(ctas, A, p, st);
    void* args[] = {&A};
    return tf_launch((void*)k_tf_iter, grid, args, p, I, st);
  };
  CK(cudaMemcpyAsync(p->d_tf, h, sizeof(double) * kTfState, cudaMemcpyHostToDevice, st));
  CK(cudaMemsetAsync(p->d_abort, 0, (4 + (size_t)grid) * sizeof(int), st));
  if (!nonlocal) {
    if ((rc = step())) return rc;
    if ((rc = read_state())) return rc;
  } else {
    const double sigma = 0.15 * (I.dx * I.N / 2.0);   // 0.15 L
    double two_s2 = 2.0 * (sigma * sigma);
    void* sargs[] = {&A, &two_s2};
    if ((rc = tf_launch((void*)k_tf_seed, grid, sargs, p, I, st))) return rc;
    // the host looks at the state every kTfAhead steps (a step after the last one returns
    // at once): a wait per step was a tenth of the call, and much more on a busy host
    for (int it = 0; it < iters; ++it) {
      SLaunchT<1> SL{};
      op_density(p, i, n_out, conv, 0, SL);
      if ((rc = op_conv(p, SL, sched_rule(I), 0, nullptr, nullptr, st))) return rc;
      if ((rc = step())) return rc;
      if ((it + 1) % kTfAhead != 0 && it + 1 < iters) continue;
      if ((rc = read_state())) return rc;
      if (h[2] != (double)kTfOk || h[3] != 0.0) break;
    }
  }
  info[0] = (h[2] == (double)kTfNoBracket) ? NAN : h[0];   // mu
  info[1] = h[3];                                          // converged
  info[2] = h[1];                                          // final dn
  info[3] = h[4];                                          // steps taken
  info[4] = h[2];                                          // status
  return BGP_OK;
}

}  // extern "C"

namespace {
// ------------------------------------------------------------ stream solver
const SKernel* solver_kernel(int N, int cfg, int k) {
  switch (N) {
#define X(n) case n: return bgp_svptr_##n(cfg, k);
    BGP_FOR_STREAM_N(X)
#undef X
    default: return nullptr;
  }
}
const SKernel* solver_conv_kernel(int M, int cfg, int k) {
  switch (M) {
#define X(m) case m: return bgp_svcptr_##m(cfg, k);
    BGP_FOR_STREAM_M(X)
#undef X
    default: return nullptr;
  }
}
enum : int { SK_TRIAL, SK_HY, SK_HX, SK_PYF, SK_PZ, SK_PYI, SK_PX };           // order of the generated tables
enum : int { SC_FWD, SC_INV, SC_PB, SC_PC, SC_PD };

constexpr int kSvSteps = 4;      // solver steps of a plane group enqueued at a time

// instances of one (ndim, N, kernel): their launches share a stream
struct SvGroup {
  int ndim, N, M;
  std::vector<int> ids;          // active instances
  int act0 = 0;                  // their section of the plan's active list
  cudaStream_t st = nullptr;
  long long batches = 0;
  bool dirty = true;             // the device's list is to be written
};

int sv_launch(bgp_plan* p, const SvGroup& g, const SKernel* k, int tiles, bool chained) {
  if (!k) return fail(BGP_ERR_UNSUPPORTED, "solver pass not compiled for this size");
  if (k->smem > 48 * 1024)
    CK(cudaFuncSetAttribute(k->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k->smem));
  const int na = (int)g.ids.size();
  SvLaunch L{p->d_sv, p->d_ctl, p->d_svsync, p->d_act + g.act0, tiles, na, {}};
  for (int q = 0; q < na && na <= kSvInline; ++q) L.inl[q] = g.ids[q];
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)std::min((long long)tiles * na, (long long)k->per_sm * p->dev->sms));
  cfg.blockDim = dim3(k->threads);
  cfg.dynamicSmemBytes = k->smem;
  cfg.stream = g.st;
  cfg.attrs = &at;
  cfg.numAttrs = chained ? 1 : 0;
  void* args[] = {&L};
  CK(cudaLaunchKernelExC(&cfg, k->fn, args));
  p->launches++;
  return BGP_OK;
}

// A solver step of a group (see bgp_solve.cuh): the passes for which `want` has a state
// bit (every bit: a whole step).
int sv_step(bgp_plan* p, const SvGroup& g, bool chained, unsigned want = ~0u) {
  const int N = g.N, M = g.M, lines = g.ndim == 2 ? N : N * N;
  // tiles of 8 lines where half a million points fill the GPU with them; of 4 lines below,
  // with the most threads per line (a few elements each) while every tile has an SM to
  // itself. 256^2, us an iteration: alone 45 with the most threads, 53 with half as many;
  // four together 93 and 68.
  const int total = lines * (int)g.ids.size();
  const int cfg = (long long)total * N >= (1 << 19) ? 2 : (total / kSvSmall > p->dev->sms ? 1 : 0);
  const int C = cfg == 2 ? 8 : kSvSmall, t = lines / C;
  int rc = BGP_OK;
  auto has = [&](unsigned bits) { return (want & bits) != 0; };
  auto run = [&](int k, int tiles) { if (!rc) { rc = sv_launch(p, g, solver_kernel(N, cfg, k), tiles, chained); chained = true; } };
  auto crun = [&](int k, int tiles) { if (!rc) { rc = sv_launch(p, g, solver_conv_kernel(M, cfg, k), tiles, chained); chained = true; } };
  auto conv = [&]() {
    const int tpl = (N + 1 + C - 1) / C;
    crun(SC_FWD, t);
    if (g.ndim == 3) crun(SC_PB, N * tpl);
    crun(SC_PC, (g.ndim == 2 ? 1 : M) * tpl);
    if (g.ndim == 3) crun(SC_PD, N * tpl);
    crun(SC_INV, t);
  };
  constexpr unsigned kTrial = 1u << ST_TRIAL | 1u << ST_INIT | 1u << ST_FINAL | 1u << ST_SWITCH, kH = 1u << ST_H | 1u << ST_MED;
  if (g.ndim == 2) {
    run(SK_TRIAL, 2 * t);
    if (M) conv();                       // the trial state's own potential
    run(SK_HX, t);
    run(SK_PZ, t);
    run(SK_PX, t);
    return rc;
  }
  // a volume's potential (of the first, refreshed or returned state), then gradient,
  // preconditioner and direction, the line search's two convolutions and its first trial
  if (M && has(1u << ST_CONV)) conv();
  if (has(1u << ST_CONV | kH)) { if (has(1u << ST_CONV | 1u << ST_H)) run(SK_HY, t); run(SK_HX, t); }
  if (has(1u << ST_CONV | kH | 1u << ST_PRE)) { run(SK_PYF, t); run(SK_PZ, t); run(SK_PYI, t); run(SK_PX, t); }
  if (M && has(1u << ST_CONV | kH | 1u << ST_PRE | 1u << ST_POLYB)) conv();
  if (M && has(1u << ST_CONV | kH | 1u << ST_PRE | 1u << ST_POLYB | 1u << ST_POLYC)) conv();
  if (has(1u << ST_CONV | kH | 1u << ST_PRE | 1u << ST_POLYB | 1u << ST_POLYC | kTrial)) run(SK_TRIAL, 3 * t);
  return rc;
}

// the stream solver's state of a plan, allocated by its first mixed solve
int sv_alloc(bgp_plan* p) {
  const int n = (int)p->inst.size();
  int rc = BGP_OK;
  if ((rc = palloc_t(p, (size_t)n, &p->d_sv))) return rc;
  if ((rc = palloc_t(p, (size_t)n, &p->d_ctl))) return rc;
  if ((rc = palloc_t(p, (size_t)n, &p->d_svsync))) return rc;
  if ((rc = palloc_t(p, (size_t)n * kSvBins, &p->d_svhist))) return rc;
  if ((rc = palloc_t(p, (size_t)n * kSvCap, &p->d_svcand))) return rc;
  if ((rc = palloc_t(p, (size_t)n, &p->d_act))) return rc;
  for (const Inst& I : p->inst) {
    // kDSums lists (the most a pass has) over its tiles of at least kSvSmall lines
    double* q = nullptr;
    if ((rc = palloc_t(p, (size_t)kDSums * (I.n / I.N / kSvSmall), &q))) return rc;
    p->svpart.push_back(q);
  }
  if (!pin_take(p->dev->device, sizeof(int) * n, &p->pin_state))
    return fail(BGP_ERR_OOM, "pinned host memory for the solver's flags");
  if ((rc = zeroed())) return rc;
  p->h_state = (int*)p->pin_state.host;
  p->d_state = (int*)p->pin_state.dev;
  return BGP_OK;
}
int sv_prepare(bgp_plan* p) {
  if (p->h_state) return BGP_OK;
  const size_t had = p->allocs.size();
  const long long bytes = p->bytes;
  const int rc = sv_alloc(p);
  if (rc) {                               // all or nothing: the next solve starts over
    for (size_t k = had; k < p->allocs.size(); ++k) cudaFree(p->allocs[k]);
    p->allocs.resize(had);
    p->bytes = bytes;
    p->svpart.clear();
    p->d_sv = nullptr;
    pin_give(&p->pin_state);
  }
  return rc;
}

// All instances of the plan in the mixed form: results in p->d_out once the stream's work
// is done.
int sv_solve(bgp_plan* p, const void* const* psi0, void* const* psi_out, const SolverParams& P, double* d_trace,
             cudaStream_t st) {
  const int n = (int)p->inst.size();
  if (n > p->grid_cap) return fail(BGP_ERR_ARG, "more instances than resident CTAs in one batch");
  int prc = sv_prepare(p);
  if (prc) return prc;
  std::vector<SvInst> hi(n);
  std::vector<SvCtl> hc(n);
  std::vector<SvGroup> groups;
  for (int i = 0; i < n; ++i) {
    const Inst& I = p->inst[i];
    SvInst& S = hi[i];
    memset(&S, 0, sizeof(S));
    S.ndim = I.ndim; S.N = I.N; S.n = I.n; S.M = I.M;
    S.kern = has_kernel(I); S.poly = S.kern && I.ndim == 3;
    S.dx = I.dx; S.dv = I.dv; S.kfac = I.kfac; S.s = I.s; S.tc = I.tc;
    S.beta2 = I.beta2; S.beta3 = I.beta3; S.Omega = I.Omega; S.inv_n = I.inv_n; S.conv_scale = I.conv_scale;
    S.pool = I.pool; S.phi2 = I.phi2; S.cb1 = I.cb1; S.cb2 = I.cb2; S.Kq = I.Kq; S.twM = I.twM;
    for (int V = 0; V < kLVariants; ++V) {
      S.tabN[V] = p->lines[i].N[V];
      S.tabF[V] = p->lines[i].F[V];
      S.tabM[V] = p->lines[i].M[V];
    }
    S.keys = I.keys;
    S.wcand = p->d_svcand + (size_t)i * kSvCap;
    S.hist = p->d_svhist + (size_t)i * kSvBins;
    S.part = p->svpart[i];
    S.in_psi = (const double2*)psi0[i];
    S.out_c = (double2*)psi_out[i];
    S.sp = P;
    S.trace = d_trace ? d_trace + (size_t)3 * P.trace_cap * i : nullptr;
    S.out = p->d_out + i;
    S.hstate = p->d_state + i;
    SvCtl& c = hc[i];
    memset(&c, 0, sizeof(c));
    c.st = ST_INIT; c.kind = KD_INIT;
    for (int q = 0; q < F_NLOG; ++q) { c.f[q] = -1; c.sc[q] = 1.0; }
    c.f[F_A] = 0; c.f[F_H] = 1; c.f[F_W] = 2;
    c.hf = -1;
    c.fp32 = 1; c.fp64_from = -1;
    c.phisc = 1.0;
    c.stop = kStopMaxit;
    c.alpha = P.alpha0; c.sigma = P.shift_min; c.med_eps = 1e-3;
    ((volatile int*)p->h_state)[i] = ST_INIT;
    const int M = S.kern ? I.M : 0;
    SvGroup* g = nullptr;
    for (SvGroup& q : groups) if (q.ndim == I.ndim && q.N == I.N && q.M == M) g = &q;
    if (!g) { groups.emplace_back(); g = &groups.back(); g->ndim = I.ndim; g->N = I.N; g->M = M; }
    g->ids.push_back(i);
  }
  CK(cudaMemcpyAsync(p->d_sv, hi.data(), sizeof(SvInst) * n, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(p->d_ctl, hc.data(), sizeof(SvCtl) * n, cudaMemcpyHostToDevice, st));
  CK(cudaMemsetAsync(p->d_svhist, 0, sizeof(unsigned) * kSvBins * (size_t)n, st));
  CK(cudaMemsetAsync(p->d_svsync, 0, sizeof(SvSync) * (size_t)n, st));
  // the first group on the caller's stream, the others on side streams that start after
  // the work enqueued so far
  if (p->side_ev.empty()) {
    cudaEvent_t e;
    CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    p->side_ev.push_back(e);
  }
  CK(cudaEventRecord(p->side_ev[0], st));
  int act0 = 0;
  for (size_t q = 0; q < groups.size(); ++q) {
    SvGroup& g = groups[q];
    g.act0 = act0;
    act0 += (int)g.ids.size();
    g.st = st;
    if (q > 0) {
      int rc = side_stream(p, (int)q, &g.st);
      if (rc) return rc;
      CK(cudaStreamWaitEvent(g.st, p->side_ev[0], 0));
    }
    while (p->sv_ev.size() < 2 * (q + 1)) {
      cudaEvent_t e;
      CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
      p->sv_ev.push_back(e);
    }
  }
  // every step ends an iteration, a trial or a level of a median search of each of its
  // instances, so this many batches are enough for any solve
  const long long most = ((long long)P.maxit + 4) * ((long long)std::max(P.ls_max, 1) + 16) + 16;
  for (bool busy = true; busy;) {
    busy = false;
    for (size_t q = 0; q < groups.size(); ++q) {
      SvGroup& g = groups[q];
      if (g.ids.empty()) continue;
      // planes: whole steps, the host two batches behind (a pass is a few us). Volumes: a
      // pass is tens of us and a skipped one a few, so the host waits for the state after
      // every trial and enqueues what it asks for
      const bool direct = g.ndim == 3;
      cudaEvent_t ev = p->sv_ev[2 * q + (direct ? 0 : g.batches & 1)];
      if (g.batches >= (direct ? 1 : 2)) CK(cudaEventSynchronize(ev));
      std::vector<int> left;
      for (int i : g.ids) if (((volatile int*)p->h_state)[i] != ST_DONE) left.push_back(i);
      if (left.size() != g.ids.size()) { g.ids.swap(left); g.dirty = true; }
      if (g.ids.empty()) continue;
      if (g.batches > most) return fail(BGP_ERR_DEVICE, "solve did not finish within its step limit");
      busy = true;
      if (g.dirty)
        CK(cudaMemcpyAsync(p->d_act + g.act0, g.ids.data(), sizeof(int) * g.ids.size(), cudaMemcpyHostToDevice, g.st));
      unsigned want = direct ? 0u : ~0u;
      if (direct) for (int i : g.ids) want |= 1u << ((volatile int*)p->h_state)[i];
      for (int s = 0; s < (direct ? 1 : kSvSteps); ++s) {
        int rc = sv_step(p, g, !(s == 0 && g.dirty), want);
        if (rc) return rc;
        g.dirty = false;
      }
      CK(cudaEventRecord(ev, g.st));
      g.batches++;
    }
  }
  for (size_t q = 1; q < groups.size(); ++q) {
    CK(cudaEventRecord(p->side_ev[q], groups[q].st));
    CK(cudaStreamWaitEvent(st, p->side_ev[q], 0));
  }
  return BGP_OK;
}
}  // namespace

extern "C" {

int bgp_solve(bgp_plan* p, const void* const* psi0, void* const* psi_out, const bgp_solver_params* sp,
              bgp_solve_result* results, double* trace, void* stream) {
  if (!p || !psi0 || !psi_out || !sp || !results) return fail(BGP_ERR_ARG, "null pointer");
  static_assert(sizeof(SolveOut) == sizeof(bgp_solve_result), "result layout");
  const int n = (int)p->inst.size();
  cudaStream_t st = (cudaStream_t)stream;
  SolverParams P{};
  P.maxit = sp->maxit; P.ls_max = sp->linesearch_max; P.stall_max = sp->linesearch_stall < 1 ? 1 : sp->linesearch_stall;
  P.restart = sp->cg_restart; P.cg_beta = sp->cg_beta; P.window = sp->conv_window;
  P.record_trace = sp->record_trace; P.trace_cap = sp->trace_cap;
  P.res_tol = sp->res_tol; P.etol = sp->energy_tol; P.alpha0 = sp->step; P.alpha_min = 1e-8;
  P.alpha_max = sp->step_max; P.shift_min = sp->precond_shift_min; P.c1 = 1e-4; P.shrink = 0.5;
  P.growth = 1.1; P.bb_min = 0.05; P.bb_max = sp->step_max; P.bb_mix = 0.5;
  // a line search of no trials never leaves the initial state: there is nothing for the
  // mixed form's launches (a trial each) to do
  P.mixed = sp->mixed && sp->linesearch_max > 0 ? 1 : 0; P.mixed_tol = sp->mixed_switch_res;
  if (P.cg_beta < 0 || P.cg_beta > 2) return fail(BGP_ERR_ARG, "cg_beta must be 0, 1 or 2");
  if (P.maxit < 0) return fail(BGP_ERR_ARG, "maxit must be >= 0");
  double* d_trace = nullptr;
  if (P.record_trace && P.trace_cap > 0) {
    CK(cudaMallocAsync((void**)&d_trace, sizeof(double) * 3 * (size_t)P.trace_cap * n, st));
  } else {
    P.record_trace = 0;
  }
  std::vector<Inst> save = p->inst;
  std::vector<int> act(n);
  for (int i = 0; i < n; ++i) {
    if (!psi0[i] || !psi_out[i]) return fail(BGP_ERR_ARG, "null field pointer");
    Inst& I = p->inst[i];
    I.prog = kProgSolve;
    I.in_psi = (const double2*)psi0[i];
    I.out_c = (double2*)psi_out[i];
    I.sp = P;
    I.trace = d_trace ? d_trace + (size_t)3 * P.trace_cap * i : nullptr;
    I.resume = 0;
    I.finished = p->d_finished;
    act[i] = i;
  }
  CK(cudaMemsetAsync(p->d_out, 0, sizeof(SolveOut) * n, st));
  // Segmented solve: each launch runs until a quarter of its instances have
  // finished; the others save their state and are relaunched with larger teams,
  // so the instances that need the most iterations soon get the whole GPU.
  int rc = BGP_OK;
  std::vector<SolveOut> outs(n);
  const bool tuning = !P.mixed && p->tune == 1 && n > 1;   // the mixed form has no relaunches
  const int ydiv = tuning ? kTuneYield[p->tune_next] : p->yield_div;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  if (tuning) {
    CK(cudaEventCreate(&ev0));
    CK(cudaEventCreate(&ev1));
    CK(cudaEventRecord(ev0, st));
  }
  if (P.mixed) {
    rc = sv_solve(p, psi0, psi_out, P, d_trace, st);
    act.clear();
    if (rc) cudaDeviceSynchronize();   // nothing of it may still run when the call returns
  }
  for (int seg = 0; !act.empty() && seg < kMaxSegments; ++seg) {
    const int na = (int)act.size();
    const int yield_at = na > 1 ? std::max(1, na / ydiv) : (1 << 30);
    for (int a : act) p->inst[a].yield_at = yield_at;
    CK(cudaMemsetAsync(p->d_finished, 0, sizeof(int), st));
    rc = launch(p, act, st);
    if (rc) break;
    CK(cudaMemcpyAsync(outs.data(), p->d_out, sizeof(SolveOut) * n, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    std::vector<int> next;
    for (int a : act) {
      if (outs[a].status == 2) {
        next.push_back(a);
        p->inst[a].resume = 1;
      }
    }
    act.swap(next);
  }
  p->inst = save;
  if (tuning) {
    float ms = 0.f;
    if (!rc && act.empty()) {
      CK(cudaEventRecord(ev1, st));
      CK(cudaEventSynchronize(ev1));
      CK(cudaEventElapsedTime(&ms, ev0, ev1));
      p->tune_ms[p->tune_next++] = ms;
      if (p->tune_next == 3) {
        int best = 0;
        for (int c = 1; c < 3; ++c) if (p->tune_ms[c] < p->tune_ms[best]) best = c;
        p->yield_div = kTuneYield[best];
        p->tune = 2;
      }
    }
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
  }
  if (!rc && !act.empty()) rc = fail(BGP_ERR_DEVICE, "solve did not finish within the relaunch limit");
  if (rc) { if (d_trace) cudaFreeAsync(d_trace, st); return rc; }
  CK(cudaMemcpyAsync(results, p->d_out, sizeof(SolveOut) * n, cudaMemcpyDeviceToHost, st));
  if (d_trace && trace)
    CK(cudaMemcpyAsync(trace, d_trace, sizeof(double) * 3 * (size_t)P.trace_cap * n, cudaMemcpyDeviceToHost, st));
  if (d_trace) CK(cudaFreeAsync(d_trace, st));
  CK(cudaStreamSynchronize(st));
  for (int i = 0; i < n; ++i)
    if (results[i].status != 0) return fail(BGP_ERR_DEVICE, "a solver team stopped on a device error");
  return BGP_OK;
}

}  // extern "C"
