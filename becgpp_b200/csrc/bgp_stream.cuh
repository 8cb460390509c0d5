// Stream passes: the Hamiltonian apply, the zero-padded convolution, the energy sums
// and the residual as plain (non-persistent) launches, one launch per axis pass over
// every tile of every instance of a batch, for every entry point but the solver's.
//
// Unlike the solver's persistent team kernel, a stream pass needs no team
// barrier: the launch boundary orders the passes, so all SMs work on one pass at
// a time and nothing waits on the host. Each pass is templated on
//   L   the line length (N, or M = 2 N for the padded axes),
//   C   the lines per tile. On a strided axis a tile groups C neighbours along the
//       contiguous axis, so each of its rows is 16 C contiguous bytes,
//   V   the line's factorization (bgp_lfft.cuh),
//   NB  the instances the launch parameters hold (1, or a batch),
// and the host's autotuner times the compiled (C, V) candidates of a plan's grid
// size on its own data and keeps the fastest.
//
// A line lives in the registers of T = L / E threads from its load to its store
// (bgp_lfft.cuh); shared memory only carries the exchanges between radix stages.
//
// H psi of an instance (operators.py:36-45 of the reference) is a sum of
// per-axis terms: along a y-line the multiplier (k_y^2/2 - Omega x k_y), along an
// x-line (k_x^2/2 + Omega y k_x), along z k_z^2/2, each applied by a forward and
// an inverse line FFT. The passes accumulate them in a scratch field A; the last
// pass adds (V + b2 rho + b3 rho^2 + phi) psi, writes H psi and each CTA's part
// of Re<psi, H psi>.
//
// The passes of one apply are a chain of programmatic dependent launches: a pass
// lets its successor start as soon as all its CTAs run, and waits for its
// predecessor only where it first reads what that wrote. The later H psi passes
// transform psi, which no pass writes, before that point, so on a grid too small to
// fill the GPU the passes of an apply overlap.
#pragma once
#include "bgp_device.cuh"
#include "bgp_lfft.cuh"

BGP_NS_BEGIN

// One instance of a stream batch (device copy).
struct SInst {
  int ndim, N, n, M;
  double dx, kfac, s, tc, beta2, beta3, Omega, dv;
  const double2* psi;     // input state
  double2* A;             // per-axis accumulator (scratch, n)
  double2* H;             // output H psi
  const double* phi;      // long-range potential (n) or null
  double* part;           // per-tile partial sums of Re<psi, H psi> (last pass)
  // zero-padded convolution (phi from |psi|^2): scratch and kernel quadrant
  double2* cb1;           // 2D: N x Mp; 3D: N x N x Mp    (Mp = conv_pitch(N))
  double2* cb2;           // 3D: N x M x Mp
  const double* Kq;       // real even quadrant of the kernel transform, (Mh)^d
  double* phi_out;        // computed potential (n), or null (only its sum is wanted)
  double conv_scale;      // -G_C dV / M^d
  const double* rho;      // the convolution's density, or null: |psi|^2
  double* gpart;          // per-tile partial sums of phi rho (last convolution pass), or null
  double hscale;          // H psi is written times this
  const double2* twM;     // w_M^t, t < M
  const double2* tabN[kLVariants];   // line-transform tables (lf_fill_table)
  const double2* tabM[kLVariants];
};

// A launch of one pass over up to NB instances of one size, passed by value (kernel
// parameter space), so nothing is staged in device memory per call. A single
// instance has its own, small parameter block: the 64-instance block is 17 KB that
// every launch would copy.
constexpr int kStreamBatch = 64;
template <int NB>
struct SLaunchT {
  SInst insts[NB];
  int ninst;
  int tiles;              // tiles of one instance in this pass
};
using SLaunch = SLaunchT<kStreamBatch>;

// Row pitch of the convolution scratch: N + 1 spectral columns, rows of whole
// 128-byte lines (N is a multiple of 8), so a tile's rows are aligned.
BGP_HD constexpr int conv_pitch(int N) { return N + 8; }

// lines per tile with the CTA filled up to a warp (the lines beyond C idle)
BGP_HD constexpr int s_cp(int L, int C, int V) { return C * lf_threads(L, V) >= 32 ? C : 32 / lf_threads(L, V); }
BGP_HD constexpr int s_threads(int L, int C, int V) { return s_cp(L, C, V) * lf_threads(L, V); }
BGP_HD constexpr size_t s_smem(int L, int C, int V) { return (size_t)s_cp(L, C, V) * lf_slots(L, V) * 16; }
// resident threads per SM the registers are budgeted for: 24 values a thread need
// about 170 registers, 16 or 12 fit in 128, 8 in 80
BGP_HD constexpr int s_min_blocks(int L, int C, int V) {
  const int E = lplan(L, V).E, want = E > 16 ? 384 : (E > 8 ? 512 : 768);
  const int b = want / s_threads(L, C, V);
  return b < 1 ? 1 : (b > 16 ? 16 : b);
}

// A compiled pass: its entry and launch geometry (evaluated at compile time).
struct SKernel {
  void* fn;
  int threads;
  size_t smem;
  int per_sm;             // CTAs per SM the registers are budgeted for
};

#if defined(__CUDACC__)

// programmatic dependent launch: let the next pass start; wait for the previous one
BGP_D void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }
BGP_D void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Thread and buffer layout of a tile: on the contiguous axis the T threads of a line
// are neighbours (and, for T <= 32, in one warp); on a strided axis the lines are.
template <int L, int C, int V, bool CONTIG>
struct Tile {
  static constexpr int T = lf_threads(L, V), CP = s_cp(L, C, V), E = lplan(L, V).E;
  static constexpr bool WARP = CONTIG && T <= 32;
  using Fft = LineFft<L, V, CONTIG ? 1 : CP, WARP>;
  int c, t;
  BGP_D Tile() {
    const int tid = threadIdx.x;
    c = CONTIG ? tid / T : tid % CP;
    t = CONTIG ? tid % T : tid / CP;
  }
  template <class F = double2>
  BGP_D F* line(double2* sm) const { return reinterpret_cast<F*>(sm) + (CONTIG ? c * lf_slots(L, V) : c); }
};

// Sums of NV values over the CTA (W warps) in a fixed order; thread 0 holds the totals.
template <int W, int NV>
BGP_D void block_sums(double (&v)[NV]) {
  __shared__ double red[NV * W];
#pragma unroll
  for (int q = 0; q < NV; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  }
  if constexpr (W > 1) {
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
      for (int q = 0; q < NV; ++q) red[q * W + (threadIdx.x >> 5)] = v[q];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        double s = 0.0;
        for (int w = 0; w < W; ++w) s += red[q * W + w];
        v[q] = s;
      }
    }
  }
}

// --------------------------------------------------------------- H psi pass
// STAGE 0: A = T(psi) on the contiguous axis; 1: A += T(psi) (3D, middle axis);
// 2: H = A + T(psi) + (V + b2 rho + b3 rho^2 + phi) psi and the CTA's part of
// Re<psi, H> (axis 0). T = inverse FFT o multiplier o forward FFT along the axis.
//
// Bound: 256^3 moves 268 MB per field and pass and is bound by HBM; a single plane
// grid is a few microseconds of latency (one tile per CTA).
template <int N, int C, int V, int STAGE, int NB>
__global__ void __launch_bounds__(s_threads(N, C, V), s_min_blocks(N, C, V))
    k_stream_h(const __grid_constant__ SLaunchT<NB> SL) {
  constexpr bool CONTIG = STAGE == 0;
  using TL = Tile<N, C, V, CONTIG>;
  constexpr int E = TL::E, T = TL::T;
  extern __shared__ double2 sm[];
  const int inst = NB == 1 ? 0 : blockIdx.x / SL.tiles, tile = blockIdx.x - inst * SL.tiles;
  const SInst& I = SL.insts[inst];
  const TL tl;
  const int c = tl.c, t = tl.t, ndim = I.ndim;
  const bool valid = c < C;
  pdl_trigger();
  // line (i, j[, k]) of this thread: element r at base + r * str; its coordinate across
  // the rotation plane (xo) and, for the trap, the squared radius of the fixed axes
  int base, str, ci = 0, cj = 0, ck = 0;
  if (STAGE == 0) {
    const int line = tile * C + c;
    base = line * N; str = 1;
    ci = line;                                   // 2D: i = line
  } else if (ndim == 2) {
    cj = tile * C + c;
    base = cj; str = N;
  } else {
    constexpr int tpl = N / C;
    const int a = tile / tpl;
    ck = (tile - a * tpl) * C + c;
    if (STAGE == 1) { ci = a; base = a * N * N + ck; str = N; }
    else { cj = a; base = a * N + ck; str = N * N; }
  }
  const double2* __restrict__ psi = I.psi;
  double2 v[E];
#pragma unroll
  for (int q = 0; q < E; ++q) v[q] = valid ? __ldg(psi + base + (t + T * q) * str) : cmk(0.0, 0.0);
  const typename TL::Fft fft{tl.line(sm), I.tabN[V], t};
  fft.template forward<false>(v);
  {
    const double dx = I.dx, Om = I.Omega, kf = I.kfac, inv = 1.0 / (double)N;
    double wx = 0.0;                             // y-line: -Omega x(i); x-line: +Omega y(j)
    if (STAGE == 2) wx = Om * ((double)(cj - N / 2) * dx);
    else if (STAGE == 1 || ndim == 2) wx = -Om * ((double)(ci - N / 2) * dx);
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int r = t + T * q, mm = (r < (N + 1) / 2) ? r : r - N;
      const double kk = kTwoPi * ((double)mm * kf);
      v[q] = cscale(v[q], (0.5 * kk * kk + wx * kk) * inv);
    }
  }
  fft.template inverse<false>(v);
  if (STAGE > 0) pdl_wait();                     // A, and phi, come from the passes before
  double acc = 0.0;
  constexpr int CH = E % 4 == 0 ? 4 : 3;         // elements in flight on the way out
#pragma unroll
  for (int q0 = 0; q0 < E; q0 += CH) {
    double2 pa[CH], pv[CH];
    double pp[CH];
#pragma unroll
    for (int u = 0; u < CH; ++u) {
      const int f = base + (t + T * (q0 + u)) * str;
      if (STAGE > 0) pa[u] = valid ? I.A[f] : cmk(0.0, 0.0);
      if (STAGE == 2) {
        pv[u] = valid ? __ldg(psi + f) : cmk(0.0, 0.0);
        pp[u] = (valid && I.phi) ? I.phi[f] : 0.0;
      }
    }
#pragma unroll
    for (int u = 0; u < CH; ++u) {
      const int r = t + T * (q0 + u), f = base + r * str;
      if (STAGE == 0) { if (valid) I.A[f] = v[q0 + u]; continue; }
      const double2 a2 = cadd(pa[u], v[q0 + u]);
      if (STAGE == 1) { if (valid) I.A[f] = a2; continue; }
      const double2 p = pv[u];
      const double rho = cabs2(p);
      // trap tc r^s from the indices (becgpp/grid.py:90-91)
      const double x = (double)(r - N / 2) * I.dx, y = (double)(cj - N / 2) * I.dx;
      double r2 = x * x + y * y;
      if (ndim == 3) { const double z = (double)(ck - N / 2) * I.dx; r2 = r2 + z * z; }
      const double Vt = (I.s <= 0.0) ? 0.0 : ((I.s == 2.0) ? I.tc * r2 : I.tc * pow(r2, 0.5 * I.s));
      const double pot = Vt + I.beta2 * rho + I.beta3 * rho * rho + pp[u];
      const double2 h = cadd(a2, cscale(p, pot));
      if (valid) I.H[f] = cscale(h, I.hscale);
      acc += p.x * h.x + p.y * h.y;
    }
  }
  if (STAGE == 2 && I.part) {
    double g[1] = {acc};
    block_sums<s_threads(N, C, V) / 32, 1>(g);
    if (threadIdx.x == 0) I.part[tile] = g[0];
  }
}

// ------------------------------------------------- zero-padded convolution
// phi = conv_scale (K * rho) on the N^d grid, cyclic in the M^d box (M = 2 N). The
// grid sits at the box's origin (a cyclic convolution commutes with the shift), so the
// upper half of every padded line is zero on the way in and unused on the way out.
//   step a  lines of the last axis: real transform, columns kk <= N kept   -> cb1
//   2D: columns along i: forward, times K^, inverse, rows i < N            -> cb1
//   3D: step b (along j) cb1 -> cb2, step c (along i: forward, K^, inverse) in cb2,
//       step d (inverse along j) cb2 -> cb1
//   last    lines of the last axis: inverse real transform, phi
// A real line of M points is one complex transform of N: z_n = x_2n + i x_(2n+1), and
//   X_k = E_k + w_M^k O_k,  E_k = (Z_k + conj Z_(N-k)) / 2,  O_k = (Z_k - conj Z_(N-k)) / 2i.

// two neighbouring values of a caller's field of doubles: one access where the field
// starts on 16 bytes (a contiguous slice of a larger array need not)
BGP_D bool on16(const double* p) { return ((size_t)p & 15) == 0; }
BGP_D double2 load_pair(const double* p, bool wide) {
  return wide ? __ldg(reinterpret_cast<const double2*>(p)) : cmk(__ldg(p), __ldg(p + 1));
}
BGP_D void store_pair(double* p, double2 v, bool wide) {
  if (wide) *reinterpret_cast<double2*>(p) = v;
  else { p[0] = v.x; p[1] = v.y; }
}

// step a (INV = 0) and the last step (INV = 1)
template <int N, int C, int V, int INV, int NB>
__global__ void __launch_bounds__(s_threads(N, C, V), s_min_blocks(N, C, V))
    k_stream_real(const __grid_constant__ SLaunchT<NB> SL) {
  using TL = Tile<N, C, V, true>;
  constexpr int E = TL::E, T = TL::T, Mp = conv_pitch(N);
  extern __shared__ double2 sm[];
  const int inst = NB == 1 ? 0 : blockIdx.x / SL.tiles, tile = blockIdx.x - inst * SL.tiles;
  const SInst& I = SL.insts[inst];
  const TL tl;
  const int t = tl.t, line = tile * C + tl.c;
  const bool valid = tl.c < C;
  double2* b = tl.line(sm);
  const typename TL::Fft fft{b, I.tabN[V], t};
  const double2* __restrict__ tw = I.twM;
  double2 v[E];
  pdl_trigger();
  if (INV == 0) {
    const double2* __restrict__ psi = I.psi + (size_t)line * N;
    const double* __restrict__ rho = I.rho + (size_t)line * N;
    const bool given = I.rho != nullptr, wide = on16(I.rho);
#pragma unroll
    for (int q = 0; q < E / 2; ++q) {
      const int n = t + T * q;
      v[q] = cmk(0.0, 0.0);
      if (valid) {
        if (given) v[q] = load_pair(rho + 2 * n, wide);
        else v[q] = cmk(cabs2(__ldg(psi + 2 * n)), cabs2(__ldg(psi + 2 * n + 1)));
      }
    }
    fft.template forward<true>(v);
    TL::Fft::sync();
#pragma unroll
    for (int q = 0; q < E; ++q) b[t + T * q] = v[q];
    TL::Fft::sync();
    double2* out = I.cb1 + (size_t)line * Mp;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int k = t + T * q;
      const double2 z = v[q], p = b[k ? N - k : 0];     // p: Z_(N-k), conjugated below
      const double2 e = cmk(0.5 * (z.x + p.x), 0.5 * (z.y - p.y));
      const double2 o = cmk(0.5 * (z.y + p.y), 0.5 * (p.x - z.x));
      if (valid) out[k] = cadd(e, cmul(o, __ldg(tw + k)));
    }
    if (t == 0 && valid) out[N] = cmk(v[0].x - v[0].y, 0.0);
  } else {
    pdl_wait();
    const double2* in = I.cb1 + (size_t)line * Mp;
#pragma unroll
    for (int q = 0; q < E; ++q) v[q] = valid ? in[t + T * q] : cmk(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < E; ++q) b[t + T * q] = v[q];
    if (t == 0) b[N] = valid ? in[N] : cmk(0.0, 0.0);
    TL::Fft::sync();
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int k = t + T * q;
      const double2 x = v[q], p = b[N - k];
      const double2 e = cmk(x.x + p.x, x.y - p.y);       // X_k + conj X_(N-k)
      const double2 d = cmk(x.x - p.x, x.y + p.y);       // X_k - conj X_(N-k)
      const double2 o = cconjmul(__ldg(tw + k), d);      // times conj w_M^k
      v[q] = cmk(e.x - o.y, e.y + o.x);                  // e + i o
    }
    fft.template inverse<true>(v);
    double* out = I.phi_out + (size_t)line * N;
    const bool store = valid && I.phi_out != nullptr, wide = on16(I.phi_out);
    const double sc = I.conv_scale;
#pragma unroll
    for (int q = 0; q < E / 2; ++q) {
      v[q] = cscale(v[q], sc);
      if (store) store_pair(out + 2 * (t + T * q), v[q], wide);
    }
    if (I.gpart) {
      // the tile's part of sum phi |psi|^2
      const double2* __restrict__ psi = I.psi + (size_t)line * N;
      double g[1] = {0.0};
#pragma unroll
      for (int q = 0; q < E / 2; ++q) {
        const int n = t + T * q;
        if (valid) g[0] += v[q].x * cabs2(__ldg(psi + 2 * n)) + v[q].y * cabs2(__ldg(psi + 2 * n + 1));
      }
      block_sums<s_threads(N, C, V) / 32, 1>(g);
      if (threadIdx.x == 0) I.gpart[tile] = g[0];
    }
  }
}

// One tile of a strided step: MODE 0: step b (forward); 1: 2D columns and 3D step c
// (forward, K^, inverse); 2: step d (inverse).
template <int M, int C, int V, int MODE>
BGP_D void pad_tile(int tile, int ndim, double2* cb1, double2* cb2, const double* Kq, const double2* tab, double2* sm) {
  using TL = Tile<M, C, V, false>;
  constexpr int E = TL::E, T = TL::T, N = M / 2, Mh = N + 1, Mp = conv_pitch(N), tpl = (Mh + C - 1) / C;
  const TL tl;
  const int t = tl.t;
  const int a = tile / tpl, kk = (tile - a * tpl) * C + tl.c;   // a: i (b, d) or jj (c); 0 in 2D
  const bool valid = tl.c < C && kk < Mh;
  const typename TL::Fft fft{tl.line(sm), tab, t};
  const double2* in;
  double2* out;
  size_t str;
  if (MODE == 1) {
    out = ndim == 2 ? cb1 + kk : cb2 + (size_t)a * Mp + kk;
    in = out;
    str = ndim == 2 ? (size_t)Mp : (size_t)M * Mp;
  } else {
    double2* x1 = cb1 + (size_t)a * N * Mp + kk;
    double2* x2 = cb2 + (size_t)a * M * Mp + kk;
    in = MODE == 0 ? x1 : x2;
    out = MODE == 0 ? x2 : x1;
    str = Mp;
  }
  double2 v[E];
#pragma unroll
  for (int q = 0; q < (MODE == 2 ? E : E / 2); ++q) v[q] = valid ? in[(size_t)(t + T * q) * str] : cmk(0.0, 0.0);
  if (MODE != 2) fft.template forward<true>(v);
  if (MODE == 1) {
    // K^ is real and even: K^[min(k, M - k)] of the quadrant's column
    const int bj = a <= N ? a : M - a;
    const double* __restrict__ K = Kq + (ndim == 2 ? (size_t)0 : (size_t)bj * Mh) + kk;
    const size_t sk = ndim == 2 ? (size_t)Mh : (size_t)Mh * Mh;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int k = t + T * q;
      const double kv = valid ? __ldg(K + (size_t)(k <= N ? k : M - k) * sk) : 0.0;
      v[q] = cscale(v[q], kv);
    }
  }
  if (MODE != 0) fft.template inverse<true>(v);
#pragma unroll
  for (int q = 0; q < (MODE == 0 ? E : E / 2); ++q)
    if (valid) out[(size_t)(t + T * q) * str] = v[q];
}
template <int M, int C, int V, int MODE, int NB>
__global__ void __launch_bounds__(s_threads(M, C, V), s_min_blocks(M, C, V))
    k_stream_pad(const __grid_constant__ SLaunchT<NB> SL) {
  extern __shared__ double2 sm[];
  const int inst = NB == 1 ? 0 : blockIdx.x / SL.tiles, tile = blockIdx.x - inst * SL.tiles;
  const SInst& I = SL.insts[inst];
  pdl_trigger();
  pdl_wait();
  pad_tile<M, C, V, MODE>(tile, I.ndim, I.cb1, I.cb2, I.Kq, I.tabM[V], sm);
}

// ------------------------------------------------------------------ energy sums
// The sums of energy_components (operators.py:10-29 of the reference) over a state as
// given: on the contiguous axis the local sums of rho = |psi|^2, on every axis the
// spectral sums  sum k^2 |psi^|^2  and, for L_z,  X sum k_y |psi^|^2  and
// Y sum k_x |psi^|^2  (Parseval along one axis). All axes' tiles are one launch: block
// b of axis slot a = b / tiles; slot 0 is the contiguous axis. Each block leaves
// kESums sums and one maximum in I.part, value q of block b at q * gridDim.x + b.
enum : int { E_N0, E_V, E_2, E_3, E_R2, E_PERP, E_Z2, E_K, E_L, kESums };
template <int N, int C, int V>
__global__ void __launch_bounds__(s_threads(N, C, V), s_min_blocks(N, C, V))
    k_stream_energy(const __grid_constant__ SLaunchT<1> SL) {
  constexpr int T = lf_threads(N, V), E = lplan(N, V).E, W = s_threads(N, C, V) / 32;
  extern __shared__ double2 sm[];
  const SInst& I = SL.insts[0];
  const int slot = blockIdx.x / SL.tiles, tile = blockIdx.x - slot * SL.tiles, ndim = I.ndim;
  const double2* __restrict__ psi = I.psi;
  const double dx = I.dx, kf = I.kfac;
  double sum[kESums], mx = 0.0, fixed = 0.0;     // fixed: the L_z coordinate of the line
#pragma unroll
  for (int q = 0; q < kESums; ++q) sum[q] = 0.0;
  double2 v[E];
  int t;
  bool valid;
  if (slot == 0) {
    const Tile<N, C, V, true> tl;
    t = tl.t;
    valid = tl.c < C;
    const int line = tile * C + tl.c;
    const int i = ndim == 2 ? line : line / N, j = line - i * N;
    const double x = (double)(i - N / 2) * dx, y3 = (double)(j - N / 2) * dx;
    if (ndim == 2) fixed = x;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int r = t + T * q;
      v[q] = valid ? __ldg(psi + (size_t)line * N + r) : cmk(0.0, 0.0);
      const double p = cabs2(v[q]);
      const double c = (double)(r - N / 2) * dx;
      // (x, y) = (x_i, x_r) in 2D; (x_i, x_j, x_r) in 3D
      const double y = ndim == 2 ? c : y3;
      const double rp = x * x + y * y;
      double r2 = rp;
      if (ndim == 3) {
        r2 = r2 + c * c;
        sum[E_PERP] += rp * p;
        sum[E_Z2] += c * c * p;
      }
      const double Vt = (I.s <= 0.0) ? 0.0 : ((I.s == 2.0) ? I.tc * r2 : I.tc * pow(r2, 0.5 * I.s));
      sum[E_N0] += p;
      sum[E_V] += Vt * p;
      sum[E_2] += p * p;
      sum[E_3] += p * p * p;
      sum[E_R2] += r2 * p;
      mx = fmax(mx, p);
    }
    const typename Tile<N, C, V, true>::Fft fft{tl.line(sm), I.tabN[V], t};
    fft.template forward<false>(v);
  } else {
    const Tile<N, C, V, false> tl;
    t = tl.t;
    valid = tl.c < C;
    // slot 1: axis 0 (x); slot 2 (3D): axis 1 (y)
    int base, str;
    if (ndim == 2) {
      base = tile * C + tl.c; str = N;
      fixed = (double)(base - N / 2) * dx;
    } else {
      constexpr int tpl = N / C;
      const int a = tile / tpl, k = (tile - a * tpl) * C + tl.c;
      base = slot == 1 ? a * N + k : a * N * N + k;
      str = slot == 1 ? N * N : N;
      fixed = (double)(a - N / 2) * dx;
    }
#pragma unroll
    for (int q = 0; q < E; ++q) v[q] = valid ? __ldg(psi + base + (t + T * q) * str) : cmk(0.0, 0.0);
    const typename Tile<N, C, V, false>::Fft fft{tl.line(sm), I.tabN[V], t};
    fft.template forward<false>(v);
  }
  double sl = 0.0;
#pragma unroll
  for (int q = 0; q < E; ++q) {
    const int r = t + T * q, mm = (r < (N + 1) / 2) ? r : r - N;
    const double kk = kTwoPi * ((double)mm * kf), a2 = cabs2(v[q]);
    sum[E_K] += kk * kk * a2;
    sl += kk * a2;
  }
  sum[E_L] = fixed * sl;
  block_sums<W, kESums>(sum);
  __shared__ double wm[W];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < W; ++w) mx = fmax(mx, wm[w]);
#pragma unroll
    for (int q = 0; q < kESums; ++q) I.part[(size_t)q * gridDim.x + blockIdx.x] = sum[q];
    I.part[(size_t)kESums * gridDim.x + blockIdx.x] = mx;
  }
}

// Sum of |H - mu psi|^2: one partial per block at part[blockIdx.x] (mu on the device).
constexpr int kResidThreads = 256;
static __global__ void __launch_bounds__(kResidThreads)
    k_stream_resid(const double2* __restrict__ psi, const double2* __restrict__ H, int n, const double* mu,
                   double* part) {
  const double m = *mu;
  double g[1] = {0.0};
  const int step = gridDim.x * kResidThreads;
  for (int f0 = blockIdx.x * kResidThreads + threadIdx.x; f0 < n; f0 += 4 * step) {
    double2 p[4], h[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int f = f0 + u * step;
      p[u] = f < n ? __ldg(psi + f) : cmk(0.0, 0.0);
      h[u] = f < n ? __ldg(H + f) : cmk(0.0, 0.0);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) g[0] += cabs2(csub(h[u], cscale(p[u], m)));
  }
  block_sums<kResidThreads / 32, 1>(g);
  if (threadIdx.x == 0) part[blockIdx.x] = g[0];
}

// Totals of lists of partials: block b adds cnt[b] values at part[b], thread by thread
// in a fixed order (or takes their maximum), into out[b] (mapped host memory or device).
struct SumArgs {
  static constexpr int kMax = 24;
  const double* part[kMax];
  int cnt[kMax], is_max[kMax];
  double scale[kMax];
  double* out;
};
static __global__ void __launch_bounds__(256) k_stream_sum(const __grid_constant__ SumArgs A) {
  const int b = blockIdx.x, n = A.cnt[b];
  const double* p = A.part[b];
  const bool is_max = A.is_max[b];
  double s = 0.0;
  for (int t = threadIdx.x; t < n; t += 256) s = is_max ? fmax(s, p[t]) : s + p[t];
  __shared__ double red[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double y = __shfl_xor_sync(0xffffffffu, s, o);
    s = is_max ? fmax(s, y) : s + y;
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) s = is_max ? fmax(s, red[w]) : s + red[w];
    A.out[b] = s * A.scale[b];
  }
}

#endif  // __CUDACC__

BGP_NS_END  // namespace bgp
