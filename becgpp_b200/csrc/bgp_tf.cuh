// Thomas-Fermi reference density on the device (becgpp/thomasfermi.py:33-120).
//
// The density n solves  mu = V_eff + b2 n + b3 n^2 + phi[n]  with  sum n dV = 1,
// V_eff = V - Omega^2 (x^2 + y^2) / 2 and phi the long-range potential of n
// (zero for the local references). One launch of k_tf_iter is one step of the
// reference's relaxed fixed point:
//   base  = V_eff + phi                      (phi = -G_C dV (K * n), from the plan)
//   mu    : sum_i rho(mu, base_i) dV = 1, by the reference's bracket expansion and
//           90 bisection halvings, three to a full-grid reduction: the seven points the
//           next three halvings can reach are summed together and the decisions follow
//           as in the one-by-one order, bit for bit (a reduction is a grid barrier
//           of several us, six more sums of a few points per thread a fraction of one;
//           25 steps at 256^2, with the convolutions: 14.6 ms with 90 reductions of one
//           sum over 592 CTAs, 5.8 ms with 30 of seven over 128)
//   n_new = rho(mu, base) / (sum rho dV)
//   dn    = sum |n_new - n| dV,  n <- (1 - relax) n + relax n_new,  n <- n / (sum n dV)
// with rho(mu, b) the upper non-negative root of b3 rho^2 + b2 rho = mu - b.
// The local references (no long-range term) use the same launch once, in mode 0:
// n = n_new, no relaxation.
//
// Work decomposition: all CTAs of the launch form one team (cooperative launch,
// bounded team barrier); every full-grid sum is a deterministic grid reduction
// (thread partials in a fixed grid-stride order, warp butterflies, warp totals
// in order, CTA partials added in CTA order after the barrier), so every CTA
// holds the same totals and takes the same bisection decisions without a
// broadcast. The arithmetic of V_eff and rho uses round-to-nearest intrinsics
// (no contraction into FMAs), the operation order of the reference's tensor
// expressions.
#pragma once
#include "bgp_common.cuh"

BGP_NS_BEGIN

struct TfArgs {
  int ndim, N, n, mode;          // mode 0: local (one mu solve), 1: one fixed-point step
  double dx, dv, tc, s, Omega, b2, b3, gc, relax;
  const double* conv;            // dV (K * n) of the current n (mode 1), else null
  double* nf;                    // density: current n in, new n out
  double* part;                  // 2 x 8 x gridDim.x partial sums
  unsigned long long* bar;       // team barrier counter
  int* abort_flag;               // status word (4 + gridDim.x ints)
  double* state;                 // out: [0] mu, [1] dn, [2] status, [3] converged, [4] steps taken
};

enum TfStatus : int { kTfOk = 0, kTfNoBracket = 1, kTfEmpty = 2, kTfBarrier = 3 };

// V_eff at flat index f (becgpp/thomasfermi.py:21-30 with becgpp/grid.py:86-91).
BGP_D double tf_veff(const TfArgs& A, int f) {
  const int N = A.N;
  int i, j, k = 0;
  if (A.ndim == 2) { i = f / N; j = f - i * N; }
  else { i = f / (N * N); const int r = f - i * N * N; j = r / N; k = r - j * N; }
  const double x = (double)(i - N / 2) * A.dx, y = (double)(j - N / 2) * A.dx;
  const double rp2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
  double r2 = rp2;
  if (A.ndim == 3) { const double z = (double)(k - N / 2) * A.dx; r2 = __dadd_rn(r2, __dmul_rn(z, z)); }
  double V = 0.0;
  if (A.s > 0.0) V = (A.s == 2.0) ? __dmul_rn(A.tc, r2) : __dmul_rn(A.tc, pow(r2, 0.5 * A.s));
  const double c = (0.5 * A.Omega) * A.Omega;
  return __dsub_rn(V, __dmul_rn(c, rp2));
}

// a / b with r = 1 / b, both rounded to nearest: the quotient q0 = a r is corrected by its
// exact remainder (Markstein, IBM J. Res. Dev. 34, 1990), which rounds it correctly; the
// same quotient as a division instruction's, in three operations that overlap with the
// other candidates'. (One thread's 28 divisions were half of a reduction of the bisection.)
BGP_HD double tf_quotient(double a, double b, double r) {
  const double q = a * r;
  return fma(fma(-q, b, a), r, q);
}
// the density's coefficients and the reciprocals its roots divide by
struct TfRoot {
  double b2, b3, r2, r3;       // r2 = 1 / b2, r3 = 1 / (2 b3) where they are used
};
BGP_HD TfRoot tf_root(double b2, double b3) {
  return TfRoot{b2, b3, fabs(b2) > 1e-30 ? 1.0 / b2 : 0.0, b3 > 1e-30 ? 1.0 / (2.0 * b3) : 0.0};
}

// Upper physical root rho >= 0 of b3 rho^2 + b2 rho = mu - b, zero where there is
// no real root (becgpp/thomasfermi.py:33-45).
BGP_D double tf_rho(double mu, double b, const TfRoot& P) {
  const double rhs = __dsub_rn(mu, b);
  if (P.b3 > 1e-30) {
    const double disc = __dadd_rn(__dmul_rn(P.b2, P.b2), __dmul_rn(4.0 * P.b3, rhs));
    if (!(disc > 0.0)) return 0.0;
    const double root = tf_quotient(__dadd_rn(-P.b2, sqrt(disc)), 2.0 * P.b3, P.r3);
    return root > 0.0 ? root : 0.0;
  }
  if (fabs(P.b2) > 1e-30) {
    const double q = tf_quotient(rhs, P.b2, P.r2);
    return q > 0.0 ? q : 0.0;
  }
  return 0.0;
}

#if defined(__CUDACC__)

constexpr int kTfSums = 7;               // most values of one reduction
constexpr int kTfHold = 4;               // base values a thread keeps in registers

// Deterministic grid-wide reduction of NV values per thread (op: 0 sum, 1 min,
// 2 max), identical totals in every CTA. sm: kTfSums * (kWarps + 1) doubles. The
// partials of the two alternating slots sit 8 values apart whatever NV is, so a
// reduction never writes where the previous one (other slot) is still being read.
template <int NV>
BGP_D bool grid_reduce(double (&v)[NV], const int (&op)[NV], double* part, int& slot, const Team& T,
                       double* sm) {
  static_assert(NV <= kTfSums, "more values than a reduction holds");
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, G = gridDim.x;
  auto comb = [](int o, double a, double b) { return o == 0 ? a + b : (o == 1 ? fmin(a, b) : fmax(a, b)); };
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    double x = v[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = comb(op[q], x, __shfl_xor_sync(0xffffffffu, x, o));
    if (lane == 0) sm[q * kWarps + w] = x;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    const int q = threadIdx.x;
    double x = sm[q * kWarps];
    for (int k = 1; k < kWarps; ++k) x = comb(op[q], x, sm[q * kWarps + k]);
    st1(part + ((size_t)slot * 8 + q) * G + blockIdx.x, x);
  }
  if (!team_sync(T)) return false;
  // warp w adds the G partials of values w, w + kWarps: lane l takes CTAs l, l+32, ...
  // in order (all values' loads in flight), then the 32 lane totals meet in a fixed
  // butterfly
  constexpr int PER = (NV + kWarps - 1) / kWarps;
  double x[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int q = w + u * kWarps;
    x[u] = 0.0;
    if (q < NV && op[q] != 0) x[u] = ld1(part + ((size_t)slot * 8 + q) * G);
  }
  for (int b = lane; b < G; b += 128) {
    double y[PER][4];
#pragma unroll
    for (int u = 0; u < PER; ++u)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int q = w + u * kWarps;
        y[u][c] = (q < NV && b + 32 * c < G) ? ld1(part + ((size_t)slot * 8 + q) * G + b + 32 * c) : x[u];
      }
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int q = w + u * kWarps;
      if (q < NV) {
#pragma unroll
        for (int c = 0; c < 4; ++c) if (b + 32 * c < G) x[u] = comb(op[q], x[u], y[u][c]);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int q = w + u * kWarps;
    if (q < NV) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x[u] = comb(op[q], x[u], __shfl_xor_sync(0xffffffffu, x[u], o));
      if (lane == 0) sm[kTfSums * kWarps + q] = x[u];
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; ++q) v[q] = sm[kTfSums * kWarps + q];
  __syncthreads();
  slot ^= 1;
  return true;
}

// One Thomas-Fermi step (see the file comment). Launched cooperatively with every
// CTA resident; kThreads threads per CTA.
__global__ void __launch_bounds__(kThreads) k_tf_iter(TfArgs A) {
  __shared__ double sm[kTfSums * (kWarps + 1)];
  Team T{(int)blockIdx.x, (int)gridDim.x, A.bar, A.abort_flag};
  // a step after the fixed point has converged or failed does nothing (the host enqueues
  // several steps before it looks)
  if (ld1(A.state + 2) != (double)kTfOk || ld1(A.state + 3) != 0.0) return;
  int slot = 0;
  const int n = A.n;
  const int first = blockIdx.x * kThreads + threadIdx.x, stride = gridDim.x * kThreads;
  const double gc = A.gc;
  const TfRoot root = tf_root(A.b2, A.b3);
  auto base = [&](int f) {
    const double v = tf_veff(A, f);
    return A.conv ? __dadd_rn(v, __dmul_rn(-gc, ld1(A.conv + f))) : v;
  };
  // the thread's base values, kept in registers when they are few
  const bool held = n <= kTfHold * stride;
  double hb[kTfHold];
  if (held) {
#pragma unroll
    for (int u = 0; u < kTfHold; ++u) hb[u] = first + u * stride < n ? base(first + u * stride) : 0.0;
  }
  auto fail = [&](int code) {
    if (blockIdx.x == 0 && threadIdx.x == 0) { A.state[2] = (double)code; A.state[3] = 0.0; A.state[4] += 1.0; }
  };
  // bracket of mu: [min base, max base + |b2| + |b3| + 1] (becgpp/thomasfermi.py:99-100)
  double lo, hi;
  {
    double v[2] = {INFINITY, -INFINITY};
    const int op[2] = {1, 2};
    for (int f = first; f < n; f += stride) { const double b = base(f); v[0] = fmin(v[0], b); v[1] = fmax(v[1], b); }
    if (!grid_reduce<2>(v, op, A.part, slot, T, sm)) { fail(kTfBarrier); return; }
    lo = v[0];
    hi = v[1] + fabs(A.b2) + fabs(A.b3) + 1.0;
  }
  // sum rho(mu[q]) dV of NV chemical potentials (q < NV), each summed in point order
  auto masses = [&](auto& mu) {
    constexpr int NV = sizeof(mu) / sizeof(double);
    double v[NV];
    int op[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) { v[q] = 0.0; op[q] = 0; }
    if (held) {
#pragma unroll
      for (int u = 0; u < kTfHold; ++u)
        if (first + u * stride < n) {
#pragma unroll
          for (int q = 0; q < NV; ++q) v[q] += tf_rho(mu[q], hb[u], root);
        }
    } else {
      for (int f = first; f < n; f += stride) {
        const double b = base(f);
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q] += tf_rho(mu[q], b, root);
      }
    }
    if (!grid_reduce<NV>(v, op, A.part, slot, T, sm)) return false;
#pragma unroll
    for (int q = 0; q < NV; ++q) mu[q] = v[q] * A.dv;
    return true;
  };
  auto mass = [&](double mu, double& out) {
    double m[1] = {mu};
    if (!masses(m)) return false;
    out = m[0];
    return true;
  };
  // expand the upper end until it holds unit mass (becgpp/thomasfermi.py:51-55)
  for (int guard = 0;; ++guard) {
    double m;
    if (!mass(hi, m)) { fail(kTfBarrier); return; }
    if (m >= 1.0) break;
    if (guard >= 200) { fail(kTfNoBracket); return; }
    hi = lo + 2.0 * (hi - lo) + 1e-9;
  }
  // 90 halvings (becgpp/thomasfermi.py:56-61), three at a time: m[0] the midpoint, m[1],
  // m[2] those of its halves, m[3..6] those of its quarters
  auto mid = [](double a, double b) { return 0.5 * (a + b); };
  for (int step = 0; step < 90; step += 3) {
    const double c = mid(lo, hi), cl = mid(lo, c), ch = mid(c, hi);
    double m[7] = {c, cl, ch, mid(lo, cl), mid(cl, c), mid(c, ch), mid(ch, hi)};
    const double p[7] = {m[0], m[1], m[2], m[3], m[4], m[5], m[6]};
    if (!masses(m)) { fail(kTfBarrier); return; }
    int k = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      double mk = m[0], pk = p[0];
#pragma unroll
      for (int q = 1; q < 7; ++q) if (q == k) { mk = m[q]; pk = p[q]; }
      const bool up = mk < 1.0;
      if (up) lo = pk; else hi = pk;
      k = 2 * k + (up ? 2 : 1);
    }
  }
  const double mu = 0.5 * (lo + hi);
  double ssum;
  if (!mass(mu, ssum)) { fail(kTfBarrier); return; }
  if (!(ssum > 0.0)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) A.state[0] = mu;
    fail(kTfEmpty);
    return;
  }
  double dn = 0.0;
  if (A.mode == 0) {
    // local reference: n = rho(mu) / (sum rho dV)
    for (int f = first; f < n; f += stride) st1(A.nf + f, __ddiv_rn(tf_rho(mu, base(f), root), ssum));
  } else {
    // relaxed update and its renormalisation (becgpp/thomasfermi.py:103-110)
    double v[2] = {0.0, 0.0};
    const int op[2] = {0, 0};
    const double a = 1.0 - A.relax, r = A.relax;
    for (int f = first; f < n; f += stride) {
      const double nn = __ddiv_rn(tf_rho(mu, base(f), root), ssum);
      const double old = ld1(A.nf + f);
      v[0] += fabs(__dsub_rn(nn, old));
      const double upd = __dadd_rn(__dmul_rn(a, old), __dmul_rn(r, nn));
      st1(A.nf + f, upd);
      v[1] += upd;
    }
    if (!grid_reduce<2>(v, op, A.part, slot, T, sm)) { fail(kTfBarrier); return; }
    dn = v[0] * A.dv;
    const double norm = v[1] * A.dv;
    for (int f = first; f < n; f += stride) st1(A.nf + f, __ddiv_rn(ld1(A.nf + f), norm));
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    A.state[0] = mu;
    A.state[1] = dn;
    A.state[2] = (double)kTfOk;
    A.state[3] = (A.mode == 0 || dn < 1e-9) ? 1.0 : 0.0;
    A.state[4] += 1.0;
  }
}

// Initial density of the fixed point, exp(-r^2 / (2 sigma^2)) with sigma = 0.15 L,
// normalised to unit mass (becgpp/thomasfermi.py:89-91). Cooperative launch.
__global__ void __launch_bounds__(kThreads) k_tf_seed(TfArgs A, double two_s2) {
  __shared__ double sm[kTfSums * (kWarps + 1)];
  Team T{(int)blockIdx.x, (int)gridDim.x, A.bar, A.abort_flag};
  int slot = 0;
  const int n = A.n, N = A.N;
  const int first = blockIdx.x * kThreads + threadIdx.x, stride = gridDim.x * kThreads;
  double v[1] = {0.0};
  const int op[1] = {0};
  for (int f = first; f < n; f += stride) {
    int i, j, k = 0;
    if (A.ndim == 2) { i = f / N; j = f - i * N; }
    else { i = f / (N * N); const int r = f - i * N * N; j = r / N; k = r - j * N; }
    const double x = (double)(i - N / 2) * A.dx, y = (double)(j - N / 2) * A.dx;
    double r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
    if (A.ndim == 3) { const double z = (double)(k - N / 2) * A.dx; r2 = __dadd_rn(r2, __dmul_rn(z, z)); }
    const double e = exp(__ddiv_rn(-r2, two_s2));
    st1(A.nf + f, e);
    v[0] += e;
  }
  if (!grid_reduce<1>(v, op, A.part, slot, T, sm)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) A.state[2] = (double)kTfBarrier;
    return;
  }
  const double norm = v[0] * A.dv;
  for (int f = first; f < n; f += stride) st1(A.nf + f, __ddiv_rn(ld1(A.nf + f), norm));
}

#endif  // __CUDACC__

BGP_NS_END  // namespace bgp
