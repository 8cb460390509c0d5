// Thomas-Fermi reference density on the device (becgpp/thomasfermi.py:33-120).
//
// The density n solves  mu = V_eff + b2 n + b3 n^2 + phi[n]  with  sum n dV = 1,
// V_eff = V - Omega^2 (x^2 + y^2) / 2 and phi the long-range potential of n
// (zero for the local references). One launch of k_tf_iter is one step of the
// reference's relaxed fixed point:
//   base  = V_eff + phi                      (phi = -G_C dV (K * n), from the plan)
//   mu    : sum_i rho(mu, base_i) dV = 1, by the reference's bracket expansion and
//           90 bisection halvings, three to a reduction: the seven points the next three
//           halvings can reach are summed together and the decisions follow in the
//           one-by-one order. A step is a chain of such reductions, bound by their latency:
//           25 steps at 256^2, with the convolutions, 14.6 ms with 90 reductions of one sum
//           over 592 CTAs, 5.8 ms with 30 of seven over 128, 4.7 ms with one division per
//           sum instead of one per point, 3.5 ms without the halvings of an interval that no
//           longer changes.
//   n_new = rho(mu, base) / (sum rho dV)
//   dn    = sum |n_new - n| dV,  n <- (1 - relax) n + relax n_new,  n <- n / (sum n dV)
// with rho(mu, b) the upper non-negative root of b3 rho^2 + b2 rho = mu - b.
// The local references (no long-range term) use the same launch once, in mode 0:
// n = n_new, no relaxation.
//
// Work decomposition: the CTAs of the launch form one team, either one thread-block
// cluster (k_tf_iter_cluster) or all resident CTAs of a cooperative launch with a bounded
// team barrier (k_tf_iter); every sum is deterministic (thread partials in a fixed
// stride order, warp butterflies, warp totals and CTA partials in fixed orders), so every
// CTA holds the same totals and takes the same bisection decisions without a
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
  int* abort_flag;               // status word (4 + gridDim.x ints), cleared once per density
  double* state;                 // out: [0] mu, [1] dn, [2] status, [3] converged, [4] steps taken
};

constexpr int kTfState = 5;      // values of TfArgs::state
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

// Upper physical root rho >= 0 of b3 rho^2 + b2 rho = mu - b, zero where there is
// no real root (becgpp/thomasfermi.py:33-45).
BGP_D double tf_rho(double mu, double b, double b2, double b3) {
  const double rhs = __dsub_rn(mu, b);
  if (b3 > 1e-30) {
    const double disc = __dadd_rn(__dmul_rn(b2, b2), __dmul_rn(4.0 * b3, rhs));
    if (!(disc > 0.0)) return 0.0;
    const double root = __ddiv_rn(__dadd_rn(-b2, sqrt(disc)), 2.0 * b3);
    return root > 0.0 ? root : 0.0;
  }
  if (fabs(b2) > 1e-30) {
    const double q = __ddiv_rn(rhs, b2);
    return q > 0.0 ? q : 0.0;
  }
  return 0.0;
}

#if defined(__CUDACC__)

constexpr int kTfSums = 7;               // most values of one reduction
constexpr int kTfHold = 4;               // base values a thread keeps in registers (grid)

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

// The team of a cooperative launch: every resident CTA, meeting at a grid barrier.
struct TfGrid {
  static constexpr int kHold = kTfHold;
  Team T;
  double *part, *sm;
  int slot;
  BGP_D int first() const { return blockIdx.x * kThreads + threadIdx.x; }
  BGP_D int stride() const { return gridDim.x * kThreads; }
  template <int NV, bool MAX>
  BGP_D bool reduce(double (&v)[NV]) {
    int op[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) op[q] = MAX ? 2 : 0;
    return grid_reduce<NV>(v, op, part, slot, T, sm);
  }
};

// The team of one thread-block cluster (up to 16 CTAs of 512 threads): partials go into
// every CTA's shared memory and the CTAs meet at the cluster's hardware barrier, which
// costs a fraction of a grid barrier through L2; the price is that 16 SMs do the sums
// (where that pays: tf_cluster in bgp_api.cu).
constexpr int kTfClThreads = 512, kTfClWarps = kTfClThreads / 32, kTfClMax = 16, kTfClHold = 8;
struct TfCluster {
  static constexpr int kHold = kTfClHold;
  double *wpart, *buf;           // kTfSums x kTfClWarps; 2 slots x 8 values x kTfClMax CTAs
  int slot;
  BGP_D int first() const { return blockIdx.x * kTfClThreads + threadIdx.x; }
  BGP_D int stride() const { return gridDim.x * kTfClThreads; }
  static BGP_D void sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  }
  // Every CTA adds the same partials in the same order. The slots alternate: a CTA writes
  // a slot again only after the barrier behind which all have read it.
  template <int NV, bool MAX>
  BGP_D bool reduce(double (&v)[NV]) {
    static_assert(NV <= 8 && NV <= kTfClWarps, "more values than a reduction holds");
    constexpr int P = NV <= 1 ? 1 : (NV <= 2 ? 2 : (NV <= 4 ? 4 : 8));
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, G = gridDim.x;
    const double none = MAX ? -INFINITY : 0.0;
    auto comb = [](double a, double b) { return MAX ? fmax(a, b) : a + b; };
    // warp: halve the values and the lanes that share one together (8 values: 9 exchanges)
    double x[P];
#pragma unroll
    for (int q = 0; q < P; ++q) x[q] = q < NV ? v[q] : none;
    int q0 = 0, o = 16;
#pragma unroll
    for (int half = P / 2; half >= 1; half /= 2) {
      const bool up = lane & o;
      if (up) q0 += half;
#pragma unroll
      for (int j = 0; j < half; ++j) {
        const double keep = up ? x[j + half] : x[j], send = up ? x[j] : x[j + half];
        x[j] = comb(keep, __shfl_xor_sync(0xffffffffu, send, o));
      }
      o /= 2;
    }
    const int same = 2 * o - 1;                // lane bits that hold the same value
#pragma unroll
    for (int k = 16; k > 0; k >>= 1)
      if (k <= o) x[0] = comb(x[0], __shfl_xor_sync(0xffffffffu, x[0], k));
    if ((lane & same) == 0 && q0 < NV) wpart[q0 * kTfClWarps + w] = x[0];
    __syncthreads();
    // CTA: warp q takes value q and sends it to every CTA
    if (w < NV) {
      double y = wpart[w * kTfClWarps + (lane & (kTfClWarps - 1))];
#pragma unroll
      for (int k = kTfClWarps / 2; k > 0; k >>= 1) y = comb(y, __shfl_xor_sync(0xffffffffu, y, k));
      if (lane < G) {
        const unsigned at = (unsigned)__cvta_generic_to_shared(buf + (slot * 8 + w) * kTfClMax + blockIdx.x);
        unsigned to;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(at), "r"(lane));
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(to), "d"(y) : "memory");
      }
    }
    __syncwarp();
    sync();
    // every warp adds the CTAs' partials: lane 4 q + j those of CTAs j, j + 4, ...
    const int q = lane >> 2;
    double y = none;
#pragma unroll
    for (int c = 0; c < kTfClMax / 4; ++c) {
      const int r = (lane & 3) + 4 * c;
      if (q < NV && r < G) y = comb(y, buf[(slot * 8 + q) * kTfClMax + r]);
    }
    y = comb(y, __shfl_xor_sync(0xffffffffu, y, 1));
    y = comb(y, __shfl_xor_sync(0xffffffffu, y, 2));
#pragma unroll
    for (int u = 0; u < NV; ++u) v[u] = __shfl_sync(0xffffffffu, y, 4 * u);
    slot ^= 1;
    return true;
  }
};

// One Thomas-Fermi step (see the file comment) by the threads of team R.
template <class R>
BGP_D void tf_step(const TfArgs& A, R& team) {
  constexpr int H = R::kHold;
  const int n = A.n, first = team.first(), stride = team.stride();
  const double gc = A.gc;
  // rho = d u with d = 2 b3 or |b2| the same for every point, so the masses of the
  // bisection add u and divide once (a division per point and candidate was half of a
  // reduction): u = sqrt(b2^2 + 4 b3 (mu - b)) - b2, or sign(b2) (mu - b), where positive
  const bool quad = A.b3 > 1e-30, lin = !quad && fabs(A.b2) > 1e-30;
  const double sgn = lin && A.b2 < 0.0 ? -1.0 : 1.0, b22 = A.b2 * A.b2, b34 = 4.0 * A.b3;
  const double per = quad ? A.dv / (2.0 * A.b3) : (lin ? A.dv / fabs(A.b2) : 0.0);
  auto base = [&](int f) {
    const double v = tf_veff(A, f);
    return A.conv ? __dadd_rn(v, __dmul_rn(-gc, ld1(A.conv + f))) : v;
  };
  // the thread's base values (times sgn), kept in registers when they are few
  const bool held = n <= H * stride;
  double hb[H];
  if (held) {
#pragma unroll
    for (int u = 0; u < H; ++u) hb[u] = first + u * stride < n ? sgn * base(first + u * stride) : 0.0;
  }
  auto fail = [&](int code) {
    if (blockIdx.x == 0 && threadIdx.x == 0) { A.state[2] = (double)code; A.state[3] = 0.0; A.state[4] += 1.0; }
  };
  // bracket of mu: [min base, max base + |b2| + |b3| + 1] (becgpp/thomasfermi.py:99-100)
  double lo, hi;
  {
    double v[2] = {-INFINITY, -INFINITY};        // -min, max
    for (int f = first; f < n; f += stride) { const double b = base(f); v[0] = fmax(v[0], -b); v[1] = fmax(v[1], b); }
    if (!team.template reduce<2, true>(v)) { fail(kTfBarrier); return; }
    lo = -v[0];
    hi = v[1] + fabs(A.b2) + fabs(A.b3) + 1.0;
  }
  // sum rho(mu[q]) dV of NV chemical potentials (q < NV), each summed in point order
  auto masses = [&](auto& mu) {
    constexpr int NV = sizeof(mu) / sizeof(double);
    double v[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) { v[q] = 0.0; mu[q] *= sgn; }
    auto add = [&](double b) {                   // b: sgn times the base value
      if (quad) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          // the roundings of tf_rho: where b3 is small against b2^2 the roots differ from
          // rounding to rounding, and the density is tf_rho over the sum of these
          const double disc = __dadd_rn(b22, __dmul_rn(b34, __dsub_rn(mu[q], b)));
          const double u = __dadd_rn(-A.b2, sqrt(fmax(disc, 0.0)));
          v[q] += disc > 0.0 && u > 0.0 ? u : 0.0;
        }
      } else {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          const double u = mu[q] - b;
          if (u > 0.0) v[q] += u;
        }
      }
    };
    if (held) {
#pragma unroll
      for (int u = 0; u < H; ++u)
        if (first + u * stride < n) add(hb[u]);
    } else {
      for (int f = first; f < n; f += stride) add(sgn * base(f));
    }
    if (!team.template reduce<NV, false>(v)) return false;
#pragma unroll
    for (int q = 0; q < NV; ++q) mu[q] = v[q] * per;
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
  auto mid = [](double a, double b) { return 0.5 * (a + b); };
  // 90 halvings (becgpp/thomasfermi.py:56-61), three at a time: m[0] the midpoint, m[1],
  // m[2] those of its halves, m[3..6] those of its quarters. Three halvings that leave the
  // interval as it was are followed by nothing else (they depend on lo and hi alone): about
  // 60 of the 90 reach neighbouring doubles.
  for (int step = 0; step < 90; step += 3) {
    const double lo0 = lo, hi0 = hi;
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
    if (lo == lo0 && hi == hi0) break;
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
    for (int f = first; f < n; f += stride) st1(A.nf + f, __ddiv_rn(tf_rho(mu, base(f), A.b2, A.b3), ssum));
  } else {
    // relaxed update and its renormalisation (becgpp/thomasfermi.py:103-110)
    double v[2] = {0.0, 0.0};
    const double a = 1.0 - A.relax, r = A.relax;
    for (int f = first; f < n; f += stride) {
      const double nn = __ddiv_rn(tf_rho(mu, base(f), A.b2, A.b3), ssum);
      const double old = ld1(A.nf + f);
      v[0] += fabs(__dsub_rn(nn, old));
      const double upd = __dadd_rn(__dmul_rn(a, old), __dmul_rn(r, nn));
      st1(A.nf + f, upd);
      v[1] += upd;
    }
    if (!team.template reduce<2, false>(v)) { fail(kTfBarrier); return; }
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

// a step after the fixed point has converged or failed does nothing (the host enqueues
// several steps before it looks)
BGP_D bool tf_over(const TfArgs& A) {
  const double status = ld1(A.state + 2), done = ld1(A.state + 3);
  return status != (double)kTfOk || done != 0.0;
}

// Launched cooperatively with every CTA resident; kThreads threads per CTA.
__global__ void __launch_bounds__(kThreads) k_tf_iter(TfArgs A) {
  __shared__ double sm[kTfSums * (kWarps + 1)];
  // (a barrier that timed out in an earlier launch shows in the status word alone when the
  // first CTA got past it)
  const int gave_up = __ldcg(A.abort_flag);
  if (tf_over(A) || gave_up != 0) return;
  TfGrid team{Team{(int)blockIdx.x, (int)gridDim.x, A.bar, A.abort_flag}, A.part, sm, 0};
  tf_step(A, team);
}
// Launched as one cluster of gridDim.x CTAs. (Its barrier has no time-out; the seed's is
// reported by the host.)
__global__ void __launch_bounds__(kTfClThreads) k_tf_iter_cluster(TfArgs A) {
  __shared__ double wpart[kTfSums * kTfClWarps], buf[2 * 8 * kTfClMax];
  if (tf_over(A)) return;
  TfCluster team{wpart, buf, 0};
  TfCluster::sync();             // every CTA has started before the first write to its buf
  tf_step(A, team);
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
