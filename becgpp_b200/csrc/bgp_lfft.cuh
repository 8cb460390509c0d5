// Line transforms of the stream passes: T = L / E threads per line, E values of
// the line in each thread's registers, and one shared-memory exchange between two
// radix stages.
//
// A line of L = r[0] r[1] .. r[n-1] values. Before stage S, with P the product of
// the radices done, the data is a(k, m), k in [0, P), m in [0, L / P) (k: the part
// of the spectral index already formed, m: what is left of the point index). Stage
// S of radix R splits m = m' + Lr a, Lr = L / (P R):
//   b -> sum_a a(k, m' + Lr a) w_R^(a b),   times w_(L/P)^(m' b),   at (k + P b, m').
// Sub-transform u = m' + Lr k, u in [0, L / R); thread t takes u = t + T s, s <
// E / R, and keeps element a (on the way in) or b (on the way out) of it in register
// slot s + (E / R) a. So the first stage reads and the last stage leaves element
// t + T q in slot q: consecutive threads on consecutive elements, straight from and
// to global memory, and a multiplier is applied between the forward and the inverse
// transform in registers. The inverse runs the stages backwards with conjugate
// twiddles. A transform pair of an n-stage line costs 2 (n - 1) exchanges; the
// in-place Stockham line in shared memory that this replaces cost 4 n + 2 (every
// stage's load and store, the multiplier's, the tile's way in and out), and shared
// memory was what bound it: the 256-point pass with a multiplier of the 3D
// convolution ran at 77 % of the L1 data pipe and 7 % of the DRAM peak.
//
// HALF transforms: on a zero-padded line the upper half of the input is zero, and
// only the lower half of the output is wanted. The first stage's radix is even, so
// its sub-transforms see a < R / 2 only and fall into two of half the length.
//
// The sums are those of the transform's definition; the twiddles come from tables
// rounded from long double (one product per stage), as in bgp_fft.cuh.
#pragma once
#include "bgp_fft.cuh"

BGP_NS_BEGIN

struct LPlan {
  int E, n, r[4];
};

// Compiled factorizations: variant 0 has the fewest exchanges its registers allow
// (E <= 16), variant 1 is the alternative with more threads per line (or, for
// lengths 2^a 3, another order), the autotuner of the applies times both; variant 2 has
// the most threads per line (the solver's passes on a grid too small to fill the GPU).
// E is a multiple of every radix, the first radix is even.
BGP_HD constexpr LPlan lplan(int L, int V) {
  switch (L) {
    case 16: return V == 1 ? LPlan{8, 2, {2, 8}} : LPlan{4, 2, {4, 4}};
    case 24: return V ? LPlan{6, 3, {6, 2, 2}} : LPlan{12, 2, {6, 4}};
    case 32: return V ? LPlan{4, 3, {4, 4, 2}} : LPlan{8, 2, {8, 4}};
    case 48: return V ? (V == 1 ? LPlan{12, 3, {4, 4, 3}} : LPlan{6, 4, {6, 2, 2, 2}}) : LPlan{12, 2, {12, 4}};
    case 64: return V ? LPlan{4, 3, {4, 4, 4}} : LPlan{8, 2, {8, 8}};
    case 96: return V == 1 ? LPlan{12, 3, {12, 4, 2}} : LPlan{12, 3, {6, 4, 4}};
    case 128: return V ? (V == 1 ? LPlan{8, 3, {8, 4, 4}} : LPlan{4, 4, {4, 4, 4, 2}}) : LPlan{16, 2, {16, 8}};
    case 192: return V == 1 ? LPlan{12, 3, {4, 4, 12}} : LPlan{12, 3, {12, 4, 4}};
    case 256: return V ? (V == 1 ? LPlan{8, 3, {8, 8, 4}} : LPlan{4, 4, {4, 4, 4, 4}}) : LPlan{16, 2, {16, 16}};
    case 384: return V == 1 ? LPlan{24, 3, {8, 8, 6}} : LPlan{12, 4, {6, 4, 4, 4}};
    case 512: return V ? LPlan{8, 3, {8, 8, 8}} : LPlan{16, 3, {16, 8, 4}};
    case 768: return V == 1 ? LPlan{24, 3, {8, 8, 12}} : LPlan{12, 4, {12, 4, 4, 4}};
    default: return LPlan{1, 1, {1, 1, 1, 1}};   // not compiled
  }
}
constexpr int kLVariants = 3;

// geometry of stage S: P = product of the earlier radices, Lr = what is left of the
// point index after it
BGP_HD constexpr int lf_P(int L, int V, int S) {
  const LPlan p = lplan(L, V);
  int P = 1;
  for (int q = 0; q < S; ++q) P *= p.r[q];
  return P;
}
BGP_HD constexpr int lf_Lr(int L, int V, int S) { return L / (lf_P(L, V, S) * lplan(L, V).r[S]); }
BGP_HD constexpr int lf_threads(int L, int V) { return L / lplan(L, V).E; }
// Exchange after stage S: element (k, m) at row k, column m, rows of odd length (the
// reads of the next stage run along a column, the lanes of a warp on distinct banks).
BGP_HD constexpr int lf_pitch(int Lr) { return Lr | 1; }
// complex slots of one line's exchange buffer (the largest exchange, and the L + 1
// spectral values of the real transforms)
BGP_HD constexpr int lf_slots(int L, int V) {
  int best = L + 1;
  for (int S = 0; S + 1 < lplan(L, V).n; ++S) {
    const int c = (L / lf_Lr(L, V, S)) * lf_pitch(lf_Lr(L, V, S));
    if (c > best) best = c;
  }
  return best | 1;
}
// Twiddle table of a length: for every stage but the last, w_L^(P m b) at b Lr + m
// (b < R, m < Lr), so the lanes of a warp (consecutive m) read consecutive values.
BGP_HD constexpr int lf_tab_off(int L, int V, int S) {
  int o = 0;
  for (int q = 0; q < S; ++q) o += lplan(L, V).r[q] * lf_Lr(L, V, q);
  return o;
}
BGP_HD constexpr int lf_tab_len(int L, int V) { return lf_tab_off(L, V, lplan(L, V).n - 1); }

// ---------------------------------------------------------- register transforms
// cos and sin of 2 pi m / R for the radices 6, 8, 12 and 16
BGP_HD constexpr double lf_cos(int R, int m) {
  const int d = (48 / R) * m % 48;             // in 48ths of a turn
  switch (d) {
    case 0: return 1.0;
    case 3: case 45: return 0.92387953251128675613;
    case 4: case 44: return 0.86602540378443864676;
    case 6: case 42: return 0.70710678118654752440;
    case 8: case 40: return 0.5;
    case 9: case 39: return 0.38268343236508977173;
    case 12: case 36: return 0.0;
    case 15: case 33: return -0.38268343236508977173;
    case 16: case 32: return -0.5;
    case 18: case 30: return -0.70710678118654752440;
    case 20: case 28: return -0.86602540378443864676;
    case 21: case 27: return -0.92387953251128675613;
    default: return -1.0;                      // 24
  }
}
BGP_HD constexpr double lf_sin(int R, int m) { return lf_cos(48, ((48 / R) * m + 36) % 48); }

// v times w_R^m (forward) or its conjugate (inverse), m and R compile-time
template <int R, int M, bool INV, class T>
BGP_HD T lf_rot(T v) {
  using Rt = typename CT<T>::R;
  constexpr int m = M % R;
  if constexpr (m == 0) {
    return v;
  } else if constexpr (4 * m == R) {
    return rot90<INV>(v);
  } else if constexpr (2 * m == R) {
    return cmake<T>(-v.x, -v.y);
  } else if constexpr (4 * m == 3 * R) {
    return rot90<!INV>(v);
  } else if constexpr (8 * m == R) {           // (1 -+ i) / sqrt 2
    return cscale(cadd(v, rot90<INV>(v)), (Rt)kR2);
  } else if constexpr (8 * m == 3 * R) {       // (-1 -+ i) / sqrt 2
    return cscale(csub(rot90<INV>(v), v), (Rt)kR2);
  } else {
    constexpr double c = lf_cos(R, m), s = lf_sin(R, m);
    return cmul(v, cmake<T>((Rt)c, (Rt)(INV ? s : -s)));
  }
}

template <int R, int A, bool INV, class T>
BGP_HD void lf_rot_all(T* v) {           // v[a] *= w_R^a, a < A
  if constexpr (A > 1) {
    lf_rot_all<R, A - 1, INV>(v);
    v[A - 1] = lf_rot<R, A - 1, INV>(v[A - 1]);
  }
}

// R-point transform of v[0..R-1], natural order in and out
template <int R, bool INV, class T>
BGP_HD void lf_dft(T* v) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2 || R == 3 || R == 4 || R == 8) {
    dft_small<R, INV>(v);
  } else if constexpr (R == 6) {
    // prime-factor map: n = 2 a + 3 b, k = 4 p + 3 q (mod 6)
    T x[2][3] = {{v[0], v[2], v[4]}, {v[3], v[5], v[1]}};
    dft_small<3, INV>(x[0]);
    dft_small<3, INV>(x[1]);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      v[(4 * p) % 6] = cadd(x[0][p], x[1][p]);
      v[(4 * p + 3) % 6] = csub(x[0][p], x[1][p]);
    }
  } else if constexpr (R == 12) {
    // prime-factor map: n = 4 a + 3 b, k = 4 p + 9 q (mod 12)
    T x[4][3];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
#pragma unroll
      for (int a = 0; a < 3; ++a) x[b][a] = v[(4 * a + 3 * b) % 12];
      dft_small<3, INV>(x[b]);
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      T y[4] = {x[0][p], x[1][p], x[2][p], x[3][p]};
      dft_small<4, INV>(y);
#pragma unroll
      for (int q = 0; q < 4; ++q) v[(4 * p + 9 * q) % 12] = y[q];
    }
  } else {
    static_assert(R == 16, "radix 1, 2, 3, 4, 6, 8, 12 or 16");
    // 4 x 4: n = 4 a + b, k = p + 4 q
    T x[4][4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
#pragma unroll
      for (int a = 0; a < 4; ++a) x[b][a] = v[4 * a + b];
      dft_small<4, INV>(x[b]);
    }
    x[1][1] = lf_rot<16, 1, INV>(x[1][1]);
    x[1][2] = lf_rot<16, 2, INV>(x[1][2]);
    x[1][3] = lf_rot<16, 3, INV>(x[1][3]);
    x[2][1] = lf_rot<16, 2, INV>(x[2][1]);
    x[2][2] = lf_rot<16, 4, INV>(x[2][2]);
    x[2][3] = lf_rot<16, 6, INV>(x[2][3]);
    x[3][1] = lf_rot<16, 3, INV>(x[3][1]);
    x[3][2] = lf_rot<16, 6, INV>(x[3][2]);
    x[3][3] = lf_rot<16, 9, INV>(x[3][3]);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      T y[4] = {x[0][p], x[1][p], x[2][p], x[3][p]};
      dft_small<4, INV>(y);
#pragma unroll
      for (int q = 0; q < 4; ++q) v[p + 4 * q] = y[q];
    }
  }
}

// forward transform whose inputs a >= R / 2 are zero (v[0..R/2-1] in, R values out)
template <int R, class T>
BGP_HD void lf_dft_half_in(T* v) {
  constexpr int H = R / 2;
  T e[H], o[H];
#pragma unroll
  for (int a = 0; a < H; ++a) { e[a] = v[a]; o[a] = v[a]; }
  lf_rot_all<R, H, false>(o);
  lf_dft<H, false>(e);
  lf_dft<H, false>(o);
#pragma unroll
  for (int b = 0; b < H; ++b) { v[2 * b] = e[b]; v[2 * b + 1] = o[b]; }
}

// inverse transform of which only the outputs a < R / 2 are wanted
template <int R, class T>
BGP_HD void lf_dft_half_out(T* v) {
  constexpr int H = R / 2;
  T e[H], o[H];
#pragma unroll
  for (int b = 0; b < H; ++b) { e[b] = v[2 * b]; o[b] = v[2 * b + 1]; }
  lf_dft<H, true>(e);
  lf_dft<H, true>(o);
  lf_rot_all<R, H, true>(o);
#pragma unroll
  for (int a = 0; a < H; ++a) v[a] = cadd(e[a], o[a]);
}

// ------------------------------------------------------- one thread's stage work
// Stage S of thread t on its registers, forward: the sub-transforms and, but for the
// last stage, the twiddles. HALF: the first stage of a line whose upper half is zero.
template <int L, int V, int S, bool HALF, class C>
BGP_HD void lf_stage_fwd(C (&v)[lplan(L, V).E], const C* tab, int t) {
  constexpr LPlan p = lplan(L, V);
  constexpr int R = p.r[S], NB = p.E / R, T = L / p.E, Lr = lf_Lr(L, V, S), off = lf_tab_off(L, V, S);
#pragma unroll
  for (int s = 0; s < NB; ++s) {
    C x[R];
#pragma unroll
    for (int a = 0; a < (HALF ? R / 2 : R); ++a) x[a] = v[s + NB * a];
    if constexpr (HALF) lf_dft_half_in<R>(x);
    else lf_dft<R, false>(x);
    if constexpr (S + 1 < p.n) {
      const int m = (t + T * s) % Lr;
#pragma unroll
      for (int b = 1; b < R; ++b) x[b] = cmul(x[b], tab[off + b * Lr + m]);
    }
#pragma unroll
    for (int b = 0; b < R; ++b) v[s + NB * b] = x[b];
  }
}
template <int L, int V, int S, bool HALF, class C>
BGP_HD void lf_stage_inv(C (&v)[lplan(L, V).E], const C* tab, int t) {
  constexpr LPlan p = lplan(L, V);
  constexpr int R = p.r[S], NB = p.E / R, T = L / p.E, Lr = lf_Lr(L, V, S), off = lf_tab_off(L, V, S);
#pragma unroll
  for (int s = 0; s < NB; ++s) {
    C x[R];
#pragma unroll
    for (int b = 0; b < R; ++b) x[b] = v[s + NB * b];
    if constexpr (S + 1 < p.n) {
      const int m = (t + T * s) % Lr;
#pragma unroll
      for (int b = 1; b < R; ++b) x[b] = cconjmul(tab[off + b * Lr + m], x[b]);
    }
    if constexpr (HALF) lf_dft_half_out<R>(x);
    else lf_dft<R, true>(x);
#pragma unroll
    for (int a = 0; a < (HALF ? R / 2 : R); ++a) v[s + NB * a] = x[a];
  }
}
// Slots of the exchange between stages S and S + 1: `b`-side (after stage S: element
// b of sub-transform s) and `a`-side (before stage S + 1: element a).
template <int L, int V, int S>
BGP_HD int lf_pos_b(int t, int s, int b) {
  constexpr LPlan p = lplan(L, V);
  constexpr int T = L / p.E, P = lf_P(L, V, S), Lr = lf_Lr(L, V, S);
  const int u = t + T * s;
  return (u / Lr + P * b) * lf_pitch(Lr) + u % Lr;
}
template <int L, int V, int S>
BGP_HD int lf_pos_a(int t, int s, int a) {
  constexpr LPlan p = lplan(L, V);
  constexpr int T = L / p.E, Lr = lf_Lr(L, V, S), Lr2 = lf_Lr(L, V, S + 1);
  const int u = t + T * s;
  return (u / Lr2) * lf_pitch(Lr) + u % Lr2 + Lr2 * a;
}

// Host emulation of a line (all its threads, stage by stage), for the CPU tests.
// x: L values in (natural order), transformed in place; inverse unnormalised.
template <int L, int V, int S, bool INV, bool HALF>
inline void lf_host_stages(double2 (*reg)[lplan(L, V).E], double2* buf, const double2* tab) {
  constexpr LPlan p = lplan(L, V);
  constexpr int T = L / p.E;
  constexpr int Q = INV ? p.n - 1 - S : S;       // the stage run now
  if constexpr (S < p.n) {
    for (int t = 0; t < T; ++t) {
      if constexpr (INV) lf_stage_inv<L, V, Q, HALF && Q == 0>(reg[t], tab, t);
      else lf_stage_fwd<L, V, Q, HALF && Q == 0>(reg[t], tab, t);
    }
    if constexpr (S + 1 < p.n) {
      constexpr int X = INV ? Q - 1 : Q;         // the exchange between X and X + 1
      constexpr int RB = p.r[X], RA = p.r[X + 1];
      for (int t = 0; t < T; ++t) {
        if (!INV) for (int s = 0; s < p.E / RB; ++s) for (int b = 0; b < RB; ++b)
          buf[lf_pos_b<L, V, X>(t, s, b)] = reg[t][s + (p.E / RB) * b];
        if (INV) for (int s = 0; s < p.E / RA; ++s) for (int a = 0; a < RA; ++a)
          buf[lf_pos_a<L, V, X>(t, s, a)] = reg[t][s + (p.E / RA) * a];
      }
      for (int t = 0; t < T; ++t) {
        if (!INV) for (int s = 0; s < p.E / RA; ++s) for (int a = 0; a < RA; ++a)
          reg[t][s + (p.E / RA) * a] = buf[lf_pos_a<L, V, X>(t, s, a)];
        if (INV) for (int s = 0; s < p.E / RB; ++s) for (int b = 0; b < RB; ++b)
          reg[t][s + (p.E / RB) * b] = buf[lf_pos_b<L, V, X>(t, s, b)];
      }
    }
    lf_host_stages<L, V, S + 1, INV, HALF>(reg, buf, tab);
  }
}
template <int L, int V, bool INV, bool HALF>
inline void lf_host_line(double2* x, const double2* tab) {
  constexpr LPlan p = lplan(L, V);
  constexpr int T = L / p.E;
  static double2 reg[T][p.E], buf[lf_slots(L, V)];
  for (int t = 0; t < T; ++t)
    for (int q = 0; q < p.E; ++q) reg[t][q] = x[t + T * q];
  lf_host_stages<L, V, 0, INV, HALF>(reg, buf, tab);
  for (int t = 0; t < T; ++t)
    for (int q = 0; q < p.E; ++q) x[t + T * q] = reg[t][q];
}
// the twiddle table of a length from its L-entry table w_L^t
template <int L, int V, int S = 0>
inline void lf_fill_table(const double2* w, double2* tab) {
  constexpr LPlan p = lplan(L, V);
  if constexpr (S + 1 < p.n) {
    constexpr int P = lf_P(L, V, S), Lr = lf_Lr(L, V, S), off = lf_tab_off(L, V, S);
    for (int b = 0; b < p.r[S]; ++b)
      for (int m = 0; m < Lr; ++m) tab[off + b * Lr + m] = w[(long)P * m * b % L];
    lf_fill_table<L, V, S + 1>(w, tab);
  }
}

#if defined(__CUDACC__)

// The exchange buffer of a tile: slot i of line c at i * LS + c * CS. On a strided
// axis the lines are interleaved (LS = lines, CS = 1), so 8 neighbouring lines fill
// one 128-byte wavefront; on the contiguous axis they are CS apart (LS = 1).
template <int L, int V, int LS, bool WARP, class C = double2>
struct LineFft {
  static constexpr LPlan p = lplan(L, V);
  static constexpr int E = p.E, T = L / E;
  C* sm;              // this line's slot 0
  const C* __restrict__ tab;
  int t;                    // thread of the line
  BGP_D static void sync() { if constexpr (WARP) __syncwarp(); else __syncthreads(); }

  template <int X, bool FWD>
  BGP_D void exchange(C (&v)[E]) const {
    constexpr int RB = p.r[X], RA = p.r[X + 1], NBB = E / RB, NBA = E / RA;
    sync();                 // the previous exchange (or use of the buffer) has been read
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int i = FWD ? lf_pos_b<L, V, X>(t, q % NBB, q / NBB) : lf_pos_a<L, V, X>(t, q % NBA, q / NBA);
      sm[i * LS] = v[q];
    }
    sync();
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int i = FWD ? lf_pos_a<L, V, X>(t, q % NBA, q / NBA) : lf_pos_b<L, V, X>(t, q % NBB, q / NBB);
      v[q] = sm[i * LS];
    }
  }
  template <bool HALF, int S = 0>
  BGP_D void forward(C (&v)[E]) const {
    lf_stage_fwd<L, V, S, HALF && S == 0>(v, tab, t);
    if constexpr (S + 1 < p.n) {
      exchange<S, true>(v);
      forward<HALF, S + 1>(v);
    }
  }
  template <bool HALF, int S = p.n - 1>
  BGP_D void inverse(C (&v)[E]) const {
    lf_stage_inv<L, V, S, HALF && S == 0>(v, tab, t);
    if constexpr (S > 0) {
      exchange<S - 1, false>(v);
      inverse<HALF, S - 1>(v);
    }
  }
};

#endif  // __CUDACC__

BGP_NS_END  // namespace bgp
