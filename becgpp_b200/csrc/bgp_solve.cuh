// The mixed-precision ground-state solver as stream passes: every step of the iteration
// is a short chain of plain launches over all active instances of a size, with all control
// on the device. (The FP64 form runs in bgp_programs.cuh's persistent kernel.) It follows
// the Riemannian PCG of becgpp/solvers.py:48-235:
//   preconditioner   sigma = max(lower median of V + 2 b2 rho + 3 b3 rho^2 (+phi)
//                    over rho > 0.05 max rho, shift_min); z = P_T[(k^2/2+sigma)^-1 g]
//   beta             pr_precond <z, g-g_prev>/<z_prev, g_prev> | pr | none,
//                    restart every cg_restart iterations
//   direction        P_T(z + beta dir), falling back to z, then P_T(g) when not descent
//   step             alpha <- alpha/2 + clamp(<s,s>/<s,y>)/2, clamped
//   Armijo           psi_t = (psi - t dir)/||.||, E_t <= E - c1 t <g,dir>, halving
//   stops            residual < res_tol, windowed energy plateau, stalled line search
//
// A step of a plane instance is four launches:
//   trial  w = psi - t dirc on every axis's lines: norm, energy and spectral sums; the
//          contiguous lines also store w (and dirc) and A = T_y w, the first axis term
//          of H w, while their spectrum is in registers
//   hx     x-lines: g = A + T_x w + pot w - mu w, its norm, the median keys, and B = the
//          x-transform of g
//   pz     y-lines: transform, divide by k^2/2 + sigma, inverse
//   px     x-lines: inverse: z, and every inner product of the next direction
// (a volume has hy, and y transforms around pz; a long-range kernel adds its
// convolution passes). What a pass cannot know before its sums are complete is decided
// by the last CTA of an instance to finish it: it adds the CTAs' partial sums in a fixed
// order and one thread runs the scalar control (ctl_*), which sets the state that says
// which of the following launches have work for the instance; the others return at
// once. A rejected trial or a wide median search simply repeats in the next step.
//
// mu is the energy's own derivative, E + Econtact + 2 Ethree + Egrav, so g forms in the
// same pass as H psi. The products with the projected z = z_raw - a psi, a = <psi, z_raw>,
// follow from those with z_raw, and <z_prev, g_prev>, |g_prev|^2 are the last
// iteration's <z, g>, |g|^2, so z and the sums share a pass.
//
// Precision. An instance starts with complex64 pool fields and FP32 line transforms (norms,
// energies, inner products and the median in FP64, a trial state rounded to its storage
// before its sums are taken, the long-range potential FP64) and hands over to FP64 fields
// and transforms once its residual is below mixed_switch_res or after kSvFailSwitch failed
// line searches in a row: the state is widened and normalised again, energy, potential and
// gradient are formed afresh, the recurrence restarts. Convergence is declared in FP64.
//
// Why not one persistent kernel: with a team barrier (3 us) after each of about ten
// phases, four lines a CTA and 128-thread teams, an iteration of one 256^2 instance took
// 91 us, most of it barrier and control latency and instruction fetch; a launch of this
// chain is about 4 us.
#pragma once
#include "bgp_programs.cuh"
#include "bgp_stream.cuh"

BGP_NS_BEGIN

enum SvState : int { ST_INIT, ST_TRIAL, ST_FINAL, ST_SWITCH, ST_CONV, ST_POLYB, ST_POLYC, ST_H, ST_MED, ST_PRE, ST_DONE };
enum SvKind : int { KD_ITER, KD_INIT, KD_FINAL, KD_SWITCH };   // what the energy and gradient under way are for
// Configurations of the solver passes (tile width, factorization), by the size of a group
// of instances: see sv_step in bgp_api.cu.
// Resident CTAs per SM their registers are budgeted for: one where a tile has an SM to
// itself (V = 2), else 384 threads in tiles of 4 lines and 512 in tiles of 8.
BGP_HD constexpr int sv_blocks(int L, int C, int V) {
  const int b = (C == 8 ? 512 : 384) / s_threads(L, C, V);
  return (b < 1 || (V == 2 && C < 8)) ? 1 : (b > 16 ? 16 : b);
}
constexpr int kSvSmall = 4;                          // lines per tile on a grid too small to fill the GPU
constexpr int kSvCap = 1024;                         // median keys ranked by one CTA
constexpr int kSvWin = 96;                           // keys wanted in the median window
constexpr int kSvGather = 256;                       // a radix bucket this small is gathered and ranked
constexpr int kSvFailSwitch = 3;                     // failed line searches that end the FP32 phase
constexpr int kSvDigit = 11, kSvBins = 1 << kSvDigit;

// direction sums (raw z), see px
enum : int { D_PZX, D_PZY, D_ZY, D_PYX, D_PYY, D_GY, D_PDX, D_PDY, D_ZG, D_GD, D_GPX, D_GPY, D_SY, D_SS, kDSums };

// Control state of an instance.
struct SvCtl {
  int st, kind, have_dirc, refresh, poly_phi;
  int f[F_NLOG];
  double sc[F_NLOG];
  int hf;                             // the state of the gradient under way: field, scale
  double hc;
  int phi_cur;
  double phisc, phisc_old;
  int fp32, fp64_from, sw_accepted;   // FP32 phase; iteration of the hand-over (-1: none); it follows a step
  int it, n_iter, n_fail, ls, stop, converged, it_ref, ntrials, ntrace, naccept, use_best, cg_reset;
  double E, E_ref, Et, ct, alpha, t, gd, beta, sigma, mu, ra, rr, best, maxrho;
  double cz, cd, cg;
  double2 cpsi;
  double zg, zg_prev, gg, gg_prev;
  double rec[kNRec], d[kDSums], qG[6];
  double mu_last;                     // of the last iterate
  double Ef, muf, massf;              // of the returned state
  // median
  double med_prev, med_eps;
  int med_valid, win_on, level, gather;
  unsigned long long win_lo, win_hi, prefix, rank;
  double nkeys, below;
};

// Counters of an instance that CTAs update while a pass runs (kept off the lines of the
// control state, which every CTA reads through L1).
struct alignas(128) SvSync {
  unsigned cnt;                       // tiles of the pass under way that are done
  unsigned wcount;                    // median keys gathered (window or bucket)
};

// Everything a pass needs about its instance (device memory, written once per solve).
struct SvInst {
  int ndim, N, n, M, kern, poly;
  double dx, dv, kfac, s, tc, beta2, beta3, Omega, inv_n, conv_scale;
  double2* pool;
  double* phi2;
  double2 *cb1, *cb2;
  const double* Kq;
  const double2* twM;
  const double2* tabN[kLVariants];
  const double2* tabM[kLVariants];
  const float2* tabF[kLVariants];     // tabN in FP32
  unsigned long long *keys, *wcand;
  unsigned* hist;                     // kSvBins
  double* part;
  const double2* in_psi;
  double2* out_c;
  SolverParams sp;
  double* trace;
  SolveOut* out;
  int* hstate;                        // its state as the host sees it (mapped memory)
};

// A pass over the active instances: work item w is tile w % tiles of the (w / tiles)-th
// active instance. The grid is at most what fits on the GPU and strides over the items,
// so a launch with nothing to do costs one wave.
constexpr int kSvInline = 8;          // active lists this short travel in the parameters
struct SvLaunch {
  const SvInst* insts;
  SvCtl* ctls;
  SvSync* sync;
  const int* act;
  int tiles, nact;
  int inl[kSvInline];
};

#if defined(__CUDACC__)

BGP_D double2* sv_field(const SvInst& I, int b) { return I.pool + (size_t)b * I.n; }

// ------------------------------------------------------------ scalar control
// (one thread of the last CTA of a pass)

BGP_D int sv_alloc(const SvCtl& S) {
  unsigned used = 0u;
#pragma unroll
  for (int q = 0; q < F_NLOG; ++q)
    if (S.f[q] >= 0) used |= 1u << S.f[q];
  if (S.hf >= 0) used |= 1u << S.hf;
  return __ffs(~used & ((1u << kNB) - 1u)) - 1;
}

BGP_D void sv_assemble(const SvInst& I, const double* s, double c2, double* comp) {
  const double dv = I.dv, inv = 1.0 / (double)I.N, c4 = c2 * c2;
  comp[1] = 0.5 * (s[S_KX] + s[S_KY] + s[S_KZ]) * inv * dv * c2;
  comp[2] = s[S_V] * dv * c2;
  comp[3] = 0.5 * I.beta2 * s[S_2] * dv * c4;
  comp[4] = (I.beta3 / 3.0) * s[S_3] * dv * (c4 * c2);
  comp[7] = (s[S_LY] - s[S_LX]) * inv * dv * c2;
  comp[5] = -I.Omega * comp[7];
  comp[6] = I.kern ? 0.5 * s[S_G] * dv * c4 : 0.0;
  comp[0] = comp[1] + comp[2] + comp[3] + comp[4] + comp[5] + comp[6];
}

BGP_D void sv_window(SvCtl& S) {
  S.win_on = S.med_valid;
  if (S.med_valid) {
    const double w = fabs(S.med_prev) * S.med_eps + 1e-300;
    S.win_lo = dkey(S.med_prev - w);
    S.win_hi = dkey(S.med_prev + w);
  }
}

// the solve ends: the lowest-residual iterate goes out and is evaluated afresh
BGP_D void sv_finish(SvCtl& S) {
  S.use_best = S.best < S.rr;
  S.mu_last = S.mu;
  const int fb = S.use_best ? F_BEST : F_PSI;
  const int keep = S.f[fb];
  const double sc = S.sc[fb];
#pragma unroll
  for (int q = 0; q < F_NLOG; ++q) if (q != F_A && q != F_H) S.f[q] = -1;
  S.f[F_PSI] = keep; S.sc[F_PSI] = sc;
  S.hf = keep;
  S.f[F_W] = sv_alloc(S);
  S.kind = KD_FINAL;
  S.st = ST_FINAL;
}

// the hand-over to FP64: the state is widened into a free field and evaluated afresh, the
// fields of earlier iterates are not read again
BGP_D void sv_switch(SvCtl& S, int accepted) {
  const int keep = S.f[F_PSI];
#pragma unroll
  for (int q = 0; q < F_NLOG; ++q) if (q != F_A && q != F_H) S.f[q] = -1;
  S.f[F_PSI] = keep;
  S.hf = keep;
  S.f[F_W] = sv_alloc(S);
  S.sw_accepted = accepted;
  S.kind = KD_SWITCH;
  S.st = ST_SWITCH;
}

// the direction and first step of iteration S.it from the sums of px; d_is_z: the last
// direction is z itself (after a failed line search)
BGP_D void sv_direction(const SvInst& I, SvCtl& S, bool d_is_z) {
  const SolverParams& P = I.sp;
  const double dv = I.dv;
  const double* r = S.d;
  const double2 a = cmk(r[D_PZX] * dv, r[D_PZY] * dv);           // <psi, z_raw> dV
  const double2 gpsi = cmk(r[D_GPX], r[D_GPY]);                  // sum conj(g) psi
  const double zy = r[D_ZY] - (a.x * r[D_PYX] + a.y * r[D_PYY]); // sum Re conj(z) (g - g_prev)
  const double zg = r[D_ZG] - (a.x * gpsi.x - a.y * gpsi.y);     // sum Re conj(g) z
  double beta = 0.0;
  if (!(S.it == 0 || S.cg_reset || P.cg_beta == 2 || (P.restart > 0 && S.it % P.restart == 0))) {
    if (P.cg_beta == 0) beta = fmax(0.0, (zy * dv) / fmax(S.zg_prev * dv, 1e-300));
    else beta = fmax(0.0, (r[D_GY] * dv) / fmax(S.gg_prev * dv, 1e-300));
    if (!isfinite(beta)) beta = 0.0;
  }
  S.beta = beta;
  S.zg = zg;
  // dirc = z + beta d - b psi,  b = <psi, z + beta d> dV (z is already projected)
  const double2 b = d_is_z ? cmk(0.0, 0.0) : cmk(beta * r[D_PDX] * dv, beta * r[D_PDY] * dv);
  const double gdd = d_is_z ? zg : r[D_GD];
  double gd = (zg + beta * gdd - (b.x * gpsi.x - b.y * gpsi.y)) * dv;
  S.cg = 0.0;
  if (d_is_z) { S.cz = 1.0 + beta; S.cd = 0.0; S.cpsi = cscale(a, -(1.0 + beta)); }
  else { S.cz = 1.0; S.cd = beta; S.cpsi = cmk(-(a.x + b.x), -(a.y + b.y)); }
  if (gd <= 0.0) {
    S.cz = 1.0; S.cd = 0.0; S.cpsi = cmk(-a.x, -a.y);
    gd = zg * dv;
  }
  if (gd <= 0.0) {
    // P_T(g) = g - psi <psi, g>,  <psi, g> = conj(sum conj(g) psi)
    const double2 pg = cmk(gpsi.x * dv, -gpsi.y * dv);
    S.cz = 0.0; S.cd = 0.0; S.cg = 1.0; S.cpsi = cmk(-pg.x, -pg.y);
    gd = (S.gg - (pg.x * gpsi.x - pg.y * gpsi.y)) * dv;
  }
  S.gd = gd;
  if (S.it > 0 && !S.cg_reset) {
    const double sy = r[D_SY] * dv;
    if (sy > 1e-30 && isfinite(sy)) {
      double bb = (r[D_SS] * dv) / sy;
      if (isfinite(bb)) {
        bb = fmin(fmax(bb, P.bb_min), P.bb_max);
        S.alpha = (1.0 - P.bb_mix) * S.alpha + P.bb_mix * bb;
      }
    }
  }
  S.alpha = fmin(fmax(S.alpha, P.alpha_min), P.alpha_max);
  S.cg_reset = 0;
  S.t = S.alpha;
  S.ls = 0;
  S.f[F_DIRC] = -1; S.f[F_W] = -1;
  S.f[F_DIRC] = sv_alloc(S);
  S.f[F_W] = sv_alloc(S);
  S.have_dirc = 0;
  S.kind = KD_ITER;
  S.st = I.poly ? ST_POLYB : ST_TRIAL;
}

// the next iteration begins (after a residual), or the solve ends at maxit
BGP_D bool sv_next_iter(const SvInst& I, SvCtl& S) {
  S.it += 1;
  if (S.it >= I.sp.maxit) { sv_finish(S); return false; }
  S.n_iter = S.it + 1;
  return true;
}

// the energy of the state under way is known (S.rec complete)
BGP_D void sv_energy_known(const SvInst& I, SvCtl& S) {
  const SolverParams& P = I.sp;
  const double dv = I.dv;
  double comp[8];
  if (S.kind == KD_FINAL) {
    sv_assemble(I, S.rec, 1.0, comp);
    S.Ef = comp[0];
    S.massf = S.rec[S_N0] * dv;
    S.muf = comp[0] + comp[3] + 2.0 * comp[4] + comp[6];
    S.mu = S.muf;
    S.hf = S.f[F_W]; S.hc = 1.0;
    S.phi_cur = 1 - S.phi_cur; S.phisc = 1.0; S.poly_phi = 0;
    S.win_on = 0;
    S.f[F_G] = sv_alloc(S);
    S.st = ST_H;
    return;
  }
  const double c = 1.0 / sqrt(S.rec[S_N0] * dv), c2 = c * c;
  sv_assemble(I, S.rec, c2, comp);
  S.Et = comp[0]; S.ct = c;
  if (S.kind == KD_ITER) {
    S.ntrials++;
    if (!(isfinite(S.Et) && S.Et <= S.E - P.c1 * S.t * S.gd)) {
      S.t = S.t * P.shrink;
      S.ls += 1;
      if (S.ls < P.ls_max && !(S.t < P.alpha_min)) { S.st = ST_TRIAL; return; }
      // failed line search
      S.n_fail++;
      S.alpha = fmax(S.alpha * 0.5, P.alpha_min);
      S.f[F_DIRC] = -1; S.f[F_W] = -1; S.f[F_DIR] = -1;
      if (S.fp32) {
        // repeated failures mean the energy change has reached the FP32 floor
        if (S.n_fail >= kSvFailSwitch || S.alpha <= P.alpha_min) { sv_switch(S, 0); return; }
      } else if (S.alpha <= P.alpha_min || S.n_fail >= P.stall_max) {
        S.stop = kStopStalled;
        sv_finish(S);
        return;
      }
      if (!sv_next_iter(I, S)) return;
      sv_direction(I, S, true);
      return;
    }
    S.n_fail = 0;
    S.naccept++;
    S.f[F_PSIP] = S.f[F_PSI]; S.sc[F_PSIP] = S.sc[F_PSI];
    S.f[F_GP] = S.f[F_G]; S.f[F_G] = -1;
    S.zg_prev = S.zg; S.gg_prev = S.gg;
    S.f[F_Z] = -1;
    S.f[F_DIR] = S.f[F_DIRC]; S.f[F_DIRC] = -1;
    S.alpha = fmin(P.alpha_max, S.t * P.growth);
  }
  S.E = S.Et;
  S.f[F_PSI] = S.f[F_W]; S.sc[F_PSI] = c; S.f[F_W] = -1;
  if (S.kind != KD_ITER) { S.f[F_PSIP] = S.f[F_PSI]; S.sc[F_PSIP] = c; }
  S.phisc_old = S.phisc;
  S.phi_cur = 1 - S.phi_cur; S.phisc = c2;
  S.mu = comp[0] + comp[3] + 2.0 * comp[4] + comp[6];
  S.maxrho = S.rec[kNSum] * c2;
  S.hf = S.f[F_PSI]; S.hc = c;
  S.f[F_G] = sv_alloc(S);
  sv_window(S);
  S.st = ST_H;
  S.poly_phi = 0;
  if (I.poly && S.kind == KD_ITER) {
    // the accepted state's potential from its parts, or every 32 accepted steps by its
    // own convolution (so rounding cannot build up over the updates)
    if (S.naccept % 32 == 0) { S.refresh = 1; S.st = ST_CONV; }
    else S.poly_phi = 1;
  }
}

// sums of the trial pass: tot = N0, V, 2, 3, K, L of the contiguous axis, max rho, then
// K, L of axis 0 (and axis 1 in 3D)
BGP_D void sv_ctl_trial(const SvInst& I, SvCtl& S, const double* tot) {
#pragma unroll
  for (int q = 0; q < kNRec; ++q) S.rec[q] = 0.0;
  S.rec[S_N0] = tot[0]; S.rec[S_V] = tot[1]; S.rec[S_2] = tot[2]; S.rec[S_3] = tot[3];
  S.rec[kNSum] = tot[6];
  S.rec[S_KX] = tot[7]; S.rec[S_LX] = tot[8];
  if (I.ndim == 2) { S.rec[S_KY] = tot[4]; S.rec[S_LY] = tot[5]; }
  else { S.rec[S_KZ] = tot[4]; S.rec[S_KY] = tot[9]; S.rec[S_LY] = tot[10]; }
  S.have_dirc = 1;
  if (S.kind == KD_FINAL || S.kind == KD_SWITCH) S.fp32 = 0;   // w is complex128
  if (I.kern && !(I.poly && S.kind == KD_ITER)) { S.refresh = 0; S.st = ST_CONV; return; }
  if (I.poly) {
    const double* G = S.qG;
    const double t = S.t;
    S.rec[S_G] = (((G[5] * t - 4.0 * G[4]) * t + (2.0 * G[2] + 4.0 * G[3])) * t - 4.0 * G[1]) * t + G[0];
  }
  sv_energy_known(I, S);
}

// sums of a convolution's last pass: phi a, phi b, phi c, phi_a a (3D line search), or
// phi |w|^2
BGP_D void sv_ctl_conv(const SvInst& I, SvCtl& S, const double* tot) {
  if (S.st == ST_POLYB) {
    S.qG[1] = tot[0]; S.qG[3] = tot[1]; S.qG[4] = tot[2]; S.qG[0] = tot[3];
    S.have_dirc = 1;
    S.st = ST_POLYC;
  } else if (S.st == ST_POLYC) {
    S.qG[2] = tot[0]; S.qG[5] = tot[2];
    S.st = ST_TRIAL;
  } else if (S.refresh) {
    S.refresh = 0;
    S.st = ST_H;
  } else {
    S.rec[S_G] = tot[0];
    sv_energy_known(I, S);
  }
}

// the preconditioner's shift is known: `sig`, the median (or its floor)
BGP_D void sv_sigma(const SvInst& I, SvCtl& S, double sig) {
  if (S.nkeys > 0.5) { S.med_prev = sig; S.med_valid = 1; }
  S.sigma = fmax(sig, I.sp.shift_min);
  S.f[F_Z] = sv_alloc(S);
  S.st = ST_PRE;
}

// residual known (ra, rr set): bookkeeping and stop tests; true when the iteration goes on
BGP_D bool sv_residual(const SvInst& I, SvCtl& S) {
  const SolverParams& P = I.sp;
  if (S.kind == KD_FINAL) {
    SolveOut o;
    o.iters = S.n_iter; o.stop = S.stop; o.converged = S.converged; o.ntrials = S.ntrials;
    o.ntrace = S.ntrace; o.best_is_final = S.use_best; o.status = 0; o.pad_ = S.naccept;
    o.E = S.E; o.resid_rel = S.rr; o.resid_abs = S.ra; o.best_resid = S.best;
    o.sigma = S.sigma; o.mu = S.mu_last; o.alpha = S.alpha; o.maxrho = S.maxrho;
    const double raf = sqrt(S.gg * I.dv);
    o.E_final = S.Ef; o.mu_final = S.muf; o.resid_abs_final = raf;
    o.resid_rel_final = raf / fmax(1.0, fabs(S.muf)); o.mass_final = S.massf;
    o.fp64_from = S.fp64_from; o.pad2_ = 0;
    *I.out = o;
    S.st = ST_DONE;
    return false;
  }
  S.ra = sqrt(S.gg * I.dv);
  S.rr = S.ra / fmax(1.0, fabs(S.mu));
  if (S.kind == KD_INIT) {
    S.f[F_GP] = S.f[F_G];
    S.f[F_BEST] = S.f[F_PSI]; S.sc[F_BEST] = S.sc[F_PSI];
    S.best = S.rr;
    S.E_ref = S.E; S.it_ref = 0;
    S.gg_prev = S.gg;
    if (P.record_trace && S.ntrace < P.trace_cap) {
      I.trace[0] = 0.0; I.trace[1] = S.E; I.trace[2] = NAN;
      S.ntrace = 1;
    }
    S.it = -1;
    return sv_next_iter(I, S);
  }
  if (S.fp32 && S.rr < P.mixed_tol) { sv_switch(S, 1); return false; }
  if (S.kind == KD_SWITCH) {
    S.fp64_from = S.it;
    S.f[F_GP] = S.f[F_G];
    S.n_fail = 0; S.cg_reset = 1;
    S.best = S.rr;
    S.f[F_BEST] = S.f[F_PSI]; S.sc[F_BEST] = S.sc[F_PSI];
    S.E_ref = S.E; S.it_ref = S.it;
    S.gg_prev = S.gg;
    if (!S.sw_accepted) return sv_next_iter(I, S);   // after failed line searches: no stop tests
  }
  if (P.record_trace && S.ntrace < P.trace_cap) {
    double* tr = I.trace + 3 * S.ntrace;
    tr[0] = (double)(S.it + 1); tr[1] = S.E; tr[2] = S.rr;
    S.ntrace++;
  }
  if (S.rr < S.best) {
    S.best = S.rr;
    S.f[F_BEST] = S.f[F_PSI]; S.sc[F_BEST] = S.sc[F_PSI];
  }
  bool stop = false;
  if (S.fp32) {
    // convergence is declared in FP64 only
  } else if (S.rr < P.res_tol) { S.converged = 1; S.stop = kStopConverged; stop = true; }
  else if (S.it - S.it_ref >= P.window) {
    const double dE = fabs(S.E - S.E_ref) / fmax(1.0, fabs(S.E));
    if (dE < P.etol) { S.converged = 1; S.stop = kStopEnergy; stop = true; }
    else { S.E_ref = S.E; S.it_ref = S.it; }
  }
  if (stop) { sv_finish(S); return false; }
  return sv_next_iter(I, S);
}

// ------------------------------------------------------------ pass skeleton
template <class S> BGP_D void sv_copy(S* dst, const S* src);

// CTA-wide totals of nv <= 16 lists of len partial sums (list q at p + q len); list `mx`
// takes the maximum. 2 W threads per list add its values in a fixed order, all lists at
// once. In shared tot.
template <int W>
BGP_D void sv_gather(const double* p, int nv, int len, int mx, double* tot) {
  constexpr int G = 2 * W > 32 ? 32 : 2 * W, U = 16;
  const int q = threadIdx.x / G, g = threadIdx.x % G;
  double x = 0.0;
  if (q < nv) {
    const double* a = p + (size_t)q * len;
    for (int i = g; i < len; i += G * U) {
      double y[U];
#pragma unroll
      for (int u = 0; u < U; ++u) y[u] = i + G * u < len ? __ldcg(a + i + G * u) : 0.0;
#pragma unroll
      for (int u = 0; u < U; ++u) x = q == mx ? fmax(x, y[u]) : x + y[u];
    }
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const double z = __shfl_xor_sync(0xffffffffu, x, o);
    x = q == mx ? fmax(x, z) : x + z;
  }
  if (g == 0 && q < nv) tot[q] = x;
}

// Sums of NV <= 16 values over the CTA (W warps) in a fixed order; value q of list q goes
// to part[q * len + tile]. Each warp reduces by a reduce-scatter (16 shuffles for up to
// 16 values; lane l ends with value scat(l)), then thread q adds the warps' totals of
// value q. Value `mx` takes the maximum.
template <int W, int NV>
BGP_D void sv_partials(const double (&v)[NV], double* part, int len, int tile, int mx = -1) {
  __shared__ double red[16 * W];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double x[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) x[q] = q < NV ? v[q] : 0.0;
  int idx = 0;
#pragma unroll
  for (int n = 8, o = 16; n >= 1; n >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int q = 0; q < n; ++q) {
      const double keep = up ? x[q + n] : x[q], send = up ? x[q] : x[q + n];
      const double y = __shfl_xor_sync(0xffffffffu, send, o);
      const bool m = mx >= 0 && idx + (up ? n : 0) + q == mx;
      x[q] = m ? fmax(keep, y) : keep + y;
    }
    if (up) idx += n;
  }
  const double z = __shfl_xor_sync(0xffffffffu, x[0], 1);
  x[0] = idx == mx ? fmax(x[0], z) : x[0] + z;
  if ((lane & 1) == 0) red[idx * W + w] = x[0];
  __syncthreads();
  for (int q = threadIdx.x; q < NV; q += W * 32) {
    double s = red[q * W];
#pragma unroll
    for (int k = 1; k < W; ++k) s = q == mx ? fmax(s, red[q * W + k]) : s + red[q * W + k];
    __stcg(part + (size_t)q * len + tile, s);
  }
  __syncthreads();
}

// Arrival of a CTA that has written the partial sums of `mine` tiles: true in every thread
// when all `total` tiles of the pass are done, and then sees all of them. (A CTA arrives
// once for its tiles of an instance: the fence and the atomic take about 2 us.)
BGP_D bool sv_last(SvSync* sy, unsigned mine, unsigned total) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(&sy->cnt, mine) + mine == total;
    if (last) { sy->cnt = 0u; __threadfence(); }
  }
  __syncthreads();
  return last != 0;
}

// the control state back to memory, and what it asks for next to the host (of a plane only
// that it is done: the write to host memory costs the pass about 1 us)
BGP_D void sv_publish(const SvInst& I, const SvCtl* cs, SvCtl* gctl) {
  sv_copy(gctl, cs);
  if (threadIdx.x == 0 && (I.ndim == 3 || cs->st == ST_DONE)) *(volatile int*)I.hstate = cs->st;
}

// The control step of the last CTA: f(totals of its partial sums) on the shared copy of
// the control state (all threads), which then goes back to memory. (One thread's scalar
// code on the state in global memory took about 20 us, a chain of dependent loads.)
template <int W, int NV, class F>
BGP_D void sv_control(const SvInst& I, SvCtl* cs, SvCtl* gctl, int nv, int len, int mx, F f) {
  __shared__ double tot[NV];
  if (nv) sv_gather<W>(I.part, nv, len, mx, tot);
  __syncthreads();
  f(tot);
  __syncthreads();
  sv_publish(I, cs, gctl);
}

template <class T> BGP_D const T* sv_tab(const SvInst& I, int V);
template <> BGP_D const double2* sv_tab<double2>(const SvInst& I, int V) { return I.tabN[V]; }
template <> BGP_D const float2* sv_tab<float2>(const SvInst& I, int V) { return I.tabF[V]; }
template <class T> BGP_D T ldf(const double2* p, size_t f) { return reinterpret_cast<const T*>(p)[f]; }
template <class T> BGP_D void stf(double2* p, size_t f, T v) { reinterpret_cast<T*>(p)[f] = v; }

// words of 8 bytes of a description or control state, copied by the CTA
template <class S>
BGP_D void sv_copy(S* dst, const S* src) {
  static_assert(sizeof(S) % 8 == 0, "copied as words of 8 bytes");
  for (int q = threadIdx.x; q < (int)(sizeof(S) / 8); q += blockDim.x)
    reinterpret_cast<unsigned long long*>(dst)[q] = reinterpret_cast<const unsigned long long*>(src)[q];
}
// a constant table into this SM's L1
BGP_D void sv_prefetch(const double2* tab, int len) {
  for (int q = 8 * threadIdx.x; q < len; q += 8 * blockDim.x)
    asm volatile("prefetch.global.L1 [%0];" ::"l"(tab + q));
}

// The work items of a CTA. The instance's description and control state are brought into
// shared memory once per instance (field by field from L2 they cost a chain of misses),
// what is constant through the solve (the first description, the twiddles of length L)
// before the wait for the previous pass. An item sees I, ctl (shared), gctl, sy, st and
// tile, and is left by `continue`.
#define SV_FOR_ITEMS(TAB, LEN)                                                             \
  __shared__ SvInst is_;                                                                   \
  __shared__ SvCtl cs_;                                                                    \
  pdl_trigger();                                                                           \
  const int items_ = SL.tiles * SL.nact;                                                   \
  int have_i_ = -1, have_c_ = -1;                                                          \
  [[maybe_unused]] unsigned mine_ = 0;                                                     \
  if (SL.nact <= kSvInline) {                                                              \
    have_i_ = SL.inl[(blockIdx.x / SL.tiles) & (kSvInline - 1)];                           \
    sv_copy(&is_, SL.insts + have_i_);                                                     \
    __syncthreads();                                                                       \
    sv_prefetch(is_.TAB, LEN);                                                             \
  }                                                                                        \
  pdl_wait();                                                                              \
  for (int item_ = blockIdx.x; item_ < items_; item_ += gridDim.x)
#define SV_ITEM                                                                            \
  const int a_ = item_ / SL.tiles, tile = item_ - a_ * SL.tiles;                           \
  const int inst_ = SL.nact <= kSvInline ? SL.inl[a_ & (kSvInline - 1)] : SL.act[a_];      \
  [[maybe_unused]] SvCtl* const gctl = SL.ctls + inst_;                                    \
  [[maybe_unused]] SvSync* const sy = SL.sync + inst_;                                     \
  if (inst_ != have_c_) {                                                                  \
    __syncthreads();                                                                       \
    sv_copy(&cs_, gctl);                                                                   \
    if (inst_ != have_i_) sv_copy(&is_, SL.insts + inst_);                                 \
    __syncthreads();                                                                       \
    have_c_ = have_i_ = inst_;                                                             \
  }                                                                                        \
  const SvInst& I = is_;                                                                   \
  SvCtl* const ctl = &cs_;                                                                 \
  const int st = ctl->st;
// the CTA's last item of the instance arrives for all of them; the others go on
#define SV_ARRIVE                                                                          \
  mine_ += 1;                                                                              \
  if (item_ + (int)gridDim.x < items_ && (item_ + (int)gridDim.x) / SL.tiles == a_) continue; \
  const unsigned all_ = mine_;                                                             \
  mine_ = 0;                                                                               \
  if (!sv_last(sy, all_, (unsigned)SL.tiles)) continue;

// line (i, j[, k]) of a strided tile along axis AX (0: x, 1: y in 3D): base and stride
// of its elements and the coordinate indices of its fixed axes
template <int N, int C, int AX>
BGP_D void sv_line(int ndim, int tile, int c, int& base, int& str, int& i, int& j, int& k) {
  i = j = k = 0;
  if (ndim == 2) { j = tile * C + c; base = j; str = N; return; }
  constexpr int tpl = N / C;
  const int a = tile / tpl;
  k = (tile - a * tpl) * C + c;
  if (AX == 1) { i = a; base = a * N * N + k; str = N; }
  else { j = a; base = a * N + k; str = N * N; }
}

// the trap tc r^s; its parameters are copied to registers (a load from the description
// would be repeated after every store)
struct SvTrap { double s, tc; };
BGP_D double sv_trap(const SvTrap& P, double r2) {
  return (P.s <= 0.0) ? 0.0 : ((P.s == 2.0) ? P.tc * r2 : P.tc * pow(r2, 0.5 * P.s));
}

// the direction's operands
struct SvDir {
  const double2 *psi, *z, *d, *g, *dirc;
  double psc, cz, cd, cg, t;
  double2 cpsi;
};
BGP_D SvDir sv_dir(const SvInst& I, const SvCtl& S) {
  SvDir D;
  D.psi = sv_field(I, S.f[F_PSI]);
  D.psc = S.sc[F_PSI];
  D.cz = S.cz; D.cd = S.cd; D.cg = S.cg; D.cpsi = S.cpsi; D.t = S.t;
  D.z = sv_field(I, S.f[F_Z]);
  D.d = S.cd != 0.0 ? sv_field(I, S.f[F_DIR]) : D.z;
  D.g = S.cg != 0.0 ? sv_field(I, S.f[F_G]) : D.z;
  D.dirc = sv_field(I, S.f[F_DIRC]);
  return D;
}
// The fields psi and dirc are formed from at one element: a caller loads a batch of
// elements before it stores any (a load cannot be moved above a store that may alias).
template <class T>
struct SvRaw { T p, a, b; };
template <class T>
BGP_D SvRaw<T> sv_load(const SvDir& D, bool have, size_t f) {
  SvRaw<T> r;
  r.p = ldf<T>(D.psi, f);
  r.a = have ? ldf<T>(D.dirc, f) : (D.cz != 0.0 ? ldf<T>(D.z, f) : ldf<T>(D.g, f));
  r.b = (!have && D.cd != 0.0) ? ldf<T>(D.d, f) : cmake<T>(0, 0);
  return r;
}
// psi (normalised) and dirc, dirc combined from its parts (rounded to the storage type)
// or as read
template <class T>
BGP_D void sv_psi_dirc(const SvDir& D, bool have, const SvRaw<T>& r, double2& p, double2& d) {
  p = cscale(to_d(r.p), D.psc);
  if (have) { d = to_d(r.a); return; }
  double2 v = cscale(to_d(r.a), D.cz != 0.0 ? D.cz : D.cg);
  if (D.cd != 0.0) v = cadd(v, cscale(to_d(r.b), D.cd));
  v = cadd(v, cmul(D.cpsi, p));
  d = to_d(to_c<T>(v));
}

// --------------------------------------------------------------------- trial
template <int N, int C, int V>
__global__ void __launch_bounds__(s_threads(N, C, V), sv_blocks(N, C, V))
    k_sv_trial(const __grid_constant__ SvLaunch SL) {
  constexpr int TH = lf_threads(N, V), E = lplan(N, V).E, W = s_threads(N, C, V) / 32;
  extern __shared__ double2 sm[];
  SV_FOR_ITEMS(tabN[V], lf_tab_len(N, V)) {
  SV_ITEM
  if (st > ST_SWITCH) continue;                  // ST_INIT, ST_TRIAL, ST_FINAL, ST_SWITCH
  auto body = [&](auto tag_) {
  using T = decltype(tag_);
  const int ndim = I.ndim, nt = SL.tiles / ndim;     // tiles of one axis
  const int slot = tile / nt, tl_ = tile - slot * nt;
  const bool have = ctl->have_dirc != 0;
  const double2* src = st == ST_INIT ? I.in_psi : sv_field(I, ctl->f[F_PSI]);
  const double ssc = ctl->sc[F_PSI];
  SvDir D{};
  if (st == ST_TRIAL) D = sv_dir(I, *ctl);
  // the state w of an element from what was loaded for it (and its direction d)
  auto load = [&](size_t f) -> SvRaw<T> {
    if (st == ST_TRIAL) return sv_load<T>(D, have, f);
    SvRaw<T> r{};
    if (st == ST_INIT) r.p = to_c<T>(__ldg(src + f));
    else if (ctl->fp32) r.p = to_c<T>(to_d(ldf<float2>(src, f)));   // widened
    else r.p = ldf<T>(src, f);
    return r;
  };
  auto state = [&](const SvRaw<T>& r, double2& d) -> T {
    if (st == ST_INIT || st == ST_SWITCH) return r.p;
    if (st == ST_FINAL) return to_c<T>(cscale(to_d(r.p), ssc));
    double2 p;
    sv_psi_dirc<T>(D, have, r, p, d);
    return to_c<T>(csub(p, cscale(d, D.t)));
  };
  constexpr int CH = C == 8 ? 2 : (E % 4 == 0 ? 4 : 3);   // elements loaded together
  const double dx = I.dx, kf = I.kfac, Om = I.Omega;
  const SvTrap trap{I.s, I.tc};
  double2* const out_c = I.out_c;
  double2* const A = sv_field(I, ctl->f[F_A]);
  T v[E];
  double sum[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, fixed = 0.0;
  if (slot == 0) {
    const Tile<N, C, V, true> tl;
    const int t = tl.t, line = tl_ * C + tl.c;
    const bool valid = tl.c < C;
    const int i = ndim == 2 ? line : line / N, j = line - i * N;
    const double x = (double)(i - N / 2) * dx, y3 = (double)(j - N / 2) * dx;
    if (ndim == 2) fixed = x;
    double2* Wf = sv_field(I, ctl->f[F_W]);
    double2* Df = st == ST_TRIAL ? sv_field(I, ctl->f[F_DIRC]) : nullptr;
    const bool store_d = st == ST_TRIAL && !have;
#pragma unroll
    for (int q0 = 0; q0 < E; q0 += CH) {
      SvRaw<T> raw[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u)
        if (valid) raw[u] = load((size_t)line * N + t + TH * (q0 + u));
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const int q = q0 + u, r = t + TH * q;
        const size_t f = (size_t)line * N + r;
        v[q] = cmake<T>(0, 0);
        if (!valid) continue;
        double2 d;
        v[q] = state(raw[u], d);
        stf<T>(Wf, f, v[q]);
        if (store_d) stf<T>(Df, f, to_c<T>(d));
        if (st == ST_FINAL) out_c[f] = to_d(v[q]);
        const double p = cabs2(to_d(v[q])), c = (double)(r - N / 2) * dx;
        const double r2 = ndim == 2 ? x * x + c * c : x * x + y3 * y3 + c * c;
        sum[0] += p;
        sum[1] += sv_trap(trap, r2) * p;
        sum[2] += p * p;
        sum[3] += p * p * p;
        sum[6] = fmax(sum[6], p);
      }
    }
    const LineFft<N, V, 1, Tile<N, C, V, true>::WARP, T> fft{tl.template line<T>(sm), sv_tab<T>(I, V), t};
    fft.template forward<false>(v);
    const double inv = 1.0 / (double)N, wx = ndim == 2 ? -Om * x : 0.0;
    double sl = 0.0;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int r = t + TH * q, mm = (r < (N + 1) / 2) ? r : r - N;
      const double kk = kTwoPi * ((double)mm * kf), a2 = cabs2(to_d(v[q]));
      sum[4] += kk * kk * a2;
      sl += kk * a2;
      v[q] = cscale(v[q], (typename CT<T>::R)((0.5 * kk * kk + wx * kk) * inv));
    }
    sum[5] = fixed * sl;
    fft.template inverse<false>(v);
    if (valid) {
#pragma unroll
      for (int q = 0; q < E; ++q) stf<T>(A, (size_t)line * N + t + TH * q, v[q]);
    }
    sv_partials<W, 7>(sum, I.part, nt, tl_, 6);
  } else {
    const Tile<N, C, V, false> tl;
    const int t = tl.t;
    const bool valid = tl.c < C;
    int base, str, i, j, k;
    if (slot == 1) sv_line<N, C, 0>(ndim, tl_, tl.c, base, str, i, j, k);
    else sv_line<N, C, 1>(ndim, tl_, tl.c, base, str, i, j, k);
    fixed = (double)((slot == 1 ? j : i) - N / 2) * dx;
#pragma unroll
    for (int q0 = 0; q0 < E; q0 += CH) {
      SvRaw<T> raw[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u)
        if (valid) raw[u] = load((size_t)base + (size_t)(t + TH * (q0 + u)) * str);
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        double2 d;
        v[q0 + u] = valid ? state(raw[u], d) : cmake<T>(0, 0);
      }
    }
    const LineFft<N, V, Tile<N, C, V, false>::CP, false, T> fft{tl.template line<T>(sm), sv_tab<T>(I, V), t};
    fft.template forward<false>(v);
    double s2[2] = {0.0, 0.0};
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int r = t + TH * q, mm = (r < (N + 1) / 2) ? r : r - N;
      const double kk = kTwoPi * ((double)mm * kf), a2 = cabs2(to_d(v[q]));
      s2[0] += kk * kk * a2;
      s2[1] += kk * a2;
    }
    s2[1] *= fixed;
    sv_partials<W, 2>(s2, I.part + (size_t)(7 + 2 * (slot - 1)) * nt, nt, tl_);
  }
  };
  if (ctl->fp32 && (st == ST_TRIAL || st == ST_INIT)) body(float2{}); else body(double2{});
  SV_ARRIVE
  const int ndim = I.ndim, nt = SL.tiles / ndim;
  sv_control<W, 11>(I, ctl, gctl, 7 + 2 * (ndim - 1), nt, 6, [&](const double* tot) {
    if (threadIdx.x == 0) sv_ctl_trial(I, *ctl, tot);
  });
  }
}

// ------------------------------------------------------- 3D: A += T_y w
template <int N, int C, int V>
__global__ void __launch_bounds__(s_threads(N, C, V), sv_blocks(N, C, V))
    k_sv_hy(const __grid_constant__ SvLaunch SL) {
  using TL = Tile<N, C, V, false>;
  constexpr int TH = TL::T, E = TL::E;
  extern __shared__ double2 sm[];
  SV_FOR_ITEMS(tabN[V], lf_tab_len(N, V)) {
  SV_ITEM
  if (st != ST_H) continue;
  auto body = [&](auto tag_) {
  using T = decltype(tag_);
  const TL tl;
  const int t = tl.t;
  const bool valid = tl.c < C;
  int base, str, i, j, k;
  sv_line<N, C, 1>(3, tile, tl.c, base, str, i, j, k);
  const double2* w = sv_field(I, ctl->hf);
  T v[E];
#pragma unroll
  for (int q = 0; q < E; ++q) v[q] = valid ? ldf<T>(w, (size_t)base + (size_t)(t + TH * q) * str) : cmake<T>(0, 0);
  const LineFft<N, V, TL::CP, false, T> fft{tl.template line<T>(sm), sv_tab<T>(I, V), t};
  fft.template forward<false>(v);
  const double inv = 1.0 / (double)N, wx = -I.Omega * ((double)(i - N / 2) * I.dx), kf = I.kfac;
#pragma unroll
  for (int q = 0; q < E; ++q) {
    const int r = t + TH * q, mm = (r < (N + 1) / 2) ? r : r - N;
    const double kk = kTwoPi * ((double)mm * kf);
    v[q] = cscale(v[q], (typename CT<T>::R)((0.5 * kk * kk + wx * kk) * inv));
  }
  fft.template inverse<false>(v);
  double2* A = sv_field(I, ctl->f[F_A]);
  if (valid) {
    constexpr int CH = E % 4 == 0 ? 4 : 3;
#pragma unroll
    for (int q0 = 0; q0 < E; q0 += CH) {
      T a[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u) a[u] = ldf<T>(A, (size_t)base + (size_t)(t + TH * (q0 + u)) * str);
#pragma unroll
      for (int u = 0; u < CH; ++u)
        stf<T>(A, (size_t)base + (size_t)(t + TH * (q0 + u)) * str, cadd(a[u], v[q0 + u]));
    }
  }
  };
  if (ctl->fp32) body(float2{}); else body(double2{});
  }
}

// r-th smallest of the cnt <= kSvCap keys at src, by counting (all threads of the CTA)
BGP_D double sv_rank(const unsigned long long* src, int cnt, unsigned long long r, unsigned long long* sk) {
  __shared__ unsigned long long found;
  if (threadIdx.x == 0) found = 0ull;
  for (int q = threadIdx.x; q < cnt; q += blockDim.x) sk[q] = __ldcg(src + q);
  __syncthreads();
  for (int q = threadIdx.x; q < cnt; q += blockDim.x) {
    const unsigned long long x = sk[q];
    unsigned long long lt = 0, le = 0;
    for (int p = 0; p < cnt; ++p) { lt += sk[p] < x; le += sk[p] <= x; }
    if (lt <= r && r < le) found = x;
  }
  __syncthreads();
  return dkey_inv(found);
}

// The next median step of an instance whose keys are written (last CTA): the rank lies
// in the window around the last median, or a radix search over the keys begins.
BGP_D void sv_median(const SvInst& I, SvCtl& S, SvSync* sy, unsigned long long* sk) {
  const unsigned m = (unsigned)S.nkeys, wc = __ldcg(&sy->wcount);
  const unsigned long long r = m ? (unsigned long long)((m - 1u) / 2u) : 0ull, below = (unsigned long long)S.below;
  const bool hit = m != 0 && S.win_on && wc <= (unsigned)kSvCap && r >= below && r < below + wc;
  double med = I.sp.shift_min;
  if (hit) med = sv_rank(I.wcand, (int)wc, r - below, sk);
  __syncthreads();
  if (threadIdx.x == 0) {
    sy->wcount = 0u;
    if (m == 0 || hit) {
      if (hit && wc > (unsigned)kSvWin) S.med_eps = fmax(S.med_eps * 0.7, 1e-12);
      else if (hit && wc < (unsigned)kSvWin / 8) S.med_eps = fmin(S.med_eps * 2.0, 0.25);
      sv_sigma(I, S, med);
    } else {
      // widen the window when the median moved out of it, narrow it when it overflowed
      if (S.win_on) S.med_eps = (wc > (unsigned)kSvCap) ? fmax(S.med_eps * 0.25, 1e-9) : fmin(S.med_eps * 4.0, 0.25);
      S.rank = r; S.prefix = 0ull; S.level = 0; S.gather = 0;
      S.st = ST_MED;
    }
  }
}

// One step of the radix search (an instance in ST_MED): level L counts digit L of the
// keys that match the prefix so far; once the rank's bucket holds at most kSvGather
// keys they are gathered and ranked.
template <int W>
BGP_D void sv_median_step(const SvInst& I, SvCtl* ctl, SvCtl* gctl, SvSync* sy, int tile, int tiles, unsigned char* smem) {
  unsigned* sh = reinterpret_cast<unsigned*>(smem);
  const int level = ctl->level, gather = ctl->gather;
  const int hi = 64 - kSvDigit * level;                  // bits above hi are fixed by the prefix
  const unsigned long long prefix = ctl->prefix;
  const long long n = I.n, lo = n * tile / tiles, end = n * (tile + 1) / tiles;
  const int shift = hi - kSvDigit > 0 ? hi - kSvDigit : 0;
  if (!gather) {
    for (int q = threadIdx.x; q < kSvBins; q += blockDim.x) sh[q] = 0u;
    __syncthreads();
  }
  for (long long f = lo + threadIdx.x; f < end; f += blockDim.x) {
    const unsigned long long key = __ldcg(I.keys + f);
    if (key == 0ull || (level > 0 && (key >> hi) != (prefix >> hi))) continue;
    if (gather) {
      const unsigned idx = atomicAdd(&sy->wcount, 1u);
      if (idx < (unsigned)kSvCap) I.wcand[idx] = key;
    } else {
      atomicAdd(&sh[(key >> shift) & (kSvBins - 1)], 1u);
    }
  }
  if (!gather) {
    __syncthreads();
    for (int q = threadIdx.x; q < kSvBins; q += blockDim.x) if (sh[q]) atomicAdd(&I.hist[q], sh[q]);
  }
  if (!sv_last(sy, 1u, tiles)) return;
  if (gather) {
    const double med = sv_rank(I.wcand, (int)__ldcg(&sy->wcount), ctl->rank, reinterpret_cast<unsigned long long*>(smem));
    if (threadIdx.x == 0) { sy->wcount = 0u; sv_sigma(I, *ctl, med); }
    __syncthreads();
    sv_publish(I, ctl, gctl);
    return;
  }
  for (int q = threadIdx.x; q < kSvBins; q += blockDim.x) {
    sh[q] = __ldcg(&I.hist[q]);
    I.hist[q] = 0u;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    // warp 0 finds the rank's bin: lane l holds the total of its 64 bins
    constexpr int per = kSvBins / 32;
    const int lane = threadIdx.x;
    unsigned long long s = 0;
    for (int q = 0; q < per; ++q) s += sh[lane * per + q];
    unsigned long long inc = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    const unsigned long long r = ctl->rank;
    __syncwarp();
    if (r >= inc - s && r < inc) {
      unsigned long long run = inc - s;
      for (int q = 0; q < per; ++q) {
        const unsigned c = sh[lane * per + q];
        if (r < run + c) {
          SvCtl& S = *ctl;
          S.prefix = prefix | ((unsigned long long)(lane * per + q) << shift);
          S.rank = r - run;
          S.level = level + 1;
          if (shift == 0) sv_sigma(I, S, dkey_inv(S.prefix));   // every bit is fixed
          else if (c <= (unsigned)kSvGather) S.gather = 1;
          break;
        }
        run += c;
      }
    }
  }
  __syncthreads();
  sv_publish(I, ctl, gctl);
}

// -------------------------------------------------- gradient and x-transform
template <int N, int C, int V>
__global__ void __launch_bounds__(s_threads(N, C, V), sv_blocks(N, C, V))
    k_sv_hx(const __grid_constant__ SvLaunch SL) {
  using TL = Tile<N, C, V, false>;
  constexpr int TH = TL::T, E = TL::E, W = s_threads(N, C, V) / 32;
  extern __shared__ double2 sm[];
  SV_FOR_ITEMS(tabN[V], lf_tab_len(N, V)) {
  SV_ITEM
  if (st == ST_MED) {
    sv_median_step<W>(I, ctl, gctl, sy, tile, SL.tiles, reinterpret_cast<unsigned char*>(sm));
    __syncthreads();
    continue;
  }
  if (st != ST_H) continue;
  auto body = [&](auto tag_) {
  using T = decltype(tag_);
  const TL tl;
  const int t = tl.t, ndim = I.ndim;
  const bool valid = tl.c < C;
  int base, str, i, j, k;
  sv_line<N, C, 0>(ndim, tile, tl.c, base, str, i, j, k);
  const double2* w = sv_field(I, ctl->hf);
  const double hc = ctl->hc;
  T v[E];
#pragma unroll
  for (int q = 0; q < E; ++q) v[q] = valid ? ldf<T>(w, (size_t)base + (size_t)(t + TH * q) * str) : cmake<T>(0, 0);
  const LineFft<N, V, TL::CP, false, T> fft{tl.template line<T>(sm), sv_tab<T>(I, V), t};
  fft.template forward<false>(v);
  const double dx = I.dx, y = (double)(j - N / 2) * dx;
  {
    const double inv = 1.0 / (double)N, wx = I.Omega * y, kf = I.kfac;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int r = t + TH * q, mm = (r < (N + 1) / 2) ? r : r - N;
      const double kk = kTwoPi * ((double)mm * kf);
      v[q] = cscale(v[q], (typename CT<T>::R)((0.5 * kk * kk + wx * kk) * inv));
    }
  }
  fft.template inverse<false>(v);
  double s[3] = {0.0, 0.0, 0.0};                  // |g|^2, keys, keys below the window
  __shared__ unsigned wn, wbase;
  unsigned long long* const wkeys = reinterpret_cast<unsigned long long*>(sm);
  {
    const double2* A = sv_field(I, ctl->f[F_A]);
    double2* G = sv_field(I, ctl->f[F_G]);
    const double mu = ctl->mu, thr = 0.05 * ctl->maxrho, phisc = ctl->phisc;
    const bool kern = I.kern != 0, poly = ctl->poly_phi != 0, keys = ctl->kind != KD_FINAL, win = ctl->win_on != 0;
    double* phi = I.phi2 + (size_t)ctl->phi_cur * I.n;
    const double* pa = I.phi2 + (size_t)(1 - ctl->phi_cur) * I.n;
    const double *pb = I.phi2 + (size_t)2 * I.n, *pc = I.phi2 + (size_t)3 * I.n;
    const double sa = ctl->phisc_old, ts = ctl->t;
    const unsigned long long lo = ctl->win_lo, hi = ctl->win_hi;
    const double z = ndim == 3 ? (double)(k - N / 2) * dx : 0.0, b2 = I.beta2, b3 = I.beta3;
    const SvTrap trap{I.s, I.tc};
    unsigned long long* const keyf = I.keys;
    // the tile's window keys, collected in shared memory (the exchange buffer; a global
    // counter's round trip per key would stall its warp)
    if (threadIdx.x == 0) wn = 0u;
    __syncthreads();
    constexpr int CH = E % 4 == 0 ? 4 : 3;
#pragma unroll
    for (int q0 = 0; q0 < E; q0 += CH) {
      T va[CH], vp[CH];
      double ph[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const size_t f = (size_t)base + (size_t)(t + TH * (q0 + u)) * str;
        va[u] = valid ? ldf<T>(A, f) : cmake<T>(0, 0);
        vp[u] = valid ? ldf<T>(w, f) : cmake<T>(0, 0);
        ph[u] = 0.0;
        if (kern && valid) {
          if (poly) ph[u] = (sa * __ldcg(pa + f) - 2.0 * ts * __ldcg(pb + f)) + ts * ts * __ldcg(pc + f);
          else ph[u] = __ldcg(phi + f);
        }
      }
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const int r = t + TH * (q0 + u);
        const size_t f = (size_t)base + (size_t)r * str;
        const double x = (double)(r - N / 2) * dx;
        double r2 = x * x + y * y;
        if (ndim == 3) r2 = r2 + z * z;
        const double2 p = cscale(to_d(vp[u]), hc);
        const double rho = cabs2(p), Vt = sv_trap(trap, r2), fl = phisc * ph[u];
        const double pot = Vt + b2 * rho + b3 * rho * rho + fl;
        const double2 h = cadd(cscale(cadd(to_d(va[u]), to_d(v[q0 + u])), hc), cscale(p, pot));
        const double2 g = csub(h, cscale(p, mu));
        v[q0 + u] = to_c<T>(g);
        if (!valid) continue;
        s[0] += cabs2(g);
        if (poly) phi[f] = ph[u];
        stf<T>(G, f, v[q0 + u]);
        if (keys) {
          unsigned long long key = 0ull;
          if (rho > thr) {
            double loc = Vt + 2.0 * b2 * rho + 3.0 * b3 * (rho * rho);
            if (kern) loc = loc + fl;
            key = dkey(loc);
            s[1] += 1.0;
            if (win) {
              if (key < lo) {
                s[2] += 1.0;
              } else if (key <= hi) {
                const unsigned idx = atomicAdd(&wn, 1u);
                if (idx < (unsigned)kSvCap) wkeys[idx] = key;
              }
            }
          }
          keyf[f] = key;
        }
      }
    }
  }
  __syncthreads();
  if (wn) {
    if (threadIdx.x == 0) wbase = atomicAdd(&sy->wcount, wn);
    __syncthreads();
    const unsigned n = wn < (unsigned)kSvCap ? wn : (unsigned)kSvCap;
    for (unsigned q = threadIdx.x; q < n; q += blockDim.x)
      if (wbase + q < (unsigned)kSvCap) I.wcand[wbase + q] = wkeys[q];
  }
  fft.template forward<false>(v);
  {
    double2* B = sv_field(I, ctl->f[F_H]);
    if (valid) {
#pragma unroll
      for (int q = 0; q < E; ++q) stf<T>(B, (size_t)base + (size_t)(t + TH * q) * str, v[q]);
    }
  }
  sv_partials<W, 3>(s, I.part, SL.tiles, tile);
  };
  if (ctl->fp32) body(float2{}); else body(double2{});
  SV_ARRIVE
  sv_control<W, 3>(I, ctl, gctl, 3, SL.tiles, -1, [&](const double* tot) {
    __shared__ int go;
    if (threadIdx.x == 0) {
      ctl->gg = tot[0]; ctl->nkeys = tot[1]; ctl->below = tot[2];
      go = sv_residual(I, *ctl);
    }
    __syncthreads();
    if (go) sv_median(I, *ctl, sy, reinterpret_cast<unsigned long long*>(sm));
    else if (threadIdx.x == 0) sy->wcount = 0u;
  });
  }
}

// ------------------------------------------------------ preconditioner passes
// MODE 0: y-lines of a volume, forward; 1: contiguous lines, forward, divide by
// k^2/2 + sigma, inverse; 2: y-lines of a volume, inverse. In place on B.
template <int N, int C, int V, int MODE>
__global__ void __launch_bounds__(s_threads(N, C, V), sv_blocks(N, C, V))
    k_sv_p(const __grid_constant__ SvLaunch SL) {
  constexpr bool CONTIG = MODE == 1;
  using TL = Tile<N, C, V, CONTIG>;
  constexpr int TH = TL::T, E = TL::E;
  extern __shared__ double2 sm[];
  SV_FOR_ITEMS(tabN[V], lf_tab_len(N, V)) {
  SV_ITEM
  if (st != ST_PRE) continue;
  auto body = [&](auto tag_) {
  using T = decltype(tag_);
  const TL tl;
  const int t = tl.t, ndim = I.ndim;
  const bool valid = tl.c < C;
  int base, str, i, j, k;
  if (CONTIG) {
    const int line = tile * C + tl.c;
    base = line * N; str = 1;
    i = ndim == 2 ? line : line / N;
    j = line - i * N;
  } else {
    sv_line<N, C, 1>(3, tile, tl.c, base, str, i, j, k);
  }
  double2* B = sv_field(I, ctl->f[F_H]);
  T v[E];
#pragma unroll
  for (int q = 0; q < E; ++q) v[q] = valid ? ldf<T>(B, (size_t)base + (size_t)(t + TH * q) * str) : cmake<T>(0, 0);
  const LineFft<N, V, CONTIG ? 1 : TL::CP, TL::WARP, T> fft{tl.template line<T>(sm), sv_tab<T>(I, V), t};
  if (MODE <= 1) fft.template forward<false>(v);
  if (MODE == 1) {
    const double kf = I.kfac, sigma = ctl->sigma;
    auto kof = [&](int m) { return kTwoPi * ((double)(m < (N + 1) / 2 ? m : m - N) * kf); };
    const double kx = kof(i), ky = ndim == 3 ? kof(j) : 0.0, kxy = kx * kx + ky * ky;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const double kr = kof(t + TH * q);
      v[q] = cscale(v[q], (typename CT<T>::R)(1.0 / (0.5 * (kxy + kr * kr) + sigma)));
    }
  }
  if (MODE >= 1) fft.template inverse<false>(v);
  if (valid) {
#pragma unroll
    for (int q = 0; q < E; ++q) stf<T>(B, (size_t)base + (size_t)(t + TH * q) * str, v[q]);
  }
  };
  if (ctl->fp32) body(float2{}); else body(double2{});
  }
}

// x-lines, inverse: z_raw, and the sums of the next direction
template <int N, int C, int V>
__global__ void __launch_bounds__(s_threads(N, C, V), sv_blocks(N, C, V))
    k_sv_px(const __grid_constant__ SvLaunch SL) {
  using TL = Tile<N, C, V, false>;
  constexpr int TH = TL::T, E = TL::E, W = s_threads(N, C, V) / 32;
  extern __shared__ double2 sm[];
  SV_FOR_ITEMS(tabN[V], lf_tab_len(N, V)) {
  SV_ITEM
  if (st != ST_PRE) continue;
  auto body = [&](auto tag_) {
  using T = decltype(tag_);
  const TL tl;
  const int t = tl.t;
  const bool valid = tl.c < C;
  int base, str, i, j, k;
  sv_line<N, C, 0>(I.ndim, tile, tl.c, base, str, i, j, k);
  const double2* B = sv_field(I, ctl->f[F_H]);
  T v[E];
#pragma unroll
  for (int q = 0; q < E; ++q) v[q] = valid ? ldf<T>(B, (size_t)base + (size_t)(t + TH * q) * str) : cmake<T>(0, 0);
  const LineFft<N, V, TL::CP, false, T> fft{tl.template line<T>(sm), sv_tab<T>(I, V), t};
  fft.template inverse<false>(v);
  double s[kDSums];
#pragma unroll
  for (int q = 0; q < kDSums; ++q) s[q] = 0.0;
  {
    const double2 *ps = sv_field(I, ctl->f[F_PSI]), *pq = sv_field(I, ctl->f[F_PSIP]);
    const double2 *G = sv_field(I, ctl->f[F_G]), *GP = sv_field(I, ctl->f[F_GP]);
    const bool has_d = ctl->f[F_DIR] >= 0;
    const double2* Df = sv_field(I, has_d ? ctl->f[F_DIR] : ctl->f[F_G]);
    double2* Z = sv_field(I, ctl->f[F_Z]);
    const double psc = ctl->sc[F_PSI], qsc = ctl->sc[F_PSIP], inv_n = I.inv_n;
    constexpr int CH = C == 8 ? 2 : (E % 4 == 0 ? 4 : 3);   // elements loaded together
    if (valid) {
#pragma unroll
      for (int q0 = 0; q0 < E; q0 += CH) {
        T rp[CH], rq[CH], rg[CH], rh[CH], rd[CH];
#pragma unroll
        for (int u = 0; u < CH; ++u) {
          const size_t f = (size_t)base + (size_t)(t + TH * (q0 + u)) * str;
          rp[u] = ldf<T>(ps, f); rq[u] = ldf<T>(pq, f); rg[u] = ldf<T>(G, f); rh[u] = ldf<T>(GP, f);
          rd[u] = has_d ? ldf<T>(Df, f) : cmake<T>(0, 0);
        }
#pragma unroll
        for (int u = 0; u < CH; ++u) {
          const size_t f = (size_t)base + (size_t)(t + TH * (q0 + u)) * str;
          const T zt = to_c<T>(cscale(to_d(v[q0 + u]), inv_n));
          stf<T>(Z, f, zt);
          const double2 z = to_d(zt), p = cscale(to_d(rp[u]), psc), qq = cscale(to_d(rq[u]), qsc);
          const double2 g = to_d(rg[u]), gp = to_d(rh[u]), d = to_d(rd[u]);
          const double2 yv = csub(g, gp), sv = csub(p, qq);
          const double2 pz = cconjmul(p, z), py = cconjmul(p, yv), gps = cconjmul(g, p), pd = cconjmul(p, d);
          s[D_PZX] += pz.x; s[D_PZY] += pz.y;
          s[D_ZY] += z.x * yv.x + z.y * yv.y;
          s[D_PYX] += py.x; s[D_PYY] += py.y;
          s[D_GY] += g.x * yv.x + g.y * yv.y;
          s[D_PDX] += pd.x; s[D_PDY] += pd.y;
          s[D_ZG] += g.x * z.x + g.y * z.y;
          s[D_GD] += g.x * d.x + g.y * d.y;
          s[D_GPX] += gps.x; s[D_GPY] += gps.y;
          s[D_SY] += sv.x * yv.x + sv.y * yv.y;
          s[D_SS] += cabs2(sv);
        }
      }
    }
  }
  sv_partials<W, kDSums>(s, I.part, SL.tiles, tile);
  };
  if (ctl->fp32) body(float2{}); else body(double2{});
  SV_ARRIVE
  sv_control<W, kDSums>(I, ctl, gctl, kDSums, SL.tiles, -1, [&](const double* tot) {
    if (threadIdx.x < kDSums) ctl->d[threadIdx.x] = tot[threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0) sv_direction(I, *ctl, false);
  });
  }
}

// ------------------------------------------------------ convolution passes
// The passes of bgp_stream.cuh's convolution on the density the state asks for: |w|^2
// of the trial (or accepted) state, or the linear and quadratic parts b = Re(conj(psi)
// dirc), c = |dirc|^2 of the trial density (3D), whose first pass stores dirc; the last
// pass also sums the potential against the density's parts.
template <int N, int C, int V, int INV>
__global__ void __launch_bounds__(s_threads(N, C, V), sv_blocks(N, C, V))
    k_sv_real(const __grid_constant__ SvLaunch SL) {
  using TL = Tile<N, C, V, true>;
  constexpr int E = TL::E, TH = TL::T, Mp = conv_pitch(N), W = s_threads(N, C, V) / 32;
  extern __shared__ double2 sm[];
  SV_FOR_ITEMS(tabN[V], lf_tab_len(N, V)) {
  SV_ITEM
  if (st != ST_CONV && st != ST_POLYB && st != ST_POLYC) continue;
  auto body = [&](auto tag_) {
  using T = decltype(tag_);
  const TL tl;
  const int t = tl.t, line = tile * C + tl.c;
  const bool valid = tl.c < C;
  double2* b = tl.line(sm);
  const typename TL::Fft fft{b, I.tabN[V], t};
  const double2* __restrict__ tw = I.twM;
  const double2* w = sv_field(I, ctl->refresh ? ctl->hf : (ctl->f[F_W] >= 0 ? ctl->f[F_W] : 0));
  SvDir D{};
  if (st != ST_CONV) D = sv_dir(I, *ctl);
  double2 v[E];
  if (INV == 0) {
    const bool store_d = st == ST_POLYB;
    double2* Df = sv_field(I, ctl->f[F_DIRC] >= 0 ? ctl->f[F_DIRC] : 0);
    constexpr int CH = (C < 8 && (E / 2) % 4 == 0) ? 4 : ((E / 2) % 3 == 0 ? 3 : 2);
#pragma unroll
    for (int q0 = 0; q0 < E / 2; q0 += CH) {
      SvRaw<T> raw[CH][2];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const size_t f = (size_t)line * N + 2 * (t + TH * (q0 + u));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (!valid) continue;
          if (st == ST_CONV) raw[u][h].p = ldf<T>(w, f + h);
          else if (st == ST_POLYC) raw[u][h].p = ldf<T>(D.dirc, f + h);
          else raw[u][h] = sv_load<T>(D, false, f + h);
        }
      }
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const size_t f = (size_t)line * N + 2 * (t + TH * (q0 + u));
        double rho[2] = {0.0, 0.0};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (!valid) continue;
          if (!store_d) { rho[h] = cabs2(to_d(raw[u][h].p)); continue; }
          double2 p, d;
          sv_psi_dirc<T>(D, false, raw[u][h], p, d);
          stf<T>(Df, f + h, to_c<T>(d));
          rho[h] = p.x * d.x + p.y * d.y;
        }
        v[q0 + u] = cmk(rho[0], rho[1]);
      }
    }
    fft.template forward<true>(v);
    TL::Fft::sync();
#pragma unroll
    for (int q = 0; q < E; ++q) b[t + TH * q] = v[q];
    TL::Fft::sync();
    double2* out = I.cb1 + (size_t)line * Mp;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const int k = t + TH * q;
      const double2 z = v[q], p = b[k ? N - k : 0];
      const double2 e = cmk(0.5 * (z.x + p.x), 0.5 * (z.y - p.y));
      const double2 o = cmk(0.5 * (z.y + p.y), 0.5 * (p.x - z.x));
      if (valid) out[k] = cadd(e, cmul(o, __ldg(tw + k)));
    }
    if (t == 0 && valid) out[N] = cmk(v[0].x - v[0].y, 0.0);
    TL::Fft::sync();                              // the buffer is free for the next item
    return;
  }
  const double2* in = I.cb1 + (size_t)line * Mp;
#pragma unroll
  for (int q = 0; q < E; ++q) v[q] = valid ? in[t + TH * q] : cmk(0.0, 0.0);
#pragma unroll
  for (int q = 0; q < E; ++q) b[t + TH * q] = v[q];
  if (t == 0) b[N] = valid ? in[N] : cmk(0.0, 0.0);
  TL::Fft::sync();
#pragma unroll
  for (int q = 0; q < E; ++q) {
    const int k = t + TH * q;
    const double2 x = v[q], p = b[N - k];
    const double2 e = cmk(x.x + p.x, x.y - p.y);
    const double2 d = cmk(x.x - p.x, x.y + p.y);
    const double2 o = cconjmul(__ldg(tw + k), d);
    v[q] = cmk(e.x - o.y, e.y + o.x);
  }
  fft.template inverse<true>(v);
  // trial and final states go to the buffer beside the current potential's; a refreshed
  // one to the current (just accepted) state's
  const int buf = st == ST_POLYB ? 2 : (st == ST_POLYC ? 3 : (ctl->refresh ? ctl->phi_cur : 1 - ctl->phi_cur));
  double* out = I.phi2 + (size_t)buf * I.n;
  const double* pa = I.phi2 + (size_t)ctl->phi_cur * I.n;
  const double sc = I.conv_scale, sa = ctl->phisc;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  if (valid) {
    constexpr int CH = (E / 2) % 2 == 0 ? 2 : 3;
#pragma unroll
    for (int q0 = 0; q0 < E / 2; q0 += CH) {
      T rp[CH][2], rd[CH][2];
      double2 ra[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const size_t f = (size_t)line * N + 2 * (t + TH * (q0 + u));
        ra[u] = cmk(0.0, 0.0);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (st == ST_CONV) { rp[u][h] = ldf<T>(w, f + h); rd[u][h] = rp[u][h]; }
          else { rp[u][h] = ldf<T>(D.psi, f + h); rd[u][h] = ldf<T>(D.dirc, f + h); }
        }
        if (st == ST_POLYB) ra[u] = __ldcg(reinterpret_cast<const double2*>(pa + f));
      }
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const size_t f = (size_t)line * N + 2 * (t + TH * (q0 + u));
        const double2 x = cscale(v[q0 + u], sc);
        *reinterpret_cast<double2*>(out + f) = x;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double ph = h ? x.y : x.x, pha = h ? ra[u].y : ra[u].x;
          if (st == ST_CONV) { s[0] += ph * cabs2(to_d(rp[u][h])); continue; }
          const double2 p = cscale(to_d(rp[u][h]), D.psc), d = to_d(rd[u][h]);
          const double da = cabs2(p), db = p.x * d.x + p.y * d.y, dc = cabs2(d);
          s[0] += ph * da;
          s[1] += ph * db;
          s[2] += ph * dc;
          s[3] += sa * pha * da;
        }
      }
    }
  }
  sv_partials<W, 4>(s, I.part, SL.tiles, tile);
  };
  if (ctl->fp32) body(float2{}); else body(double2{});
  if (INV == 0) continue;
  SV_ARRIVE
  sv_control<W, 4>(I, ctl, gctl, 4, SL.tiles, -1, [&](const double* tot) {
    if (threadIdx.x == 0) sv_ctl_conv(I, *ctl, tot);
  });
  }
}

template <int M, int C, int V, int MODE>
__global__ void __launch_bounds__(s_threads(M, C, V), s_min_blocks(M, C, V))
    k_sv_pad(const __grid_constant__ SvLaunch SL) {
  extern __shared__ double2 sm[];
  SV_FOR_ITEMS(tabM[V], lf_tab_len(M, V)) {
  SV_ITEM
  if (st != ST_CONV && st != ST_POLYB && st != ST_POLYC) continue;
  pad_tile<M, C, V, MODE>(tile, I.ndim, I.cb1, I.cb2, I.Kq, I.tabM[V], sm);
  }
}

#endif  // __CUDACC__

BGP_NS_END  // namespace bgp
