// gbf_f64_pair.cuh — per-cell device code of the FP64 step in increment form
// with FP32-pair arithmetic; shared by the single-domain kernels (gbf_f64.cu)
// and the batched ones (gbf_ensemble.cu).
//
// State, inputs and results are the plain FP64 step's: P and S in FP64. Only
// what a step adds to them is formed from FP32 pairs (gbf_pair.cuh):
//   * the Newton's equations at the start of a step are
//       F1(P, S) - A1 = dt/phi div1,   F2(P, S) - A2 = dt/phi div2 + rho02 beta2 P_k S - src
//     (A: the targets of cpu.cpp:260-291, whose masses are F at P_k = 0), so
//     no mass is ever formed and subtracted again: the increments (dP, dS)
//     solve  r + [F(x + d) - F(x)] = 0, the bracket written in increments;
//   * pressures enter as differences from the row's hydrostatic P_hs(j), so
//     gravity and the hydrostatic gradient cancel before any rounding;
//   * 1 - S_e = S / (1 - S_wr) and ln S_e = ln(1 - .) are taken without
//     forming S_e, so kr2 keeps its relative accuracy as S -> 0.
// An increment is then accurate to about 2^-45 of itself, and P + dP, S + dS
// are rounded once in FP64. The arithmetic that forms masses of 1000 kg/m^3 in
// FP64 and recovers P through rho0 beta from their rounding (1e-13) loses more:
// the error against 64-bit increments is 1e-12 of P there and 1e-16 here.
#pragma once

#include "gbf_domain.h"
#include "gbf_pair.cuh"

// A row's constants: P_hs(j), P_hs(j) - P_atm as a pair, and what rounding
// leaves of rho01 g h2 minus the rows' differences of P_hs (above, below).
struct GbfPairRow {
  double phs;
  GbfPf pp;
  float eu, ed;
};
__device__ __forceinline__ double pair_row_phs(const gbf_model& m, int j) {  // gbf_p_hydrostatic, each operation rounded
  return __dadd_rn(m.P_atm, __dmul_rn(__dmul_rn(__dmul_rn((double)j, m.ro01), m.g), m.h2));
}
__device__ __forceinline__ GbfPairRow gbf_pair_row(const gbf_model& m, int j) {
  GbfPairRow r;
  r.phs = pair_row_phs(m, j);
  const double pp = __dsub_rn(r.phs, m.P_atm), H = __dmul_rn(__dmul_rn(m.ro01, m.g), m.h2);
  r.pp.h = __double2float_rn(pp);
  r.pp.l = __double2float_rn(__dsub_rn(pp, (double)r.pp.h));
  r.eu = __double2float_rn(__dsub_rn(H, __dsub_rn(r.phs, pair_row_phs(m, j - 1))));
  r.ed = __double2float_rn(__dsub_rn(H, __dsub_rn(pair_row_phs(m, j + 1), r.phs)));
  return r;
}

// Model constants as pairs. Mobilities x density are held times 2^e (`scale`)
// so that pairs of physical size (1e-4 and smaller) keep their low parts away
// from FP32's underflow; the weights dt / h^2 carry 2^-e.
struct GbfPairConsts {
  int nx, ny, nz, noflow;
  unsigned pl, n, nint;
  GbfFastDiv dnx, dny, dix, diy;
  int ri0, rk0, rn;  // rate source cells (rn = 0: none)
  int max_iter;
  float Patm;
  GbfPf k1, k2, rk1;     // rho01 beta1, rho02 beta2, 1 / (rho01 beta1)
  GbfPf ro1, ro2;        // rho01, rho02
  GbfPf g1, g2, ghd;     // g h2 rho01 beta1, g h2 rho02 beta2, g h2 (rho02 - rho01)
  GbfPf wx, wy, wz;      // dt / h1^2, dt kv / h2^2, dt / h3^2 (over the scale)
  GbfPf c1, c2;          // 1 / mu (times the scale)
  GbfPf K[2], phip[2], rphi[2], inv[2], E3p[2], pd[2], ilam[2];
  double phi_d[2], inv_d[2], E1[2], E2[2], E3[2];  // 1 / (1 - S_wr); Brooks-Corey exponents over ln 2
  float E1f[2], E2f[2];
  float taylor[2][4];    // (1 / lambda + n) / (n + 1), n = 1..4
  double ro1_d, ro2_d, beta1_d, beta2_d, Patm_d, k1_d, k2_d;  // the densities' constants
  double dtsrc_d, rro2_d;  // dt x the rate source per volume, 1 / rho02
};
GbfPairConsts gbf_pair_consts(const gbf_model& m);
// The pair step solves the Newton's equations to round-off. The reference's 7
// iterations (and more) do too; a model that asks for fewer stops before, and
// keeps the plain FP64 passes (gbf_f64_cell.cuh).
inline bool gbf_pair_applies(const gbf_model& m) { return m.newton_iterations >= 7; }
// Fill rows[0, ny) for the model (stream-ordered on st).
int gbf_pair_fill_rows(const gbf_model& m, GbfPairRow* rows, cudaStream_t st);

// Arrays of a pair step beside GbfF64Step's P, S, Pn, Sn.
struct GbfPairWork {
  float2 *D, *L1, *L2, *Pk;  // P - P_hs(j), mobility x density of both phases, capillary pressure (where S is not 0)
  const GbfPairRow* rows;
  // drop-in (NULL: none): the caller's (P, S) that pass 1 reads and copies to
  // s.P, s.S; it also writes the density arrays s.ro1, s.ro2
  const double *P_from, *S_from;
};

__device__ __forceinline__ GbfPf pf_ld(const float2* p) {
  const float2 v = __ldg(p);
  return {v.x, v.y};
}
__device__ __forceinline__ void pf_st(float2* p, GbfPf a) { *p = make_float2(a.h, a.l); }

// Brooks-Corey functions of om = 1 - S_e = S / (1 - S_wr): kr1 = S_e^e1, w =
// 1 - S_e^e2 (kr2 = om^2 w) and P_k / P_d = S_e^(-1/lambda). Beyond the
// tables' range (S_e <= 2^-11, S far below 0, NaN) they come from CUDA's
// functions, with the FP64 passes' limits (S_e = 0: kr1 = 0, P_k infinite;
// S_e < 0: NaN).
__device__ __forceinline__ bool pair_om_ok(float om) { return om < 0.9995f && om > -0.25f; }
static __device__ __noinline__ double pair_pow_general(double om, double E) {
  return exp2(E * log(1.0 - om));
}
// P_k(S) (rare: the Newton's changes of S beyond its expansion's range).
static __device__ __noinline__ GbfPf pair_pk(const GbfPairConsts& C, int md, GbfPf S) {
  const double om = __dmul_rn(pf_to_double(S), C.inv_d[md]);
  const float omf = pf_from_double(om).h;
  if (!pair_om_ok(omf)) return pf_mul(C.pd[md], pf_from_double(pair_pow_general(om, C.E3[md])));
  return pf_mul(C.pd[md], pf_exp2(pf_mul(pf_from_double(gbf_ln1m(om, omf)), C.E3p[md])));
}

// Pass 1 at cell c (every cell): D, L1, L2, P_k (DROPIN: and the copy of the
// caller's state, the reference's density arrays). The Brooks-Corey functions
// keep FP64's accuracy (an error of kr would act in the same direction step
// after step, while the roundings of the pair products do not): 14 FP64
// instructions where there is DNAPL, one elsewhere.
template <bool DROPIN>
__device__ __forceinline__ void gbf_pair_props_cell(const GbfPairConsts& C, const gbf_cells& cells,
                                                    const GbfF64Step& s, const GbfPairWork& w, unsigned c) {
  const unsigned row = gbf_div(c, C.dnx), j = row - gbf_div(row, C.dny) * (unsigned)C.ny;
  const int md = cells.media ? __ldg(cells.media + c) : 0;
  double P, S;
  if (DROPIN) {
    P = w.P_from[c];
    S = w.S_from[c];
    const_cast<double*>(s.P)[c] = P;
    const_cast<double*>(s.S)[c] = S;
    s.ro1[c] = C.ro1_d * (1. + C.beta1_d * (P - C.Patm_d));
    s.ro2[c] = C.ro2_d * (1. + C.beta2_d * (P - C.Patm_d));
  } else {
    P = __ldg(s.P + c);
    S = __ldg(s.S + c);
  }
  const GbfPairRow R = w.rows[j];
  const GbfPf D = pf_from_double(__dsub_rn(P, R.phs));
  const GbfPf Pp = pf_add(R.pp, D);
  const float K = cells.K ? __ldg(cells.K + c) : 0.f;
  auto over_mu = [&](const GbfPf& rmu) { return cells.K ? pf_mulf(rmu, K) : pf_mul(rmu, C.K[md]); };  // K / mu
  GbfPf l1 = over_mu(C.c1), l2 = {0.f, 0.f};
  if (!gbf_is_zero(S)) {  // S = 0: kr1 = 1, kr2 = 0, and P_k = P_d is not stored
    const double om = __dmul_rn(S, C.inv_d[md]);
    const GbfPf omp = pf_from_double(om);
    GbfPf kr1, w2, pk = C.pd[md];
    if (pair_om_ok(omp.h)) {
      const double l = gbf_ln1m(om, omp.h);
      const GbfPf lp = pf_from_double(l);
      kr1 = pf_from_double(gbf_exp2(__dmul_rn(l, C.E1[md]), __fmul_rn(lp.h, C.E1f[md])));
      w2 = pf_from_double(gbf_one_minus_exp2(__dmul_rn(l, C.E2[md]), __fmul_rn(lp.h, C.E2f[md])));
      pk = pf_mul(pk, pf_exp2(pf_mul(lp, C.E3p[md])));
    } else {
      kr1 = pf_from_double(pair_pow_general(om, C.E1[md]));
      w2 = pf_from_double(1.0 - pair_pow_general(om, C.E2[md]));
      pk = pf_mul(pk, pf_from_double(pair_pow_general(om, C.E3[md])));
    }
    l1 = pf_mul(l1, kr1);
    l2 = pf_mul(pf_mul(over_mu(C.c2), pf_mul(pf_mul(omp, omp), w2)), pf_add(C.ro2, pf_mul_raw(C.k2, Pp)));
    pf_st(w.Pk + c, pk);
  }
  pf_st(w.D + c, D);
  pf_st(w.L1 + c, pf_mul(l1, pf_add(C.ro1, pf_mul_raw(C.k1, Pp))));
  pf_st(w.L2 + c, l2);
}

// a - b, normalised
__device__ __forceinline__ GbfPf pf_diff(GbfPf a, GbfPf b) {
  const GbfPf s = pf_two_sum(a.h, -b.h);
  return pf_fast(s.h, __fadd_rn(s.l, __fsub_rn(a.l, b.l)));
}
// Upwinded flux through a face with potential x (from the minus to the plus side).
__device__ __forceinline__ GbfPf pair_face(GbfPf x, GbfPf Lm, GbfPf Lp) {
  const bool f = x.h >= 0.f;
  return pf_mul_raw(x, GbfPf{f ? Lm.h : Lp.h, f ? Lm.l : Lp.l});
}
// w (out - in)
__device__ __forceinline__ GbfPf pair_net(GbfPf out, GbfPf in, GbfPf w) {
  const GbfPf s = pf_two_sum(out.h, -in.h);
  return pf_mul_raw(GbfPf{s.h, __fadd_rn(s.l, __fsub_rn(out.l, in.l))}, w);
}
__device__ __forceinline__ GbfPf pair_sum3(GbfPf a, GbfPf b, GbfPf c) {
  const GbfPf s = pf_two_sum(a.h, b.h), t = pf_two_sum(s.h, c.h);
  return pf_fast(t.h, __fadd_rn(__fadd_rn(t.l, s.l), __fadd_rn(__fadd_rn(a.l, b.l), c.l)));
}

// A thread's sums of phi A (both phases), A1 = rho1 (1 - S) - r1, A2 = rho02
// (1 + beta2 (P - P_atm)) S - r2: in FP64, but for phi r1, a 1e-6 part of the
// water mass, summed as a pair.
struct GbfPairMass {
  double m1 = 0., m2 = 0.;
  GbfPf r1 = {0.f, 0.f};
};

// The rate source of a cell: dt src / phi in FP64 as a pair and its remainder
// (the same every step, so its rounding would add up), and S + ds + remainder.
static __device__ __noinline__ GbfPf pair_source(double dtsrc, double phi, double& rest) {
  const double sd = dtsrc / phi;
  const GbfPf sp = pf_from_double(sd);
  rest = sd - pf_to_double(sp);
  return sp;
}
static __device__ __noinline__ double pair_add_rest(double S, double ds, double rest, double rro2) {
  return S + __fma_rn(rest, rro2, ds);
}
// roS1, roS2, roS1_old, roS2_old of the mass update (GBF_OUT_MASS_ARRAYS).
static __device__ __noinline__ void pair_mass_arrays(const GbfPairConsts& C, const GbfF64Step& s, unsigned c, double P,
                                                     double S, GbfPf r1, GbfPf r2) {
  const double pa = P - C.Patm_d, q1 = __fma_rn(C.k1_d, pa, C.ro1_d) * (1. - S), q2 = __fma_rn(C.k2_d, pa, C.ro2_d) * S;
  s.roS1_old[c] = q1;
  s.roS2_old[c] = q2;
  s.roS1[c] = q1 - pf_to_double(r1);
  s.roS2[c] = q2 - pf_to_double(r2);
}

// The Newton's equations of a cell with DNAPL, d = (dp, ds):
//   r1 + k1 dp (1 - S - ds) - rho1 ds = 0,
//   r2 + k2 (dp + P_k(S + ds) - P_k(S)) (S + ds) + rho2 ds = 0, rho2 at P + P_k(S),
// r2 with the k2 P_k S that the targets leave out (cpu.cpp:63 vs :306).
// The Jacobian and its inverse are FP32, the residual pairs: a step leaves
// 2^-21 of itself, so two or three reach round-off.
__device__ __forceinline__ void pair_newton(const GbfPairConsts& C, int md, GbfPf Pp, GbfPf S, GbfPf Pk, GbfPf r1,
                                            GbfPf r2, GbfPf& dp, GbfPf& ds) {
  const GbfPf rho1 = pf_add(C.ro1, pf_mul_raw(C.k1, Pp));
  const GbfPf rho2 = pf_add(C.ro2, pf_mul_raw(C.k2, pf_add(Pp, Pk)));
  const GbfPf omS = pf_sub(GbfPf{1.f, 0.f}, S);
  const GbfPf Se = pf_sub(GbfPf{1.f, 0.f}, pf_mul(S, C.inv[md]));
  r2 = pf_add(r2, pf_mul(pf_mul(C.k2, Pk), S));
  const GbfPf slope = pf_div(pf_mul(Pk, C.ilam[md]), Se);  // dP_k/dS
  const float rSe = pf_rcp(Se.h);
  float J11 = __fmul_rn(C.k1.h, omS.h), mJ12 = rho1.h, J21 = __fmul_rn(C.k2.h, S.h);
  const float share = __fmul_rn(J21, slope.h);
  float J22 = __fadd_rn(rho2.h, share);
  float inv = pf_rcp(__fmaf_rn(J11, J22, __fmul_rn(mJ12, J21)));
  const float ratio = fabsf(__fmul_rn(share, pf_rcp(rho2.h)));  // the capillary term's part of J22
  GbfPf G1 = r1, G2 = r2;
  for (int it = 0;; it++) {
    const float ep = -__fmul_rn(inv, __fmaf_rn(J22, G1.h, __fmul_rn(mJ12, G2.h)));
    const float es = -__fmul_rn(inv, __fmaf_rn(J11, G2.h, -__fmul_rn(J21, G1.h)));
    dp = it ? pf_addf(dp, ep) : GbfPf{ep, 0.f};
    ds = it ? pf_addf(ds, es) : GbfPf{es, 0.f};
    const float x = __fmul_rn(__fmul_rn(ds.h, C.inv[md].h), rSe);  // relative change of S_e
    if (it > 0) {
      // what the step leaves: the Jacobian's error (2^-21) or its change over the increments,
      // of the step; small enough once below 2^-54 of S and of P
      const float q = fmaxf(4.77e-7f, it > 1 ? 0.f : __fmul_rn(8.f, fabsf(x)));
      const float lim_s = __fmul_rn(5.55e-17f, fabsf(__fadd_rn(S.h, ds.h)));
      const float lim_p = __fmul_rn(5.55e-17f, __fadd_rn(fabsf(Pp.h), C.Patm));
      const bool done =
          (__fmul_rn(q, fabsf(es)) <= lim_s || fabsf(es) <= __fmul_rn(2.8e-14f, fabsf(ds.h))) &&
          (__fmul_rn(q, fabsf(ep)) <= lim_p || fabsf(ep) <= __fmul_rn(2.8e-14f, fabsf(dp.h)));
      if (done || it + 1 >= C.max_iter || !(fabsf(ep) < 3e38f && fabsf(es) < 3e38f)) break;
    }
    // residual at the new point
    const GbfPf omn = pf_sub(omS, ds), Sn = pf_add(S, ds);
    GbfPf dPk;
    if (fabsf(x) < 0.0156f && __fmul_rn(ratio, fabsf(x)) < 5.96e-8f) {
      // P_k((1 - x)^-a - 1) = slope ds (1 + (a + 1)/2 x (1 + (a + 2)/3 x (1 + ...))), a = 1 / lambda
      const float* a = C.taylor[md];
      const float t = __fmul_rn(__fmul_rn(x, a[0]),
                                __fmaf_rn(__fmul_rn(x, a[1]), __fmaf_rn(__fmul_rn(x, a[2]), __fmaf_rn(x, a[3], 1.f), 1.f), 1.f));
      const GbfPf lin = pf_mul(slope, ds);
      dPk = pf_fast(lin.h, __fmaf_rn(lin.h, t, lin.l));
    } else {
      dPk = pf_sub(pair_pk(C, md, Sn), Pk);
    }
    const GbfPf dpk = pf_add(dp, dPk);
    G1 = pf_sub(pf_add(r1, pf_mul(pf_mul(C.k1, dp), omn)), pf_mul(rho1, ds));
    G2 = pf_add(pf_add(r2, pf_mul(pf_mul(C.k2, dpk), Sn)), pf_mul(rho2, ds));
    if (it > 0 || fabsf(x) > 1e-4f) {  // the Jacobian at the new point
      J11 = __fmul_rn(C.k1.h, omn.h);
      mJ12 = __fmaf_rn(C.k1.h, dp.h, rho1.h);
      J21 = __fmul_rn(C.k2.h, Sn.h);
      const float sl = __fmul_rn(__fmul_rn(__fadd_rn(Pk.h, dPk.h), C.ilam[md].h),
                                 pf_rcp(__fmaf_rn(-ds.h, C.inv[md].h, Se.h)));
      J22 = __fmaf_rn(C.k2.h, __fmaf_rn(sl, Sn.h, dpk.h), rho2.h);
      inv = pf_rcp(__fmaf_rn(J11, J22, __fmul_rn(mJ12, J21)));
    }
  }
}

// Pass 2 at interior cell (i, j, k) = c: fluxes, Newton, next state (the
// water-only form where no DNAPL is in the cell or flows through its faces).
template <bool MASS>
__device__ __forceinline__ void gbf_pair_step_cell(const GbfPairConsts& C, const gbf_cells& cells,
                                                   const GbfF64Step& s, const GbfPairWork& w, int i, int j, int k,
                                                   unsigned c, GbfPairMass& acc, unsigned& bad) {
  const unsigned nx = (unsigned)C.nx, pl = C.pl;
  const int md = cells.media ? __ldg(cells.media + c) : 0;
  const GbfPairRow R = w.rows[j];
  const GbfPf D = pf_ld(w.D + c);
  const GbfPf Pp = pf_add(R.pp, D);  // P - P_atm
  // face potentials times h; gravity g h2 (rho_a - rho01) with the centre cell's density
  const GbfPf xm = pf_diff(pf_ld(w.D + c - 1), D), xp = pf_diff(D, pf_ld(w.D + c + 1));
  const GbfPf zm = pf_diff(pf_ld(w.D + c - pl), D), zp = pf_diff(D, pf_ld(w.D + c + pl));
  const GbfPf yu = pf_addf(pf_diff(pf_ld(w.D + c - nx), D), R.eu), yd = pf_addf(pf_diff(D, pf_ld(w.D + c + nx)), R.ed);
  const bool noflow = C.noflow && j == C.ny - 2;
  const GbfPf zero = {0.f, 0.f};
  GbfPf rphi;
  float phif = 0.f;
  if (cells.phi) {
    phif = __ldg(cells.phi + c);
    const float q = pf_rcp(phif);
    rphi = pf_fast(q, __fmul_rn(__fmaf_rn(-phif, q, 1.f), q));
  } else {
    rphi = C.rphi[md];
  }
  GbfPf r1;
  {
    const GbfPf Lc = pf_ld(w.L1 + c), G = pf_mul(C.g1, Pp);
    const GbfPf y1 = pf_add(yu, G), y2 = noflow ? zero : pf_add(yd, G);
    const GbfPf f = pair_sum3(
        pair_net(pair_face(xp, Lc, pf_ld(w.L1 + c + 1)), pair_face(xm, pf_ld(w.L1 + c - 1), Lc), C.wx),
        pair_net(pair_face(y2, Lc, pf_ld(w.L1 + c + nx)), pair_face(y1, pf_ld(w.L1 + c - nx), Lc), C.wy),
        pair_net(pair_face(zp, Lc, pf_ld(w.L1 + c + pl)), pair_face(zm, pf_ld(w.L1 + c - pl), Lc), C.wz));
    r1 = pf_mul(f, rphi);
  }
  const double Sd = __ldg(s.S + c), Pd = __ldg(s.P + c);
  const bool src = C.rn > 0 && j == 1 && (unsigned)(i - C.ri0) < (unsigned)C.rn && (unsigned)(k - C.rk0) < (unsigned)C.rn;
  const GbfPf Lc = pf_ld(w.L2 + c), Lxm = pf_ld(w.L2 + c - 1), Lxp = pf_ld(w.L2 + c + 1);
  const GbfPf Lyu = pf_ld(w.L2 + c - nx), Lyd = pf_ld(w.L2 + c + nx);
  const GbfPf Lzm = pf_ld(w.L2 + c - pl), Lzp = pf_ld(w.L2 + c + pl);
  const bool dnapl = !gbf_is_zero(Sd) || src || Lc.h != 0.f || Lxm.h != 0.f || Lxp.h != 0.f || Lyu.h != 0.f ||
                     Lyd.h != 0.f || Lzm.h != 0.f || Lzp.h != 0.f;
  if (MASS) acc.r1 = pf_add(acc.r1, cells.phi ? pf_mulf(r1, phif) : pf_mul(r1, C.phip[md]));
  double Sn;
  GbfPf dp, r2 = zero;
  if (dnapl) {
    const GbfPf G = pf_add(pf_mul(C.g2, Pp), C.ghd);
    const GbfPf y1 = pf_add(yu, G), y2 = noflow ? zero : pf_add(yd, G);
    const GbfPf f = pair_sum3(pair_net(pair_face(xp, Lc, Lxp), pair_face(xm, Lxm, Lc), C.wx),
                              pair_net(pair_face(y2, Lc, Lyd), pair_face(y1, Lyu, Lc), C.wy),
                              pair_net(pair_face(zp, Lc, Lzp), pair_face(zm, Lzm, Lc), C.wz));
    r2 = pf_mul(f, rphi);
    double rest = 0.;  // what the pair r2 leaves of the source
    if (src) r2 = pf_sub(r2, pair_source(C.dtsrc_d, cells.phi ? gbf_f2d(phif) : C.phi_d[md], rest));
    GbfPf ds;
    pair_newton(C, md, Pp, pf_from_double(Sd), gbf_is_zero(Sd) ? C.pd[md] : pf_ld(w.Pk + c), r1, r2, dp, ds);
    const double dsd = pf_to_double(ds);
    Sn = __dadd_rn(Sd, dsd);
    if (src) Sn = pair_add_rest(Sd, dsd, rest, C.rro2_d);
    if (MASS) {
      const double phi = cells.phi ? gbf_f2d(phif) : C.phi_d[md];
      const double pa = __dsub_rn(Pd, C.Patm_d), q1 = __fma_rn(C.k1_d, pa, C.ro1_d);
      acc.m1 = __fma_rn(phi, __fma_rn(-q1, Sd, q1), acc.m1);
      acc.m2 = __fma_rn(phi, __fma_rn(__fma_rn(C.k2_d, pa, C.ro2_d), Sd, __dsub_rn(rest, pf_to_double(r2))), acc.m2);
    }
  } else {
    dp = pf_neg(pf_mul(r1, C.rk1));  // rho01 beta1 dP = -r1
    Sn = Sd;
    if (MASS) {
      const double phi = cells.phi ? gbf_f2d(phif) : C.phi_d[md];
      acc.m1 = __fma_rn(phi, __fma_rn(C.k1_d, __dsub_rn(Pd, C.Patm_d), C.ro1_d), acc.m1);
    }
  }
  if (s.roS1) pair_mass_arrays(C, s, c, Pd, Sd, r1, r2);
  const double Pn = __dadd_rn(Pd, pf_to_double(dp));
  if (!gbf_is_finite(Pn) || !gbf_is_finite(Sn)) bad = 1;
  s.Pn[c] = Pn;
  s.Sn[c] = Sn;
}
