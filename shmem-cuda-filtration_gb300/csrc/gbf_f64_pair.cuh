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
// An increment is then accurate to about 2^-46 of itself, and P + dP, S + dS
// are rounded once in FP64. The arithmetic that forms masses of 1000 kg/m^3 in
// FP64 and recovers P through rho0 beta from their rounding loses about
// 2^-53 / beta1 of P: with beta1 = 1e-9 and P near hydrostatic the error against
// 64-bit increments is 8e-13 of P there and 4e-17 here. Cells that pairs do not
// hold are refused, and taken again in FP64 (pair_cell_again):
//   * S_e below 2^-11, capillary pressure above a limit (`ratio` in
//     pair_newton), and a Newton that 7 iterations do not end. The limit keeps P_k
//     and its slope in FP32's range and the Newton's convergence quadratic: near
//     residual water the reference's 7 iterations stop before they converge, and
//     what they leave is the result;
//   * a change of a phase's mass above 2^-5 of its density, where 2^-46 of it
//     would show beside FP64's 2^-53. With the reference's compressibilities and
//     white noise of 1000 and 10,000 Pa in P the mean errors of S are 1.6e-17 and
//     1.8e-17, the plain FP64 passes' 2.4e-17 (without the limit 1.8e-17, 1.4e-16);
//   * P further than 2^-5 P_atm from hydrostatic (2^-5 / beta1 where that is
//     more) in the cell or next to it. P - P_hs is a multiple of P's last place,
//     2^-53 to 2^-52 of P: nearer than that it fits the pair's 48 bits, further
//     away the cell's face potentials are taken from FP64 differences. So are
//     those at pressures above 32 / beta1, where the water's weight is that of
//     32 times its density and fluxes of 2^3 of the limit above cancel.
// The looks for these cost 24 of 660 us a step at 256^3 where no cell is refused.
// Where many are (192^3, us a step): 10,000 Pa off hydrostatic everywhere with
// the reference's compressibilities, all wet 624 -> 1030, all dry 176 -> 460;
// noise of 10,000 Pa 20,800 and 2400; S_e 1e-6 everywhere 18,200. The plain
// passes take about 3700, since they form each mobility once; cells like these
// are few in a state that time steps have smoothed.
// S below about 1e-13 has no mobility in pairs (om^3 is below FP32's range; in
// FP64 it would move 1e-26 of itself a step).
#pragma once

#include "gbf_f64_cell.cuh"
#include "gbf_pair.cuh"

constexpr float kPairMost = 0.03125f;  // 2^-5: the largest change of a cell (of its density or saturation) in pairs

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
  float Patm;
  float far;          // limit of |P - P_hs|: 2^-5 of P_atm or 1 / beta1
  float deep;         // limit of P - P_atm: 32 / beta1
  float rro1, rro2;   // 1 / rho0
  double H_d;         // rho01 g h2
  GbfPf k1, k2, rk1;     // rho01 beta1, rho02 beta2, 1 / (rho01 beta1)
  GbfPf ro1, ro2;        // rho01, rho02
  GbfPf g1, g2, ghd;     // g h2 rho01 beta1, g h2 rho02 beta2, g h2 (rho02 - rho01)
  GbfPf wx, wy, wz;      // dt / h1^2, dt kv / h2^2, dt / h3^2 (over the scale)
  GbfPf c1, c2;          // 1 / mu (times the scale)
  GbfPf K[2], phip[2], rphi[2], inv[2], E3p[2], pd[2], ilam[2];
  double phi_d[2], inv_d[2], E1[2], E2[2];  // 1 / (1 - S_wr); Brooks-Corey exponents over ln 2
  float E1f[2], E2f[2];
  float taylor[2][4];    // (1 / lambda + n) / (n + 1), n = 1..4
  double ro1_d, ro2_d, beta1_d, beta2_d, Patm_d, k1_d, k2_d;  // the densities' constants
  double dtsrc_d, rro2_d;  // dt x the rate source per volume, 1 / rho02
};
inline GbfPairConsts gbf_pair_consts(const gbf_model& m) {
  GbfPairConsts C = {};
  const GbfDerived d = gbf_derive(m);
  C.nx = m.nx; C.ny = m.ny; C.nz = m.nz;
  C.noflow = m.bc_mode == GBF_BC_HYDROSTATIC_SIDES;
  C.pl = (unsigned)m.nx * (unsigned)m.ny;
  C.n = C.pl * (unsigned)m.nz;
  C.nint = (unsigned)(m.nx - 2) * (unsigned)(m.ny - 2) * (unsigned)(m.nz - 2);
  C.dnx = gbf_fast_div((unsigned)m.nx);
  C.dny = gbf_fast_div((unsigned)m.ny);
  C.dix = gbf_fast_div((unsigned)m.nx - 2);
  C.diy = gbf_fast_div((unsigned)m.ny - 2);
  if (d.src != 0.) {
    C.rn = m.rate_cells;
    C.ri0 = m.nx / 2 - m.rate_cells / 2;
    C.rk0 = m.nz / 2 - m.rate_cells / 2;
  }
  C.Patm = (float)fabs(m.P_atm);
  C.far = (float)(0x1p-5 * fmax(fabs(m.P_atm), 1. / m.beta1));
  C.deep = (float)(32. / m.beta1);
  C.rro1 = (float)(1. / m.ro01);
  C.rro2 = (float)(1. / m.ro02);
  C.H_d = m.ro01 * m.g * m.h2;
  // 2^e that brings the water mobility x density of media 0 to about 1
  int e = 0;
  const double L = m.K[0] * m.ro01 / m.mu1;
  if (L > 0. && isfinite(L)) frexp(L, &e);
  e = e < -60 ? -60 : e > 60 ? 60 : e;
  const double sc = ldexp(1.0, -e), log2e = 1.4426950408889634074;
  C.k1 = pf_const(m.ro01 * m.beta1);
  C.k2 = pf_const(m.ro02 * m.beta2);
  C.rk1 = pf_const(1.0 / (m.ro01 * m.beta1));
  C.ro1 = pf_const(m.ro01);
  C.ro2 = pf_const(m.ro02);
  C.g1 = pf_const(m.g * m.h2 * m.ro01 * m.beta1);
  C.g2 = pf_const(m.g * m.h2 * m.ro02 * m.beta2);
  C.ghd = pf_const(m.g * m.h2 * (m.ro02 - m.ro01));
  C.wx = pf_const(m.dt / (m.h1 * m.h1) / sc);
  C.wy = pf_const(m.dt * m.kv / (m.h2 * m.h2) / sc);
  C.wz = pf_const(m.dt / (m.h3 * m.h3) / sc);
  C.c1 = pf_const(sc / m.mu1);
  C.c2 = pf_const(sc / m.mu2);
  C.dtsrc_d = m.dt * d.src;
  C.rro2_d = 1.0 / m.ro02;
  for (int md = 0; md < 2; md++) {
    C.K[md] = pf_const(m.K[md]);
    C.phi_d[md] = m.m[md];
    C.phip[md] = pf_const(m.m[md]);
    C.rphi[md] = pf_const(1.0 / m.m[md]);
    C.inv[md] = pf_const(d.inv_1mswr[md]);
    C.inv_d[md] = d.inv_1mswr[md];
    C.E1[md] = d.e1[md] * log2e;
    C.E2[md] = d.e2[md] * log2e;
    C.E1f[md] = (float)C.E1[md];
    C.E2f[md] = (float)C.E2[md];
    C.E3p[md] = pf_const(d.m_inv_lam[md] * log2e);
    C.pd[md] = pf_const(m.P_d[md]);
    C.ilam[md] = pf_const(d.inv_lam_1mswr[md]);
    for (int n = 1; n <= 4; n++) C.taylor[md][n - 1] = (float)((1.0 / m.lambda[md] + n) / (n + 1));
  }
  C.ro1_d = m.ro01; C.ro2_d = m.ro02; C.beta1_d = m.beta1; C.beta2_d = m.beta2; C.Patm_d = m.P_atm;
  C.k1_d = m.ro01 * m.beta1; C.k2_d = m.ro02 * m.beta2;
  return C;
}
// Models of the pair step. It solves the Newton's equations to round-off, as
// the reference's 7 iterations (and more) do; a model that asks for fewer stops
// before, and keeps the plain FP64 passes (gbf_f64_cell.cuh). So does one whose
// constants, or the exponents of 2 that S_e >= 2^-11 gives (11 / lambda in P_k),
// are too near the ends of FP32's range for products of two or three of them
// and the low parts of their pairs.
inline bool gbf_pair_applies(const gbf_model& m) {
  auto fits = [](double x) { return fabs(x) >= 0x1p-40 && fabs(x) <= 0x1p40; };
  const GbfDerived d = gbf_derive(m);
  bool ok = m.newton_iterations >= 7 && fits(m.ro01) && fits(m.ro02) && fits(m.ro01 * m.beta1) && m.beta1 > 0. &&
            fits(1. / m.beta1) && (m.beta2 == 0. || fits(m.ro02 * m.beta2)) && (m.g == 0. || fits(m.g * m.h2)) &&
            fits(m.dt / (m.h1 * m.h1) / m.mu1) && fits(m.dt * m.kv / (m.h2 * m.h2) / m.mu1) &&
            fits(m.dt / (m.h3 * m.h3) / m.mu1) && fits(m.mu1) && fits(m.mu2) && fabs(m.P_atm) <= 0x1p40;
  for (int md = 0; md < 2; md++)
    ok = ok && m.lambda[md] >= 0.125 && m.lambda[md] <= 1024. && d.inv_1mswr[md] <= 0x1p10 && fits(m.m[md]) &&
         m.P_d[md] <= 0x1p40 && m.K[md] >= 0. && m.K[md] <= 0x1p40;
  return ok;
}
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
  const float2 v = *p;  // written by pass 1, which may still run when this kernel starts: no __ldg
  return {v.x, v.y};
}
__device__ __forceinline__ void pf_st(float2* p, GbfPf a) { *p = make_float2(a.h, a.l); }

// Brooks-Corey functions of om = 1 - S_e = S / (1 - S_wr): kr1 = S_e^e1, w =
// 1 - S_e^e2 (kr2 = om^2 w) and P_k / P_d = S_e^(-1/lambda). Beyond the
// tables' range (S_e <= 2^-11, S far below 0, NaN) the mobilities come from
// CUDA's functions, with the FP64 passes' limits (S_e = 0: kr1 = 0; S_e < 0:
// NaN), and P_k is infinite, which sends the cell itself to pair_cell_f64.
__device__ __forceinline__ bool pair_om_ok(float om) { return om < 0.9995f && om > -0.25f; }
static __device__ __noinline__ double pair_pow_general(double om, double E) {
  return exp2(E * log(1.0 - om));
}
__device__ __forceinline__ GbfPf pair_pk_none() { return {__uint_as_float(0x7f800000u), 0.f}; }
// P_k(S) (rare: the Newton's changes of S beyond its expansion's range).
static __device__ __noinline__ GbfPf pair_pk(const GbfPairConsts& C, int md, GbfPf S) {
  const double om = __dmul_rn(pf_to_double(S), C.inv_d[md]);
  const float omf = pf_from_double(om).h;
  if (!pair_om_ok(omf)) return pair_pk_none();
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
    P = s.P[c];
    S = s.S[c];
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
      pk = pair_pk_none();
    }
    l1 = pf_mul(l1, kr1);
    l2 = pf_mul(pf_mul(over_mu(C.c2), pf_mul(pf_mul(omp, omp), w2)), pf_add(C.ro2, pf_mul_raw(C.k2, Pp)));
    pf_st(w.Pk + c, pk);
  }
  // NaN: pass 2 refuses the cells whose potentials use it
  pf_st(w.D + c, fabsf(D.h) <= C.far && Pp.h <= C.deep ? D : GbfPf{__uint_as_float(0x7fffffffu), 0.f});
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
// w (out - in); MAG: mag + w times the larger of the two
template <bool MAG>
__device__ __forceinline__ GbfPf pair_net(GbfPf out, GbfPf in, GbfPf w, float& mag) {
  if (MAG) mag = __fmaf_rn(w.h, fmaxf(fabsf(out.h), fabsf(in.h)), mag);
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
// 2^-21 of itself, so two or three reach round-off, and it ends there whatever
// newton_tol is (an end at newton_tol = 1e-11 errs by 1.7e-16 of P where this
// one errs by 8e-17). False: it did not, or the cell is none for pairs (see the
// top of this file).
__device__ __forceinline__ bool pair_newton(const GbfPairConsts& C, int md, GbfPf Pp, GbfPf S, GbfPf Pk, GbfPf r1,
                                            GbfPf r2, GbfPf& dp, GbfPf& ds) {
  const GbfPf rho1 = pf_add(C.ro1, pf_mul_raw(C.k1, Pp));
  const GbfPf rho2 = pf_add(C.ro2, pf_mul_raw(C.k2, pf_add(Pp, Pk)));
  const GbfPf omS = pf_sub(GbfPf{1.f, 0.f}, S);
  const GbfPf Se = pf_sub(GbfPf{1.f, 0.f}, pf_mul(S, C.inv[md]));
  r2 = pf_add(r2, pf_mul(pf_mul(C.k2, Pk), S));
  const GbfPf slope = pf_div(pf_mul(Pk, C.ilam[md]), Se);  // dP_k/dS
  const float rSe = __fmul_rn(C.inv[md].h, pf_rcp(Se.h));  // relative change of S_e per change of S
  float J11 = __fmul_rn(C.k1.h, omS.h), mJ12 = rho1.h, J21 = __fmul_rn(C.k2.h, S.h);
  const float share = __fmul_rn(J21, slope.h), rrho2 = pf_rcp(rho2.h);
  float J22 = __fadd_rn(rho2.h, share);
  float inv = pf_rcp(__fmaf_rn(J11, J22, __fmul_rn(mJ12, J21)));
  const float ratio = fabsf(__fmul_rn(share, rrho2));  // the capillary term's part of J22
  // what the pairs' 2^-46 of P_k leave of S is below 2^-54 with ratio <= 2^-8
  if (!(ratio <= 3.90625e-3f)) return false;
  const float rb = fmaxf(__fmul_rn(C.k1.h, pf_rcp(rho1.h)), fabsf(__fmul_rn(C.k2.h, rrho2)));  // of the densities, per change of P
  GbfPf G1 = r1, G2 = r2;
  for (int it = 0; it < 7; it++) {
    const float ep = -__fmul_rn(inv, __fmaf_rn(J22, G1.h, __fmul_rn(mJ12, G2.h)));
    const float es = -__fmul_rn(inv, __fmaf_rn(J11, G2.h, -__fmul_rn(J21, G1.h)));
    dp = it ? pf_addf(dp, ep) : GbfPf{ep, 0.f};
    ds = it ? pf_addf(ds, es) : GbfPf{es, 0.f};
    const float x = __fmul_rn(ds.h, rSe);  // relative change of S_e
    if (!(fabsf(x) <= 0.5f && fabsf(ds.h) <= kPairMost)) return false;
    // what the step leaves: the Jacobian's error (2^-21) or its change since the point it was formed
    // at, of the step; small enough once below 2^-54 of S and of P
    const float chg = it > 1 ? __fmaf_rn(fabsf(ep), rb, fabsf(__fmul_rn(es, rSe))) : __fmaf_rn(fabsf(dp.h), rb, fabsf(x));
    const float q = fmaxf(4.77e-7f, __fmul_rn(8.f, chg));
    const float Pa = __fadd_rn(fabsf(Pp.h), C.Patm);
    const float lim_s = __fmul_rn(5.55e-17f, fabsf(__fadd_rn(S.h, ds.h))), lim_p = __fmul_rn(5.55e-17f, Pa);
    if ((__fmul_rn(q, fabsf(es)) <= lim_s || fabsf(es) <= __fmul_rn(2.8e-14f, fabsf(ds.h))) &&
        (__fmul_rn(q, fabsf(ep)) <= lim_p || fabsf(ep) <= __fmul_rn(2.8e-14f, fabsf(dp.h))))
      return true;
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
  return false;
}

// The Newton's equations of pair_newton in FP64. False: not a cell for
// increments, or no end within 7 iterations.
__device__ __forceinline__ bool pair_newton_f64(const gbf_model& m, const GbfDerived& d, int md, double P, double S,
                                                double r1, double r2, double& dp, double& ds) {
  const double inv = d.inv_1mswr[md], om = S * inv, Se = 1. - om, k1 = m.ro01 * m.beta1, k2 = m.ro02 * m.beta2;
  if (!(om > -0.25 && om < 0.9995)) return false;
  const double Pk = m.P_d[md] * exp(d.m_inv_lam[md] * log1p(-om)), pa = P - m.P_atm;
  const double rho1 = m.ro01 * (1. + m.beta1 * pa), rho2 = m.ro02 * (1. + m.beta2 * (pa + Pk));
  r2 += k2 * Pk * S;
  double dPk = 0.;
  dp = ds = 0.;
  for (int it = 0; it < 7; it++) {
    const double Sn = S + ds, slope = (Pk + dPk) * d.inv_lam_1mswr[md] / (Se - ds * inv);
    if (it == 0 && !(fabs(k2 * S * slope) <= 0x1p-8 * fabs(rho2))) return false;
    const double G1 = r1 + k1 * dp * (1. - Sn) - rho1 * ds, G2 = r2 + k2 * (dp + dPk) * Sn + rho2 * ds;
    const double J11 = k1 * (1. - Sn), J12 = -(rho1 + k1 * dp), J21 = k2 * Sn;
    const double J22 = rho2 + k2 * (dp + dPk + slope * Sn), rdet = 1. / (J11 * J22 - J12 * J21);
    const double ep = -rdet * (J22 * G1 - J12 * G2), es = -rdet * (J11 * G2 - J21 * G1);
    dp += ep;
    ds += es;
    if (!(fabs(ds * inv) <= 0.5 * fabs(Se))) return false;
    if (fabs(ep) <= 0x1p-50 * fabs(dp) + 0x1p-56 * fabs(P) && fabs(es) <= 0x1p-50 * fabs(ds) + 0x1p-56 * fabs(S)) return true;
    dPk = Pk * expm1(d.m_inv_lam[md] * log1p(-ds * inv / Se));
  }
  return false;
}

// The step of one cell in FP64 and in increments, its stencil's mobilities
// formed here since no pass keeps them in FP64. Returns its part of the masses.
static __device__ __noinline__ double2 pair_cell_f64(const gbf_model& m, const GbfDerived& d, const gbf_cells& cells,
                                                     const GbfF64Step& s, int i, int j, int k) {
#ifdef GBF_COUNT_FP64_CELL
  GBF_COUNT_FP64_CELL;  // the tests' build for the CPU
#endif
  const GbfGeo g = gbf_geo(m);
  const size_t c = gbf_idx(g, i, j, k);
  double S[7], P[7], L1[7], L2[7];
  auto at = [&](int t) {
    const size_t st = t < 3 ? 1 : t < 5 ? (size_t)g.nx : g.pl;
    return t == 0 ? c : (t & 1) ? c - st : c + st;
  };
#pragma unroll
  for (int t = 0; t < 7; t++) {
    S[t] = s.S[at(t)];
    P[t] = s.P[at(t)];
  }
  const int md = gbf_media_at(cells, c);
  const double phi = cells.phi ? (double)cells.phi[c] : m.m[md], dtphi = m.dt / phi;
  const bool src = d.src != 0. && j == 1 && gbf_in_rate_patch(m, i, k);
  bool dry = !src;
#pragma unroll
  for (int t = 0; t < 7; t++) dry = dry && gbf_is_zero(S[t]);
#pragma unroll 1
  for (int t = 0; t < 7; t++) {
    const int mt = gbf_media_at(cells, at(t));
    const double K = cells.K ? (double)cells.K[at(t)] : m.K[mt], pa = P[t] - m.P_atm;
    double k1 = 1., k2 = 0.;
    if (!gbf_is_zero(S[t])) {
      const double om = S[t] * d.inv_1mswr[mt], l = log1p(-om);
      k1 = exp(d.e1[mt] * l);
      k2 = om * om * -expm1(d.e2[mt] * l);
    }
    L1[t] = K * k1 * d.neg_inv_mu1 * (m.ro01 * (1. + m.beta1 * pa));
    L2[t] = K * k2 * d.neg_inv_mu2 * (m.ro02 * (1. + m.beta2 * pa));
  }
  const bool noflow_bottom = m.bc_mode == GBF_BC_HYDROSTATIC_SIDES && j == g.ny - 2;
  const GbfF64Faces faces = gbf_f64_faces(d, s.P, c, g.nx, g.pl);
  const double ro1 = m.ro01 * (1. + m.beta1 * (P[0] - m.P_atm)), ro2 = m.ro02 * (1. + m.beta2 * (P[0] - m.P_atm));
  const double r1 = dtphi * gbf_f64_divergence(m, d, faces, ro1 * m.g, noflow_bottom, L1);
  const double q1 = ro1 * (1. - S[0]), q2 = ro2 * S[0];
  double r2 = 0., Pn = P[0], Sn = S[0];
  if (dry) {
    Pn -= r1 / (m.ro01 * m.beta1);
  } else {
    double dp, ds;
    r2 = dtphi * gbf_f64_divergence(m, d, faces, ro2 * m.g, noflow_bottom, L2);
    if (src) r2 -= dtphi * d.src;
    if (pair_newton_f64(m, d, md, P[0], S[0], r1, r2, dp, ds)) {
      Pn += dp;
      Sn += ds;
    } else {
      gbf_f64_newton(m, d, md, log((1. - S[0] - m.S_wr[md]) / (1. - m.S_wr[md])), q1 - r1, q2 - r2, Pn, Sn);
    }
  }
  if (s.roS1) {
    s.roS1_old[c] = q1;
    s.roS2_old[c] = q2;
    s.roS1[c] = q1 - r1;
    s.roS2[c] = q2 - r2;
  }
  if (!gbf_is_finite(Pn) || !gbf_is_finite(Sn)) atomicOr(s.status, GBF_DEV_NONFINITE);
  s.Pn[c] = Pn;
  s.Sn[c] = Sn;
  return make_double2(phi * (q1 - r1), phi * (q2 - r2));
}
// (*a - *b) + H as a pair.
static __device__ __noinline__ GbfPf pair_diff64(const double* a, const double* b, double H) {
  return pf_from_double(__dadd_rn(__dsub_rn(*a, *b), H));
}

// What stands in S of the next state at a cell that the pairs refused, for its
// differences of P - P_hs or for good, until it is taken again: NaNs of its own.
constexpr int kPairRefused = 0x7ffaf64c;
__device__ __forceinline__ double pair_refused(bool differences) { return __hiloint2double(kPairRefused, differences ? 1 : 0); }

// Pass 2 at interior cell (i, j, k) = c: fluxes, Newton, next state (the
// water-only form where no DNAPL is in the cell or flows through its faces).
// False, and a mark left in S: not a cell for pairs (see the top of this file).
// FAR: such a cell again, its potentials from FP64 differences (without a mark).
template <bool MASS, bool FAR>
__device__ __forceinline__ bool gbf_pair_step_cell(const GbfPairConsts& C, const gbf_cells& cells,
                                                   const GbfF64Step& s, const GbfPairWork& w, int i, int j, int k,
                                                   unsigned c, GbfPairMass& acc, unsigned& bad) {
  const unsigned nx = (unsigned)C.nx, pl = C.pl;
  const int md = cells.media ? __ldg(cells.media + c) : 0;
  const GbfPairRow R = w.rows[j];
  const double Pd = s.P[c];
  const GbfPf D = FAR ? pf_from_double(__dsub_rn(Pd, R.phs)) : pf_ld(w.D + c);
  const GbfPf Pp = pf_add(R.pp, D);  // P - P_atm
  // face potentials times h; gravity g h2 (rho_a - rho01) with the centre cell's density
  GbfPf xm = pf_ld(w.D + c - 1), xp = pf_ld(w.D + c + 1), yu = pf_ld(w.D + c - nx), yd = pf_ld(w.D + c + nx);
  GbfPf zm = pf_ld(w.D + c - pl), zp = pf_ld(w.D + c + pl);
  if (FAR) {
    const double* P = s.P + c;
    xm = pair_diff64(P - 1, P, 0.);
    xp = pair_diff64(P, P + 1, 0.);
    zm = pair_diff64(P - pl, P, 0.);
    zp = pair_diff64(P, P + pl, 0.);
    yu = pair_diff64(P - nx, P, C.H_d);
    yd = pair_diff64(P, P + nx, C.H_d);
  } else {
    xm = pf_diff(xm, D);
    xp = pf_diff(D, xp);
    zm = pf_diff(zm, D);
    zp = pf_diff(D, zp);
    yu = pf_addf(pf_diff(yu, D), R.eu);
    yd = pf_addf(pf_diff(D, yd), R.ed);
  }
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
  // a phase's net change of density in the cell and 2^-3 of that through its faces (FAR), over rho0; a NaN shows
  auto change = [&](GbfPf r, float mag, float rro) {
    return __fmul_rn(FAR ? __fmaf_rn(mag, __fmul_rn(0.125f, rphi.h), fabsf(r.h)) : fabsf(r.h), rro);
  };
  float mag = 0.f, most;
  {
    const GbfPf Lc = pf_ld(w.L1 + c), G = pf_mul(C.g1, Pp);
    const GbfPf y1 = pf_add(yu, G), y2 = noflow ? zero : pf_add(yd, G);
    const GbfPf f = pair_sum3(
        pair_net<FAR>(pair_face(xp, Lc, pf_ld(w.L1 + c + 1)), pair_face(xm, pf_ld(w.L1 + c - 1), Lc), C.wx, mag),
        pair_net<FAR>(pair_face(y2, Lc, pf_ld(w.L1 + c + nx)), pair_face(y1, pf_ld(w.L1 + c - nx), Lc), C.wy, mag),
        pair_net<FAR>(pair_face(zp, Lc, pf_ld(w.L1 + c + pl)), pair_face(zm, pf_ld(w.L1 + c - pl), Lc), C.wz, mag));
    r1 = pf_mul(f, rphi);
    most = change(r1, mag, C.rro1);
    mag = 0.f;
  }
  const double Sd = s.S[c];
  const bool src = C.rn > 0 && j == 1 && (unsigned)(i - C.ri0) < (unsigned)C.rn && (unsigned)(k - C.rk0) < (unsigned)C.rn;
  const GbfPf Lc = pf_ld(w.L2 + c), Lxm = pf_ld(w.L2 + c - 1), Lxp = pf_ld(w.L2 + c + 1);
  const GbfPf Lyu = pf_ld(w.L2 + c - nx), Lyd = pf_ld(w.L2 + c + nx);
  const GbfPf Lzm = pf_ld(w.L2 + c - pl), Lzp = pf_ld(w.L2 + c + pl);
  const bool dnapl = !gbf_is_zero(Sd) || src || Lc.h != 0.f || Lxm.h != 0.f || Lxp.h != 0.f || Lyu.h != 0.f ||
                     Lyd.h != 0.f || Lzm.h != 0.f || Lzp.h != 0.f;
  double Sn;
  bool ok;
  GbfPf dp, r2 = zero;
  if (dnapl) {
    const GbfPf G = pf_add(pf_mul(C.g2, Pp), C.ghd);
    const GbfPf y1 = pf_add(yu, G), y2 = noflow ? zero : pf_add(yd, G);
    const GbfPf f = pair_sum3(pair_net<FAR>(pair_face(xp, Lc, Lxp), pair_face(xm, Lxm, Lc), C.wx, mag),
                              pair_net<FAR>(pair_face(y2, Lc, Lyd), pair_face(y1, Lyu, Lc), C.wy, mag),
                              pair_net<FAR>(pair_face(zp, Lc, Lzp), pair_face(zm, Lzm, Lc), C.wz, mag));
    r2 = pf_mul(f, rphi);
    ok = most <= kPairMost && change(r2, mag, C.rro2) <= kPairMost;
    double rest = 0.;  // what the pair r2 leaves of the source
    if (src) r2 = pf_sub(r2, pair_source(C.dtsrc_d, cells.phi ? gbf_f2d(phif) : C.phi_d[md], rest));
    GbfPf ds;
    ok = ok && pair_newton(C, md, Pp, pf_from_double(Sd), gbf_is_zero(Sd) ? C.pd[md] : pf_ld(w.Pk + c), r1, r2, dp, ds);
    const double dsd = pf_to_double(ds);
    Sn = __dadd_rn(Sd, dsd);
    if (src) Sn = pair_add_rest(Sd, dsd, rest, C.rro2_d);
    if (MASS && ok) {
      const double phi = cells.phi ? gbf_f2d(phif) : C.phi_d[md];
      const double pa = __dsub_rn(Pd, C.Patm_d), q1 = __fma_rn(C.k1_d, pa, C.ro1_d);
      acc.m1 = __fma_rn(phi, __fma_rn(-q1, Sd, q1), acc.m1);
      acc.m2 = __fma_rn(phi, __fma_rn(__fma_rn(C.k2_d, pa, C.ro2_d), Sd, __dsub_rn(rest, pf_to_double(r2))), acc.m2);
    }
  } else {
    dp = pf_neg(pf_mul(r1, C.rk1));  // rho01 beta1 dP = -r1
    Sn = Sd;
    ok = most <= kPairMost;
    if (MASS && ok) {
      const double phi = cells.phi ? gbf_f2d(phif) : C.phi_d[md];
      acc.m1 = __fma_rn(phi, __fma_rn(C.k1_d, __dsub_rn(Pd, C.Patm_d), C.ro1_d), acc.m1);
    }
  }
  if (!ok) {
    if (!FAR) s.Sn[c] = pair_refused(most != most);
    return false;
  }
  if (MASS) acc.r1 = pf_add(acc.r1, cells.phi ? pf_mulf(r1, phif) : pf_mul(r1, C.phip[md]));
  if (s.roS1) pair_mass_arrays(C, s, c, Pd, Sd, r1, r2);
  const double Pn = __dadd_rn(Pd, pf_to_double(dp));
  if (!gbf_is_finite(Pn) || !gbf_is_finite(Sn)) bad = 1;
  s.Pn[c] = Pn;
  s.Sn[c] = Sn;
  return true;
}

// Interior cell number t.
__device__ __forceinline__ unsigned pair_cell(const GbfPairConsts& C, unsigned t, int& i, int& j, int& k) {
  const unsigned r = gbf_div(t, C.dix), q = gbf_div(r, C.diy);
  i = (int)(1u + t - r * C.dix.d);
  j = (int)(1u + r - q * C.diy.d);
  k = (int)(1u + q);
  return (unsigned)i + (unsigned)j * (unsigned)C.nx + (unsigned)k * C.pl;
}
__device__ __forceinline__ bool pair_is_refused(const GbfPairConsts& C, const GbfF64Step& s, unsigned t) {
  int i, j, k;
  return __double2hiint(s.Sn[pair_cell(C, t, i, j, k)]) == kPairRefused;
}
// A cell that gbf_pair_step_cell refused; its part of the masses.
template <bool MASS>
static __device__ __noinline__ double2 pair_cell_again(const GbfPairConsts& C, const gbf_model& m, const GbfDerived& d,
                                                       const gbf_cells& cells, const GbfF64Step& s,
                                                       const GbfPairWork& w, unsigned t) {
  int i, j, k;
  const unsigned c = pair_cell(C, t, i, j, k);
  if (__double2loint(s.Sn[c])) {
    GbfPairMass acc;
    unsigned bad = 0;
    if (gbf_pair_step_cell<MASS, true>(C, cells, s, w, i, j, k, c, acc, bad)) {
      if (bad) atomicOr(s.status, GBF_DEV_NONFINITE);
      return make_double2(acc.m1 - pf_to_double(acc.r1), acc.m2);
    }
  }
  return pair_cell_f64(m, d, cells, s, i, j, k);
}
// Pass 2 at interior cells t0, t0 + stride, .. below t1, summed into acc; every
// thread of the block calls it. The cells that the pairs refuse are taken after
// the others: calls among the pair arithmetic cost it registers (256^3, none
// refused: pass 2 488 us with them there, 470 after the others, 447 without
// any). Up to an eighth of a block's cells, they are listed and shared out
// evenly, in a fixed order: a warp pays for the FP64 of one lane what it pays
// for 32. More than that, a thread takes its own, whose neighbours' are in its
// warp.
template <bool MASS>
__device__ __forceinline__ void gbf_pair_step_cells(const GbfPairConsts& C, const gbf_model& m, const GbfDerived& d,
                                                    const gbf_cells& cells, const GbfF64Step& s, const GbfPairWork& w,
                                                    unsigned t0, unsigned stride, unsigned t1, GbfPairMass& acc) {
  unsigned bad = 0, first = t1, last = 0;  // of the refused cells
  for (unsigned t = t0; t < t1; t += stride) {
    int i, j, k;
    const unsigned c = pair_cell(C, t, i, j, k);
    if (!gbf_pair_step_cell<MASS, false>(C, cells, s, w, i, j, k, c, acc, bad)) {
      first = min(first, t);
      last = t;
    }
  }
  if (bad) atomicOr(s.status, GBF_DEV_NONFINITE);
  auto again = [&](unsigned t) {
    const double2 phiA = pair_cell_again<MASS>(C, m, d, cells, s, w, t);
    if (MASS) {
      acc.m1 += phiA.x;
      acc.m2 += phiA.y;
    }
  };
#ifdef __CUDACC__
  if (!__syncthreads_or(first < t1)) return;
  // 512 B: with 2 KB a block programmatic launches no longer overlap (40 steps of 40^3 788 -> 942 us)
  constexpr unsigned kList = 128;
  __shared__ unsigned list[kList], warps[32];
  unsigned n = 0;  // this thread's
  for (unsigned t = first; t < t1 && t <= last; t += stride) n += pair_is_refused(C, s, t);
  const unsigned lane = threadIdx.x & 31u;
  unsigned rank = n;  // cells of the threads before, in the warp and in the block
  for (unsigned o = 1; o < 32u; o <<= 1) {
    const unsigned v = __shfl_up_sync(0xffffffffu, rank, o);
    if (lane >= o) rank += v;
  }
  if (lane == 31u) warps[threadIdx.x >> 5] = rank;
  __syncthreads();
  rank -= n;
  unsigned total = 0;
  for (unsigned q = 0; q < blockDim.x >> 5; q++) {
    if (q < threadIdx.x >> 5) rank += warps[q];
    total += warps[q];
  }
  if (total * 8u > (t1 - (t0 - threadIdx.x) + stride - 1u) / stride * blockDim.x) {  // the block's cells: t0 is its first plus threadIdx.x
    for (unsigned t = first; t < t1 && t <= last; t += stride)
      if (pair_is_refused(C, s, t)) again(t);
    return;
  }
  unsigned t = first;
  for (unsigned base = 0; base < total; base += kList) {
    for (; t < t1 && t <= last && rank < base + kList; t += stride)
      if (pair_is_refused(C, s, t)) list[rank++ - base] = t;
    __syncthreads();
    for (unsigned q = threadIdx.x; q < kList && base + q < total; q += blockDim.x) again(list[q]);
    __syncthreads();
  }
#else
  for (unsigned t = first; t < t1 && t <= last; t += stride)
    if (pair_is_refused(C, s, t)) again(t);
#endif
}
