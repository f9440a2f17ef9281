// gbf_eager.cu — one FP64 kernel per hot-path function of the reference.
//
// These are the kernels behind the drop-in's default (eager) mode: each
// reference function call launches its own kernel and writes the reference's
// arrays, so any caller of the defines.h function set sees exactly the
// reference's intermediate state. Semantics follow the reference CPU path
// (cpu.cpp), which is the oracle:
//   * a 3-D iteration space covered by a flat grid-stride loop (the reference
//     GPU kernels' blockIdx.y / BlockNY split, gpu.cu:61-62, leaves cells
//     untouched whenever ceil(Ny/4) != 4; this mapping has no such gap);
//   * model.newton_iterations Newton iterations (7 in the reference CPU path,
//     defines.h:15; the reference GPU kernel runs one, gpu.cu:342-374);
//   * boundary values of the CPU's in-place i->j->k sweep (cpu.cpp:44-54),
//     computed race-free in two kernels (gather to scratch, then scatter).
//
// This translation unit is compiled with -fmad=false so that every
// multiply-add rounds like the oracle's; only pow() may differ in the last
// bit between CUDA and the host libm.
//
// The kernels are bound by GB300's FP64 pipe (a DADD of one warp holds an SM's
// for 20 cycles), so they leave out FP64 work whose result is known exactly,
// and nothing else; every array keeps the bits of the plain expressions:
//   * divisions by grid and fluid constants through their reciprocals (exact_div);
//   * cells without DNAPL (S2 = 0, so S_e = 1): pow(1, x) = 1, kr2 = 0, and
//     the DNAPL fluxes of a cell whose neighbourhood has no DNAPL mobility;
//   * P2 = P1, as a1 leaves it: the phases' potentials are the same numbers;
//   * the Newton (k_newton): P_k and its slope again only when S2 moved, and
//     an end at a fixed point or a 2-cycle of the iteration.
// Small grids launch small blocks (eager_block): 3375 cells in blocks of 256
// would queue on 14 of the 152 SMs' FP64 pipes.
// us a call, before -> now: 100x84x61 of two media, a fifth of the cells with
// DNAPL, newton 1589 -> 358, mass 320 -> 126, props 253 -> 82, velocity 112 ->
// 47; 15^3 newton 125 -> 35, mass 31 -> 15, props 21 -> 8, velocity 20 -> 7.5.
#include <math.h>

#include <mutex>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "gbf_pair.cuh"

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ int media_at(const gbf_cells& c, size_t idx) { return c.media ? c.media[idx] : 0; }
__device__ __forceinline__ double K_at(const gbf_model& m, const gbf_cells& c, size_t idx, int md) {
  return c.K ? (double)c.K[idx] : m.K[md];
}
__device__ __forceinline__ double phi_at(const gbf_model& m, const gbf_cells& c, size_t idx, int md) {
  return c.phi ? (double)c.phi[idx] : m.m[md];
}

__device__ __forceinline__ bool same_bits(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }
// A divisor and its correctly rounded reciprocal (r = 0: divide).
struct Recip {
  double b, r;
};
Recip recip(double b) { return {b, b > 0x1p-100 && b < 0x1p100 ? 1.0 / b : 0.0}; }
__device__ __noinline__ double plain_div(double a, double b) { return a / b; }
// a / b, correctly rounded, in 5 FP64 instructions (a division takes about 10):
// the quotient by the reciprocal is within two units in the last place; a
// residual step brings it within one, and by Markstein's theorem (IBM J. Res.
// Dev. 34, 1990) the next is then correctly rounded. The residuals are exact
// away from underflow and overflow; other dividends (but zeros, over a positive
// number) are divided.
__device__ __forceinline__ double exact_div(double a, const Recip& d) {
  const unsigned e = ((unsigned)__double2hiint(a) >> 20) & 0x7ffu;
  if (e - 200u < 1600u && d.r != 0.0) {
    double q = __dmul_rn(a, d.r);
    q = __fma_rn(__fma_rn(-q, d.b, a), d.r, q);
    return __fma_rn(__fma_rn(-q, d.b, a), d.r, q);
  }
  if (gbf_is_zero(a) && (unsigned)__double2hiint(d.b) - 1u < 0x7fefffffu) return a;  // b > 0 and finite, without the FP64 unit
  return plain_div(a, d.b);
}

// Constants of a model, each by the expression (and roundings) of the plain
// kernels (the host code of this file is compiled without contraction).
struct EagerConsts {
  double e1[2], e2[2], mil[2], mil1[2];  // Brooks-Corey exponents; -1/lambda, -1/lambda - 1
  Recip om_swr[2], lam_swr[2];           // 1 - S_wr, lambda (1 - S_wr)
  double PkS1[2];                        // dP_k/dS at S_e = 1
  bool one;                              // S = 0 is S_e = 1, its P_k and slope finite, in both media (every model of use)
  double Xi1w[2];                        // Xi1 of the table's K at S_e = 1
  Recip mu1, mu2, h1, h2, h3, hh1, hh2, hh3;  // hh: 2 h
  double dtphi[2];                       // dt / phi of the table
  bool flux;                             // finite pressures have finite potentials: no zero mobility meets a NaN
};
EagerConsts eager_consts(const gbf_model& m) {
  EagerConsts C;
  C.one = true;
  for (int md = 0; md < 2; md++) {
    const double lam = m.lambda[md], swr = m.S_wr[md];
    C.e1[md] = (2. + 3. * lam) / lam;
    C.e2[md] = (2. + lam) / lam;
    C.mil[md] = (-1.) / lam;
    C.mil1[md] = ((-1.) / lam) - 1.;
    C.om_swr[md] = recip(1 - swr);
    C.lam_swr[md] = recip(lam * (1 - swr));
    C.PkS1[md] = m.P_d[md] / (lam * (1 - swr));
    C.one = C.one && (1. - swr) / (1. - swr) == 1. && isfinite(C.PkS1[md]) && isfinite(m.P_d[md]);
    C.Xi1w[md] = -1. * m.K[md] / m.mu1;
    C.dtphi[md] = m.dt / m.m[md];
  }
  C.flux = fabs(m.h1) > 0. && fabs(m.h2) > 0. && fabs(m.h3) > 0. && isfinite(m.g) && isfinite(m.kv);
  C.mu1 = recip(m.mu1);
  C.mu2 = recip(m.mu2);
  C.h1 = recip(m.h1);
  C.h2 = recip(m.h2);
  C.h3 = recip(m.h3);
  C.hh1 = recip(2. * m.h1);
  C.hh2 = recip(2. * m.h2);
  C.hh3 = recip(2. * m.h3);
  return C;
}

// The pow() calls of a block's cells, made dense: each cell that needs its
// pair of them puts two jobs on a list in shared memory, and the block's
// threads take the jobs in turn. A warp holds the FP64 pipe for a whole pow()
// however few of its lanes want one (100x84x61, a fifth of the cells with
// DNAPL: k_newton 516 -> 358 us, k_props 106 -> 82), and a small grid's block has
// twice as many threads as cells, so that a cell's two run side by side.
struct PowJobs {
  double S[kThreads], r[2][kThreads];  // S2 of a cell; its two results
  unsigned char md[kThreads];
  unsigned short list[2 * kThreads];
  int n;
};
// Every thread of the block calls it: the jobs of the threads with `need`,
// done; returns whether any thread said `any`. E[k]: the exponents of the cell's
// media; Fn(k, md, pow) is what the cell wants of its k-th pow().
template <class Fn>
__device__ __forceinline__ bool pow_jobs(PowJobs& jobs, bool any, bool need, double S2, int md, const gbf_model& m,
                                         const EagerConsts& C, const double (&E0)[2], const double (&E1)[2], Fn fn) {
  if (threadIdx.x == 0) jobs.n = 0;
  __syncthreads();
  if (need) {
    const int q = atomicAdd(&jobs.n, 2);
    jobs.S[threadIdx.x] = S2;
    jobs.md[threadIdx.x] = (unsigned char)md;
    jobs.list[q] = (unsigned short)(2 * threadIdx.x);
    jobs.list[q + 1] = (unsigned short)(2 * threadIdx.x + 1);
  }
  if (!__syncthreads_or(any)) return false;
  for (int q = threadIdx.x; q < jobs.n; q += blockDim.x) {
    const int t = jobs.list[q] >> 1, k = jobs.list[q] & 1, d = jobs.md[t];
    const double S_e = exact_div(1. - jobs.S[t] - m.S_wr[d], C.om_swr[d]);
    jobs.r[k][t] = fn(k, d, S_e, pow(S_e, k ? E1[d] : E0[d]));
  }
  __syncthreads();
  return true;
}

// a1 (cpu.cpp:57-74): every cell; blocks of `per` cells.
__global__ void k_props(const gbf_model m, const EagerConsts C, gbf_arrays a, gbf_cells cells, unsigned per) {
  __shared__ PowJobs jobs;
  const GbfGeo g = gbf_geo(m);
  for (size_t b = (size_t)blockIdx.x * per; b < g.n; b += (size_t)gridDim.x * per) {
    const size_t c = b + threadIdx.x;
    const bool mine = threadIdx.x < per && c < g.n;
    int md = 0;
    double S2 = 0., P1 = 0.;
    if (mine) {
      md = media_at(cells, c);
      S2 = a.S2[c];
      P1 = a.P1[c];
    }
    const bool wet = mine && !(gbf_is_zero(S2) && C.one);
    const bool some = pow_jobs(jobs, wet, wet, S2, md, m, C, C.e1, C.e2, [](int k, int, double S_e, double p) {
      return k ? (1. - S_e) * (1. - S_e) * (1 - p) : p;
    });
    if (mine) {
      const double P2 = P1 + 0.0;
      double Xi1, Xi2;
      if (!some || !wet) {  // S_e = (1 - S_wr) / (1 - S_wr) = 1: kr1 = 1, kr2 = 0
        Xi1 = cells.K ? exact_div(-(double)cells.K[c], C.mu1) : C.Xi1w[md];
        Xi2 = -0.0;
      } else {
        const double K = K_at(m, cells, c, md);
        Xi1 = exact_div(-1. * K * jobs.r[0][threadIdx.x], C.mu1);
        Xi2 = exact_div(-1. * K * jobs.r[1][threadIdx.x], C.mu2);
      }
      a.P2[c] = P2;
      a.Xi1[c] = Xi1;
      a.Xi2[c] = Xi2;
      a.ro1[c] = m.ro01 * (1. + (m.beta1) * (P1 - m.P_atm));
      a.ro2[c] = m.ro02 * (1. + (m.beta2) * (P2 - m.P_atm));
    }
    __syncthreads();  // the jobs' arrays, before the next cells'
  }
}

// One direction of a2 (cpu.cpp:77-160): both phases' pressure gradients at a
// cell, one-sided on the faces (lo: c is the direction's first cell, hi: its
// last); P2's is P1's where its values are.
struct Grad {
  double g1, g2;
};
__device__ __forceinline__ Grad eager_gradient(const double* P1, const double* P2, size_t c, size_t st, bool lo, bool hi,
                                               const Recip& h, const Recip& hh) {
  const size_t p = hi ? c : c + st, q = lo ? c : c - st;
  const double a1 = P1[p], b1 = P1[q], a2 = P2[p], b2 = P2[q];
  const Recip& d = lo || hi ? h : hh;
  Grad r;
  r.g1 = exact_div(a1 - b1, d);
  r.g2 = r.g1;
  if (!same_bits(a1, a2) || !same_bits(b1, b2)) r.g2 = plain_div(a2 - b2, d.b);
  return r;
}

// a2 (cpu.cpp:77-160): every cell; one-sided differences on the faces, where
// the mobility multiplies the difference before the division.
__global__ void k_velocity(const gbf_model m, const EagerConsts C, gbf_arrays a) {
  const GbfGeo g = gbf_geo(m);
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < g.n; c += (size_t)gridDim.x * blockDim.x) {
    const unsigned q = (unsigned)c / (unsigned)g.nx;
    const int i = (int)((unsigned)c - q * (unsigned)g.nx), k = (int)(q / (unsigned)g.ny), j = (int)(q - (unsigned)k * (unsigned)g.ny);
    const double Xi1 = a.Xi1[c], Xi2 = a.Xi2[c];
    const bool x = i == 0 || i == g.nx - 1, z = k == 0 || k == g.nz - 1;
    if (x) {
      const size_t p = i == 0 ? c + 1 : c, r = i == 0 ? c : c - 1;
      a.u1x[c] = exact_div(Xi1 * (a.P1[p] - a.P1[r]), C.h1);
      a.u2x[c] = exact_div(Xi2 * (a.P2[p] - a.P2[r]), C.h1);
    } else {
      const Grad d = eager_gradient(a.P1, a.P2, c, 1, false, false, C.h1, C.hh1);
      a.u1x[c] = Xi1 * d.g1;
      a.u2x[c] = Xi2 * d.g2;
    }
    {
      const double kX1 = m.kv * Xi1, kX2 = m.kv * Xi2;
      const Grad d = eager_gradient(a.P1, a.P2, c, (size_t)g.nx, j == 0, j == g.ny - 1, C.h2, C.hh2);
      a.u1y[c] = kX1 * (d.g1 - a.ro1[c] * m.g);
      a.u2y[c] = kX2 * (d.g2 - a.ro2[c] * m.g);
    }
    if (z) {
      const size_t p = k == 0 ? c + g.pl : c, r = k == 0 ? c : c - g.pl;
      a.u1z[c] = exact_div(Xi1 * (a.P1[p] - a.P1[r]), C.h3);
      a.u2z[c] = exact_div(Xi2 * (a.P2[p] - a.P2[r]), C.h3);
    } else {
      const Grad d = eager_gradient(a.P1, a.P2, c, g.pl, false, false, C.h3, C.hh3);
      a.u1z[c] = Xi1 * d.g1;
      a.u2z[c] = Xi2 * d.g2;
    }
  }
}

// Donor-cell divergence of one direction (cpu.cpp:260-262), reference order.
__device__ __noinline__ double plain_upwind(double x1, double x2, double Xc, double rc, double Xm, double rm, double Xp,
                                            double rp, double h) {
  return (((x2 + fabs(x2)) / 2.0 - (x1 - fabs(x1)) / 2.0) * (-1) * Xc * rc - (x1 + fabs(x1)) / 2.0 * (-1) * Xm * rm +
          (x2 - fabs(x2)) / 2.0 * (-1) * Xp * rp) / h;
}
__device__ __forceinline__ double upwind_div(double x1, double x2, double Xc, double rc, double Xm, double rm,
                                             double Xp, double rp, const Recip& h) {
  if (!gbf_is_finite(x1) || !gbf_is_finite(x2)) return plain_upwind(x1, x2, Xc, rc, Xm, rm, Xp, rp, h.b);
  // (x + |x|) / 2 and (x - |x|) / 2 of a finite x are x or +0, by its sign bit (-0: +0 and -0)
  const bool n1 = __double2hiint(x1) < 0, n2 = __double2hiint(x2) < 0;
  const double p1 = n1 ? 0. : x1, m1 = n1 ? x1 : 0., p2 = n2 ? 0. : x2, m2 = n2 ? x2 : 0.;
  return exact_div(-(p2 - m1) * Xc * rc - -p1 * Xm * rm + -m2 * Xp * rp, h);
}

__device__ __forceinline__ void interior_cell(const GbfGeo& g, size_t t, int& i, int& j, int& k) {
  const unsigned ix = (unsigned)g.nx - 2, iy = (unsigned)g.ny - 2, q = (unsigned)t / ix, r = q / iy;
  i = 1 + (int)((unsigned)t - q * ix);
  j = 1 + (int)(q - r * iy);
  k = 1 + (int)r;
}

// The face potentials of a phase at cell c, and its divergence (cpu.cpp:236-262).
struct Faces {
  double x1, x2, y1, y2, z1, z2;  // without gravity
};
__device__ __forceinline__ Faces eager_faces(const double* P, size_t c, size_t nx, size_t pl, const EagerConsts& C) {
  const double p = P[c];
  Faces f;
  f.z2 = exact_div(-(P[c + pl] - p), C.h3);
  f.z1 = exact_div(-(p - P[c - pl]), C.h3);
  f.x2 = exact_div(-(P[c + 1] - p), C.h1);
  f.x1 = exact_div(-(p - P[c - 1]), C.h1);
  f.y2 = exact_div(-(P[c + nx] - p), C.h2);
  f.y1 = exact_div(-(p - P[c - nx]), C.h2);
  return f;
}
__device__ __forceinline__ double eager_divergence(const gbf_model& m, const EagerConsts& C, const Faces& f, bool closed,
                                                   const double* Xi, const double* ro, size_t c, size_t nx, size_t pl) {
  const double X = Xi[c], r = ro[c];
  const double y2 = closed ? 0 : f.y2 + r * m.g, y1 = f.y1 + r * m.g;
  const double f3 = upwind_div(f.z1, f.z2, X, r, Xi[c - pl], ro[c - pl], Xi[c + pl], ro[c + pl], C.h3);
  const double f1 = upwind_div(f.x1, f.x2, X, r, Xi[c - 1], ro[c - 1], Xi[c + 1], ro[c + 1], C.h1);
  const double f2 = m.kv * upwind_div(y1, y2, X, r, Xi[c - nx], ro[c - nx], Xi[c + nx], ro[c + nx], C.h2);
  return f1 + f2 + f3;
}
// The DNAPL divergence of a cell that has some around it (a call, so that its
// FP64 instructions are not issued predicated off for the other cells).
__device__ __noinline__ double eager_divergence2(const gbf_model& m, const EagerConsts& C, const gbf_arrays& a, Faces f,
                                                 bool same, bool closed, size_t c, size_t nx, size_t pl) {
  if (!same) f = eager_faces(a.P2, c, nx, pl, C);
  return eager_divergence(m, C, f, closed, a.Xi2, a.ro2, c, nx, pl);
}

// a3 (cpu.cpp:218-291): interior cells.
__global__ void k_mass(const gbf_model m, const EagerConsts C, gbf_arrays a, gbf_cells cells) {
  const GbfGeo g = gbf_geo(m);
  const size_t nint = (size_t)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  const bool noflow_bottom = (m.bc_mode == GBF_BC_HYDROSTATIC_SIDES);
  const double src = (m.source_mode == GBF_SOURCE_RATE && m.rate_cells > 0)
                         ? m.rate / (double)(m.rate_cells * m.rate_cells) / (m.h1 * m.h2 * m.h3)
                         : 0.0;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nint; t += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    interior_cell(g, t, i, j, k);
    const size_t c = gbf_idx(g, i, j, k), pl = g.pl, nx = g.nx;
    const size_t nb[7] = {c, c - 1, c + 1, c - nx, c + nx, c - pl, c + pl};
    const double roS1 = a.ro1[c] * (1 - a.S2[c]);
    const double roS2 = a.ro2[c] * a.S2[c];
    const bool closed = noflow_bottom && j == g.ny - 2;
    // P2 equal to P1 at the seven cells; DNAPL immobile there, and every number that its zero mobility multiplies finite
    bool same = true, still = C.flux;
#pragma unroll
    for (int q = 0; q < 7; q++) {
      const double p2 = a.P2[nb[q]];
      same = same && same_bits(p2, a.P1[nb[q]]);
      still = still && gbf_is_zero(a.Xi2[nb[q]]) && gbf_is_finite(p2) && gbf_is_finite(a.ro2[nb[q]]);
    }
    const Faces f = eager_faces(a.P1, c, nx, pl, C);
    const double f1 = eager_divergence(m, C, f, closed, a.Xi1, a.ro1, c, nx, pl);
    const double dtphi = cells.phi ? plain_div(m.dt, (double)cells.phi[c]) : C.dtphi[media_at(cells, c)];
    double A1 = roS1 - dtphi * f1, A2;
    const bool in_src = src != 0.0 && j == 1 && gbf_in_rate_patch(m, i, k);
    // roS2 - dtphi (+-0): roS2 itself, but for roS2 = -0
    if (still && !in_src && __double_as_longlong(roS2) != (long long)0x8000000000000000ull && gbf_is_finite(dtphi)) {
      A2 = roS2;
    } else {
      const double gsum = eager_divergence2(m, C, a, f, same, closed, c, nx, pl);
      A2 = in_src ? roS2 - dtphi * (gsum - src) : roS2 - dtphi * gsum;
    }
    a.roS1_old[c] = roS1;
    a.roS2_old[c] = roS2;
    a.roS1[c] = A1;
    a.roS2[c] = A2;
  }
}

// a4 (cpu.cpp:293-320): interior cells, in place; blocks of `per` cells. The
// iteration is a map of (P1, S2) with everything else fixed: once it returns
// the point it was given every later iteration does, and once it returns the
// point before, the later ones alternate between the two, so the last one's
// result is known. (Rounding leaves nearly every cell at one or the other
// after 2 to 5 of the reference's 7 iterations.)
__global__ void k_newton(const gbf_model m, const EagerConsts C, gbf_arrays a, gbf_cells cells, unsigned per) {
  __shared__ PowJobs jobs;
  const GbfGeo g = gbf_geo(m);
  const size_t nint = (size_t)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  const bool tol = m.newton_tol > 0;
  const int N = m.newton_iterations;
  for (size_t b = (size_t)blockIdx.x * per; b < nint; b += (size_t)gridDim.x * per) {
    const size_t t = b + threadIdx.x;
    const bool mine = threadIdx.x < per && t < nint;
    size_t c = 0;
    int md = 0;
    double roS1 = 0., roS2 = 0., P1 = 0., S2 = 0.;
    if (mine) {
      int i, j, k;
      interior_cell(g, t, i, j, k);
      c = gbf_idx(g, i, j, k);
      md = media_at(cells, c);
      roS1 = a.roS1[c];
      roS2 = a.roS2[c];
      P1 = a.P1[c];
      S2 = a.S2[c];
    }
    bool active = mine;
    const double pd = m.P_d[md];
    // Without DNAPL (S2 = 0, roS2 = 0) every product with S2 is zero, dS too,
    // and the step in P1 is the one of the general form with those zeros left out.
    if (mine && C.one && gbf_is_zero(S2) && gbf_is_zero(roS2) && gbf_is_finite(P1) && gbf_is_finite(roS1) && !tol) {
      const double F1P = m.ro01 * (m.beta1);
      double Pb = P1;
      for (int w = 1; w <= N; w++) {
        const double F1 = m.ro01 * (1. + (m.beta1) * (P1 - m.P_atm)) - roS1;
        const double F2S = m.ro02 * (1 + (m.beta2) * (P1 + pd - m.P_atm));
        const double Pn = P1 - 1 / (F1P * F2S) * (F2S * F1);
        const bool fixed = same_bits(Pn, P1), cycle = w > 1 && same_bits(Pn, Pb);
        Pb = P1;
        P1 = Pn;
        if (fixed) break;
        if (cycle) {
          if ((N - w) & 1) P1 = Pb;
          break;
        }
      }
      S2 = 0.;
      active = false;
    }
    double Pb = P1, Sb = S2, Sk = 0., P_k = 0., SPkS = 0., omS = 0., F1P = 0., F2P = 0.;  // b: the point before
    for (int w = 1; w <= N; w++) {
      const bool moved = active && (w == 1 || !same_bits(S2, Sk)), wet = moved && !(gbf_is_zero(S2) && C.one);
      // P_k and dP_k/dS where S2 moved (at S_e = 1 without pow)
      if (!pow_jobs(jobs, active, wet, S2, md, m, C, C.mil, C.mil1, [&](int k, int d, double, double p) {
            const double v = m.P_d[d] * p;
            return k ? exact_div(v, C.lam_swr[d]) : v;
          }))
        break;
      if (active) {
        if (moved) {
          Sk = S2;
          P_k = wet ? jobs.r[0][threadIdx.x] : pd;
          SPkS = S2 * (wet ? jobs.r[1][threadIdx.x] : C.PkS1[md]);
          omS = 1. - S2;
          F1P = m.ro01 * (m.beta1) * omS;
          F2P = m.ro02 * (m.beta2) * S2;
        }
        const double r1 = m.ro01 * (1. + (m.beta1) * (P1 - m.P_atm));
        const double pk = P1 + P_k - m.P_atm;
        const double F1 = r1 * omS - roS1;
        const double F2 = m.ro02 * (1. + (m.beta2) * pk) * S2 - roS2;
        const double F1S = -r1;
        const double F2S = m.ro02 * (1 + (m.beta2) * (pk + SPkS));
        const double det = F1P * F2S - F1S * F2P;
        const double inv = 1 / det;
        const double dP = inv * (F2S * F1 - F1S * F2);
        const double dS = inv * (F1P * F2 - F2P * F1);
        const double Pn = P1 - dP, Sn = S2 - dS;
        const bool fixed = same_bits(Pn, P1) && same_bits(Sn, S2);
        const bool cycle = w > 1 && same_bits(Pn, Pb) && same_bits(Sn, Sb);
        Pb = P1;
        Sb = S2;
        P1 = Pn;
        S2 = Sn;
        if (tol && fabs(dS) <= m.newton_tol && fabs(dP) <= m.newton_tol * fabs(P1)) {
          active = false;
        } else if (fixed) {
          active = false;
        } else if (cycle) {
          if ((N - w) & 1) {
            P1 = Pb;
            S2 = Sb;
          }
          active = false;
        }
      }
    }
    if (mine) {
      a.P1[c] = P1;
      a.S2[c] = S2;
    }
    __syncthreads();  // the jobs' arrays, before the next cells'
  }
}

// a5, pass 1: the value the reference's sweep leaves at every boundary cell,
// into scratch[0 .. nb) (S2) and scratch[nb .. 2nb) (P1). Reads only.
__global__ void __launch_bounds__(kThreads) k_boundary_gather(const gbf_model m, gbf_arrays a, double* scratch) {
  const GbfGeo g = gbf_geo(m);
  const size_t nb = gbf_boundary_count(g);
  const double* ro1 = a.ro1;
  auto ro1_top = [ro1, &g](int i) { return ro1[(size_t)i + (size_t)g.nx]; };
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nb; t += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    gbf_boundary_cell(g, t, i, j, k);
    scratch[t] = gbf_sweep_S<double>(m, g, a.S2, a.S2, i, j, k);
    scratch[nb + t] = gbf_sweep_P<double>(m, g, a.P1, a.P1, i, j, k, ro1_top);
  }
}

// a5, pass 2: scatter.
__global__ void __launch_bounds__(kThreads) k_boundary_scatter(const gbf_model m, gbf_arrays a, const double* scratch) {
  const GbfGeo g = gbf_geo(m);
  const size_t nb = gbf_boundary_count(g);
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nb; t += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    gbf_boundary_cell(g, t, i, j, k);
    size_t c = gbf_idx(g, i, j, k);
    a.S2[c] = scratch[t];
    a.P1[c] = scratch[nb + t];
  }
}

// Scratch of gbf_boundary_f64_noalloc: a fixed array of this library in
// device memory, 8 MiB, held by every GPU that loads the library until the
// process exits. In host code the name is only a stand-in for the array, not
// its device address: host code passes the address that
// cudaGetSymbolAddress returns for the current device (noalloc_scratch).
constexpr size_t kNoAllocScratchDoubles = (size_t)1 << 20;
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocScratchDoubles];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
// Per device: the array's address and the id of the CUDA context it was looked
// up in. A context that is destroyed (cudaDeviceReset, a reset of the primary
// context) and created again may load the library's module elsewhere, so the
// address is valid only while the context it came from is current.
double* g_noalloc_ptr[kNoAllocMaxDevices] = {};
unsigned long long g_noalloc_ctx[kNoAllocMaxDevices] = {};
PFN_cuCtxGetCurrent_v4000 g_ctx_current = nullptr;
PFN_cuCtxGetId_v12000 g_ctx_id = nullptr;
bool g_ctx_queries_resolved = false;

// Id of the calling thread's current CUDA context (cuCtxGetId: unique for the
// life of the process), or 0 when no context is current or the driver cannot
// tell. The driver functions are reached through the runtime's entry-point
// query, so libgbflow does not link libcuda. Called with g_noalloc_mu held.
unsigned long long current_context_id() {
  if (!g_ctx_queries_resolved) {
    g_ctx_queries_resolved = true;
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 4000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      g_ctx_current = (PFN_cuCtxGetCurrent_v4000)f;
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      g_ctx_id = (PFN_cuCtxGetId_v12000)f;
  }
  if (!g_ctx_current || !g_ctx_id) return 0;
  CUcontext c = nullptr;
  if (g_ctx_current(&c) != CUDA_SUCCESS || !c) return 0;
  unsigned long long id = 0;
  return g_ctx_id(c, &id) == CUDA_SUCCESS ? id : 0;
}

// Device address of g_noalloc_scratch on the current device, looked up with
// that device current (cudaGetSymbolAddress) on the first call, and again
// whenever the current context is not the one the address came from (or
// cannot be identified); otherwise the cached address.
int noalloc_scratch(double** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return gbf_cuda_check(e, "gbf_boundary_f64_noalloc: cudaGetDevice");
  if (dev < 0 || dev >= kNoAllocMaxDevices) return gbf_fail(GBF_ERR_ARG, "gbf_boundary_f64_noalloc: device index");
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  const unsigned long long ctx = current_context_id();
  if (!g_noalloc_ptr[dev] || ctx == 0 || ctx != g_noalloc_ctx[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) return gbf_cuda_check(e != cudaSuccess ? e : cudaErrorInvalidSymbol,
                                                      "gbf_boundary_f64_noalloc: cudaGetSymbolAddress");
    g_noalloc_ptr[dev] = (double*)p;
    g_noalloc_ctx[dev] = current_context_id();  // the lookup made a context current if none was
  }
  *out = g_noalloc_ptr[dev];
  return GBF_OK;
}

// Block size of an FP64-bound kernel over n cells: 256, or what spreads a
// small grid over every SM.
int eager_block(size_t n) {
  const size_t per = (n + (size_t)gbf_num_sms() - 1) / (size_t)gbf_num_sms();
  return per >= (size_t)kThreads ? kThreads : (int)((per + 31) / 32 * 32);
}

int check_model(const gbf_model* m, const char* where) {
  if (!m || m->nx < 3 || m->ny < 3 || m->nz < 3) return gbf_fail(GBF_ERR_ARG, where);
  return GBF_OK;
}

int launched(const char* where) {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GBF_OK : gbf_cuda_check(e, where);
}

// Start-of-step phase masses of interior cells from a state (P, S): what
// assign_rS_nr leaves in roS1_old, roS2_old (cpu.cpp:222-225, 286-287) with
// the densities of assign_ro1_ro2 at P2 = P1 (cpu.cpp:63-74). FP64 state, or
// the split state (dP from the hydrostatic profile, S in FP32) when P is NULL.
// Boundary cells get 0.
__global__ void __launch_bounds__(kThreads) k_roS_old(const gbf_model m, const double* P, const double* S,
                                                      const float* dPf, const float* Sf, int px, double* o1,
                                                      double* o2) {
  const GbfGeo g = gbf_geo(m);
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < g.n; c += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(c % g.nx), j = (int)((c / g.nx) % g.ny), k = (int)(c / g.pl);
    if (gbf_is_boundary(g, i, j, k)) {
      o1[c] = 0.;
      o2[c] = 0.;
      continue;
    }
    const size_t q = c + (size_t)(px - g.nx) * ((size_t)j + (size_t)k * g.ny);  // the split state's rows are px apart
    const double p = P ? P[c] : gbf_p_hydrostatic(m, j) + (double)dPf[q];
    const double s = S ? S[c] : (double)Sf[q];
    const double ro1 = m.ro01 * (1. + (m.beta1) * (p - m.P_atm));
    const double ro2 = m.ro02 * (1. + (m.beta2) * (p - m.P_atm));
    o1[c] = ro1 * (1 - s);
    o2[c] = ro2 * s;
  }
}

}  // namespace

int gbf_roS_old_launch(const gbf_model& m, const double* P, const double* S, const float* dPf, const float* Sf, int px,
                       double* o1, double* o2, cudaStream_t st) {
  k_roS_old<<<gbf_grid_for(gbf_geo(m).n, kThreads), kThreads, 0, st>>>(m, P, S, dPf, Sf, px, o1, o2);
  GBF_CUDA(cudaGetLastError());
  return GBF_OK;
}

extern "C" {

int gbf_props_f64(const gbf_model* m, gbf_arrays a, gbf_cells cells, void* stream) {
  if (int s = check_model(m, "gbf_props_f64")) return s;
  const size_t n = gbf_geo(*m).n;
  const int b = eager_block(n), threads = b <= kThreads / 2 ? 2 * b : kThreads;
  k_props<<<gbf_grid_for(n, b), threads, 0, (cudaStream_t)stream>>>(*m, eager_consts(*m), a, cells, (unsigned)b);
  return launched("gbf_props_f64");
}

int gbf_velocity_f64(const gbf_model* m, gbf_arrays a, void* stream) {
  if (int s = check_model(m, "gbf_velocity_f64")) return s;
  const size_t n = gbf_geo(*m).n;
  const int b = eager_block(n);
  k_velocity<<<gbf_grid_for(n, b), b, 0, (cudaStream_t)stream>>>(*m, eager_consts(*m), a);
  return launched("gbf_velocity_f64");
}

int gbf_mass_f64(const gbf_model* m, gbf_arrays a, gbf_cells cells, void* stream) {
  if (int s = check_model(m, "gbf_mass_f64")) return s;
  size_t nint = (size_t)(m->nx - 2) * (m->ny - 2) * (m->nz - 2);
  const int b = eager_block(nint);
  k_mass<<<gbf_grid_for(nint, b), b, 0, (cudaStream_t)stream>>>(*m, eager_consts(*m), a, cells);
  return launched("gbf_mass_f64");
}

int gbf_newton_f64(const gbf_model* m, gbf_arrays a, gbf_cells cells, void* stream) {
  if (int s = check_model(m, "gbf_newton_f64")) return s;
  size_t nint = (size_t)(m->nx - 2) * (m->ny - 2) * (m->nz - 2);
  const int b = eager_block(nint), threads = b <= kThreads / 2 ? 2 * b : kThreads;
  k_newton<<<gbf_grid_for(nint, b), threads, 0, (cudaStream_t)stream>>>(*m, eager_consts(*m), a, cells, (unsigned)b);
  return launched("gbf_newton_f64");
}

size_t gbf_boundary_scratch_doubles(const gbf_model* m) {
  if (!m || m->nx < 3 || m->ny < 3 || m->nz < 3) return 0;
  return 2 * gbf_boundary_count(gbf_geo(*m));
}

int gbf_boundary_f64(const gbf_model* m, gbf_arrays a, double* scratch, void* stream) {
  if (int s = check_model(m, "gbf_boundary_f64")) return s;
  if (!scratch) return gbf_fail(GBF_ERR_ARG, "gbf_boundary_f64: scratch");
  size_t nb = gbf_boundary_count(gbf_geo(*m));
  unsigned grid = gbf_grid_for(nb, kThreads);
  k_boundary_gather<<<grid, kThreads, 0, (cudaStream_t)stream>>>(*m, a, scratch);
  k_boundary_scatter<<<grid, kThreads, 0, (cudaStream_t)stream>>>(*m, a, scratch);
  return launched("gbf_boundary_f64");
}

// The boundary pass for callers that cannot allocate device memory when they
// apply the boundary conditions. Same kernels and results as
// gbf_boundary_f64; the gather scratch is the library's fixed device array
// g_noalloc_scratch instead of a caller buffer. Allocates nothing: no
// cudaMalloc, cudaFree or allocating library routine. The first call on a
// device looks up the array's address there (cudaGetSymbolAddress), and so
// does the first call after that device's context was destroyed and created
// again, so make those calls before any stream capture. Every call on a device uses the
// same array, which keeps the last call's contents: the gather fills every
// slot the scatter reads, so nothing needs clearing, and calls that overlap
// on the same GPU (from several streams or host threads) race on it.
int gbf_boundary_f64_noalloc(const gbf_model* m, gbf_arrays a, void* stream) {
  if (int s = check_model(m, "gbf_boundary_f64_noalloc")) return s;
  const size_t nb = gbf_boundary_count(gbf_geo(*m));
  if (2 * nb > kNoAllocScratchDoubles)
    return gbf_fail(GBF_ERR_ARG, "gbf_boundary_f64_noalloc: more than 524288 boundary cells (its fixed 8 MiB "
                                 "scratch holds 2 doubles per boundary cell); use gbf_boundary_f64");
  double* scratch = nullptr;
  if (int s = noalloc_scratch(&scratch)) return s;
  const unsigned grid = gbf_grid_for(nb, kThreads);
  k_boundary_gather<<<grid, kThreads, 0, (cudaStream_t)stream>>>(*m, a, scratch);
  k_boundary_scatter<<<grid, kThreads, 0, (cudaStream_t)stream>>>(*m, a, scratch);
  return launched("gbf_boundary_f64_noalloc");
}

}  // extern "C"
