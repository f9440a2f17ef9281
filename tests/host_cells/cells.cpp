// cells.cpp — the per-cell device code of the FP64 step, compiled for the CPU
// and driven as the kernels drive it: pass 1 over every cell, pass 2 over the
// interior, the face pass.
#include "cuda_on_host.h"

#include <vector>

#include "gbf_f64_cell.cuh"
static long g_fp64_cells;  // cells that the pair step gave to FP64
#define GBF_COUNT_FP64_CELL g_fp64_cells++
#include "gbf_f64_pair.cuh"

namespace {
void faces(const gbf_model& m, const GbfGeo& g, const GbfF64Step& s) {
  for (size_t t = 0; t < gbf_boundary_count(g); t++) gbf_f64_boundary_cell(m, s, g, t);
}
}  // namespace

extern "C" {

// The number of such cells since the last call.
long host_fp64_cells(void) {
  const long n = g_fp64_cells;
  g_fp64_cells = 0;
  return n;
}
int host_pair_applies(const gbf_model* m) { return gbf_pair_applies(*m); }

// `steps` steps of (P, S) in place by the pair step (pair) or the plain FP64
// passes; masses[steps][2]. Returns the status bits.
unsigned host_f64_steps(const gbf_model* mp, const int* media, const float* K, const float* phi, double* P, double* S,
                        int steps, int pair, double* masses) {
  const gbf_model m = *mp;
  const GbfGeo g = gbf_geo(m);
  const GbfDerived d = gbf_derive(m);
  const gbf_cells cells = {media, K, phi};
  const size_t n = g.n;
  std::vector<double> Pn(P, P + n), Sn(S, S + n), work(pair ? 0 : 5 * n);
  std::vector<float2> pw(pair ? 4 * n : 0);
  std::vector<GbfPairRow> rows;
  for (int j = 0; j < m.ny; j++) rows.push_back(gbf_pair_row(m, j));
  const GbfPairConsts C = gbf_pair_consts(m);
  GbfPairWork w = {};
  w.D = pw.data();
  w.L1 = w.D + n;
  w.L2 = w.L1 + n;
  w.Pk = w.L2 + n;
  w.rows = rows.data();
  unsigned bad = 0;
  for (int q = 0; q < steps; q++) {
    GbfF64Step s = {};
    s.P = P;
    s.S = S;
    s.Pn = Pn.data();
    s.Sn = Sn.data();
    s.status = &bad;
    double m1 = 0., m2 = 0.;
    if (pair) {
      for (unsigned c = 0; c < n; c++) gbf_pair_props_cell<false>(C, cells, s, w, c);
    } else {
      s.L1 = work.data();
      s.L2 = s.L1 + n;
      s.ro1 = s.L2 + n;
      s.ro2 = s.ro1 + n;
      s.lnSe = s.ro2 + n;
      for (size_t c = 0; c < n; c++) gbf_f64_props_cell(m, d, cells, s, 0, g, c);
    }
    if (pair) {
      for (unsigned t = 0; t < 64; t++) {  // as 64 threads
        GbfPairMass acc;
        gbf_pair_step_cells<true>(C, m, d, cells, s, w, t, 64, C.nint, acc);
        m1 += acc.m1 - pf_to_double(acc.r1);
        m2 += acc.m2;
      }
    } else {
      for (int k = 1; k < m.nz - 1; k++)
        for (int j = 1; j < m.ny - 1; j++)
          for (int i = 1; i < m.nx - 1; i++) gbf_f64_flux_newton_cell(m, d, cells, s, g, i, j, k, m1, m2, bad);
    }
    faces(m, g, s);
    masses[2 * q] = m1 * d.V;
    masses[2 * q + 1] = m2 * d.V;
    memcpy(P, Pn.data(), n * sizeof(double));
    memcpy(S, Sn.data(), n * sizeof(double));
  }
  return bad;
}

// The table-driven functions at x[0, n): ln(1 - x), 2^x, 1 - 2^x, 2^x as a pair (hi + lo).
void host_pair_functions(int n, const double* x, double* ln1m, double* exp2_, double* om_exp2, double* exp2_pair) {
  for (int q = 0; q < n; q++) {
    const GbfPf p = pf_from_double(x[q]);
    if (ln1m) ln1m[q] = gbf_ln1m(x[q], p.h);
    if (exp2_) exp2_[q] = gbf_exp2(x[q], p.h);
    if (om_exp2) om_exp2[q] = gbf_one_minus_exp2(x[q], p.h);
    if (exp2_pair) {
      const GbfPf e = pf_exp2(p);
      exp2_pair[q] = (double)e.h + (double)e.l;
    }
  }
}
}
