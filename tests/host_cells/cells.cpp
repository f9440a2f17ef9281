// cells.cpp — per-cell device code of the FP64 step, compiled for the CPU.
#include "cuda_on_host.h"

#include "gbf_pair.cuh"

extern "C" {

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
