// gbf_f64.cu — FP64 step of one domain: two passes plus a face pass.
//
// GB300 executes FP64 at about 1/58 of its FP32 rate (measured 1.2 TFLOP/s
// DFMA against 6.7 TB/s of HBM): any step whose arithmetic is FP64 is bound
// by that pipe (measured 8.73 ms a step at 256^3: 85% of it active, DRAM at
// 4%). The step therefore forms its increments in FP32 pairs
// (gbf_f64_pair.cuh) and takes the FP64 pipe 6 warp instructions per 32 cells
// without DNAPL (with phase masses), about 25 with:
//   pass 1 (k_pair_props, every cell): pressure against the row's hydrostatic
//     value, mobility x density of both phases, capillary pressure, as pairs
//     (32 bytes a cell written, 24 without DNAPL);
//   pass 2 (k_pair_step, interior cells): upwinded face fluxes with gravity
//     (cpu.cpp:218-291) and the 2x2 Newton (cpu.cpp:293-320) in increments,
//     the next FP64 state (ping-pong), phase-mass partial sums on request.
// Two passes, not one tile: a cell's properties cost half of its fluxes and
// Newton, so they are not computed again for halos, and the 64 bytes a cell
// that this moves beside the state are hidden behind the arithmetic. Both are
// bound by instruction issue, with the FP64 pipe about half busy; 256^3,
// heterogeneous, a fifth of the cells with DNAPL: pass 1 201 us (223 with the
// DNAPL mobility formed and P_k stored in every cell), pass 2 470 us (3.7 and
// 2.2 TB/s of 44 and 62 bytes a cell; 447 without the looks for cells that
// pairs do not hold), where the FP64 passes took 2460 and
// 6270. Pass 1 keeps to 32 registers for eight blocks an SM: at 40 it takes 226
// us, and on small grids fewer blocks of the next kernel fit beside it (40
// steps of 40^3 778 -> 881 us). Pass 2 takes 64 registers for four blocks an SM:
// at three (80 registers) its latencies show, 808 us; at five and six it spills
// (627, 764).
//   face pass (k_f64_boundary): the reference's sweep-ordered boundary
//     values (cpu.cpp:44-54, 323-403) into the next state.
// A model with fewer Newton iterations than the reference's 7, whose iterates
// stop before convergence, and one whose constants do not fit FP32 pairs run the
// plain FP64 passes (k_f64_props, k_f64_flux_newton; per-cell code in
// gbf_f64_cell.cuh).
#include "gbf_f64_cell.cuh"
#include "gbf_f64_pair.cuh"

namespace {

constexpr int kThreads = 256;

__global__ void __launch_bounds__(kThreads) k_f64_props(const gbf_model m, const GbfDerived d, const gbf_cells cells,
                                                        const GbfF64Step s, const int flags) {
  gbf_pdl_begin();
  const GbfGeo g = gbf_geo(m);
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < g.n; c += (size_t)gridDim.x * blockDim.x)
    gbf_f64_props_cell(m, d, cells, s, flags, g, c);
}

__global__ void __launch_bounds__(kThreads) k_f64_flux_newton(const gbf_model m, const GbfDerived d,
                                                              const gbf_cells cells, const GbfF64Step s) {
  gbf_pdl_begin();
  const GbfGeo g = gbf_geo(m);
  const size_t ix = (size_t)g.nx - 2, iy = (size_t)g.ny - 2;
  const size_t nint = ix * iy * (size_t)(g.nz - 2);
  double msum1 = 0., msum2 = 0.;
  unsigned bad = 0;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nint; t += (size_t)gridDim.x * blockDim.x) {
    const int i = 1 + (int)(t % ix), j = 1 + (int)((t / ix) % iy), k = 1 + (int)(t / (ix * iy));
    gbf_f64_flux_newton_cell(m, d, cells, s, g, i, j, k, msum1, msum2, bad);
  }
  if (bad) atomicOr(s.status, GBF_DEV_NONFINITE);
  if (s.mass_partials) gbf_block_sum2<kThreads>(msum1, msum2, d.V, s.mass_partials + 2 * blockIdx.x);
}

template <bool DROPIN>
__global__ void __launch_bounds__(kThreads, 8) k_pair_props(const GbfPairConsts C, const gbf_cells cells,
                                                         const GbfF64Step s, const GbfPairWork w) {
  gbf_pdl_begin();
  for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c < C.n; c += gridDim.x * blockDim.x)
    gbf_pair_props_cell<DROPIN>(C, cells, s, w, c);
}

template <bool MASS, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_pair_step(const __grid_constant__ GbfPairConsts C,
                                                          const __grid_constant__ gbf_model m,
                                                          const __grid_constant__ GbfDerived d,
                                                          const __grid_constant__ gbf_cells cells,
                                                          const __grid_constant__ GbfF64Step s,
                                                          const __grid_constant__ GbfPairWork w) {
  gbf_pdl_begin();
  GbfPairMass acc;
  gbf_pair_step_cells<MASS>(C, m, d, cells, s, w, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, C.nint, acc);
  if (MASS) gbf_block_sum2<NT>(acc.m1 - pf_to_double(acc.r1), acc.m2, d.V, s.mass_partials + 2 * blockIdx.x);
}

__global__ void __launch_bounds__(kThreads) k_density(double ro0, double beta, double Patm, const double* P,
                                                      double* out, size_t n) {
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x)
    out[c] = ro0 * (1. + beta * (P[c] - Patm));
}

__global__ void k_pair_rows(const gbf_model m, GbfPairRow* rows) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < m.ny; j += gridDim.x * blockDim.x) rows[j] = gbf_pair_row(m, j);
}

__global__ void __launch_bounds__(kThreads) k_f64_boundary(const gbf_model m, const GbfF64Step s, const GbfMassTail tail) {
  gbf_pdl_begin();
  unsigned blocks = gridDim.x;
  if (tail.out && blockIdx.x == --blocks) {
    gbf_mass_tail(tail);
    return;
  }
  const GbfGeo g = gbf_geo(m);
  const size_t nb = gbf_boundary_count(g);
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nb; t += (size_t)blocks * blockDim.x)
    gbf_f64_boundary_cell(m, s, g, t);
}

}  // namespace

namespace {
// Block size of the pair step's passes over n cells: 64 where 256 would leave
// less than a few blocks an SM. Time of a step with 256, 128, 64, 32 threads:
// 40^3 17.3, 15.9, 15.1, 14.8 us; 64^3 25.5, 23.8, 23.4, 26.4 us; with 256 and
// 64 threads 68^3 (the cut) 28.9, 26.3, 80^3 34.7, 34.0, 96^3 51.2, 50.6,
// 112^3 74.7, 75.1.
unsigned pair_threads(size_t n) { return n < (size_t)gbf_num_sms() * 2048 ? 64u : (unsigned)kThreads; }
}  // namespace

// Blocks of the flux pass: one wave (its per-block mass partials).
unsigned gbf_f64_flux_grid(const gbf_model& m) {
  const size_t nint = (size_t)(m.nx - 2) * (m.ny - 2) * (m.nz - 2);
  const unsigned t = gbf_pair_applies(m) ? pair_threads(gbf_geo(m).n) : (unsigned)kThreads;
  return gbf_grid_for(nint, (int)t, 1024 / (int)t);
}

int gbf_density_launch(const gbf_model& m, int phase, const double* P, double* out, cudaStream_t st) {
  const size_t n = gbf_geo(m).n;
  k_density<<<gbf_grid_for(n, kThreads), kThreads, 0, st>>>(phase == 1 ? m.ro01 : m.ro02, phase == 1 ? m.beta1 : m.beta2,
                                                           m.P_atm, P, out, n);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GBF_OK : gbf_cuda_check(e, "gbf_density_launch");
}

int gbf_pair_fill_rows(const gbf_model& m, GbfPairRow* rows, cudaStream_t st) {
  k_pair_rows<<<gbf_grid_for((size_t)m.ny, kThreads), kThreads, 0, st>>>(m, rows);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GBF_OK : gbf_cuda_check(e, "gbf_pair_fill_rows");
}

int gbf_f64_launch_step(const gbf_model& m, const GbfDerived& d, const gbf_cells& cells, const GbfF64Step& s,
                        const GbfPairConsts* pc, const GbfPairWork* pair, int props_flags, double* mass_out,
                        cudaStream_t st, GbfTimer* tm) {
  const GbfGeo g = gbf_geo(m);
  const unsigned fg = gbf_f64_flux_grid(m);
  const bool mass = s.mass_partials && mass_out;
  cudaError_t err = cudaSuccess;
  // programmatic launches up to 4M cells. us a step with, without: 40^3 15.0, 20.1; 96^3 51.2, 54.1; 128^3 108.7,
  // 104.9; 144^3 150.9, 151.1; 160^3 (4.1M) 181.3, 186.8; 176^3 242, 237; 256^3 669, 661
  const bool pdl = g.n < (4u << 20);
  unsigned threads = kThreads;
  auto go = [&](auto kern, unsigned blocks, auto... args) {
    if (err == cudaSuccess) err = gbf_launch(pdl, kern, blocks, threads, 0, st, args...);
  };
  cudaEvent_t e = gbf_timer_begin(tm, st);
  if (pair) {
    threads = pair_threads(g.n);
    const unsigned pg = gbf_grid_for(g.n, (int)threads, 2048 / (int)threads);
    go(pair->P_from ? k_pair_props<true> : k_pair_props<false>, pg, *pc, cells, s, *pair);
    if (props_flags) {  // the outputs P2, Xi, u of the state the step starts from
      GbfF64Step o = s;
      o.L1 = nullptr;
      threads = kThreads;
      go(k_f64_props, gbf_grid_for(g.n, kThreads, 4), m, d, cells, o, props_flags);
    }
  } else {
    go(k_f64_props, gbf_grid_for(g.n, kThreads, 4), m, d, cells, s, props_flags);
  }
  gbf_timer_end(tm, GBF_K_PROPS, e, st);
  e = gbf_timer_begin(tm, st);
  if (pair) {
    threads = pair_threads(g.n);
    go(threads == 64 ? (mass ? k_pair_step<true, 64> : k_pair_step<false, 64>)
                     : (mass ? k_pair_step<true, kThreads> : k_pair_step<false, kThreads>),
       fg, *pc, m, d, cells, s, *pair);
    threads = kThreads;
  } else {
    go(k_f64_flux_newton, fg, m, d, cells, s);
  }
  gbf_timer_end(tm, GBF_K_FLUX_NEWTON, e, st);
  e = gbf_timer_begin(tm, st);
  const GbfMassTail tail = {s.mass_partials, (int)fg, mass ? mass_out : nullptr, 0.0};
  go(k_f64_boundary, gbf_grid_for(gbf_boundary_count(g), kThreads, 4) + (mass ? 1 : 0), m, s, tail);
  gbf_timer_end(tm, GBF_K_BOUNDARY, e, st);
  return err == cudaSuccess ? GBF_OK : gbf_cuda_check(err, "gbf_f64_launch_step");
}
