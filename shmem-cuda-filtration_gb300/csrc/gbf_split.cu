// gbf_split.cu — split-precision step: FP32 pressure, saturation, K, phi and
// fluxes; FP64 (or FP32-pair) per-cell phase masses and one wide-precision
// residual per cell.
//
// State (per cell):
//   dP  = P - P_hs(j), FP32, with P_hs(j) = P_atm + j rho01 g h2 the
//         hydrostatic profile of the initial state (main.cpp:114). Vertical
//         potentials then read -(dP(j+1) - dP(j))/h2 + (rho_c - rho01) g: the
//         two large hydrostatic terms cancel exactly before anything is rounded.
//   S   = S2, FP32.
//   M1, M2 (interior cells): the phase masses per pore volume the
//         reference's mass update starts from, ro1 (1 - S2) and ro2 S2 with
//         ro2 at P2 = P1 (cpu.cpp:224-225), in FP64 (GBF_PREC_SPLIT), as an
//         unevaluated sum of two FP32 (GBF_PREC_SPLIT_DF), or as FP32 defects
//         over c1(j) (1 - S), c2(j) S (GBF_PREC_SPLIT_DEFECT).
// The tile routine (gbf_split_tile.cuh) does the fused update of one column
// tile; this file holds the single-domain kernels and the host side.
#include <math.h>

#include <algorithm>

#include "gbf_split_x2.cuh"

GbfPatchConsts gbf_patch_consts(const gbf_model& m) {
  GbfPatchConsts P = {};
  if (m.source_mode != GBF_SOURCE_DIRICHLET_PATCH || m.source < 0) return P;
  P.n = 2 * m.source + 1;
  P.i0 = m.nx / 2 - m.source;
  P.k0 = m.nz / 2 - m.source;
  P.S2 = m.S2_gr;
  P.nmr2 = -m.ro02 / m.mu2;
  P.gh2 = m.g * m.h2;
  P.wy = m.dt * m.kv / (m.h2 * m.h2);
  for (int md = 0; md < 2; md++) {
    P.K[md] = m.K[md];
    P.se_b[md] = -1.0 / (1.0 - m.S_wr[md]);
    P.e2[md] = (2. + m.lambda[md]) / m.lambda[md];
  }
  return P;
}

GbfSplitConsts gbf_split_consts(const gbf_model& m, int px) {
  GbfSplitConsts C = {};
  C.px = px;
  C.nx = m.nx; C.ny = m.ny; C.nz = m.nz;
  C.noflow_bottom = (m.bc_mode == GBF_BC_HYDROSTATIC_SIDES);
  const double V = m.h1 * m.h2 * m.h3;
  double src = 0.0;
  if (m.source_mode == GBF_SOURCE_RATE && m.rate_cells > 0) {
    C.rn = m.rate_cells;
    C.ri0 = m.nx / 2 - m.rate_cells / 2;
    C.rk0 = m.nz / 2 - m.rate_cells / 2;
    src = m.rate / (double)(m.rate_cells * m.rate_cells) / V;
  } else {  // the cells under the Dirichlet patch (the PATCH tiles; gbf_patch_consts)
    const GbfPatchConsts P = gbf_patch_consts(m);
    C.rn = P.n;
    C.ri0 = P.i0;
    C.rk0 = P.k0;
  }
  const double H = m.ro01 * m.g * m.h2;
  C.H = (float)H;
  C.ro01 = (float)m.ro01; C.ro02 = (float)m.ro02; C.beta1 = (float)m.beta1; C.beta2 = (float)m.beta2;
  C.bmax = C.beta1 > C.beta2 ? C.beta1 : C.beta2;
  C.cfl1 = (float)(1.0 / m.ro01); C.cfl2 = (float)(1.0 / m.ro02);
  C.nmr1 = (float)(-m.ro01 / m.mu1);
  C.nmr2 = (float)(-m.ro02 / m.mu2);
  C.ro01b1 = (float)(m.ro01 * m.beta1);
  C.ro02b2 = (float)(m.ro02 * m.beta2);
  for (int md = 0; md < 2; md++) {
    const double lam = m.lambda[md], swr = m.S_wr[md];
    C.K[md] = (float)m.K[md];
    C.m[md] = (float)m.m[md];
    C.se_b[md] = (float)(-1.0 / (1.0 - swr));
    C.e1[md] = (float)((2. + 3. * lam) / lam);
    C.e2[md] = (float)((2. + lam) / lam);
    C.m_inv_lam[md] = (float)(-1. / lam);
    C.inv_lam_1mswr[md] = (float)(1.0 / (lam * (1.0 - swr)));
    C.P_d[md] = (float)m.P_d[md];
  }
  C.H_d = H; C.beta1_d = m.beta1; C.beta2_d = m.beta2; C.ro01_d = m.ro01; C.ro02_d = m.ro02;
  C.dtsrc_d = m.dt * src;
  C.V = V;
  C.ro01b1_d = m.ro01 * m.beta1;
  C.ro02b2_d = m.ro02 * m.beta2;
  C.ro01b1_lo = (float)(C.ro01b1_d - (double)C.ro01b1);
  C.ro02b2_lo = (float)(C.ro02b2_d - (double)C.ro02b2);
  C.gh1 = (float)(m.g * m.ro01 * m.beta1 * m.h2);
  C.gh2 = (float)(m.g * m.ro02 * m.beta2 * m.h2);
  C.ghd = (float)(m.g * (m.ro02 - m.ro01) * m.h2);
  C.wx = (float)(m.dt / (m.h1 * m.h1));
  C.wy = (float)(m.dt * m.kv / (m.h2 * m.h2));
  C.wz = (float)(m.dt / (m.h3 * m.h3));
  C.H_df = gbf_df_from_double(H);
  C.beta1_df = gbf_df_from_double(m.beta1);
  C.beta2_df = gbf_df_from_double(m.beta2);
  C.ro01_df = gbf_df_from_double(m.ro01);
  C.ro02_df = gbf_df_from_double(m.ro02);
  C.dtsrc_df = gbf_df_from_double(C.dtsrc_d);
  for (int md = 0; md < 2; md++) {
    C.m_d[md] = m.m[md];
    C.m_df[md] = gbf_df_from_double(m.m[md]);
    C.dtsrc_m_d[md] = C.dtsrc_d / m.m[md];
    C.dtsrc_m_df[md] = gbf_df_from_double(C.dtsrc_m_d[md]);
  }
  return C;
}

namespace {

constexpr int kThreads = 256;

int tiles_x(const GbfSplitConsts& C) { return (C.nx - 2 + kSplitTX - 1) / kSplitTX; }
int tiles_y(const GbfSplitConsts& C) { return (C.ny - 2 + kSplitTY - 1) / kSplitTY; }
// The plain-load tile on one grid (grids without TMA staging). Block b runs
// tile b mod (tiles of a chunk layer) of the k chunk kc0 + b / (tiles of a
// layer), kchunk planes from 1 + kchunk kc; G.mass_partials is that launch's
// first partial.
template <int MR, bool CFL, bool PATCH>
__global__ void __launch_bounds__(kSplitThreads, 4) k_split_step(const GbfSplitConsts C, const GbfSplitGrid G,
                                                              const int kchunk, const int kc0) {
  gbf_pdl_begin();
  __shared__ GbfSplitPlane pl[2];
  const int ntx = (C.nx - 2 + kSplitTX - 1) / kSplitTX, nty = (C.ny - 2 + kSplitTY - 1) / kSplitTY;
  const int b = blockIdx.x;
  const int tx = b % ntx, ty = (b / ntx) % nty, kc = kc0 + b / (ntx * nty);
  const int k0 = 1 + kc * kchunk;
  const int k1 = min(k0 + kchunk, C.nz - 1);
  GbfSplitAcc<MR> acc;
  split_tile<MR, kSplitTX, kSplitTY, false, CFL, PATCH>(C, G, 1 + tx * kSplitTX, 1 + ty * kSplitTY, k0, k1, pl, acc);
  if (acc.bad) atomicOr(G.status, GBF_DEV_NONFINITE);
  if (G.mass_partials) split_block_mass<MR>(acc, C.V, G.mass_partials + 2 * blockIdx.x);
  if constexpr (CFL) split_block_cfl<kSplitThreads>(acc.cfl1, acc.cfl2, G.cfl_out);
}

// Boundary cells [0, nb) of gbf_boundary_cell's enumeration (all, or all but
// the x faces that the x-pair tile writes).
__global__ void __launch_bounds__(kThreads) k_split_boundary(const gbf_model m, int px, const GbfSplitGrid G, float H,
                                                             size_t nb, int k_lo, int k_hi, const GbfMassTail tail) {
  gbf_pdl_begin();
  unsigned blocks = gridDim.x;
  if (tail.out && blockIdx.x == --blocks) {
    gbf_mass_tail(tail);
    return;
  }
  const GbfGeo g = gbf_geo(m, px);
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nb; t += (size_t)blocks * blockDim.x) {
    int i, j, k;
    gbf_boundary_cell(g, t, i, j, k);
    if (k < k_lo || k >= k_hi) continue;  // planes [k_lo, k_hi) only (a slab of the host pipeline)
    const size_t c = gbf_idx(g, i, j, k);
    G.Sn[c] = gbf_sweep_S<float>(m, g, G.Sn, G.S, i, j, k);
    G.dPn[c] = gbf_split_sweep_dP(m, g, G.dPn, G.dP, i, j, k, H);
  }
}

// Per interior row j: c1(j) times the sum of the row's interior porosities
// (FP64), one block per row.
__global__ void k_defect_k1_rows(const gbf_model m, const float* phi, const int* media, double* rows) {
  __shared__ double red[256];
  const int nx = m.nx, ny = m.ny, nz = m.nz, j = 1 + blockIdx.x;
  const size_t n = (size_t)(nx - 2) * (nz - 2);
  double a = 0.;
  for (size_t t = threadIdx.x; t < n; t += blockDim.x) {
    const int i = 1 + (int)(t % (nx - 2)), k = 1 + (int)(t / (nx - 2));
    const size_t c = (size_t)i + (size_t)j * nx + (size_t)k * nx * ny;
    a += phi ? (double)phi[c] : m.m[media ? media[c] : 0];
  }
  red[threadIdx.x] = a;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) rows[blockIdx.x] = (double)gbf_defect_row(m, j).c1 * red[0];
}
__global__ void k_defect_k1_sum(const double* rows, int nrows, double V, double* out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double a = 0.;
    for (int q = 0; q < nrows; q++) a += rows[q];
    *out = a * V;
  }
}

// The state conversions of cells [c0, c1): each block kConvCells consecutive
// cells, the loads of a thread's cells in flight together.
constexpr int kConvPer = 4, kConvCells = kConvPer * kThreads;
template <int MR>
__global__ void __launch_bounds__(kThreads) k_split_init(const gbf_model m, int px, const GbfFastDiv dnx,
                                                         const GbfFastDiv dny, const GbfRowConst* rows, const double* P,
                                                         const double* S, float* dP0, float* dP1, float* S0, float* S1, double* M1,
                                                         double* M2, unsigned c0, unsigned c1) {
  const unsigned b = c0 + blockIdx.x * kConvCells + threadIdx.x;
  double p[kConvPer], s[kConvPer];
#pragma unroll
  for (int u = 0; u < kConvPer; u++) {
    const unsigned c = b + u * kThreads;
    if (c < c1) {
      p[u] = P[c];
      s[u] = S[c];
    }
  }
#pragma unroll
  for (int u = 0; u < kConvPer; u++) {
    const unsigned c = b + u * kThreads;
    if (c < c1) {
      const unsigned r = gbf_div(c, dnx), j = r - gbf_div(r, dny) * dny.d, q = c + r * (unsigned)(px - m.nx);
      float dp, sf;
      gbf_split_init_cell<MR, false>(m, p[u], s[u], rows[j], dp, sf, M1, M2, q);
      dP0[q] = dp;
      dP1[q] = dp;  // the next-state buffer's faces are rewritten every step; they start equal
      S0[q] = sf;
      S1[q] = sf;
    }
  }
}

__global__ void __launch_bounds__(kThreads) k_split_to_f64(unsigned pad, const GbfFastDiv dnx,
                                                           const GbfFastDiv dny, const GbfRowConst* rows, const float* dPf, const float* Sf,
                                                           double* P, double* S, unsigned c0, unsigned c1) {
  const unsigned b = c0 + blockIdx.x * kConvCells + threadIdx.x;
  float p[kConvPer], s[kConvPer];
#pragma unroll
  for (int u = 0; u < kConvPer; u++) {
    const unsigned c = b + u * kThreads;
    if (c < c1) {
      const unsigned q = pad ? c + gbf_div(c, dnx) * pad : c;  // pad: the padding of a row
      if (P) p[u] = dPf[q];
      if (S) s[u] = Sf[q];
    }
  }
#pragma unroll
  for (int u = 0; u < kConvPer; u++) {
    const unsigned c = b + u * kThreads;
    if (c < c1) {
      if (P) {
        const unsigned r = gbf_div(c, dnx), j = r - gbf_div(r, dny) * dny.d;
        P[c] = gbf_split_P(p[u], rows[j]);
      }
      if (S) S[c] = gbf_f2d_all(s[u]);
    }
  }
}

__global__ void k_split_rows(const gbf_model m, GbfRowConst* rows) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < m.ny; j += gridDim.x * blockDim.x) rows[j] = gbf_row_const(m, j);
}

}  // namespace

// k planes per CTA of a grid of `tiles` column tiles and `nzi` interior
// planes, run with `slots` CTAs resident at a time: the CTAs run in waves,
// and the last wave of an uneven count leaves slots idle. Among k ranges of
// at least 16 planes (or the whole column), take the one with the fewest
// plane-times: waves x (planes per CTA + about 1.5 for the prologue, which
// builds the first plane and loads the plane below it). Grids that fill
// less than one wave may go down to 2 planes per CTA: there the planes a CTA
// marches through are the step's latency (40^3: 8 planes 19.4 us a step, 2
// planes 13.0).
int gbf_split_kchunk_waves(long long tiles, int nzi, long long slots, double* cost_out = nullptr) {
  if (nzi < 1) nzi = 1;
  if (slots < 1) slots = 1;
  const int max_chunks = (nzi + 1) / 2;
  int best = nzi;
  double best_cost = 1e300;
  for (int chunks = 1; chunks <= max_chunks; chunks++) {
    const int kc = (nzi + chunks - 1) / chunks;
    const long long ctas = tiles * ((nzi + kc - 1) / kc);
    if (chunks > 1 && kc < 16 && ctas > slots) continue;
    const double cost = (double)((ctas + slots - 1) / slots) * (kc + 1.5);
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best = kc;
    }
  }
  if (cost_out) *cost_out = best_cost;
  return best;
}

namespace {
constexpr int kPairTX[kPairShapes] = {64, 32, 16}, kPairTY[kPairShapes] = {8, 16, 32};
long long pair_tiles(const GbfSplitConsts& C, int shape) {
  return (long long)((C.nx - 1 + kPairTX[shape] - 1) / kPairTX[shape]) *
         ((C.ny - 2 + kPairTY[shape] - 1) / kPairTY[shape]);
}
}  // namespace

// Resident CTAs per SM (launch bounds and shared memory): the 32x8 plain-load
// tile 4, the x-pair tiles gbf_pair_ctas: 3 in the defect form (2 in the 16x32
// shape, 77 KB of shared memory), else 2. The x-pair shape is the one with the
// fewest plane-times: a grid's rows fill 64 lanes badly where nx is just above
// a multiple of 64 or small (13x300x280: 68.6 us a step with 64x8, 29.7 with
// 16x32; 151x97x83: 31.2 and 29.3 with 32x16), and the three cost the same a
// plane.
GbfSplitPlan gbf_split_plan(const GbfSplitConsts& C, int mr, bool tma) {
  const long long sms = gbf_num_sms();
  if (!tma) {
    const int kc = gbf_split_kchunk_waves((long long)tiles_x(C) * tiles_y(C), C.nz - 2, 4 * sms);
    return {0, kc, kc};
  }
  GbfSplitPlan plan = {};
  double best = 1e300;
  for (int shape = 0; shape < kPairShapes; shape++) {
    const int ctas = mr == kMassDefect && shape == kPair16x32 ? 2 : gbf_pair_ctas(mr);
    double cost;
    const int kc = gbf_split_kchunk_waves(pair_tiles(C, shape), C.nz - 2, ctas * sms, &cost);
    if (shape == kPair64x8) plan.kchunk_cfl = kc;
    if (cost < best - 1e-9) {
      best = cost;
      plan.shape = shape;
      plan.kchunk = kc;
    }
  }
  return plan;
}

// The step tiles of k chunks [kc0, kc0 + nkc) (kchunk planes each): the
// x-pair tile with TMA staging (maps), else the plain-load tile.
namespace {
// The Dirichlet patch's pre-pass, one thread per patch cell (gbf_split_patch_cell).
__global__ void __launch_bounds__(kThreads) k_split_patch(const GbfSplitConsts C, const GbfPatchConsts P,
                                                          const GbfSplitGrid G) {
  gbf_pdl_begin();
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < P.n * P.n; t += gridDim.x * blockDim.x)
    gbf_split_patch_cell(C, P, G, t);
}
}  // namespace

template <int MR, bool PATCH>
int launch_plain(const GbfSplitConsts& C, const GbfSplitGrid& G, cudaStream_t st, int kchunk, int kc0, int nkc) {
  const unsigned blocks = (unsigned)(tiles_x(C) * tiles_y(C) * nkc);
  GBF_CUDA(gbf_launch(true, G.cfl_out ? k_split_step<MR, true, PATCH> : k_split_step<MR, false, PATCH>, blocks, kSplitThreads, 0,
                      st, C, G, kchunk, kc0));
  return GBF_OK;
}

// The step tiles of k chunks [kc0, kc0 + nkc) (kchunk planes each): the
// x-pair tile with TMA staging (maps), else the plain-load tile. Under a
// Dirichlet patch (G.patch_in set) the PATCH instantiations.
int launch_chunks(const GbfSplitConsts& C, const GbfSplitGrid& G, int mr, int shape, const GbfTmaSet* maps, int buf,
                  cudaStream_t st, int kchunk, int kc0, int nkc) {
  if (maps) {
    if (shape != kPair64x8) maps++;
    return G.K ? gbf_launch_x2_fields(shape, C, G, mr, maps, buf, st, kchunk, kc0, nkc)
               : gbf_launch_x2_table(shape, C, G, mr, maps, buf, st, kchunk, kc0, nkc);
  }
  auto form = [&](auto tag) {
    constexpr int MR = decltype(tag)::value;
    return G.patch_in ? launch_plain<MR, true>(C, G, st, kchunk, kc0, nkc) : launch_plain<MR, false>(C, G, st, kchunk, kc0, nkc);
  };
  return mr == kMassDefect ? form(std::integral_constant<int, kMassDefect>{})
         : mr == kMassDF   ? form(std::integral_constant<int, kMassDF>{})
                           : form(std::integral_constant<int, kMassDefectDF>{});
}
// The shape of a step's tiles (CFL numbers: 64x8), and the tiles of a chunk layer.
int step_shape(const GbfSplitGrid& G, const GbfSplitPlan& plan) { return G.cfl_out ? kPair64x8 : plan.shape; }
long long layer_tiles(const GbfSplitConsts& C, int shape, const GbfTmaSet* maps) {
  return maps ? pair_tiles(C, shape) : (long long)tiles_x(C) * tiles_y(C);
}

int gbf_split_launch_domain(const gbf_model& m, const GbfSplitConsts& C, const GbfSplitGrid& G, int mr,
                            double* mass_out, cudaStream_t st, GbfTimer* tm, const GbfTmaSet* maps, int buf,
                            double k1v, const GbfSplitPlan& plan) {
  const int shape = step_shape(G, plan), kchunk = G.cfl_out ? plan.kchunk_cfl : plan.kchunk;
  const int nkc = (C.nz - 2 + kchunk - 1) / kchunk;
  const unsigned blocks = (unsigned)(layer_tiles(C, shape, maps) * nkc);
  cudaEvent_t e = gbf_timer_begin(tm, st);
  if (G.patch_in) {  // the Dirichlet patch's FP64 inflow, timed with the step kernel
    const GbfPatchConsts P = gbf_patch_consts(m);
    GBF_CUDA(gbf_launch(true, k_split_patch, gbf_grid_for((size_t)P.n * P.n, kThreads), kThreads, 0, st, C, P, G));
  }
  // TMA staging (maps): the x-pair tile; else the plain-load tile
  if (int s = launch_chunks(C, G, mr, shape, maps, buf, st, kchunk, 0, nkc)) return s;
  gbf_timer_end(tm, GBF_K_SPLIT_STEP, e, st);
  e = gbf_timer_begin(tm, st);
  // one cell per thread (row segments, as the ensembles' face pass walks
  // them, measured 8.6 -> 10.4 us on 256^3: too few warps for a latency-bound pass)
  const size_t nb = maps ? gbf_boundary_count_no_xfaces(gbf_geo(m)) : gbf_boundary_count(gbf_geo(m));
  const bool mass = G.mass_partials && mass_out;
  const GbfMassTail tail = {G.mass_partials, (int)blocks, mass ? mass_out : nullptr, gbf_is_defect(mr) ? k1v : 0.0};
  GBF_CUDA(gbf_launch(true, k_split_boundary, gbf_grid_for(nb, kThreads, 4) + (mass ? 1 : 0), kThreads, 0, st, m, C.px, G, C.H, nb,
                      0, C.nz, tail));
  gbf_timer_end(tm, GBF_K_SPLIT_BOUNDARY, e, st);
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? GBF_OK : gbf_cuda_check(err, "gbf_split_launch_domain");
}

// The host-resident pipeline's slabs (gbf_split_advance_host): one k chunk
// layer of the step each, about 1M cells (16 MB each way) or more, so that a
// slab's copies outlast its few launches, at most 16, at least 4 planes.
constexpr long long kPipeSlabCells = 1ll << 20;
int pipe_slabs(const GbfSplitConsts& C) {
  const long long cells = (long long)C.nx * C.ny * C.nz;
  return (int)std::min(16ll, std::max(1ll, cells / kPipeSlabCells));
}
int pipe_kchunk(const GbfSplitConsts& C) {
  const int s = pipe_slabs(C);
  return std::max(4, (C.nz - 2 + s - 1) / s);
}
bool gbf_split_pipelined(const gbf_model& m) {
  const GbfSplitConsts C = gbf_split_consts(m);
  return pipe_slabs(C) >= 2 && (C.nz - 2 + pipe_kchunk(C) - 1) / pipe_kchunk(C) >= 2;
}

// Mass-partial slots: the largest CTA count of the grid's launches.
unsigned gbf_split_blocks(const gbf_model& m, int mr) {
  const GbfSplitConsts C = gbf_split_consts(m);
  const GbfSplitPlan a = gbf_split_plan(C, mr, false), b = gbf_split_plan(C, mr, true);
  const int kp = pipe_kchunk(C);
  auto ctas = [&](long long tiles, int kc) { return tiles * ((C.nz - 2 + kc - 1) / kc); };
  long long most = ctas((long long)tiles_x(C) * tiles_y(C), std::min(a.kchunk, kp));
  most = std::max(most, ctas(pair_tiles(C, kPair64x8), std::min(b.kchunk_cfl, kp)));
  return (unsigned)std::max(most, ctas(pair_tiles(C, b.shape), std::min(b.kchunk, kp)));
}

// ----------------------------------------------------------------- host side

// A field of the caller's cells (nx a row) to rows px apart.
__global__ void __launch_bounds__(kThreads) k_split_pitch(const unsigned* src, unsigned* dst, GbfFastDiv dnx, unsigned pad,
                                                          unsigned n) {
  for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
    dst[c + gbf_div(c, dnx) * pad] = src[c];
}
static int pitch_field(gbf_domain* d, const void* src, const void* dst) {
  const unsigned n = (unsigned)gbf_geo(d->m).n;
  k_split_pitch<<<gbf_grid_for(n, kThreads), kThreads, 0, d->stream>>>((const unsigned*)src, (unsigned*)dst,
                                                                       gbf_fast_div((unsigned)d->m.nx),
                                                                       (unsigned)(d->px - d->m.nx), n);
  GBF_CUDA(cudaGetLastError());
  return GBF_OK;
}
int gbf_split_pitch_media(gbf_domain* d) {
  if (d->split_cells.media == d->cells.media) return GBF_OK;
  return pitch_field(d, d->cells.media, d->split_cells.media);
}

int gbf_split_alloc(gbf_domain* d) {
  const gbf_model& m = d->m;
  // Grids with K and porosity fields and no media table, or with the media
  // table (or one medium) and no field, run the x-pair tile: TMA staging wants
  // rows of whole 16-byte units, so the split state's and the fields' rows are
  // padded to that. Measured against the plain-load tile, us a step: 256^3 of
  // the media table under the Dirichlet patch 322 -> 214, 255x253x251 with
  // fields 271 -> 193, 67x45x150 of the table 36.5 -> 31.4, 40^3 15.1 -> 13.0.
  const bool fields = d->cells.K && d->cells.phi && !d->cells.media, table = !d->cells.K && !d->cells.phi;
  const int pitch = (m.nx + 3) / 4 * 4;
  const bool tma = (fields || table) && gbf_tma_eligible(pitch, 64) &&
                   (double)pitch * m.ny * m.nz < 2147483648.0;
  d->px = tma ? pitch : m.nx;
  const GbfSplitPlan plan = gbf_split_plan(gbf_split_consts(m), gbf_mass_rep(d->precision), tma);
  d->split_plan[0] = plan.shape;
  d->split_plan[1] = plan.kchunk;
  d->split_plan[2] = plan.kchunk_cfl;
  const size_t n = (size_t)d->px * m.ny * m.nz;
  int s = GBF_OK;
  for (int b = 0; b < 2 && !s; b++) {
    s |= gbf_domain_alloc(d, (void**)&d->Pf[b], n * sizeof(float));
    s |= gbf_domain_alloc(d, (void**)&d->Sf[b], n * sizeof(float));
  }
  // FP64 masses or FP32 pairs: 8 bytes per cell and phase; FP32 defects: 4
  const int mb = gbf_mass_bytes(gbf_mass_rep(d->precision));
  if (!s) s |= gbf_domain_alloc(d, (void**)&d->M1, n * mb);
  if (!s) s |= gbf_domain_alloc(d, (void**)&d->M2, n * mb);
  d->split_cells = d->cells;
  // the cell fields in padded rows; a drop-in's media array that TMA cannot take in place is copied too
  if (!s && (d->px != m.nx || (tma && ((uintptr_t)d->cells.media & 15) != 0))) {
    auto padded = [&](const void* src, const void** dst) {
      if (!src || s) return;
      s |= gbf_domain_alloc(d, (void**)dst, n * 4);
      if (!s) s |= pitch_field(d, src, *dst);
    };
    padded(d->cells.K, (const void**)&d->split_cells.K);
    padded(d->cells.phi, (const void**)&d->split_cells.phi);
    padded(d->cells.media, (const void**)&d->split_cells.media);
  }
  // the defect form's water-mass part left out of the tiles' sums
  d->defect_k1v = 0.0;
  if (!s && gbf_is_defect(gbf_mass_rep(d->precision)))
    s |= gbf_defect_k1(d->m, d->cells.phi, d->cells.media, &d->defect_k1v, nullptr);  // after the cells' copies
  // per-block mass partials of the split step kernel
  if (!s) s |= gbf_domain_alloc(d, (void**)&d->split_partials, 2 * sizeof(double) * gbf_split_blocks(d->m, gbf_mass_rep(d->precision)));
  // the row table of the state conversions
  if (!s) s |= gbf_domain_alloc(d, (void**)&d->split_rows, sizeof(GbfRowConst) * (size_t)d->m.ny);
  if (!s) s |= gbf_split_fill_rows(d->m, d->split_rows, d->stream);
  // the Dirichlet patch's inflow, one FP32 pair per patch cell
  const int pn = gbf_patch_consts(d->m).n;
  if (!s && pn > 0) {  // zeroed: entries outside the interior are never written (nor used)
    s |= gbf_domain_alloc(d, (void**)&d->split_patch, sizeof(float2) * (size_t)pn * pn);
    if (!s) s |= gbf_cuda_check(cudaMemset(d->split_patch, 0, sizeof(float2) * (size_t)pn * pn), "gbf_split_alloc");
  }
  if (s) return GBF_ERR_NOMEM;
  if (tma) {
    // boxes of the x-pair tile, 64x8 and the plan's: halo planes {TX + 8, TY + 2}
    // (K, or the media indices), interior rows {TX, TY}
    GbfTmaSet h[2] = {};
    int e = GBF_OK;
    const int px = d->px, shapes[2] = {kPair64x8, d->split_plan[0]};
    const gbf_cells& c = d->split_cells;
    const void* k = fields ? (const void*)c.K : (const void*)c.media;
    for (int q = 0; q < 2 && !e; q++) {
      const int tx = kPairTX[shapes[q]], ty = kPairTY[shapes[q]];
      auto box = [&](void* map, const void* base, int eb, int bx, int by) {
        if (!e) e |= gbf_tma_encode_box(map, base, eb, m.nx, m.ny, m.nz, px, bx, by);
      };
      for (int b = 0; b < 2; b++) {
        box(&h[q].dP[b], d->Pf[b], 4, tx + 8, ty + 2);
        box(&h[q].S[b], d->Sf[b], 4, tx + 8, ty + 2);
      }
      if (k) box(&h[q].K, k, 4, tx + 8, ty + 2);
      box(&h[q].M1, d->M1, mb, tx, ty);
      box(&h[q].M2, d->M2, mb, tx, ty);
      if (fields) box(&h[q].phi, c.phi, 4, tx, ty);
    }
    if (!e) e |= gbf_domain_alloc(d, &d->tma, sizeof(h));
    if (e) return GBF_ERR_CUDA;
    GBF_CUDA(cudaMemcpy(d->tma, h, sizeof(h), cudaMemcpyHostToDevice));
  }
  return GBF_OK;
}

int gbf_defect_k1(const gbf_model& m, const float* phi_dev, const int* media_dev, double* k1v_host,
                  cudaStream_t st) {
  const int nrows = m.ny - 2;
  double* rows = nullptr;
  GBF_CUDA(cudaMallocAsync((void**)&rows, (nrows + 1) * sizeof(double), st));
  k_defect_k1_rows<<<nrows, 256, 0, st>>>(m, phi_dev, media_dev, rows);
  k_defect_k1_sum<<<1, 32, 0, st>>>(rows, nrows, m.h1 * m.h2 * m.h3, rows + nrows);
  GBF_CUDA(cudaGetLastError());
  GBF_CUDA(cudaMemcpyAsync(k1v_host, rows + nrows, sizeof(double), cudaMemcpyDeviceToHost, st));
  GBF_CUDA(cudaStreamSynchronize(st));
  GBF_CUDA(cudaFreeAsync(rows, st));
  return GBF_OK;
}

int gbf_split_fill_rows(const gbf_model& m, GbfRowConst* rows, cudaStream_t st) {
  k_split_rows<<<gbf_grid_for((size_t)m.ny, kThreads), kThreads, 0, st>>>(m, rows);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GBF_OK : gbf_cuda_check(e, "gbf_split_fill_rows");
}

int gbf_split_init_state(const gbf_model& m, int px, const GbfRowConst* rows, const double* P_dev, const double* S_dev,
                         float* const dPf[2], float* const Sf[2], double* M1, double* M2, int mr, size_t c0, size_t c1,
                         cudaStream_t st) {
  const GbfFastDiv dnx = gbf_fast_div((unsigned)m.nx), dny = gbf_fast_div((unsigned)m.ny);
  const unsigned blocks = (unsigned)((c1 - c0 + kConvCells - 1) / kConvCells);
  auto kern = mr == kMassDefect ? k_split_init<kMassDefect> : mr == kMassDF ? k_split_init<kMassDF> : k_split_init<kMassDefectDF>;
  kern<<<blocks, kThreads, 0, st>>>(m, px, dnx, dny, rows, P_dev, S_dev, dPf[0], dPf[1], Sf[0], Sf[1], M1, M2,
                                    (unsigned)c0, (unsigned)c1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GBF_OK : gbf_cuda_check(e, "gbf_split_init_state");
}

int gbf_split_upload(gbf_domain* d, const double* P1, const double* S2, cudaMemcpyKind kind) {
  const size_t n = gbf_geo(d->m).n, b = n * sizeof(double);
  const double *P = P1, *S = S2;
  double* tmp = nullptr;
  const double* mP = (const double*)gbf_mapped_host(P1);
  const double* mS = (const double*)gbf_mapped_host(S2);
  if (kind == cudaMemcpyHostToDevice && mP && mS) {  // page-locked: read in place
    P = mP;
    S = mS;
  } else if (kind == cudaMemcpyHostToDevice) {  // stage through device memory
    GBF_CUDA(cudaMallocAsync((void**)&tmp, 2 * b, d->stream));
    GBF_CUDA(cudaMemcpyAsync(tmp, P1, b, cudaMemcpyHostToDevice, d->stream));
    GBF_CUDA(cudaMemcpyAsync(tmp + n, S2, b, cudaMemcpyHostToDevice, d->stream));
    P = tmp;
    S = tmp + n;
  }
  d->cur = 0;
  if (int e = gbf_split_init_state(d->m, d->px, d->split_rows, P, S, d->Pf, d->Sf, d->M1, d->M2, gbf_mass_rep(d->precision), 0,
                                   n, d->stream))
    return e;
  if (tmp) GBF_CUDA(cudaFreeAsync(tmp, d->stream));
  return GBF_OK;
}

int gbf_split_step(gbf_domain* d) {
  const int nxt = d->cur ^ 1;
  GbfSplitGrid G;
  G.dP = d->Pf[d->cur];
  G.S = d->Sf[d->cur];
  G.dPn = d->Pf[nxt];
  G.Sn = d->Sf[nxt];
  if (d->borrowed)  // the caller's media array: read as it is now
    if (int e = gbf_split_pitch_media(d)) return e;
  G.K = d->split_cells.K;
  G.phi = d->split_cells.phi;
  G.media = d->split_cells.media;
  G.M1 = d->M1;
  G.M2 = d->M2;
  G.mass_partials = nullptr;
  G.status = d->status;
  G.cfl_out = nullptr;
  G.patch_in = d->split_patch;
  double* mass_out = nullptr;
  if ((d->out_flags & GBF_OUT_MASS) && d->mass_hist && d->mass_count < d->mass_cap) {
    G.mass_partials = d->split_partials;
    mass_out = d->mass_hist + 2 * d->mass_count;
    if ((d->out_flags & GBF_OUT_CFL) && d->cfl_hist) G.cfl_out = d->cfl_hist + 2 * d->mass_count;
    d->mass_count++;
  }
  const GbfSplitConsts C = gbf_split_consts(d->m, d->px);
  int s = gbf_split_launch_domain(d->m, C, G, gbf_mass_rep(d->precision), mass_out, d->stream, &d->timer,
                                  (const GbfTmaSet*)d->tma, d->cur, d->defect_k1v,
                                  {d->split_plan[0], d->split_plan[1], d->split_plan[2]});
  if (s) return s;
  d->cur = nxt;
  d->steps++;
  return GBF_OK;
}

int gbf_split_download(gbf_domain* d, int field, double* host) {
  const size_t n = gbf_geo(d->m).n, b = n * sizeof(double);
  if (field != GBF_FIELD_P1 && field != GBF_FIELD_S2)
    return gbf_fail(GBF_ERR_STATE, "split precision keeps P1 and S2 only");
  double* tmp = (double*)gbf_mapped_host(host);  // page-locked: written in place
  const bool staged = tmp == nullptr;
  if (staged) GBF_CUDA(cudaMallocAsync((void**)&tmp, b, d->stream));
  if (int e = gbf_split_state_to_f64(d->m, d->px, d->split_rows, d->Pf[d->cur], d->Sf[d->cur],
                                     field == GBF_FIELD_P1 ? tmp : nullptr, field == GBF_FIELD_S2 ? tmp : nullptr, 0, n,
                                     d->stream))
    return e;
  if (staged) {
    GBF_CUDA(cudaMemcpyAsync(host, tmp, b, cudaMemcpyDeviceToHost, d->stream));
    GBF_CUDA(cudaFreeAsync(tmp, d->stream));
  }
  GBF_CUDA(cudaStreamSynchronize(d->stream));
  return GBF_OK;
}

int gbf_split_state_to_f64(const gbf_model& m, int px, const GbfRowConst* rows, const float* dPf, const float* Sf, double* P,
                           double* S, size_t c0, size_t c1, cudaStream_t st) {
  const unsigned blocks = (unsigned)((c1 - c0 + kConvCells - 1) / kConvCells);
  k_split_to_f64<<<blocks, kThreads, 0, st>>>((unsigned)(px - m.nx), gbf_fast_div((unsigned)m.nx),
                                              gbf_fast_div((unsigned)m.ny), rows, dPf, Sf, P, S, (unsigned)c0,
                                              (unsigned)c1);
  GBF_CUDA(cudaGetLastError());
  return GBF_OK;
}

// One step of a grid from host FP64 arrays to host FP64 arrays, pipelined
// over slabs of planes (one k chunk layer of the step each): the copy engines
// move slab s + 1 in and slab s - 1 out while the compute stream converts slab
// s, steps the chunk layer of slab s - 1 (its tiles read the first plane of
// slab s), applies the boundary rules to its planes (they read nothing outside
// the slab but the start-of-step state) and converts it back. The state equals
// upload + step + download bit for bit; the phase masses sum the same cells in
// other partial blocks (within 1e-11 relative). Grids without a Dirichlet patch.
namespace {
int split_advance_host(gbf_domain* d, const double* P_in, const double* S_in, double* P_out, double* S_out) {
  const gbf_model& m = d->m;
  const GbfGeo g = gbf_geo(m);
  const size_t n = g.n, pl = g.pl;
  const int mr = gbf_mass_rep(d->precision);
  const GbfSplitConsts C = gbf_split_consts(m, d->px);
  const GbfTmaSet* maps = (const GbfTmaSet*)d->tma;
  const int kp = pipe_kchunk(C), ns = (C.nz - 2 + kp - 1) / kp;  // slabs = k chunks
  auto pa = [&](int q) { return q == 0 ? 0 : 1 + q * kp; };
  auto pb = [&](int q) { return q == ns - 1 ? C.nz : 1 + (q + 1) * kp; };
  if (!d->pipe_in) {
    GBF_CUDA(cudaStreamCreateWithFlags(&d->pipe_in, cudaStreamNonBlocking));
    GBF_CUDA(cudaStreamCreateWithFlags(&d->pipe_out, cudaStreamNonBlocking));
  }
  while ((int)d->pipe_ev.size() < 2 + 2 * ns) {
    cudaEvent_t e;
    GBF_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    d->pipe_ev.push_back(e);
  }
  if (!d->pipe_stage && gbf_domain_alloc(d, (void**)&d->pipe_stage, 2 * sizeof(double) * n))
    return gbf_fail(GBF_ERR_NOMEM, "gbf_domain_advance_host");
  double *stP = d->pipe_stage, *stS = d->pipe_stage + n;
  cudaStream_t cs = d->stream;
  // the upload's resets (gbf_domain_upload), then everything on the stream so far first
  d->cur = 0;
  d->mass_count = 0;
  d->steps = 0;
  if (d->cfl_hist) GBF_CUDA(cudaMemsetAsync(d->cfl_hist, 0, 2 * sizeof(float) * (size_t)d->mass_cap, cs));
  GBF_CUDA(cudaMemsetAsync(d->status, 0, sizeof(unsigned), cs));
  GBF_CUDA(cudaEventRecord(d->pipe_ev[0], cs));
  GBF_CUDA(cudaStreamWaitEvent(d->pipe_in, d->pipe_ev[0], 0));
  GBF_CUDA(cudaStreamWaitEvent(d->pipe_out, d->pipe_ev[0], 0));
  for (int q = 0; q < ns; q++) {  // host -> device, every slab in order
    const size_t c0 = (size_t)pa(q) * pl, b = ((size_t)pb(q) * pl - c0) * sizeof(double);
    GBF_CUDA(cudaMemcpyAsync(stP + c0, P_in + c0, b, cudaMemcpyDefault, d->pipe_in));
    GBF_CUDA(cudaMemcpyAsync(stS + c0, S_in + c0, b, cudaMemcpyDefault, d->pipe_in));
    GBF_CUDA(cudaEventRecord(d->pipe_ev[2 + q], d->pipe_in));
  }
  GbfSplitGrid G;
  G.dP = d->Pf[0];
  G.S = d->Sf[0];
  G.dPn = d->Pf[1];
  G.Sn = d->Sf[1];
  G.K = d->split_cells.K;
  G.phi = d->split_cells.phi;
  G.media = d->split_cells.media;
  G.M1 = d->M1;
  G.M2 = d->M2;
  G.mass_partials = nullptr;
  G.status = d->status;
  G.cfl_out = nullptr;
  G.patch_in = nullptr;
  double* mass_out = nullptr;
  if ((d->out_flags & GBF_OUT_MASS) && d->mass_hist && d->mass_cap > 0) {
    G.mass_partials = d->split_partials;
    mass_out = d->mass_hist;
    if ((d->out_flags & GBF_OUT_CFL) && d->cfl_hist) G.cfl_out = d->cfl_hist;
    d->mass_count = 1;
  }
  const int shape = G.cfl_out ? kPair64x8 : d->split_plan[0];
  const long long tiles = layer_tiles(C, shape, maps);
  const size_t nb = maps ? gbf_boundary_count_no_xfaces(g) : gbf_boundary_count(g);
  for (int q = 0; q <= ns; q++) {
    if (q < ns) {  // slab q in: FP64 -> split state, both buffers
      const size_t c0 = (size_t)pa(q) * pl, c1 = (size_t)pb(q) * pl;
      GBF_CUDA(cudaStreamWaitEvent(cs, d->pipe_ev[2 + q], 0));
      if (int e = gbf_split_init_state(m, d->px, d->split_rows, stP, stS, d->Pf, d->Sf, d->M1, d->M2, mr, c0, c1, cs)) return e;
    }
    if (q > 0) {  // slab q - 1: its chunk layer of the step, its boundary cells, out
      const int r = q - 1;
      const size_t c0 = (size_t)pa(r) * pl, c1 = (size_t)pb(r) * pl;
      GbfSplitGrid Gr = G;
      if (Gr.mass_partials) Gr.mass_partials += 2 * (size_t)tiles * r;
      if (int s = launch_chunks(C, Gr, mr, shape, maps, 0, cs, kp, r, 1)) return s;
      // the last slab's pass also sums the masses of all (every slab's tiles precede it on the stream)
      const bool sum = mass_out && q == ns;
      const GbfMassTail tail = {G.mass_partials, (int)(tiles * ns), sum ? mass_out : nullptr,
                                gbf_is_defect(mr) ? d->defect_k1v : 0.0};
      GBF_CUDA(gbf_launch(true, k_split_boundary, gbf_grid_for(nb, kThreads, 4) + (sum ? 1 : 0), kThreads, 0, cs, m, C.px, G, C.H,
                          nb, pa(r), pb(r), tail));
      if (int e = gbf_split_state_to_f64(m, d->px, d->split_rows, d->Pf[1], d->Sf[1], stP, stS, c0, c1, cs)) return e;
      GBF_CUDA(cudaGetLastError());
      GBF_CUDA(cudaEventRecord(d->pipe_ev[2 + ns + r], cs));
      GBF_CUDA(cudaStreamWaitEvent(d->pipe_out, d->pipe_ev[2 + ns + r], 0));
      const size_t b = (c1 - c0) * sizeof(double);
      GBF_CUDA(cudaMemcpyAsync(P_out + c0, stP + c0, b, cudaMemcpyDefault, d->pipe_out));
      GBF_CUDA(cudaMemcpyAsync(S_out + c0, stS + c0, b, cudaMemcpyDefault, d->pipe_out));
    }
  }
  GBF_CUDA(cudaGetLastError());
  GBF_CUDA(cudaEventRecord(d->pipe_ev[1], d->pipe_out));
  GBF_CUDA(cudaStreamWaitEvent(cs, d->pipe_ev[1], 0));
  d->cur = 1;
  d->steps = 1;
  d->uploaded = true;
  GBF_CUDA(cudaStreamSynchronize(cs));
  return GBF_OK;
}
}  // namespace

int gbf_split_advance_host(gbf_domain* d, const double* P_in, const double* S_in, double* P_out, double* S_out) {
  const int s = split_advance_host(d, P_in, S_in, P_out, S_out);
  if (s) {  // an error part-way: no copy may still read or write the caller's arrays after the return
    if (d->pipe_in) cudaStreamSynchronize(d->pipe_in);
    if (d->pipe_out) cudaStreamSynchronize(d->pipe_out);
    cudaStreamSynchronize(d->stream);
  }
  return s;
}

int gbf_split_launches_per_step(gbf_domain* d) {
  return 2 + (d->split_patch ? 1 : 0) + (d->borrowed && d->split_cells.media != d->cells.media ? 1 : 0);
}

// ----------------------------------------------------------- diagnostics
// The bounded mbarrier wait of the TMA tiles, run on a barrier phase that
// never completes (arrival count 2, one arrival, no copy in flight): every
// thread must give up after `tries` rounds and the block reports
// GBF_DEV_TIMEOUT, as the tiles do when a plane never arrives.
namespace {
__global__ void k_diag_wait(unsigned tries, unsigned* status) {
  __shared__ unsigned long long bar;
  if (threadIdx.x == 0) {
    gbf_mbar_init(&bar, 2);
    gbf_mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(gbf_smem_u32(&bar)) : "memory");
  const bool ok = gbf_mbar_wait(&bar, 0u, tries);
  if (__syncthreads_or(!ok) && threadIdx.x == 0) atomicOr(status, GBF_DEV_TIMEOUT);
}
}  // namespace

extern "C" int gbf_diag_bounded_wait(unsigned tries, double* ms) {
  unsigned* st = nullptr;
  GBF_CUDA(cudaMalloc((void**)&st, sizeof(unsigned)));
  GBF_CUDA(cudaMemset(st, 0, sizeof(unsigned)));
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  cudaEventRecord(a, nullptr);
  k_diag_wait<<<1, 256>>>(tries, st);
  cudaEventRecord(b, nullptr);
  unsigned h = 0;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(&h, st, sizeof(unsigned), cudaMemcpyDeviceToHost);
  float t = 0.f;
  if (e == cudaSuccess) cudaEventElapsedTime(&t, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(st);
  if (e != cudaSuccess) return gbf_cuda_check(e, "gbf_diag_bounded_wait");
  if (ms) *ms = t;
  return (h & GBF_DEV_TIMEOUT) ? gbf_fail(GBF_ERR_TIMEOUT, "bounded wait gave up (diagnostic)") : GBF_OK;
}
