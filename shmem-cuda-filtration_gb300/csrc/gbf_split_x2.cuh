// gbf_split_x2.cuh — the x-pair TMA tile on one grid: its kernel and launch,
// instantiated for grids with K and porosity fields and for grids of the
// media table in files that compile in parallel.
#pragma once

#include <type_traits>

#include "gbf_split_tile.cuh"

namespace {

// x-pair tiles (TMA staging): TX x TY cells from x0 = TX t, t such that x0 <= nx - 2
template <int TX>
__host__ __device__ int tiles_x2(const GbfSplitConsts& C) { return (C.nx - 1 + TX - 1) / TX; }
template <int TY>
__host__ __device__ int tiles_y2(const GbfSplitConsts& C) { return (C.ny - 2 + TY - 1) / TY; }

// The x-pair tile on one grid: one tile (TX x TY cells, a k range) per CTA,
// blocks mapped to tiles and k chunks as in k_split_step.
template <int MR, int TX, int TY, bool CFL, bool PATCH, bool TAB>
__global__ void __launch_bounds__(TX / 2 * TY, gbf_pair_ctas(MR)) k_split_step_x2(const GbfSplitConsts C,
                                                                         const GbfSplitGrid G, const int kchunk,
                                                                         const int kc0, const GbfTmaSet* maps,
                                                                         int buf) {
  extern __shared__ __align__(128) unsigned char dyn[];
  using Cta = GbfPairCta<TX, TY, MR>;
  Cta& cta = *reinterpret_cast<Cta*>(dyn);
  if (gbf_smem_u32(dyn) & 127u) {  // the TMA destinations need it; never expected to fire
    if (threadIdx.x == 0) atomicOr(G.status, GBF_DEV_TIMEOUT);
    return;
  }
  const int ntx = tiles_x2<TX>(C), nty = tiles_y2<TY>(C);
  const int b = blockIdx.x;
  const int tx = b % ntx, ty = (b / ntx) % nty, kc = kc0 + b / (ntx * nty);
  const int k0 = 1 + kc * kchunk;
  const int k1 = min(k0 + kchunk, C.nz - 1);
  if (threadIdx.x == 0) gbf_pair_bars_init(cta.bars);
  gbf_pdl_begin();
  __syncthreads();
  unsigned phases = 0;
  GbfSplitAcc<MR> acc;
  split_tile_x2<MR, TX, TY, CFL, TX / 2 * TY, PATCH, TAB>(C, G, TX * tx, 1 + TY * ty, k0,
                                                                         k1, cta.bars, cta.body, acc, maps, buf,
                                                                         &phases);
  if (acc.bad) atomicOr(G.status, GBF_DEV_NONFINITE);
  if (G.mass_partials) split_block_mass<MR, TX / 2 * TY>(acc, C.V, G.mass_partials + 2 * blockIdx.x);
  if constexpr (CFL) split_block_cfl<TX / 2 * TY>(acc.cfl1, acc.cfl2, G.cfl_out);
}

}  // namespace

// The step tiles of k chunks [kc0, kc0 + nkc) (kchunk planes each).
template <int MR, int TX, int TY, bool TAB, bool CFL, bool PATCH>
int launch_x2(const GbfSplitConsts& C, const GbfSplitGrid& G, const GbfTmaSet* maps, int buf, cudaStream_t st,
              int kchunk, int kc0, int nkc) {
  const unsigned blocks = (unsigned)(tiles_x2<TX>(C) * tiles_y2<TY>(C) * nkc);
  const int bytes = (int)sizeof(GbfPairCta<TX, TY, MR>);
  GBF_CUDA(cudaFuncSetAttribute(k_split_step_x2<MR, TX, TY, CFL, PATCH, TAB>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  GBF_CUDA(gbf_launch(true, k_split_step_x2<MR, TX, TY, CFL, PATCH, TAB>, blocks, TX / 2 * TY, (size_t)bytes, st, C, G, kchunk, kc0,
                      maps, buf));
  return GBF_OK;
}

// All forms of one shape and flavour: mr the masses, the Dirichlet patch when
// G.patch_in, CFL numbers when G.cfl_out (shapes compiled with CFL only).
template <int TX, int TY, bool TAB, bool CFL>
int launch_x2_form(const GbfSplitConsts& C, const GbfSplitGrid& G, int mr, const GbfTmaSet* maps, int buf,
                   cudaStream_t st, int kchunk, int kc0, int nkc) {
  auto go = [&](auto tag) {
    constexpr int MR = decltype(tag)::value;
    if constexpr (CFL)
      if (G.cfl_out)
        return G.patch_in ? launch_x2<MR, TX, TY, TAB, true, true>(C, G, maps, buf, st, kchunk, kc0, nkc)
                          : launch_x2<MR, TX, TY, TAB, true, false>(C, G, maps, buf, st, kchunk, kc0, nkc);
    return G.patch_in ? launch_x2<MR, TX, TY, TAB, false, true>(C, G, maps, buf, st, kchunk, kc0, nkc)
                      : launch_x2<MR, TX, TY, TAB, false, false>(C, G, maps, buf, st, kchunk, kc0, nkc);
  };
  return mr == kMassDefect ? go(std::integral_constant<int, kMassDefect>{})
         : mr == kMassDF   ? go(std::integral_constant<int, kMassDF>{})
                           : go(std::integral_constant<int, kMassDefectDF>{});
}
// The instantiations, by translation unit. shape: kPairShapes' index.
int gbf_launch_x2_fields(int shape, const GbfSplitConsts& C, const GbfSplitGrid& G, int mr, const GbfTmaSet* maps,
                         int buf, cudaStream_t st, int kchunk, int kc0, int nkc);
int gbf_launch_x2_table(int shape, const GbfSplitConsts& C, const GbfSplitGrid& G, int mr, const GbfTmaSet* maps,
                        int buf, cudaStream_t st, int kchunk, int kc0, int nkc);
int gbf_launch_x2_fields_narrow(int shape, const GbfSplitConsts& C, const GbfSplitGrid& G, int mr, const GbfTmaSet* maps,
                                int buf, cudaStream_t st, int kchunk, int kc0, int nkc);
int gbf_launch_x2_table_narrow(int shape, const GbfSplitConsts& C, const GbfSplitGrid& G, int mr, const GbfTmaSet* maps,
                               int buf, cudaStream_t st, int kchunk, int kc0, int nkc);
