// gbf_split_fields.cu — the 64x8 x-pair tile of grids with K and porosity fields.
#include "gbf_split_x2.cuh"

int gbf_launch_x2_fields(int shape, const GbfSplitConsts& C, const GbfSplitGrid& G, int mr, const GbfTmaSet* maps, int buf,
    cudaStream_t st, int kchunk, int kc0, int nkc) {
  if (shape != kPair64x8) return gbf_launch_x2_fields_narrow(shape, C, G, mr, maps, buf, st, kchunk, kc0, nkc);
  return launch_x2_form<64, 8, false, true>(C, G, mr, maps, buf, st, kchunk, kc0, nkc);
}
