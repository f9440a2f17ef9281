// gbf_split_fields_narrow.cu — the narrower x-pair tiles of grids with K and porosity fields.
#include "gbf_split_x2.cuh"

int gbf_launch_x2_fields_narrow(int shape, const GbfSplitConsts& C, const GbfSplitGrid& G, int mr, const GbfTmaSet* maps, int buf,
    cudaStream_t st, int kchunk, int kc0, int nkc) {
  return shape == kPair32x16 ? launch_x2_form<32, 16, false, false>(C, G, mr, maps, buf, st, kchunk, kc0, nkc)
                             : launch_x2_form<16, 32, false, false>(C, G, mr, maps, buf, st, kchunk, kc0, nkc);
}
