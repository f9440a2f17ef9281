// gbf_split_table_narrow.cu — the narrower x-pair tiles of grids of the media table.
#include "gbf_split_x2.cuh"

int gbf_launch_x2_table_narrow(int shape, const GbfSplitConsts& C, const GbfSplitGrid& G, int mr, const GbfTmaSet* maps, int buf,
    cudaStream_t st, int kchunk, int kc0, int nkc) {
  return shape == kPair32x16 ? launch_x2_form<32, 16, true, false>(C, G, mr, maps, buf, st, kchunk, kc0, nkc)
                             : launch_x2_form<16, 32, true, false>(C, G, mr, maps, buf, st, kchunk, kc0, nkc);
}
