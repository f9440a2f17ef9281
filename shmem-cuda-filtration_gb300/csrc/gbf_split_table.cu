// gbf_split_table.cu — the 64x8 x-pair tile of grids of the media table (the
// drop-in's physics, and homogeneous grids).
#include "gbf_split_x2.cuh"

int gbf_launch_x2_table(int shape, const GbfSplitConsts& C, const GbfSplitGrid& G, int mr, const GbfTmaSet* maps, int buf,
    cudaStream_t st, int kchunk, int kc0, int nkc) {
  if (shape != kPair64x8) return gbf_launch_x2_table_narrow(shape, C, G, mr, maps, buf, st, kchunk, kc0, nkc);
  return launch_x2_form<64, 8, true, true>(C, G, mr, maps, buf, st, kchunk, kc0, nkc);
}
