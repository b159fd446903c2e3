// The fused CGFDM stage with 32 x 8 column tiles (two CTAs per SM), in
// namespace cgfdm::ty8: the same source as cgfdm_stage.cu, compiled for the
// other tile height, for batches and the ring pipeline (the split pipeline
// sweeps a 32 x 8 item in two 4-row sweeps).
#define CG_TILE_Y 8
#define CG_CTAS_PER_SM 2
#define CG_TILE_NS ty8
#include "cgfdm_stage.cu"
