// The CGFDM stage kernel of halo-linked parts (32 x 4 tiles).
#define CG_STAGE_SET 3
#include "cgfdm_stage.cu"
