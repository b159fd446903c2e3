// The CGFDM stage kernel with mixed-precision storage (32 x 4 tiles).
#define CG_STAGE_SET 2
#include "cgfdm_stage.cu"
