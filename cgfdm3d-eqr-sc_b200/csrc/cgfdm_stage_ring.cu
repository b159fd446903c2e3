// The ring pipeline of the CGFDM stage kernel on 32 x 4 tiles.
#define CG_STAGE_SET 4
#include "cgfdm_stage.cu"
