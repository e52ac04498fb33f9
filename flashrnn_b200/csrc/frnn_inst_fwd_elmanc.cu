// Instantiates the fwd time loops of the elmanc cell.
#define FRNN_INST_CELL CELL_ELMAN_CLIP
#define FRNN_INST_BWD 0
#define FRNN_INST_LANE lane_fwd_elmanc
#define FRNN_INST_BIG big_fwd_elmanc
#define FRNN_INST_PACK big_pack_elmanc
#include "frnn_inst.cuh"
