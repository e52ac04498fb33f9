// Instantiates the bwd time loops of the elmanc cell.
#define FRNN_INST_CELL CELL_ELMAN_CLIP
#define FRNN_INST_BWD 1
#define FRNN_INST_LANE lane_bwd_elmanc
#define FRNN_INST_HELP lane_bwd_help_elmanc
#define FRNN_INST_BIG big_bwd_elmanc
#include "frnn_inst.cuh"
