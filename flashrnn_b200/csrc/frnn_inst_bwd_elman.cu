// Instantiates the bwd time loops of the elman cell.
#define FRNN_INST_CELL CELL_ELMAN
#define FRNN_INST_BWD 1
#define FRNN_INST_LANE lane_bwd_elman
#define FRNN_INST_HELP lane_bwd_help_elman
#define FRNN_INST_BIG big_bwd_elman
#include "frnn_inst.cuh"
