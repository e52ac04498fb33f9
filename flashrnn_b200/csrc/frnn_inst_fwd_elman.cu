// Instantiates the fwd time loops of the elman cell.
#define FRNN_INST_CELL CELL_ELMAN
#define FRNN_INST_BWD 0
#define FRNN_INST_LANE lane_fwd_elman
#define FRNN_INST_STREAM stream_fwd_elman
#include "frnn_inst.cuh"
