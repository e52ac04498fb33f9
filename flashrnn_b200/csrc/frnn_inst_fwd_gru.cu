// Instantiates the fwd time loops of the gru cell.
#define FRNN_INST_CELL CELL_GRU
#define FRNN_INST_BWD 0
#define FRNN_INST_LANE lane_fwd_gru
#define FRNN_INST_STREAM stream_fwd_gru
#include "frnn_inst.cuh"
