// Instantiates the bwd time loops of the gru cell.
#define FRNN_INST_CELL CELL_GRU
#define FRNN_INST_BWD 1
#define FRNN_INST_LANE lane_bwd_gru
#define FRNN_INST_HELP lane_bwd_help_gru
#define FRNN_INST_DR lane_bwd_dr_gru
#define FRNN_INST_BIG big_bwd_gru
#include "frnn_inst.cuh"
