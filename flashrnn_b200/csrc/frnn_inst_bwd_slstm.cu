// Instantiates the bwd time loops of the slstm cell.
#define FRNN_INST_CELL CELL_SLSTM
#define FRNN_INST_BWD 1
#define FRNN_INST_LANE lane_bwd_slstm
#define FRNN_INST_HELP lane_bwd_help_slstm
#define FRNN_INST_DR lane_bwd_dr_slstm
#define FRNN_INST_BIG big_bwd_slstm
#include "frnn_inst.cuh"
