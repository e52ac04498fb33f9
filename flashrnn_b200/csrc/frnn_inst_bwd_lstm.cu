// Instantiates the bwd time loops of the lstm cell.
#define FRNN_INST_CELL CELL_LSTM
#define FRNN_INST_BWD 1
#define FRNN_INST_LANE lane_bwd_lstm
#define FRNN_INST_HELP lane_bwd_help_lstm
#define FRNN_INST_DR lane_bwd_dr_lstm
#define FRNN_INST_BIG big_bwd_lstm
#include "frnn_inst.cuh"
