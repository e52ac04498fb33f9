// Instantiates the fwd time loops of the lstm cell.
#define FRNN_INST_CELL CELL_LSTM
#define FRNN_INST_BWD 0
#define FRNN_INST_LANE lane_fwd_lstm
#define FRNN_INST_BIG big_fwd_lstm
#define FRNN_INST_PACK big_pack_lstm
#include "frnn_inst.cuh"
