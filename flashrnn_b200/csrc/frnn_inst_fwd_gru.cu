// Instantiates the fwd time loops of the gru cell.
#define FRNN_INST_CELL CELL_GRU
#define FRNN_INST_BWD 0
#define FRNN_INST_LANE lane_fwd_gru
#define FRNN_INST_BIG big_fwd_gru
#define FRNN_INST_PACK big_pack_gru
#include "frnn_inst.cuh"
