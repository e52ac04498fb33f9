// Instantiates the fwd time loops of the slstm cell.
#define FRNN_INST_CELL CELL_SLSTM
#define FRNN_INST_BWD 0
#define FRNN_INST_LANE lane_fwd_slstm
#define FRNN_INST_BIG big_fwd_slstm
#define FRNN_INST_PACK big_pack_slstm
#include "frnn_inst.cuh"
