// Instantiates the fwd time loops of the elman cell.
#define FRNN_INST_CELL CELL_ELMAN
#define FRNN_INST_BWD 0
#define FRNN_INST_LANE lane_fwd_elman
#define FRNN_INST_BIG big_fwd_elman
#define FRNN_INST_PACK big_pack_elman
#include "frnn_inst.cuh"
