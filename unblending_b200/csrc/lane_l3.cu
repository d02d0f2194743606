// Lane kernels for 3 layer(s).
#define UNB_SOLVER_LAYERS 3
#include "lane_layers.cuh"
