// k_expert_mma for Q8_0 weights.
#define EXPERT_MMA_QT QT_Q8_0
#include "expert_mma_inst.cuh"
