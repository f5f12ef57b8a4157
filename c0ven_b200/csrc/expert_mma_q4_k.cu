// k_expert_mma for Q4_K weights.
#define EXPERT_MMA_QT QT_Q4_K
#include "expert_mma_inst.cuh"
