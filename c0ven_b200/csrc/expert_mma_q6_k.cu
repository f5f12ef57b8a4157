// k_expert_mma for Q6_K weights.
#define EXPERT_MMA_QT QT_Q6_K
#include "expert_mma_inst.cuh"
