// k_expert_mma for Q6_K weights (expert_mma.cuh).
#define EXPERT_MMA_QT moe::QT_Q6_K
#include "expert_mma_inst.cuh"
