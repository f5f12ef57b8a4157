// k_expert_mma for Q4_K weights (expert_mma.cuh).
#define EXPERT_MMA_QT moe::QT_Q4_K
#include "expert_mma_inst.cuh"
