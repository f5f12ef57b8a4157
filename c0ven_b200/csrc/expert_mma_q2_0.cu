// k_expert_mma for Q2_0 weights (expert_mma.cuh).
#define EXPERT_MMA_QT moe::QT_Q2_0
#include "expert_mma_inst.cuh"
