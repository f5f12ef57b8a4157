// k_expert_mma for Q8_0 weights (expert_mma.cuh).
#define EXPERT_MMA_QT moe::QT_Q8_0
#include "expert_mma_inst.cuh"
