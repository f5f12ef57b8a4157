// k_expert_mma for IQ3_XXS weights (expert_mma.cuh).
#define EXPERT_MMA_QT moe::QT_IQ3_XXS
#include "expert_mma_inst.cuh"
