// k_expert_mma for IQ3_S weights (expert_mma.cuh).
#define EXPERT_MMA_QT moe::QT_IQ3_S
#include "expert_mma_inst.cuh"
