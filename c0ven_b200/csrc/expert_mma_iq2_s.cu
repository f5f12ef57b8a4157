// k_expert_mma for IQ2_S weights (expert_mma.cuh).
#define EXPERT_MMA_QT moe::QT_IQ2_S
#include "expert_mma_inst.cuh"
