// k_expert_mma for IQ4_NL weights (expert_mma.cuh).
#define EXPERT_MMA_QT moe::QT_IQ4_NL
#include "expert_mma_inst.cuh"
