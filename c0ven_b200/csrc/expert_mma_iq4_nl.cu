// k_expert_mma for IQ4_NL weights.
#define EXPERT_MMA_QT QT_IQ4_NL
#include "expert_mma_inst.cuh"
