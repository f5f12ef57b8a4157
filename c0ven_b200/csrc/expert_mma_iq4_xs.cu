// k_expert_mma for IQ4_XS weights.
#define EXPERT_MMA_QT QT_IQ4_XS
#include "expert_mma_inst.cuh"
