// FP32 instances of the TMA step, compiled beside the others (fit_tma.cu).
#define WK_TMA_TYPE float
#define WK_TMA_PART WK_TMA_TYPE, false
#include "fit_tma.cu"
