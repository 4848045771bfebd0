// FP64 row-group instances of the TMA step, compiled beside the others (fit_tma.cu).
#define WK_TMA_TYPE double
#define WK_TMA_PART WK_TMA_TYPE, true
#include "fit_tma.cu"
