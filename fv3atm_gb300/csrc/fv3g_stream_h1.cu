// fv3g_stream_h1.cu -- the marching FP64 substep, hord 1.
#include "fv3g_stream.cuh"

FV3G_STREAM_INSTANTIATE(1)
