// fv3g_stream_h8.cu -- the marching FP64 substep, hord 8.
#include "fv3g_stream.cuh"

FV3G_STREAM_INSTANTIATE(8)
