// fv3g_stream_h5.cu -- the marching FP64 substep, hord 5.
#include "fv3g_stream.cuh"

FV3G_STREAM_INSTANTIATE(5)
