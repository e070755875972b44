// axg_stream_mono.cu -- the streamed step's kernels for the monopole.
#define AXG_STREAM_POLE axg::POLE_MONO
#include "axg_stream_impl.cuh"
