// axg_stream_quad.cu -- the streamed step's kernels for the quadrupole.
#define AXG_STREAM_POLE axg::POLE_QUAD
#include "axg_stream_impl.cuh"
