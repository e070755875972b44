// axg_stream_di.cu -- the streamed step's kernels for the dipole.
#define AXG_STREAM_POLE axg::POLE_DI
#include "axg_stream_impl.cuh"
