// axg_stream_host.h -- launching the streamed step's kernels (axg_stream.cuh),
// which are compiled per pole type in axg_stream_{mono,di,quad}.cu.
#pragma once

#include <cuda_runtime.h>

#include "axg_stream.cuh"

namespace axg {

enum StreamKind { kElemPass = 0, kPointPass = 1 };

// what a launch of a step is: its kernel (streamed: the element blocks come
// from HBM)
struct StreamKernel {
  int kind, mode;
  bool patched, anel, kahan, streamed;
};

// CTAs of a launch's work
inline int32_t stream_blocks(const StreamWork &w) {
  return w.nb_se + w.nb_fe + w.nb_cp + w.nb_si + w.nb_sp + w.nb_fp + w.nb_rec;
}

// One launch for a solve or for several solves (with programmatic stream
// serialization); the memory-variable update of a symplectic step over
// n_groups groups; the element pass's resident CTAs per SM.
template <int POLE>
cudaError_t stream_launch(const StreamKernel &k, const StreamOne &p, const SpecDev &sp, cudaStream_t s);
template <int POLE>
cudaError_t stream_launch(const StreamKernel &k, const StreamMany &p, const SpecDev &sp, cudaStream_t s);
template <int POLE>
cudaError_t stream_memvar(const StreamOne &p, const SpecDev &sp, int32_t n_groups, cudaStream_t s);
template <int POLE>
cudaError_t stream_elem_ctas(const StreamKernel &k, int *per_sm);
#ifdef AXG_DEVICE_CHECKS
template <int POLE>
cudaError_t stream_check_record(int32_t *out8);  // the translation unit's g_axg_check
#endif

}  // namespace axg
