// axg_stream_impl.cuh -- the launchers of axg_stream_host.h for one pole type
// (AXG_STREAM_POLE, set by the file that includes this).
#include "axg_stream_host.h"

namespace axg {
namespace {

template <class... KArgs, class... Args>
cudaError_t launch(void (*kernel)(KArgs...), unsigned grid, cudaStream_t s, bool pdl, Args &&...args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kGrpThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

unsigned blocks(const StreamOne &p) { return (unsigned)stream_blocks(p.w); }
unsigned blocks(const StreamMany &p) { return (unsigned)p.start[p.n]; }

// CTAs per SM of the scattered element pass.  Quadrupole steps, 4 / 3 CTAs: from
// L2 12.9 / 14.0 us on 13 390 elements, from HBM 20.1 / 17.0 on 18 944, 23.9 /
// 23.6 on 25 802, 32.4 / 33.2 on 32 298 (3 waves either way), 73.2 / 71.3 on
// 70 528.  Stiffness calls likewise: 15.9 / 13.9 us on 16 900, 53.3 / 51.3 on 62 500,
// 103.6 / 100.1 on 129 600; dipole 14.6 / 12.7, 49.4 / 44.5, 95.5 / 86.8.  Several solves' launches, whose waves fill, keep 4: six solves on
// 5 664 and 18 944 elements 9.67 / 9.95 ms for 96 steps.
template <int POLE, int MODE, bool ANEL, bool KAHAN, class P>
auto scatter_of(const StreamKernel &k) -> void (*)(P, SpecDev) {
  if constexpr (ANEL) return scatter_kernel<POLE, MODE, ANEL, KAHAN, 3, P>;
  else if constexpr (POLE == POLE_MONO || P::kMany) return scatter_kernel<POLE, MODE, ANEL, KAHAN, 4, P>;
  else return k.streamed ? scatter_kernel<POLE, MODE, ANEL, KAHAN, 3, P> : scatter_kernel<POLE, MODE, ANEL, KAHAN, 4, P>;
}

template <int POLE, int MODE, bool KAHAN, class P>
auto patched_or(const StreamKernel &k) -> void (*)(P, SpecDev) {
  return k.patched ? patch_kernel<POLE, MODE, KAHAN, P> : scatter_of<POLE, MODE, false, KAHAN, P>(k);
}

// The scattered element pass of a Newmark step does not depend on the
// precision mode (it reads the stored prediction); the patched one also
// finishes points.
template <int POLE, class P>
auto elem_kernel(const StreamKernel &k) -> void (*)(P, SpecDev) {
  if (k.mode == MODE_FORCE) return patched_or<POLE, MODE_FORCE, false, P>(k);
  if (k.mode == MODE_NEWMARK) {
    if (!k.patched)
      return k.anel ? scatter_of<POLE, MODE_NEWMARK, true, false, P>(k)
                    : scatter_of<POLE, MODE_NEWMARK, false, false, P>(k);
    return k.kahan ? patch_kernel<POLE, MODE_NEWMARK, true, P> : patch_kernel<POLE, MODE_NEWMARK, false, P>;
  }
  if (k.anel)
    return k.kahan ? scatter_of<POLE, MODE_SYMPLECTIC, true, true, P>(k)
                   : scatter_of<POLE, MODE_SYMPLECTIC, true, false, P>(k);
  return k.kahan ? patched_or<POLE, MODE_SYMPLECTIC, true, P>(k) : patched_or<POLE, MODE_SYMPLECTIC, false, P>(k);
}

template <int POLE, int MODE, class P>
auto point_kernel_of(const StreamKernel &k) -> void (*)(P) {
  if (k.patched) return k.kahan ? point_kernel<POLE, MODE, true, true, P> : point_kernel<POLE, MODE, true, false, P>;
  return k.kahan ? point_kernel<POLE, MODE, false, true, P> : point_kernel<POLE, MODE, false, false, P>;
}

template <int POLE, class P>
cudaError_t launch_step(const StreamKernel &k, const P &p, const SpecDev &sp, cudaStream_t s) {
  if (k.kind == kElemPass) return launch(elem_kernel<POLE, P>(k), blocks(p), s, true, p, sp);
  auto fn = k.mode == MODE_NEWMARK      ? point_kernel_of<POLE, MODE_NEWMARK, P>(k)
            : k.mode == MODE_SYMPLECTIC ? point_kernel_of<POLE, MODE_SYMPLECTIC, P>(k)
            : k.patched                 ? point_kernel<POLE, MODE_FORCE, true, false, P>
                                        : point_kernel<POLE, MODE_FORCE, false, false, P>;
  return launch(fn, blocks(p), s, true, p);
}

}  // namespace

template <int POLE>
cudaError_t stream_launch(const StreamKernel &k, const StreamOne &p, const SpecDev &sp, cudaStream_t s) {
  return launch_step<POLE>(k, p, sp, s);
}
template <int POLE>
cudaError_t stream_launch(const StreamKernel &k, const StreamMany &p, const SpecDev &sp, cudaStream_t s) {
  return launch_step<POLE>(k, p, sp, s);
}

template <int POLE>
cudaError_t stream_memvar(const StreamOne &p, const SpecDev &sp, int32_t n_groups, cudaStream_t s) {
  return launch(memvar_kernel<POLE>, (unsigned)((n_groups + kGrpWarps - 1) / kGrpWarps), s, false, p, sp, n_groups);
}

template <int POLE>
cudaError_t stream_elem_ctas(const StreamKernel &k, int *per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, elem_kernel<POLE, StreamOne>(k), kGrpThreads, 0);
}

#ifdef AXG_DEVICE_CHECKS
template <int POLE>
cudaError_t stream_check_record(int32_t *out8) {
  return cudaMemcpyFromSymbol(out8, g_axg_check, 8 * sizeof(int32_t));
}
template cudaError_t stream_check_record<AXG_STREAM_POLE>(int32_t *);
#endif

template cudaError_t stream_launch<AXG_STREAM_POLE>(const StreamKernel &, const StreamOne &, const SpecDev &,
                                                    cudaStream_t);
template cudaError_t stream_launch<AXG_STREAM_POLE>(const StreamKernel &, const StreamMany &, const SpecDev &,
                                                    cudaStream_t);
template cudaError_t stream_memvar<AXG_STREAM_POLE>(const StreamOne &, const SpecDev &, int32_t, cudaStream_t);
template cudaError_t stream_elem_ctas<AXG_STREAM_POLE>(const StreamKernel &, int *);

}  // namespace axg
