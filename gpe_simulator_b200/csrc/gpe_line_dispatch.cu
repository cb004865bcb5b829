// Dispatch of the run-time-length sweeps by mode.
#include "gpe_line.cuh"

namespace gpe {

template <typename R, bool ZT, int MODE>
cudaError_t line_one(int ax, const Phys& ph, const Sweep& sw, const FastOps& op, const LineGeo& g,
                     const LineShape& sh, size_t smem, cudaStream_t st);
template <typename R, bool ZT, int MODE>
cudaError_t line_batch_one(int ax, const Phys* phs, const Sweep* sws, int count, const FastOps& op,
                           const LineGeo& g, const LineShape& sh, size_t smem, cudaStream_t st);

template <typename R>
cudaError_t launch_line(int ax, const Phys& ph, const Sweep& sw, const FastOps& op, const LineGeo& g,
                        const LineShape& sh, size_t smem, cudaStream_t st) {
  switch (op.mode) {
    case FM_Z1: return line_one<R, true, FM_Z1>(ax, ph, sw, op, g, sh, smem, st);
    case FM_Z2: return line_one<R, true, FM_Z2>(ax, ph, sw, op, g, sh, smem, st);
    case FM_Z21: return line_one<R, true, FM_Z21>(ax, ph, sw, op, g, sh, smem, st);
    case FM_XKIN: return line_one<R, false, FM_XKIN>(ax, ph, sw, op, g, sh, smem, st);
    case FM_DIAGR: return line_one<R, true, FM_DIAGR>(ax, ph, sw, op, g, sh, smem, st);
    case FM_DIAGK: return line_one<R, false, FM_DIAGK>(ax, ph, sw, op, g, sh, smem, st);
    case FM_LZ: return line_one<R, false, FM_LZ>(ax, ph, sw, op, g, sh, smem, st);
    default: break;
  }
  if (ax == FZ) return line_one<R, true, FM_PLAIN>(ax, ph, sw, op, g, sh, smem, st);
  return line_one<R, false, FM_PLAIN>(ax, ph, sw, op, g, sh, smem, st);
}

template <typename R>
cudaError_t launch_line_batch(int ax, const Phys* phs, const Sweep* sws, int count, const FastOps& op,
                              const LineGeo& g, const LineShape& sh, size_t smem, cudaStream_t st) {
  switch (op.mode) {
    case FM_Z1: return line_batch_one<R, true, FM_Z1>(ax, phs, sws, count, op, g, sh, smem, st);
    case FM_Z2: return line_batch_one<R, true, FM_Z2>(ax, phs, sws, count, op, g, sh, smem, st);
    case FM_XKIN: return line_batch_one<R, false, FM_XKIN>(ax, phs, sws, count, op, g, sh, smem, st);
    case FM_DIAGR: return line_batch_one<R, true, FM_DIAGR>(ax, phs, sws, count, op, g, sh, smem, st);
    case FM_DIAGK: return line_batch_one<R, false, FM_DIAGK>(ax, phs, sws, count, op, g, sh, smem, st);
    case FM_PLAIN: break;
    default: return cudaErrorInvalidValue;
  }
  if (ax == FZ) return line_batch_one<R, true, FM_PLAIN>(ax, phs, sws, count, op, g, sh, smem, st);
  return line_batch_one<R, false, FM_PLAIN>(ax, phs, sws, count, op, g, sh, smem, st);
}

#define GPE_LINE_DISPATCH(R)                                                                                     \
  template cudaError_t launch_line<R>(int, const Phys&, const Sweep&, const FastOps&, const LineGeo&,            \
                                      const LineShape&, size_t, cudaStream_t);                              \
  template cudaError_t launch_line_batch<R>(int, const Phys*, const Sweep*, int, const FastOps&, const LineGeo&, \
                                            const LineShape&, size_t, cudaStream_t);
GPE_LINE_DISPATCH(float)
GPE_LINE_DISPATCH(double)

}  // namespace gpe
