// gpe_line_impl.cuh -- launch wrappers of the run-time-length sweeps (one translation
// unit per precision and group of modes holds the kernels: gpe_line_<prec>_<group>.cu).
#pragma once
#include "gpe_line.cuh"

namespace gpe {

template <typename K> static cudaError_t line_attr(K kern, int& attr_dev) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (attr_dev == dev) return cudaSuccess;
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, kern);
  int optin = 0;
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
  if (e == cudaSuccess) attr_dev = dev;
  return e;
}

template <typename R, bool ZT, int MODE, int RMAX>
cudaError_t line_one_r(int ax, const Phys& ph, const Sweep& sw, const FastOps& op, const LineGeo& g,
                     const LineShape& sh, size_t smem, cudaStream_t st) {
  constexpr auto kern = &k_line<R, ZT, MODE, RMAX>;
  static int attr_dev = -1;
  const cudaError_t e = line_attr(kern, attr_dev);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)sh.tiles);
  cfg.blockDim = dim3((unsigned)sh.T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = op.pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, ph, sw, op, g, sh, ax);
}

template <typename R, bool ZT, int MODE, int RMAX>
cudaError_t line_batch_one_r(int ax, const Phys* phs, const Sweep* sws, int count, const FastOps& op,
                           const LineGeo& g, const LineShape& sh, size_t smem, cudaStream_t st) {
  constexpr auto kern = &k_line_batch<R, ZT, MODE, RMAX>;
  static int attr_dev = -1;
  const cudaError_t e = line_attr(kern, attr_dev);
  if (e != cudaSuccess) return e;
  kern<<<dim3((unsigned)sh.tiles, (unsigned)count), sh.T, smem, st>>>(phs, sws, op, g, sh, ax);
  return cudaGetLastError();
}

// by the largest radix of the geometry
template <typename R, bool ZT, int MODE>
cudaError_t line_one(int ax, const Phys& ph, const Sweep& sw, const FastOps& op, const LineGeo& g,
                     const LineShape& sh, size_t smem, cudaStream_t st) {
  return g.rmax <= 8 ? line_one_r<R, ZT, MODE, 8>(ax, ph, sw, op, g, sh, smem, st)
                     : line_one_r<R, ZT, MODE, 16>(ax, ph, sw, op, g, sh, smem, st);
}
template <typename R, bool ZT, int MODE>
cudaError_t line_batch_one(int ax, const Phys* phs, const Sweep* sws, int count, const FastOps& op,
                           const LineGeo& g, const LineShape& sh, size_t smem, cudaStream_t st) {
  return g.rmax <= 8 ? line_batch_one_r<R, ZT, MODE, 8>(ax, phs, sws, count, op, g, sh, smem, st)
                     : line_batch_one_r<R, ZT, MODE, 16>(ax, phs, sws, count, op, g, sh, smem, st);
}

#define GPE_LINE_ONE(R, ZT, MODE)                                                                               \
  template cudaError_t line_one<R, ZT, MODE>(int, const Phys&, const Sweep&, const FastOps&, const LineGeo&,   \
                                             const LineShape&, size_t, cudaStream_t);
#define GPE_LINE_BOTH(R, ZT, MODE)                                                                              \
  GPE_LINE_ONE(R, ZT, MODE)                                                                                     \
  template cudaError_t line_batch_one<R, ZT, MODE>(int, const Phys*, const Sweep*, int, const FastOps&,         \
                                                   const LineGeo&, const LineShape&, size_t, cudaStream_t);

}  // namespace gpe
