// Run-time-length sweeps, float: fused z sweep.
#include "gpe_line_impl.cuh"
namespace gpe {
GPE_LINE_ONE(float, true, FM_Z21)
}  // namespace gpe
