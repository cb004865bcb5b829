// Run-time-length sweeps, double: fused z sweep.
#include "gpe_line_impl.cuh"
namespace gpe {
GPE_LINE_ONE(double, true, FM_Z21)
}  // namespace gpe
