// Run-time-length sweeps, float: first and last z sweep of a step.
#include "gpe_line_impl.cuh"
namespace gpe {
GPE_LINE_BOTH(float, true, FM_Z1)
GPE_LINE_BOTH(float, true, FM_Z2)
}  // namespace gpe
