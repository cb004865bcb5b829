// Run-time-length sweeps, double: first and last z sweep of a step.
#include "gpe_line_impl.cuh"
namespace gpe {
GPE_LINE_BOTH(double, true, FM_Z1)
GPE_LINE_BOTH(double, true, FM_Z2)
}  // namespace gpe
