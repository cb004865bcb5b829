// Run-time-length sweeps, double: plain transforms.
#include "gpe_line_impl.cuh"
namespace gpe {
GPE_LINE_BOTH(double, true, FM_PLAIN)
GPE_LINE_BOTH(double, false, FM_PLAIN)
}  // namespace gpe
