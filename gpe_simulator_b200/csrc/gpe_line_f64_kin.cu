// Run-time-length sweeps, double: x sweep with the kinetic factor.
#include "gpe_line_impl.cuh"
namespace gpe {
GPE_LINE_BOTH(double, false, FM_XKIN)
}  // namespace gpe
