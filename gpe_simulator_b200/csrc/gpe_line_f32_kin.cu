// Run-time-length sweeps, float: x sweep with the kinetic factor.
#include "gpe_line_impl.cuh"
namespace gpe {
GPE_LINE_BOTH(float, false, FM_XKIN)
}  // namespace gpe
