// Run-time-length sweeps, double: diagnostic sweeps.
#include "gpe_line_impl.cuh"
namespace gpe {
GPE_LINE_BOTH(double, true, FM_DIAGR)
GPE_LINE_BOTH(double, false, FM_DIAGK)
GPE_LINE_ONE(double, false, FM_LZ)
}  // namespace gpe
