// Run-time-length sweeps, float: diagnostic sweeps.
#include "gpe_line_impl.cuh"
namespace gpe {
GPE_LINE_BOTH(float, true, FM_DIAGR)
GPE_LINE_BOTH(float, false, FM_DIAGK)
GPE_LINE_ONE(float, false, FM_LZ)
}  // namespace gpe
