// Run-time-length sweeps, float: plain transforms.
#include "gpe_line_impl.cuh"
namespace gpe {
GPE_LINE_BOTH(float, true, FM_PLAIN)
GPE_LINE_BOTH(float, false, FM_PLAIN)
}  // namespace gpe
