// General-length axis passes instantiated for storage double, arithmetic double.
#include "fm_generic_impl.cuh"

namespace fm {
FM_BLUE_INST(double, double)
}  // namespace fm
