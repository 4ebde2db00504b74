// General-length axis passes instantiated for storage float, arithmetic double.
#include "fm_generic_impl.cuh"

namespace fm {
FM_BLUE_INST(float, double)
}  // namespace fm
