// General-length axis passes instantiated for storage float, arithmetic float.
#include "fm_generic_impl.cuh"

namespace fm {
FM_BLUE_INST(float, float)
}  // namespace fm
