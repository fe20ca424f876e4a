// Even-model stages in FP64.
#include "even_impl.cuh"

namespace pgb {
PGB_EVEN_INST(double)
}  // namespace pgb
