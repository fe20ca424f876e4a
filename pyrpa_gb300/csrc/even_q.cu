// Even-model stages in double-float.
#include "even_impl.cuh"

namespace pgb {
PGB_EVEN_INST(dfl)
}  // namespace pgb
