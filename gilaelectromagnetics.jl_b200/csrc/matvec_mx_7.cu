// matvec_mx_7.cu -- mixed-radix passes, lengths listed below.
#include "matvec_mx_impl.cuh"

namespace gila {
GILA_MX_PART(7, 32, 36, 108, 112, 240, 250, 420, 432)
}  // namespace gila
