// matvec_mx_3.cu -- mixed-radix passes, lengths listed below.
#include "matvec_mx_impl.cuh"

namespace gila {
GILA_MX_PART(3, 192, 6, 20, 50, 84, 144, 200, 288, 360, 486)
}  // namespace gila
