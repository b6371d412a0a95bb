// matvec_mx_2.cu -- mixed-radix passes, lengths listed below.
#include "matvec_mx_impl.cuh"

namespace gila {
GILA_MX_PART(2, 8, 18, 54, 80, 150, 196, 294, 350, 490)
}  // namespace gila
