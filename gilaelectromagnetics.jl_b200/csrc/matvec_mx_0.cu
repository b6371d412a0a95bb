// matvec_mx_0.cu -- mixed-radix passes, lengths listed below.
#include "matvec_mx_impl.cuh"

namespace gila {
GILA_MX_PART(0, 64, 12, 14, 60, 70, 162, 168, 320, 324, 504)
}  // namespace gila
