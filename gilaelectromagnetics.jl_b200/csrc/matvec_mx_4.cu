// matvec_mx_4.cu -- mixed-radix passes, lengths listed below.
#include "matvec_mx_impl.cuh"

namespace gila {
GILA_MX_PART(4, 4, 24, 48, 90, 140, 210, 280, 378, 480)
}  // namespace gila
