// matvec_mx_5.cu -- mixed-radix passes, lengths listed below.
#include "matvec_mx_impl.cuh"

namespace gila {
GILA_MX_PART(5, 96, 28, 42, 98, 126, 216, 270, 392, 450)
}  // namespace gila
