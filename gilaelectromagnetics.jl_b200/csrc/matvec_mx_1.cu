// matvec_mx_1.cu -- mixed-radix passes, lengths listed below.
#include "matvec_mx_impl.cuh"

namespace gila {
GILA_MX_PART(1, 384, 10, 16, 56, 72, 160, 180, 300, 336, 500)
}  // namespace gila
