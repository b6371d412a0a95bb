// matvec_mx_6.cu -- mixed-radix passes, lengths listed below.
#include "matvec_mx_impl.cuh"

namespace gila {
GILA_MX_PART(6, 30, 40, 100, 120, 224, 252, 400, 448)
}  // namespace gila
