/* dp_pk_semi.cu -- the packed kernels of SEMI_GLOBAL_ (dp_pk.cuh). */
#include "dp_pk.cuh"

namespace gb {
PkKernel pk_kernel_semi(PkVariant v, int start) { return pk_kernel<SEMI_GLOBAL_>(v, start); }
} // namespace gb
