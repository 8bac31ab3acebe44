/* dp_pk_global.cu -- the packed kernels of GLOBAL_ (dp_pk.cuh). */
#include "dp_pk.cuh"

namespace gb {
PkKernel pk_kernel_global(PkVariant v, int start) { return pk_kernel<GLOBAL_>(v, start); }
} // namespace gb
