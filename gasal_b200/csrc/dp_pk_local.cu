/* dp_pk_local.cu -- the packed kernels of LOCAL_ (dp_pk.cuh). */
#include "dp_pk.cuh"

namespace gb {
PkKernel pk_kernel_local(PkVariant v, int start) { return pk_kernel<LOCAL_>(v, start); }
} // namespace gb
