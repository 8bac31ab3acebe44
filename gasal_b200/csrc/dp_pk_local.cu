/* dp_pk_local.cu -- the packed kernels of LOCAL_ (dp_pk.cuh). */
#include "dp_pk.cuh"

namespace gb {
cudaError_t pk_visit_local(int group, int start, bool fast, const PkLaunchFn &f)
{
    return pk_visit<LOCAL_>(group, start, fast, f);
}
} // namespace gb
