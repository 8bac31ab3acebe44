/* dp_pk_global.cu -- the packed kernels of GLOBAL_ (dp_pk.cuh). */
#include "dp_pk.cuh"

namespace gb {
cudaError_t pk_visit_global(int group, int start, bool fast, const PkLaunchFn &f)
{
    return pk_visit<GLOBAL_>(group, start, fast, f);
}
} // namespace gb
