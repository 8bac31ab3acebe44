/* dp_pk_semi.cu -- the packed kernels of SEMI_GLOBAL_ (dp_pk.cuh). */
#include "dp_pk.cuh"

namespace gb {
cudaError_t pk_visit_semi(int group, int start, bool fast, const PkLaunchFn &f)
{
    return pk_visit<SEMI_GLOBAL_>(group, start, fast, f);
}
} // namespace gb
