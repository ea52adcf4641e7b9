// Path pools with the basic vertex programs, and with smooth translucent objects.  The 16-round draw is
// compiled once, out of line (PT_OUTLINE_TEA): beside the traversal and the other programs its inlined
// copies overflow the instruction cache.
#define PT_OUTLINE_TEA
#include "pt_pool.cuh"

namespace pt {

pt_status launch_path_pools(const SceneDev& S0, const WfDev& w, uint64_t n, bool multi, bool adjoint, PoolPrograms programs, int refill,
                            cudaStream_t stream)
{
  if (programs == POOL_ALL) return launch_path_pools_all(S0, w, n, multi, adjoint, refill, stream);
  if (adjoint) return launch_pool_scenes<true, POOL_TRANSLUCENT>(S0, w, n, multi, refill, stream);
  if (programs == POOL_TRANSLUCENT) return launch_pool_scenes<false, POOL_TRANSLUCENT>(S0, w, n, multi, refill, stream);
  return launch_pool_scenes<false, POOL_BASIC>(S0, w, n, multi, refill, stream);
}

}  // namespace pt
