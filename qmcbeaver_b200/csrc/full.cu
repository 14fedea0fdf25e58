// full.cu -- instantiations of the full-evaluation / refresh kernel (kernels.cuh).
#include "kernels.cuh"
#include "launches.h"

namespace qmcb {

template <bool kRest>
static const void *full_fn_of(bool mixed, bool extras)
{
  if (mixed)
    return extras ? (const void *)k_full<float, MIXED_TI, true, kRest> : (const void *)k_full<float, MIXED_TI, false, kRest>;
  return extras ? (const void *)k_full<double, double, true, kRest> : (const void *)k_full<double, double, false, kRest>;
}

const void *full_fn(bool mixed, bool extras, bool rest)
{
  return rest ? full_fn_of<true>(mixed, extras) : full_fn_of<false>(mixed, extras);
}

}  // namespace qmcb
