// full.cu -- instantiations of the full-evaluation / refresh kernel (kernels.cuh).
#include "kernels.cuh"
#include "launches.h"

namespace qmcb {

template <bool kRest>
static const void *full_fn_of(bool mixed, bool extras)
{
  if (mixed)
    return extras ? (const void *)k_full<float, MIXED_TI, true, kRest, false>
                  : (const void *)k_full<float, MIXED_TI, false, kRest, false>;
  return extras ? (const void *)k_full<double, double, true, kRest, false>
                : (const void *)k_full<double, double, false, kRest, false>;
}

const void *rest_dense_fn(bool mixed)
{
  return mixed ? (const void *)k_full<float, MIXED_TI, true, true, true>
               : (const void *)k_full<double, double, true, true, true>;
}

const void *full_fn(bool mixed, bool extras, bool rest)
{
  return rest ? full_fn_of<true>(mixed, extras) : full_fn_of<false>(mixed, extras);
}

}  // namespace qmcb
