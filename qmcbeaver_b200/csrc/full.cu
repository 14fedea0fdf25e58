// full.cu -- instantiations of the full-evaluation / refresh kernel (kernels.cuh).
#include "kernels.cuh"
#include "launches.h"

namespace qmcb {

const void *full_fn(bool mixed, bool extras)
{
  if (mixed) return extras ? (const void *)k_full<float, MIXED_TI, true> : (const void *)k_full<float, MIXED_TI, false>;
  return extras ? (const void *)k_full<double, double, true> : (const void *)k_full<double, double, false>;
}

}  // namespace qmcb
