// move.cu -- instantiations of the one-determinant move kernel (kernels.cuh).
#include "kernels.cuh"
#include "launches.h"

namespace qmcb {

template <bool kMetropolis, typename TS, typename TI>
static const void *move_fn_of(bool extras, bool ginv)
{
  if (ginv)
    return extras ? (const void *)k_move<kMetropolis, TS, TI, true, true, false>
                  : (const void *)k_move<kMetropolis, TS, TI, false, true, false>;
  return extras ? (const void *)k_move<kMetropolis, TS, TI, true, false, false>
                : (const void *)k_move<kMetropolis, TS, TI, false, false, false>;
}

const void *move_dense_fn(bool metropolis)
{
  return metropolis ? (const void *)k_move<true, double, double, true, false, true>
                    : (const void *)k_move<false, double, double, true, false, true>;
}

const void *move_fn(bool metropolis, bool mixed, bool extras, bool ginv)
{
  if (mixed)
    return metropolis ? move_fn_of<true, float, MIXED_TI>(extras, ginv) : move_fn_of<false, float, MIXED_TI>(extras, ginv);
  return metropolis ? move_fn_of<true, double, double>(extras, ginv) : move_fn_of<false, double, double>(extras, ginv);
}

}  // namespace qmcb
