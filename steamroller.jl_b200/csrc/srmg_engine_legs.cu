// srmg_engine_legs.cu -- the persistent kernel's instances for one leg of a V-cycle, the
// coarse levels between them run by a cluster (srmg_coarse.cu).  In a source file of their
// own: beside the whole cycle's instances the compiler stops inlining the phases that
// both call, and a mixed solve takes 2140 us instead of 1820.
#include "srmg_engine.cuh"
#include "srmg_internal.h"

const void *srmg::engine_legs_kernel(int threads) {
  return threads == kEngineNarrow ? (const void *)k_engine_vcycle<double, kEngineNarrow, true>
                                  : (const void *)k_engine_vcycle<double, kEngineWide, true>;
}
