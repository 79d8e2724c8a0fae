// wg_agg_lowcard.cu — launches of the shared-memory kernel of plans without a
// compiled shape (wg_lowcard.cuh), in a translation unit of its own.
#include "wg_internal.h"
#include "wg_launch.cuh"
#include "wg_lowcard.cuh"

namespace wg {

int lowcard_threads(int ctas_per_sm) { return wgd::kLcThreads / ctas_per_sm; }
int lowcard_rows(int threads) { return threads * wgd::kLcRows; }

template <int NA>
static void launch_t(const LaunchSpec& ls, cudaStream_t st) {
  cudaFuncSetAttribute(wgd::lowcard_kernel<NA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ls.smem_bytes);
  wgd::lowcard_kernel<NA><<<ls.grid, ls.block, ls.smem_bytes, st>>>(ls.P);
}

void launch_lowcard(const LaunchSpec& ls, cudaStream_t st) {
  if (ls.P.L.n_aggs <= 4) launch_t<4>(ls, st);
  else launch_t<8>(ls, st);
}

}  // namespace wg
