// wg_agg_lowcard.cu — launches of the column-at-a-time kernel of plans without a
// compiled shape (wg_lowcard.cuh), with its groups in shared memory or in a
// key window, and of the kernels around a window (wg_window.cuh).
#include "wg_internal.h"
#include "wg_launch.cuh"
#include "wg_window.cuh"

#include <algorithm>

namespace wg {

int lowcard_threads(int ctas_per_sm) { return wgd::kLcThreads / ctas_per_sm; }
int lowcard_rows(int threads) { return threads * wgd::kLcRows; }

template <int NA>
static void launch_t(const LaunchSpec& ls, cudaStream_t st) {
  cudaFuncSetAttribute(wgd::lowcard_kernel<NA, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ls.smem_bytes);
  wgd::lowcard_kernel<NA, true><<<ls.grid, ls.block, ls.smem_bytes, st>>>(ls.P);
}

// The window of the launch, then its slots (at most `slots`), empty.
void launch_window_begin(const LaunchSpec& ls, int sms, cudaStream_t st) {
  wgd::KeyWindow* w = const_cast<wgd::KeyWindow*>(ls.P.win);
  if (ls.win_known) wgd::window_set_kernel<<<1, 1, 0, st>>>(wgd::KeyWindow{ls.win_base, (unsigned long long)ls.win_slots}, w);
  else wgd::window_sample_kernel<<<1, wgd::kWinThreads, 0, st>>>(ls.P, (unsigned long long)ls.win_slots, w);
  const int64_t words = ls.win_slots * ls.P.L.slot_words;
  wgd::window_init_kernel<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(sms * 8, words / 2048)), 256, 0, st>>>(ls.P);
}

void launch_window_rows(const LaunchSpec& ls, int sms, cudaStream_t st) {
  const int block = wgd::kLcThreads / 2;
  const int64_t per = (int64_t)block * wgd::kLcRows;
  const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(2 * sms, (ls.P.n_items + per - 1) / per));
  if (ls.P.L.n_aggs <= 4) wgd::lowcard_kernel<4, false><<<grid, block, 0, st>>>(ls.P);
  else wgd::lowcard_kernel<8, false><<<grid, block, 0, st>>>(ls.P);
}

void launch_window_fold(const LaunchSpec& ls, int sms, cudaStream_t st) {
  const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(sms * 8, (ls.win_slots + 255) / 256));
  if (ls.P.L.n_aggs <= 4) wgd::window_fold_kernel<4><<<grid, 256, 0, st>>>(ls.P);
  else wgd::window_fold_kernel<8><<<grid, 256, 0, st>>>(ls.P);
}

void launch_lowcard(const LaunchSpec& ls, cudaStream_t st) {
  if (ls.P.L.n_aggs <= 4) launch_t<4>(ls, st);
  else launch_t<8>(ls, st);
}

}  // namespace wg
