// wg_agg_static.cu — the fused kernel instantiated for every compiled query
// shape (wg_shapes.cuh): one-row, vector and tile-staged variants.
#include "wg_internal.h"
#include "wg_launch.cuh"
#include "wg_star.cuh"
#include "wg_lean.cuh"
#include "wg_window.cuh"

#include <algorithm>
#include <cstdlib>

namespace wg {

// The star-join shape's lean kernel (wg_star.cuh) when the launch is the
// vector kernel with a shared table and the plan has its physical form
// (WG_STAR_LEAN=0 keeps the generic vector kernel).
template <bool FIXED>
static void launch_star_t(const LaunchSpec& l, cudaStream_t st) {
  cudaFuncSetAttribute(wgd::starjoin_dense_kernel<FIXED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)l.smem_bytes);
  wgd::starjoin_dense_kernel<FIXED><<<l.grid, 768, l.smem_bytes, st>>>(l.P);
}

static bool launch_star_lean(const LaunchSpec& ls, cudaStream_t st) {
  static const bool on = [] {
    const char* v = std::getenv("WG_STAR_LEAN");
    return !v || std::atoi(v) != 0;
  }();
  if (!on || ls.vec == 0 || !ls.smem || ls.tile || ls.stage || ls.block != 768 || !wgd::starjoin_dense_ok(ls.P))
    return false;
  // two words of fixed-point float SUM per slot while two CTAs still fit an SM
  // (ls.smem_bytes holds for two: it was sized for at least one float copy)
  LaunchSpec l = ls;
  constexpr int sw = wgd::ShapeStarJoin::slot_words;
  const int64_t fixed_bytes = (int64_t)l.P.smem_slots * ((sw + 2) | 1) * 8;
  const bool fixed = fixed_bytes <= l.smem_half;
  l.P.smem_rep = fixed ? -1 : 1;
  l.P.smem_sw = fixed ? (sw + 2) | 1 : sw | 1;
  l.smem_bytes = (size_t)l.P.smem_slots * l.P.smem_sw * 8;
  if (fixed) launch_star_t<true>(l, st);
  else launch_star_t<false>(l, st);
  return true;
}

// Shapes that group by one hashed integer key, on the vector path with a shared
// table: lean_group_kernel, one CTA of 1024 threads per SM or two of 512.
template <class C, bool FIXED>
static void launch_lean_t(const LaunchSpec& l, unsigned block, cudaStream_t st) {
  cudaFuncSetAttribute(wgd::lean_group_kernel<C, FIXED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)l.smem_bytes);
  wgd::lean_group_kernel<C, FIXED><<<l.grid, block, l.smem_bytes, st>>>(l.P);
}

template <class C>
static bool launch_lean(const LaunchSpec& ls, cudaStream_t st) {
  if (ls.vec == 0 || !ls.smem || ls.tile) return false;
  LaunchSpec l = ls;
  const bool whole = ls.block == 1024;  // the table takes a whole SM
  constexpr bool any_float = wgd::lean_float_sums<C>() > 0;
  // fixed-point float SUMs widen the slots: taken while the table keeps its CTAs per SM
  const int64_t room = whole ? ls.smem_whole : ls.smem_half;
  const bool fixed = any_float && (int64_t)l.P.smem_slots * wgd::lean_stride<C>(true) * 8 <= room;
  l.P.smem_rep = fixed ? -1 : 1;
  l.P.smem_sw = wgd::lean_stride<C>(fixed);
  l.smem_bytes = (size_t)l.P.smem_slots * l.P.smem_sw * 8;
  const unsigned block = whole ? wgd::kLeanThreads : wgd::kLeanThreads / 2;
  if (fixed) launch_lean_t<C, any_float>(l, block, st);
  else launch_lean_t<C, false>(l, block, st);
  return true;
}

template <class C>
static bool launch_window_t(const LaunchSpec& ls, int sms, cudaStream_t st) {
  const int64_t per = (int64_t)wgd::kWinBlock * wgd::kWinRows;
  const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(2 * sms, (ls.P.n_items + per - 1) / per));
  wgd::window_group_kernel<C><<<grid, wgd::kWinBlock, 0, st>>>(ls.P);
  return true;
}

bool launch_window_static(const LaunchSpec& ls, int sms, cudaStream_t st) {
  using namespace wgd;
  if (ls.vec == 0) return false;  // unaligned columns or a selection
  switch (ls.P.shape) {
    case SHAPE_GROUPBY: return launch_window_t<ShapeGroupBy>(ls, sms, st);
    case SHAPE_BATCH_I64: return launch_window_t<ShapeBatchI64>(ls, sms, st);
    case SHAPE_BATCH_F64: return launch_window_t<ShapeBatchF64>(ls, sms, st);
    case SHAPE_IPV4: return launch_window_t<ShapeIPv4>(ls, sms, st);
    default: return false;
  }
}

void launch_static_shape(const LaunchSpec& ls, cudaStream_t st) {
  using namespace wgd;
  switch (ls.P.shape) {
    case SHAPE_STARJOIN:
      if (launch_star_lean(ls, st)) return;
      launch_pipeline_t<ShapeStarJoin::n_aggs, StatShape<ShapeStarJoin>>(ls, st);
      return;
    case SHAPE_GROUPBY:
      if (launch_lean<ShapeGroupBy>(ls, st)) return;
      launch_pipeline_t<ShapeGroupBy::n_aggs, StatShape<ShapeGroupBy>>(ls, st);
      return;
    case SHAPE_HIGHCARD: launch_pipeline_t<ShapeHighCard::n_aggs, StatShape<ShapeHighCard>>(ls, st); return;
    case SHAPE_BATCH_I64:
      if (launch_lean<ShapeBatchI64>(ls, st)) return;
      launch_pipeline_t<ShapeBatchI64::n_aggs, StatShape<ShapeBatchI64>>(ls, st);
      return;
    case SHAPE_BATCH_F64:
      if (launch_lean<ShapeBatchF64>(ls, st)) return;
      launch_pipeline_t<ShapeBatchF64::n_aggs, StatShape<ShapeBatchF64>>(ls, st);
      return;
    case SHAPE_IPV4:
      if (launch_lean<ShapeIPv4>(ls, st)) return;
      launch_pipeline_t<ShapeIPv4::n_aggs, StatShape<ShapeIPv4>>(ls, st);
      return;
    default: return;
  }
}

}  // namespace wg
