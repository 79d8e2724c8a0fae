// wg_agg_static.cu — the fused kernel instantiated for every compiled query
// shape (wg_shapes.cuh): one-row, vector and tile-staged variants.
#include "wg_internal.h"
#include "wg_launch.cuh"
#include "wg_star.cuh"

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

void launch_static_shape(const LaunchSpec& ls, cudaStream_t st) {
  using namespace wgd;
  switch (ls.P.shape) {
    case SHAPE_STARJOIN:
      if (launch_star_lean(ls, st)) return;
      launch_pipeline_t<ShapeStarJoin::n_aggs, StatShape<ShapeStarJoin>>(ls, st);
      return;
    case SHAPE_GROUPBY: launch_pipeline_t<ShapeGroupBy::n_aggs, StatShape<ShapeGroupBy>>(ls, st); return;
    case SHAPE_HIGHCARD: launch_pipeline_t<ShapeHighCard::n_aggs, StatShape<ShapeHighCard>>(ls, st); return;
    case SHAPE_BATCH_I64: launch_pipeline_t<ShapeBatchI64::n_aggs, StatShape<ShapeBatchI64>>(ls, st); return;
    case SHAPE_BATCH_F64: launch_pipeline_t<ShapeBatchF64::n_aggs, StatShape<ShapeBatchF64>>(ls, st); return;
    case SHAPE_IPV4: launch_pipeline_t<ShapeIPv4::n_aggs, StatShape<ShapeIPv4>>(ls, st); return;
    default: return;
  }
}

}  // namespace wg
