// wg_window.cuh — GROUP BY over one integer key drawn from a range of up to a few
// hundred thousand values: the groups' state in HBM (resident in L2), indexed by key - base.
//
// Between what fits a CTA's shared memory and the tables of tens of millions of
// groups (wg_hc.cuh), a row of the HBM hash table costs a key read that everything
// else waits for, a warp-wide match for rows of one group, and then an L2 atomic per
// sum. Identifiers, codes, prefixes and string ids mostly come from a range
// not much wider than their distinct count: then the slot is an offset, nothing is read
// before the updates, and the bound is the L2 atomics (10^8 rows into 65536 groups, a sum
// and a count each: 1228 us, 163 G atomics/s of the 190 measured at most, against
// 2262 us through the hash table; 2 * 10^7 rows of string ids into 10^5 groups 342
// against 869 us).
//
// A one-CTA kernel samples the input (kWinSamples rows, spread over it) and sets the
// window, none when the sampled keys span more slots than the buffer holds or when
// some key is so frequent that its atomics would serialise (the hash-table
// kernel combines such rows per warp first). The window kernel and the
// hash-table kernel are both launched; the one the sample did not choose returns at
// once, so the host waits for nothing. Rows outside the window update the hash table
// directly. A last kernel folds the window's groups into it.
#pragma once

#include "wg_lowcard.cuh"

namespace wgd {

constexpr int kWinThreads = 1024;
constexpr int kWinSamples = 8 * kWinThreads;
constexpr int kWinBins = 8192;
// Sampled rows of one bin (of kWinBins, by key hash) from which a key counts as hot: 0.5% of the rows.
constexpr uint32_t kWinHot = 40;

// The window of a launch, from a sample of the plan's rows (no join).
static __global__ void __launch_bounds__(kWinThreads) window_sample_kernel(const __grid_constant__ Plan P,
                                                                           unsigned long long slots, KeyWindow* out) {
  __shared__ uint32_t bin[kWinBins];
  __shared__ long long s_lo, s_hi;
  __shared__ unsigned s_most;
  for (int i = threadIdx.x; i < kWinBins; i += kWinThreads) bin[i] = 0;
  if (threadIdx.x == 0) { s_lo = 0x7FFFFFFFFFFFFFFFLL; s_hi = -0x7FFFFFFFFFFFFFFFLL - 1; s_most = 0; }
  __syncthreads();
  const DynShape sh{P};
  long long lo = 0x7FFFFFFFFFFFFFFFLL, hi = -0x7FFFFFFFFFFFFFFFLL - 1;
  for (int s = threadIdx.x; s < kWinSamples; s += kWinThreads) {
    const int64_t item = (P.n_items / kWinSamples) * s + (P.n_items % kWinSamples) * s / kWinSamples;
    const SrcGlobal src{P.sel ? (int64_t)__ldg(P.sel + item) : item};
    ExprVals ev;
    eval_exprs(P, sh, src, -1, ev);
    const Val v = fetch(P, sh, src, P.L.key_vcol[0], -1, ev);
    if (v.null) continue;
    const long long k = (long long)v.lo;
    lo = k < lo ? k : lo;
    hi = k > hi ? k : hi;
    atomicAdd(&bin[(uint32_t)((v.lo * 0x9E3779B97F4A7C15ULL) >> 51)], 1u);
  }
  for (int o = 16; o > 0; o >>= 1) {
    const long long l2 = __shfl_down_sync(WG_FULL_MASK, lo, o), h2 = __shfl_down_sync(WG_FULL_MASK, hi, o);
    lo = l2 < lo ? l2 : lo;
    hi = h2 > hi ? h2 : hi;
  }
  if ((threadIdx.x & 31) == 0) { atomicMin(&s_lo, lo); atomicMax(&s_hi, hi); }
  __syncthreads();
  unsigned most = 0;
  for (int i = threadIdx.x; i < kWinBins; i += kWinThreads) most = max(most, bin[i]);
  most = __reduce_max_sync(WG_FULL_MASK, most);
  if ((threadIdx.x & 31) == 0) atomicMax(&s_most, most);
  __syncthreads();
  if (threadIdx.x != 0) return;
  const unsigned long long last = (unsigned long long)s_hi - (unsigned long long)s_lo;  // span - 1
  KeyWindow w;
  w.base = 0;
  w.n = 0;
  if (s_hi >= s_lo && last < slots && s_most < kWinHot) {
    // room on both sides for keys the sample missed
    const unsigned long long n = min(slots, last + 1 + (last >> 3) + 64);
    w.n = n;
    w.base = (long long)((unsigned long long)s_lo - (n - 1 - last) / 2);
  }
  *out = w;
}

// A window known beforehand (a join payload's value range, a dictionary's ids).
static __global__ void window_set_kernel(KeyWindow w, KeyWindow* out) { *out = w; }

// The window's slots, empty.
static __global__ void window_init_kernel(const __grid_constant__ Plan P) {
  __shared__ unsigned long long init[WG_MAX_SLOT_WORDS];
  const int sw = P.L.slot_words;
  if (threadIdx.x < (unsigned)sw) init[threadIdx.x] = P.L.init[threadIdx.x];
  __syncthreads();
  fill_pattern(P.wslots, (int64_t)P.win->n * sw, sw, sw, init, (int64_t)blockIdx.x * blockDim.x + threadIdx.x,
               (int64_t)gridDim.x * blockDim.x);
}

// The window's groups into the hash table.
template <int NA>
__global__ void window_fold_kernel(const __grid_constant__ Plan P) {
  Credit cr;
  const LayoutAcc ly{P.L};
  const int sw = P.L.slot_words;
  const KeyWindow w = *P.win;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < w.n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long* s = P.wslots + i * sw;
    const unsigned long long rows = s[1];
    if (rows == 0) continue;
    unsigned long long* g = find_global(ly, P.T, (unsigned long long)w.base + i, 0, false, P.err, &cr);
    if (g == nullptr) continue;
    Contrib<NA> c;
    slot_contrib<NA>(ly, s, c);
    apply<NA, false>(ly, g, c, rows);
  }
  cr.release(P.T);
}

// The rows of a compiled shape without a join: kWinRows per lane, their updates
// in flight together.
constexpr int kWinRows = 4;
constexpr int kWinBlock = 512;
template <class C>
__global__ void __launch_bounds__(kWinBlock, 2) window_group_kernel(const __grid_constant__ Plan P) {
  static_assert(C::key_words == 1 && C::has_join == 0, "one integer key, no join");
  const KeyWindow w = *P.win;
  if (w.n == 0) return;
  constexpr int U = kWinRows, NA = C::n_aggs;
  const StatShape<C> sh{P};
  Credit cr;
  const int lane = threadIdx.x & 31;
  const int64_t step = (int64_t)gridDim.x * (blockDim.x >> 5) * (32 * U);
  int64_t base = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 * U);
  const bool test = P.minmax_test != 0;
  FarQueue queue;
  far_init(queue, base);
  for (;;) {
    unsigned far = 0;
    for (; base < P.n_items; base += step) {
      const int64_t r0 = base + (int64_t)lane * U;
      SrcRow rw[U];
      load_rows<U>(P, sh, r0, rw);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        bool a = r0 + u < P.n_items;
#pragma unroll
        for (int f = 0; f < C::n_filters; ++f) a = a && pred_val(P, sh, f, rw[u].v[C::filt_col(f)]);
        if (!a) continue;
        ExprVals ev;
        eval_exprs(P, sh, rw[u], -1, ev);
        const unsigned long long d = fetch(P, sh, rw[u], C::key_vcol(0), -1, ev).lo - (unsigned long long)w.base;
        if (d >= w.n) { far |= 1u << u; continue; }
        Contrib<NA> c;
        make_contrib<NA>(P, sh, rw[u], -1, ev, c);
        apply<NA, false>(sh, P.wslots + d * C::slot_words, c, 1ULL, 1, test);
      }
      if (__any_sync(WG_FULL_MASK, far != 0)) break;
    }
    if (base >= P.n_items) break;
    far_rows<StatShape<C>, U, false>(P, &queue, far, &cr, base + (int64_t)lane * U);
    base += step;
  }
  far_flush<StatShape<C>>(P, &queue, &cr);
  cr.release(P.T);
}

}  // namespace wgd
