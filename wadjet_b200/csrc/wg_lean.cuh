// wg_lean.cuh — the row loop of compiled shapes that group by one hashed integer key in
// a CTA's shared-memory table, with every launch choice fixed at compile time.
//
// pipeline_vec_kernel serves every physical form of a shape (dense or hashed
// groups, float-SUM copies, warp combine, HBM-table rows), deciding per row
// from the plan: 234 warp instructions per 32 rows of the group-by shape, whose
// shared-memory work is five operations, so it was bound by instruction issue
// (1969 us at 2^28 rows, 4096 groups; 1405 here; the columns take 1149 us at the
// copy peak). Here a row is its loads, the comparison, a 32-bit multiply-shift hash,
// one key read and its updates; the first probes of a lane's rows are read
// together. Float SUMs accumulate in scaled fixed point (f64_to_fixed_scaled)
// while the wider slots leave the table its CTAs per SM.
//
// Keys drawn from a range no larger than the table (identifiers, codes) need no
// hash: each CTA samples one row per thread, spread over the input, and when the
// sampled keys span at most the table's slots, slot = key - base for a window
// around them. (4096 keys hashed into 5760 slots take 2.2 probes on average.)
//
// A row whose key finds no slot (outside the window, the table at its fill limit,
// no free slot within kLeanProbes steps, the key equal to the empty pattern) goes to
// the HBM table, 32 of a warp's at a time, by the shape's own code. (2^24 rows into 3000
// sparse keys with a hint of 300, a sixth of them without a slot: 1.95 ms a row at a time and
// interpreted, 0.54 so.)
#pragma once

#include "wg_lowcard.cuh"

namespace wgd {

// Rows per lane and an L2 prefetch two chunks ahead, group-by shape at 2^28 rows
// and 4096 groups (with rows for the HBM table handled in the loop, 1570 us as it was then): 4
// without 1570, 2 without 1673, 4 with 1832, 2 with 1831 us; the next chunk's loads held
// in registers (spills) 2962 with 4 and 3141 with 2.
constexpr int kLeanRows = 4;
constexpr int kLeanProbes = 16;    // slots a key is looked for in (two in a thousand keys of a table 3/4 full need more)
constexpr int kLeanThreads = 1024; // per SM (64 registers each), in one CTA or two

template <class C>
constexpr int lean_float_sums() {
  int n = 0;
  for (int a = 0; a < C::n_aggs; ++a) n += C::agg_kind(a) == K_SUM_F64;
  return n;
}
// Words per shared slot: the layout's, two per fixed-point float SUM, made odd.
template <class C>
constexpr int lean_stride(bool fixed) {
  return (C::slot_words + (fixed ? 2 * lean_float_sums<C>() : 0)) | 1;
}

// A thread's place among s_limit, held before it installs a key, so that the table never
// holds more: with a check before and an add after, every thread between the two passed
// the limit, and a small table (256 slots, 32 of them spare) filled.
__device__ __forceinline__ bool reserve_group(int* s_groups, int s_limit) {
  if (*((volatile int*)s_groups) >= s_limit) return false;
  if (atomicAdd(s_groups, 1) < s_limit) return true;
  atomicSub(s_groups, 1);
  return false;
}

// The stride of a key's probes: its own, so that a table near its limit has no long runs.
__device__ __forceinline__ uint32_t lean_step(unsigned long long k) {
  return 1u + ((uint32_t)((k * 0x9E3779B97F4A7C15ULL) >> 32) & 31u);
}

// Insert or find from slot h on within `probes` slots: the slot's index, -1 when the key has none.
template <int SW>
static __device__ __noinline__ int lean_insert(unsigned long long* sm, int S, unsigned long long k, uint32_t h, int probes,
                                               int* s_groups, int s_limit) {
  if (k == WG_EMPTY_KEY) return -1;
  const uint32_t step = lean_step(k);
  for (; probes > 0; --probes) {
    unsigned long long* s = sm + h * SW;
    const unsigned long long cur = *((volatile unsigned long long*)s);
    if (cur == k) return (int)h;
    if (cur == WG_EMPTY_KEY) {
      if (!reserve_group(s_groups, s_limit)) return -1;
      const unsigned long long old = atomicCAS(s, WG_EMPTY_KEY, k);
      if (old == WG_EMPTY_KEY) return (int)h;
      atomicSub(s_groups, 1);
      if (old == k) return (int)h;
    }
    h += step;
    if (h >= (uint32_t)S) h -= (uint32_t)S;
  }
  return -1;
}

// What a CTA takes from its sample of the input.
struct LeanSample {
  long long lo, hi;     // smallest and largest sampled key
  unsigned exp;         // exponent field of the largest float SUM input
};

// apply<NA, true> with one copy of each float SUM, or fixed-point ones.
template <class C, bool FIXED>
__device__ __forceinline__ void lean_apply(unsigned long long* s, const Contrib<C::n_aggs>& c, double scale) {
  atomicAdd((unsigned*)(s + 1), 1u);
  int nf = 0;
#pragma unroll
  for (int a = 0; a < C::n_aggs; ++a) {
    unsigned long long* t = s + C::agg_off(a);
    const unsigned long long w = c.w0[a];
    switch (C::agg_kind(a)) {
      case K_SUM_I64: smem_add_limbs((unsigned*)t, 2, w, 0); break;
      case K_SUM_F64: {
        unsigned long long lo, hi;
        if (FIXED && f64_to_fixed_scaled(as_f(w), scale, lo, hi))
          smem_add_limbs((unsigned*)(s + C::slot_words + 2 * nf), 4, lo, hi);
        else if (as_f(w) != 0.0)
          atomicAdd((double*)t, as_f(w));
        ++nf;
        break;
      }
      case K_MIN_I64: if ((long long)w < *(volatile long long*)t) atomicMin((long long*)t, (long long)w); break;
      case K_MAX_I64: if ((long long)w > *(volatile long long*)t) atomicMax((long long*)t, (long long)w); break;
      case K_MIN_F64: if (w < *(volatile unsigned long long*)t) atomicMin(t, w); break;
      case K_MAX_F64: if (w > *(volatile unsigned long long*)t) atomicMax(t, w); break;
      default: break;
    }
  }
}

// Rows [begin, end): chunk c of 32 * kLeanRows rows for c = first, first + step, ...
// (begin a multiple of kLeanRows, columns 16-byte aligned, no validity
// bitmaps). DENSE: slot = key - base, else hashed.
template <class C, bool FIXED, bool DENSE>
__device__ __forceinline__ void lean_rows(const Plan& P, int64_t begin, int64_t end, int64_t first, int64_t step,
                                          unsigned long long* sm, int S, long long base_key, int* s_groups,
                                          double scale, Credit* cr) {
  static_assert(C::key_words == 1 && C::has_join == 0, "one integer key, no join");
  constexpr int U = kLeanRows, NA = C::n_aggs, SW = lean_stride<C>(FIXED);
  const StatShape<C> sh{P};
  const int lane = threadIdx.x & 31;
  const int s_limit = (S * 7) / 8;
  int64_t base = begin + first * (32 * U);
  FarQueue queue;
  far_init(queue, base);
  for (;;) {
    // the common rows; a chunk with rows for the HBM table leaves the loop, so
    // that the call below holds no registers through it
    unsigned far = 0;
    for (; base < end; base += step * (32 * U)) {
      const int64_t r0 = base + (int64_t)lane * U;
      SrcRow rw[U];
      load_rows<U>(P, sh, r0, rw, end);
      unsigned act = 0;
      unsigned long long cur[U];
      uint32_t h[U];
      auto key_of = [&](int u, ExprVals& ev) {
        eval_exprs(P, sh, rw[u], -1, ev);
        return fetch(P, sh, rw[u], C::key_vcol(0), -1, ev).lo;
      };
#pragma unroll
      for (int u = 0; u < U; ++u) {
        bool a = r0 + u < end;
#pragma unroll
        for (int f = 0; f < C::n_filters; ++f) a = a && pred_val(P, sh, f, rw[u].v[C::filt_col(f)]);
        ExprVals ev;
        const unsigned long long k = key_of(u, ev);
        if (DENSE) {
          const unsigned long long d = k - (unsigned long long)base_key;
          far |= a && d >= (unsigned long long)S ? 1u << u : 0u;
          a = a && d < (unsigned long long)S;
          h[u] = (uint32_t)d;
        } else {
          h[u] = __umulhi((uint32_t)((k * 0x9E3779B97F4A7C15ULL) >> 32), (uint32_t)S);
        }
        act |= a ? 1u << u : 0u;
      }
      if (!DENSE) {
#pragma unroll
        for (int u = 0; u < U; ++u) cur[u] = *((volatile unsigned long long*)(sm + h[u] * SW));
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!((act >> u) & 1u)) continue;
        ExprVals ev;
        const unsigned long long k = key_of(u, ev);
        int at = (int)h[u];
        if (!DENSE) {
          unsigned long long c = cur[u];
          int probes = kLeanProbes;
          if (c != k && c != WG_EMPTY_KEY) {
            const int step = (int)lean_step(k);
            do {
              at += step;
              if (at >= S) at -= S;
              c = *((volatile unsigned long long*)(sm + at * SW));
            } while (c != k && c != WG_EMPTY_KEY && --probes > 0);
          }
          if (c == WG_EMPTY_KEY && *((volatile int*)s_groups) >= s_limit) at = -1;
          else if (c == WG_EMPTY_KEY) at = lean_insert<SW>(sm, S, k, (uint32_t)at, probes, s_groups, s_limit);
          else if (c != k) at = -1;
          if (at < 0) { far |= 1u << u; continue; }
        }
        Contrib<NA> c;
        make_contrib<NA>(P, sh, rw[u], -1, ev, c);
        lean_apply<C, FIXED>(sm + at * SW, c, scale);
      }
      if (__any_sync(WG_FULL_MASK, far != 0)) break;
    }
    if (base >= end) break;
    far_rows<StatShape<C>, U, false>(P, &queue, far, cr, base + (int64_t)lane * U);
    base += step * (32 * U);
  }
  far_flush<StatShape<C>>(P, &queue, cr);
}

// One row per thread, spread over [begin, end) so that neither order nor a
// quiet start decides: the keys' range and the largest float SUM input. Every
// thread of the CTA calls it; *out is shared.
template <class C>
__device__ __forceinline__ void lean_sample(const Plan& P, int64_t begin, int64_t end, LeanSample* out) {
  const StatShape<C> sh{P};
  if (threadIdx.x == 0) {
    out->lo = 0x7FFFFFFFFFFFFFFFLL;
    out->hi = -0x7FFFFFFFFFFFFFFFLL - 1;
    out->exp = 0;
  }
  __syncthreads();
  long long lo = 0x7FFFFFFFFFFFFFFFLL, hi = -0x7FFFFFFFFFFFFFFFLL - 1;
  unsigned ex = 0;
  const int64_t n = end - begin;
  if (n > 0) {
    const SrcGlobal src{begin + (int64_t)((n / blockDim.x) * threadIdx.x + (n % blockDim.x) * threadIdx.x / blockDim.x)};
    ExprVals ev;
    eval_exprs(P, sh, src, -1, ev);
    lo = hi = (long long)fetch(P, sh, src, C::key_vcol(0), -1, ev).lo;
    if (lean_float_sums<C>() > 0) {
      Contrib<C::n_aggs> c;
      make_contrib<C::n_aggs>(P, sh, src, -1, ev, c);
#pragma unroll
      for (int a = 0; a < C::n_aggs; ++a)
        if (C::agg_kind(a) == K_SUM_F64) {
          const unsigned e = (unsigned)(c.w0[a] >> 52) & 0x7FFu;
          if (e != 0x7FFu && e > ex) ex = e;
        }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const long long l2 = __shfl_down_sync(WG_FULL_MASK, lo, o), h2 = __shfl_down_sync(WG_FULL_MASK, hi, o);
    lo = l2 < lo ? l2 : lo;
    hi = h2 > hi ? h2 : hi;
  }
  ex = __reduce_max_sync(WG_FULL_MASK, ex);
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&out->lo, lo);
    atomicMax(&out->hi, hi);
    if (ex) atomicMax(&out->exp, ex);
  }
  __syncthreads();
}

// Whether the sampled keys fit a window of S slots, and its first key: the
// spare slots half on either side.
__device__ __forceinline__ bool lean_window(const LeanSample& s, int S, long long* base) {
  const unsigned long long span = (unsigned long long)s.hi - (unsigned long long)s.lo;  // (wraps right when hi >= lo)
  if (s.hi < s.lo || span >= (unsigned long long)S) return false;
  *base = (long long)((unsigned long long)s.lo - ((unsigned long long)S - 1 - span) / 2);
  return true;
}

// A sampled CTA's rows, dense or hashed.
template <class C, bool FIXED>
__device__ __forceinline__ bool lean_run(const Plan& P, int64_t begin, int64_t end, int64_t first, int64_t step,
                                         unsigned long long* sm, int S, const LeanSample& smp, int* s_groups,
                                         long long* base, Credit* cr) {
  const double scale = FIXED ? fixed_scale(fixed_exponent_of(smp.exp)) : 1.0;
  const bool dense = lean_window(smp, S, base);
  if (dense) lean_rows<C, FIXED, true>(P, begin, end, first, step, sm, S, *base, s_groups, scale, cr);
  else lean_rows<C, FIXED, false>(P, begin, end, first, step, sm, S, 0, s_groups, scale, cr);
  return dense;
}

template <class C, bool FIXED>
__global__ void __launch_bounds__(kLeanThreads, 1) lean_group_kernel(const __grid_constant__ Plan P) {
  extern __shared__ unsigned long long sm[];
  __shared__ int s_groups;
  __shared__ LeanSample smp;
  Credit cr;
  const int S = P.smem_slots;
  smem_table_init(P, sm, S, &s_groups);
  lean_sample<C>(P, 0, P.n_items, &smp);
  const int64_t wpb = blockDim.x >> 5;
  long long base = 0;
  const bool dense = lean_run<C, FIXED>(P, 0, P.n_items, (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5),
                                        (int64_t)gridDim.x * wpb, sm, S, smp, &s_groups, &base, &cr);
  __syncthreads();
  smem_table_flush<C::n_aggs>(P, sm, S, cr, FIXED ? fixed_exponent_of(smp.exp) : 64, dense, base);
  cr.release(P.T);
}

}  // namespace wgd
