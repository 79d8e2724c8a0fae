// wg_lowcard.cuh — the fused pipeline for any plan (no compiled shape) whose
// groups fit a CTA's shared memory.
//
// What bounds it: a plan without a compiled shape is interpreted, so the cost
// of a row is the instructions of its plan's steps, then the shared-memory
// atomics of its updates. Two choices follow.
//
//  - Column at a time over kLcRows rows per lane. Every decision a step takes
//    from the plan (a column's class, an operator, an aggregate's kind) is the
//    same for all rows, so it is taken once per step and kLcRows rows, and the
//    rows' loads and hash probes are in flight together. One row at a time, the
//    interpreter took every decision per row and each load waited for the last.
//  - Keys apart from accumulators, and the accumulators copied. A key's slot in
//    the CTA's key table is its group's index; the accumulators of group i lie in
//    up to 32 copies, lane l adding to copy l % copies. With a handful of
//    groups a warp's lanes meet on the same words: 32-bit shared atomics then
//    serialise and float adds (compare-and-swap loops) replay once per lane.
//    As many copies as fit the CTA's share of shared memory are taken; the
//    flush folds them with shuffles and updates the HBM table once per group.
//
// The copies are for the groups that the caller expects, and an estimate may be ten
// times too low. Where many of a CTA's rows found no slot, it hands its groups to the
// HBM table and goes on with as many slots of one copy as its shared memory holds
// (lc_rest, apart from the common loop, whose registers it would take). 2^24 rows into
// 1000 groups with a hint of 100: 36.6 ms with probes as long as the full table and
// a row at a time into the HBM table, 0.54 now, 0.33 with the right hint; into 10,000 by
// two keys with a hint of 1000 35.3 and 2.3 ms.
//
// Packed keys, NULL keys, a scalar aggregate (no key) and NULL counters take
// this path too. Rows whose key finds no slot (none free within kLcProbes, or a key
// outside a dense range) go to the HBM table, 32 of a warp's at a time; a warp that
// still meets many such rows stops looking for slots.
//
// Measured on B200, against pipeline_kernel: 30,000,001 rows, 6 groups by two
// int32 keys, seven aggregates over nullable columns 14.74 -> 1.58 ms (both
// bound by instruction issue and its latencies, not by the 1.33 GB read); a LEFT
// join of 2^24 + 3 rows on sparse int64 keys with duplicates, 50 groups 4.37 ->
// 0.89 ms. Shared memory beyond the tables' need costs: 64 KB more of it per CTA left so
// little L1 that the first query took 2.3 ms. Rows per lane x threads per SM, the first query: 2 x 1024 1.58, 3 x
// 1024 1.50, 4 x 768 1.66, 2 x 768 1.81, 4 x 512 1.85, 2 x 1536 1.86 ms; the second
// 0.89, 0.88, 0.96, 1.05, 1.06, 0.87; 2^21 rows into 1000 groups 93, 104, 110, 103,
// 104, 106 us.
#pragma once

#include "wg_shapes.cuh"

#include <type_traits>

namespace wgd {

constexpr int kLcRows = 2;         // rows per lane
constexpr int kLcThreads = 1024;   // per SM (64 registers each): two CTAs of 512, or one when the table needs the SM

// kLcRows values of one virtual column.
struct LcVals {
  unsigned long long lo[kLcRows], hi[kLcRows];
  unsigned null;  // bit u: row u is NULL
};

// The rows a lane works on: input row base + off and build row (or a direct
// join's payload bits).
struct LcRowSet {
  int64_t base;
  uint32_t off[kLcRows];
  int32_t brow[kLcRows];
  __device__ __forceinline__ int64_t row(int u) const { return base + off[u]; }
};

#define WG_LC_EACH(u) _Pragma("unroll") for (int u = 0; u < kLcRows; ++u)
#define WG_LC_LIVE(u, m) WG_LC_EACH(u) if (((m) >> u) & 1u)

// Column j (an input or payload column) of the rows in `live` (0 elsewhere).
__device__ __forceinline__ void lc_load(const Plan& P, const LcRowSet& r, int j, unsigned live, LcVals& v) {
  v.null = 0;
  WG_LC_EACH(u) { v.lo[u] = 0; v.hi[u] = 0; }
  const int nin = P.n_in;
  if (j < nin) {
    const void* d = P.in[j].data;
    switch (P.in[j].cls) {
      case WG_CLS_I32:
        WG_LC_LIVE(u, live) v.lo[u] = (unsigned long long)(long long)__ldcs((const int32_t*)d + r.row(u));
        break;
      case WG_CLS_F32:
        WG_LC_LIVE(u, live) v.lo[u] = as_w((double)__ldcs((const float*)d + r.row(u)));
        break;
      case WG_CLS_DEC:
        WG_LC_LIVE(u, live) {
          const longlong2 t = __ldcs((const longlong2*)d + r.row(u));
          v.lo[u] = (unsigned long long)t.y;
          v.hi[u] = (unsigned long long)t.x;
        }
        break;
      default:
        WG_LC_LIVE(u, live) v.lo[u] = (unsigned long long)__ldcs((const long long*)d + r.row(u));
        break;
    }
    if (P.in[j].valid != nullptr) {
      WG_LC_LIVE(u, live) v.null |= is_null(P.in[j], r.row(u)) ? 1u << u : 0u;
    }
    return;
  }
  {
    const DCol& c = P.join.pay[j - nin];
    if (P.join.direct) {  // brow holds the payload's 32 bits
      WG_LC_EACH(u) v.lo[u] = c.cls == WG_CLS_F32 ? as_w((double)__int_as_float(r.brow[u]))
                                                  : (unsigned long long)(long long)r.brow[u];
      return;
    }
    unsigned have = 0;
    WG_LC_EACH(u) have |= r.brow[u] >= 0 ? 1u << u : 0u;
    have &= live;
    v.null = live & ~have;  // an unmatched LEFT row
    switch (c.cls) {
      case WG_CLS_I32:
        WG_LC_LIVE(u, have) v.lo[u] = (unsigned long long)(long long)__ldg((const int32_t*)c.data + r.brow[u]);
        break;
      case WG_CLS_F32:
        WG_LC_LIVE(u, have) v.lo[u] = as_w((double)__ldg((const float*)c.data + r.brow[u]));
        break;
      case WG_CLS_DEC:
        WG_LC_LIVE(u, have) {
          const longlong2 t = __ldg((const longlong2*)c.data + r.brow[u]);
          v.lo[u] = (unsigned long long)t.y;
          v.hi[u] = (unsigned long long)t.x;
        }
        break;
      default:
        WG_LC_LIVE(u, have) v.lo[u] = (unsigned long long)__ldg((const long long*)c.data + r.brow[u]);
        break;
    }
    if (c.valid != nullptr) {
      WG_LC_LIVE(u, have) v.null |= is_null(c, r.brow[u]) ? 1u << u : 0u;
    }
    return;
  }
}

// Predicate f on the rows in `live`: the rows that pass. The comparison is
// reduced to which of less / equal / greater / unordered the operator accepts.
__device__ __forceinline__ unsigned lc_filter(const Plan& P, const LcRowSet& r, int f, unsigned live) {
  LcVals v;
  lc_load(P, r, P.filt[f].col, live, v);
  const int op = P.filt[f].op;
  const unsigned accept = op == WG_OP_EQ ? 2u : op == WG_OP_NE ? 13u : op == WG_OP_LT ? 1u : op == WG_OP_LE ? 3u
                          : op == WG_OP_GT ? 4u : 6u;
  unsigned pass = 0;
  if (P.filt[f].cls == WG_CLS_I32 || P.filt[f].cls == WG_CLS_I64) {
    const long long c = P.filt[f].ci;
    WG_LC_LIVE(u, live) {
      const long long x = (long long)v.lo[u];
      pass |= (accept & (x < c ? 1u : x == c ? 2u : 4u)) ? 1u << u : 0u;
    }
  } else {
    const double c = P.filt[f].cf;  // exact in binary64 for a float32 column
    WG_LC_LIVE(u, live) {
      const double x = as_f(v.lo[u]);
      pass |= (accept & (x < c ? 1u : x == c ? 2u : x > c ? 4u : 8u)) ? 1u << u : 0u;
    }
  }
  return pass & ~v.null;
}

// Probe of the rows in `live`: brow and the rows that match. The first slot of
// every row's probe is loaded before any is examined; a collision falls back
// to the one-row probe.
__device__ __forceinline__ unsigned lc_probe(const Plan& P, LcRowSet& r, unsigned live, const LcVals& k) {
  const JoinView& j = P.join;
  unsigned hit = 0;
  live &= ~k.null;
  if (j.direct && j.dense) {
    unsigned in = 0;
    WG_LC_LIVE(u, live) in |= k.lo[u] - (unsigned long long)j.base < j.mask ? 1u << u : 0u;
    if (j.dense == 2) {
      WG_LC_LIVE(u, in) r.brow[u] = (int32_t)__ldg((const uint32_t*)j.slots + (k.lo[u] - (unsigned long long)j.base));
      return in;
    }
    unsigned long long s[kLcRows];
    WG_LC_LIVE(u, in) s[u] = __ldg((const unsigned long long*)j.slots + (k.lo[u] - (unsigned long long)j.base));
    WG_LC_LIVE(u, in) {
      if ((uint32_t)s[u] == (uint32_t)k.lo[u]) { hit |= 1u << u; r.brow[u] = (int32_t)(s[u] >> 32); }
    }
    return hit;
  }
  if (j.direct) {
    WG_LC_LIVE(u, live) {
      int32_t b = -1;
      if (join_direct(j, (int64_t)k.lo[u], b, P.err)) hit |= 1u << u;
      r.brow[u] = b;
    }
    return hit;
  }
  if (j.bloom != nullptr) {
    WG_LC_LIVE(u, live) {
      if (!bloom_contains(j.bloom, j.bloom_mask, bloom_hash_int((long long)k.lo[u]))) live &= ~(1u << u);
    }
  }
  if (j.flavor == 0) {
    WG_LC_LIVE(u, live) {
      if ((long long)k.lo[u] < INT32_MIN || (long long)k.lo[u] > INT32_MAX) live &= ~(1u << u);
    }
    unsigned long long s[kLcRows];
    WG_LC_LIVE(u, live) s[u] = __ldg((const unsigned long long*)j.slots + fib_slot(k.lo[u], j.shift));
    WG_LC_LIVE(u, live) {
      int32_t b = (int32_t)(s[u] >> 32);
      if (b != -1 && (uint32_t)s[u] != (uint32_t)k.lo[u]) b = join_head(j, (int64_t)k.lo[u], P.err);
      r.brow[u] = b;
      hit |= b >= 0 ? 1u << u : 0u;
    }
  } else {
    longlong2 s[kLcRows];
    WG_LC_LIVE(u, live) s[u] = __ldg((const longlong2*)j.slots + fib_slot(k.lo[u], j.shift));
    WG_LC_LIVE(u, live) {
      int32_t b = (int32_t)(uint32_t)s[u].y;
      if (b != -1 && (unsigned long long)s[u].x != k.lo[u]) b = join_head(j, (int64_t)k.lo[u], P.err);
      r.brow[u] = b;
      hit |= b >= 0 ? 1u << u : 0u;
    }
  }
  return hit;
}

// Projection e of the rows in `live` (eval_expr's semantics; the host has
// checked the program, and an entry's type is the same for every row). The
// stack is a shift register with its top in `top`: no entry is addressed by a
// run-time depth, which would cost a select per entry and operation.
__device__ __forceinline__ void lc_eval(const Plan& P, const LcRowSet& r, int e, unsigned live,
                                        unsigned long long* out, unsigned& null) {
  const ExprD& x = P.expr[e];
  unsigned long long top[kLcRows], s0[kLcRows], s1[kLcRows], s2[kLcRows];
  WG_LC_EACH(u) { top[u] = 0; s0[u] = 0; s1[u] = 0; s2[u] = 0; }
  unsigned fl = 0;  // bit i: the entry i below the top holds a float
  null = 0;
#pragma unroll 1
  for (int k = 0; k < x.n_ops; ++k) {
    const int opc = x.opc[k];
    if (opc <= WG_EXPR_CONST_F) {
      WG_LC_EACH(u) { s2[u] = s1[u]; s1[u] = s0[u]; s0[u] = top[u]; }
      bool isf = opc == WG_EXPR_CONST_F;
      if (opc == WG_EXPR_COL) {
        const int j = x.arg[k];
        LcVals w;
        lc_load(P, r, j, live, w);
        null |= w.null;
        const int cls = P.vcls[j];
        isf = !(cls == WG_CLS_I32 || cls == WG_CLS_I64);
        if (cls == WG_CLS_DEC) {
          const double b = P.vdiv_b[j], y = P.vdiv_y[j];
          WG_LC_EACH(u) w.lo[u] = as_w(div_by_recip(int128_to_f64((int64_t)w.hi[u], w.lo[u]), b, y));
        }
        WG_LC_EACH(u) top[u] = w.lo[u];
      } else {
        WG_LC_EACH(u) top[u] = (unsigned long long)x.imm[k];
      }
      fl = fl << 1 | (isf ? 1u : 0u);
    } else {
      const bool bf = fl & 1u, af = fl & 2u;
      const bool ints = opc == WG_EXPR_SHR || opc == WG_EXPR_AND || (!af && !bf && opc != WG_EXPR_DIV);
      if (ints) {
        WG_LC_EACH(u) {
          const unsigned long long a = s0[u], b = top[u];
          top[u] = opc == WG_EXPR_SHR ? (unsigned long long)((long long)a >> (b & 63)) : opc == WG_EXPR_AND ? (a & b)
                   : opc == WG_EXPR_ADD ? a + b : opc == WG_EXPR_SUB ? a - b : a * b;
        }
      } else {
        if (!af) { WG_LC_EACH(u) s0[u] = as_w(__ll2double_rn((long long)s0[u])); }
        if (!bf) { WG_LC_EACH(u) top[u] = as_w(__ll2double_rn((long long)top[u])); }
        if (opc == WG_EXPR_DIV) {
          WG_LC_EACH(u) top[u] = as_w(__ddiv_rn(as_f(s0[u]), as_f(top[u])));
        } else {
          WG_LC_EACH(u) {
            const double a = as_f(s0[u]), b = as_f(top[u]);
            top[u] = as_w(opc == WG_EXPR_ADD ? __dadd_rn(a, b) : opc == WG_EXPR_SUB ? __dsub_rn(a, b) : __dmul_rn(a, b));
          }
        }
      }
      WG_LC_EACH(u) { s0[u] = s1[u]; s1[u] = s2[u]; }
      fl = (fl >> 2) << 1 | (ints ? 0u : 1u);
    }
  }
  const bool widen = x.result_cls == WG_CLS_F64 && !(fl & 1u);
  WG_LC_EACH(u) out[u] = widen ? as_w(__ll2double_rn((long long)top[u])) : top[u];
}

// The plan's projections of the current rows, evaluated once per step. Indexed
// at run time: they live in local memory, two stores and loads of which cost
// less than keeping them in registers through the step.
struct LcExprs {
  unsigned long long v[WG_MAX_EXPRS * kLcRows];
  unsigned null[WG_MAX_EXPRS];
};

// Virtual column j of the rows in `live`.
__device__ __forceinline__ void lc_value(const Plan& P, const LcRowSet& r, const LcExprs& ev, int j, unsigned live,
                                         LcVals& v) {
  const int e = j - P.n_in - (P.has_join ? P.join.n_pay : 0);
  if (e < 0) {
    lc_load(P, r, j, live, v);
  } else {
    WG_LC_EACH(u) v.lo[u] = ev.v[e * kLcRows + u];
    v.null = ev.null[e] & live;
  }
}

// Slots a key is looked for in before it counts as having none: probes of a full
// table are instructions of every row. (Keys at half load do not need so many, also where small
// packed keys hash to neighbouring slots.)
constexpr int kLcProbes = 32;

// A key's slot in the CTA's key table of S slots, inserting it: [0, S) a regular
// key, S the key equal to the empty pattern, S + 1 the NULL key; -1 when it has
// none or is outside a dense range (or, with the groups in a key window in HBM,
// outside the window or NULL).
template <bool SH>
__device__ __forceinline__ int lc_slot(const Plan& P, const KeyWindow& w, unsigned long long* keys, int S,
                                       unsigned long long k0, unsigned long long k1, bool knull) {
  if (!SH) {
    const unsigned long long d = k0 - (unsigned long long)w.base;
    return !knull && d < w.n ? (int)d : -1;
  }
  const int kw = P.L.key_words;
  if (kw == 0) return 0;
  if (knull) return S + 1;
  if (P.gdense) {
    const uint32_t d = (uint32_t)k0 - (uint32_t)P.gmin;
    return d < (uint32_t)S ? (int)d : -1;
  }
  const int probes = min(S, kLcProbes);
  if (kw == 1) {
    if (k0 == WG_EMPTY_KEY) return S;
    uint32_t h = __umulhi((uint32_t)((k0 * 0x9E3779B97F4A7C15ULL) >> 32), (uint32_t)S);
    for (int p = 0; p < probes; ++p) {
      unsigned long long* s = keys + h;
      const unsigned long long cur = *((volatile unsigned long long*)s);
      if (cur == k0) return (int)h;
      if (cur == WG_EMPTY_KEY) {
        const unsigned long long old = atomicCAS(s, WG_EMPTY_KEY, k0);
        if (old == WG_EMPTY_KEY || old == k0) return (int)h;
      }
      h = h + 1 == (uint32_t)S ? 0u : h + 1;
    }
    return -1;
  }
  if (k0 == ~0ULL && k1 == ~0ULL) return S;
  const unsigned long long m = (k0 ^ 0x9E3779B97F4A7C15ULL) * (k1 * 0x517CC1B727220A95ULL + 0x9E3779B97F4A7C15ULL | 1ULL);
  uint32_t h = __umulhi((uint32_t)(m >> 32), (uint32_t)S);
  for (int p = 0; p < probes; ++p) {
    unsigned long long* s = keys + 2 * h;
    // the words change once, from {~0, ~0} to the key: a read with neither ~0
    // is the complete key, anything else is settled by the 16-byte CAS
    const U128 cur = read128(s);
    if (cur.lo != ~0ULL && cur.hi != ~0ULL) {
      if (cur.lo == k0 && cur.hi == k1) return (int)h;
    } else {
      U128 e; e.lo = ~0ULL; e.hi = ~0ULL;
      U128 k; k.lo = k0; k.hi = k1;
      const U128 old = cas128((U128*)s, e, k);
      if (old.lo == e.lo && old.hi == e.hi) return (int)h;
      if (old.lo == k0 && old.hi == k1) return (int)h;
    }
    h = h + 1 == (uint32_t)S ? 0u : h + 1;
  }
  return -1;
}

// Group keys of the rows in `live`, packed as make_key does; returns the rows that have one.
__device__ __forceinline__ unsigned lc_make_keys(const Plan& P, const LcRowSet& r, const LcExprs& ev, unsigned live,
                                                 unsigned long long (&k0)[kLcRows], unsigned long long (&k1)[kLcRows],
                                                 unsigned& knull) {
  const Layout& L = P.L;
  unsigned bad = 0;
  knull = 0;
  WG_LC_EACH(u) { k0[u] = 0; k1[u] = 0; }
  if (L.key_words > 0) {
#pragma unroll 1
    for (int k = 0; k < L.n_keys; ++k) {
      LcVals v;
      lc_value(P, r, ev, L.key_vcol[k], live, v);
      if (L.key_words == 1) {
        knull = v.null;
        WG_LC_LIVE(u, live & ~v.null) k0[u] = v.lo[u];
        break;
      }
      const bool w0 = L.key_word[k] == 0, i32 = L.key_i32[k] != 0;
      const int sh = L.key_shift[k];
      WG_LC_LIVE(u, live) {
        if ((v.null >> u) & 1u) {
          if (L.null_word < 0) { bad |= 1u << u; continue; }
          const unsigned long long m = 1ULL << (L.null_shift + k);
          if (L.null_word == 0) k0[u] |= m; else k1[u] |= m;
        } else {
          const unsigned long long w = i32 ? (unsigned long long)(uint32_t)v.lo[u] << sh : v.lo[u];
          if (w0) k0[u] |= w; else k1[u] |= w;
        }
      }
    }
    if (bad) set_error(P.err, WG_DERR_NULL_PACKED);
  }
  return live & ~bad;
}

// Group keys of the rows in `live` and their shared slots; returns the rows
// that have one, `far` the rows that have none.
template <bool SH>
__device__ __forceinline__ unsigned lc_keys(const Plan& P, const KeyWindow& w, const LcRowSet& r, const LcExprs& ev,
                                            unsigned live, unsigned long long* keys, int S, int (&slot)[kLcRows],
                                            unsigned& far) {
  unsigned long long k0[kLcRows], k1[kLcRows];
  unsigned knull;
  live = lc_make_keys(P, r, ev, live, k0, k1, knull);
  WG_LC_EACH(u) slot[u] = 0;
  far = 0;
  WG_LC_LIVE(u, live) {
    slot[u] = lc_slot<SH>(P, w, keys, S, k0[u], k1[u], (knull >> u) & 1u);
    far |= slot[u] < 0 ? 1u << u : 0u;
  }
  return live & ~far;
}

// The updates of the rows in `live`, aggregate by aggregate (apply<NA, SH>'s,
// with 32-bit NULL counters in shared memory); acc: the lane's copy of the
// accumulators (SH), or the window's slots past their key word.
template <bool SH>
__device__ __forceinline__ void lc_count(unsigned long long* p) {
  if (SH) atomicAdd((unsigned*)p, 1u);
  else atomicAdd(p, 1ULL);
}

template <bool SH>
__device__ __forceinline__ void lc_update(const Plan& P, const LcRowSet& r, const LcExprs& ev, unsigned live,
                                          unsigned long long* acc, const int (&slot)[kLcRows]) {
  const Layout& L = P.L;
  const int kw = L.key_words, aw = SH ? P.smem_sw : L.slot_words;
  unsigned long long* t[kLcRows];  // the row's group, indexed like a slot (key words first)
  WG_LC_EACH(u) t[u] = acc + (int64_t)slot[u] * aw - kw;
  WG_LC_LIVE(u, live) lc_count<SH>(t[u] + kw);
#pragma unroll 1
  for (int a = 0; a < L.n_aggs; ++a) {
    const int kind = L.agg[a].kind, off = L.agg[a].off, noff = L.agg[a].null_off, vcol = L.agg[a].vcol;
    if (vcol < 0 || (kind == K_COUNT && noff < 0)) continue;
    LcVals v;
    lc_value(P, r, ev, vcol, live, v);
    if (noff >= 0) {
      WG_LC_LIVE(u, live & v.null) lc_count<SH>(t[u] + noff);
    }
    const unsigned m = live & ~v.null;
    switch (kind) {
      case K_SUM_I64:
        WG_LC_LIVE(u, m) {
          if (SH) smem_add_limbs((unsigned*)(t[u] + off), 2, v.lo[u], 0);
          else if (v.lo[u]) atomicAdd(t[u] + off, v.lo[u]);
        }
        break;
      case K_SUM_F64: {
        const int cls = P.vcls[vcol];
        const bool ints = cls == WG_CLS_I32 || cls == WG_CLS_I64;
        WG_LC_LIVE(u, m) {
          const double d = ints ? __ll2double_rn((long long)v.lo[u]) : as_f(v.lo[u]);
          if (d != 0.0) atomicAdd((double*)(t[u] + off), d);
        }
        break;
      }
      case K_SUM_DEC:
        WG_LC_LIVE(u, m) {
          if (SH) smem_add_limbs((unsigned*)(t[u] + off), 4, v.lo[u], v.hi[u]);
          else atomic_add128(t[u] + off, v.lo[u], v.hi[u]);
        }
        break;
      case K_MIN_I64:
        WG_LC_LIVE(u, m) {
          if ((long long)v.lo[u] < *(volatile long long*)(t[u] + off)) atomicMin((long long*)(t[u] + off), (long long)v.lo[u]);
        }
        break;
      case K_MAX_I64:
        WG_LC_LIVE(u, m) {
          if ((long long)v.lo[u] > *(volatile long long*)(t[u] + off)) atomicMax((long long*)(t[u] + off), (long long)v.lo[u]);
        }
        break;
      case K_MIN_F64:
        WG_LC_LIVE(u, m) {
          const unsigned long long o = f64_to_ord(as_f(v.lo[u]));
          if (o < *(volatile unsigned long long*)(t[u] + off)) atomicMin(t[u] + off, o);
        }
        break;
      case K_MAX_F64:
        WG_LC_LIVE(u, m) {
          const unsigned long long o = f64_to_ord(as_f(v.lo[u]));
          if (o > *(volatile unsigned long long*)(t[u] + off)) atomicMax(t[u] + off, o);
        }
        break;
      case K_MIN_DEC: case K_MAX_DEC:  // 16-byte compare-and-swap: in HBM only
        if (!SH) {
          WG_LC_LIVE(u, m) {
            if (kind == K_MIN_DEC) atomic_min128((U128*)(t[u] + off), v.lo[u], v.hi[u]);
            else atomic_max128((U128*)(t[u] + off), v.lo[u], v.hi[u]);
          }
        }
        break;
      default: break;  // COUNT
    }
  }
}

// One row without a slot, into the HBM table: of a compiled shape row by row, of
// any other plan by the same steps as the common rows'.
template <class Sh>
static __device__ __noinline__ void lc_far_row(const Plan& P, int64_t row, int32_t brow, Credit* cr) {
  const Sh sh{P};
  if constexpr (std::is_same<Sh, DynShape>::value) {
    LcRowSet r;
    r.base = row;
    WG_LC_EACH(u) { r.off[u] = 0; r.brow[u] = brow; }
    LcExprs ev;
#pragma unroll 1
    for (int e = 0; e < P.n_exprs; ++e) lc_eval(P, r, e, 1u, ev.v + e * kLcRows, ev.null[e]);
    unsigned long long k0[kLcRows], k1[kLcRows];
    unsigned knull;
    if (!lc_make_keys(P, r, ev, 1u, k0, k1, knull)) return;
    unsigned long long* g = find_global(sh, P.T, k0[0], k1[0], (knull & 1u) != 0, P.err, cr);
    const int slot[kLcRows] = {0, 0};
    if (g != nullptr) lc_update<false>(P, r, ev, 1u, g + P.L.key_words, slot);
  } else {
    constexpr int NA = Sh::kAggs;
    const SrcGlobal src{row};
    ExprVals ev;
    Contrib<NA> c;
    eval_exprs(P, sh, src, brow, ev);
    unsigned long long k0, k1;
    bool knull;
    if (!make_key(P, sh, src, brow, ev, k0, k1, knull)) return;
    make_contrib<NA>(P, sh, src, brow, ev, c);
    unsigned long long* g = find_global(sh, P.T, k0, k1, knull, P.err, cr);
    if (g != nullptr) apply<NA, false>(sh, g, c, 1ULL, 1, P.minmax_test != 0);
  }
}

// The lane of the n-th set bit of m (n below its count).
__device__ __forceinline__ int nth_lane(unsigned m, int n) {
  int at = 0;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const int c = __popc(m & ((1u << s) - 1u));
    if (n >= c) {
      n -= c;
      m >>= s;
      at += s;
    }
  }
  return at;
}

// Rows for the HBM table, gathered per warp until there are 32, one in each lane: a
// row there is some hundreds of instructions and dependent reads, which cost a warp
// the same for one row as for 32. In local memory, as it is used rarely: shared
// memory taken for it would come out of the L1 cache, which the plan's steps use.
struct FarQueue {
  int64_t row;
  int32_t brow;
  int n;           // rows in the queue (all lanes the same, as are the fields below)
  int far, mark;   // rows that came here since the last look, and how many the next one waits for
  int64_t from;    // the row at which the warp began to count them
};

__device__ __forceinline__ void far_init(FarQueue& q, int64_t from) {
  q.row = 0;
  q.brow = -1;
  q.n = q.far = 0;
  q.mark = 64;
  q.from = from;
}

template <class Sh>
static __device__ __noinline__ void far_flush(const Plan& P, FarQueue* q, Credit* cr) {
  if ((int)(threadIdx.x & 31) < q->n) lc_far_row<Sh>(P, q->row, q->brow, cr);
  q->n = 0;
  __syncwarp();
}

// Whether more than one in `share` of the warp's rows had no slot, looked at every q->mark such rows.
static __device__ __noinline__ bool lc_too_many(FarQueue* q, int64_t base, int share) {
  if (q->far < q->mark) return false;
  const int64_t step = (int64_t)gridDim.x * (blockDim.x >> 5) * (32 * kLcRows);
  const int64_t rows = ((base - q->from) / step + 1) * (32 * kLcRows);
  const bool many = (int64_t)q->far * share > rows;
  q->far = 0;
  q->from = base + step;
  return many;
}

// Every lane of the warp calls it: the rows row0 + u of the set bits u of `far`
// (JOIN: two rows, row0 and row1, with their build rows). Returns lc_too_many, of
// the rows up to base, where a share is given; one call for both, as every call in a
// row loop costs the loop registers.
template <class Sh, int U, bool JOIN>
static __device__ __noinline__ bool far_rows(const Plan& P, FarQueue* q, unsigned far, Credit* cr, int64_t row0, int64_t row1 = 0,
                                             int32_t b0 = -1, int32_t b1 = -1, int64_t base = 0, int share = 0) {
  static_assert(!JOIN || U == 2, "two rows per lane with build rows");
  const int lane = threadIdx.x & 31;
  int n = q->n;
#pragma unroll 1
  for (int u = 0; u < U; ++u) {
    const unsigned m = __ballot_sync(WG_FULL_MASK, (far >> u) & 1u);
    if (m == 0) continue;
    const int c = __popc(m);
    const int64_t row = JOIN ? (u ? row1 : row0) : row0 + u;
    const int32_t brow = u ? b1 : b0;
    // row i of the step goes to lane n + i, past lane 31 to lane n + i - 32 once the queue has run
    auto put = [&](int i) {
      const bool in = i >= 0 && i < c;
      const int from = in ? nth_lane(m, i) : lane;
      const int64_t r = __shfl_sync(WG_FULL_MASK, row, from);
      const int32_t b = JOIN ? __shfl_sync(WG_FULL_MASK, brow, from) : -1;
      if (in) {
        q->row = r;
        q->brow = b;
      }
    };
    put(lane - n);
    if (n + c >= 32) {
      lc_far_row<Sh>(P, q->row, q->brow, cr);
      __syncwarp();
      put(lane + 32 - n);
    }
    n = (n + c) & 31;
    q->far += c;
  }
  q->n = n;
  return share > 0 && lc_too_many(q, base, share);
}

// The CTA's groups folded over their R copies (R consecutive lanes per group) and
// added to the HBM table. CTAs start at different groups, as smem_table_flush.
template <int NA>
__device__ __forceinline__ void lc_flush(const Plan& P, const unsigned long long* keys, const unsigned long long* acc,
                                         int S, int R, Credit* cr) {
  const LayoutAcc ly{P.L};
  const Layout& L = P.L;
  const int kw = L.key_words, aw = P.smem_sw, S2 = S + 2;
  const int lane = threadIdx.x & 31, per = 32 / R, copy = lane & (R - 1);
  const int step = (int)(blockDim.x >> 5) * per;
  const int off0 = (int)(((long long)blockIdx.x * S2) / max(1, (int)gridDim.x));
  for (int i0 = (int)(threadIdx.x >> 5) * per; i0 < S2; i0 += step) {
    const int n = i0 + lane / R;
    const bool have = n < S2;
    const int i = have ? (n + off0 < S2 ? n + off0 : n + off0 - S2) : 0;
    const unsigned long long* s = acc + ((size_t)copy * S2 + i) * aw - kw;
    unsigned long long rows = have ? s[kw] : 0ULL;
    Contrib<NA> c;
    slot_contrib<NA>(ly, s, c);
    for (int o = R >> 1; o > 0; o >>= 1) {
      rows += __shfl_xor_sync(WG_FULL_MASK, rows, o);
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        if (a >= L.n_aggs) continue;
        const int kind = L.agg[a].kind;
        const unsigned long long b0 = __shfl_xor_sync(WG_FULL_MASK, c.w0[a], o);
        const unsigned long long b1 = kind_words(kind) == 2 ? __shfl_xor_sync(WG_FULL_MASK, c.w1[a], o) : 0ULL;
        combine(kind, c.w0[a], c.w1[a], b0, b1);
        if (L.agg[a].null_off >= 0) c.nul[a] += __shfl_xor_sync(WG_FULL_MASK, c.nul[a], o);
      }
    }
    if (copy != 0 || !have || rows == 0) continue;
    unsigned long long k0 = 0, k1 = 0;
    const bool knull = kw > 0 && i == S + 1;
    if (kw > 0 && !knull) {
      if (i == S) { k0 = kw == 1 ? WG_EMPTY_KEY : ~0ULL; k1 = ~0ULL; }
      else if (P.gdense) k0 = (unsigned long long)P.gmin + (unsigned long long)i;
      else { k0 = keys[(size_t)i * kw]; if (kw == 2) k1 = keys[(size_t)i * 2 + 1]; }
    }
    unsigned long long* g = find_global(ly, P.T, k0, k1, knull, P.err, cr);
    if (g != nullptr) apply<NA, false>(ly, g, c, rows);
  }
}

// The rows of the warp from base on. SH: groups in the CTA's shared memory, S slots
// at sm and the copy of the accumulators that the lane adds to at mine; otherwise
// in the key window win, its accumulators at mine. REST: after the CTA's second layout.
// Returns the row at which the warp stopped: the end of the input, or where its CTA
// is to change the layout.
template <int NA, bool SH, bool REST>
__device__ __forceinline__ int64_t lc_rows(const Plan& P, const KeyWindow& win, unsigned long long* sm, int S,
                                           unsigned long long* mine, int64_t base, FarQueue* queue, volatile int* s_quit,
                                           Credit* cr) {
  const int lane = threadIdx.x & 31;
  const int64_t step = (int64_t)gridDim.x * (blockDim.x >> 5) * (32 * kLcRows);
  const int jt = P.has_join ? (P.join.direct ? WG_JOIN_INNER : P.join.jtype) : WG_JOIN_INNER;
  bool look = !REST || S > 0;  // for shared slots
  for (; base < P.n_items; base += step) {
    bool quit = false;
    LcRowSet r;
    r.base = P.sel ? 0 : base;
    unsigned live = 0;
    WG_LC_EACH(u) {
      const int i = u * 32 + lane;
      const bool in = base + i < P.n_items;
      live |= in ? 1u << u : 0u;
      r.off[u] = !in ? 0u : P.sel ? __ldg(P.sel + base + i) : (uint32_t)i;
      r.brow[u] = -1;
    }
#pragma unroll 1
    for (int f = 0; f < P.n_filters; ++f) live = lc_filter(P, r, f, live);
    if (P.has_join) {
      LcVals k;
      lc_load(P, r, P.probe_col, live, k);
      if (P.join.part_shift != 0) {  // rows of another pass over a partitioned build
        WG_LC_LIVE(u, live) {
          if (!join_pass_mine(P.join, (k.null >> u) & 1u, (long long)k.lo[u])) live &= ~(1u << u);
        }
      }
      const unsigned hit = lc_probe(P, r, live, k);
      if (jt == WG_JOIN_INNER) live = hit;
      else if (jt == WG_JOIN_LEFT) { WG_LC_EACH(u) if (!((hit >> u) & 1u)) r.brow[u] = -1; }
      else { live = jt == WG_JOIN_SEMI ? hit : live & ~hit; WG_LC_EACH(u) r.brow[u] = -1; }
    }
    const bool chained = P.has_join && !P.join.direct && jt != WG_JOIN_SEMI && jt != WG_JOIN_ANTI;
    while (__any_sync(WG_FULL_MASK, live != 0)) {
      int32_t nxt[kLcRows];
      if (chained) {
        WG_LC_EACH(u) nxt[u] = ((live >> u) & 1u) && r.brow[u] >= 0 ? __ldg(P.join.next + r.brow[u]) : -1;
      }
      LcExprs ev;
#pragma unroll 1
      for (int e = 0; e < P.n_exprs; ++e) lc_eval(P, r, e, live, ev.v + e * kLcRows, ev.null[e]);
      unsigned far = live;
      if (!REST || look) {
        int slot[kLcRows];
        const unsigned have = lc_keys<SH>(P, win, r, ev, live, sm, S, slot, far);
        lc_update<SH>(P, r, ev, have, mine, slot);
      }
      if (__any_sync(WG_FULL_MASK, far != 0)) {
        // Another layout holds more groups. Where there is none (left), a row without a slot has cost
        // the probes on top of its way through the HBM table: 2^24 rows into 1000 groups with a fifth
        // of them without took 1.8 ms, all of them 1.35.
        const int share = !SH || (P.gdense && !REST) ? 0 : !REST && P.smem_more > 0 ? 16 : 6;
        const bool many = far_rows<DynShape, kLcRows, true>(P, queue, far, cr, r.row(0), r.row(1), r.brow[0], r.brow[1], base, share);
        if (REST) {
          look = look && !many;
        } else if (SH) {
          if (many) *s_quit = 1;
          __syncwarp();
          quit = __any_sync(WG_FULL_MASK, *s_quit != 0);
        }
      }
      if (!chained) break;  // at most one match per row
      live = 0;             // arenaNext chain (join.go:2700)
      WG_LC_EACH(u) {
        r.brow[u] = nxt[u];
        live |= nxt[u] >= 0 ? 1u << u : 0u;
      }
    }
    if (SH && !REST && quit) return base + step;
  }
  return base;
}

__device__ __forceinline__ void lc_init(const Plan& P, unsigned long long* sm, int S, int R, const unsigned long long* init) {
  const int kw = P.L.key_words, key_words = P.gdense ? 0 : S * kw;
  for (int i = threadIdx.x; i < key_words; i += blockDim.x) sm[i] = kw == 1 ? WG_EMPTY_KEY : ~0ULL;
  __syncthreads();
  fill_pattern(sm + key_words, (int64_t)R * (S + 2) * P.smem_sw, P.smem_sw, P.L.slot_words - kw, init + kw, threadIdx.x, blockDim.x);
  __syncthreads();
}

// The rest of a CTA's rows with P.smem_more slots of one copy, none where that is 0.
template <int NA>
static __device__ __noinline__ void lc_rest(const Plan& P, unsigned long long* sm, const unsigned long long* init, int64_t base,
                                            FarQueue* queue, Credit* cr) {
  const int S = P.smem_more;
  unsigned long long* acc = sm + S * P.L.key_words;
  if (S > 0) lc_init(P, sm, S, 1, init);
  queue->far = 0;
  queue->mark = 128;
  queue->from = base;
  lc_rows<NA, true, true>(P, KeyWindow{0, 0}, sm, S, acc, base, queue, nullptr, cr);
  __syncthreads();
  if (S > 0) lc_flush<NA>(P, sm, acc, S, 1, cr);
}

// SH: groups in the CTA's shared memory; otherwise in the launch's key window
// (wg_window.cuh), nothing when it has none.
template <int NA, bool SH>
__global__ void __launch_bounds__(kLcThreads, 1) lowcard_kernel(const __grid_constant__ Plan P) {
  extern __shared__ __align__(16) unsigned long long sm[];
  __shared__ int s_quit;
  __shared__ unsigned long long s_init[WG_MAX_SLOT_WORDS];
  KeyWindow win;
  win.base = 0;
  win.n = 0;
  if (!SH) {
    win = *P.win;
    if (win.n == 0) return;
  }
  Credit cr;
  int64_t base = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 * kLcRows);
  FarQueue queue;
  far_init(queue, base);
  if (SH) {
    const int S = P.smem_slots, R = P.smem_rep;
    unsigned long long* acc = sm + (P.gdense ? 0 : S * P.L.key_words);
    if (threadIdx.x < (unsigned)P.L.slot_words) s_init[threadIdx.x] = P.L.init[threadIdx.x];
    if (threadIdx.x == 0) s_quit = 0;
    lc_init(P, sm, S, R, s_init);
    unsigned long long* mine = acc + (size_t)(threadIdx.x & (unsigned)(R - 1)) * (S + 2) * P.smem_sw;
    base = lc_rows<NA, true, false>(P, win, sm, S, mine, base, &queue, &s_quit, &cr);
    __syncthreads();
    lc_flush<NA>(P, sm, acc, S, R, &cr);
    if (s_quit) {
      __syncthreads();  // the table is read before it is laid out anew
      lc_rest<NA>(P, sm, s_init, base, &queue, &cr);
    }
  } else {
    lc_rows<NA, false, false>(P, win, sm, 0, P.wslots + P.L.key_words, base, &queue, nullptr, &cr);
  }
  far_flush<DynShape>(P, &queue, &cr);
  cr.release(P.T);
}

#undef WG_LC_EACH
#undef WG_LC_LIVE

}  // namespace wgd
