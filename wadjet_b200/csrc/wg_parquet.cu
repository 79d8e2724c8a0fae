// wg_parquet.cu — batches on the device: the upload of decoded host batches and
// Parquet column chunks decoded on the GPU.
//
// The reference's native scan decodes each page on the host
// (ColumnPageReader.decodeValues, internal/storage/parquet/page_reader.go:607;
// the RLE / bit-packed hybrid, rle.go) and copies the values into a
// batch.Vector (scan/columnar_native.go:470-707). Here only the encoded page
// bytes cross to the device and the decode runs there:
//
// Every chunk of a batch goes through the same few launches, over slices of
// its pages (about kSliceRows rows each), so a batch fills the SMs whatever its
// page count:
//
//  1. definition levels: the hybrid stream expanded to a valid byte per row
//     (level 1 = a value, 0 = NULL);
//  2. the bytes packed into validity words, their popcounts scanned, so the
//     rank of a row among the non-NULL rows is a prefix plus one popcount;
//  3. values: PLAIN values copied (by rank where the chunk has NULLs), or
//     dictionary indices expanded from the hybrid stream and gathered from the
//     dictionary with the reference's bounds check, each widened on the way
//     (DECIMAL's INT64 to Int128 as Int128From); a dictionary chunk with NULLs
//     writes its non-NULL values densely and
//  4. scatters them to their rows by rank.
//
// A hybrid stream's run headers lie one run apart, so walking them is a chain of
// dependent reads. Writers cut long stretches into equal runs; once a header is
// known, the next 32 such headers are read at once at its stride, and as many as
// hold the same byte are runs of the same length (a header fixes its run's
// bytes, so each match proves the next position). One thread walking every
// header, and one CTA per page, held 2^21 rows of five columns to 1.9 ms of
// kernels, 0.14 ms now (values 76 us, levels 27, scatter 23).
#include "wg_internal.h"
#include "wg_device.cuh"

#include <cub/cub.cuh>

#include <algorithm>
#include <climits>

using namespace wg;

struct wg_batch {
  wg::Ctx* ctx = nullptr;
  std::vector<wg::DevBuf> data, valid;  // an uploaded batch's columns
  wg::DevBuf arena;                     // a decoded batch's columns, values and validity words
  wg::DevBuf sel;
  std::vector<wg_column> cols;
  int64_t len = 0, sel_len = 0;
  bool has_sel = false;
};

namespace {

using namespace wgd;

constexpr int kPageThreads = 256;
constexpr int kRuns = 256;
constexpr int64_t kSliceRows = 8192;
constexpr int kMaxSlices = 64;

struct PageD {
  int64_t row0, n;            // the page's rows within the chunk
  int64_t def_off, def_len;   // level bytes in the batch's byte image (def_len < 0: no levels)
  int64_t data_off, data_len; // values section in the byte image
  int32_t enc;
  int32_t chunk;
};

struct ChunkD {
  int32_t es;              // physical width: 4 or 8
  int32_t widen;           // INT64 DECIMAL values to Int128
  int32_t nullable;        // some page has definition levels
  int32_t dict_enc;        // some page is dictionary-encoded
  int64_t dict_off;        // the dictionary's values in the byte image
  int64_t dict_len;
  uint8_t* vbytes;         // valid flag per row of the chunk
  uint64_t* vwords;        // validity words
  int64_t word0;           // the chunk's first word in the batch's popcount prefix
  char* dense;             // non-NULL values in row order (the column itself when nothing is NULL)
  char* out;               // the column
  int64_t rows;
};

struct BatchArgs {
  const ChunkD* chunks;
  const PageD* pages;
  const uint8_t* bytes;                 // byte image: pages, dictionaries
  const unsigned long long* wprefix;    // non-NULL rows before each 64-row word, over all nullable chunks
  unsigned long long* wcount;
  int32_t* err;
};

struct Run {
  int64_t out0, n;    // values [out0, out0 + n) of the stream
  int64_t off, blen;  // bit-packed: the run's bytes
  int32_t kind;       // 0 = repeated value, 1 = bit-packed
  int32_t value;
};

// Value j of a bit-packed run whose bytes are p[0, blen): the reference reads
// up to four little-endian bytes from the value's first byte, bytes past the
// run's end reading as zero, and masks bit_width bits (decodeBitPackedRange,
// rle.go:214-250). The two aligned words that hold the four bytes are read; the
// byte image ends with at least eight spare bytes.
__device__ __forceinline__ int32_t bitpacked_value(const uint8_t* p, int64_t blen, int bw, int64_t j) {
  if (bw == 0) return 0;
  const int64_t bit = j * bw;
  const int64_t byte = bit >> 3;
  const int sh = (int)(bit & 7);
  const int64_t rem = blen - byte;
  if (rem <= 0) return 0;
  const uintptr_t a = reinterpret_cast<uintptr_t>(p + byte);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
  uint32_t raw = __funnelshift_r(__ldg(w), __ldg(w + 1), (uint32_t)(a & 3) * 8);
  if (rem < 4) raw &= (1u << (8 * (uint32_t)rem)) - 1u;
  const int32_t mask = bw >= 32 ? -1 : (int32_t)((1u << bw) - 1u);
  return (int32_t)(raw >> sh) & mask;
}

// Values [k0, k1) of the RLE / bit-packed hybrid stream p[0, len) with bit
// width bw and `count` values, handed to sink(k, value) (decodeAllBatch,
// rle.go:219-275). Every thread of the CTA calls it. A stream that ends before
// k1, a varint that runs off it or a repeated value missing its bytes sets
// WG_DERR_BAD_PAGE, as the reference returns an error there; the slice that
// ends at `count` walks the whole stream.
template <class Sink>
__device__ void hybrid_decode(const uint8_t* p, int64_t len, int bw, int64_t count, int64_t k0, int64_t k1,
                              const Sink& sink, int32_t* err) {
  __shared__ Run runs[kRuns];
  __shared__ int s_nruns, s_done;
  const int lane = threadIdx.x & 31;
  const int vbytes = (bw + 7) / 8;
  int64_t off = 0, pos = 0;  // warp 0's walk
  for (;;) {
    if (threadIdx.x < 32) {
      int nr = 0, done = 0;
      while (nr + 32 <= kRuns) {
        if (off >= len || pos >= k1) { done = 1; break; }
        const uint32_t b0 = p[off];
        if (b0 & 0x80) {  // a longer varint: one run, every lane the same walk
          unsigned long long h = 0;
          int shift = 0;
          bool ok = false;
          while (off < len && shift < 64) {
            const uint8_t b = p[off++];
            h |= (unsigned long long)(b & 0x7F) << shift;
            if (!(b & 0x80)) { ok = true; break; }
            shift += 7;
          }
          if (!ok) { if (lane == 0) set_error(err, WG_DERR_BAD_PAGE); done = 1; break; }
          Run r;
          r.out0 = pos;
          r.off = 0;
          r.blen = 0;
          r.value = 0;
          if ((h & 1ULL) == 0) {  // repeated value: count = header >> 1, then ceil(bw / 8) value bytes
            const int64_t c = (int64_t)(h >> 1);
            if (off + vbytes > len) { if (lane == 0) set_error(err, WG_DERR_BAD_PAGE); done = 1; break; }
            for (int i = 0; i < vbytes; ++i) r.value |= (int32_t)p[off + i] << (8 * i);
            off += vbytes;
            r.kind = 0;
            r.n = c < count - pos ? c : count - pos;
          } else {  // bit-packed: header >> 1 groups of 8 values, groups * bw bytes
            const int64_t groups = (int64_t)(h >> 1);
            if (groups <= 0) continue;
            if (groups > LLONG_MAX / 8 || (bw > 0 && groups > LLONG_MAX / bw)) {
              if (lane == 0) set_error(err, WG_DERR_BAD_PAGE);
              done = 1;
              break;
            }
            const int64_t nv = groups * 8;
            r.kind = 1;
            r.n = nv < count - pos ? nv : count - pos;
            r.off = off;
            int64_t bc = groups * bw;
            if (bc > len - off) bc = len - off;
            r.blen = bc;
            off += bc;
          }
          pos += r.n;
          if (r.n > 0 && pos > k0) {
            if (lane == 0) runs[nr] = r;
            ++nr;
          }
          continue;
        }
        if (b0 == 1) { ++off; continue; }  // a bit-packed run of no groups
        // one-byte header: the run's bytes and values, and as many runs like it as follow
        const bool packed = b0 & 1u;
        const int64_t nv = packed ? (int64_t)(b0 >> 1) * 8 : (int64_t)(b0 >> 1);
        const int64_t body = packed ? (int64_t)(b0 >> 1) * bw : (int64_t)vbytes;
        const int64_t at = off + lane * (1 + body);
        const bool like = at < len && p[at] == b0 && (lane == 0 || nv == 0 || pos + lane * nv < k1);
        const unsigned m = __ballot_sync(WG_FULL_MASK, like);
        const int n = m == WG_FULL_MASK ? 32 : __ffs(~m) - 1;  // lane 0 always matches
        const bool mine = lane < n;
        Run r;
        r.out0 = pos + lane * nv;
        r.n = nv < count - r.out0 ? nv : count - r.out0;
        r.off = at + 1;
        r.blen = 0;
        r.value = 0;
        r.kind = packed ? 1 : 0;
        bool bad = false;
        if (packed) {
          r.blen = body < len - r.off ? body : len - r.off;
        } else if (mine) {
          bad = r.off + vbytes > len;
          for (int i = 0; i < vbytes && !bad; ++i) r.value |= (int32_t)p[r.off + i] << (8 * i);
        }
        const unsigned badm = __ballot_sync(WG_FULL_MASK, mine && bad);
        const bool keep = mine && !bad && r.n > 0 && r.out0 + r.n > k0;
        const unsigned km = __ballot_sync(WG_FULL_MASK, keep);
        if (keep) runs[nr + __popc(km & ((1u << lane) - 1u))] = r;
        nr += __popc(km);
        if (badm) {
          if (lane == 0) set_error(err, WG_DERR_BAD_PAGE);
          done = 1;
          break;
        }
        pos += n * nv;
        if (pos > count) pos = count;
        off += n * (1 + body);
      }
      if (done && pos < k1 && lane == 0) set_error(err, WG_DERR_BAD_PAGE);  // fewer values than the page has
      if (lane == 0) {
        s_nruns = nr;
        s_done = done;
      }
    }
    __syncthreads();
    const int nr = s_nruns;
    if (nr > 0) {
      const int64_t base = runs[0].out0 > k0 ? runs[0].out0 : k0;
      const int64_t last = runs[nr - 1].out0 + runs[nr - 1].n;
      const int64_t end = last < k1 ? last : k1;
      int lo = 0;  // the last run starting at or before the thread's value: near the one before
      for (int64_t o = base + threadIdx.x; o < end; o += blockDim.x) {
        for (int step = 0; step < 4 && lo + 1 < nr && runs[lo + 1].out0 <= o; ++step) ++lo;
        if (lo + 1 < nr && runs[lo + 1].out0 <= o) {
          int hi = nr - 1;
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (runs[mid].out0 <= o) lo = mid; else hi = mid - 1;
          }
        }
        const Run& r = runs[lo];
        sink(o, r.kind == 0 ? r.value : bitpacked_value(p + r.off, r.blen, bw, o - r.out0));
      }
    }
    const int done = s_done;
    __syncthreads();  // the table is reused
    if (done) break;
  }
}

// Slice blockIdx.x of a page's n values.
__device__ __forceinline__ void slice_of(int64_t n, int64_t& k0, int64_t& k1) {
  const int64_t per = ((n + gridDim.x - 1) / gridDim.x + 63) & ~int64_t(63);
  k0 = (int64_t)blockIdx.x * per;
  k1 = k0 + per < n ? k0 + per : n;
  if (k0 > n) k0 = n;
}

__device__ __forceinline__ int64_t rank_of(const BatchArgs& a, const ChunkD& c, int64_t r) {
  if (!c.nullable) return r;
  const int64_t w = r >> 6;
  const int b = (int)(r & 63);
  const uint64_t below = b ? (c.vwords[w] & ((~0ULL) >> (64 - b))) : 0ULL;
  return (int64_t)(a.wprefix[c.word0 + w] - a.wprefix[c.word0]) + __popcll(below);
}

// One physical value (es bytes, aligned) stored at slot i of `to`, widened for DECIMAL.
__device__ __forceinline__ void put_value(const ChunkD& c, char* to, int64_t i, const uint8_t* src) {
  if (c.widen) {
    const long long v = *(const long long*)src;
    longlong2 d;
    d.x = v < 0 ? -1LL : 0LL;  // Int128From: Hi is the sign extension (decimal.go:17)
    d.y = v;
    ((longlong2*)to)[i] = d;
  } else if (c.es == 4) {
    ((uint32_t*)to)[i] = *(const uint32_t*)src;
  } else {
    ((unsigned long long*)to)[i] = *(const unsigned long long*)src;
  }
}

__device__ __forceinline__ void put_zero(const ChunkD& c, char* to, int64_t i) {
  if (c.widen) {
    longlong2 z;
    z.x = 0;
    z.y = 0;
    ((longlong2*)to)[i] = z;
  } else if (c.es == 4) {
    ((uint32_t*)to)[i] = 0u;
  } else {
    ((unsigned long long*)to)[i] = 0ULL;
  }
}

struct DefSink {
  uint8_t* v;
  __device__ __forceinline__ void operator()(int64_t k, int32_t level) const { v[k] = level == 1 ? 1 : 0; }
};

struct DictSink {
  const ChunkD& c;
  const uint8_t* dict;
  int64_t dense0;
  int32_t* err;
  __device__ __forceinline__ void operator()(int64_t k, int32_t idx) const {
    // the gather loops' bounds check (columnar_native.go:480-486): uint(idx) >= len is an error
    if ((uint64_t)(uint32_t)idx >= (uint64_t)c.dict_len) { set_error(err, WG_DERR_BAD_PAGE); return; }
    put_value(c, c.dense, dense0 + k, dict + (int64_t)(uint32_t)idx * c.es);
  }
};

// Grid (slices, pages).
__global__ void __launch_bounds__(kPageThreads) def_levels_kernel(const BatchArgs a) {
  const PageD pg = a.pages[blockIdx.y];
  const ChunkD& c = a.chunks[pg.chunk];
  if (!c.nullable) return;
  int64_t k0, k1;
  slice_of(pg.n, k0, k1);
  if (k0 >= k1) return;
  uint8_t* v = c.vbytes + pg.row0;
  if (pg.def_len < 0) {  // a required page inside a nullable chunk: every row has a value
    for (int64_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) v[k] = 1;
    return;
  }
  hybrid_decode(a.bytes + pg.def_off, pg.def_len, 1, pg.n, k0, k1, DefSink{v}, a.err);
}

// Validity words and their popcounts from the per-row flags (grid.y: chunk).
__global__ void pack_valid_kernel(const BatchArgs a) {
  const ChunkD& c = a.chunks[blockIdx.y];
  if (!c.nullable) return;
  const int64_t nwords = (c.rows + 63) / 64;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += (int64_t)gridDim.x * blockDim.x) {
    uint64_t bits = 0;
    const int64_t r0 = w * 64;
    const uint8_t* v = c.vbytes + r0;
    if (r0 + 64 <= c.rows) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {  // eight flags (0 or 1) at a time: the byte's bits gathered by a multiply
        const unsigned long long f = *(const unsigned long long*)(v + 8 * q);
        bits |= ((f * 0x0102040810204080ULL) >> 56) << (8 * q);
      }
    } else {
      for (int b = 0; r0 + b < c.rows; ++b) bits |= (uint64_t)(v[b] != 0) << b;
    }
    c.vwords[w] = bits;
    a.wcount[c.word0 + w] = (unsigned long long)__popcll(bits);
  }
}

// Grid (slices, pages).
__global__ void __launch_bounds__(kPageThreads) values_kernel(const BatchArgs a) {
  const PageD pg = a.pages[blockIdx.y];
  const ChunkD& c = a.chunks[pg.chunk];
  const int64_t d0 = rank_of(a, c, pg.row0);
  const int64_t cnt = rank_of(a, c, pg.row0 + pg.n) - d0;
  const uint8_t* data = a.bytes + pg.data_off;
  int64_t k0, k1;
  if (pg.enc == WG_ENC_PLAIN) {
    if (pg.data_len < cnt * c.es) {  // PLAIN data shorter than the page's values
      if (threadIdx.x == 0) set_error(a.err, WG_DERR_BAD_PAGE);
      return;
    }
    if (!c.nullable || c.dict_enc) {  // non-NULL values in order
      slice_of(cnt, k0, k1);
      for (int64_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) put_value(c, c.dense, d0 + k, data + k * c.es);
    } else {  // straight to their rows
      slice_of(pg.n, k0, k1);
      for (int64_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const int64_t r = pg.row0 + k;
        if ((c.vwords[r >> 6] >> (r & 63)) & 1ULL) put_value(c, c.out, r, data + (rank_of(a, c, r) - d0) * c.es);
        else put_zero(c, c.out, r);
      }
    }
    return;
  }
  // dictionary indices: one bit-width byte, then the hybrid stream
  if (cnt == 0) return;
  if (pg.data_len < 1 || data[0] > 32) {
    if (threadIdx.x == 0) set_error(a.err, WG_DERR_BAD_PAGE);
    return;
  }
  slice_of(cnt, k0, k1);
  if (k0 >= k1) return;
  hybrid_decode(data + 1, pg.data_len - 1, (int)data[0], cnt, k0, k1, DictSink{c, a.bytes + c.dict_off, d0, a.err}, a.err);
}

// Non-NULL values of the dictionary chunks with NULLs to their rows; NULL rows
// get zero bytes (grid.y: chunk).
__global__ void scatter_kernel(const BatchArgs a) {
  const ChunkD& c = a.chunks[blockIdx.y];
  if (!c.nullable || !c.dict_enc) return;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < c.rows; r += (int64_t)gridDim.x * blockDim.x) {
    if (!((c.vwords[r >> 6] >> (r & 63)) & 1ULL)) { put_zero(c, c.out, r); continue; }
    const int64_t k = rank_of(a, c, r);
    if (c.widen) ((longlong2*)c.out)[r] = ((const longlong2*)c.dense)[k];
    else if (c.es == 4) ((uint32_t*)c.out)[r] = ((const uint32_t*)c.dense)[k];
    else ((unsigned long long*)c.out)[r] = ((const unsigned long long*)c.dense)[k];
  }
}

unsigned grid_for_rows(Ctx* ctx, int64_t n, int block) {
  int64_t b = (n + block - 1) / block;
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(b, (int64_t)ctx->sm_count * 16));
}

// Physical width of a column type's PLAIN values (4 or 8), 0 when the GPU path has none.
int64_t phys_width(int32_t type_id) {
  if (type_id == WG_TYPE_DECIMAL) return 8;
  const int64_t e = elem_size(type_id);
  return e == 4 || e == 8 ? e : 0;
}

// What a chunk's pages ask for; refuses what the decode does not take.
wg_status check_chunk(const wg_column_chunk& ch, ChunkD* c, int64_t* rows) {
  if (ch.n_pages < 0 || (ch.n_pages > 0 && !ch.pages)) return fail(WG_E_INVALID, "bad column chunk");
  const int64_t es = phys_width(ch.type_id);
  if (es == 0 || elem_size(ch.type_id) == 0) return fail(WG_E_UNSUPPORTED, "column type is not on the GPU decode path");
  std::memset(c, 0, sizeof(*c));
  c->es = (int32_t)es;
  c->widen = ch.type_id == WG_TYPE_DECIMAL;
  *rows = 0;
  for (int p = 0; p < ch.n_pages; ++p) {
    const wg_page& pg = ch.pages[p];
    if (pg.num_values < 0 || pg.def_len < 0 || pg.data_len < 0 || (pg.def_len > 0 && !pg.def_levels) ||
        (pg.data_len > 0 && !pg.data))
      return fail(WG_E_INVALID, "bad page descriptor");
    if (pg.encoding != WG_ENC_PLAIN && pg.encoding != WG_ENC_PLAIN_DICTIONARY && pg.encoding != WG_ENC_RLE_DICTIONARY)
      return fail(WG_E_UNSUPPORTED, "page encoding is not on the GPU decode path (PLAIN and dictionary are)");
    if (pg.def_levels) c->nullable = 1;
    if (pg.encoding != WG_ENC_PLAIN) c->dict_enc = 1;
    *rows += pg.num_values;
  }
  if (c->dict_enc && (!ch.dict || ch.dict_len < 0)) return fail(WG_E_INVALID, "dictionary page missing");
  c->dict_len = c->dict_enc ? ch.dict_len : 0;
  return WG_OK;
}

constexpr int64_t align_up(int64_t v, int64_t a) { return (v + a - 1) & ~(a - 1); }

// Chunks [0, n_chunks) of `chunks` into their columns (cd: out, vwords and the
// checked facts set). Scratch the ledger has no room for splits the group.
wg_status decode_group(Ctx* ctx, const wg_column_chunk* chunks, ChunkD* cd, int n_chunks, int64_t rows) {
  std::vector<PageD> pd;
  std::vector<HostPiece> pieces(2);  // the chunk and page tables (set below), then the pages' bytes
  // the byte image: the chunk and page tables, then dictionaries, levels and values (16-byte aligned each)
  int64_t n_pages = 0, max_page = 0;
  bool any_null = false, any_scatter = false;
  for (int i = 0; i < n_chunks; ++i) n_pages += chunks[i].n_pages;
  const int64_t chunk_at = 0, page_at = align_up((int64_t)sizeof(ChunkD) * n_chunks, 16);
  int64_t image = align_up(page_at + (int64_t)sizeof(PageD) * n_pages, 16);
  auto place = [&](const void* src, int64_t len) {
    const int64_t at = image;
    if (len > 0) pieces.push_back(HostPiece{src, at, len});
    image += align_up(len, 16);
    return at;
  };
  int64_t nwords = 0, vbytes = 0, dense = 0;
  std::vector<int64_t> vb_at((size_t)n_chunks), dense_at((size_t)n_chunks);
  for (int i = 0; i < n_chunks; ++i) {
    const wg_column_chunk& ch = chunks[i];
    ChunkD& c = cd[i];
    if (c.nullable) {
      any_null = true;
      c.word0 = nwords;
      nwords += (rows + 63) / 64;
      vb_at[(size_t)i] = vbytes;
      vbytes += align_up(rows, 256);
      if (c.dict_enc) {
        any_scatter = true;
        dense_at[(size_t)i] = dense;
        dense += align_up(rows * elem_size(ch.type_id), 256);
      }
    }
    if (c.dict_len > 0) c.dict_off = place(ch.dict, c.dict_len * c.es);
    int64_t row = 0;
    for (int p = 0; p < ch.n_pages; ++p) {
      const wg_page& pg = ch.pages[p];
      PageD d{};
      d.row0 = row;
      d.n = pg.num_values;
      d.enc = pg.encoding;
      d.chunk = i;
      d.def_len = pg.def_levels ? pg.def_len : -1;
      d.def_off = pg.def_levels ? place(pg.def_levels, pg.def_len) : 0;
      d.data_len = pg.data_len;
      d.data_off = place(pg.data, pg.data_len);
      row += pg.num_values;
      max_page = std::max(max_page, pg.num_values);
      pd.push_back(d);
    }
  }
  image = align_up(image + 16, 256);  // bitpacked_value reads whole words
  // scratch: the byte image, valid flags, popcounts and their prefix, dense values, the scan's storage
  size_t scan_bytes = 0;
  if (any_null) {
    if (nwords >= INT_MAX) return fail(WG_E_UNSUPPORTED, "batch too large");
    cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                  (int)(nwords + 1), ctx->stream);
  }
  const int64_t vb0 = image, wc0 = vb0 + vbytes, wp0 = wc0 + align_up((nwords + 1) * 8, 256),
                dn0 = wp0 + align_up((nwords + 1) * 8, 256), sc0 = dn0 + dense;
  DevBuf scratch;
  const wg_status room = take_block(ctx, sc0 + (int64_t)scan_bytes + 256, &scratch);
  if (room == WG_E_NOMEM && n_chunks > 1) {
    const int half = n_chunks / 2;
    set_error("");
    WG_TRY(decode_group(ctx, chunks, cd, half, rows));
    return decode_group(ctx, chunks + half, cd + half, n_chunks - half, rows);
  }
  WG_TRY(room);
  char* sp = scratch.as<char>();
  for (int i = 0; i < n_chunks; ++i) {
    ChunkD& c = cd[i];
    c.dense = c.out;
    if (c.nullable) {
      c.vbytes = (uint8_t*)(sp + vb0 + vb_at[(size_t)i]);
      if (c.dict_enc) c.dense = sp + dn0 + dense_at[(size_t)i];
    }
  }
  pieces[0] = HostPiece{cd, chunk_at, (int64_t)sizeof(ChunkD) * n_chunks};
  pieces[1] = HostPiece{pd.data(), page_at, (int64_t)(sizeof(PageD) * pd.size())};
  WG_TRY(send_pieces(ctx, pieces, image, sp));
  if (rows > 0 && n_pages > 0) {
    BatchArgs a;
    a.chunks = (const ChunkD*)(sp + chunk_at);
    a.pages = (const PageD*)(sp + page_at);
    a.bytes = (const uint8_t*)sp;
    a.wcount = (unsigned long long*)(sp + wc0);
    a.wprefix = (const unsigned long long*)(sp + wp0);
    a.err = ctx->dev_error;
    const unsigned slices = (unsigned)std::max<int64_t>(1, std::min<int64_t>(kMaxSlices, (max_page + kSliceRows - 1) / kSliceRows));
    // a grid's second dimension holds 65535: more pages than that take several launches
    constexpr int64_t kPagesPerLaunch = 65535;
    const unsigned row_grid = std::max(1u, grid_for_rows(ctx, rows, 256) / (unsigned)std::max(1, std::min(n_chunks, 8)));
    if (any_null) {
      for (int64_t p0 = 0; p0 < n_pages; p0 += kPagesPerLaunch) {
        BatchArgs ap2 = a;
        ap2.pages += p0;
        def_levels_kernel<<<dim3(slices, (unsigned)std::min(kPagesPerLaunch, n_pages - p0)), kPageThreads, 0, ctx->stream>>>(ap2);
        ctx->count_launch();
      }
      WG_CUDA_TRY(cudaMemsetAsync(a.wcount + nwords, 0, 8, ctx->stream));
      pack_valid_kernel<<<dim3(std::max(1u, row_grid / 8), (unsigned)n_chunks), 256, 0, ctx->stream>>>(a);
      cub::DeviceScan::ExclusiveSum(sp + sc0, scan_bytes, a.wcount, (unsigned long long*)(sp + wp0), (int)(nwords + 1),
                                    ctx->stream);
      ctx->count_launch(2);
    }
    for (int64_t p0 = 0; p0 < n_pages; p0 += kPagesPerLaunch) {
      BatchArgs ap2 = a;
      ap2.pages += p0;
      values_kernel<<<dim3(slices, (unsigned)std::min(kPagesPerLaunch, n_pages - p0)), kPageThreads, 0, ctx->stream>>>(ap2);
      ctx->count_launch();
    }
    if (any_scatter) {
      scatter_kernel<<<dim3(row_grid, (unsigned)n_chunks), 256, 0, ctx->stream>>>(a);
      ctx->count_launch();
    }
    WG_CUDA_TRY(cudaGetLastError());
  }
  // a malformed page says so in the error word
  int32_t err = 0;
  {
    std::lock_guard<std::mutex> g(ctx->mu);
    WG_CUDA_TRY(cudaMemcpyAsync(ctx->host_scalar, ctx->dev_error, 4, cudaMemcpyDeviceToHost, ctx->stream));
    WG_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    err = *(const int32_t*)ctx->host_scalar;
  }
  park_block(ctx, &scratch);  // the stream is idle: the wait above
  const wg_status st = device_error_status(ctx, err);
  if (err == WG_DERR_BAD_PAGE)
    return fail(WG_E_INVALID, "malformed Parquet page (levels or indices end early, an index is past the "
                              "dictionary, or PLAIN data is shorter than its values)");
  return st;
}

wg_status decode_batch(Ctx* ctx, const wg_column_chunk* chunks, int n_chunks, int64_t rows, wg_batch* b) {
  std::vector<ChunkD> cd((size_t)n_chunks);
  // the columns: one allocation, values then validity words of each
  int64_t arena = 0;
  std::vector<int64_t> valid_at((size_t)n_chunks, -1);
  for (int i = 0; i < n_chunks; ++i) {
    ChunkD& c = cd[(size_t)i];
    int64_t r = 0;
    WG_TRY(check_chunk(chunks[i], &c, &r));
    if (r != rows) return fail(WG_E_INVALID, "column chunks of one batch must hold the same number of rows");
    if (rows == 0) c.nullable = 0;
    c.rows = rows;
    arena += align_up(std::max<int64_t>(rows * elem_size(chunks[i].type_id), 16), 256);
    if (c.nullable) {
      valid_at[(size_t)i] = arena;
      arena += align_up((rows + 63) / 64 * 8, 256);
    }
  }
  WG_TRY(take_block(ctx, arena, &b->arena));
  int64_t at = 0;
  for (int i = 0; i < n_chunks; ++i) {
    ChunkD& c = cd[(size_t)i];
    wg_column col{};
    c.out = b->arena.as<char>() + at;
    at += align_up(std::max<int64_t>(rows * elem_size(chunks[i].type_id), 16), 256);
    if (c.nullable) {
      c.vwords = (uint64_t*)(b->arena.as<char>() + valid_at[(size_t)i]);
      at = valid_at[(size_t)i] + align_up((rows + 63) / 64 * 8, 256);
    }
    col.type_id = chunks[i].type_id;
    col.scale = chunks[i].scale;
    col.data = c.out;
    col.valid_words = c.nullable ? c.vwords : nullptr;
    col.len = rows;
    b->cols.push_back(col);
  }
  return decode_group(ctx, chunks, cd.data(), n_chunks, rows);
}

}  // namespace

extern "C" {

wg_status wg_batch_upload(wg_ctx* ctx, const wg_batch_desc* host, wg_batch** out) {
  if (!ctx || !host || !out) return fail(WG_E_INVALID, "NULL argument");
  *out = nullptr;
  WG_TRY(ensure_device(ctx));
  StagedBatch sb;
  WG_TRY(stage_batch(ctx, host, &sb));
  WG_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  wg_batch* b = new wg_batch();
  b->ctx = ctx;
  b->data = std::move(sb.data);
  b->valid = std::move(sb.valid);
  b->sel = std::move(sb.sel);
  b->cols = sb.cols;
  b->len = host->len;
  b->has_sel = host->sel != nullptr;
  b->sel_len = host->sel_len;
  *out = b;
  return WG_OK;
}

wg_status wg_batch_decode(wg_ctx* ctx, const wg_column_chunk* chunks, int32_t n_chunks, wg_batch** out) {
  if (!ctx || !out || n_chunks < 1 || !chunks) return fail(WG_E_INVALID, "NULL argument");
  *out = nullptr;
  WG_TRY(ensure_device(ctx));
  if (chunks[0].n_pages < 0 || (chunks[0].n_pages > 0 && !chunks[0].pages)) return fail(WG_E_INVALID, "bad column chunk");
  int64_t rows = 0;
  for (int p = 0; p < chunks[0].n_pages; ++p) rows += chunks[0].pages[p].num_values;
  wg_batch* b = new wg_batch();
  b->ctx = ctx;
  b->len = rows;
  const wg_status st = decode_batch(ctx, chunks, n_chunks, rows, b);
  if (st != WG_OK) {
    cudaStreamSynchronize(ctx->stream);  // nothing still reads the buffers freed here
    delete b;
    return st;
  }
  *out = b;
  return WG_OK;
}

wg_status wg_batch_device_desc(wg_batch* b, wg_batch_desc* out, wg_column* cols, int32_t max_cols) {
  if (!b || !out) return fail(WG_E_INVALID, "NULL argument");
  const int32_t n = (int32_t)b->cols.size();
  out->ncols = n;
  out->_pad = 0;
  out->len = b->len;
  out->sel = b->has_sel ? b->sel.as<uint32_t>() : nullptr;
  out->sel_len = b->has_sel ? b->sel_len : 0;
  out->cols = cols;
  if (!cols || max_cols < n) return fail(WG_E_INVALID, "cols has room for fewer columns than the batch holds");
  for (int32_t i = 0; i < n; ++i) cols[i] = b->cols[(size_t)i];
  return WG_OK;
}

wg_status wg_batch_destroy(wg_batch* b) {
  if (!b) return WG_OK;
  ensure_device(b->ctx);
  cudaStreamSynchronize(b->ctx->stream);
  if (b->arena.get()) {
    cudaDeviceSynchronize();  // as cudaFree would: no other stream still reads the columns
    park_block(b->ctx, &b->arena);
  }
  delete b;
  return WG_OK;
}

}  // extern "C"
