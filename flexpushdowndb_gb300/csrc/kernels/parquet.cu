// Parquet column decoding on the device: the data half of Arrow's
// parquet::arrow::FileReader::ReadTable that ParquetReader::readImpl drives
// (fpdb-tuple/src/parquet/ParquetReader.cpp:12-42), after the host has read
// the footer and page headers (host/parquet_meta.cpp). The page formats are
// the public Apache Parquet specification's: PLAIN values (little-endian
// fixed width; byte arrays as a 4-byte length then the bytes), dictionary
// pages (PLAIN) with data pages of RLE / bit-packed hybrid indices behind a
// bit-width byte, definition levels of optional columns as a 4-byte length
// and an RLE / bit-packed hybrid run (v1) or a separate uncompressed prefix
// (v2), and the snappy block format.
//
// Launches:
//   parquet_snappy_kernel  one warp per snappy page: lane 0 reads each
//                          element's tag (literal, or a copy with a 1-, 2- or
//                          4-byte offset) and the warp moves its bytes, 32 at
//                          a time (copies whose source overlaps their output
//                          go in steps of the offset);
//   parquet_runs_kernel    one warp per page of more than 8,192 dictionary
//                          indices in several runs: skips (and checks) its
//                          definition levels and finds the run that each
//                          8,192nd index lies in;
//   parquet_pages_kernel   one CTA per 8,192 values of a page: thread 0 walks
//                          byte-array lengths (data and dictionary pages) and
//                          reads the dictionary indices' run headers, up to
//                          256 a round, and every thread then decodes the
//                          round's indices that lie in the CTA's part of the
//                          page, a fixed-width column's straight into its
//                          values;
//   parquet_values_kernel  per plain data page and value: fixed-width values
//                          copied into the output column; byte arrays (plain
//                          or dictionary-encoded) get their source and
//                          length;
//   then per utf8 column a prefix sum of the lengths and a byte copy.
#include <algorithm>
#include <cstring>
#include <vector>

#include "../host/parquet_meta.h"
#include "common.cuh"
#include "launch.h"

namespace gfpdb {
namespace {

struct PageDev {
  const uint8_t* body;    // page body on the device (after its header)
  uint8_t* inflated;      // snappy pages: the decompressed body (v2: the values part)
  const uint8_t* values;  // set by parquet_runs_kernel or parquet_pages_kernel: the first value byte
  int32_t body_len;
  int32_t inflated_len;
  int32_t values_len;     // set with `values`
  int32_t type;           // PageType
  int32_t encoding;
  int32_t snappy;         // 1: the values live in `inflated`
  int32_t num_values;
  int32_t v2_levels;      // data page v2: level bytes ahead of the values
  int32_t v1_def;         // data page v1 of an optional column
  int32_t width;          // fixed-width bytes, 0 for byte arrays
  int32_t dict_page;      // data pages: their dictionary page's index, -1
  int32_t n_parts;
  int32_t walked;         // 1: parquet_runs_kernel has set values and the parts' runs
  int32_t first_part;     // its first part in the read's list
  int32_t late_from;      // the parts from this value on are decoded in the read's second round (kPqNever: none)
  int32_t walk_at, walk_done;  // where the walk over the runs stopped: a header's place, the values before it
  int64_t first_row;
  int64_t dict_base;      // byte-array dictionary pages: first entry in dict_ptr / dict_len
  int32_t* idx;           // dictionary-encoded columns: per-row entry
  uint64_t* row_ptr;      // byte-array columns: per-row value address
  int32_t* row_len;       //   and length
  uint8_t* fixed_out;     // fixed-width columns: the output values
};

struct DictArrays {
  uint64_t* ptr;  // byte-array dictionary entries: address
  int32_t* len;   //   and length
};

__device__ __forceinline__ uint32_t le32(const uint8_t* p) {
  return static_cast<uint32_t>(p[0]) | (static_cast<uint32_t>(p[1]) << 8) | (static_cast<uint32_t>(p[2]) << 16) |
         (static_cast<uint32_t>(p[3]) << 24);
}

// Snappy block format: a varint of the uncompressed length, then elements.
__device__ void snappy_warp(const uint8_t* src, int32_t n, uint8_t* dst, int32_t cap, DevStatus* st, int page) {
  const int lane = threadIdx.x & 31;
  int32_t ip = 0;
  int ok = 1;
  if (lane == 0) {
    uint32_t ulen = 0;
    int shift = 0;
    ok = 0;
    while (ip < n && shift <= 28) {
      const uint8_t b = src[ip++];
      ulen |= static_cast<uint32_t>(b & 0x7f) << shift;
      if (!(b & 0x80)) {
        ok = ulen == static_cast<uint32_t>(cap) ? 1 : 0;
        break;
      }
      shift += 7;
    }
  }
  ok = __shfl_sync(0xffffffffu, ok, 0);
  if (!ok) {
    if (lane == 0) raise_status(st, GFPDB_EINVAL, 100000 + page);
    return;
  }
  int32_t op = 0;
  for (;;) {
    int32_t kind = 0, len = 0, off = 0, lit = 0;
    if (lane == 0) {
      if (ip >= n) {
        kind = -1;
      } else {
        const uint8_t tag = src[ip++];
        const int t = tag & 3;
        if (t == 0) {
          len = (tag >> 2) + 1;
          if (len > 60) {
            const int nb = len - 60;
            len = 0;
            if (ip + nb > n) {
              kind = -2;
            } else {
              for (int k = 0; k < nb; ++k) len |= static_cast<int32_t>(src[ip + k]) << (8 * k);
              ip += nb;
              len += 1;
            }
          }
          lit = ip;
          ip += len;
          if (kind == 0) kind = (len <= 0 || ip > n) ? -2 : 1;
        } else {
          const int nb = t == 1 ? 1 : (t == 2 ? 2 : 4);
          if (ip + nb > n) {
            kind = -2;
          } else {
            if (t == 1) {
              len = 4 + ((tag >> 2) & 7);
              off = ((tag >> 5) << 8) | src[ip];
            } else {
              len = 1 + (tag >> 2);
              off = t == 2 ? (src[ip] | (src[ip + 1] << 8)) : static_cast<int32_t>(le32(src + ip));
            }
            ip += nb;
            kind = (off <= 0 || off > op) ? -2 : 2;
          }
        }
        if (kind > 0 && (len > cap - op)) kind = -2;
      }
    }
    kind = __shfl_sync(0xffffffffu, kind, 0);
    if (kind < 0) {
      if (kind == -2 && lane == 0) raise_status(st, GFPDB_EINVAL, 100000 + page);
      break;
    }
    len = __shfl_sync(0xffffffffu, len, 0);
    off = __shfl_sync(0xffffffffu, off, 0);
    lit = __shfl_sync(0xffffffffu, lit, 0);
    if (kind == 1) {
      for (int32_t i = lane; i < len; i += 32) dst[op + i] = src[lit + i];
    } else {
      const int32_t step = off < 32 ? off : 32;  // a step never reads what it writes
      for (int32_t base = 0; base < len; base += step) {
        const int32_t i = base + lane;
        if (lane < step && i < len) dst[op + i] = dst[op + i - off];
        __syncwarp();
      }
    }
    __syncwarp();
    op += len;
  }
  if (lane == 0 && op != cap) raise_status(st, GFPDB_EINVAL, 100000 + page);
}

__global__ void __launch_bounds__(256) parquet_snappy_kernel(PageDev* pages, const int32_t* list, int32_t n,
                                                             DevStatus* st) {
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t w = warp; w < n; w += warps) {
    __syncwarp();
    const int p = list[w];
    const PageDev& pg = pages[p];
    const int32_t skip = pg.type == parquet::PAGE_DATA_V2 ? pg.v2_levels : 0;
    snappy_warp(pg.body + skip, pg.body_len - skip, pg.inflated, pg.inflated_len, st, p);
  }
}

// One run header of an RLE / bit-packed hybrid stream at p[*at]: returns
// false past the end.
__device__ __forceinline__ bool run_header(const uint8_t* p, int32_t n, int32_t* at, uint32_t* h) {
  uint32_t v = 0;
  for (int shift = 0; shift <= 28; shift += 7) {
    if (*at >= n) return false;
    const uint8_t b = p[(*at)++];
    v |= static_cast<uint32_t>(b & 0x7f) << shift;
    if (!(b & 0x80)) {
      *h = v;
      return true;
    }
  }
  return false;
}

__device__ __forceinline__ void copy_value(const uint8_t* src, uint8_t* dst, int w) {
  if (w == 8 && !(reinterpret_cast<uintptr_t>(src) & 7)) {
    *reinterpret_cast<uint64_t*>(dst) = *reinterpret_cast<const uint64_t*>(src);
  } else if (w == 4 && !(reinterpret_cast<uintptr_t>(src) & 3)) {
    *reinterpret_cast<uint32_t*>(dst) = *reinterpret_cast<const uint32_t*>(src);
  } else {
    for (int k = 0; k < w; ++k) dst[k] = src[k];
  }
}

constexpr int kPqThreads = 256;
constexpr int kPqRuns = 256;  // run headers read per round
// Dictionary indices of a page that one CTA decodes: 32 per thread. One CTA
// per page left most SMs without a warp (a 4M-row, 7-column file of
// 131,072-row pages is 237 pages; the pass took 460 us at 12% occupancy) and
// the longest page set its length; with parts, word-wide index reads and one
// copy per span of chunks the whole read of that file went from 1,118 to 680 us
// (653 with copying and decoding overlapped, see kPqBatch).
constexpr int kPqPart = 8192;
constexpr int32_t kPqNever = INT32_MAX;

struct PagePart {
  int32_t page;
  int32_t first;     // the part's first value in the page
  int32_t at, done;  // the run it lies in: the header's place among the page's values, the values before the run
};

// The page's values, behind its levels. With definition levels, false (and an
// error) where one says null or they are malformed. One thread.
__device__ bool page_values(const PageDev& pg, int32_t w, DevStatus* st, const uint8_t** values, int32_t* values_len) {
  const uint8_t* base;
  int32_t blen;
  if (pg.snappy) {
    base = pg.inflated;
    blen = pg.inflated_len;
  } else {
    const int32_t skip = pg.type == parquet::PAGE_DATA_V2 ? pg.v2_levels : 0;
    base = pg.body + skip;
    blen = pg.body_len - skip;
  }
  int ok = 1;
  if (pg.v1_def) {  // 4-byte length, then the levels: every one must be 1 (no nulls)
    ok = 0;
    if (blen >= 4) {
      const int32_t len = static_cast<int32_t>(le32(base));
      if (len >= 0 && len <= blen - 4) {
        const uint8_t* lv = base + 4;
        int32_t at = 0, seen = 0;
        ok = 1;
        while (seen < pg.num_values && ok) {
          uint32_t h;
          if (!run_header(lv, len, &at, &h)) {
            ok = 0;
            break;
          }
          if (h & 1) {  // bit-packed: (h >> 1) groups of 8 one-bit levels
            const int32_t bytes = static_cast<int32_t>(h >> 1);
            if (bytes > len - at) {
              ok = 0;
              break;
            }
            for (int32_t b = 0; b < bytes && ok; ++b) {
              const int32_t valid = pg.num_values - seen - 8 * b;
              const uint32_t need = valid >= 8 ? 0xffu : ((1u << (valid > 0 ? valid : 0)) - 1u);
              if ((lv[at + b] & need) != need) ok = 0;  // a 0 level: a null
            }
            at += bytes;
            seen += 8 * bytes;
          } else {  // RLE: (h >> 1) copies of a one-byte level
            if (at >= len || lv[at] != 1) {
              ok = 0;
              break;
            }
            ++at;
            seen += static_cast<int32_t>(h >> 1);
          }
        }
        base += 4 + len;
        blen -= 4 + len;
      }
    }
    if (!ok) raise_status(st, GFPDB_EUNSUPPORTED, 200000 + w);  // nulls, or bad levels
  }
  *values = base;
  *values_len = blen;
  return ok != 0;
}

// One warp per page of several parts and runs: where each part's first run
// begins, so that no part walks the headers of the ones before it. 16M rows of
// four columns in 1M-value pages of 504-value runs, as Arrow writes them, take
// 1.4 ms, of 8-value runs 7.8 ms (8.4 and 211 with each part walking from the
// page's first run, 6.4 and 35 with a CTA per page). A header's place follows from the one before. The page goes through
// shared memory kPqWindow bytes at a time, so that short runs cost no memory
// round trip each, and runs of one length, the usual case, are taken up to 32 a
// step: each lane looks for the same header where it would be.
//
// Batches are decoded one after the other, so a page of many runs that all
// differ would hold up the ones behind it, each in turn: after `steps` steps
// the walk stops, and the page's remaining parts wait for the read's second
// round, in which the walks of all its pages go on together.
constexpr int kPqWindow = 1024;
constexpr int kPqWalkThreads = 128;

__global__ void __launch_bounds__(kPqWalkThreads) parquet_runs_kernel(PageDev* pages, const int32_t* list, int32_t n,
                                                                      PagePart* parts, int32_t steps, int32_t late,
                                                                      DevStatus* st) {
  __shared__ uint4 s_window[kPqWalkThreads / 32][kPqWindow / 16];
  const int lane = threadIdx.x & 31;
  uint4* const window = s_window[threadIdx.x >> 5];
  const uint8_t* const bytes = reinterpret_cast<const uint8_t*>(window);
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t item = warp; item < n; item += warps) {
    const int32_t w = list[item];
    PageDev& pg = pages[w];
    const int32_t num_values = pg.num_values, n_parts = pg.n_parts;
    PagePart* const part = parts + pg.first_part;
    int32_t at = 1, done = 0;
    if (late) {
      if (pg.late_from == kPqNever) continue;
      at = pg.walk_at;
      done = pg.walk_done;
    } else {
      if (lane == 0) {
        const uint8_t* values = nullptr;
        int32_t len = 0;
        const bool ok = page_values(pg, w, st, &values, &len);
        pg.values = ok ? values : nullptr;
        pg.values_len = ok ? len : 0;
      }
      __syncwarp();
    }
    const uint8_t* const base = pg.values;
    const int32_t blen = pg.values_len;
    const int bw = blen > 0 ? base[0] : 99;
    if (bw > 32) continue;  // the parts report it
    int32_t next = done > kPqPart ? (done + kPqPart - 1) / kPqPart : 1;  // the first part that is not found yet
    int64_t from = 0, to = 0;  // the window: bytes [from, to) of the values, all of them real ones
    int pad = 0;               // bytes of the window before `from`
    for (int32_t step = 0; next < n_parts; ++step) {
      if (step == steps) {
        if (lane == 0) {
          pg.late_from = next * kPqPart;
          pg.walk_at = at;
          pg.walk_done = done;
          st->aux[0] = 1;
        }
        break;
      }
      if (at + 5 > to && to < blen) {  // a header is 5 bytes at most
        // whole 16-byte lines (the buffers start on one, and end 16 bytes
        // after the last page)
        __syncwarp();
        const uintptr_t first = reinterpret_cast<uintptr_t>(base + at) & ~uintptr_t{15};
        pad = static_cast<int>(reinterpret_cast<uintptr_t>(base + at) - first);
        from = at;
        to = at + kPqWindow - pad;
        if (to > blen) to = blen;
#pragma unroll
        for (int k = 0; k < kPqWindow / 16 / 32; ++k) {
          const uintptr_t line = first + 16 * static_cast<uintptr_t>(lane + 32 * k);
          if (line < reinterpret_cast<uintptr_t>(base + blen)) window[lane + 32 * k] = __ldg(reinterpret_cast<const uint4*>(line));
        }
        __syncwarp();
      }
      // runs that all differ, with one-byte headers: one after the other
      const int shift = pad - static_cast<int>(from);  // window byte of value byte 0
      if (at < to) {
        uint32_t h = bytes[at + shift];
        for (; step != steps; ++step) {
          const int32_t count = h & 1 ? static_cast<int32_t>(h >> 1) * 8 : static_cast<int32_t>(h >> 1);
          const int32_t after = at + 1 + (h & 1 ? static_cast<int32_t>(h >> 1) * bw : (bw + 7) / 8);
          if (h >= 0x80 || count == 0 || after + 5 > to) break;
          const uint32_t h2 = bytes[after + shift];
          if (h2 == h) break;
          if (count > num_values - done) break;
          done += count;
          for (; next < n_parts && next * kPqPart < done; ++next)
            if (lane == 0) {
              part[next].at = at;
              part[next].done = done - count;
            }
          at = after;
          h = h2;
        }
        if (next >= n_parts) break;
        if (step == steps) {
          --step;  // the loop's head sees it again
          continue;
        }
      }
      const uint8_t* const here = bytes + at + shift;
      int32_t head = 0;
      uint32_t h = 0;
      bool good = run_header(here, static_cast<int32_t>(to - at), &head, &h);
      const int64_t body = h & 1 ? static_cast<int64_t>(h >> 1) * bw : (bw + 7) / 8;
      const int64_t count = h & 1 ? static_cast<int64_t>(h >> 1) * 8 : h >> 1;
      good = good && count > 0 && body <= blen - at - head;
      if (!good) {  // the parts from here on meet it and report it
        for (int32_t p = next + lane; p < n_parts; p += 32) {
          part[p].at = at;
          part[p].done = done;
        }
        break;
      }
      // the same header where this lane's run would be: in the window first,
      // beyond it only if no lane's run there differs
      const int64_t stride = head + body;
      const int64_t mine = at + lane * stride, before = done + lane * count;
      const bool fits = mine + stride <= blen, near = mine + head <= to;
      auto same = [&](const uint8_t* there) {
        for (int b = 0; b < head; ++b)
          if (there[b] != here[b]) return false;
        return true;
      };
      const int in_window = __popc(__ballot_sync(0xffffffffu, near));
      uint32_t differs = __ballot_sync(0xffffffffu, !fits || (near && !same(bytes + mine + shift)));
      if (differs == 0 || __ffs(static_cast<int>(differs)) - 1 >= in_window)
        differs |= __ballot_sync(0xffffffffu, fits && !near && !same(base + mine));
      const int runs = differs != 0 ? __ffs(static_cast<int>(differs)) - 1 : 32;  // 1 at least
      if (lane < runs) {
        int64_t p = (before + kPqPart - 1) / kPqPart;
        for (p = p < 1 ? 1 : p; p < n_parts && p * kPqPart < before + count; ++p) {
          part[p].at = static_cast<int32_t>(mine);
          part[p].done = static_cast<int32_t>(before);
        }
      }
      const int64_t reached = done + runs * count;
      if (reached >= num_values) break;
      at += static_cast<int32_t>(runs * stride);
      done = static_cast<int32_t>(reached);
      next = done > kPqPart ? (done + kPqPart - 1) / kPqPart : 1;
    }
  }
}

// One CTA per part of a page: kPqPart consecutive values where the page
// holds dictionary indices, the whole of any other page. Thread 0
// does the sequential parts (byte-array lengths, and the run headers from the
// part's first run, or its page's, to its end; pages that are not walked have
// their levels skipped here too); the dictionary indices of each round of up to kPqRuns runs that lie in
// the part are then decoded by every thread, a value finding its run by binary
// search over the runs' first values. A fixed-width column's
// index is looked up in its dictionary page at once and the value written
// to the output column (the dictionary page's body is read as the host laid
// it out, not through fields another CTA of this launch sets); a byte-array
// column's index is kept for parquet_values_kernel, which runs after the
// dictionary pages' entries are known.
__global__ void __launch_bounds__(kPqThreads) parquet_pages_kernel(PageDev* pages, int32_t n_pages,
                                                                   const PagePart* __restrict__ items, int64_t n_items,
                                                                   int32_t late, DictArrays dicts, DevStatus* st) {
  __shared__ int32_t s_first[kPqRuns + 1];  // the page value index each run starts at; then the round's end
  __shared__ int32_t s_start[kPqRuns];      // bit-packed runs: first byte; RLE runs: -1
  __shared__ uint32_t s_value[kPqRuns];     // RLE runs: the value
  __shared__ int32_t s_n, s_ok, s_at, s_done, s_bw, s_blen;
  __shared__ const uint8_t* s_base;
  __shared__ uint4 s_window[kPqWindow / 16];
  for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x) {
    __syncthreads();  // the previous part's shared state is no longer read
    const PagePart part = items[item];
    const int32_t w = part.page;
    PageDev& pg = pages[w];
    const int32_t part_lo = part.first;
    if ((part_lo >= pg.late_from) != (late != 0)) continue;  // the read's other round decodes it
    const int32_t num_values = pg.num_values;
    const int32_t part_hi = num_values - part_lo < kPqPart ? num_values : part_lo + kPqPart;
    const uint8_t* base;
    int32_t blen;
    if (threadIdx.x == 0) {
      int ok = 1;
      if (pg.walked) {
        base = pg.values;
        blen = pg.values_len;
        ok = base != nullptr;  // else parquet_runs_kernel has reported why
      } else {
        ok = page_values(pg, w, st, &base, &blen);
        if (ok && part_lo == 0) {  // for parquet_values_kernel
          pg.values = base;
          pg.values_len = blen;
        }
      }
      s_base = base;
      s_blen = blen;
      if (ok) {
        // (a page walked or checked here has one part)
        const bool bytes_walk = pg.width == 0 && (pg.type == parquet::PAGE_DICTIONARY || pg.encoding == parquet::ENC_PLAIN);
        if (bytes_walk) {  // byte arrays: each value's address and length
          const bool dict = pg.type == parquet::PAGE_DICTIONARY;
          int32_t at = 0;
          for (int32_t e = 0; e < pg.num_values; ++e) {
            int32_t len = -1;
            if (blen - at >= 4) {
              len = static_cast<int32_t>(le32(base + at));
              at += 4;
            }
            if (len < 0 || len > blen - at) {
              raise_status(st, GFPDB_EINVAL, (dict ? 300000 : 400000) + w);
              ok = 0;
              break;
            }
            if (dict) {
              dicts.ptr[pg.dict_base + e] = reinterpret_cast<uint64_t>(base + at);
              dicts.len[pg.dict_base + e] = len;
            } else {
              pg.row_ptr[pg.first_row + e] = reinterpret_cast<uint64_t>(base + at);
              pg.row_len[pg.first_row + e] = len;
            }
            at += len;
          }
        } else if (pg.width > 0 && (pg.type == parquet::PAGE_DICTIONARY || pg.encoding == parquet::ENC_PLAIN) &&
                   static_cast<int64_t>(pg.num_values) * pg.width > blen) {
          raise_status(st, GFPDB_EINVAL, 400000 + w);
          ok = 0;
        }
      }
      const bool indices = ok && pg.type != parquet::PAGE_DICTIONARY && pg.encoding != parquet::ENC_PLAIN;
      s_bw = blen > 0 ? base[0] : 99;
      if (indices && (s_bw > 32 || pg.dict_page < 0 || pg.dict_page >= n_pages)) {
        raise_status(st, GFPDB_EINVAL, 500000 + w);
        ok = 0;
      }
      s_ok = indices ? ok : 0;
      s_at = part.at;
      s_done = part.done;
    }
    __syncthreads();
    if (!s_ok) continue;
    // Dictionary indices: a bit-width byte, then RLE / bit-packed hybrid runs.
    base = s_base;
    blen = s_blen;
    const int32_t bw = s_bw;
    const uint32_t mask = bw == 32 ? 0xffffffffu : ((1u << bw) - 1u);
    const int32_t width = pg.width;
    const int64_t first_row = pg.first_row;
    uint8_t* const fixed_out = pg.fixed_out;
    int32_t* const idx_out = pg.idx;
    // a fixed-width column's dictionary: its page's values as laid out on
    // the host (dictionary pages carry no levels), its entry count and bytes
    const uint8_t* dvals = nullptr;
    int64_t dlen = 0;
    int32_t dn = 0;
    if (width > 0) {
      const PageDev& dp = pages[pg.dict_page];
      dvals = dp.snappy ? dp.inflated : dp.body;
      dlen = dp.snappy ? dp.inflated_len : dp.body_len;
      dn = dp.num_values;
    }
    for (;;) {
      // the next kPqWindow bytes: a header read from memory waits for the one
      // before it, from shared memory it costs a tenth of that
      const int32_t from = s_at;
      const uintptr_t line = reinterpret_cast<uintptr_t>(base + from) & ~uintptr_t{15};
      const int pad = static_cast<int>(reinterpret_cast<uintptr_t>(base + from) - line);
      const int32_t to = blen - from < kPqWindow - pad ? blen : from + kPqWindow - pad;
      if (threadIdx.x < kPqWindow / 16 && line + 16 * threadIdx.x < reinterpret_cast<uintptr_t>(base + to))
        s_window[threadIdx.x] = __ldg(reinterpret_cast<const uint4*>(line) + threadIdx.x);
      __syncthreads();
      if (threadIdx.x == 0) {
        const uint8_t* const window = reinterpret_cast<const uint8_t*>(s_window) + pad;
        int32_t n = 0, at = from, done = s_done;
        while (n < kPqRuns && done < part_hi) {
          if (at + 9 > to && to < blen) break;  // a header or an RLE run may go past the window
          uint32_t h;
          int32_t head = 0;
          if (!run_header(window + (at - from), to - at, &head, &h)) {
            s_ok = 0;
            break;
          }
          at += head;
          int64_t count;
          if (h & 1) {
            const int64_t groups = h >> 1;
            if (groups * bw > blen - at) {
              s_ok = 0;
              break;
            }
            s_start[n] = at;
            at += static_cast<int32_t>(groups * bw);
            count = groups * 8;
          } else {
            const int32_t vb = (bw + 7) / 8;
            if (vb > blen - at) {
              s_ok = 0;
              break;
            }
            uint32_t v = 0;
            for (int k = 0; k < vb; ++k) v |= static_cast<uint32_t>(window[at - from + k]) << (8 * k);
            at += vb;
            s_start[n] = -1;
            s_value[n] = v;
            count = h >> 1;
          }
          if (count <= 0) {
            s_ok = 0;
            break;
          }
          s_first[n] = done;
          done += static_cast<int32_t>(count < num_values - done ? count : num_values - done);
          if (done > part_lo) ++n;  // a run wholly before the part is passed over
        }
        s_first[n] = done;
        s_n = s_ok ? n : -1;
        s_at = at;
        s_done = done;
        if (!s_ok) raise_status(st, GFPDB_EINVAL, 500000 + w);
      }
      __syncthreads();
      const int32_t n = s_n;
      if (n < 0) break;
      const int32_t v0 = s_first[0] > part_lo ? s_first[0] : part_lo, v1 = s_first[n] < part_hi ? s_first[n] : part_hi;
      // unrolled so that several values' loads are in flight together
#pragma unroll 4
      for (int32_t v = v0 + static_cast<int32_t>(threadIdx.x); v < v1; v += kPqThreads) {
        int32_t lo = 0, hi = n - 1;  // the run holding v: the last with s_first <= v
        while (lo < hi) {
          const int32_t mid = (lo + hi + 1) >> 1;
          if (s_first[mid] <= v) lo = mid;
          else hi = mid - 1;
        }
        uint32_t idx;
        if (s_start[lo] < 0) {
          idx = s_value[lo];
        } else {
          // the value's bits from the two aligned words around them (32 bits
          // at most; the buffers start 16-byte aligned and carry 16 bytes of
          // tail padding)
          const int64_t bit = static_cast<int64_t>(v - s_first[lo]) * bw;
          const uintptr_t q = reinterpret_cast<uintptr_t>(base + s_start[lo]) + static_cast<uintptr_t>(bit >> 3);
          const uint32_t* al = reinterpret_cast<const uint32_t*>(q & ~uintptr_t{3});
          const uint32_t sh = 8u * static_cast<uint32_t>(q & 3u) + static_cast<uint32_t>(bit & 7);
          idx = __funnelshift_r(__ldg(al), __ldg(al + 1), sh) & mask;
        }
        if (width > 0) {
          if (idx >= static_cast<uint32_t>(dn) || (static_cast<int64_t>(idx) + 1) * width > dlen) {
            raise_status(st, GFPDB_EINVAL, 600000 + w);
            continue;
          }
          // the value's 4-byte words from the two aligned words around each
          // (the arena and the inflated buffer carry 16 bytes of tail padding)
          const uint8_t* sp = dvals + static_cast<int64_t>(idx) * width;
          const uint32_t* al = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(sp) & ~uintptr_t{3});
          const uint32_t sh = 8u * static_cast<uint32_t>(reinterpret_cast<uintptr_t>(sp) & 3u);
          const uint32_t w0 = __ldg(al), w1 = __ldg(al + 1);
          if (width == 4) {
            reinterpret_cast<uint32_t*>(fixed_out)[first_row + v] = __funnelshift_r(w0, w1, sh);
          } else {
            const uint2 d = make_uint2(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, __ldg(al + 2), sh));
            reinterpret_cast<uint2*>(fixed_out)[first_row + v] = d;
          }
        } else {
          idx_out[first_row + v] = static_cast<int32_t>(idx);
        }
      }
      const bool more = s_done < part_hi;
      __syncthreads();  // the runs are read before thread 0 rewrites them
      if (!more) break;
    }
  }
}

// blockIdx.y: a data page (index into `list`, whose first is the read's
// first-th); values over x.
__global__ void __launch_bounds__(256) parquet_values_kernel(const PageDev* pages, const int32_t* list, int32_t first,
                                                             int32_t late, DictArrays dicts, DevStatus* st) {
  const PageDev& pg = pages[list[blockIdx.y]];
  const bool dict = pg.encoding != parquet::ENC_PLAIN;
  const PageDev* dp = dict ? &pages[pg.dict_page] : nullptr;
  // the read's other round has all its indices, or its dictionary
  if ((pg.late_from != kPqNever || (dict && dp->late_from != kPqNever)) != (late != 0)) return;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < pg.num_values; i += stride) {
    const int64_t row = pg.first_row + i;
    if (pg.width > 0) {
      // bounds: a page whose levels or sizes were bad has values_len 0
      // plain values only: a fixed-width dictionary page is decoded to its
      // values by the page pass and never listed here
      if (dict || (i + 1) * pg.width > pg.values_len) {
        raise_status(st, GFPDB_EINVAL, 600000 + first + static_cast<int32_t>(blockIdx.y));
        continue;
      }
      // the value's 4-byte words from the two aligned words around each
      // (the arena and the inflated buffer carry 16 bytes of tail padding)
      const uint8_t* sp = pg.values + i * pg.width;
      const uint32_t* al = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(sp) & ~uintptr_t{3});
      const uint32_t sh = 8u * static_cast<uint32_t>(reinterpret_cast<uintptr_t>(sp) & 3u);
      uint32_t* dw = reinterpret_cast<uint32_t*>(pg.fixed_out + row * pg.width);
      for (int k = 0; k < pg.width / 4; ++k) dw[k] = __funnelshift_r(al[k], al[k + 1], sh);
    } else if (dict) {
      const int32_t e = pg.idx[row];
      if (e < 0 || e >= dp->num_values) {
        raise_status(st, GFPDB_EINVAL, 600000 + first + static_cast<int32_t>(blockIdx.y));
        pg.row_ptr[row] = 0;
        pg.row_len[row] = 0;
        continue;
      }
      pg.row_ptr[row] = dicts.ptr[dp->dict_base + e];
      pg.row_len[row] = dicts.len[dp->dict_base + e];
    }
  }
}

__global__ void parquet_bytes_kernel(const uint64_t* __restrict__ ptr, const int32_t* __restrict__ offs, int64_t n,
                                     uint8_t* __restrict__ out) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n; r += stride) {
    const uint8_t* src = reinterpret_cast<const uint8_t*>(ptr[r]);
    const int32_t o = offs[r], len = offs[r + 1] - o;
    for (int32_t k = 0; k < len; ++k) out[o + k] = src[k];
  }
}

constexpr int64_t kPqCopyGap = 64 * 1024;

// A read's chunks are copied and decoded in batches of about kPqBatch bytes:
// while one batch is decoded on the caller's stream the next ones are copied
// on a stream of the read's own. Reads of a single batch use the caller's
// stream alone. (72.6 MB, 4M rows: 558 us of copying and then decoding as one
// batch, 496 us in batches.)
constexpr int64_t kPqBatch = 8 << 20;
// Steps that a batch's walk over a page's runs may take: runs of one length are
// done before (a 1M-value page of 504-value runs takes 66).
constexpr int32_t kPqWalkSteps = 256;

// Byte arrays of a page that are walked with their batch, about 0.3 us each. The
// walks of longer pages, which the batches behind would wait for in turn, go on
// together in the second round: 2M rows of three columns with utf8 dictionaries
// of 5,000 entries (five batches) take 1.9 ms, plain utf8 pages 36 (5.8 and 141
// walked with each batch; 1.8 and 36 without batches).
constexpr int32_t kPqEarlyLengths = 128;

// Compressed pages an SM that are waited for before they are inflated. A warp
// takes one page, from beginning to end, and each launch is as long as its
// longest page: 33 MB of four columns in five batches took 322 ms, inflated
// batch by batch, and takes 82 (82 without batches).
constexpr int kPqInflatePerSm = 16;

// Whether the file's bytes show that all of a page's indices lie in one run: its
// parts then need no walk (a batch would wait about 8 us for it; a look at each
// page of a file of small ones takes as long). Levels and compressed pages are
// not looked into.
bool one_run(const uint8_t* file, const parquet::PageInfo& pg) {
  if (pg.codec != parquet::CODEC_UNCOMPRESSED || pg.v1_def_levels) return false;
  const int64_t skip = pg.type == parquet::PAGE_DATA_V2 ? pg.v2_levels : 0;
  uint64_t h = 0;
  for (int k = 0; k < 5 && skip + 1 + k < pg.compressed; ++k) {
    const uint8_t b = file[pg.data_offset + skip + 1 + k];
    h |= static_cast<uint64_t>(b & 0x7f) << (7 * k);
    if ((b & 0x80) == 0) return static_cast<int64_t>(h & 1 ? (h >> 1) * 8 : h >> 1) >= pg.num_values;
  }
  return false;
}

// The copies' stream, two batches ahead of the decoding; nothing it started is
// left running when it goes.
struct CopyStream {
  cudaStream_t s = nullptr;
  cudaEvent_t ev[2] = {nullptr, nullptr};  // behind the copies of the even and of the odd batches
  ~CopyStream() {
    if (s != nullptr) {
      (void)cudaStreamSynchronize(s);
      (void)cudaStreamDestroy(s);
    }
    for (cudaEvent_t e : ev)
      if (e != nullptr) (void)cudaEventDestroy(e);
  }
  void open(cudaStream_t after) {
    GF_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    for (cudaEvent_t& e : ev) GF_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    GF_CUDA(cudaEventRecord(ev[0], after));
    GF_CUDA(cudaStreamWaitEvent(s, ev[0], 0));
  }
  void copied(size_t batch) { GF_CUDA(cudaEventRecord(ev[batch & 1], s)); }
  void await(size_t batch, cudaStream_t by) { GF_CUDA(cudaStreamWaitEvent(by, ev[batch & 1], 0)); }
};

int grid_parquet(int64_t n) {
  int64_t b = (n + 255) / 256;
  const int64_t cap = static_cast<int64_t>(num_sms()) * 8;
  if (b > cap) b = cap;
  return static_cast<int>(b < 1 ? 1 : b);
}

}  // namespace

TupleSetPtr parquet_read(const uint8_t* file, int64_t size, const std::vector<std::string>& names, int64_t start_pos,
                         int64_t end_pos, cudaStream_t s) {
  const parquet::Layout L = parquet::read_layout(file, size, names, start_pos, end_pos);
  const int64_t rows = L.num_rows;
  if (rows > INT32_MAX) fail(GFPDB_EUNSUPPORTED, "a Parquet read of more than 2^31 - 1 rows");
  const int nc = static_cast<int>(L.columns.size());

  // the column chunks' bytes on the device, in batches; within one, chunks
  // that follow each other in the file with at most kPqCopyGap bytes between
  // them share one copy (a copy costs about 3 us besides its bytes)
  struct Span {
    int64_t begin, end, at;  // file bytes [begin, end) at byte `at` of the arena
  };
  struct Batch {
    size_t chunk_end, span_end;              // its last chunk and span, plus one
    size_t item_end = 0, walk_end = 0, snappy_end = 0, data_end = 0;  // the same in the lists below
    int64_t bytes = 0;
  };
  std::vector<Span> spans;
  std::vector<Batch> batches;
  std::vector<int64_t> chunk_at(L.chunks.size());
  int64_t arena_bytes = 0;
  for (size_t c = 0; c < L.chunks.size(); ++c) {
    const auto& ch = L.chunks[c];
    const bool fresh = batches.empty() || batches.back().bytes >= kPqBatch;
    if (fresh) batches.push_back(Batch{c, spans.size()});
    Batch& b = batches.back();
    if (!fresh && ch.begin >= spans.back().end && ch.begin - spans.back().end <= kPqCopyGap)
      spans.back().end = ch.end;
    else
      spans.push_back(Span{ch.begin, ch.end, arena_bytes});
    chunk_at[c] = spans.back().at + (ch.begin - spans.back().begin);
    arena_bytes = (chunk_at[c] + (ch.end - ch.begin) + 15) / 16 * 16;
    b.bytes += ch.end - ch.begin;
    b.chunk_end = c + 1;
    b.span_end = spans.size();
  }
  auto arena = make_buffer(arena_bytes + 16, s);  // tail padding: 4-byte word reads past a value's end
  CopyStream copies;
  if (batches.size() > 1) copies.open(s);
  auto copy_batch = [&](size_t b) {
    if (b >= batches.size()) return;
    for (size_t k = b > 0 ? batches[b - 1].span_end : 0; k < batches[b].span_end; ++k)
      copy_h2d(arena->as<uint8_t>() + spans[k].at, file + spans[k].begin, spans[k].end - spans[k].begin,
               copies.s != nullptr ? copies.s : s);
    if (copies.s != nullptr) copies.copied(b);
  };
  // the first copies run while the host lays the pages out; the others come
  // after the page descriptors, which would wait behind them
  copy_batch(0);
  copy_batch(1);

  // per-column outputs and working arrays
  std::vector<BufferPtr> fixed(nc), row_ptr(nc), row_len(nc), idx(nc);
  std::vector<bool> has_dict(nc, false);
  for (const auto& pg : L.pages)
    if (pg.type != parquet::PAGE_DICTIONARY && pg.encoding != parquet::ENC_PLAIN) has_dict[pg.column] = true;
  for (int c = 0; c < nc; ++c) {
    const DType t = L.columns[c].dtype;
    if (t == DType::Utf8) {
      row_ptr[c] = make_buffer((rows > 0 ? rows : 1) * 8, s);
      row_len[c] = make_buffer((rows > 0 ? rows : 1) * 4, s);
    } else {
      fixed[c] = make_buffer((rows > 0 ? rows : 1) * dtype_width(t), s);
    }
    if (has_dict[c] && t == DType::Utf8) idx[c] = make_buffer((rows > 0 ? rows : 1) * 4, s);
  }

  // page descriptors
  std::vector<PageDev> pd(L.pages.size());
  std::vector<int32_t> snappy_list, data_list, walk_list;
  std::vector<PagePart> item_list;
  int64_t inflate_bytes = 0, dict_entries = 0;
  std::vector<int64_t> inflate_at(L.pages.size(), -1);
  bool second_round = false;
  int32_t looked_at = -1;  // a chunk
  bool walk = false;
  size_t batch = 0;  // pages come in the order of their chunks
  auto end_batch = [&] {
    batches[batch].item_end = item_list.size();
    batches[batch].walk_end = walk_list.size();
    batches[batch].snappy_end = snappy_list.size();
    batches[batch].data_end = data_list.size();
    ++batch;
  };
  for (size_t p = 0; p < L.pages.size(); ++p) {
    const auto& pg = L.pages[p];
    while (static_cast<size_t>(pg.chunk) >= batches[batch].chunk_end) end_batch();
    const bool v2 = pg.type == parquet::PAGE_DATA_V2;
    const bool snappy = pg.codec == parquet::CODEC_SNAPPY && !(v2 && !pg.v2_compressed);
    if (snappy) {
      inflate_at[p] = inflate_bytes;
      inflate_bytes += (static_cast<int64_t>(pg.uncompressed) - (v2 ? pg.v2_levels : 0) + 15) / 16 * 16;
      snappy_list.push_back(static_cast<int32_t>(p));
    } else if ((v2 ? pg.compressed - pg.v2_levels : pg.compressed) !=
               (v2 ? pg.uncompressed - pg.v2_levels : pg.uncompressed)) {
      fail(GFPDB_EINVAL, "Parquet uncompressed page sizes disagree");
    }
    // data pages the values pass reads: plain pages, and dictionary-encoded
    // byte-array pages (a fixed-width column's dictionary indices become
    // values in the page pass)
    const bool fixed_dict = L.columns[pg.column].dtype != DType::Utf8 && pg.encoding != parquet::ENC_PLAIN;
    if (pg.type != parquet::PAGE_DICTIONARY && !fixed_dict) data_list.push_back(static_cast<int32_t>(p));
    const bool indices = pg.type != parquet::PAGE_DICTIONARY && pg.encoding != parquet::ENC_PLAIN;
    // byte-array pages whose lengths a thread walks
    const bool lengths = L.columns[pg.column].dtype == DType::Utf8 && !indices;
    const bool late = lengths && batches.size() > 1 && pg.num_values > kPqEarlyLengths;
    pd[p].late_from = late ? 0 : kPqNever;
    second_round |= late;
    pd[p].first_part = static_cast<int32_t>(item_list.size());
    for (int64_t first = 0; first == 0 || (indices && first < pg.num_values); first += kPqPart)
      item_list.push_back(PagePart{static_cast<int32_t>(p), static_cast<int32_t>(first), 1, 0});
    if (item_list.size() > INT32_MAX) fail(GFPDB_EUNSUPPORTED, "a Parquet read of too many pages");
    pd[p].n_parts = static_cast<int32_t>(item_list.size()) - pd[p].first_part;
    if (pd[p].n_parts > 1) {  // a chunk's pages are walked or not by its first one
      if (pg.chunk != looked_at) {
        looked_at = pg.chunk;
        walk = !one_run(file, pg);
      }
      if (walk) {
        pd[p].walked = 1;
        walk_list.push_back(static_cast<int32_t>(p));
      }
    }
  }
  while (batch < batches.size()) end_batch();
  auto inflated = make_buffer(inflate_bytes + 16, s);
  for (size_t p = 0; p < L.pages.size(); ++p) {
    const auto& pg = L.pages[p];
    const int c = pg.column;
    const bool v2 = pg.type == parquet::PAGE_DATA_V2;
    PageDev& d = pd[p];
    d.body = arena->as<uint8_t>() + chunk_at[pg.chunk] + (pg.data_offset - L.chunks[pg.chunk].begin);
    d.body_len = pg.compressed;
    d.snappy = inflate_at[p] >= 0 ? 1 : 0;
    d.inflated = d.snappy ? inflated->as<uint8_t>() + inflate_at[p] : nullptr;
    d.inflated_len = d.snappy ? pg.uncompressed - (v2 ? pg.v2_levels : 0) : 0;
    d.type = pg.type;
    d.encoding = pg.encoding;
    d.num_values = pg.num_values;
    d.v2_levels = pg.v2_levels;
    d.v1_def = pg.v1_def_levels ? 1 : 0;
    d.width = L.columns[c].dtype == DType::Utf8 ? 0 : dtype_width(L.columns[c].dtype);
    d.dict_page = pg.dict_page;
    d.first_row = pg.first_row;
    if (pg.type == parquet::PAGE_DICTIONARY && d.width == 0) {
      d.dict_base = dict_entries;
      dict_entries += pg.num_values;
    }
    d.idx = idx[c] ? idx[c]->as<int32_t>() : nullptr;
    d.row_ptr = row_ptr[c] ? row_ptr[c]->as<uint64_t>() : nullptr;
    d.row_len = row_len[c] ? row_len[c]->as<int32_t>() : nullptr;
    d.fixed_out = fixed[c] ? fixed[c]->as<uint8_t>() : nullptr;
  }
  DictArrays dicts{};
  BufferPtr dict_ptr, dict_len;
  if (dict_entries > 0) {
    dict_ptr = make_buffer(dict_entries * 8, s);
    dict_len = make_buffer(dict_entries * 4, s);
    dicts.ptr = dict_ptr->as<uint64_t>();
    dicts.len = dict_len->as<int32_t>();
  }
  auto status = make_filled(sizeof(DevStatus), 0, s);
  DevStatus* st = status->as<DevStatus>();
  const int64_t np = static_cast<int64_t>(pd.size());
  auto pages_dev = make_buffer((np > 0 ? np : 1) * static_cast<int64_t>(sizeof(PageDev)), s);
  // the parts, then the lists of pages to walk, to inflate and to copy values of
  const size_t item_bytes = item_list.size() * sizeof(PagePart);
  std::vector<char> lists_host(item_bytes + (walk_list.size() + snappy_list.size() + data_list.size()) * 4);
  {
    char* to = lists_host.data();
    auto append = [&](const void* from, size_t bytes) {
      if (bytes > 0) std::memcpy(to, from, bytes);
      to += bytes;
    };
    append(item_list.data(), item_bytes);
    append(walk_list.data(), walk_list.size() * 4);
    append(snappy_list.data(), snappy_list.size() * 4);
    append(data_list.data(), data_list.size() * 4);
  }
  auto lists = make_buffer(static_cast<int64_t>(lists_host.size()) + 16, s);
  PagePart* items = lists->as<PagePart>();
  int32_t* walk_dev = reinterpret_cast<int32_t*>(lists->as<char>() + item_bytes);
  if (np > 0) GF_CUDA(cudaMemcpyAsync(pages_dev->data(), pd.data(), np * sizeof(PageDev), cudaMemcpyHostToDevice, s));
  if (!lists_host.empty())
    GF_CUDA(cudaMemcpyAsync(items, lists_host.data(), lists_host.size(), cudaMemcpyHostToDevice, s));
  PageDev* pages = pages_dev->as<PageDev>();
  const int32_t* snappy_dev = walk_dev + walk_list.size();
  const int32_t* data_dev = snappy_dev + snappy_list.size();

  // the walks, parts and values of the pages of batches (from, to]
  auto decode = [&](const Batch& from, const Batch& to, bool late) {
    if (to.walk_end > from.walk_end) {
      const int64_t n = static_cast<int64_t>(to.walk_end - from.walk_end), most = static_cast<int64_t>(num_sms()) * 16;
      ProfScope prof("parquet_runs_kernel", s);
      parquet_runs_kernel<<<static_cast<int>(std::min((n + 3) / 4, most)), 128, 0, s>>>(
          pages, walk_dev + from.walk_end, static_cast<int32_t>(n), items, late ? -1 : kPqWalkSteps, late ? 1 : 0, st);
      after_launch("parquet_runs_kernel");
      prof.stop(0.0);
    }
    if (to.item_end > from.item_end) {
      ProfScope prof("parquet_pages_kernel", s);
      const int64_t n = static_cast<int64_t>(to.item_end - from.item_end), most = static_cast<int64_t>(num_sms()) * 8;
      parquet_pages_kernel<<<static_cast<int>(std::min(n, most)), kPqThreads, 0, s>>>(
          pages, static_cast<int32_t>(np), items + from.item_end, n, late ? 1 : 0, dicts, st);
      after_launch("parquet_pages_kernel");
      prof.stop(0.0);
    }
    // each data page's values over up to 64 blocks of 256 threads
    int64_t most = 0;
    for (size_t k = from.data_end; k < to.data_end; ++k) most = std::max<int64_t>(most, L.pages[data_list[k]].num_values);
    const int gx = static_cast<int>(std::min<int64_t>(64, std::max<int64_t>(1, (most + 255) / 256)));
    for (size_t at = from.data_end; at < to.data_end; at += 65535) {  // grid y limit
      const int gy = static_cast<int>(std::min<size_t>(65535, to.data_end - at));
      ProfScope prof("parquet_values_kernel", s);
      parquet_values_kernel<<<dim3(gx, gy), 256, 0, s>>>(pages, data_dev + at, static_cast<int32_t>(at), late ? 1 : 0,
                                                         dicts, st);
      after_launch("parquet_values_kernel");
      prof.stop(0.0);
    }
  };
  Batch from{};
  for (size_t b = 0; b < batches.size(); ++b) {
    const Batch& to = batches[b];
    if (copies.s != nullptr) copies.await(b, s);
    const size_t compressed = to.snappy_end - from.snappy_end;
    if (compressed > 0 && compressed < static_cast<size_t>(num_sms()) * kPqInflatePerSm && b + 1 < batches.size()) {
      copy_batch(b + 2);
      continue;  // decoded with the next one
    }
    if (to.snappy_end > from.snappy_end) {
      const int64_t n = static_cast<int64_t>(to.snappy_end - from.snappy_end);
      ProfScope prof("parquet_snappy_kernel", s);
      parquet_snappy_kernel<<<grid_parquet(n * 32), 256, 0, s>>>(pages, snappy_dev + from.snappy_end,
                                                                 static_cast<int32_t>(n), st);
      after_launch("parquet_snappy_kernel");
      double bytes = 0;
      for (size_t k = from.snappy_end; k < to.snappy_end; ++k) bytes += pd[snappy_list[k]].inflated_len;
      prof.stop(bytes);
    }
    decode(from, to, false);
    copy_batch(b + 2);
    from = to;
  }
  if (second_round) decode(Batch{}, batches.back(), true);
  DevStatus h;
  GF_CUDA(cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, s));
  sync(s);
  if (h.code == 0 && h.aux[0] != 0 && !second_round) {  // a batch's walks were cut short
    decode(Batch{}, batches.back(), true);
    GF_CUDA(cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, s));
    sync(s);
  }
  if (h.code != 0)
    fail(h.code, std::string(h.code == GFPDB_EUNSUPPORTED ? "Parquet column with nulls (definition levels)"
                                                         : "malformed Parquet page data") +
                     " (page " + std::to_string(h.detail % 100000) + ")");

  std::vector<Field> fields;
  std::vector<ColumnPtr> cols;
  for (int c = 0; c < nc; ++c) {
    const DType t = L.columns[c].dtype;
    fields.push_back(Field{L.columns[c].name, t});
    if (t != DType::Utf8) {
      cols.push_back(make_fixed_column(t, rows, fixed[c]));
      continue;
    }
    auto offs = make_buffer((rows + 1) * 4, s);
    const int64_t total = rows > 0 ? exclusive_scan_i32(row_len[c]->as<int32_t>(), offs->as<int32_t>(), rows, s) : 0;
    if (rows == 0) GF_CUDA(cudaMemsetAsync(offs->data(), 0, 4, s));
    auto bytes = make_buffer(total > 0 ? total : 1, s);
    if (total > 0) {
      ProfScope prof("parquet_bytes_kernel", s);
      parquet_bytes_kernel<<<grid_parquet(rows), 256, 0, s>>>(row_ptr[c]->as<uint64_t>(), offs->as<int32_t>(), rows,
                                                              bytes->as<uint8_t>());
      after_launch("parquet_bytes_kernel");
      prof.stop(2.0 * static_cast<double>(total));
    }
    cols.push_back(make_utf8_column(rows, offs, bytes));
  }
  sync(s);  // the page descriptors (host vector) and the arena are released on return
  return TupleSet::make(std::move(fields), std::move(cols), rows);
}

}  // namespace gfpdb
