// Delimited-text ingest into typed device columns.
//
// Replaces CSVReader::read and the reference's SIMD CSV path
// (fpdb-tuple/src/csv/CSVReader.cpp:15-103; find_indexes at
// fpdb-tuple/src/arrow/SIMDParserHelpers.cpp:13-201; per-field std::stoi /
// std::stol / date parsing and ArrayBuilder appends at
// fpdb-tuple/src/arrow/CSVToArrowSIMDChunkParser.cpp:183-313). Parsing rules:
// fields split on the delimiter, rows on '\n' (a trailing '\r' is dropped),
// an optional header line is skipped, and a field wrapped in double quotes
// has the quotes removed (the reference strips surrounding quotes through
// startEndOffsets_, CSVToArrowSIMDChunkParser.cpp:371-373).
//
// Types: int32 / int64 (optional sign, decimal digits), decimal(p, s) text
// into int64 scaled by 10^s with exact integer arithmetic (the reference reads
// decimals as double; here they are exact cents), date32 from YYYY-MM-DD
// (days since 1970-01-01 by Howard Hinnant's public-domain days_from_civil
// algorithm), and utf8 (bytes copied as they are).
//
// Kernels: the text is cut into 32 KiB tiles. A separator is a delimiter or a
// newline; in a well-formed text every row has n_fields separators, so the
// field that ends at the g-th separator of the text is row g / n_fields,
// field g % n_fields.
// (1) csv_index_kernel: each 16 bytes' separator bits (kept for the next
// pass), per tile the separator count and the position of its last separator;
// (2) csv_fields_kernel: every tile's numeric fields converted, per utf8
// field where it lies in its tile, and per utf8 column and tile the bytes (a
// newline at any position but the last field of a row marks the row
// malformed); (3) csv_strings_kernel: every tile's utf8 offsets and bytes,
// all columns in one pass over the text. Separator counts and byte counts are
// also added up per bucket of tiles, so a block finds how many come before
// its tile from the buckets before it and the tiles of its own bucket, while
// its text is on the way: no scan pass stands between the others.
//
// 2M lineitem rows (482 MB of text, 16 columns, 6 of them utf8) take 85 +
// 310 + 280 us. With the fields converted byte by byte, a prefix sum per utf8
// column and a copy kernel per utf8 column that went to the text again, the
// same rows took 1,260 us of kernels (110 index, 49 scan, 470 fields, 150
// prefix sums, 465 copies). Tiles of 32 KiB at five blocks an SM measured
// faster than 16 KiB ones (1,109 against 1,140 us the call): a column's rows
// of a tile fill more of its last warp step, and per-tile work halves.
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "launch.h"

namespace gfpdb {

namespace {

constexpr int kCsvThreads = 256;
constexpr int kCsvChunk = 128;                              // bytes per thread
constexpr int kCsvTile = kCsvThreads * kCsvChunk;           // bytes per tile

// The sum of v over the tiles before `tile`, from the sums of whole buckets
// of 1 << shift tiles and the tiles of its own bucket. The warp works together.
template <typename T>
__device__ __forceinline__ int64_t sum_before(const unsigned long long* __restrict__ buckets, const T* __restrict__ v,
                                              int64_t tile, int shift) {
  const int lane = threadIdx.x & 31;
  const int64_t bucket = tile >> shift;
  int64_t sum = 0;
#pragma unroll 4
  for (int64_t i = lane; i < bucket; i += 32) sum += static_cast<int64_t>(buckets[i]);
#pragma unroll 4
  for (int64_t i = (bucket << shift) + lane; i < tile; i += 32) sum += v[i];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
  return sum;
}

// Bytes [at, at + 16) of the text (zeros past its end); at is a multiple of 16.
__device__ __forceinline__ uint4 load16(const uint8_t* text, int64_t n, int64_t at) {
  if (at + 16 <= n) return __ldg(reinterpret_cast<const uint4*>(text + at));
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    w[k] = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b)
      if (at + 4 * k + b < n) w[k] |= static_cast<uint32_t>(text[at + 4 * k + b]) << (8 * b);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// 0x80 in every byte of w that is a separator (equal to the pattern's byte
// or a newline), 0 elsewhere: a byte x is zero where ((x & 0x7F) + 0x7F) | x
// has its high bit clear (exact: no carry crosses a byte).
__device__ __forceinline__ uint32_t separator_bytes(uint32_t w, uint32_t dpat) {
  const uint32_t a = w ^ dpat, b = w ^ 0x0A0A0A0Au;
  const uint32_t ta = ((a & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | a;
  const uint32_t tb = ((b & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | b;
  return ~((ta & tb) | 0x7F7F7F7Fu);
}

// Bit i set when byte i of the 16 is a separator. The 0x80 bytes gather by
// dot products with the bits' weights, two words to a byte (times 128).
__device__ __forceinline__ uint32_t separator_bits16(const uint4& v, uint32_t dpat) {
  uint32_t lo = __dp4a(separator_bytes(v.x, dpat), 0x08040201u, 0u);
  lo = __dp4a(separator_bytes(v.y, dpat), 0x80402010u, lo);
  uint32_t hi = __dp4a(separator_bytes(v.z, dpat), 0x08040201u, 0u);
  hi = __dp4a(separator_bytes(v.w, dpat), 0x80402010u, hi);
  return (lo >> 7) | (hi << 1);
}

// (1) per tile: separators, and the position of the last one (-1: none).
// Bound by the text's stream: each warp reads 4 KiB in eight coalesced 16-byte
// loads per lane, all in flight together.
__global__ void __launch_bounds__(kCsvThreads, 6)
    csv_index_kernel(const uint8_t* __restrict__ text, int64_t n, uint8_t delim, int32_t* __restrict__ tile_count,
                     int64_t* __restrict__ tile_last, uint16_t* __restrict__ masks,
                     unsigned long long* __restrict__ buckets, int shift, unsigned long long* __restrict__ last_byte) {
  constexpr int kPieces = kCsvTile / 16;          // 16-byte pieces of a tile
  constexpr int kEach = kPieces / kCsvThreads;    // pieces of a thread
  __shared__ int s_cnt[kCsvThreads / 32], s_last[kCsvThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tile0 = static_cast<int64_t>(blockIdx.x) * kCsvTile;
  const int piece0 = warp * (kPieces / (kCsvThreads / 32)) + lane;
  const uint32_t dpat = static_cast<uint32_t>(delim) * 0x01010101u;
  uint16_t* const out = masks + static_cast<int64_t>(blockIdx.x) * kPieces + piece0;
  const bool whole = tile0 + kCsvTile <= n;
  uint4 v[kEach];
#pragma unroll
  for (int k = 0; k < kEach; ++k)
    v[k] = whole ? __ldg(reinterpret_cast<const uint4*>(text + tile0) + piece0 + 32 * k)
                 : load16(text, n, tile0 + (piece0 + 32 * k) * 16);
  int cnt = 0, last = -1;
#pragma unroll
  for (int k = 0; k < kEach; ++k) {
    const int at = (piece0 + 32 * k) * 16;
    uint32_t m = separator_bits16(v[k], dpat);
    if (!whole && tile0 + at + 16 > n) m &= n > tile0 + at ? (1u << (n - tile0 - at)) - 1u : 0u;  // bytes past the end
    out[32 * k] = static_cast<uint16_t>(m);
    cnt += __popc(m);
    if (m != 0) last = at + 31 - __clz(static_cast<int>(m));
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  last = __reduce_max_sync(0xffffffffu, last);
  if (lane == 0) {
    s_cnt[warp] = cnt;
    s_last[warp] = last;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kCsvThreads / 32; ++w) {
      cnt += s_cnt[w];
      last = s_last[w] > last ? s_last[w] : last;
    }
    tile_count[blockIdx.x] = cnt;
    tile_last[blockIdx.x] = last >= 0 ? tile0 + last : -1;
    atomicAdd(buckets + (blockIdx.x >> shift), static_cast<unsigned long long>(cnt));
    if (blockIdx.x == gridDim.x - 1) *last_byte = text[n - 1];
  }
}

__device__ __forceinline__ int32_t days_from_civil(int32_t y, uint32_t m, uint32_t d) {
  y -= m <= 2;
  const int32_t era = (y >= 0 ? y : y - 399) / 400;
  const uint32_t yoe = static_cast<uint32_t>(y - era * 400);
  const uint32_t doy = (153 * (m + (m > 2 ? -3 : 9)) + 2) / 5 + d - 1;
  const uint32_t doe = yoe * 365 + yoe / 4 - yoe / 100 + doy;
  return era * 146097 + static_cast<int32_t>(doe) - 719468;
}

struct CsvOut {
  void* data;         // fixed-width output; utf8: the bytes
  int32_t* offs;      // utf8: the offsets
  int32_t type;       // ColTypeCode
  int32_t decimal;    // 1: decimal text -> scaled int64
  int32_t scale;
  int32_t pow10;      // 10^scale
  int32_t field;      // the line's field
  int32_t utf8;       // which utf8 column this is (-1: fixed width)
};

constexpr int kCsvMaxOut = 32;
constexpr int kCsvMaxFields = 256;

struct CsvParams {
  const uint8_t* text;
  int64_t n;                   // text bytes
  int64_t n_tiles;
  int32_t bucket_shift;        // log2 of the tiles in a bucket
  int32_t pad;
  int64_t n_buckets;
  const unsigned long long* sep_buckets;  // separators of each bucket of tiles
  const int32_t* tile_count;   // separators of each tile
  const int64_t* tile_last;    // position of each tile's last separator (-1: none)
  int64_t* tile_row;           // row (the header counts) << 8 | field of each tile's first separator
  const uint64_t* chunk_masks; // separator bits (csv_index_kernel)
  unsigned long long* byte_buckets;  // [utf8 column][bucket] bytes of its tiles' fields
  int64_t* tile_bytes;         // [utf8 column][tile] bytes of the tile's fields
  uint32_t* spans;             // [utf8 column][data row] the field in its tile: length << 16 | first byte (kCsvFar)
  int64_t* far;                // per tile, its kCsvFar field: first text byte, length
  int64_t n_rows;              // data rows (after the header)
  uint32_t inv_fields;         // ceil(2^32 / n_fields), 0 for one field
  int32_t n_fields;
  int32_t n_out;
  int32_t n_utf8;
  int32_t header;              // 1: the first row is skipped
  int32_t virtual_end;         // 1: the text does not end with '\n' (a newline is implied at n)
  DevStatus* st;
  int32_t utf8_out[kCsvMaxOut];  // output of each utf8 column
  CsvOut out[kCsvMaxOut];
};

__device__ __forceinline__ bool parse_int(const uint8_t* t, int64_t b, int64_t e, int64_t* v) {
  if (b >= e) return false;
  bool neg = false;
  if (t[b] == '-' || t[b] == '+') {
    neg = t[b] == '-';
    ++b;
  }
  if (b >= e) return false;
  uint64_t acc = 0;
  for (int64_t i = b; i < e; ++i) {
    const uint32_t d = static_cast<uint32_t>(t[i]) - '0';
    if (d > 9) return false;
    acc = acc * 10 + d;
  }
  *v = neg ? static_cast<int64_t>(0ull - acc) : static_cast<int64_t>(acc);
  return true;
}

__device__ __forceinline__ bool parse_decimal(const uint8_t* t, int64_t b, int64_t e, int scale, int64_t* v) {
  if (b >= e) return false;
  bool neg = false;
  if (t[b] == '-' || t[b] == '+') {
    neg = t[b] == '-';
    ++b;
  }
  uint64_t acc = 0;
  int frac = -1;  // digits seen after the point, -1 before it
  bool any = false;
  for (int64_t i = b; i < e; ++i) {
    const uint8_t c = t[i];
    if (c == '.') {
      if (frac >= 0) return false;
      frac = 0;
      continue;
    }
    const uint32_t d = static_cast<uint32_t>(c) - '0';
    if (d > 9) return false;
    if (frac >= 0) {
      if (frac == scale) return false;  // more fractional digits than the scale holds
      ++frac;
    }
    acc = acc * 10 + d;
    any = true;
  }
  if (!any) return false;
  for (int k = frac < 0 ? 0 : frac; k < scale; ++k) acc *= 10;
  *v = neg ? static_cast<int64_t>(0ull - acc) : static_cast<int64_t>(acc);
  return true;
}

__device__ __forceinline__ bool parse_date(const uint8_t* t, int64_t b, int64_t e, int32_t* v) {
  if (e - b != 10 || t[b + 4] != '-' || t[b + 7] != '-') return false;
  int32_t y = 0;
  uint32_t m = 0, d = 0;
  for (int i = 0; i < 4; ++i) {
    const uint32_t x = static_cast<uint32_t>(t[b + i]) - '0';
    if (x > 9) return false;
    y = y * 10 + static_cast<int32_t>(x);
  }
  for (int i = 5; i < 7; ++i) {
    const uint32_t x = static_cast<uint32_t>(t[b + i]) - '0';
    if (x > 9) return false;
    m = m * 10 + x;
  }
  for (int i = 8; i < 10; ++i) {
    const uint32_t x = static_cast<uint32_t>(t[b + i]) - '0';
    if (x > 9) return false;
    d = d * 10 + x;
  }
  if (m < 1 || m > 12 || d < 1 || d > 31) return false;
  *v = days_from_civil(y, m, d);
  return true;
}

__device__ __forceinline__ void csv_malformed(DevStatus* st, int64_t row) {
  raise_status(st, GFPDB_EINVAL, static_cast<int32_t>(row < 0 ? 0 : (row < INT32_MAX ? row : INT32_MAX)));
}

// A tile's text and separators in shared memory.
//
// The text holds the kCsvFront bytes before the tile too, so that the tile's
// first field is read from shared memory unless it starts further back (a
// "far" field). The separators' positions are stored by (field, row) so that
// consecutive lanes take one field of consecutive rows. A tile with more than
// kCsvSepCap separators (fields of under 8 bytes on average) is worked off in
// as many equal parts as keep each within it.
constexpr int kCsvFront = 256;
constexpr int kCsvTextLines = (kCsvFront + kCsvTile + 32) / 16;  // 16-byte lines of a tile's text
constexpr int kCsvSepCap = 4096;
constexpr int kCsvWarps = kCsvThreads / 32;
constexpr int kCsvParts = 16;  // most parts of a tile: each of 2,048 bytes
constexpr uint32_t kCsvFar = 0xFFFFu;  // first byte of a span that starts before the tile's text

// The separators of one part of a tile, on rows row0 (the header counts) to
// row0 + rows - 1: the first is field c0 of row0, the last field c1 of the
// last row. Field c of row0 + r ends at pos[(c + 1) * rs + r] and starts one
// past pos[c * rs + r] (row 0 of pos repeats field n_fields - 1 one row on),
// unless it is the part's first and far. Data rows are r in [lo, hi).
struct CsvPart {
  int64_t row0;
  int32_t c0, c1, rows, lo, hi, far;
};

struct CsvTileShared {
  uint4 text[kCsvTextLines];                     // byte i: text byte tile0 - kCsvFront + i
  int32_t warp_cnt[kCsvWarps];
  int32_t bound[kCsvParts + 1];                  // separators before each kCsvParts-th of the tile, and in all of it
  int32_t c0;                                    // field of the tile's first separator
  int64_t q0;                                    //   and its row (the header counts)
  int64_t prev;                                  // the separator before the part, as a byte of `text` (may lie before it)
  CsvPart part;
  uint16_t pos[1];                               // separators, as bytes of `text`: csv_pos_slots() of them
};

// pos holds fields + 1 rows of kCsvSepCap / fields + 3.
constexpr int csv_pos_slots(int fields) { return (fields + 1) * (kCsvSepCap / fields + 3); }
constexpr int csv_fields_smem(int fields) {
  return static_cast<int>(sizeof(CsvTileShared)) + 2 * csv_pos_slots(fields);
}

__device__ __forceinline__ unsigned div_fields(const CsvParams& p, unsigned j) {
  return p.inv_fields == 0 ? j : __umulhi(j, p.inv_fields);  // exact for j * n_fields < 2^32
}

// The 32 KiB tile and the kCsvFront bytes before it into `text`, without a barrier.
__device__ __forceinline__ void stage_tile(const CsvParams& p, uint4* text) {
  constexpr int kEach = kCsvTile / 16 / kCsvThreads;
  const int64_t tile0 = static_cast<int64_t>(blockIdx.x) * kCsvTile;
  uint4 v[kEach];
  if (tile0 + kCsvTile <= p.n) {
    const uint4* src = reinterpret_cast<const uint4*>(p.text + tile0) + threadIdx.x;
#pragma unroll
    for (int k = 0; k < kEach; ++k) v[k] = __ldg(src + k * kCsvThreads);
  } else {
#pragma unroll
    for (int k = 0; k < kEach; ++k) v[k] = load16(p.text, p.n, tile0 + (threadIdx.x + k * kCsvThreads) * 16);
  }
  if (threadIdx.x < kCsvFront / 16)
    text[threadIdx.x] = blockIdx.x > 0 ? load16(p.text, p.n, tile0 - kCsvFront + threadIdx.x * 16) : make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int k = 0; k < kEach; ++k) text[kCsvFront / 16 + threadIdx.x + k * kCsvThreads] = v[k];
}

// Reports the first malformed row of a chunk: its separators again, the first
// one field c of `row`.
__device__ __noinline__ void malformed_row(const CsvParams& p, const uint8_t* chunk, uint4 mask, int bits, int cnt, int c,
                                           int64_t row) {
  const uint32_t m[4] = {mask.x, mask.y, mask.z, mask.w};
  for (int k = 0, b = 0; k < cnt; ++k, ++b) {
    bool is_nl = true;
    if (k < bits) {
      while ((m[b >> 5] >> (b & 31) & 1u) == 0) ++b;
      is_nl = chunk[b] == '\n';
    }
    if (is_nl != (c == p.n_fields - 1)) {
      csv_malformed(p.st, row);
      return;
    }
    if (++c == p.n_fields) {
      c = 0;
      ++row;
    }
  }
}

// Stages the block's tile and calls visit(part) for each of its parts, every
// thread with the same part, between block barriers.
template <class Visit>
__device__ __forceinline__ void walk_tile(const CsvParams& p, CsvTileShared& sh, Visit&& visit) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tile0 = static_cast<int64_t>(blockIdx.x) * kCsvTile;
  const int64_t at = tile0 + static_cast<int64_t>(threadIdx.x) * kCsvChunk;
  const int F = p.n_fields;
  const uint4 mask = __ldg(reinterpret_cast<const uint4*>(p.chunk_masks) + at / kCsvChunk);
  stage_tile(p, sh.text);
  // the implied newline after an unterminated last line belongs to the chunk
  // holding the last byte
  const bool has_end = p.virtual_end && p.n > at && p.n <= at + kCsvChunk;
  const int bits = __popc(mask.x) + __popc(mask.y) + __popc(mask.z) + __popc(mask.w);
  const int cnt = bits + (has_end ? 1 : 0);
  int incl = cnt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += y;
  }
  if (lane == 31) sh.warp_cnt[warp] = incl;
  if (warp == 0) {
    const int64_t g0 = sum_before(p.sep_buckets, p.tile_count, blockIdx.x, p.bucket_shift);
    if (lane == 0) {
      sh.q0 = g0 / F;
      sh.c0 = static_cast<int>(g0 - sh.q0 * F);
      p.tile_row[blockIdx.x] = sh.q0 << 8 | sh.c0;
    }
  } else if (warp == 1) {  // the last separator before the tile
    int64_t prev = -1;
    for (int64_t t = static_cast<int64_t>(blockIdx.x) - 1; t >= 0; t -= 32) {
      const int64_t x = t - lane >= 0 ? p.tile_last[t - lane] : -1;
      const unsigned found = __ballot_sync(0xffffffffu, x >= 0);
      if (found != 0) {
        prev = __shfl_sync(0xffffffffu, x, __ffs(static_cast<int>(found)) - 1);
        break;
      }
    }
    if (lane == 0) sh.prev = prev - tile0 + kCsvFront;
  }
  __syncthreads();
  int before = incl - cnt, tot = 0;  // separators before this thread's chunk, and in the tile
#pragma unroll
  for (int w = 0; w < kCsvWarps; ++w) {
    const int c = sh.warp_cnt[w];
    if (w < warp) before += c;
    tot += c;
  }
  if (tot == 0) return;  // uniform over the block
  const int rs = kCsvSepCap / F + 3;
  int parts = 1;
  if (tot > kCsvSepCap) {
    constexpr int kShare = kCsvThreads / kCsvParts;
    if (threadIdx.x % kShare == 0) sh.bound[threadIdx.x / kShare] = before;
    if (threadIdx.x == 0) sh.bound[kCsvParts] = tot;
    __syncthreads();
    for (bool fits = false; !fits && parts < kCsvParts;) {
      parts *= 2;
      fits = true;
      for (int i = 0; i < kCsvParts; i += kCsvParts / parts)
        fits = fits && sh.bound[i + kCsvParts / parts] - sh.bound[i] <= kCsvSepCap;
    }
  }
  const uint8_t* text = reinterpret_cast<const uint8_t*>(sh.text);
  for (int part = 0; part < parts; ++part) {
    int begin = 0, end = tot;
    bool mine = true;
    if (parts > 1) {
      begin = sh.bound[part * (kCsvParts / parts)];
      end = sh.bound[(part + 1) * (kCsvParts / parts)];
      mine = static_cast<int>(threadIdx.x) / (kCsvThreads / parts) == part;
      if (begin == end) continue;  // uniform over the block
    }
    // field c0 of the part's first separator, and where this thread's first
    // one lies: field c, r rows on
    const unsigned j0 = static_cast<unsigned>(sh.c0 + begin);
    const unsigned jr = div_fields(p, j0);
    const int c0 = static_cast<int>(j0 - jr * F);
    const unsigned j = static_cast<unsigned>(c0 + before - begin);
    const int r = static_cast<int>(div_fields(p, j));
    const int c = static_cast<int>(j) - r * F;
    if (threadIdx.x == kCsvThreads - 1) {  // the part's description, ready at the barrier
      CsvPart& pt = sh.part;
      const unsigned jl = static_cast<unsigned>(c0 + end - begin - 1);
      const int rl = static_cast<int>(div_fields(p, jl));
      pt.row0 = sh.q0 + jr;
      pt.c0 = c0;
      pt.c1 = static_cast<int>(jl) - rl * F;
      pt.rows = rl + 1;
      pt.far = sh.prev < -1 ? 1 : 0;
      pt.lo = pt.row0 < p.header ? static_cast<int>(p.header - pt.row0) : 0;
      const int64_t data_end = p.n_rows + p.header - pt.row0;
      pt.hi = data_end < pt.rows ? static_cast<int>(data_end > 0 ? data_end : 0) : pt.rows;
      if (!pt.far) sh.pos[c0 * rs] = static_cast<uint16_t>(sh.prev);  // -1: 0xFFFF
    }
    if (mine && cnt > 0) {
      const int i0 = kCsvFront + static_cast<int>(threadIdx.x) * kCsvChunk;
      const uint8_t* chunk = text + i0;
      uint16_t* at_pos = sh.pos + (c + 1) * rs + r;
      const int wrap = F * rs - 1;
      uint32_t m = mask.x;
      uint32_t m1 = mask.y, m2 = mask.z, m3 = mask.w;
      int hi = 0;            // bytes of the chunk behind m
      int left = F - 1 - c;  // fields after this one in its row
      bool bad = false;
      for (int k = 0; k < bits; ++k) {
        while (m == 0) {
          m = m1;
          m1 = m2;
          m2 = m3;
          hi += 32;
        }
        const int b = __ffs(static_cast<int>(m)) - 1 + hi;
        m &= m - 1;
        bad |= (chunk[b] == '\n') != (left == 0);
        *at_pos = static_cast<uint16_t>(i0 + b);
        at_pos += rs;
        if (--left < 0) {
          left = F - 1;
          at_pos -= wrap;
          at_pos[-rs] = static_cast<uint16_t>(i0 + b);
        }
      }
      if (has_end) {  // the implied newline
        *at_pos = static_cast<uint16_t>(p.n - tile0 + kCsvFront);
        bad |= left != 0;
      }
      if (bad) malformed_row(p, chunk, mask, bits, cnt, c, sh.q0 + jr + r - p.header);
    }
    __syncthreads();
    visit(sh.part);
    if (parts > 1) {
      __syncthreads();
      if (threadIdx.x == 0) sh.prev = sh.pos[(sh.part.c1 + 1) * rs + sh.part.rows - 1];
      __syncthreads();  // the next part writes pos and reads prev
    }
  }
}

// Drops a carriage return before the row's newline and surrounding quotes.
template <class I>
__device__ __forceinline__ void trim_field(const uint8_t* t, I& b, I& e, bool row_end) {
  if (row_end && e > b && t[e - 1] == '\r') --e;
  if (e - b >= 2 && t[b] == '"' && t[e - 1] == '"') {
    ++b;
    --e;
  }
}

// 0x80 in some byte when a byte of t (text ^ '0') is not a digit.
__device__ __forceinline__ uint32_t not_digits(uint32_t t) { return ((t + 0x76767676u) | t) & 0x80808080u; }

// Value of four digits, the first in the lowest byte.
__device__ __forceinline__ uint32_t four_digits(uint32_t t) {
  return __dp4a(t, 0x0000010Au, 0u) * 100u + __dp4a(t, 0x010A0000u, 0u);
}

// Bytes [i, i + 4) of the text in shared memory.
__device__ __forceinline__ uint32_t text_word(const uint32_t* s, int i) {
  return __funnelshift_r(s[i >> 2], s[(i >> 2) + 1], 8u * (static_cast<unsigned>(i) & 3u));
}

// Value of the len (0 to 8) digits that end before byte e: the eight bytes
// before e as two words, the bytes that are not the field's masked to zeros.
// *bad gets bits when one is not a digit.
__device__ __forceinline__ uint32_t digits8(const uint32_t* s, int e, int len, uint32_t* bad) {
  const int i = e - 8;
  const uint32_t w0 = s[i >> 2], w1 = s[(i >> 2) + 1], w2 = s[(i >> 2) + 2];
  const unsigned sh = 8u * (static_cast<unsigned>(i) & 3u);
  const uint32_t mlo = len > 4 ? ~0u << (8 * (8 - len)) : 0u;
  const uint32_t mhi = len >= 4 ? ~0u : len > 0 ? ~0u << (8 * (4 - len)) : 0u;
  const uint32_t lo = (__funnelshift_r(w0, w1, sh) ^ 0x30303030u) & mlo;
  const uint32_t hi = (__funnelshift_r(w1, w2, sh) ^ 0x30303030u) & mhi;
  *bad |= not_digits(lo) | not_digits(hi);
  return four_digits(lo) * 10000u + four_digits(hi);
}

// The same for 1 to 4 digits: the four bytes before e.
__device__ __forceinline__ uint32_t digits4(const uint32_t* s, int e, int len, uint32_t* bad) {
  const uint32_t t = (text_word(s, e - 4) ^ 0x30303030u) & (~0u << (8 * (4 - len)));
  *bad |= not_digits(t);
  return four_digits(t);
}

// One numeric field, bytes [b, e) of the text in shared memory: eight digits
// at a time for the common lengths, else byte by byte.
__device__ __forceinline__ bool parse_number(const CsvOut& o, const uint32_t* s, int b, int e, int64_t* v) {
  const uint8_t* t = reinterpret_cast<const uint8_t*>(s);
  const uint8_t c0 = b < e ? t[b] : 0;
  const int d0 = b + ((c0 == '-' || c0 == '+') ? 1 : 0);  // first digit
  uint32_t bad = 0;
  if (o.decimal) {
    const int dot = e - 1 - o.scale;
    if (o.scale >= 1 && o.scale <= 4 && dot >= d0 && dot - d0 <= 8 && t[dot] == '.') {
      const int64_t x = static_cast<int64_t>(digits8(s, dot, dot - d0, &bad)) * o.pow10 + digits4(s, e, o.scale, &bad);
      *v = c0 == '-' ? -x : x;
      return bad == 0;
    }
    return parse_decimal(t, b, e, o.scale, v);
  }
  if (e > d0 && e - d0 <= 8) {
    const int64_t x = digits8(s, e, e - d0, &bad);
    *v = c0 == '-' ? -x : x;
    return bad == 0;
  }
  return parse_int(t, b, e, v);
}

// A YYYY-MM-DD field: its ten bytes as three words.
__device__ __forceinline__ bool parse_date_words(const uint32_t* s, int b, int e, int32_t* v) {
  if (e - b != 10) return false;
  const uint32_t ty = text_word(s, b) ^ 0x30303030u;
  const uint32_t tm = text_word(s, b + 4) ^ 0x2D30302Du;                // "-MM-": the dashes to 0
  const uint32_t td = (text_word(s, b + 8) ^ 0x00003030u) & 0x0000FFFFu;
  const uint32_t bad = not_digits(ty) | (((tm + 0x7F76767Fu) | tm) & 0x80808080u) | not_digits(td);
  const uint32_t m = __dp4a(tm, 0x00010A00u, 0u), d = __dp4a(td, 0x0000010Au, 0u);
  if (bad != 0 || m < 1 || m > 12 || d < 1 || d > 31) return false;
  *v = days_from_civil(static_cast<int32_t>(four_digits(ty)), m, d);
  return true;
}

__device__ __forceinline__ void store_number(const CsvParams& p, const CsvOut& o, int64_t row, bool ok, int64_t v) {
  if (o.type == CT_DATE32) {
    static_cast<int32_t*>(o.data)[row] = static_cast<int32_t>(v);
  } else if (o.type == CT_I32) {
    if (v < INT32_MIN || v > INT32_MAX) ok = false;
    static_cast<int32_t*>(o.data)[row] = static_cast<int32_t>(v);
  } else {
    static_cast<int64_t*>(o.data)[row] = v;
  }
  if (!ok) csv_malformed(p.st, row);
}

// (2) every field, by the separator that ends it: a warp takes one column, 32
// rows at a time, so every lane makes the same conversion and stores coalesced
// into the column. Bound by issue (the conversions, and the lists of
// separators), so positions and rows are 32-bit offsets into the tile and
// what a column needs is set up once per tile.
__global__ void __launch_bounds__(kCsvThreads, 5) csv_fields_kernel(const __grid_constant__ CsvParams p) {
  extern __shared__ uint4 s_mem[];
  CsvTileShared& sh = *reinterpret_cast<CsvTileShared*>(s_mem);
  __shared__ unsigned long long s_bytes[kCsvMaxOut];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < kCsvMaxOut) s_bytes[threadIdx.x] = 0;  // walk_tile's barrier comes before its use
  const int64_t shift = static_cast<int64_t>(blockIdx.x) * kCsvTile - kCsvFront;  // text byte of sh.text's first
  const uint32_t* s = reinterpret_cast<const uint32_t*>(sh.text);
  const uint8_t* t = reinterpret_cast<const uint8_t*>(sh.text);
  const int rs = kCsvSepCap / p.n_fields + 3;
  const int share = p.n_out > 0 && p.n_out < kCsvWarps ? kCsvWarps / p.n_out : 1;  // warps of a column
  walk_tile(p, sh, [&](const CsvPart& pt) {
    for (int k = warp / share; k < p.n_out; k += kCsvWarps / share) {
      const CsvOut& o = p.out[k];
      const int c = o.field;
      const bool row_end = c == p.n_fields - 1;
      const bool far = pt.far && c == pt.c0;  // the field of row 0
      int first = pt.c0 > c || far ? 1 : 0;
      first = pt.lo > first ? pt.lo : first;
      int end = pt.rows - (pt.c1 < c ? 1 : 0);
      end = pt.hi < end ? pt.hi : end;
      const uint16_t* const from = sh.pos + c * rs;
      const int64_t row_base = pt.row0 - p.header;
      const int r0 = first + (warp % share) * 32 + lane, step = 32 * share;
      if (far && lane == 0 && warp % share == 0 && pt.lo == 0 && pt.hi > 0) {
        int64_t fb = sh.prev + 1 + shift, fe = from[rs] + shift;
        trim_field(p.text, fb, fe, row_end);
        if (o.type == CT_UTF8) {
          p.far[2 * blockIdx.x] = fb;
          p.far[2 * blockIdx.x + 1] = fe - fb;
          p.spans[o.utf8 * p.n_rows + row_base] = kCsvFar;
          atomicAdd(&s_bytes[o.utf8], static_cast<unsigned long long>(fe - fb));
        } else {
          int64_t v = 0;
          int32_t day = 0;
          const bool ok = o.type == CT_DATE32 ? parse_date(p.text, fb, fe, &day)
                          : o.decimal         ? parse_decimal(p.text, fb, fe, o.scale, &v)
                                              : parse_int(p.text, fb, fe, &v);
          store_number(p, o, row_base, ok, o.type == CT_DATE32 ? day : v);
        }
      }
      if (o.type == CT_UTF8) {
        uint32_t* const spans = p.spans + o.utf8 * p.n_rows + row_base;
        unsigned sum = 0;  // a tile's fields of one column but the far one: under 2^16 bytes
        for (int r = r0; r < end; r += step) {
          int b = (from[r] + 1) & 0xFFFF, e = from[rs + r];
          trim_field(t, b, e, row_end);
          spans[r] = static_cast<uint32_t>(e - b) << 16 | static_cast<uint32_t>(b);
          sum += e - b;
        }
        sum = __reduce_add_sync(0xffffffffu, sum);
        if (lane == 0) atomicAdd(&s_bytes[o.utf8], static_cast<unsigned long long>(sum));
      } else if (o.type == CT_DATE32) {
        int32_t* const out = static_cast<int32_t*>(o.data) + row_base;
        for (int r = r0; r < end; r += step) {
          int b = (from[r] + 1) & 0xFFFF, e = from[rs + r];
          trim_field(t, b, e, row_end);
          int32_t day = 0;
          if (!parse_date_words(s, b, e, &day)) csv_malformed(p.st, row_base + r);
          out[r] = day;
        }
      } else {
        for (int r = r0; r < end; r += step) {
          int b = (from[r] + 1) & 0xFFFF, e = from[rs + r];
          trim_field(t, b, e, row_end);
          int64_t v = 0;
          const bool ok = parse_number(o, s, b, e, &v);
          store_number(p, o, row_base + r, ok, v);
        }
      }
      __syncwarp();
    }
  });
  __syncthreads();
  for (int k = threadIdx.x; k < p.n_out; k += kCsvThreads)
    if (p.out[k].utf8 >= 0) {
      const int u = p.out[k].utf8;
      p.tile_bytes[u * p.n_tiles + blockIdx.x] = static_cast<int64_t>(s_bytes[u]);
      if (s_bytes[u] != 0) atomicAdd(p.byte_buckets + u * p.n_buckets + (blockIdx.x >> p.bucket_shift), s_bytes[u]);
    }
}

// (3) utf8 offsets and bytes. A warp takes a column of the tile, or with up to
// four columns a run of a column's rows (csv_share of them a column: a single
// column by one warp of the eight took 372 us the call for 3M strings of 20
// bytes, 221 with all eight), 32 rows at a time: their lengths, a warp scan for
// the offsets, then each lane copies its string into the warp's buffer in
// shared memory (words between a head and a tail of at most three bytes), laid
// out as the output's 16-byte lines, and the warp writes the buffer out in
// whole 16-byte stores with byte stores at its two ends. Groups of strings too
// long for the buffer go out a word of the output per lane, whichever rows its
// bytes are of (1.4M strings of 60 bytes: 251 us the call, 537 string by string
// with a byte per lane and one warp).
constexpr int kCsvStage = 1536;                            // bytes of a warp's buffer besides its alignment
constexpr int kCsvOutLines = (kCsvStage + 32) / 16;        // 16-byte lines of a warp's buffer
constexpr int csv_share(int columns) { return columns >= 1 && columns <= kCsvWarps / 2 ? kCsvWarps / columns : 1; }
constexpr int csv_strings_smem(int columns) {
  const int warps = columns * csv_share(columns);
  return (kCsvTextLines + (warps < kCsvWarps ? warps : kCsvWarps) * kCsvOutLines) * 16;
}

// kRuns: warps share a column's rows.
template <bool kRuns>
__global__ void __launch_bounds__(kCsvThreads, 5) csv_strings_kernel(const __grid_constant__ CsvParams p) {
  extern __shared__ uint4 s_mem[];
  __shared__ int32_t s_run[kCsvWarps];  // bytes of each warp's run of rows
  uint4* const s_text = s_mem;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // where this tile's separators begin and the next one's (the last tile's
  // end: a whole number of rows)
  const int64_t begin = p.tile_row[blockIdx.x];
  const int64_t end_row = blockIdx.x + 1 < gridDim.x ? p.tile_row[blockIdx.x + 1] : (p.n_rows + p.header) << 8;
  stage_tile(p, s_text);
  bool staged = false;  // the barrier after the staging, behind the first column's loads
  const uint32_t* s = reinterpret_cast<const uint32_t*>(s_text);
  const uint8_t* t = reinterpret_cast<const uint8_t*>(s_text);
  uint4* const s_out = s_mem + kCsvTextLines + warp * kCsvOutLines;
  uint32_t* const ow = reinterpret_cast<uint32_t*>(s_out);
  uint16_t* const oh = reinterpret_cast<uint16_t*>(s_out);
  uint8_t* const ob = reinterpret_cast<uint8_t*>(s_out);
  const int share = kRuns ? csv_share(p.n_utf8) : 1;
  auto length = [&](uint32_t span) {
    return (span & 0xFFFFu) == kCsvFar ? static_cast<int32_t>(p.far[2 * blockIdx.x + 1]) : static_cast<int32_t>(span >> 16);
  };
  for (int u = warp / share; u < p.n_utf8; u += kCsvWarps / share) {
    const CsvOut& o = p.out[p.utf8_out[u]];
    // the column's data rows whose separator lies in the tile
    int64_t row0 = (begin >> 8) + (o.field < (begin & 255) ? 1 : 0) - p.header;
    int64_t row1 = (end_row >> 8) + (o.field < (end_row & 255) ? 1 : 0) - p.header;
    if (row0 < 0) row0 = 0;
    if (row1 > p.n_rows) row1 = p.n_rows;
    uint8_t* const out = static_cast<uint8_t*>(o.data);
    const uint32_t* const spans = p.spans + u * p.n_rows;
    const int part = kRuns ? warp % share : 0;
    if (kRuns && row1 > row0) {  // this warp's run of them
      const int64_t run = (row1 - row0 + share - 1) / share;
      row0 = row0 + part * run < row1 ? row0 + part * run : row1;
      row1 = row0 + run < row1 ? row0 + run : row1;
      int32_t bytes = 0;  // a column holds less than 2^31 bytes (checked before the launch)
#pragma unroll 4
      for (int64_t r = row0 + lane; r < row1; r += 32) bytes += length(__ldg(spans + r));
      bytes = __reduce_add_sync(0xffffffffu, bytes);
      if (lane == 0) s_run[warp] = bytes;
    } else if (kRuns && lane == 0) {
      s_run[warp] = 0;
    }
    // a column's spans are loaded a group ahead of their use
    uint32_t ahead = row0 + lane < row1 ? __ldg(spans + row0 + lane) : 0u;
    int32_t base = static_cast<int32_t>(
        sum_before(p.byte_buckets + u * p.n_buckets, p.tile_bytes + u * p.n_tiles, blockIdx.x, p.bucket_shift));
    if (!staged) {
      __syncthreads();
      staged = true;
    }
    if (kRuns)
      for (int w = warp - part; w < warp; ++w) base += s_run[w];
    for (int64_t r = row0 + lane; r - lane < row1; r += 32) {
      const bool have = r < row1;
      const uint32_t span = ahead;
      ahead = r + 32 < row1 ? __ldg(spans + r + 32) : 0u;
      const bool far = have && (span & 0xFFFFu) == kCsvFar;
      const int b = static_cast<int>(span & 0xFFFFu);
      const int32_t len = length(span);
      int32_t incl = len;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
      }
      const int32_t total = __shfl_sync(0xffffffffu, incl, 31);
      const int32_t at = base + incl - len;
      if (have) {
        o.offs[r] = at;
        if (r == p.n_rows - 1) o.offs[r + 1] = at + len;
      }
      if (total <= kCsvStage && !__any_sync(0xffffffffu, far)) {
        const int a0 = base & 15;  // buffer byte 0 is the output's 16-byte line
        int d = a0 + incl - len;
        const int dend = d + len;
        int i = b;
        if ((d & 1) != 0 && d < dend) ob[d++] = t[i++];
        if ((d & 2) != 0 && d + 2 <= dend) {
          oh[d >> 1] = static_cast<uint16_t>(t[i] | t[i + 1] << 8);
          d += 2;
          i += 2;
        }
        // word-aligned now, unless fewer than two bytes are left
        const unsigned shl = 8u * (static_cast<unsigned>(i) & 3u);
        int w = i >> 2;
        uint32_t lo = s[w];
        const int words = (dend - d) >> 2;
        uint32_t* const to = ow + (d >> 2);
#pragma unroll 4
        for (int x = 0; x < words; ++x) {
          const uint32_t hi = s[++w];
          to[x] = __funnelshift_r(lo, hi, shl);
          lo = hi;
        }
        d += words > 0 ? 4 * words : 0;
        if (d < dend) {  // the last one to three bytes
          uint32_t x = __funnelshift_r(lo, s[w + 1], shl);
          if (d + 2 <= dend) {
            oh[d >> 1] = static_cast<uint16_t>(x);
            x >>= 16;
            d += 2;
          }
          if (d < dend) ob[d] = static_cast<uint8_t>(x);
        }
        __syncwarp();
        const int end = a0 + total;
        uint8_t* const line0 = out + (base - a0);
        const int v0 = (a0 + 15) / 16, v1 = end / 16;  // whole lines [v0, v1)
        if (v0 <= v1) {
          for (int q = v0 + lane; q < v1; q += 32) reinterpret_cast<uint4*>(line0)[q] = s_out[q];
          if (lane < 16) {
            if (lane >= a0 && v0 == 1) line0[lane] = ob[lane];
          } else if (16 * v1 + lane - 16 < end) {
            line0[16 * v1 + lane - 16] = ob[16 * v1 + lane - 16];
          }
        } else if (lane >= a0 && lane < end) {  // within one line
          line0[lane] = ob[lane];
        }
        __syncwarp();  // the buffer is rewritten by the next group
      } else {
        // word by word of the output: where each row's bytes begin in it, and
        // what its text lies at from there, in the warp's buffer
        int32_t* const off = reinterpret_cast<int32_t*>(s_out);
        int32_t* const from = off + 33;
        off[lane + 1] = at + len;
        if (lane == 0) off[0] = base;
        from[lane] = b - at;  // a far row's bytes are read from the text itself
        const int far_row = __ffs(static_cast<int>(__ballot_sync(0xffffffffu, far))) - 1;  // one at most
        const uint8_t* const far_text = far_row >= 0 ? p.text + p.far[2 * blockIdx.x] : nullptr;
        __syncwarp();
        const int32_t far_at = far_row >= 0 ? off[far_row] : 0;
        const int32_t end = base + total;
        auto byte = [&](int row, int32_t q) { return row == far_row ? far_text[q - far_at] : t[from[row] + q]; };
        const int32_t w0 = (base + 3) >> 2, w1 = end >> 2;  // whole words [w0, w1)
        {  // the bytes before and after them, three at most each
          const int32_t head = 4 * w0 < end ? 4 * w0 : end, tail = 4 * w1 > head ? 4 * w1 : head;
          const int32_t q = lane < 4 ? base + lane : tail + lane - 4;
          if (lane < 4 ? q < head : lane < 8 && q < end) {
            int row = lane < 4 ? 0 : static_cast<int>(row1 - (r - lane) < 32 ? row1 - (r - lane) : 32) - 1;
            while (off[row + 1] <= q) ++row;
            while (off[row] > q) --row;
            out[q] = byte(row, q);
          }
        }
        int row = 0;
        int32_t row_end = off[1], place = from[0];
        for (int32_t w = w0 + lane; w < w1; w += 32) {
          const int32_t q = 4 * w;
          if (q >= row_end) {
            do ++row;
            while (off[row + 1] <= q);  // q < end
            row_end = off[row + 1];
            place = from[row];
          }
          uint32_t x;
          const bool one = q + 4 <= row_end;
          if (row != far_row && (one || off[row + 2] >= q + 4)) {
            x = text_word(s, place + q);
            if (!one) {  // its last bytes are the next row's first ones
              const uint32_t next = ~0u << (8 * (row_end - q));
              x = (x & ~next) | (text_word(s, from[row + 1] + q) & next);
            }
          } else if (one) {
            const uint8_t* const f = far_text + (q - far_at);
            x = f[0] | f[1] << 8 | f[2] << 16 | static_cast<uint32_t>(f[3]) << 24;
          } else {
            x = 0;
            int at_row = row;
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
              while (off[at_row + 1] <= q + k) ++at_row;
              x |= static_cast<uint32_t>(byte(at_row, q + k)) << (8 * k);
            }
          }
          reinterpret_cast<uint32_t*>(out)[w] = x;
        }
        __syncwarp();  // the buffer is rewritten by the next group
      }
      base += total;
    }
  }
  if (!staged) __syncthreads();  // a warp without a column
}

}  // namespace

TupleSetPtr csv_parse(const char* device_text, int64_t n_bytes, char delimiter, bool has_header,
                      const std::vector<CsvField>& fields, const std::vector<int>& emit, cudaStream_t s) {
  if (fields.empty()) fail(GFPDB_EINVAL, "CSV schema has no fields");
  if (static_cast<int>(emit.size()) > kCsvMaxOut) fail(GFPDB_EUNSUPPORTED, "too many CSV columns to emit");
  if (static_cast<int>(fields.size()) > 256) fail(GFPDB_EUNSUPPORTED, "too many CSV fields per line");
  if (n_bytes >= (int64_t{1} << 40)) fail(GFPDB_EUNSUPPORTED, "CSV text too large");
  const uint8_t* text = reinterpret_cast<const uint8_t*>(device_text);
  allow_shared(csv_fields_kernel, csv_fields_smem(1));  // the most
  allow_shared(csv_strings_kernel<true>, csv_strings_smem(kCsvWarps));  // the most
  allow_shared(csv_strings_kernel<false>, csv_strings_smem(kCsvWarps));
  if ((reinterpret_cast<uintptr_t>(text) & 15u) != 0) fail(GFPDB_EINVAL, "CSV text must be 16-byte aligned");

  if (static_cast<int>(fields.size()) > kCsvMaxFields) fail(GFPDB_EUNSUPPORTED, "too many CSV fields per line");
  const int F = static_cast<int>(fields.size());
  // (1) separators per tile and per bucket of tiles. One scratch buffer: the
  // buckets (cleared: separators, the text's last byte, then per emitted utf8
  // column its bytes), the separator bits, then the tiles' rows. A bucket
  // holds about as many tiles as there are buckets, 256 at least.
  const int64_t n_tiles = n_bytes > 0 ? (n_bytes + kCsvTile - 1) / kCsvTile : 0;
  if (n_tiles >= INT32_MAX) fail(GFPDB_EUNSUPPORTED, "CSV text too large");
  int n_utf8 = 0;
  for (int f : emit) n_utf8 += fields[f].type == DType::Utf8 ? 1 : 0;
  const int64_t nt = std::max<int64_t>(n_tiles, 1);
  int shift = 8;
  while ((nt >> shift) > (int64_t{1} << shift)) ++shift;
  const int64_t nb = (nt >> shift) + 1;
  constexpr int64_t kChunkWords = kCsvTile / 64;  // words of separator bits of a tile
  const int64_t bucket_words = (nb * (1 + n_utf8) + 2) / 2 * 2;
  auto scratch = make_buffer((bucket_words + nt * kChunkWords + nt * (5 + n_utf8)) * 8, s);
  auto* sep_buckets = scratch->as<unsigned long long>();
  unsigned long long* last_byte = sep_buckets + nb;
  unsigned long long* byte_buckets = last_byte + 1;
  uint64_t* masks = reinterpret_cast<uint64_t*>(sep_buckets + bucket_words);  // 16-byte aligned
  int64_t* tile_last = reinterpret_cast<int64_t*>(masks + nt * kChunkWords);
  int64_t* tile_row = tile_last + nt;
  int64_t* far = tile_row + nt;
  int64_t* tile_bytes = far + 2 * nt;
  int32_t* tile_count = reinterpret_cast<int32_t*>(tile_bytes + nt * n_utf8);
  std::vector<unsigned long long> sums(bucket_words, 0);
  sums[nb] = '\n';
  if (n_tiles > 0) {
    GF_CUDA(cudaMemsetAsync(sep_buckets, 0, bucket_words * 8, s));
    ProfScope prof("csv_index_kernel", s);
    csv_index_kernel<<<static_cast<int>(n_tiles), kCsvThreads, 0, s>>>(
        text, n_bytes, static_cast<uint8_t>(delimiter), tile_count, tile_last, reinterpret_cast<uint16_t*>(masks),
        sep_buckets, shift, last_byte);
    after_launch("csv_index_kernel");
    prof.stop(static_cast<double>(n_bytes));
    GF_CUDA(cudaMemcpyAsync(sums.data(), sep_buckets, (nb + 1) * 8, cudaMemcpyDeviceToHost, s));
    sync(s);
  }
  const bool virtual_end = n_bytes > 0 && sums[nb] != '\n';
  int64_t seps = virtual_end ? 1 : 0;
  for (int64_t b = 0; b < nb; ++b) seps += static_cast<int64_t>(sums[b]);
  if (seps % F != 0)
    fail(GFPDB_EINVAL, "malformed CSV field or wrong field count near data row " + std::to_string(seps / F));
  const int64_t lines = seps / F;
  const int64_t skip = has_header && lines > 0 ? 1 : 0;
  const int64_t n_rows = lines - skip;

  // (2) fields
  std::vector<Field> out_fields;
  std::vector<BufferPtr> bufs(emit.size()), offs(emit.size());
  CsvParams* pp = new CsvParams;
  std::unique_ptr<CsvParams> holder(pp);
  CsvParams& p = *pp;
  std::memset(&p, 0, sizeof(p));
  p.text = text;
  p.n = n_bytes;
  p.n_tiles = nt;
  p.bucket_shift = shift;
  p.n_buckets = nb;
  p.sep_buckets = sep_buckets;
  p.byte_buckets = byte_buckets;
  p.tile_count = tile_count;
  p.tile_last = tile_last;
  p.tile_row = tile_row;
  p.chunk_masks = masks;
  p.tile_bytes = tile_bytes;
  auto spans = make_buffer(n_utf8 * n_rows * 4, s);
  p.spans = spans->as<uint32_t>();
  p.far = far;
  p.n_rows = n_rows;
  p.n_fields = F;
  p.inv_fields = F == 1 ? 0u : static_cast<uint32_t>(((uint64_t{1} << 32) + F - 1) / F);
  p.n_out = static_cast<int32_t>(emit.size());
  p.header = static_cast<int32_t>(skip);
  p.virtual_end = virtual_end ? 1 : 0;
  auto status = make_filled(sizeof(DevStatus), 0, s);
  p.st = status->as<DevStatus>();
  std::vector<bool> taken(fields.size(), false);
  std::vector<size_t> utf8;
  for (size_t k = 0; k < emit.size(); ++k) {
    const CsvField& f = fields[emit[k]];
    if (taken[emit[k]]) fail(GFPDB_EINVAL, "CSV column '" + f.name + "' projected twice");
    taken[emit[k]] = true;
    out_fields.push_back(Field{f.name, f.type});
    CsvOut& o = p.out[k];
    o.type = static_cast<int32_t>(f.type);
    o.decimal = f.decimal ? 1 : 0;
    o.scale = f.scale;
    o.pow10 = 1;
    for (int d = 0; d < f.scale; ++d) o.pow10 *= 10;  // scale <= 9
    o.field = emit[k];
    o.utf8 = -1;
    if (f.type == DType::Utf8) {
      o.utf8 = p.n_utf8++;
      p.utf8_out[o.utf8] = static_cast<int32_t>(k);
      utf8.push_back(k);
    } else {
      bufs[k] = make_buffer(n_rows * dtype_width(f.type), s);
      o.data = bufs[k]->data();
    }
  }
  if (n_tiles > 0) {
    ProfScope prof("csv_fields_kernel", s);
    csv_fields_kernel<<<static_cast<int>(n_tiles), kCsvThreads, csv_fields_smem(F), s>>>(p);
    after_launch("csv_fields_kernel");
    double out_w = 0;
    for (auto& f : out_fields) out_w += f.type == DType::Utf8 ? 4 : dtype_width(f.type);
    prof.stop(static_cast<double>(n_bytes) + static_cast<double>(n_rows) * out_w);
  }
  // One synchronization for the parse status and the utf8 columns' sizes (the
  // parse status first: a malformed text reports as such).
  std::vector<int64_t> totals(utf8.size(), 0);
  {
    if (n_tiles > 0 && !utf8.empty())
      GF_CUDA(cudaMemcpyAsync(sums.data(), byte_buckets, nb * n_utf8 * 8, cudaMemcpyDeviceToHost, s));
    DevStatus hs;
    GF_CUDA(cudaMemcpyAsync(&hs, status->data(), sizeof(DevStatus), cudaMemcpyDeviceToHost, s));
    sync(s);
    if (hs.code == GFPDB_EINVAL)
      fail(GFPDB_EINVAL, "malformed CSV field or wrong field count near data row " + std::to_string(hs.detail));
    raise_device_status(hs, "CSV parse");
    for (size_t u = 0; u < utf8.size() && n_tiles > 0; ++u) {
      for (int64_t b = 0; b < nb; ++b) totals[u] += static_cast<int64_t>(sums[u * nb + b]);
      if (totals[u] > INT32_MAX) fail(GFPDB_EUNSUPPORTED, "utf8 column exceeds 2 GiB of bytes");
    }
  }
  // (3) utf8 offsets and bytes
  double string_bytes = 0;
  for (size_t u = 0; u < utf8.size(); ++u) {
    const size_t k = utf8[u];
    offs[k] = make_buffer((n_rows + 1) * 4, s);
    bufs[k] = make_buffer(totals[u], s);
    p.out[k].data = bufs[k]->data();
    p.out[k].offs = offs[k]->as<int32_t>();
    if (n_rows == 0) GF_CUDA(cudaMemsetAsync(offs[k]->data(), 0, 4, s));
    string_bytes += static_cast<double>(totals[u]) + 4.0 * static_cast<double>(n_rows);
  }
  if (n_rows > 0 && !utf8.empty()) {
    ProfScope prof("csv_strings_kernel", s);
    const auto strings = csv_share(n_utf8) > 1 ? csv_strings_kernel<true> : csv_strings_kernel<false>;
    strings<<<static_cast<int>(n_tiles), kCsvThreads, csv_strings_smem(n_utf8), s>>>(p);
    after_launch("csv_strings_kernel");
    prof.stop(static_cast<double>(n_bytes) + string_bytes + 4.0 * static_cast<double>(n_rows) * n_utf8);
  }
  std::vector<ColumnPtr> cols;
  for (size_t k = 0; k < emit.size(); ++k)
    cols.push_back(out_fields[k].type == DType::Utf8 ? make_utf8_column(n_rows, offs[k], bufs[k])
                                                     : make_fixed_column(out_fields[k].type, n_rows, bufs[k]));
  return TupleSet::make(std::move(out_fields), std::move(cols), n_rows);
}

}  // namespace gfpdb
