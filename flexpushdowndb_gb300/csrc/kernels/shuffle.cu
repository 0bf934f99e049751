// Hash partitioning of a TupleSet's rows into slots: the GPU form of
// ShuffleKernel2::shuffle (fpdb-executor/src/physical/shuffle/ShuffleKernel2.cpp:28-125),
// which hashes the shuffle columns of every row (RecordBatchHasher), appends
// the row id to the list of slot hash % numSlots, takes the rows in slot order
// and slices the result into one TupleSet per slot. Rows keep their input
// order within a slot.
//
// Here the slot of a row is a fast range of a 64-bit mix of the row's key
// hash (row_key_hash: integers by value, utf8 by bytes), independent of the
// low bits that join and group tables index by and of the bloom's block bits.
// The reference's partition function is Arrow's HashMultiColumn; which slot a
// key lands in does not change any query's result, only that equal keys land
// in the same slot.
//
// Three launches, all stable and without global atomics, over tiles of 256
// rows per warp of a block (4096 rows for 16 warps, 2048 for 8):
//   shuffle_count_kernel   hashes the tile's rows (several key loads in flight
//                          per thread), keeps each row's slot in 16 bits and
//                          counts the slots by shared-memory atomics; the
//                          counts land slot-major in a [slots][tiles] matrix;
//   shuffle_scan_kernel    one block per slot: its tiles' counts become
//                          offsets within the slot, and the slot's total;
//   shuffle_scatter_kernel ranks the tile's rows (a lane's peers with the same
//                          slot from one ballot per slot bit) and gives every
//                          row its place in the tile's slot order (input order
//                          kept); then each column is read in row order, put
//                          into shared memory in slot order and written from
//                          there, so reads are whole lines and writes whole
//                          sectors of one slot's run. utf8 columns are
//                          gathered afterwards through the inverse permutation
//                          that the same kernel writes.
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "launch.h"

namespace gfpdb {
namespace {

constexpr int kShufMaxFixed = 24;   // fixed-width columns scattered per launch
constexpr int kShufRowsPerWarp = 256;
constexpr int kShufPerLane = kShufRowsPerWarp / 32;
constexpr int kShufUnroll = 8;      // key loads in flight per thread

struct ShufKeys {
  DevCol keys[kMaxKeyColumns];
  int32_t n_keys;
  uint32_t slots;
  int64_t n;       // rows
  int32_t tile;    // rows per block: warps * kShufRowsPerWarp
  int32_t pad;
  int64_t ntiles;
};

struct ShufScatter {
  const void* src[kShufMaxFixed];
  void* dst[kShufMaxFixed];
  int8_t width[kShufMaxFixed];
  int32_t n_fixed;
  int32_t pad;
  const uint16_t* row_slot;  // slot of each row
  const int32_t* starts;     // [slots][ntiles] rows of the slot in earlier tiles
  const int32_t* totals;     // [slots] rows of the slot
  int32_t* inverse;          // inverse[out row] = input row (utf8 columns), or null
};

__device__ __forceinline__ uint32_t slot_of(uint64_t h, uint32_t slots) {
  const uint64_t g = mix64(h ^ 0x5851f42d4c957f2dull);
  return static_cast<uint32_t>(((g >> 32) * slots) >> 32);
}

// Lanes of the warp whose slot equals this lane's (the lane itself
// included), from one ballot per slot bit: the live lanes agreeing with this
// lane on every bit.
template <int kBits>
__device__ __forceinline__ unsigned slot_peers(uint32_t s, bool live) {
  unsigned peers = __ballot_sync(0xffffffffu, live);
#pragma unroll
  for (int b = 0; b < kBits; ++b) {
    const unsigned ones = __ballot_sync(0xffffffffu, (s >> b) & 1u);
    peers &= ((s >> b) & 1u) ? ones : ~ones;
  }
  return peers;
}

enum ShufKeyKind { kKeyI32, kKeyI64, kKeyAny };

// The multiplies of three 64-bit mixes a row hold it (issue 68%, math pipe
// throttle): 62 us for 20M int64 keys, as before it also wrote the slots. The
// scatter reads the 2-byte slot instead of hashing the key again.
template <int kKind>
__global__ void __launch_bounds__(512)
    shuffle_count_kernel(const __grid_constant__ ShufKeys p, uint16_t* row_slot, int32_t* counts) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  int32_t* hist = reinterpret_cast<int32_t*>(s_raw);
  const int64_t begin = static_cast<int64_t>(blockIdx.x) * p.tile;
  const int rows = static_cast<int>(begin + p.tile < p.n ? p.tile : p.n - begin);
  const int step = blockDim.x;
  for (uint32_t i = threadIdx.x; i < p.slots; i += step) hist[i] = 0;
  __syncthreads();
  row_slot += begin;
  for (int base = threadIdx.x; base < rows; base += kShufUnroll * step) {
    uint64_t h[kShufUnroll];
#pragma unroll
    for (int u = 0; u < kShufUnroll; ++u) {
      const int i = base + u * step;
      h[u] = 0;
      if (i < rows) {
        if (kKind == kKeyI32) h[u] = static_cast<uint64_t>(static_cast<int64_t>(__ldcs(static_cast<const int*>(p.keys[0].data) + begin + i)));
        else if (kKind == kKeyI64) h[u] = static_cast<uint64_t>(__ldcs(static_cast<const long long*>(p.keys[0].data) + begin + i));
        else h[u] = row_key_hash(p.keys, p.n_keys, begin + i);
      }
    }
#pragma unroll
    for (int u = 0; u < kShufUnroll; ++u) {
      const int i = base + u * step;
      if (kKind != kKeyAny) h[u] = row_key_combine(kRowKeySeed, hash_key(static_cast<int64_t>(h[u])));
      if (i < rows) {
        const uint32_t s = slot_of(h[u], p.slots);
        row_slot[i] = static_cast<uint16_t>(s);
        atomicAdd(&hist[s], 1);
      }
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < p.slots; i += step)
    counts[static_cast<int64_t>(i) * p.ntiles + blockIdx.x] = hist[i];
}

// Inclusive prefix sum of one value per thread over the block; *total is the
// block's sum. warp_sums: 32 words that no thread uses when it is called.
template <class T>
__device__ __forceinline__ T block_inclusive_scan(T v, T* warp_sums, T* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const T t = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += t;
  }
  if (lane == 31) warp_sums[warp] = v;
  __syncthreads();
  T w = lane < nw ? warp_sums[lane] : T{0};
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const T t = __shfl_up_sync(0xffffffffu, w, d);
    if (lane >= d) w += t;
  }
  *total = __shfl_sync(0xffffffffu, w, 31);
  const T before = __shfl_sync(0xffffffffu, w, warp > 0 ? warp - 1 : 0);
  __syncthreads();
  return warp > 0 ? v + before : v;
}

// Block s: counts[s][0, ntiles) becomes its exclusive prefix sum, in place.
__global__ void __launch_bounds__(1024) shuffle_scan_kernel(int32_t* counts, int64_t ntiles, int32_t* totals) {
  __shared__ int32_t warp_sums[32];
  int32_t* row = counts + static_cast<int64_t>(blockIdx.x) * ntiles;
  int32_t run = 0;
  for (int64_t at = 0; at < ntiles; at += blockDim.x) {
    const int64_t i = at + threadIdx.x;
    const int32_t v = i < ntiles ? row[i] : 0;
    int32_t sum;
    const int32_t incl = block_inclusive_scan(v, warp_sums, &sum);
    if (i < ntiles) row[i] = run + incl - v;
    run += sum;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = run;
}

// Dynamic shared memory of the scatter: a column of the tile in slot order,
// the output row of each of its places, per-slot words, per-warp counts.
constexpr int64_t shuf_scatter_smem(int64_t tile, int64_t slots) {
  return tile * 12 + slots * 4 + (tile / kShufRowsPerWarp) * slots * 2;
}

// Bound by latency: a tile goes through a chain of barriers (rank, scan, and
// two a column), so what counts is how many tiles an SM has in flight. 8 rows
// a lane keep it to 40 registers, three blocks of 16 warps an SM. 20M rows of
// 20 bytes over 256 slots: 197 us (237 us with 16 rows a lane and 32 warps an
// SM, 228 us with the next column's loads ahead of the writes at 64
// registers, 246 us with tiles of 2048 rows). Reading the rows in slot order
// straight from memory, a lookup per lane in the L1, and ranking them twice
// took 305 us.
template <int kBits>
__global__ void __launch_bounds__(512, 3) shuffle_scatter_kernel(const __grid_constant__ ShufKeys p,
                                                                 const __grid_constant__ ShufScatter q) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ int64_t warp_sums[32];
  const int tile = p.tile;
  const int nw = blockDim.x >> 5;
  const int slots = static_cast<int>(p.slots);
  uint64_t* stage8 = reinterpret_cast<uint64_t*>(s_raw);  // [tile]
  uint32_t* stage4 = reinterpret_cast<uint32_t*>(s_raw);
  int32_t* sdest = reinterpret_cast<int32_t*>(stage8 + tile);     // [tile] output row of each place
  int32_t* delta = sdest + tile;                                  // [slots] output row less place
  uint16_t* wcnt = reinterpret_cast<uint16_t*>(delta + slots);    // [warps][slots]
  const int64_t begin = static_cast<int64_t>(blockIdx.x) * tile;
  const int rows = static_cast<int>(begin + tile < p.n ? tile : p.n - begin);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r0 = warp * kShufRowsPerWarp + lane;  // this lane's rows: r0 + 32 j

  uint32_t at[kShufPerLane];  // slot | rank among the warp's rows of the slot << 16, later the row's place
#pragma unroll
  for (int j = 0; j < kShufPerLane; ++j)
    at[j] = r0 + 32 * j < rows ? __ldcs(q.row_slot + begin + r0 + 32 * j) : 0u;
  for (int i = threadIdx.x; i < nw * slots; i += blockDim.x) wcnt[i] = 0;
  __syncthreads();

  uint16_t* mine = wcnt + warp * slots;
  const unsigned below = (1u << lane) - 1u;
#pragma unroll
  for (int j = 0; j < kShufPerLane; ++j) {
    const bool live = r0 + 32 * j < rows;
    const uint32_t s = at[j];
    const unsigned peers = slot_peers<kBits>(s, live);
    const uint32_t had = mine[s];
    __syncwarp();
    if (live && (peers & below) == 0) mine[s] = static_cast<uint16_t>(had + __popc(peers));
    __syncwarp();
    at[j] = s | (had + __popc(peers & below)) << 16;
  }
  __syncthreads();

  // Slots in order, a block's width at a time: where the slot begins in the
  // tile's order and in the output, and where each warp's rows of it begin.
  // One scan carries both sums: a tile's rows in the low 14 bits.
  int64_t run = 0;
  for (int s0 = 0; s0 < slots; s0 += blockDim.x) {
    const int s = s0 + threadIdx.x;
    int32_t mid = 0;
    int64_t both = 0;
    if (s < slots) {
      for (int w = 0; w < nw; ++w) mid += wcnt[w * slots + s];
      both = static_cast<int64_t>(q.totals[s]) << 14 | mid;
    }
    int64_t sum;
    const int64_t excl = run + block_inclusive_scan(both, warp_sums, &sum) - both;
    run += sum;
    if (s < slots) {
      int32_t place = static_cast<int32_t>(excl & 0x3FFF);
      delta[s] = static_cast<int32_t>(excl >> 14) + q.starts[static_cast<int64_t>(s) * p.ntiles + blockIdx.x] - place;
      for (int w = 0; w < nw; ++w) {
        const int32_t c = wcnt[w * slots + s];
        wcnt[w * slots + s] = static_cast<uint16_t>(place);
        place += c;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kShufPerLane; ++j) {
    const uint32_t s = at[j] & 0xFFFFu;
    at[j] = mine[s] + (at[j] >> 16);
    if (r0 + 32 * j < rows) sdest[at[j]] = static_cast<int32_t>(at[j]) + delta[s];
  }

  for (int c = 0; c < q.n_fixed; ++c) {
    if (q.width[c] == 8) {
      const long long* src = static_cast<const long long*>(q.src[c]) + begin;
      long long* dst = static_cast<long long*>(q.dst[c]);
      long long v[kShufPerLane];
#pragma unroll
      for (int j = 0; j < kShufPerLane; ++j) v[j] = r0 + 32 * j < rows ? __ldcs(src + r0 + 32 * j) : 0;
      __syncthreads();  // the column before it has left the stage
#pragma unroll
      for (int j = 0; j < kShufPerLane; ++j)
        if (r0 + 32 * j < rows) stage8[at[j]] = static_cast<uint64_t>(v[j]);
      __syncthreads();
#pragma unroll 4
      for (int i = threadIdx.x; i < rows; i += blockDim.x) dst[sdest[i]] = static_cast<long long>(stage8[i]);
    } else {
      const int* src = static_cast<const int*>(q.src[c]) + begin;
      int* dst = static_cast<int*>(q.dst[c]);
      int v[kShufPerLane];
#pragma unroll
      for (int j = 0; j < kShufPerLane; ++j) v[j] = r0 + 32 * j < rows ? __ldcs(src + r0 + 32 * j) : 0;
      __syncthreads();
#pragma unroll
      for (int j = 0; j < kShufPerLane; ++j)
        if (r0 + 32 * j < rows) stage4[at[j]] = static_cast<uint32_t>(v[j]);
      __syncthreads();
#pragma unroll 4
      for (int i = threadIdx.x; i < rows; i += blockDim.x) dst[sdest[i]] = static_cast<int>(stage4[i]);
    }
  }
  if (q.inverse != nullptr) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kShufPerLane; ++j)
      if (r0 + 32 * j < rows) stage4[at[j]] = static_cast<uint32_t>(begin + r0 + 32 * j);
    __syncthreads();
    for (int i = threadIdx.x; i < rows; i += blockDim.x) q.inverse[sdest[i]] = static_cast<int32_t>(stage4[i]);
  }
}

}  // namespace

ShuffleResult shuffle_rows(const TupleSetPtr& in_ts, const std::vector<std::string>& keys, int64_t num_slots,
                           cudaStream_t s) {
  if (keys.empty() || keys.size() > static_cast<size_t>(kMaxKeyColumns))
    fail(GFPDB_EINVAL, "a shuffle key has 1 to 8 columns");
  if (num_slots < 1 || num_slots > kShuffleMaxSlots)
    fail(GFPDB_EINVAL, "shuffle slots must be 1 to " + std::to_string(kShuffleMaxSlots));
  TupleSetPtr in = resolved(in_ts, s);
  const int64_t n = in->num_rows();
  if (n > INT32_MAX) fail(GFPDB_EUNSUPPORTED, "a shuffle input has at most 2^31 - 1 rows");

  ShufKeys p;
  std::memset(&p, 0, sizeof(p));
  for (size_t i = 0; i < keys.size(); ++i) {
    const auto& c = in->column(in->require_column(keys[i]));
    if (c->type == DType::Float64) fail(GFPDB_EUNSUPPORTED, "float64 shuffle column '" + keys[i] + "'");
    p.keys[i] = DevCol{c->data, c->offsets, static_cast<int32_t>(c->type), 0};
  }
  p.n_keys = static_cast<int32_t>(keys.size());
  p.slots = static_cast<uint32_t>(num_slots);
  p.n = n;

  ShuffleResult r;
  r.offsets.assign(num_slots + 1, 0);
  r.offsets[num_slots] = n;
  if (n == 0) {
    r.rows = in;
    return r;
  }

  // 16 warps a tile: runs of one slot are twice as long as with 8. Inputs that
  // would leave an SM with less than two such tiles take 8.
  const int warps = n >= static_cast<int64_t>(num_sms()) * 2 * 16 * kShufRowsPerWarp ? 16 : 8;
  p.tile = warps * kShufRowsPerWarp;
  p.ntiles = (n + p.tile - 1) / p.tile;
  const int blocks = static_cast<int>(p.ntiles);
  const int64_t smem_scatter = shuf_scatter_smem(p.tile, num_slots);
  const auto scatter = num_slots <= 32    ? shuffle_scatter_kernel<5>
                       : num_slots <= 256 ? shuffle_scatter_kernel<8>
                                          : shuffle_scatter_kernel<10>;
  allow_shared(scatter, smem_scatter);

  const int64_t cells = num_slots * p.ntiles;
  auto row_slot = make_buffer(n * 2, s);
  auto starts = make_buffer((cells + num_slots) * 4, s);
  int32_t* totals = starts->as<int32_t>() + cells;
  {
    ProfScope prof("shuffle_count_kernel", s);
    const auto count = p.n_keys == 1 && p.keys[0].type == CT_I64    ? shuffle_count_kernel<kKeyI64>
                       : p.n_keys == 1 && p.keys[0].type != CT_UTF8 ? shuffle_count_kernel<kKeyI32>
                                                                    : shuffle_count_kernel<kKeyAny>;
    count<<<blocks, warps * 32, num_slots * 4, s>>>(p, row_slot->as<uint16_t>(), starts->as<int32_t>());
    after_launch("shuffle_count_kernel");
    prof.stop(static_cast<double>(n) * (4.0 * p.n_keys + 2.0) + static_cast<double>(cells) * 4.0);
  }
  {
    ProfScope prof("shuffle_scan_kernel", s);
    const int64_t threads = std::min<int64_t>(1024, (p.ntiles + 31) / 32 * 32);
    shuffle_scan_kernel<<<static_cast<int>(num_slots), static_cast<int>(threads), 0, s>>>(starts->as<int32_t>(),
                                                                                          p.ntiles, totals);
    after_launch("shuffle_scan_kernel");
    prof.stop(2.0 * static_cast<double>(cells) * 4.0);
  }

  // Output columns: fixed-width ones scattered by the kernel (in groups of
  // kShufMaxFixed, the ranking repeated per group), utf8 ones gathered
  // through the inverse permutation.
  std::vector<ColumnPtr> out(in->num_columns());
  std::vector<int> fixed, utf8;
  for (int i = 0; i < in->num_columns(); ++i) (in->column(i)->type == DType::Utf8 ? utf8 : fixed).push_back(i);
  BufferPtr inverse;
  if (!utf8.empty()) inverse = make_buffer(n * 4, s);
  size_t at = 0;
  do {
    ShufScatter q;
    std::memset(&q, 0, sizeof(q));
    q.row_slot = row_slot->as<uint16_t>();
    q.starts = starts->as<int32_t>();
    q.totals = totals;
    const size_t take = std::min<size_t>(kShufMaxFixed, fixed.size() - at);
    for (size_t j = 0; j < take; ++j) {
      const auto& c = in->column(fixed[at + j]);
      const int w = dtype_width(c->type);
      auto buf = make_buffer(n * w, s);
      q.src[j] = c->data;
      q.dst[j] = buf->data();
      q.width[j] = static_cast<int8_t>(w);
      out[fixed[at + j]] = make_fixed_column(c->type, n, buf);
    }
    q.n_fixed = static_cast<int32_t>(take);
    if (at == 0 && inverse) q.inverse = inverse->as<int32_t>();
    ProfScope prof("shuffle_scatter_kernel", s);
    scatter<<<blocks, warps * 32, smem_scatter, s>>>(p, q);
    after_launch("shuffle_scatter_kernel");
    double bytes = static_cast<double>(n) * 2.0 + (q.inverse ? n * 4.0 : 0.0);
    for (size_t j = 0; j < take; ++j) bytes += 2.0 * n * q.width[j];
    prof.stop(bytes);
    at += take;
  } while (at < fixed.size());
  if (!utf8.empty()) {
    std::vector<GatherSpec> specs;
    for (int i : utf8) specs.push_back(GatherSpec{in->column(i).get(), inverse->as<int32_t>()});
    auto g = gather_columns(specs, n, s);
    for (size_t j = 0; j < utf8.size(); ++j) out[utf8[j]] = g[j];
  }

  std::vector<int32_t> rows(num_slots);
  GF_CUDA(cudaMemcpyAsync(rows.data(), totals, static_cast<size_t>(num_slots) * 4, cudaMemcpyDeviceToHost, s));
  sync(s);
  for (int64_t i = 0; i < num_slots; ++i) r.offsets[i + 1] = r.offsets[i] + rows[i];
  r.rows = TupleSet::make(in->fields(), std::move(out), n);
  return r;
}

TupleSetPtr slice_rows(const TupleSetPtr& ts, int64_t at, int64_t len) {
  std::vector<ColumnPtr> cols;
  for (int i = 0; i < ts->num_columns(); ++i) {
    const auto& c = ts->column(i);
    auto sl = std::make_shared<Column>(*c);
    sl->length = len;
    if (c->valid != nullptr) {
      if (at % 32 != 0) fail(GFPDB_EUNSUPPORTED, "a slice of a nullable column must start at a multiple of 32 rows");
      sl->valid = c->valid + at / 32;
    }
    if (c->type == DType::Utf8) sl->offsets = c->offsets + at;
    else sl->data = static_cast<const char*>(c->data) + at * dtype_width(c->type);
    cols.push_back(sl);
  }
  return TupleSet::make(ts->fields(), std::move(cols), len);
}

}  // namespace gfpdb
