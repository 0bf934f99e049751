// Hash group-by with exact integer aggregates.
//
// Replaces the Arrow hash aggregate (hash_sum / hash_count / hash_min_max)
// that GroupArrowKernel drives (fpdb-executor/src/physical/group/GroupArrowKernel.cpp:127-154,
// fpdb-executor/src/physical/aggregate/function/Sum.cpp:63-74, Count.cpp:91-104)
// and the native GroupKernel (fpdb-executor/src/physical/group/GroupKernel.cpp:263-300).
//
// Keys: up to two key columns packed into one 64-bit word (32 bits per int32 /
// date32 column, 64 bits for one int64 column); a utf8 key column is first
// mapped to dense int32 codes by a device string dictionary that persists
// across batches. Wider keys (three to eight columns, or two whose widths add
// up to more than 64 bits) are written as fixed-width records of their
// values (utf8 columns by their codes) and mapped to dense int32 codes by the
// same dictionary over the records, and the table groups by that code; the
// key columns are recovered from the records at finalisation. The all-ones
// word marks an empty slot, so the one key that packs to all-ones gets a
// dedicated extra slot at index `capacity`.
//
// Aggregation: each CTA first folds its rows into a shared-memory table
// (64-bit atomicCAS on keys, accumulators as pairs of native 32-bit atomics)
// and merges the table into the global open-addressing table once at the
// end, so low-cardinality group-bys (a handful to a few thousand groups) cost
// one global atomic per group per CTA rather than per row. Rows whose key
// does not fit the shared table collect in a per-warp queue and go to the
// global table 32 at a time. New groups are counted per CTA in shared memory
// and added to the table's count once per CTA. Integer sums are 64-bit
// two's-complement additions, which are associative and commutative, so
// results are bit-exact whatever order the atomics land in.
//
// Table size: at most half full for an upper bound on the groups (groups so
// far plus the batch's rows). A large batch whose rows are known on the host
// is first counted with a HyperLogLog sketch of its keys, and the table is
// sized for that estimate instead: a batch of 20M rows over 1.8M distinct
// keys gets 4M slots (96 MB with two accumulators) rather than 64M (1.5 GB)
// to fill and to scan at finalisation.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "eval.cuh"
#include "launch.h"

namespace gfpdb {

namespace {

constexpr int kGroupThreads = 256;
constexpr int kGroupSmemSlotsMax = 1024;  // slots of a CTA's shared-memory table
constexpr int kGroupQueue = 64;           // rows of a warp waiting for the global table (two rounds of 32)
// group_update_plain_kernel's table takes in a key on its second sight: a bit
// per hash value remembers the first. Keys seen once would otherwise fill the
// table before the frequent ones have all come by.
constexpr int kGroupSeenBits = 1 << 16;
constexpr int kGroupSmemProbes = 4;       // shared-memory slots a row tries before the global table
constexpr uint32_t kDictSpinLimit = 1u << 20;

struct AccDev {
  int8_t fn;  // AGG_SUM / AGG_COUNT / AGG_MIN / AGG_MAX / AGG_COUNT_STAR
  int8_t vt;
  int16_t pad;
  int32_t pad2;
  Operand in;
};

struct GroupParams {
  int64_t n_rows;          // exact, or the capacity when n_dev is set
  const int64_t* n_dev;    // device row count of a deferred batch
  int32_t n_keys;
  int32_t n_acc;
  int32_t key_bits[2];
  DevCol key_cols[2];
  AccDev acc[kMaxAggs];
  DevCol cols[kMaxCols];
  uint64_t* keys;             // slot i's key at keys[i * key_stride], its accumulators from accs[i * acc_stride]
  unsigned long long* accs;
  uint64_t mask;
  int32_t key_stride, acc_stride;
  int32_t sm_slots;
  int32_t float_sums;         // a float64 sum is among the accumulators
  DevStatus* st;  // aux[0]: groups claimed, aux[1]: special slot used
  Program prog;
};

// A batch's columns are read once: streaming loads (evict-first) leave the
// L2 to the table, which every row revisits.
__device__ __forceinline__ int64_t load_int_stream(const DevCol& c, int64_t row) {
  if (c.type == CT_I64) return __ldcs(static_cast<const long long*>(c.data) + row);
  return __ldcs(static_cast<const int*>(c.data) + row);
}

__device__ __forceinline__ uint64_t pack_key(const GroupParams& p, int64_t row) {
  if (p.n_keys == 0) return 0;  // a non-grouped aggregate: one group
  if (p.n_keys == 1) {
    const int64_t v = load_int_stream(p.key_cols[0], row);
    return p.key_bits[0] == 64 ? static_cast<uint64_t>(v) : static_cast<uint64_t>(static_cast<uint32_t>(v));
  }
  const uint32_t a = static_cast<uint32_t>(load_int_stream(p.key_cols[0], row));
  const uint32_t b = static_cast<uint32_t>(load_int_stream(p.key_cols[1], row));
  return (static_cast<uint64_t>(a) << 32) | b;
}

// Identity of each accumulator: 0 for sums and counts, +inf / INT64_MAX for
// MIN, -inf / INT64_MIN for MAX (as bit patterns).
__host__ __device__ __forceinline__ unsigned long long acc_identity(int fn, int vt) {
  if (fn == AGG_MIN) return vt == VT_F64 ? 0x7ff0000000000000ull : static_cast<unsigned long long>(INT64_MAX);
  if (fn == AGG_MAX) return vt == VT_F64 ? 0xfff0000000000000ull : static_cast<unsigned long long>(INT64_MIN);
  return 0ull;
}

__device__ __forceinline__ void acc_combine(unsigned long long* addr, int fn, int vt, unsigned long long v) {
  switch (fn) {
    case AGG_SUM:
      if (vt == VT_F64) atomicAdd(reinterpret_cast<double*>(addr), __longlong_as_double(static_cast<long long>(v)));
      else atomicAdd(addr, v);
      break;
    case AGG_COUNT:
    case AGG_COUNT_STAR: atomicAdd(addr, v); break;
    case AGG_MIN:
    case AGG_MAX: {
      if (vt == VT_F64) {
        const double x = __longlong_as_double(static_cast<long long>(v));
        unsigned long long old = *reinterpret_cast<volatile unsigned long long*>(addr);
        for (;;) {
          const double cur = __longlong_as_double(static_cast<long long>(old));
          const bool better = fn == AGG_MIN ? x < cur : x > cur;
          if (!better) break;
          const unsigned long long prev = atomicCAS(addr, old, v);
          if (prev == old) break;
          old = prev;
        }
      } else if (fn == AGG_MIN) {
        atomicMin(reinterpret_cast<long long*>(addr), static_cast<long long>(v));
      } else {
        atomicMax(reinterpret_cast<long long*>(addr), static_cast<long long>(v));
      }
      break;
    }
  }
}

// acc_combine on a shared-memory accumulator. 64-bit atomics there are
// compare-and-swap loops, which rows of one key on many lanes drag through
// round after round; 32-bit additions are native. A 64-bit sum is its low
// half's additions, each passing its carry on (the old value tells), and its
// high half's: together the same two's-complement sum. A minimum or maximum
// that does not improve on the value read needs no atomic (it only ever
// moves one way).
__device__ __forceinline__ void smem_combine(unsigned long long* addr, int fn, int vt, unsigned long long v) {
  if (fn == AGG_COUNT || fn == AGG_COUNT_STAR) {
    atomicAdd(reinterpret_cast<unsigned*>(addr), 1u);  // a CTA counts fewer than 2^31 rows: no carry
  } else if (fn == AGG_SUM && vt != VT_F64) {
    unsigned* w = reinterpret_cast<unsigned*>(addr);
    const unsigned lo = static_cast<unsigned>(v);
    const unsigned old = atomicAdd(w, lo);
    const unsigned hi = static_cast<unsigned>(v >> 32) + (old + lo < lo ? 1u : 0u);
    if (hi != 0) atomicAdd(w + 1, hi);
  } else if (fn != AGG_SUM && vt != VT_F64) {
    const long long cur = *reinterpret_cast<volatile long long*>(addr), x = static_cast<long long>(v);
    if (fn == AGG_MIN ? x < cur : x > cur) acc_combine(addr, fn, vt, v);
  } else {
    acc_combine(addr, fn, vt, v);
  }
}

// Global slot of a key that is not the all-ones word, continuing from its
// home slot `slot` whose content `s` the caller has already read; claims an
// empty slot for a new key. Returns UINT64_MAX (and raises GFPDB_ENOMEM) if
// the table is full.
__device__ __forceinline__ uint64_t global_slot_from(const GroupParams& p, uint64_t key, uint64_t slot, uint64_t s,
                                                     unsigned* claims) {
  for (uint64_t i = 0; i <= p.mask; ++i) {
    if (i > 0) s = *reinterpret_cast<volatile uint64_t*>(p.keys + slot * p.key_stride);
    if (s == kEmptySlot) {
      s = atomicCAS(reinterpret_cast<unsigned long long*>(p.keys + slot * p.key_stride), static_cast<unsigned long long>(kEmptySlot),
                    static_cast<unsigned long long>(key));
      if (s == kEmptySlot) {
        atomicAdd(claims, 1u);
        return slot;
      }
    }
    if (s == key) return slot;
    slot = (slot + 1) & p.mask;
  }
  raise_status(p.st, GFPDB_ENOMEM, 20);
  return UINT64_MAX;
}

// The all-ones key has its own slot at index capacity.
__device__ __forceinline__ uint64_t special_slot(const GroupParams& p) {
  if (atomicExch(reinterpret_cast<unsigned long long*>(&p.st->aux[1]), 1ull) == 0ull)
    atomicAdd(reinterpret_cast<unsigned long long*>(&p.st->aux[0]), 1ull);
  return p.mask + 1;
}

// `claims` counts the groups this call creates: a CTA's shared-memory
// counter, added to the table's count once per CTA (one global address
// taking an atomic per new group would serialise the L2 on it).
__device__ __forceinline__ uint64_t global_slot(const GroupParams& p, uint64_t key, unsigned* claims) {
  if (key == kEmptySlot) return special_slot(p);
  const uint64_t slot = hash_key(static_cast<int64_t>(key)) & p.mask;
  return global_slot_from(p, key, slot, *reinterpret_cast<volatile uint64_t*>(p.keys + slot * p.key_stride), claims);
}

// The value of an aggregate's input that is no plain column (out of line: the
// update's loads of four aggregates would otherwise carry four interpreters).
__device__ __noinline__ unsigned long long program_value(const GroupParams& p, const AccDev& a, int64_t row) {
  return static_cast<unsigned long long>(operand_row(p.prog, p.cols, a.in, row, p.st));
}

__device__ __forceinline__ unsigned long long row_value(const GroupParams& p, const AccDev& a, int64_t row) {
  if (a.fn == AGG_COUNT || a.fn == AGG_COUNT_STAR) return 1ull;
  if (a.in.kind == OPND_COL) {  // a plain column (float64 as its bits), streamed
    const DevCol& c = p.cols[a.in.col];
    if (c.type == CT_I64 || c.type == CT_F64)
      return static_cast<unsigned long long>(__ldcs(static_cast<const long long*>(c.data) + row));
    return static_cast<unsigned long long>(static_cast<int64_t>(__ldcs(static_cast<const int*>(c.data) + row)));
  }
  return program_value(p, a, row);
}

// A row into the global table; the first values are asked for before the slot.
template <int A>
__device__ __forceinline__ void add_global(const GroupParams& p, uint64_t key, int64_t row, unsigned* claims) {
  uint64_t g = UINT64_MAX;
  if constexpr (A == 0) {
    global_slot(p, key, claims);
  } else if constexpr (A == 1) {
    const unsigned long long v = row_value(p, p.acc[0], row);
    g = global_slot(p, key, claims);
    if (g != UINT64_MAX) acc_combine(p.accs + g * p.acc_stride, p.acc[0].fn, p.acc[0].vt, v);
  } else {
    for (int a0 = 0; a0 < p.n_acc; a0 += 4) {
      unsigned long long v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = a0 + u < p.n_acc ? row_value(p, p.acc[a0 + u], row) : 0ull;
      if (a0 == 0) {
        g = global_slot(p, key, claims);
        if (g == UINT64_MAX) break;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (a0 + u < p.n_acc)
          acc_combine(p.accs + g * p.acc_stride + a0 + u, p.acc[a0 + u].fn, p.acc[a0 + u].vt, v[u]);
    }
  }
}

// Bytes of a CTA's dynamic shared memory: the table and the warps' queues.
constexpr int64_t group_smem(int64_t slots, int n_acc) {
  return slots * (8 + 8 * n_acc) + kGroupThreads / 32 * kGroupQueue * 12;
}

// Every row straight to the global table (the caller expects many groups).
// Bound by the latency of its atomics, so registers count: 40 to 48 of them,
// five to six CTAs an SM. With the first four values loaded before the slot is
// looked up (62 registers) 4M rows of 200k keys took 17 us more (175, call).
template <int A>
__global__ void __launch_bounds__(kGroupThreads) group_update_global_kernel(const __grid_constant__ GroupParams p) {
  __shared__ unsigned s_claims;
  const int64_t n_rows = clamp_rows(p.n_dev, p.n_rows);
  const int64_t first = static_cast<int64_t>(blockIdx.x) * kGroupThreads;
  if (first >= n_rows) return;
  if (threadIdx.x == 0) s_claims = 0;
  __syncthreads();
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kGroupThreads;
  for (int64_t r = first + threadIdx.x; r < n_rows; r += stride) {
    const uint64_t g = global_slot(p, pack_key(p, r), &s_claims);
    if (A == 0 || g == UINT64_MAX) continue;
    for (int a = 0; a < (A < 2 ? A : p.n_acc); ++a)
      acc_combine(p.accs + g * p.acc_stride + a, p.acc[a].fn, p.acc[a].vt, row_value(p, p.acc[a], r));
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_claims != 0)
    atomicAdd(reinterpret_cast<unsigned long long*>(&p.st->aux[0]), static_cast<unsigned long long>(s_claims));
}

// Any accumulators, any batch; large exact batches of plain aggregates take
// group_update_plain_kernel. A: the accumulators, 2 for any number. Issue and
// the latency of shared-memory atomics hold it, so five CTAs an SM, which 48
// registers allow: with the next key loaded a step ahead (63 registers, four
// CTAs) 20M rows of 100 keys took 572 us instead of 533 for a computed sum and
// a count, 645 instead of 586 for six aggregates. One accumulator's value and
// the next key are loaded ahead all the same (100 keys 331 us, 351 without).
// One CTA of 1,024 threads an SM with a table of most of its shared memory,
// tried for batches of 2M rows and more, took 31 ms instead of 8 for 20M rows
// of a float64 sum: one address for all of an SM's rows.
template <int A>
__global__ void __launch_bounds__(kGroupThreads, 5) group_update_kernel(const __grid_constant__ GroupParams p) {
  constexpr int NT = kGroupThreads;
  constexpr bool kAhead = A == 1;
  extern __shared__ unsigned long long s_mem[];
  __shared__ int s_scan[NT / 32 + 1];
  __shared__ unsigned s_claims;
  const int S = p.sm_slots;  // a power of two
  const int n_acc = A < 2 ? A : p.n_acc;
  uint64_t* s_keys = reinterpret_cast<uint64_t*>(s_mem);
  unsigned long long* s_acc = s_mem + S;  // [accumulator][slot]
  uint64_t* s_qkey = reinterpret_cast<uint64_t*>(s_acc + static_cast<int64_t>(S) * n_acc);
  int32_t* s_qrow = reinterpret_cast<int32_t*>(s_qkey + (NT / 32) * kGroupQueue);
  const int64_t n_rows = clamp_rows(p.n_dev, p.n_rows);
  // A grid sized for a capacity can be far larger than the rows that arrive:
  // CTAs without rows leave before touching shared memory (uniform per CTA).
  if (static_cast<int64_t>(blockIdx.x) * NT >= n_rows) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_claims = 0;
  for (int i = threadIdx.x; i < S; i += NT) s_keys[i] = kEmptySlot;
  for (int a = 0; a < n_acc; ++a) {
    const unsigned long long v = acc_identity(p.acc[a].fn, p.acc[a].vt);
    for (int i = threadIdx.x; i < S; i += NT) s_acc[a * S + i] = v;
  }
  __syncthreads();
  // the warp's rows waiting for the global table, a ring of kGroupQueue; the
  // first n (at most 32) go into it together, one per lane
  uint64_t* q_key = s_qkey + warp * kGroupQueue;
  int32_t* q_row = s_qrow + warp * kGroupQueue;
  unsigned head = 0, tail = 0;  // the same in every lane
  auto drain = [&](int n) {
    if (lane < n) {
      const unsigned e = (head + lane) & (kGroupQueue - 1);
      add_global<A>(p, q_key[e], q_row[e], &s_claims);
    }
    __syncwarp();
    head += n;
  };
  const int64_t stride = static_cast<int64_t>(gridDim.x) * NT;
  int64_t base = static_cast<int64_t>(blockIdx.x) * NT + warp * 32;
  uint64_t next = kAhead && base + lane < n_rows ? pack_key(p, base + lane) : 0;
  for (; base < n_rows; base += stride) {
    const int64_t r = base + lane;
    const uint64_t key = kAhead ? next : r < n_rows ? pack_key(p, r) : 0;
    if (kAhead && r + stride < n_rows) next = pack_key(p, r + stride);
    const unsigned long long v0 = kAhead && r < n_rows ? row_value(p, p.acc[0], r) : 0ull;
    int found = -1;
    if (r < n_rows && key != kEmptySlot) {
      // A short probe run: with few groups the table is sparse and a key is
      // found or placed in a step or two; with many groups (high-cardinality
      // keys) the table is soon full and a longer run only delays the row's
      // trip to the global table.
      int slot = static_cast<int>(hash_key(static_cast<int64_t>(key))) & (S - 1);
      for (int i = 0; i < kGroupSmemProbes; ++i) {
        uint64_t k = *reinterpret_cast<volatile uint64_t*>(s_keys + slot);
        if (k == kEmptySlot) {
          k = atomicCAS(reinterpret_cast<unsigned long long*>(s_keys + slot),
                        static_cast<unsigned long long>(kEmptySlot), static_cast<unsigned long long>(key));
          if (k == kEmptySlot) k = key;
        }
        if (k == key) {
          found = slot;
          break;
        }
        slot = (slot + 1) & (S - 1);
      }
    }
    // The warp's rows all go to one slot: their float64 sum is added up in
    // registers. A double has no native shared-memory addition, and 32 lanes'
    // compare-and-swap loops on one address go round 32 times (a float64 sum
    // without keys over 20M rows: 790 us, 8,600 with a loop a row).
    int same = 0;
    if (A > 0 && p.float_sums && __all_sync(0xffffffffu, found >= 0)) __match_all_sync(0xffffffffu, found, &same);
    if (found >= 0) {
      auto combine = [&](int a, unsigned long long v) {
        unsigned long long* to = s_acc + a * S + found;
        if (same && p.acc[a].fn == AGG_SUM && p.acc[a].vt == VT_F64) {
          double x = __longlong_as_double(static_cast<long long>(v));
#pragma unroll
          for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
          if (lane == 0) atomicAdd(reinterpret_cast<double*>(to), x);
        } else {
          smem_combine(to, p.acc[a].fn, p.acc[a].vt, v);
        }
      };
      if (A == 1) combine(0, v0);
      else for (int a = 0; a < n_acc; ++a) combine(a, row_value(p, p.acc[a], r));
    }
    const unsigned m = __ballot_sync(0xffffffffu, r < n_rows && found < 0);
    if (m != 0) {
      if (m >> lane & 1u) {
        const unsigned e = (tail + __popc(m & ((1u << lane) - 1u))) & (kGroupQueue - 1);
        q_key[e] = key;
        q_row[e] = static_cast<int32_t>(r);
      }
      tail += __popc(m);
      __syncwarp();
      if (tail - head >= 32) drain(32);
    }
  }
  if (tail != head) drain(static_cast<int>(tail - head));
  __syncthreads();
  // Merge into the global table: the occupied slots are listed first (a
  // block scan), so each thread merges about one group, and every group's
  // global insert and atomics run in the same round instead of one after
  // another on the threads that hold several.
  int c = 0;
  for (int i = threadIdx.x; i < S; i += NT) c += s_keys[i] != kEmptySlot ? 1 : 0;
  uint16_t* s_occ = reinterpret_cast<uint16_t*>(s_qkey);  // the queues are empty: at most kGroupSmemSlotsMax entries
  int occupied;
  int o = block_exclusive_sum<NT>(c, &occupied, s_scan);
  for (int i = threadIdx.x; i < S; i += NT)
    if (s_keys[i] != kEmptySlot) s_occ[o++] = static_cast<uint16_t>(i);
  __syncthreads();
  for (int j = threadIdx.x; j < occupied; j += NT) {
    const int i = s_occ[j];
    const uint64_t g = global_slot(p, s_keys[i], &s_claims);
    if (g == UINT64_MAX) continue;
    for (int a = 0; a < n_acc; ++a)
      acc_combine(p.accs + g * p.acc_stride + a, p.acc[a].fn, p.acc[a].vt, s_acc[a * S + i]);
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_claims != 0)
    atomicAdd(reinterpret_cast<unsigned long long*>(&p.st->aux[0]), static_cast<unsigned long long>(s_claims));
}

// Exact batches of kGroupPlainRows rows and more whose aggregates are counts
// and sums, minima or maxima of plain integer columns. Bound by issue and by
// the lanes that wait: the code is straight where the kernel above interprets
// each accumulator of each row (373 instructions per 32 rows here), two rows
// of a lane are in flight, and rows that miss the shared table queue up until
// they fill two rounds of a warp. 1024 threads with two rows each: 512 with
// four took 1.6 times as long, 768 with two or three 1.25 times. SUM, COUNT
// and MAX, the whole call, against the kernel above: 20M rows of 1000 keys 348
// against 568 us, of Zipf(1.1) keys over 10M values 605 against 811; 1M rows
// of 10, 1000, 20k and 500k keys 104 to 152 against 125 to 201, 250k rows 87 to
// 124 against 91 to 146, 100k rows the same both ways, so batches from about
// 200k rows on take it. A row reads its set's four one-byte tags and then one
// key: with the four keys read instead the random 16-byte reads' bank
// conflicts cost 20M rows of 1000 keys 35 us more.
struct PlainAcc {
  const void* col;   // null: a count
  int32_t wide;      // int64 column
  int32_t at;        // the accumulator's place in a slot
  int64_t flip;      // -1 for a minimum, which is kept as the maximum of ~x
};

constexpr int64_t kGroupPlainRows = 3 << 16;
constexpr int kPlainAccs = 4;
constexpr int kPlainThreads = 1024;
constexpr int kPlainRows = 2;  // rows of a lane in flight
constexpr int kPlainQueue = 2 * 32 * kPlainRows;  // a warp's rows waiting for the global table
constexpr int kPlainWays = 4;  // neighbouring slots of the shared table that a key can go into

struct PlainParams {
  const void* key[2];
  int32_t n_keys;
  int32_t wide_key;          // one int64 key
  uint32_t n;                // rows
  int32_t n_add;             // sums and counts
  PlainAcc acc[kPlainAccs];  // the sums and counts, then the others
};

constexpr int64_t plain_smem(int64_t slots, int n_acc) {
  return slots * (8 + 8 * n_acc + 1) + kGroupSeenBits / 8 + kPlainThreads / 32 * kPlainQueue * 12;
}

__device__ __forceinline__ void red_add(unsigned long long* at, unsigned long long v) {
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(at), "l"(v) : "memory");
}

// Adds x and y to accumulators atx and aty of every lane's slot (null: none).
// Two lanes take a slot's two sums, so that both reach the L2 in one request:
// 190 G rows/s of random slots, as with one sum, against 100 with a lane
// sending one after the other.
__device__ __forceinline__ void add_pair(unsigned long long* acc, int atx, unsigned long long x, int aty,
                                         unsigned long long y, int lane) {
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int src = r * 16 + (lane >> 1);
    auto* a = reinterpret_cast<unsigned long long*>(
        __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(acc), src));
    const unsigned long long vx = __shfl_sync(0xffffffffu, x, src), vy = __shfl_sync(0xffffffffu, y, src);
    if (a != nullptr) red_add(a + (lane & 1 ? aty : atx), lane & 1 ? vy : vx);
  }
  __syncwarp();
}

// A warp's rows (those that are live) into the global table: key[u] with
// values v[u][a], minima and maxima as maxima of v ^ flip. kBeside: a slot is
// its key and three accumulators, 32 bytes read in one load.
template <int A, bool kBeside>
__device__ __forceinline__ void plain_global(const GroupParams& p, const PlainParams& pp,
                                             const uint64_t (&key)[kPlainRows], const uint64_t (&h)[kPlainRows],
                                             const unsigned long long (&v)[kPlainRows][A],
                                             const bool (&live)[kPlainRows], int lane, unsigned* claims) {
  uint64_t slot[kPlainRows][4];
  uint64_t g[kPlainRows];
  bool pend[kPlainRows], home[kPlainRows];
  auto stride = [&] { return static_cast<uint64_t>(kBeside ? 4 : p.key_stride); };
#pragma unroll
  for (int u = 0; u < kPlainRows; ++u) {
    g[u] = h[u] & p.mask;
    if (live[u]) {
      const uint64_t* at = p.keys + g[u] * stride();
      if (kBeside)
        asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                     : "=l"(slot[u][0]), "=l"(slot[u][1]), "=l"(slot[u][2]), "=l"(slot[u][3])
                     : "l"(at)
                     : "memory");
      else
        slot[u][0] = *reinterpret_cast<const volatile uint64_t*>(at);
    }
  }
  __syncwarp();
  bool any = false;
#pragma unroll
  for (int u = 0; u < kPlainRows; ++u) {
    home[u] = live[u] && slot[u][0] == key[u] && key[u] != kEmptySlot;
    pend[u] = live[u] && !home[u];
    if (pend[u] && key[u] == kEmptySlot) {
      g[u] = special_slot(p);
      pend[u] = false;
    }
    any = any || pend[u];
  }
  // New keys and keys that are not in their home slot: all of the warp's go on
  // together, a claim or a step to the next slot at a time.
  for (uint64_t i = 0; __any_sync(0xffffffffu, any); ++i) {
    uint64_t old[kPlainRows];
#pragma unroll
    for (int u = 0; u < kPlainRows; ++u) {
      old[u] = pend[u] ? slot[u][0] : 0;
      if (pend[u] && old[u] == kEmptySlot)
        old[u] = atomicCAS(reinterpret_cast<unsigned long long*>(p.keys + g[u] * stride()),
                           static_cast<unsigned long long>(kEmptySlot), static_cast<unsigned long long>(key[u]));
    }
    any = false;
#pragma unroll
    for (int u = 0; u < kPlainRows; ++u) {
      if (!pend[u]) continue;
      if (old[u] == kEmptySlot) atomicAdd(claims, 1u);
      pend[u] = old[u] != kEmptySlot && old[u] != key[u];
      if (pend[u] && i == p.mask) {
        raise_status(p.st, GFPDB_ENOMEM, 20);  // the table is full
        pend[u] = false;
        g[u] = UINT64_MAX;
      }
      if (pend[u]) {
        g[u] = (g[u] + 1) & p.mask;
        slot[u][0] = *reinterpret_cast<const volatile uint64_t*>(p.keys + g[u] * stride());
        any = true;
      }
    }
  }
#pragma unroll
  for (int u = 0; u < kPlainRows; ++u) {
    if (!__any_sync(0xffffffffu, live[u])) continue;
    unsigned long long* acc =
        live[u] && g[u] != UINT64_MAX ? p.accs + g[u] * (kBeside ? 4 : p.acc_stride) : nullptr;
    if constexpr (A >= 2)
      if (pp.n_add >= 2) add_pair(acc, pp.acc[0].at, v[u][0], pp.acc[1].at, v[u][1], lane);
    if constexpr (A >= 4)
      if (pp.n_add >= 4) add_pair(acc, pp.acc[2].at, v[u][2], pp.acc[3].at, v[u][3], lane);
    if (acc != nullptr) {
      if (pp.n_add == 1) red_add(acc + pp.acc[0].at, v[u][0]);
      if constexpr (A >= 3)
        if (pp.n_add == 3) red_add(acc + pp.acc[2].at, v[u][2]);
#pragma unroll
      for (int a = 0; a < A; ++a) {
        if (a < pp.n_add) continue;
        const int at = pp.acc[a].at;
        const long long flip = pp.acc[a].flip;
        const long long x = static_cast<long long>(v[u][a]);
        if (kBeside && home[u]) {  // an extremum moves one way only: what is no better than an older one needs no atomic
          const long long cur = static_cast<long long>(at == 0 ? slot[u][1] : at == 1 ? slot[u][2] : slot[u][3]);
          if (x <= (cur ^ flip)) continue;
        }
        if (flip) asm volatile("red.relaxed.gpu.global.min.s64 [%0], %1;" ::"l"(acc + at), "l"(~x) : "memory");
        else asm volatile("red.relaxed.gpu.global.max.s64 [%0], %1;" ::"l"(acc + at), "l"(x) : "memory");
      }
    }
    __syncwarp();
  }
}

template <int A, bool kBeside>
__global__ void __launch_bounds__(kPlainThreads) group_update_plain_kernel(const __grid_constant__ GroupParams p,
                                                                               const __grid_constant__ PlainParams pp) {
  constexpr int U = kPlainRows;
  extern __shared__ __align__(16) unsigned long long s_mem[];
  __shared__ unsigned s_claims;
  const int S = p.sm_slots;  // a multiple of kPlainWays
  uint64_t* s_keys = reinterpret_cast<uint64_t*>(s_mem);
  unsigned long long* s_acc = s_mem + S;  // [accumulator][slot]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t* q_key = reinterpret_cast<uint64_t*>(s_acc) + static_cast<int64_t>(S) * A;
  uint32_t* q_row = reinterpret_cast<uint32_t*>(q_key + kPlainThreads / 32 * kPlainQueue);
  unsigned* s_seen = q_row + kPlainThreads / 32 * kPlainQueue;
  uint32_t* s_tags = s_seen + kGroupSeenBits / 32;  // a byte per slot, 0 while it is empty
  q_key += warp * kPlainQueue;
  q_row += warp * kPlainQueue;
  unsigned head = 0, tail = 0;  // the same in every lane
  if (threadIdx.x == 0) s_claims = 0;
  for (int i = threadIdx.x; i < S; i += kPlainThreads) {
    s_keys[i] = kEmptySlot;
#pragma unroll
    for (int a = 0; a < A; ++a) s_acc[a * S + i] = a < pp.n_add ? 0ull : static_cast<unsigned long long>(INT64_MIN);
  }
  for (int i = threadIdx.x; i < kGroupSeenBits / 32; i += kPlainThreads) s_seen[i] = 0;
  for (int i = threadIdx.x; i < S / kPlainWays; i += kPlainThreads) s_tags[i] = 0;
  __syncthreads();

  // Rows past the end stand for the last row and are not live: every load is
  // in range without a test of its own.
  const uint32_t last = pp.n - 1;
  auto load_keys = [&](uint32_t r0, uint64_t (&k)[U]) {
    if (pp.n_keys == 1 && pp.wide_key) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        k[u] = static_cast<uint64_t>(__ldcs(static_cast<const long long*>(pp.key[0]) + min(r0 + 32 * u, last)));
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        k[u] = 0;
        if (pp.n_keys > 0) k[u] = static_cast<uint32_t>(__ldcs(static_cast<const int*>(pp.key[0]) + min(r0 + 32 * u, last)));
        if (pp.n_keys > 1)
          k[u] = k[u] << 32 | static_cast<uint32_t>(__ldcs(static_cast<const int*>(pp.key[1]) + min(r0 + 32 * u, last)));
      }
    }
  };
  const uint32_t stride = gridDim.x * (kPlainThreads * U);
  uint32_t base = (blockIdx.x * (kPlainThreads / 32) + warp) * (32 * U);
  uint64_t next[U];
  load_keys(base + lane, next);
  auto load_values = [&](const uint32_t (&r)[U], unsigned long long (&v)[U][A]) {
#pragma unroll
    for (int a = 0; a < A; ++a) {
      const PlainAcc& d = pp.acc[a];
      if (d.col == nullptr) {
#pragma unroll
        for (int u = 0; u < U; ++u) v[u][a] = 1ull;
      } else if (d.wide) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          v[u][a] = static_cast<unsigned long long>(__ldcs(static_cast<const long long*>(d.col) + r[u])) ^
                    static_cast<unsigned long long>(d.flip);
      } else {
#pragma unroll
        for (int u = 0; u < U; ++u)
          v[u][a] = static_cast<unsigned long long>(static_cast<long long>(__ldcs(static_cast<const int*>(d.col) + r[u]))) ^
                    static_cast<unsigned long long>(d.flip);
      }
    }
  };
  for (;;) {
    uint64_t key[U];
    uint32_t row[U];
    unsigned long long v[U][A];
    uint64_t h[U];
    if (tail - head >= 32 * U || base >= pp.n) {
      // Waiting rows, a full warp of them: only about a quarter of a step's
      // rows miss the shared table, and they would go through the global
      // table's round trips at that share of a warp.
      if (tail == head) break;
      bool live[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned e = head + lane + 32 * u;
        live[u] = e - head < tail - head;
        key[u] = q_key[e & (kPlainQueue - 1)];
        row[u] = live[u] ? q_row[e & (kPlainQueue - 1)] : last;
        h[u] = hash_key(static_cast<int64_t>(key[u]));
      }
      head += tail - head < 32 * U ? tail - head : 32 * U;
      load_values(row, v);
      plain_global<A, kBeside>(p, pp, key, h, v, live, lane, &s_claims);
      continue;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      key[u] = next[u];
      row[u] = min(base + lane + 32 * u, last);
    }
    load_values(row, v);
    load_keys(base + stride + lane, next);  // a step ahead of their use
    int found[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      h[u] = hash_key(static_cast<int64_t>(key[u]));
      const bool is_row = base + lane + 32 * u < pp.n;
      const int set = static_cast<int>(__umulhi(static_cast<unsigned>(h[u] >> 32), static_cast<unsigned>(S / kPlainWays)));
      const int at = kPlainWays * set;
      const uint32_t tag = (static_cast<uint32_t>(h[u]) >> 24) | 1u;  // not a bit of the seen bits' index
      const uint32_t tags = *reinterpret_cast<const volatile uint32_t*>(s_tags + set);
      const uint32_t same = __vcmpeq4(tags, tag * 0x01010101u);
      const bool can = is_row && key[u] != kEmptySlot;
      int way = -1;
      if (can && same != 0) {
        way = (__ffs(static_cast<int>(same)) - 1) >> 3;
        if (*reinterpret_cast<const volatile uint64_t*>(s_keys + at + way) != key[u]) {  // another key's tag
          way = -1;
          for (int j = 0; j < kPlainWays; ++j)
            if (*reinterpret_cast<const volatile uint64_t*>(s_keys + at + j) == key[u]) way = j;
        }
      }
      if (can && way < 0 && (tags >> 24) == 0) {  // slots fill in order: the last one is empty while any is
        const unsigned bit = static_cast<unsigned>(h[u]) & (kGroupSeenBits - 1);
        if (atomicOr(s_seen + (bit >> 5), 1u << (bit & 31)) >> (bit & 31) & 1u)  // not its first sight
          for (int j = 0; j < kPlainWays && way < 0; ++j) {
            const unsigned long long old = atomicCAS(reinterpret_cast<unsigned long long*>(s_keys + at + j),
                                                     static_cast<unsigned long long>(kEmptySlot),
                                                     static_cast<unsigned long long>(key[u]));
            if (old == kEmptySlot) reinterpret_cast<uint8_t*>(s_tags)[at + j] = static_cast<uint8_t>(tag);
            if (old == kEmptySlot || old == key[u]) way = j;
          }
      }
      __syncwarp();
      found[u] = way < 0 ? -1 : at + way;
      const bool miss = is_row && way < 0;
      const unsigned m = __ballot_sync(0xffffffffu, miss);
      if (miss) {
        const unsigned e = (tail + __popc(m & ((1u << lane) - 1u))) & (kPlainQueue - 1);
        q_key[e] = key[u];
        q_row[e] = row[u];
      }
      tail += __popc(m);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (found[u] >= 0) {
#pragma unroll
        for (int a = 0; a < A; ++a) {
          unsigned long long* to = s_acc + a * S + found[u];
          if (a < pp.n_add) {
            smem_combine(to, AGG_SUM, VT_I64, v[u][a]);
          } else if (static_cast<long long>(v[u][a]) > *reinterpret_cast<volatile long long*>(to)) {
            atomicMax(reinterpret_cast<long long*>(to), static_cast<long long>(v[u][a]));
          }
        }
      }
      __syncwarp();
    }
    base += stride;
  }
  __syncthreads();
  // the shared table's groups
  for (int i0 = warp * (32 * U); i0 < S; i0 += kPlainThreads * U) {
    uint64_t key[U], h[U];
    unsigned long long v[U][A];
    bool live[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = min(i0 + lane + 32 * u, S - 1);
      key[u] = s_keys[i];
      live[u] = i0 + lane + 32 * u < S && key[u] != kEmptySlot;
      h[u] = hash_key(static_cast<int64_t>(key[u]));
#pragma unroll
      for (int a = 0; a < A; ++a) v[u][a] = s_acc[a * S + i];
    }
    plain_global<A, kBeside>(p, pp, key, h, v, live, lane, &s_claims);
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_claims != 0)
    atomicAdd(reinterpret_cast<unsigned long long*>(&p.st->aux[0]), static_cast<unsigned long long>(s_claims));
}

// HyperLogLog sketch (Flajolet, Fusy, Gandouet, Meunier 2007) of a batch's
// packed keys: 2^12 registers, each the largest leading-zero rank + 1 of
// the hashes that fall in it. Registers gather per CTA in shared memory.
constexpr int kSketchBits = 12;
constexpr int kSketchRegs = 1 << kSketchBits;

__global__ void __launch_bounds__(256) group_sketch_kernel(const __grid_constant__ GroupParams p,
                                                           unsigned* __restrict__ regs) {
  __shared__ unsigned s_regs[kSketchRegs];
  for (int i = threadIdx.x; i < kSketchRegs; i += blockDim.x) s_regs[i] = 0;
  __syncthreads();
  const int64_t n = clamp_rows(p.n_dev, p.n_rows);
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  // four keys in flight per thread (past the end: the last key again, which
  // changes no maximum)
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n; r += 4 * stride) {
    uint64_t key[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) key[u] = pack_key(p, r + u * stride < n ? r + u * stride : n - 1);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      // a hash unrelated to the slot hash (another constant before the mixer)
      const uint64_t h = mix64(key[u] ^ 0xd6e8feb86659fd93ull);
      const unsigned idx = static_cast<unsigned>(h >> (64 - kSketchBits));
      const unsigned rank = static_cast<unsigned>(__clzll((h << kSketchBits) | (1ull << (kSketchBits - 1)))) + 1u;
      if (rank > s_regs[idx]) atomicMax(&s_regs[idx], rank);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kSketchRegs; i += blockDim.x) {
    const unsigned v = s_regs[i];
    if (v > *reinterpret_cast<volatile unsigned*>(regs + i)) atomicMax(regs + i, v);
  }
}

// Fills words [0, n) with a pattern of `period` words, 16 bytes a store: a
// 4M-slot table of 134 MB in 44 us (98 us with a thread storing one slot's
// words one after another).
struct InitPattern {
  unsigned long long word[kMaxAggs + 1];
  int32_t period;
};

__global__ void __launch_bounds__(256) group_init_kernel(unsigned long long* __restrict__ out, uint64_t n,
                                                         const __grid_constant__ InitPattern pat) {
  __shared__ unsigned long long s_word[kMaxAggs + 1];
  if (threadIdx.x < kMaxAggs + 1) s_word[threadIdx.x] = pat.word[threadIdx.x];
  __syncthreads();
  const uint64_t stride = 2 * static_cast<uint64_t>(gridDim.x) * blockDim.x;
  uint64_t i = 2 * (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x);
  unsigned m = static_cast<unsigned>(i % pat.period);
  const unsigned step = static_cast<unsigned>(stride % pat.period);
  for (; i < n; i += stride) {
    const unsigned m1 = m + 1 == static_cast<unsigned>(pat.period) ? 0 : m + 1;
    if (i + 1 < n) *reinterpret_cast<ulonglong2*>(out + i) = make_ulonglong2(s_word[m], s_word[m1]);
    else out[i] = s_word[m];
    m += step;
    if (m >= static_cast<unsigned>(pat.period)) m -= pat.period;
  }
}

// A table's slots: slot i's key at keys[i * key_stride], its accumulators
// from accs[i * acc_stride].
struct TableView {
  uint64_t* keys;
  unsigned long long* accs;
  int32_t key_stride, acc_stride;
};

// Move every group of an old table into a larger one (accumulators copied).
__global__ void group_rehash_kernel(TableView old, uint64_t old_cap, TableView to, uint64_t mask, int n_acc,
                                    DevStatus* st) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i <= old_cap; i += stride) {
    uint64_t dst;
    if (i == old_cap) {
      dst = mask + 1;  // the special slot stays special: its key word is never written, its accumulators move
    } else {
      const uint64_t key = old.keys[i * old.key_stride];
      if (key == kEmptySlot) continue;
      uint64_t slot = hash_key(static_cast<int64_t>(key)) & mask;
      bool ok = false;
      for (uint64_t k = 0; k <= mask; ++k) {
        const unsigned long long prev = atomicCAS(reinterpret_cast<unsigned long long*>(to.keys + slot * to.key_stride),
                                                  static_cast<unsigned long long>(kEmptySlot),
                                                  static_cast<unsigned long long>(key));
        if (prev == kEmptySlot) {
          ok = true;
          break;
        }
        slot = (slot + 1) & mask;
      }
      if (!ok) {
        raise_status(st, GFPDB_ENOMEM, 21);
        continue;
      }
      dst = slot;
    }
    for (int a = 0; a < n_acc; ++a) to.accs[dst * to.acc_stride + a] = old.accs[i * old.acc_stride + a];
  }
}

struct OutAggDev {
  int8_t kind;  // 0: copy accumulator, 1: avg = sum / count
  int8_t out_type;  // DType code of the output column
  int8_t vt;
  int8_t pad;
  int32_t a0, a1;  // accumulator indices
  void* dst;
};

struct FinalParams {
  const uint64_t* keys;  // strides as in GroupParams
  const unsigned long long* accs;
  int32_t key_stride, acc_stride;
  uint64_t cap;  // special slot at index cap
  const int64_t* special_dev;  // non-zero once the all-ones key has a group
  int32_t n_acc;
  int32_t n_keys;
  int32_t n_out;
  int32_t key_bits[2];
  void* key_dst[2];
  int32_t key_type[2];
  OutAggDev outs[kMaxAggs];
  unsigned long long* counter;
};

__device__ __forceinline__ void store_typed(void* dst, int64_t pos, int type, int64_t v) {
  if (type == CT_I64 || type == CT_F64) static_cast<long long*>(dst)[pos] = v;
  else static_cast<int*>(dst)[pos] = static_cast<int32_t>(v);
}

// Each warp lists the live slots of kSteps consecutive 32-slot steps with
// one atomic on the output counter. Large tables take several steps per
// atomic (one address taking an atomic per 32 slots would queue them);
// small ones one step per warp, so that more warps share the few slots.
constexpr uint64_t kFinalChunkedSlots = 1ull << 20;

template <int kSteps>
__global__ void __launch_bounds__(256) group_finalize_kernel(const __grid_constant__ FinalParams p) {
  const int lane = threadIdx.x & 31;
  const uint32_t below = (1u << lane) - 1u;
  const uint64_t n_slots = p.cap + 1;
  const uint64_t warp0 = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const uint64_t n_warps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
  constexpr uint64_t kChunk = 32 * kSteps;
  for (uint64_t base = warp0 * kChunk; base < n_slots; base += n_warps * kChunk) {
    uint64_t key[kSteps];
    uint32_t m[kSteps];
    int total = 0;
#pragma unroll
    for (int k = 0; k < kSteps; ++k) {
      const uint64_t i = base + k * 32 + lane;
      bool live = false;
      key[k] = 0;
      if (i < p.cap) {
        key[k] = p.keys[i * p.key_stride];
        live = key[k] != kEmptySlot;
      } else if (i == p.cap) {
        key[k] = kEmptySlot;
        live = *p.special_dev != 0;
      }
      m[k] = __ballot_sync(0xffffffffu, live);
      total += __popc(m[k]);
    }
    if (total == 0) continue;
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(p.counter, static_cast<unsigned long long>(total));
    at = __shfl_sync(0xffffffffu, at, 0);
    // a column at a time, every step's value loaded before the first is stored
    // (4M slots, 1.8M groups, four columns: 74 us; 142 us a row at a time)
    int64_t pos[kSteps];  // -1: no live slot
#pragma unroll
    for (int k = 0; k < kSteps; ++k) {
      pos[k] = (m[k] >> lane & 1u) ? static_cast<int64_t>(at) + __popc(m[k] & below) : -1;
      at += __popc(m[k]);
    }
    if (p.n_keys == 1) {
#pragma unroll
      for (int k = 0; k < kSteps; ++k)
        if (pos[k] >= 0)
          store_typed(p.key_dst[0], pos[k], p.key_type[0],
                      p.key_bits[0] == 64 ? static_cast<int64_t>(key[k])
                                          : static_cast<int32_t>(static_cast<uint32_t>(key[k])));
    } else if (p.n_keys == 2) {
#pragma unroll
      for (int k = 0; k < kSteps; ++k) {
        if (pos[k] < 0) continue;
        store_typed(p.key_dst[0], pos[k], p.key_type[0], static_cast<int32_t>(static_cast<uint32_t>(key[k] >> 32)));
        store_typed(p.key_dst[1], pos[k], p.key_type[1], static_cast<int32_t>(static_cast<uint32_t>(key[k])));
      }
    }
    const unsigned long long* acc = p.accs + (base + lane) * p.acc_stride;
    const uint64_t step = static_cast<uint64_t>(32) * p.acc_stride;
    for (int j = 0; j < p.n_out; ++j) {
      const OutAggDev& o = p.outs[j];
      unsigned long long a[kSteps];
#pragma unroll
      for (int k = 0; k < kSteps; ++k) a[k] = pos[k] >= 0 ? acc[k * step + o.a0] : 0ull;
      if (o.kind == 0) {
#pragma unroll
        for (int k = 0; k < kSteps; ++k)
          if (pos[k] >= 0) store_typed(o.dst, pos[k], o.out_type, static_cast<int64_t>(a[k]));
      } else {
#pragma unroll
        for (int k = 0; k < kSteps; ++k) {
          if (pos[k] < 0) continue;
          const unsigned long long c = acc[k * step + o.a1];
          const double sum = o.vt == VT_F64 ? __longlong_as_double(static_cast<long long>(a[k]))
                                            : static_cast<double>(static_cast<long long>(a[k]));
          static_cast<double*>(o.dst)[pos[k]] = c == 0 ? 0.0 : sum / static_cast<double>(c);
        }
      }
    }
  }
}

// ------------------------------------------------------- string dictionary

struct DictDev {
  uint64_t* slot_hash;
  uint32_t* slot_code;  // 0 = not published yet, else code + 1
  int64_t* code_off;
  int32_t* code_len;
  uint8_t* heap;
  uint64_t mask;
  int64_t code_cap;
  int64_t heap_cap;
  DevStatus* st;  // aux[0]: codes, aux[1]: heap bytes
};

__device__ __forceinline__ uint64_t dict_hash(const uint8_t* s, int32_t n) {
  uint64_t h = hash_bytes(s, n);
  return h == kEmptySlot ? kEmptySlot - 1 : h;
}

// Values are utf8 strings (offs, bytes) or, with offs null, fixed-width
// records of `width` bytes each.
__global__ void __launch_bounds__(256) dict_encode_kernel(const int32_t* __restrict__ offs, const uint8_t* __restrict__ bytes,
                                                          int32_t width, int64_t n, int32_t* __restrict__ out_codes,
                                                          DictDev d) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n; r += stride) {
    const int64_t b = offs != nullptr ? offs[r] : r * width;
    const int32_t len = offs != nullptr ? offs[r + 1] - static_cast<int32_t>(b) : width;
    const uint8_t* str = bytes + b;
    const uint64_t h = dict_hash(str, len);
    uint64_t slot = h & d.mask;
    int32_t code = -1;
    for (uint64_t i = 0; i <= d.mask && code < 0; ++i, slot = (slot + 1) & d.mask) {
      uint64_t s = *reinterpret_cast<volatile uint64_t*>(d.slot_hash + slot);
      if (s == kEmptySlot) {
        s = atomicCAS(reinterpret_cast<unsigned long long*>(d.slot_hash + slot),
                      static_cast<unsigned long long>(kEmptySlot), static_cast<unsigned long long>(h));
        if (s == kEmptySlot) {
          // This thread owns the new entry: store its bytes, then publish.
          const unsigned long long c = atomicAdd(reinterpret_cast<unsigned long long*>(&d.st->aux[0]), 1ull);
          const unsigned long long off = atomicAdd(reinterpret_cast<unsigned long long*>(&d.st->aux[1]),
                                                   static_cast<unsigned long long>(len));
          if (static_cast<int64_t>(c) >= d.code_cap || static_cast<int64_t>(off) + len > d.heap_cap) {
            raise_status(d.st, GFPDB_ENOMEM, 30);
            st_release32(d.slot_code + slot, 0xFFFFFFFFu);
            break;
          }
          for (int32_t k = 0; k < len; ++k) d.heap[off + k] = str[k];
          d.code_off[c] = static_cast<int64_t>(off);
          d.code_len[c] = len;
          __threadfence();
          st_release32(d.slot_code + slot, static_cast<uint32_t>(c) + 1u);
          code = static_cast<int32_t>(c);
          break;
        }
      }
      if (s != h) continue;
      // Same hash: wait (bounded) until the owner has published, then compare bytes.
      uint32_t pub = 0;
      for (uint32_t spin = 0; spin < kDictSpinLimit; ++spin) {
        pub = ld_acquire32(d.slot_code + slot);
        if (pub != 0) break;
        __nanosleep(32);
      }
      if (pub == 0) {
        raise_status(d.st, GFPDB_ETIMEDOUT, 31);
        break;
      }
      if (pub == 0xFFFFFFFFu) break;  // owner ran out of space; error already raised
      const int32_t c = static_cast<int32_t>(pub - 1u);
      if (d.code_len[c] != len) continue;
      const uint8_t* other = d.heap + d.code_off[c];
      bool eq = true;
      for (int32_t k = 0; eq && k < len; ++k) eq = other[k] == str[k];
      if (eq) code = c;
    }
    if (code < 0) raise_status(d.st, GFPDB_ENOMEM, 32);
    out_codes[r] = code < 0 ? 0 : code;
  }
}

__global__ void dict_rehash_kernel(DictDev d, int64_t n_codes) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; c < n_codes; c += stride) {
    const uint64_t h = dict_hash(d.heap + d.code_off[c], d.code_len[c]);
    uint64_t slot = h & d.mask;
    for (uint64_t i = 0; i <= d.mask; ++i, slot = (slot + 1) & d.mask) {
      const unsigned long long prev = atomicCAS(reinterpret_cast<unsigned long long*>(d.slot_hash + slot),
                                                static_cast<unsigned long long>(kEmptySlot),
                                                static_cast<unsigned long long>(h));
      if (prev == kEmptySlot) {
        d.slot_code[slot] = static_cast<uint32_t>(c) + 1u;
        break;
      }
    }
  }
}

__global__ void dict_lengths_kernel(const int32_t* codes, int64_t n, const int32_t* code_len, int32_t* lens) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n; r += stride)
    lens[r] = code_len[codes[r]];
}

// Key records: each record's values written at fixed offsets (4-byte words;
// an 8-byte value as two), and back into columns.
struct RecordCols {
  DevCol cols[kMaxKeyColumns];
  int32_t off[kMaxKeyColumns];    // byte offset of the column in a record
  int32_t width[kMaxKeyColumns];  // 4 or 8
  int32_t n_cols;
  int32_t rec_width;              // multiple of 4
};

__global__ void group_record_pack_kernel(const __grid_constant__ RecordCols rc, int64_t n, uint32_t* out) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int words = rc.rec_width / 4;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n; r += stride) {
    uint32_t* rec = out + r * words;
    for (int k = 0; k < rc.n_cols; ++k) {
      const int64_t v = load_int(rc.cols[k], r);
      rec[rc.off[k] / 4] = static_cast<uint32_t>(v);
      if (rc.width[k] == 8) rec[rc.off[k] / 4 + 1] = static_cast<uint32_t>(static_cast<uint64_t>(v) >> 32);
    }
  }
}

__global__ void group_record_split_kernel(const __grid_constant__ RecordCols rc, int64_t n, const int32_t* codes,
                                          const int64_t* code_off, const uint8_t* heap, void* const* dst) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n; r += stride) {
    const uint32_t* rec = reinterpret_cast<const uint32_t*>(heap + code_off[codes[r]]);
    for (int k = 0; k < rc.n_cols; ++k) {
      const uint32_t lo = rec[rc.off[k] / 4];
      if (rc.width[k] == 8)
        static_cast<uint64_t*>(dst[k])[r] = (static_cast<uint64_t>(rec[rc.off[k] / 4 + 1]) << 32) | lo;
      else
        static_cast<uint32_t*>(dst[k])[r] = lo;
    }
  }
}

__global__ void dict_copy_kernel(const int32_t* codes, int64_t n, const int64_t* code_off, const uint8_t* heap,
                                 const int32_t* offs, uint8_t* out) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n; r += stride) {
    const uint8_t* src = heap + code_off[codes[r]];
    const int32_t o = offs[r], len = offs[r + 1] - o;
    for (int32_t k = 0; k < len; ++k) out[o + k] = src[k];
  }
}

int grid_for(int64_t n) {
  int64_t blocks = (n + 255) / 256;
  int64_t cap = static_cast<int64_t>(num_sms()) * 8;
  if (blocks > cap) blocks = cap;
  return static_cast<int>(blocks < 1 ? 1 : blocks);
}

// Tables above this many slots (32 MB of keys) are sized by a sketch when
// the batch allows it.
constexpr uint64_t kSketchMinSlots = 1ull << 22;

bool stream_capturing(cudaStream_t s) {
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(s, &c) == cudaSuccess && c != cudaStreamCaptureStatusNone;
}

uint64_t next_pow2(uint64_t x) {
  uint64_t c = 1;
  while (c < x) c <<= 1;
  return c;
}

DevStatus read_status(const DevStatus* d, cudaStream_t s) {
  DevStatus h;
  GF_CUDA(cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, s));
  sync(s);
  return h;
}

// Distinct keys of a batch, estimated from its HyperLogLog sketch (the raw
// estimate alpha_m m^2 / sum 2^-M[j], with linear counting over the empty
// registers in the small range); standard error about 1.04 / sqrt(2^12).
double sketch_distinct(const GroupParams& p, int64_t n, cudaStream_t s) {
  auto regs = make_filled(kSketchRegs * 4, 0, s);
  // enough CTAs to stream the keys at full occupancy (16 KB of registers
  // each); their merges mostly find the global registers already as large
  int64_t blocks = (n + 1023) / 1024;
  if (blocks > static_cast<int64_t>(num_sms()) * 8) blocks = static_cast<int64_t>(num_sms()) * 8;
  {
    ProfScope prof("group_sketch_kernel", s);
    group_sketch_kernel<<<static_cast<int>(blocks < 1 ? 1 : blocks), 256, 0, s>>>(p, regs->as<unsigned>());
    after_launch("group_sketch_kernel");
    prof.stop(static_cast<double>(n) * 8);
  }
  std::vector<unsigned> h(kSketchRegs);
  GF_CUDA(cudaMemcpyAsync(h.data(), regs->data(), kSketchRegs * 4, cudaMemcpyDeviceToHost, s));
  sync(s);
  double sum = 0;
  int zeros = 0;
  for (unsigned v : h) {
    sum += 1.0 / static_cast<double>(uint64_t{1} << v);  // v <= 64 - kSketchBits + 1
    zeros += v == 0 ? 1 : 0;
  }
  const double m = kSketchRegs;
  double e = 0.7213 / (1.0 + 1.079 / m) * m * m / sum;
  if (e <= 2.5 * m && zeros > 0) e = m * std::log(m / zeros);
  return e;
}

class StringDict {
 public:
  BufferPtr slot_hash, slot_code, code_off, code_len, heap, status;
  uint64_t cap = 0;
  int64_t code_cap = 0, heap_cap = 0;
  int64_t codes_upper = 0, heap_upper = 0;  // host-side upper bounds

  DictDev dev() const {
    DictDev d;
    d.slot_hash = slot_hash->as<uint64_t>();
    d.slot_code = slot_code->as<uint32_t>();
    d.code_off = code_off->as<int64_t>();
    d.code_len = code_len->as<int32_t>();
    d.heap = heap->as<uint8_t>();
    d.mask = cap - 1;
    d.code_cap = code_cap;
    d.heap_cap = heap_cap;
    d.st = status->as<DevStatus>();
    return d;
  }

  void ensure(int64_t more_codes, int64_t more_bytes, cudaStream_t s) {
    if (!status) status = make_filled(sizeof(DevStatus), 0, s);
    int64_t codes_real = 0, bytes_real = 0;
    const bool grow_slots = static_cast<uint64_t>(2 * (codes_upper + more_codes)) > cap;
    const bool grow_codes = codes_upper + more_codes > code_cap;
    const bool grow_heap = heap_upper + more_bytes > heap_cap;
    if (!(grow_slots || grow_codes || grow_heap)) return;
    if (cap > 0) {
      DevStatus h = read_status(status->as<DevStatus>(), s);
      raise_device_status(h, "string dictionary");
      codes_real = h.aux[0];
      bytes_real = h.aux[1];
      codes_upper = codes_real;
      heap_upper = bytes_real;
    }
    const int64_t need_codes = codes_upper + more_codes;
    const int64_t need_bytes = heap_upper + more_bytes;
    if (need_codes > code_cap) {
      int64_t nc = static_cast<int64_t>(next_pow2(static_cast<uint64_t>(need_codes < 1024 ? 1024 : need_codes)));
      auto off = make_buffer(nc * 8, s), len = make_buffer(nc * 4, s);
      if (codes_real > 0) {
        GF_CUDA(cudaMemcpyAsync(off->data(), code_off->data(), codes_real * 8, cudaMemcpyDeviceToDevice, s));
        GF_CUDA(cudaMemcpyAsync(len->data(), code_len->data(), codes_real * 4, cudaMemcpyDeviceToDevice, s));
      }
      code_off = off;
      code_len = len;
      code_cap = nc;
    }
    if (need_bytes > heap_cap) {
      int64_t nb = static_cast<int64_t>(next_pow2(static_cast<uint64_t>(need_bytes < 4096 ? 4096 : need_bytes)));
      auto hp = make_buffer(nb, s);
      if (bytes_real > 0) GF_CUDA(cudaMemcpyAsync(hp->data(), heap->data(), bytes_real, cudaMemcpyDeviceToDevice, s));
      heap = hp;
      heap_cap = nb;
    }
    uint64_t want = next_pow2(static_cast<uint64_t>(2 * need_codes < 1024 ? 1024 : 2 * need_codes));
    if (want > cap) {
      slot_hash = make_filled(static_cast<int64_t>(want) * 8, 0xFF, s);
      slot_code = make_filled(static_cast<int64_t>(want) * 4, 0, s);
      cap = want;
      if (codes_real > 0) {
        dict_rehash_kernel<<<grid_for(codes_real), 256, 0, s>>>(dev(), codes_real);
        after_launch("dict_rehash_kernel");
      }
    }
  }

  BufferPtr encode(const Column& c, cudaStream_t s) {
    const int64_t n = c.length;
    int32_t ends[2] = {0, 0};
    if (n > 0) {
      GF_CUDA(cudaMemcpyAsync(&ends[0], c.offsets, 4, cudaMemcpyDeviceToHost, s));
      GF_CUDA(cudaMemcpyAsync(&ends[1], c.offsets + n, 4, cudaMemcpyDeviceToHost, s));
      sync(s);
    }
    ensure(n, ends[1] - ends[0], s);
    auto codes = make_buffer(n * 4, s);
    if (n > 0) {
      dict_encode_kernel<<<grid_for(n), 256, 0, s>>>(c.offsets, static_cast<const uint8_t*>(c.data), 0, n,
                                                     codes->as<int32_t>(), dev());
      after_launch("dict_encode_kernel");
    }
    codes_upper += n;
    heap_upper += ends[1] - ends[0];
    return codes;
  }

  // n records of `width` bytes each (4-byte aligned; the heap keeps every
  // record at a multiple of its width, so records stay aligned).
  BufferPtr encode_records(const void* records, int64_t n, int32_t width, cudaStream_t s) {
    ensure(n, n * width, s);
    auto codes = make_buffer(n * 4, s);
    if (n > 0) {
      dict_encode_kernel<<<grid_for(n), 256, 0, s>>>(nullptr, static_cast<const uint8_t*>(records), width, n,
                                                     codes->as<int32_t>(), dev());
      after_launch("dict_encode_kernel");
    }
    codes_upper += n;
    heap_upper += n * width;
    return codes;
  }

  ColumnPtr decode(const int32_t* codes, int64_t n, cudaStream_t s) {
    auto offs = make_buffer((n + 1) * 4, s);
    int64_t total = 0;
    if (n > 0) {
      auto lens = make_buffer(n * 4, s);
      dict_lengths_kernel<<<grid_for(n), 256, 0, s>>>(codes, n, code_len->as<int32_t>(), lens->as<int32_t>());
      after_launch("dict_lengths_kernel");
      total = exclusive_scan_i32(lens->as<int32_t>(), offs->as<int32_t>(), n, s);
    } else {
      GF_CUDA(cudaMemsetAsync(offs->data(), 0, 4, s));
    }
    auto bytes = make_buffer(total, s);
    if (n > 0 && total > 0) {
      dict_copy_kernel<<<grid_for(n), 256, 0, s>>>(codes, n, code_off->as<int64_t>(), heap->as<uint8_t>(),
                                                   offs->as<int32_t>(), bytes->as<uint8_t>());
      after_launch("dict_copy_kernel");
    }
    return make_utf8_column(n, offs, bytes);
  }
};

}  // namespace

class GroupTable {
 public:
  std::vector<std::string> group_cols;
  std::vector<GroupAggregate> aggs;
  int64_t hint = 0;

  bool compiled = false;
  std::vector<DType> key_types;
  std::vector<int32_t> key_bits;
  std::vector<AccDev> accs;           // internal accumulators
  std::vector<OutAggDev> outs;        // user aggregates -> accumulators
  std::vector<DType> out_types;
  Program prog{};
  ColumnSlots slots;
  std::vector<std::unique_ptr<StringDict>> dicts;  // per key column (utf8 only)
  bool wide = false;                        // keys as records, grouped by record code
  RecordCols records{};
  std::unique_ptr<StringDict> record_dict;

  BufferPtr keys, accbuf, status;  // accbuf is keys where a slot's key and accumulators lie together
  TableView view{};
  uint64_t cap = 0;
  int64_t groups_upper = 0;

  void compile(const TupleSet& ts) {
    if (group_cols.size() > static_cast<size_t>(kMaxKeyColumns))
      fail(GFPDB_EUNSUPPORTED, "group-by over more than 8 key columns");
    int bits = 0;
    for (auto& g : group_cols) {
      DType t = ts.field(ts.require_column(g)).type;
      if (t == DType::Float64) fail(GFPDB_EUNSUPPORTED, "float64 group keys");
      key_types.push_back(t);
      int b = t == DType::Int64 ? 64 : 32;
      key_bits.push_back(b);
      bits += b;
      dicts.emplace_back(t == DType::Utf8 ? new StringDict() : nullptr);
    }
    if (group_cols.size() > 2 || bits > 64) {
      wide = true;
      std::memset(&records, 0, sizeof(records));
      records.n_cols = static_cast<int32_t>(group_cols.size());
      for (size_t k = 0; k < group_cols.size(); ++k) {
        records.off[k] = records.rec_width;
        records.width[k] = key_types[k] == DType::Int64 ? 8 : 4;  // utf8 columns as their int32 codes
        records.rec_width += records.width[k];
      }
      record_dict.reset(new StringDict());
    }
    std::memset(&prog, 0, sizeof(prog));
    for (auto& a : aggs) {
      OutAggDev o{};
      auto add_acc = [&](int8_t fn, int8_t vt, Operand in) {
        if (static_cast<int>(accs.size()) >= kMaxAggs) fail(GFPDB_EUNSUPPORTED, "too many aggregates");
        AccDev d{};
        d.fn = fn;
        d.vt = vt;
        d.in = in;
        accs.push_back(d);
        return static_cast<int32_t>(accs.size() - 1);
      };
      if (a.fn == AGG_AVG_REDUCE) {
        // AvgReduce (fpdb-executor/src/physical/aggregate/function/AvgReduce.cpp:21-84):
        // the first phase's AVG_INTERMEDIATE_SUM_<name> and
        // AVG_INTERMEDIATE_COUNT_<name> columns, each summed, divided at
        // finalisation.
        auto column = [](const std::string& n) {
          auto e = std::make_shared<Expr>();
          e->kind = Expr::Column;
          e->name = n;
          return ExprPtr(e);
        };
        DType sum_t, cnt_t;
        Operand sum_in = compile_value(column(kAvgIntermediateSum + a.name), ts.fields(), prog, slots, &sum_t);
        Operand cnt_in = compile_value(column(kAvgIntermediateCount + a.name), ts.fields(), prog, slots, &cnt_t);
        if (cnt_t == DType::Float64 || cnt_t == DType::Utf8 || sum_t == DType::Utf8)
          fail(GFPDB_EINVAL, "AVG_REDUCE '" + a.name + "' needs a numeric sum and an integer count column");
        o.kind = 1;
        o.vt = sum_t == DType::Float64 ? VT_F64 : VT_I64;
        o.a0 = add_acc(AGG_SUM, o.vt, sum_in);
        o.a1 = add_acc(AGG_SUM, VT_I64, cnt_in);
        o.out_type = static_cast<int8_t>(DType::Float64);
        out_types.push_back(DType::Float64);
      } else if (a.fn == AGG_COUNT_STAR || (a.fn == AGG_COUNT && !a.expr)) {
        Operand none{};
        none.kind = OPND_LIT;
        o.kind = 0;
        o.a0 = add_acc(AGG_COUNT_STAR, VT_I64, none);
        o.out_type = static_cast<int8_t>(DType::Int64);
        out_types.push_back(DType::Int64);
      } else {
        if (!a.expr) fail(GFPDB_EINVAL, "aggregate '" + a.name + "' needs an input expression");
        DType in_t;
        Operand in = compile_value(a.expr, ts.fields(), prog, slots, &in_t);
        const int8_t vt = in_t == DType::Float64 ? VT_F64 : VT_I64;
        if (a.fn == AGG_SUM) {
          o.a0 = add_acc(AGG_SUM, vt, in);
          DType ot = vt == VT_F64 ? DType::Float64 : DType::Int64;
          o.out_type = static_cast<int8_t>(ot);
          out_types.push_back(ot);
        } else if (a.fn == AGG_COUNT) {
          o.a0 = add_acc(AGG_COUNT, VT_I64, in);
          o.out_type = static_cast<int8_t>(DType::Int64);
          out_types.push_back(DType::Int64);
        } else if (a.fn == AGG_MIN || a.fn == AGG_MAX) {
          o.a0 = add_acc(a.fn, vt, in);
          o.out_type = static_cast<int8_t>(in_t);
          out_types.push_back(in_t);
        } else {  // AVG: sum and count, divided at finalisation
          o.kind = 1;
          o.vt = vt;
          o.a0 = add_acc(AGG_SUM, vt, in);
          Operand none{};
          none.kind = OPND_LIT;
          o.a1 = add_acc(AGG_COUNT_STAR, VT_I64, none);
          o.out_type = static_cast<int8_t>(DType::Float64);
          out_types.push_back(DType::Float64);
        }
      }
      outs.push_back(o);
    }
    compiled = true;
  }

  // Tables of kPackedSlots slots and more, too large for the L2 to keep whole,
  // put a slot's key beside its accumulators when they fill 16 or 32 bytes
  // (one or three accumulators): a row then touches one sector instead of
  // two or three.
  static constexpr uint64_t kPackedSlots = 1ull << 20;

  void init_table(uint64_t new_cap, cudaStream_t s) {
    const int na = static_cast<int>(accs.size());
    // Empty keys are all-ones and sum / count accumulators start at zero, so
    // without MIN / MAX a table with separate keys comes pre-filled (no init
    // kernel; inside a captured plan from the graph's fill regions).
    bool zero_init = true;
    for (int a = 0; a < na; ++a) zero_init &= accs[a].fn != AGG_MIN && accs[a].fn != AGG_MAX;
    const bool packed = new_cap >= kPackedSlots && (na == 1 || na == 3);
    const int64_t n_slots = static_cast<int64_t>(new_cap + 1);
    InitPattern pat{};
    pat.period = packed ? na + 1 : na > 0 ? na : 1;
    if (packed) pat.word[0] = kEmptySlot;
    for (int a = 0; a < na; ++a) pat.word[packed ? a + 1 : a] = acc_identity(accs[a].fn, accs[a].vt);
    auto init = [&](const BufferPtr& b) {
      const uint64_t words = static_cast<uint64_t>(n_slots) * pat.period;
      group_init_kernel<<<grid_for(static_cast<int64_t>(words / 2 + 1)), 256, 0, s>>>(b->as<unsigned long long>(), words,
                                                                                      pat);
      after_launch("group_init_kernel");
    };
    BufferPtr nk, nacc;
    TableView to{};
    if (packed) {
      nk = nacc = make_buffer(n_slots * 8 * (na + 1), s);
      init(nk);
      to = TableView{nk->as<uint64_t>(), nk->as<unsigned long long>() + 1, na + 1, na + 1};
    } else {
      nk = make_filled(n_slots * 8, 0xFF, s);
      const int64_t acc_bytes = n_slots * 8 * (na > 0 ? na : 1);
      if (zero_init) {
        nacc = make_filled(acc_bytes, 0, s);
      } else {
        nacc = make_buffer(acc_bytes, s);
        init(nacc);
      }
      to = TableView{nk->as<uint64_t>(), nacc->as<unsigned long long>(), 1, na};
    }
    if (!status) status = make_filled(sizeof(DevStatus), 0, s);
    if (cap > 0) {
      group_rehash_kernel<<<grid_for(static_cast<int64_t>(cap + 1)), 256, 0, s>>>(view, cap, to, new_cap - 1, na,
                                                                                 status->as<DevStatus>());
      after_launch("group_rehash_kernel");
    }
    keys = nk;
    accbuf = nacc;
    view = to;
    cap = new_cap;
  }

  // group_update_plain_kernel's parameters, or false when an accumulator is
  // not an integer sum, minimum or maximum of a column or a count.
  static bool plain_params(const GroupParams& p, PlainParams* out) {
    if (p.n_acc < 1 || p.n_acc > kPlainAccs) return false;
    std::memset(out, 0, sizeof(*out));
    out->n = static_cast<uint32_t>(p.n_rows);
    out->n_keys = p.n_keys;
    out->wide_key = p.n_keys == 1 && p.key_bits[0] == 64;
    for (int k = 0; k < p.n_keys; ++k) {
      if ((p.key_cols[k].type == CT_I64) != (out->wide_key != 0)) return false;
      out->key[k] = p.key_cols[k].data;
    }
    int n = 0;
    for (int pass = 0; pass < 2; ++pass) {  // sums and counts first
      for (int a = 0; a < p.n_acc; ++a) {
        const AccDev& d = p.acc[a];
        const bool count = d.fn == AGG_COUNT || d.fn == AGG_COUNT_STAR;
        if ((count || d.fn == AGG_SUM) != (pass == 0)) continue;
        PlainAcc& o = out->acc[n++];
        o.at = a;
        if (count) continue;
        if (d.vt == VT_F64 || d.in.kind != OPND_COL) return false;
        const DevCol& c = p.cols[d.in.col];
        if (c.type != CT_I64 && c.type != CT_I32 && c.type != CT_DATE32) return false;
        o.col = c.data;
        o.wide = c.type == CT_I64;
        o.flip = d.fn == AGG_MIN ? -1 : 0;
      }
      if (pass == 0) out->n_add = n;
    }
    return true;
  }

  void update(const TupleSet& batch, cudaStream_t s) {
    if (!compiled) compile(batch);
    // String keys are dictionary-encoded from exact inputs; other batches
    // may carry their row count on the device.
    TupleSetPtr exact_holder;
    const TupleSet* tsp = &batch;
    bool utf8_key = false;
    for (auto t : key_types) utf8_key |= t == DType::Utf8;
    if ((utf8_key || wide) && !batch.exact()) {
      exact_holder = batch.resolve(s);
      tsp = exact_holder.get();
    }
    const TupleSet& ts = *tsp;
    const int64_t n = ts.num_rows();
    if (n >= INT32_MAX) fail(GFPDB_EUNSUPPORTED, "group-by batch must have fewer than 2^31 rows");

    GroupParams* pp = new GroupParams;
    std::unique_ptr<GroupParams> holder(pp);
    GroupParams& p = *pp;
    std::memset(&p, 0, sizeof(p));
    p.n_rows = n;
    p.n_dev = ts.rows_dev();
    p.n_keys = static_cast<int32_t>(group_cols.size());
    p.n_acc = static_cast<int32_t>(accs.size());
    std::vector<BufferPtr> code_bufs;
    if (wide && n > 0) {
      RecordCols rc = records;
      for (int k = 0; k < rc.n_cols; ++k) {
        const auto& c = ts.column(group_cols[k]);
        if (c->type != key_types[k]) fail(GFPDB_EINVAL, "group key column changed type between batches");
        if (c->type == DType::Utf8) {
          auto codes = dicts[k]->encode(*c, s);
          code_bufs.push_back(codes);
          rc.cols[k] = DevCol{codes->data(), nullptr, CT_I32, 0};
        } else {
          rc.cols[k] = DevCol{c->data, nullptr, static_cast<int32_t>(c->type), 0};
        }
      }
      auto recs = make_buffer(n * rc.rec_width, s);
      group_record_pack_kernel<<<grid_for(n), 256, 0, s>>>(rc, n, recs->as<uint32_t>());
      after_launch("group_record_pack_kernel");
      auto codes = record_dict->encode_records(recs->data(), n, rc.rec_width, s);
      code_bufs.push_back(codes);
      p.n_keys = 1;
      p.key_bits[0] = 32;
      p.key_cols[0] = DevCol{codes->data(), nullptr, CT_I32, 0};
    } else if (n > 0) {
      for (int k = 0; k < p.n_keys; ++k) {
        const auto& c = ts.column(group_cols[k]);
        if (c->type != key_types[k]) fail(GFPDB_EINVAL, "group key column changed type between batches");
        p.key_bits[k] = key_bits[k];
        if (c->type == DType::Utf8) {
          auto codes = dicts[k]->encode(*c, s);
          code_bufs.push_back(codes);
          p.key_cols[k] = DevCol{codes->data(), nullptr, CT_I32, 0};
        } else {
          p.key_cols[k] = DevCol{c->data, nullptr, static_cast<int32_t>(c->type), 0};
        }
      }
    }

    // Size the table so that it stays at most half full.
    int64_t bound = groups_upper + n;
    if (hint > 0 && bound > hint) bound = groups_upper > hint ? groups_upper : hint;
    uint64_t want = next_pow2(static_cast<uint64_t>(2 * bound < 1024 ? 1024 : 2 * bound));
    if (want > cap && cap > 0) {
      // Upper bound says grow: read the real group count first.
      DevStatus h = read_status(status->as<DevStatus>(), s);
      raise_device_status(h, "group-by");
      groups_upper = h.aux[0];
      bound = groups_upper + n;
      if (hint > 0 && bound > hint) bound = groups_upper > hint ? groups_upper : hint;
      want = next_pow2(static_cast<uint64_t>(2 * bound < 1024 ? 1024 : 2 * bound));
    }
    if (want > cap && want > kSketchMinSlots && hint == 0 && n > 0 && p.n_keys > 0 && ts.exact() &&
        !deferred_mode() && !stream_capturing(s)) {
      // A large table for a batch whose rows are on the host: size it for
      // the batch's estimated distinct keys (with a quarter to spare) over
      // the exact groups so far instead of its row count.
      const double est = sketch_distinct(p, n, s);
      int64_t fresh = static_cast<int64_t>(est * 1.25) + 1024;
      if (fresh > n) fresh = n;
      const int64_t known = cap > 0 ? groups_upper : 0;  // exact: read above
      const int64_t b2 = known + fresh;
      // at most 5/8 full with the spare quarter taken, half full without: a
      // table half the size costs the update a little and saves more around
      // it (three accumulators, 0.9M groups of 20M rows, 2M slots against 4M:
      // init 23 against 43 us, update 396 against 371, finalize 44 against
      // 74; six, 20M rows of 1M keys: the call 1,150 against 1,225 us). With
      // fewer accumulators there is less around it, and longer runs cost
      // more: half full at most (20M rows of 1M keys: no accumulators 520
      // against 654 us, one 619 against 761, two 923 against 998).
      const int64_t slots = accs.size() < 3 ? 2 * b2 : b2 + b2 * 3 / 5;
      const uint64_t w2 = next_pow2(static_cast<uint64_t>(slots < 1024 ? 1024 : slots));
      if (w2 < want) want = w2 > cap ? w2 : cap;
    }
    if (want > cap) init_table(want, s);
    if (n == 0) return;

    for (int a = 0; a < p.n_acc; ++a) p.acc[a] = accs[a];
    bind_columns(slots, ts, p.cols, kMaxCols);
    p.prog = prog;
    p.keys = view.keys;
    p.accs = view.accs;
    p.key_stride = view.key_stride;
    p.acc_stride = view.acc_stride;
    p.mask = cap - 1;
    p.st = status->as<DevStatus>();
    // Shared-memory pre-aggregation unless the caller expects many groups.
    const int per_slot = 8 + 8 * p.n_acc;
    const bool use_smem = hint == 0 || hint <= 4096;
    for (int a = 0; a < p.n_acc; ++a) p.float_sums |= accs[a].fn == AGG_SUM && accs[a].vt == VT_F64;
    ProfScope prof("group_update_kernel", s);
    PlainParams plain;
    if (use_smem && ts.exact() && n >= kGroupPlainRows && plain_params(p, &plain)) {
      using PlainKernel = void (*)(GroupParams, PlainParams);
      static const PlainKernel table[kPlainAccs] = {group_update_plain_kernel<1, false>, group_update_plain_kernel<2, false>,
                                                    group_update_plain_kernel<3, false>, group_update_plain_kernel<4, false>};
      const bool beside = p.n_acc == 3 && p.key_stride == 4;
      const PlainKernel fn = beside ? group_update_plain_kernel<3, true> : table[p.n_acc - 1];
      p.sm_slots = static_cast<int32_t>((max_smem_optin() - 1024 - plain_smem(0, 0)) / (per_slot + 1)) / kPlainWays * kPlainWays;
      const int64_t dyn = plain_smem(p.sm_slots, p.n_acc);
      allow_shared(fn, dyn);
      const int64_t step = kPlainThreads * kPlainRows;
      fn<<<static_cast<int>(std::min<int64_t>(num_sms(), (n + step - 1) / step)), kPlainThreads, dyn, s>>>(p, plain);
    } else {
      using Kernel = void (*)(GroupParams);
      static const Kernel table[2][3] = {{group_update_global_kernel<0>, group_update_global_kernel<1>, group_update_global_kernel<2>},
                                         {group_update_kernel<0>, group_update_kernel<1>, group_update_kernel<2>}};
      const Kernel fn = table[use_smem ? 1 : 0][std::min(p.n_acc, 2)];
      int sm_slots = kGroupSmemSlotsMax;
      // dynamic plus static shared memory stays within the 48 KB a launch
      // gets without opting in to more
      while (group_smem(sm_slots, p.n_acc) > 47 * 1024) sm_slots >>= 1;
      p.sm_slots = sm_slots;
      const size_t dyn = static_cast<size_t>(use_smem ? group_smem(sm_slots, p.n_acc) : 0);
      // 16 rows a thread amortise a CTA's table, but while that leaves SMs
      // without a CTA four rows do
      int64_t blocks = (n + kGroupThreads * 16 - 1) / (kGroupThreads * 16);
      blocks = std::max(blocks, std::min<int64_t>(num_sms(), (n + kGroupThreads * 4 - 1) / (kGroupThreads * 4)));
      // one wave: as many CTAs as fit on every SM at once
      int per_sm = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kGroupThreads, dyn) != cudaSuccess || per_sm < 1)
        per_sm = 1;
      int64_t max_blocks = static_cast<int64_t>(num_sms()) * per_sm;
      if (blocks > max_blocks) blocks = max_blocks;
      if (blocks < 1) blocks = 1;
      fn<<<static_cast<int>(blocks), kGroupThreads, dyn, s>>>(p);
    }
    after_launch("group_update_kernel");
    double w = 0;
    for (int k = 0; k < p.n_keys; ++k) w += p.key_bits[k] / 8;
    if (wide) w += records.rec_width - 4;
    for (size_t i = 0; i < slots.types.size(); ++i) w += dtype_width(slots.types[i]);
    prof.stop(static_cast<double>(n) * w);
    if (p.n_dev) prof.set_bytes_model(p.n_dev, n, w, nullptr, 0, ts.rows_owner());
    groups_upper += n;
    if (hint > 0 && groups_upper > hint) groups_upper = hint;
  }

  TupleSetPtr finalize(const TupleSet* schema_src, cudaStream_t s) {
    std::vector<Field> fields;
    for (size_t k = 0; k < group_cols.size(); ++k)
      fields.push_back(Field{group_cols[k], compiled ? key_types[k] : DType::Int64});
    for (size_t j = 0; j < aggs.size(); ++j)
      fields.push_back(Field{aggs[j].name, compiled ? out_types[j] : DType::Int64});
    if (!compiled || cap == 0) return TupleSet::make_empty(fields, s);
    (void)schema_src;
    bool utf8_key = wide;
    for (auto t : key_types) utf8_key |= t == DType::Utf8;
    // Deferred: outputs sized for every slot, the group count stays on the
    // device and the status block is checked at the end of the plan.
    const bool defer = deferred_mode() && !utf8_key;
    int64_t n_groups = static_cast<int64_t>(cap) + 1;
    if (defer) {
      defer_check(status, status->as<DevStatus>(), "group-by");
    } else {
      DevStatus h = read_status(status->as<DevStatus>(), s);
      raise_device_status(h, "group-by");
      for (auto& d : dicts)
        if (d && d->status) raise_device_status(read_status(d->status->as<DevStatus>(), s), "string dictionary");
      if (record_dict && record_dict->status)
        raise_device_status(read_status(record_dict->status->as<DevStatus>(), s), "group key dictionary");
      n_groups = h.aux[0];
    }
    FinalParams fp;
    std::memset(&fp, 0, sizeof(fp));
    fp.keys = view.keys;
    fp.accs = view.accs;
    fp.key_stride = view.key_stride;
    fp.acc_stride = view.acc_stride;
    fp.cap = cap;
    fp.special_dev = &status->as<DevStatus>()->aux[1];
    fp.n_acc = static_cast<int32_t>(accs.size());
    fp.n_keys = static_cast<int32_t>(group_cols.size());
    std::vector<BufferPtr> key_out(group_cols.size());
    BufferPtr record_codes;
    if (wide) {  // the table's key is the record code
      fp.n_keys = 1;
      record_codes = make_buffer(n_groups * 4, s);
      fp.key_dst[0] = record_codes->data();
      fp.key_type[0] = CT_I32;
      fp.key_bits[0] = 32;
    }
    for (size_t k = 0; k < group_cols.size() && !wide; ++k) {
      DType t = key_types[k] == DType::Utf8 ? DType::Int32 : key_types[k];
      key_out[k] = make_buffer(n_groups * dtype_width(t), s);
      fp.key_dst[k] = key_out[k]->data();
      fp.key_type[k] = static_cast<int32_t>(t);
      fp.key_bits[k] = key_bits[k];
    }
    std::vector<BufferPtr> agg_out(aggs.size());
    fp.n_out = static_cast<int32_t>(aggs.size());
    for (size_t j = 0; j < aggs.size(); ++j) {
      agg_out[j] = make_buffer(n_groups * dtype_width(out_types[j]), s);
      fp.outs[j] = outs[j];
      fp.outs[j].dst = agg_out[j]->data();
    }
    auto counter = make_filled(8, 0, s);
    fp.counter = counter->as<unsigned long long>();
    {
      ProfScope prof("group_finalize_kernel", s);
      if (cap + 1 >= kFinalChunkedSlots)
        group_finalize_kernel<8><<<grid_for(static_cast<int64_t>((cap + 1) / 8)), 256, 0, s>>>(fp);
      else
        group_finalize_kernel<1><<<grid_for(static_cast<int64_t>(cap + 1)), 256, 0, s>>>(fp);
      after_launch("group_finalize_kernel");
      prof.stop(static_cast<double>(cap + 1) * 8);
    }
    if (wide) {
      std::vector<void*> dst(group_cols.size());
      for (size_t k = 0; k < group_cols.size(); ++k) {
        key_out[k] = make_buffer(n_groups * records.width[k], s);
        dst[k] = key_out[k]->data();
      }
      auto dst_dev = make_buffer(static_cast<int64_t>(dst.size() * sizeof(void*)), s);
      GF_CUDA(cudaMemcpyAsync(dst_dev->data(), dst.data(), dst.size() * sizeof(void*), cudaMemcpyHostToDevice, s));
      if (n_groups > 0) {
        group_record_split_kernel<<<grid_for(n_groups), 256, 0, s>>>(
            records, n_groups, record_codes->as<int32_t>(), record_dict->code_off->as<int64_t>(),
            record_dict->heap->as<uint8_t>(), dst_dev->as<void*>());
        after_launch("group_record_split_kernel");
      }
      sync(s);  // dst (host vector) is read by the copy above
    }
    std::vector<ColumnPtr> cols;
    for (size_t k = 0; k < group_cols.size(); ++k) {
      if (key_types[k] == DType::Utf8) cols.push_back(dicts[k]->decode(key_out[k]->as<int32_t>(), n_groups, s));
      else cols.push_back(make_fixed_column(key_types[k], n_groups, key_out[k]));
    }
    for (size_t j = 0; j < aggs.size(); ++j) cols.push_back(make_fixed_column(out_types[j], n_groups, agg_out[j]));
    if (defer)
      return TupleSet::make_deferred(std::move(fields), std::move(cols), n_groups, counter,
                                     reinterpret_cast<const int64_t*>(counter->data()));
    return TupleSet::make(std::move(fields), std::move(cols), n_groups);
  }
};

std::shared_ptr<GroupTable> group_table_create(const std::vector<std::string>& group_cols,
                                               const std::vector<GroupAggregate>& aggs, int64_t groups_hint) {
  auto g = std::make_shared<GroupTable>();
  g->group_cols = group_cols;
  g->aggs = aggs;
  g->hint = groups_hint;
  return g;
}

void group_table_update(GroupTable& g, const TupleSet& batch, cudaStream_t s) { g.update(batch, s); }

TupleSetPtr group_table_finalize(GroupTable& g, cudaStream_t s) { return g.finalize(nullptr, s); }

}  // namespace gfpdb
