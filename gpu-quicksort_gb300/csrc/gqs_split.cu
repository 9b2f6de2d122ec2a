// The split sort: quicksort's partition with hundreds of pivots at once, and an on-chip sort of the
// ranges it leaves.
//
// A binary partition level reads and writes every key to gain one bit of order, and a sort of 2^28
// keys needs about fifteen before its ranges fit on chip. Here one level puts every key into one
// of up to 1024 ranges, so two levels reach ranges of a few thousand keys at 2^28, and one level
// reaches them below four million keys:
//   split_map      one CTA a segment: a map of a key to its range, from a sample of the segment
//   split_count    every key's range, counted
//   split_starts   where every range starts; ranges still too long become segments of the next level
//   split_scatter  every key to its range (d -> dn at the first level, dn -> d at the second)
//   local_sort     every range sorted in shared memory, into d
// Plain sorts of at most kSmallMax keys take two kernels instead: split_small (every CTA makes the
// map for itself, then scatters into ranges with room for kLocal keys each, so that nothing is
// counted first) and local_small over those ranges.
// Device time against the persistent kernel's binary levels, which took these sorts before: 2^28 u32 10.7 to 3.10 ms, 2^26 f64
// 5.05 to 1.86 ms, 2^20 u32 84 to 27 us (that was with a split of its own in front).
// The order of keys inside a range does not matter to the next step, so a key's place in it
// is the old value of a counter (one shared-memory atomic), not a stable rank.
//
// What cannot be sorted so (a range that stays longer than the on-chip sort takes, because the map's
// sample missed its keys) is listed for the persistent kernel's quicksort; Queue::left counts it.
//
// The reference's counterparts: gqsort_kernel's partition (GPU-Quicksort_OpenCL_1.2/
// QuicksortKernels.cl:102-240) generalised from one pivot, and lqsort_kernel (267-421).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "gqs_device.cuh"
#include "gqs_launch.h"

// Fields and arguments that only the bounds-check build has.
#ifdef GQS_CHECK
#define GQS_CHECK_ONLY(...) __VA_ARGS__
#else
#define GQS_CHECK_ONLY(...)
#endif

namespace gqs {
namespace {

template <class T>
using BOf = typename KeyOps<T>::B;

constexpr int kThreads = 512;                   // of the map, count and scatter kernels
constexpr uint32_t kTileCtas = 2;               // of the scatter kernels on an SM: three spill their keys (2^28 u32: 3.10 to 3.66 ms)
constexpr uint32_t kMaxBins = 1024;             // ranges one segment is split into (bin_room: the map may make more)
constexpr uint32_t kBinSlots = 2564;            // bin_room(kMaxBins)
constexpr uint32_t kMaxCells = 4096;
constexpr uint32_t kMaxParts = 256;             // cells divided further
constexpr uint32_t kMaxSub = 2048;              // cells that those are divided into
constexpr uint32_t kPartSub = 128;              // and at most so many for one
constexpr uint32_t kWarpBin = 256;              // longer ones of unequal keys are sorted by a warp each, beyond this by the CTA
constexpr int kCandidates = 4;
constexpr uint32_t kOver = 32;                  // samples a range of a counted level
constexpr uint32_t kCluster = 4;                // CTAs of a small sort that take the sample together
constexpr uint32_t kCopyChunk = 32768;          // keys of one record of a range of equal keys
constexpr uint32_t kSmallOver = 10;             // samples a range of a small sort (its ranges have room for three times their mean)

template <class B>
struct Sizes {
  // Keys one CTA sorts on chip, and its CTAs: 256 threads, three on an SM. 2^28 u32 takes 3.37 ms so; with 512 threads and two CTAs
  // 3.54, with four CTAs (fewer registers) 3.42, with two 3.48.
  static constexpr uint32_t kLocal = sizeof(B) == 8 ? 4096 : 8192;
  static constexpr uint32_t kSortThreads = 256, kSortCtas = 3;
  static constexpr uint32_t kTarget = kLocal / 16 * 7;  // mean keys of a range (6/16: 2^28 u32 3.45 ms)
  static constexpr int kTileRows = 64 / (int)sizeof(B);  // keys a thread of a tile
  static constexpr uint32_t kTile = kThreads * kTileRows;
  static constexpr int kLocalRows = (int)(kLocal / kSortThreads);
  static constexpr int kBlock = sizeof(B) == 8 ? 8 : 16;     // keys of one network of the on-chip sort
  static constexpr uint32_t kShortBin = kBlock / 2 + 1;      // longest bin that these put in order
  static constexpr uint32_t kTiny = sizeof(B) == 8 ? 128 : 256;
  // keys of a sample: at the first level of a plain sort (one CTA), at other levels, and in a small sort (two CTAs an SM)
  static constexpr uint32_t kMaxSample = sizeof(B) == 8 ? 16384 : 24576, kMaxSample2 = sizeof(B) == 8 ? 8192 : 12288;
  static constexpr uint32_t kSmallSample = sizeof(B) == 8 ? 3328 : 5120;
  static constexpr size_t kSmallMax = sizeof(B) == 8 ? 1u << 19 : 1u << 21;
};
template <class T>
using EngineCfg = Cfg<T, 16, sizeof(BOf<T>) == 8 ? 6144 : 12288, sizeof(BOf<T>) == 8 ? 4096 : 8192, 3, sizeof(BOf<T>) == 8 ? 4 : 8>;
template <class T>
constexpr bool kFloating = !KeyOps<T>::kIdentity;

constexpr uint32_t kEqual = 1u << 30, kBinMask = 0xffffu;  // in a map's table: all keys of the range are equal; the range

// A segment being split: its keys, and the map of a key to its range.
struct SegRec {
  unsigned long long start;
  unsigned long long lo, span;  // keys are clamped to [lo, lo + span]
  uint32_t len, k, cells;       // cells allocated, of the segment and of its parts
  uint32_t bin0, cell0, tile0;  // its counters, map cells and tiles
  uint32_t sh, bins, used;      // entries of the table; cell of a key: (key - lo) >> sh, or by value:
  float flo, scale;             // (key - flo) * scale
  uint32_t top;                 // greatest value of that
  uint32_t kind;                // BY_VALUE, PARTS, and how many Part records there are
};
enum : uint32_t { BY_VALUE = 1u << 31, PARTS = 1u << 30, PART_COUNT = PARTS - 1u };
// A cell with more than the sample of one range, divided further: equal steps between its least and greatest sampled key, or
// (mult 0) the keys below, equal to and above one value that makes up nearly all of them.
template <class B>
struct Part {
  B lo, span;
  uint32_t right, left, mult;  // the span shifted to just below 2^32, times mult / 2^32
  uint32_t sub;                // its cells in the table start here
  __device__ __forceinline__ uint32_t of(B key) const {
    if (!mult) return sub + (key >= lo ? 1u : 0u) + (key > lo ? 1u : 0u);
    B y = (key < lo ? lo : key) - lo;
    y = y < span ? y : span;
    return sub + __umulhi((uint32_t)(y >> right) << left, mult);
  }
};
enum : uint32_t { IN_DN = 1, EQUAL = 2 };
struct Bucket {
  unsigned long long start;
  uint32_t len, flags;
  unsigned long long value;  // EQUAL: all keys are this
};
struct alignas(256) Ctl {
  unsigned long long alloc[2];  // (segments << 32) | tiles, per level
  unsigned long long leftovers;
  uint32_t bins[2], cells[2];
  uint32_t buckets;
};

// The tables of one level.
struct Level {
  SegRec* seg;
  uint32_t* bin;   // keys per range, then the next output position in it (from the segment's start)
  unsigned long long* value;  // kEqual ranges: the keys, as the map orders them
  uint32_t* eq;               // 1: a kEqual range
  uint32_t* cell;
  void* part;      // the records of the cells with a map of their own (part_room(k) for a segment, at bin0 / 4)
  uint32_t segs, bins, cells;  // how many there is room for
  uint32_t index;
};
struct Tables {
  Ctl* ctl;
  Bucket* bucket;
  unsigned long long* left;  // (start, end) of the ranges left to the quicksort
  uint32_t buckets;          // records there is room for
  uint32_t tile_keys;
  uint32_t lefts;            // records of `left` that there is room for
  unsigned long long n;      // every key index is below it
};
// The state of a small plain sort. The cursors and the count of finished CTAs are zero between sorts: the last CTA of
// local_small leaves them so.
struct Small {
  uint32_t cursor[kBinSlots];              // next place in every range
  uint32_t done;                           // CTAs of local_small that have finished
  uint32_t bins;
  unsigned long long left;                 // 1: all of the sort is left to the persistent kernel
  unsigned long long table[2];             // (then: [0, n))
  uint32_t eq[kBinSlots];                  // 1: all keys of the range are equal (the cursor counts them, none is moved)
  unsigned long long value[kBinSlots];     // to this (as the map orders keys)
};

__device__ __forceinline__ uint32_t ceil_log2(uint32_t v) { return v <= 1u ? 0u : 32u - (uint32_t)__clz(v - 1u); }

// Counters of a segment split k ways: at most k + 1 ranges, and two for each single value with the sample of 1.5 ranges.
__device__ __host__ __forceinline__ uint32_t bin_room(uint32_t k) { return 2u * k + k / 2u + 4u; }
__device__ __host__ __forceinline__ uint32_t part_room(uint32_t k) { return k / 2u + 1u < kMaxParts ? k / 2u + 1u : kMaxParts; }
__device__ __host__ __forceinline__ uint32_t sub_room(uint32_t k) { return 8u * k + 32u < kMaxSub ? 8u * k + 32u : kMaxSub; }
__device__ __forceinline__ uint32_t cell_count(uint32_t k) {
  const uint32_t l = ceil_log2(4u * k);
  return 1u << (l < 8u ? 8u : l > 12u ? 12u : l);
}

// False: no room (only segments that overlap, which no valid table has, can need more than there is).
__device__ __forceinline__ bool add_segment(const Tables& t, const Level& v, unsigned long long start, uint32_t len, uint32_t k) {
  SegRec r{};
  r.start = start;
  r.len = len;
  r.k = k;
  r.cells = cell_count(k) + sub_room(k);
  r.bin0 = atomicAdd(&t.ctl->bins[v.index], bin_room(k));
  r.cell0 = atomicAdd(&t.ctl->cells[v.index], r.cells);
  const uint32_t tiles = (len + t.tile_keys - 1u) / t.tile_keys;
  const unsigned long long old = atomicAdd(&t.ctl->alloc[v.index], (1ull << 32) | (unsigned long long)tiles);
  r.tile0 = (uint32_t)old;
  const uint32_t at = (uint32_t)(old >> 32);
  if (at >= v.segs || r.bin0 + bin_room(k) > v.bins || r.cell0 + r.cells > v.cells) return false;
  v.seg[at] = r;
  return true;
}

// Ranges for `len` keys: enough for a mean of kTarget keys, or with more than kMaxBins needed and a
// second level to come, the square root.
template <class B>
__device__ __host__ __forceinline__ uint32_t range_count(uint32_t len, bool more_levels) {
  const uint32_t want = (len + Sizes<B>::kTarget - 1u) / Sizes<B>::kTarget;
  if (want <= 2u) return 2u;
  if (want <= kMaxBins) return want;
  if (!more_levels) return kMaxBins;
  const uint32_t r = (uint32_t)ceilf(sqrtf((float)want));
  return r < kMaxBins ? r : kMaxBins;
}

// Zeroes `bytes` (a multiple of 4) at p with the calling CTA.
__device__ __forceinline__ void clear(void* p, size_t bytes) {
  for (uint32_t i = threadIdx.x; i < bytes / 4; i += blockDim.x) static_cast<volatile uint32_t*>(p)[i] = 0u;
}

// ---- segments: short ones are sorted or listed, long ones are to be split -------------------
template <class T>
__global__ void __launch_bounds__(256) split_plan_segments(SortArgs<T> a, Tables t, Level v, const unsigned long long* offsets,
                                                           const unsigned long long* nseg_dev, uint32_t nseg,
                                                           unsigned long long n, uint32_t pairs, uint32_t levels) {
  using B = BOf<T>;
  __shared__ unsigned long long placed_sum;
  const uint32_t seg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  pdl_wait();
  pdl_trigger();
  if (nseg_dev) {
    const unsigned long long m = *nseg_dev;
    if (m > nseg) {
      if (seg == 0 && lane == 0) set_error(a.q, ST_INVALID, m);
      return;
    }
    nseg = (uint32_t)m;
  }
  if (threadIdx.x == 0) placed_sum = 0ull;
  __syncthreads();
  if (seg < nseg) {
    const unsigned long long s = offsets[pairs ? 2ull * seg : seg], e = offsets[pairs ? 2ull * seg + 1 : seg + 1];
    if (s > e || e > n) {  // malformed segment table
      if (lane == 0) set_error(a.q, ST_INVALID, seg);
    } else if (e > s) {
      const unsigned long long m = e - s;
      if (m <= Sizes<B>::kTiny) {
        unsigned long long tiny = 0;
        const unsigned long long placed = place_small<EngineCfg<T>>(a, 1u, s, m, tiny);
        if (lane == 0) atomicAdd(&placed_sum, placed);
      } else if (lane == 0) {
        bool room = m < (1ull << 31);
        if (m <= Sizes<B>::kLocal) {
          const uint32_t at = atomicAdd(&t.ctl->buckets, 1u);
          room = at < t.buckets;
          if (room) t.bucket[at] = Bucket{s, (uint32_t)m, 0u, 0ull};
        } else if (room) {
          room = add_segment(t, v, s, (uint32_t)m, range_count<B>((uint32_t)m, levels > 1u));
        }
        if (!room) set_error(a.q, ST_CAPACITY, seg);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && placed_sum) {
    atomicAdd(&a.q->total, placed_sum);
    atomicAdd(&a.q->done, placed_sum);
    atomicAdd(&a.q->tiny_keys, placed_sum);
  }
}

// ---- the map of a segment, from a sample of its keys --------------------------------------------
__device__ __forceinline__ int bits_of(uint32_t v) { return 32 - __clz((int)v); }
__device__ __forceinline__ int bits_of(uint64_t v) { return 64 - __clzll((long long)v); }

// A key of a floating type as a float (a double rounded towards zero, beyond the float range cut
// off), in the keys' order.
template <class T>
__device__ __forceinline__ float as_float(BOf<T> key) {
  if constexpr (sizeof(BOf<T>) == 4) {
    return __uint_as_float((uint32_t)KeyOps<T>::raw(key));
  } else {
    const uint64_t r = KeyOps<T>::raw(key);
    const uint32_t hi = (uint32_t)(r >> 32), mag = hi & 0x7fffffffu;
    uint32_t f = __funnelshift_l((uint32_t)r, mag, 3) - (896u << 23);  // the exponent's bias from 1023 to 127
    f = mag < 0x38100000u ? 0u : mag >= 0x47f00000u ? 0x7f7fffffu : f;
    return __uint_as_float(f | (hi & 0x80000000u));
  }
}
// Both ends and their distance are ordinary floats.
__device__ __forceinline__ bool finite_span(float a, float b, float w) {
  return w > 0.f && w < 3e38f && fabsf(a) < 3e38f && fabsf(b) < 3e38f;
}

// The range of a key: a table's entry for its cell, or (a cell with many samples) for the part of the cell that it is in, and so
// on. Cells are equal steps of the integer that orders the keys, or (floating types, where that spreads the sample more evenly)
// of their value. Every step of it keeps the order of the keys, and every kernel computes the same. VALUE and PARTS_ say what
// the segment's kind asks for: a map of integer cells without parts is one table read and a few integer instructions a key.
template <class T>
struct KeyMap {
  using B = BOf<T>;
  B lo, span;
  uint32_t sh, used, top, kind;
  float flo, scale;
  GQS_CHECK_ONLY(Queue* q; uint32_t bins;)
  __device__ __forceinline__ void load(const SegRec& r GQS_CHECK_ONLY(, Queue* q_)) {
    lo = (B)r.lo;
    span = (B)r.span;
    sh = r.sh;
    used = r.used;
    top = r.top;
    kind = r.kind;
    flo = r.flo;
    scale = r.scale;
#ifdef GQS_CHECK
    q = q_;
    bins = r.bins;
    check(r.cells, r.k);
#endif
  }
#ifdef GQS_CHECK
  // The map's tables are as large as was reserved for them.
  __device__ __forceinline__ void check(uint32_t cells, uint32_t k) {
    if (GQS_OK(used <= cells && used <= kMaxCells + kMaxSub && top < used && bins <= bin_room(k) && bins <= kBinSlots &&
                   (kind & PART_COUNT) <= part_room(k),
               q, 0xD203ull))
      return;
    lo = span = 0;
    sh = top = kind = 0u;
    used = 1u;
    bins = bins < kBinSlots ? bins : kBinSlots;
  }
#endif
  __device__ __forceinline__ B offset(B key) const {
    const B x = (key < lo ? lo : key) - lo;
    return x < span ? x : span;
  }
  template <bool VALUE>
  __device__ __forceinline__ uint32_t cell(B key) const {
    if constexpr (VALUE) {
      const uint32_t u = __float2uint_rz(__fmul_rn(__fsub_rn(as_float<T>(lo + offset(key)), flo), scale));
      return u < top ? u : top;
    } else {
      return (uint32_t)(offset(key) >> sh);
    }
  }
  // (tables of short() entries take the mark of a part and kEqual from the two highest bits)
  template <bool VALUE, bool PARTS_, class E>
  __device__ __forceinline__ uint32_t bin(B key, const E* tab, const Part<B>* part) const {
    constexpr int kTop = sizeof(E) * 8 - 1;
    uint32_t e = tab[cell<VALUE>(key)];
    if constexpr (PARTS_) {
#ifdef GQS_CHECK
      for (int depth = 0; e >> kTop; ++depth) {
        const uint32_t p = e & ((1u << kTop) - 1u);
        if (!GQS_OK(p < (kind & PART_COUNT) && depth < 4, q, 0xD204ull)) return 0u;
        const uint32_t at = part[p].of(key);
        if (!GQS_OK(at < used, q, 0xD205ull)) return 0u;
        e = tab[at];
      }
#else
      while (e >> kTop) e = tab[part[e & ((1u << kTop) - 1u)].of(key)];
#endif
      if (sizeof(E) == 2 && e >> 14) e ^= 1u << 14 ^ kEqual;
    }
    if (!GQS_OK((e & kBinMask) < bins, q, 0xD206ull)) return 0u;
    return e;
  }
  static __device__ __forceinline__ uint16_t narrow(uint32_t e) { return (uint16_t)((e & 0x3fffu) | (e >> 16 & 0xc000u)); }
};
// Calls f.template operator()<VALUE, PARTS_>() with what `kind` says.
template <class T, class F>
__device__ __forceinline__ void by_kind(uint32_t kind, F&& f) {
  if (kFloating<T> && (kind & BY_VALUE)) {
    if (kind & PARTS) f.template operator()<kFloating<T>, true>();
    else f.template operator()<kFloating<T>, false>();
  } else {
    if (kind & PARTS) f.template operator()<false, true>();
    else f.template operator()<false, false>();
  }
}

template <class B>
__device__ __forceinline__ B warp_min(B v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const B w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w < v ? w : v;
  }
  return v;
}
template <>
__device__ __forceinline__ uint32_t warp_min<uint32_t>(uint32_t v) { return __reduce_min_sync(0xffffffffu, v); }
template <class B>
__device__ __forceinline__ B warp_max(B v) { return ~warp_min<B>(~v); }

template <class B>
__device__ __forceinline__ void prefetch_l2(const B* p, uint32_t len, uint32_t tid, uint32_t nt) {
  const char* const c = reinterpret_cast<const char*>(p);
  for (uint32_t i = tid * 128u; i < len * sizeof(B); i += nt * 128u) asm volatile("prefetch.global.L2 [%0];" ::"l"(c + i));
}

// Exclusive scan over the CTA of one value a thread; returns the sum through `total`.
template <int NT>
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* wsum, uint32_t& total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
    if ((int)lane >= o) inc += u;
  }
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  const uint32_t w = lane < NT / 32 ? wsum[lane] : 0u;
  total = __reduce_add_sync(0xffffffffu, w);
  const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u);
  __syncthreads();
  return inc - v + before;
}

template <class B>
struct MapSmem {
  uint32_t tab[kMaxCells + kMaxSub];  // samples per cell, then the map's table
  Part<B> part[kMaxParts];
  uint16_t node[kMaxCells + kMaxSub];  // the part that a cell is divided into (kNone: it is not)
  uint32_t weight[kMaxParts];          // two for each single value in the part
  uint32_t entry[kMaxParts], owner[kMaxParts];  // the part's own cell, and the part that that is in
  uint32_t before[kMaxParts], extra[kMaxParts];  // samples, and weights, in front of it
  uint32_t least[2][kMaxParts], greatest[2][kMaxParts];  // high and low words (32-bit keys: [0])
  uint32_t candidate[kCandidates][kMaxParts];  // indexes of samples
  uint32_t equal[kCandidates][kMaxParts];
  uint32_t cell2[kMaxCells];  // samples per cell by value
  B wmin[kCluster * kThreads / 32], wmax[kCluster * kThreads / 32];
  uint32_t wsum[kThreads / 32];
  unsigned long long spread[2][kThreads / 32];
  alignas(16) B sample[1];  // as many as the launch has room for
};
constexpr uint32_t kNone = 0xffffu, kWhole = 0xfffeu;  // no part; nor will there be one (the keys are equal)

// Latency: a chain of small steps by one CTA, 22 to 32 us at the first level of a large sort (its sample is read from HBM) and a few
// without one. Maps that divide cells take 40 us and more; a warp a part and four samples at a time took 100003 zipf words from 78 to
// 44 us.
// Makes the map of src[0, len) for about k ranges: sm.tab and sm.part are its tables, `bins` its ranges (at most bin_room(k));
// equal(bin, value) is called for each range that holds only keys equal to value. `salt` varies the sample. Every CTA that
// calls it with the same arguments makes the same map; the CL CTAs of a cluster read a part of the sample each and hand it round.
template <class T, uint32_t CL = 1, class F>
__device__ __forceinline__ void make_map(MapSmem<BOf<T>>& sm, const BOf<T>* src, uint32_t len, uint32_t k, uint32_t salt,
                                         uint32_t over_sample, uint32_t max_sample, KeyMap<T>& map, uint32_t& bins, F&& equal) {
  using B = BOf<T>;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t cells = cell_count(k);
  uint32_t S = over_sample * k;
  S = S < 1024u ? 1024u : S;
  S = S > max_sample ? max_sample : S;
  if (S > len) S = len;
  const uint32_t step = len / S;
  B mn = kmax<B>(), mx = B(0);
  namespace cg = cooperative_groups;
  const uint32_t rank = CL > 1u ? cg::this_cluster().block_rank() : 0u;
  const uint32_t i1 = S * (rank + 1u) / CL;
  if (CL > 1u) cg::this_cluster().sync();  // the others have started
  constexpr uint32_t U = CL > 1u ? 4u : 8u;  // loads under way at a time
  for (uint32_t i0 = S * rank / CL + tid; i0 < i1; i0 += U * kThreads) {
    B x[U];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      // one key at a pseudo-random place of each of S equal parts
      const uint32_t i = i0 + u * kThreads;
      uint32_t h = i * 2654435761u + salt * 40503u;
      h ^= h >> 15;
      h *= 0x85ebca6bu;
      if (i < i1) x[u] = KeyOps<T>::key(src[(uint32_t)(((unsigned long long)i * len) / S) + __umulhi(h, step)]);
    }
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t i = i0 + u * kThreads;
      if (i >= i1) break;
#pragma unroll
      for (uint32_t c = 0; c < CL; ++c) *(CL > 1u ? cg::this_cluster().map_shared_rank(&sm.sample[i], c) : &sm.sample[i]) = x[u];
      mn = x[u] < mn ? x[u] : mn;
      mx = x[u] > mx ? x[u] : mx;
    }
  }
  for (uint32_t i = tid; i < cells; i += kThreads) {
    sm.tab[i] = 0u;
    if (kFloating<T>) sm.cell2[i] = 0u;
  }
  mn = warp_min<B>(mn);
  mx = warp_max<B>(mx);
  if (lane < CL) {
    const uint32_t at = rank * (kThreads / 32) + warp;
    *(CL > 1u ? cg::this_cluster().map_shared_rank(&sm.wmin[at], lane) : &sm.wmin[at]) = mn;
    *(CL > 1u ? cg::this_cluster().map_shared_rank(&sm.wmax[at], lane) : &sm.wmax[at]) = mx;
  }
  if (CL > 1u) cg::this_cluster().sync();
  else __syncthreads();
  constexpr uint32_t kWarps = CL * kThreads / 32;
  mn = sm.wmin[lane & (kWarps - 1u)];
  mx = sm.wmax[lane & (kWarps - 1u)];
  for (uint32_t i = 32u + lane; i < kWarps; i += 32u) {
    mn = sm.wmin[i] < mn ? sm.wmin[i] : mn;
    mx = sm.wmax[i] > mx ? sm.wmax[i] : mx;
  }
  mn = warp_min<B>(mn);
  mx = warp_max<B>(mx);
  // one cell more at each end, for the keys outside the sample's
  map.lo = mn ? mn - 1u : mn;
  const B hi = mx != kmax<B>() ? mx + 1u : mx;
  map.span = hi - map.lo;
  const int over = bits_of(map.span) - (31 - __clz(cells));
  map.sh = over > 0 ? (uint32_t)over : 0u;
  map.top = (uint32_t)(map.span >> map.sh);
  map.used = map.top + 1u;
  map.kind = 0u;
  map.flo = map.scale = 0.f;
  if (mn == mx) {  // one value (so far): the keys below, equal, above
    bins = map.used;
    map.kind = PARTS;  // for the mark
    if (tid < map.used) sm.tab[tid] = tid | (map.lo + (B)tid == mn ? kEqual : 0u);
    if (tid == 0) equal((uint32_t)(mn - map.lo), mn);
    __syncthreads();
    return;
  }
  for (uint32_t i = tid; i < S; i += kThreads) atomicAdd(&sm.tab[map.template cell<false>(sm.sample[i])], 1u);
  if constexpr (kFloating<T>) {
    KeyMap<T> other = map;
    other.kind = BY_VALUE;
    other.used = cells;
    other.top = cells - 1u;
    other.lo = mn;
    other.span = mx - mn;
    other.flo = as_float<T>(mn);
    const float b = as_float<T>(mx), w = __fsub_rn(b, other.flo);
    other.scale = __fdiv_rn((float)cells, w);
    if (finite_span(other.flo, b, w) && other.scale < 3e38f) {  // the same in every thread
      for (uint32_t i = tid; i < S; i += kThreads) atomicAdd(&sm.cell2[other.template cell<true>(sm.sample[i])], 1u);
      __syncthreads();
      unsigned long long sq[2] = {0ull, 0ull};
      for (uint32_t i = tid; i < cells; i += kThreads) {
        sq[0] += (unsigned long long)sm.tab[i] * sm.tab[i];
        sq[1] += (unsigned long long)sm.cell2[i] * sm.cell2[i];
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        sq[0] += __shfl_xor_sync(0xffffffffu, sq[0], o);
        sq[1] += __shfl_xor_sync(0xffffffffu, sq[1], o);
      }
      if (lane == 0) {
        sm.spread[0][warp] = sq[0];
        sm.spread[1][warp] = sq[1];
      }
      __syncthreads();
      sq[0] = sq[1] = 0ull;
      for (int i = 0; i < kThreads / 32; ++i) {
        sq[0] += sm.spread[0][i];
        sq[1] += sm.spread[1][i];
      }
      if (sq[1] < sq[0]) {
        map = other;
        for (uint32_t i = tid; i < cells; i += kThreads) sm.tab[i] = sm.cell2[i];
      }
    }
  }
  const bool by_value = kFloating<T> && map.kind;
  __syncthreads();
  // Cells with the sample of 1.5 ranges and more are divided, and their parts again, twice. (A range may end with nearly a whole
  // cell more than its share: of the words of a pair sort, whose cells are that full more often, one in a few hundred ranges was
  // longer than kLocal then and cost its sort the persistent kernel, 33 us; theirs are divided from one range's sample on. Other
  // keys lose by more parts: 1.86 to 1.95 ms for 2^27 f32.)
  const uint32_t halves = KeyOps<T>::kIdentity && sizeof(B) == 8 && over_sample > kSmallOver ? 2u : 3u;
  constexpr uint32_t R = kMaxCells / kThreads;
  auto heavy = [&](uint32_t c) { return 2u * c * k >= halves * S; };
  uint32_t limit[4] = {0u, 0u, 0u, 0u};  // parts made by the end of each round
  uint32_t first = 0u, end = cells, rounds = 0u;
  for (uint32_t round = 0; round < 3u; ++round) {
    const uint32_t per = (end - first + kThreads - 1u) / kThreads, e0 = first + tid * per;
    uint32_t mine = 0u, total;
    for (uint32_t i = 0; i < per; ++i) {
      const uint32_t c = e0 + i < end ? sm.tab[e0 + i] : 0u;
      if (heavy(c) && !(round && sm.node[e0 + i] == kWhole)) mine += (1u << 16) + min(4u * (c * k / S) + 4u, kPartSub);
    }
    uint32_t at = block_scan<kThreads>(mine, sm.wsum, total);
    const uint32_t n0 = limit[round], n1 = min(n0 + (total >> 16), part_room(k));
    if (n1 == n0) break;
    ++rounds;
    limit[round + 1u] = n1;
    uint32_t last = min(end + (total & 0xffffu), cells + sub_room(k));
    for (uint32_t i = 0; i < per; ++i) {
      const uint32_t e = e0 + i;
      if (e >= end) break;
      const uint32_t c = sm.tab[e];
      uint32_t node = kNone;
      if (heavy(c) && !(round && sm.node[e] == kWhole)) {
        const uint32_t sub = min(4u * (c * k / S) + 4u, kPartSub), p = n0 + (at >> 16), from = end + (at & 0xffffu);
        at += (1u << 16) + sub;
        if (p < n1) {
          sm.entry[p] = e;
          sm.part[p].sub = from;
          sm.part[p].mult = from + sub <= last ? sub : 0u;  // 0: no room
          sm.weight[p] = 0u;
          sm.least[0][p] = sm.least[1][p] = ~0u;
          sm.greatest[0][p] = sm.greatest[1][p] = 0u;
#pragma unroll
          for (int j = 0; j < kCandidates; ++j) {
            sm.candidate[j][p] = ~0u;
            sm.equal[j][p] = 0u;
          }
          if (from + sub <= last) node = p;
        }
      }
      sm.node[e] = (uint16_t)node;
    }
    for (uint32_t i = end + tid; i < last; i += kThreads) {
      sm.tab[i] = 0u;
      sm.node[i] = (uint16_t)kNone;
    }
    __syncthreads();
    // f(i, x, p) for every sample i, x, that is in a part p of this round; four at a time, each a chain of dependent reads
    auto in_parts = [&](auto&& f) {
      for (uint32_t i0 = tid; i0 < S; i0 += 4u * kThreads) {
        B x[4];
        uint32_t p[4];
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u) {
          x[u] = sm.sample[i0 + u * kThreads < S ? i0 + u * kThreads : i0];
          p[u] = sm.node[by_value ? map.template cell<kFloating<T>>(x[u]) : map.template cell<false>(x[u])];
        }
        for (uint32_t r = 0; r < round; ++r)
#pragma unroll
          for (uint32_t u = 0; u < 4u; ++u)
            if (p[u] < n0) p[u] = sm.node[sm.part[p[u]].of(x[u])];
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u)
          if (p[u] < kWhole && i0 + u * kThreads < S) f(i0 + u * kThreads, x[u], p[u]);
      }
    };
    // The atomics are looked at first, as a part of many samples would keep them busy, and of 32 bits: a part's extremes are
    // found by high words first, then by low words.
    auto lower = [](uint32_t& m, uint32_t x) {
      if (x < *(volatile uint32_t*)&m) atomicMin(&m, x);
    };
    auto raise = [](uint32_t& m, uint32_t x) {
      if (x > *(volatile uint32_t*)&m) atomicMax(&m, x);
    };
    constexpr int kHigh = sizeof(B) == 8 ? 32 : 0;
    in_parts([&](uint32_t i, B x, uint32_t p) {
      // the first samples of four parts of the sample: a frequent value most likely
      lower(sm.candidate[i / kThreads % kCandidates][p], i);
      lower(sm.least[0][p], (uint32_t)(x >> kHigh));
      raise(sm.greatest[0][p], (uint32_t)(x >> kHigh));
    });
    __syncthreads();
    in_parts([&](uint32_t, B x, uint32_t p) {
#pragma unroll
      for (int j = 0; j < kCandidates; ++j)
        if (sm.candidate[j][p] != ~0u && x == sm.sample[sm.candidate[j][p]]) atomicAdd(&sm.equal[j][p], 1u);
      if (sizeof(B) == 8) {
        if ((uint32_t)(x >> kHigh) == sm.least[0][p]) lower(sm.least[1][p], (uint32_t)x);
        if ((uint32_t)(x >> kHigh) == sm.greatest[0][p]) raise(sm.greatest[1][p], (uint32_t)x);
      }
    });
    __syncthreads();
    for (uint32_t p = n0 + warp; p < n1; p += kThreads / 32) {
      Part<B> part = sm.part[p];
      const uint32_t e = sm.entry[p], sub = part.mult;
      if (!sub) continue;
      uint32_t most = 0u;
#pragma unroll
      for (int j = 0; j < kCandidates; ++j)
        if (sm.equal[j][p] > most) {
          most = sm.equal[j][p];
          part.lo = sm.sample[sm.candidate[j][p]];
        }
      if ((sm.tab[e] - most) * k <= S) {  // the others are a range at most
        part.mult = 0u;
        if (lane == 0) {
          sm.weight[p] = 2u;
          sm.node[part.sub + 1u] = (uint16_t)kWhole;
        }
      } else {
        auto whole = [&](const uint32_t (&w)[2][kMaxParts]) { return sizeof(B) == 8 ? (B)w[0][p] << kHigh | w[1][p] : (B)w[0][p]; };
        part.lo = whole(sm.least);
        part.span = whole(sm.greatest) - part.lo;
        const int bits = bits_of(part.span);
        part.right = bits > 32 ? (uint32_t)bits - 32u : 0u;
        part.left = bits < 32 ? 32u - (uint32_t)bits : 0u;
        const unsigned long long top = (unsigned long long)((uint32_t)(part.span >> part.right) << part.left) + 1ull;
        part.mult = (uint32_t)(((unsigned long long)sub << 32) / top);
      }
      // the part that this one's cell is in: the last of the round before whose cells start at or before it
      uint32_t o = 0u;
      if (round)
        for (uint32_t j = limit[round - 1u] + lane; j < n0; j += 32u)
          if (sm.node[sm.entry[j]] == j && sm.part[j].sub <= e) o = j + 1u;
      o = __reduce_max_sync(0xffffffffu, o);
      __syncwarp();
      if (lane == 0) {
        sm.part[p] = part;
        sm.owner[p] = o ? o - 1u : kNone;
      }
    }
    __syncthreads();
    in_parts([&](uint32_t, B x, uint32_t p) { atomicAdd(&sm.tab[sm.part[p].of(x)], 1u); });
    __syncthreads();
    first = end;
    end = last;
  }
  const uint32_t parts = limit[rounds];
  if (!parts) {
    const uint32_t per = cells > kThreads ? cells / kThreads : 1u, c0 = tid * per;
    uint32_t c[R], sum = 0u, total;
#pragma unroll
    for (uint32_t r = 0; r < R; ++r) {
      c[r] = r < per && c0 + r < cells ? sm.tab[c0 + r] : 0u;
      sum += c[r];
    }
    uint32_t before = block_scan<kThreads>(sum, sm.wsum, total);
#pragma unroll
    for (uint32_t r = 0; r < R; ++r) {
      if (r < per && c0 + r < cells) sm.tab[c0 + r] = before * k / S;
      before += c[r];
    }
    bins = k + 1u;
  } else {
    // A range starts wherever k / S of the samples in front make a whole number; a single value's range is its own (one
    // step before it and one behind it).
    for (uint32_t p = tid; p < parts; p += kThreads)
      if (sm.node[sm.entry[p]] == p && !sm.part[p].mult)
        for (uint32_t o = sm.owner[p]; o != kNone; o = sm.owner[o]) atomicAdd(&sm.weight[o], 2u);
    __syncthreads();
    const uint32_t per = cells > kThreads ? cells / kThreads : 1u, c0 = tid * per;
    auto sum_of = [&](uint32_t e) {
      const uint32_t p = sm.node[e];
      return sm.tab[e] + (p >= kWhole ? 0u : sm.weight[p] << 16);
    };
    auto settle = [&](uint32_t e, uint32_t before, uint32_t extra) {
      const uint32_t p = sm.node[e];
      if (p >= kWhole) {
        sm.tab[e] = before * k / S + extra;
      } else {
        sm.tab[e] = 0x80000000u | p;
        sm.before[p] = before;
        sm.extra[p] = extra;
      }
    };
    uint32_t sum = 0u, total;
    for (uint32_t r = 0; r < per; ++r)
      if (c0 + r < cells) sum += sum_of(c0 + r);
    uint32_t at = block_scan<kThreads>(sum, sm.wsum, total);
    for (uint32_t r = 0; r < per; ++r)
      if (c0 + r < cells) {
        const uint32_t c = sum_of(c0 + r);
        settle(c0 + r, at & 0xffffu, at >> 16);
        at += c;
      }
    for (uint32_t round = 0; round < rounds; ++round) {
      __syncthreads();
      for (uint32_t p = limit[round] + warp; p < limit[round + 1u]; p += kThreads / 32) {  // its cells 32 at a time
        if (sm.tab[sm.entry[p]] != (0x80000000u | p)) continue;
        const Part<B> part = sm.part[p];
        uint32_t in_front = sm.before[p] | (sm.extra[p] << 16);
        const uint32_t sub = part.mult ? part.of(kmax<B>()) - part.sub + 1u : 3u;
        for (uint32_t i0 = 0; i0 < sub; i0 += 32u) {
          const uint32_t i = i0 + lane, e = part.sub + i;
          const uint32_t c = i < sub ? sum_of(e) + (part.mult || i >= 2u ? 0u : 1u << 16) : 0u;
          uint32_t inc = c;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if ((int)lane >= o) inc += u;
          }
          const uint32_t front = in_front + inc - c;
          if (i < sub) settle(e, front & 0xffffu, front >> 16);
          if (!part.mult && i == 1u) {
            equal(sm.tab[e], part.lo);
            sm.tab[e] |= kEqual;
          }
          in_front += __shfl_sync(0xffffffffu, inc, 31);
        }
      }
    }
    bins = k + 1u + (total >> 16);
    map.kind |= PARTS | parts;
    map.used = end;
  }
  __syncthreads();
  if (!by_value && map.sh == 0u) {  // a range that is one cell of one value: nothing left to sort in it
    bool any = false;
    for (uint32_t i = tid; i <= map.top; i += kThreads) {
      const uint32_t b = sm.tab[i];
      auto apart = [&](uint32_t j) { return !(sm.tab[j] >> 31) && (sm.tab[j] & kBinMask) != b; };
      if (b < kEqual && (i == 0u ? map.lo == B(0) : apart(i - 1u)) && (i == map.top ? hi == kmax<B>() : apart(i + 1u))) {
        equal(b, map.lo + (B)i);
        sm.tab[i] = b | kEqual;  // (the others compare what kBinMask leaves)
        any = true;
      }
    }
    if (__syncthreads_or(any)) map.kind |= PARTS;
  }
  __syncthreads();
}

template <class T>
__global__ void __launch_bounds__(kThreads) split_map(const BOf<T>* src, Tables t, Level v, uint32_t plain_n, uint32_t levels,
                                                      uint32_t max_sample, Queue* q) {
  using B = BOf<T>;
  extern __shared__ __align__(16) unsigned char split_dyn[];
  MapSmem<B>& sm = *reinterpret_cast<MapSmem<B>*>(split_dyn);
  const uint32_t tid = threadIdx.x;
  pdl_wait();
  pdl_trigger();
  if (plain_n) {  // the first kernel of its sort, one CTA
    clear(q, sizeof(Queue));
    clear(t.ctl, sizeof(Ctl));
    __threadfence();
    __syncthreads();
  }
#ifdef GQS_PROFILE
  if (tid == 0) atomicCAS(&q->lvl_start, 0ull, (unsigned long long)global_timer_ns());
#endif
  if (ld_relaxed(&q->error)) return;  // set before this grid started, if at all: the same for every thread
  if (plain_n) {
    if (tid == 0) add_segment(t, v, 0ull, plain_n, range_count<B>(plain_n, levels > 1u));
    __threadfence();
    __syncthreads();
  }
  const uint32_t nseg = (uint32_t)(__ldcg(&t.ctl->alloc[v.index]) >> 32);
  for (uint32_t s = blockIdx.x; s < nseg; s += gridDim.x) {
    SegRec* const rec = v.seg + s;
    const uint32_t k = __ldcg(&rec->k), bin0 = __ldcg(&rec->bin0), cell0 = __ldcg(&rec->cell0);
    for (uint32_t i = tid; i < bin_room(k); i += kThreads) {
      v.bin[bin0 + i] = 0u;
      v.eq[bin0 + i] = 0u;
    }
    KeyMap<T> map;
    uint32_t bins;
    if (!GQS_OK(__ldcg(&rec->start) + __ldcg(&rec->len) <= t.n, q, 0xD207ull)) continue;
    make_map<T>(sm, src + __ldcg(&rec->start), __ldcg(&rec->len), k, s, kOver, max_sample, map, bins, [&](uint32_t b, B x) {
      if (!GQS_OK(b < bin_room(k), q, 0xD208ull)) return;
      v.eq[bin0 + b] = 1u;
      v.value[bin0 + b] = x;
    });
#ifdef GQS_CHECK
    map.q = q;
    map.bins = bins;
    map.check(__ldcg(&rec->cells), k);
#endif
    for (uint32_t i = tid; i < map.used; i += kThreads) v.cell[cell0 + i] = sm.tab[i];
    Part<B>* const out = static_cast<Part<B>*>(v.part) + bin0 / 4u;
    for (uint32_t i = tid; i < (map.kind & PART_COUNT); i += kThreads) out[i] = sm.part[i];
    if (tid == 0) {
      rec->lo = map.lo;
      rec->span = map.span;
      rec->sh = map.sh;
      rec->used = map.used;
      rec->top = map.top;
      rec->kind = map.kind;
      rec->flo = map.flo;
      rec->scale = map.scale;
      rec->bins = bins;
    }
    __syncthreads();
  }
}

// ---- tiles of the segments of a level --------------------------------------------------------
// The segment of tile `t`: the last one whose first tile is at most t.
__device__ __forceinline__ uint32_t find_segment(const SegRec* seg, uint32_t nseg, uint32_t t) {
  uint32_t lo = 0u, hi = nseg;
  while (hi - lo > 1u) {
    const uint32_t mid = (lo + hi) >> 1;
    if (seg[mid].tile0 <= t) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Every key's range, counted: reads the keys once. Bound by shared memory (a cell and a count each, seven wavefronts a row of 32)
// 62 to 70 % of the rate, half the copy bandwidth: 2^25 u32 in 35 to 40 us. Three CTAs on an SM hide its loads, eight under way a thread.
template <class T>
__global__ void __launch_bounds__(kThreads, 3) split_count(const BOf<T>* src, Tables t, Level v, Queue* q) {
  using B = BOf<T>;
  __shared__ uint32_t tab[kMaxCells + kMaxSub];
  __shared__ uint32_t cnt[kBinSlots];
  __shared__ Part<B> part[kMaxParts];
  const uint32_t tid = threadIdx.x;
  pdl_wait();
  pdl_trigger();
  if (ld_relaxed(&q->error)) return;
  const unsigned long long al = t.ctl->alloc[v.index];
  const uint32_t tile_keys = t.tile_keys;
  const uint32_t nseg = (uint32_t)(al >> 32), tiles = (uint32_t)al;
  const uint32_t t0 = (uint32_t)((unsigned long long)tiles * blockIdx.x / gridDim.x);
  const uint32_t t1 = (uint32_t)((unsigned long long)tiles * (blockIdx.x + 1u) / gridDim.x);
  if (t0 >= t1) return;
  uint32_t s = find_segment(v.seg, nseg, t0), tile = t0;
  while (tile < t1) {
    const SegRec r = v.seg[s];
    const uint32_t seg_tiles = (r.len + tile_keys - 1u) / tile_keys;
    const uint32_t end = r.tile0 + seg_tiles < t1 ? r.tile0 + seg_tiles : t1;
    KeyMap<T> map;
    map.load(r GQS_CHECK_ONLY(, q));
    __syncthreads();
    for (uint32_t i = tid; i < map.used; i += kThreads) tab[i] = v.cell[r.cell0 + i];
    for (uint32_t i = tid; i < (map.kind & PART_COUNT); i += kThreads) part[i] = static_cast<const Part<B>*>(v.part)[r.bin0 / 4u + i];
    for (uint32_t i = tid; i < r.bins; i += kThreads) cnt[i] = 0u;
    __syncthreads();
    // keys [k0, k1) of the segment
    const uint32_t k0 = (tile - r.tile0) * tile_keys;
    const uint32_t last = (end - r.tile0) * tile_keys, k1 = last < r.len ? last : r.len;
    const B* const p = src + r.start;
    by_kind<T>(map.kind, [&]<bool VALUE, bool PARTS_>() {
      constexpr uint32_t U = 8;
      uint32_t i = k0 + tid;
      for (; i + (U - 1u) * kThreads < k1; i += U * kThreads) {
        B x[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) x[u] = p[i + u * kThreads];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) atomicAdd(&cnt[map.template bin<VALUE, PARTS_>(KeyOps<T>::key(x[u]), tab, part) & kBinMask], 1u);
      }
      for (; i < k1; i += kThreads) atomicAdd(&cnt[map.template bin<VALUE, PARTS_>(KeyOps<T>::key(p[i]), tab, part) & kBinMask], 1u);
    });
    __syncthreads();
    for (uint32_t b = tid; b < r.bins; b += kThreads)
      if (cnt[b]) atomicAdd(&v.bin[r.bin0 + b], cnt[b]);
    tile = end;
    ++s;
  }
}

// One CTA a segment: where every range starts; the ranges become records of the on-chip sort, or
// segments of the next level.
template <class T>
__global__ void __launch_bounds__(kThreads) split_starts(Tables t, Level v, Level next, uint32_t levels, Queue* q) {
  using B = BOf<T>;
  __shared__ uint32_t wsum[kThreads / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  pdl_wait();
  pdl_trigger();
  if (ld_relaxed(&q->error)) return;
  const uint32_t nseg = (uint32_t)(t.ctl->alloc[v.index] >> 32);
  const bool more = v.index + 1u < levels;
  const uint32_t side = v.index == 0u ? (uint32_t)IN_DN : 0u;
  for (uint32_t s = blockIdx.x; s < nseg; s += gridDim.x) {
    const SegRec r = v.seg[s];
    if (tid == 0) {
      atomicAdd(&q->part_keys, (unsigned long long)r.len);
      atomicAdd(&q->part_jobs, 1u);
      atomicMax(&q->max_depth, v.index);
#ifdef GQS_PROFILE
      level_note(q, v.index, 0, r.len);
#endif
    }
    constexpr uint32_t R = (kBinSlots + kThreads - 1) / kThreads;
    uint32_t c[R], sum = 0u, total;
    bool still = false, moves = false;
#pragma unroll
    for (uint32_t i = 0; i < R; ++i) {
      const uint32_t b = tid * R + i;
      c[i] = b < r.bins ? __ldcg(&v.bin[r.bin0 + b]) : 0u;
      sum += c[i];
      if (!c[i]) continue;
      if (!v.eq[r.bin0 + b]) moves = true;
      else if (side && c[i] == r.len) still = true;
    }
    still = __syncthreads_or(still);
    moves = __syncthreads_or(moves);
    if (!moves && tid == 0) v.seg[s].bins = 0u;  // only equal keys: nothing to scatter
    if (still) {                                 // of one value, and already in d
      if (tid == 0) {
        atomicAdd(&q->total, (unsigned long long)r.len);
        atomicAdd(&q->done, (unsigned long long)r.len);
      }
      continue;
    }
    uint32_t at = block_scan<kThreads>(sum, wsum, total);
#pragma unroll
    for (uint32_t i = 0; i < R; ++i) {
      const uint32_t b = tid * R + i;
      const unsigned long long start = r.start + at;
      const bool eq = c[i] && v.eq[r.bin0 + b];
      if (b < r.bins) v.bin[r.bin0 + b] = at;
      const bool split_again = !eq && more && c[i] > Sizes<B>::kLocal;
      if (split_again && !add_segment(t, next, start, c[i], range_count<B>(c[i], false))) set_error(q, ST_INTERNAL, s);
      const uint32_t recs = !c[i] || split_again ? 0u : eq ? (c[i] + kCopyChunk - 1u) / kCopyChunk : 1u;
      uint32_t inc = recs;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if ((int)lane >= o) inc += u;
      }
      uint32_t first = 0u;
      if (lane == 31 && inc) first = atomicAdd(&t.ctl->buckets, inc);
      first = __shfl_sync(0xffffffffu, first, 31) + inc - recs;
      if (recs && !GQS_OK(first + recs <= t.buckets && start + c[i] <= r.start + r.len, q, 0xD209ull)) continue;
      for (uint32_t j = 0; j < recs; ++j) {
        const uint32_t off = j * kCopyChunk;
        t.bucket[first + j] = eq ? Bucket{start + off, c[i] - off < kCopyChunk ? c[i] - off : kCopyChunk, EQUAL, v.value[r.bin0 + b]}
                                 : Bucket{start, c[i], side, 0ull};
      }
      at += c[i];
    }
    __syncthreads();
  }
}

// ---- a tile's keys to their ranges --------------------------------------------------------------
template <class B>
struct TileSmem {
  alignas(16) B keys[Sizes<B>::kTile];
  uint32_t cnt[kBinSlots];
  uint32_t gbase[kBinSlots];
  uint32_t wsum[kThreads / 32];
  uint16_t bin[Sizes<B>::kTile];
};

// One tile: `here` keys in registers (row j, thread tid: key j * kThreads + tid). Counts them by range with one shared atomic
// each, reserves every range's share with reserve(range,
// count), groups the keys by range in shared memory, calls between(), then puts each key with put(range, first, key, index):
// the tile's part of the range is key indexes [.., ..) of the groups and starts at `first` - index of its first.
// The reservation's round trip to L2 is hidden behind the grouping, the next tile's loads (between) behind the writes.
// Bound by shared-memory wavefronts: of random cells and counters, a row of 32 keys takes about 3.5 for the cell, 2.5 for the
// count, 2.8 for the place, 3.5 for the write and 2 to 4 for reading back in order: 17 in all, 69 % of the rate at 2^25 u32 (96 us). A place from a second atomic (2.8)
// costs less than the counter's start read again (3.5), and leaves half the registers for what is remembered of each key: 2^28 u32
// 3.37 to 3.10 ms, 2^27 f32 1.87 to 1.72.
template <class T, bool VALUE, bool PARTS_, bool COUNT_EQUAL, class E, class Reserve, class Between, class Put>
__device__ __forceinline__ void scatter_tile(TileSmem<BOf<T>>& sm, const KeyMap<T>& map, const E* tab, const Part<BOf<T>>* part,
                                             uint32_t bins, const BOf<T> (&key)[Sizes<BOf<T>>::kTileRows], uint32_t here,
                                             Reserve&& reserve, Between&& between, Put&& put) {
  using B = BOf<T>;
  constexpr int ROWS = Sizes<B>::kTileRows;
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  // Without parts: the keys' ranges, two in a word, and a second atomic for their places, once the counters hold the ranges' starts.
  // With parts, where hot counters make atomics slow: (range << 16) | place in the tile's part of it. kLeft: not moved.
  uint32_t at[PARTS_ ? ROWS : ROWS / 2] = {};
  constexpr uint32_t kLeft = PARTS_ ? ~0u : 0xffffu;
  auto range_of = [&](int j) { return j & 1 ? at[j / 2] >> 16 : at[j / 2] & 0xffffu; };
  auto same_row = [&](uint32_t b) { return __all_sync(0xffffffffu, b == __shfl_sync(0xffffffffu, b, 0)); };
  const bool full = !PARTS_ && here == (uint32_t)ROWS * kThreads;
  uint32_t moved = here;
  bool runs = false;
  if constexpr (PARTS_) {
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      at[j] = kLeft;
      if ((uint32_t)j * kThreads + tid < here) {
        const uint32_t b = map.template bin<VALUE, PARTS_>(key[j], tab, part);
        if (b < kEqual) at[j] = (b << 16) | atomicAdd(&sm.cnt[b], 1u);
        else if (COUNT_EQUAL) atomicAdd(&sm.cnt[b & kBinMask], 1u << 16);
      }
    }
  } else if (full) {
#pragma unroll
    for (int j = 0; j < ROWS; j += 2)
      at[j / 2] = map.template bin<VALUE, PARTS_>(key[j], tab, part) | map.template bin<VALUE, PARTS_>(key[j + 1], tab, part) << 16;
    // 32 adds to one counter run one by one: where rows seem to be of one range each, one add a row
    const bool r0 = same_row(range_of(0)), r1 = same_row(range_of(ROWS / 2));
    runs = r0 || r1;
    if (!runs) {
#pragma unroll
      for (int j = 0; j < ROWS; ++j) atomicAdd(&sm.cnt[range_of(j)], 1u);
    } else {
#pragma unroll
      for (int j = 0; j < ROWS; ++j) {
        const uint32_t b = range_of(j);
        if (!same_row(b)) atomicAdd(&sm.cnt[b], 1u);
        else if (lane == 0) atomicAdd(&sm.cnt[b], 32u);
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      uint32_t b = kLeft;
      if ((uint32_t)j * kThreads + tid < here) {
        b = map.template bin<VALUE, PARTS_>(key[j], tab, part);
        atomicAdd(&sm.cnt[b], 1u);
      }
      at[j / 2] |= b << 16 * (j & 1);
    }
  }
  __syncthreads();
  // range tid * per + i in thread tid; the first one's reservation is under way while the keys are grouped
  const uint32_t per = (bins + kThreads - 1u) / kThreads, b0 = tid * per;
  uint32_t base0 = 0u, ex0;
  {
    // in a counter: the keys to move, and above them those that are only counted
    constexpr uint32_t kMoved = COUNT_EQUAL ? 0xffffu : ~0u;
    auto all = [](uint32_t c) { return COUNT_EQUAL ? (c & 0xffffu) + (c >> 16) : c; };
    uint32_t sum = 0u, total;
    for (uint32_t i = 0; i < per; ++i)
      if (b0 + i < bins) sum += sm.cnt[b0 + i] & kMoved;
    const uint32_t c0 = b0 < bins ? sm.cnt[b0] : 0u;
    if (c0) base0 = reserve(b0, all(c0));
    ex0 = block_scan<kThreads>(sum, sm.wsum, total);
    if (PARTS_) moved = total;
    uint32_t ex = ex0;
    for (uint32_t i = 0; i < per; ++i)
      if (b0 + i < bins) {
        const uint32_t c = sm.cnt[b0 + i];
        sm.cnt[b0 + i] = ex;
        if (i) sm.gbase[b0 + i] = c ? reserve(b0 + i, all(c)) - ex : 0u;
        ex += c & kMoved;
      }
  }
  __syncthreads();
  if constexpr (PARTS_) {
#pragma unroll
    for (int j = 0; j < ROWS; ++j)
      if (at[j] != kLeft) {
        const uint32_t i = sm.cnt[at[j] >> 16] + (at[j] & 0xffffu);
        if (!GQS_OK(i < here, map.q, 0xD20Aull)) continue;
        sm.keys[i] = key[j];
        sm.bin[i] = (uint16_t)(at[j] >> 16);  // cheaper than to find it again
      }
  } else if (full && !runs) {
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      const uint32_t i = atomicAdd(&sm.cnt[range_of(j)], 1u);
      if (GQS_OK(i < here, map.q, 0xD20Aull)) sm.keys[i] = key[j];
    }
  } else if (full) {
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      const uint32_t b = range_of(j);
      uint32_t i = 0u;
      if (!same_row(b)) {
        i = atomicAdd(&sm.cnt[b], 1u);
      } else {
        if (lane == 0) i = atomicAdd(&sm.cnt[b], 32u);
        i = __shfl_sync(0xffffffffu, i, 0) + lane;
      }
      if (GQS_OK(i < here, map.q, 0xD20Aull)) sm.keys[i] = key[j];
    }
  } else {
#pragma unroll
    for (int j = 0; j < ROWS; ++j)
      if (range_of(j) != kLeft) {
        const uint32_t i = atomicAdd(&sm.cnt[range_of(j)], 1u);
        if (GQS_OK(i < here, map.q, 0xD20Aull)) sm.keys[i] = key[j];
      }
  }
  if (b0 < bins) sm.gbase[b0] = base0 - ex0;
  between();
  __syncthreads();
  auto one = [&](uint32_t i) {
    const B k = sm.keys[i];
    const uint32_t b = PARTS_ ? sm.bin[i] : map.template bin<VALUE, PARTS_>(k, tab, part);
    put(b, sm.gbase[b] + i, k);
  };
  if (full) {
#pragma unroll
    for (int j = 0; j < ROWS; ++j) one((uint32_t)j * kThreads + tid);
  } else {
#pragma unroll 1
    for (uint32_t i = tid; i < moved; i += kThreads) one(i);
  }
}

template <class B>
struct ScatterSmem {
  TileSmem<B> tile;
  uint16_t tab[kMaxCells + kMaxSub];
  Part<B> part[kMaxParts];
};

template <class T>
__global__ void __launch_bounds__(kThreads, kTileCtas) split_scatter(const BOf<T>* src, BOf<T>* dst, Tables t, Level v, Queue* q) {
  using B = BOf<T>;
  constexpr int ROWS = Sizes<B>::kTileRows;
  extern __shared__ __align__(16) unsigned char split_dyn[];
  ScatterSmem<B>& sm = *reinterpret_cast<ScatterSmem<B>*>(split_dyn);
  const uint32_t tid = threadIdx.x;
  pdl_wait();
  pdl_trigger();
  if (ld_relaxed(&q->error)) return;
  const unsigned long long al = t.ctl->alloc[v.index];
  const uint32_t tile_keys = t.tile_keys;
  const uint32_t nseg = (uint32_t)(al >> 32), tiles = (uint32_t)al;
  const uint32_t t0 = (uint32_t)((unsigned long long)tiles * blockIdx.x / gridDim.x);
  const uint32_t t1 = (uint32_t)((unsigned long long)tiles * (blockIdx.x + 1u) / gridDim.x);
  if (t0 >= t1) return;
  uint32_t s = find_segment(v.seg, nseg, t0), seg_t0 = v.seg[s].tile0, seg_len = v.seg[s].len;
  unsigned long long start = v.seg[s].start;
  uint32_t bins = 0u, len;
  uint32_t* cursor = nullptr;
  B* out = nullptr;
  KeyMap<T> map;
  B key[ROWS];
  auto load = [&](uint32_t tile) {
    const uint32_t k0 = (tile - seg_t0) * tile_keys;
    len = seg_len - k0 < tile_keys ? seg_len - k0 : tile_keys;
    const B* const p = src + start + k0 + tid;
    if (len == (uint32_t)ROWS * kThreads) {
#pragma unroll
      for (int j = 0; j < ROWS; ++j) key[j] = KeyOps<T>::key(p[j * kThreads]);
    } else {
#pragma unroll
      for (int j = 0; j < ROWS; ++j)
        if ((uint32_t)j * kThreads + tid < len) key[j] = KeyOps<T>::key(p[j * kThreads]);
    }
  };
  load(t0);
  bool fresh = true;  // the tile is of another segment than the one before
  auto advance = [&](uint32_t tile) {
    fresh = false;
    if (tile + 1u >= t1) return;
    const uint32_t seg_end = seg_t0 + (seg_len + tile_keys - 1u) / tile_keys;
    if (tile + 1u == seg_end) {
      ++s;
      seg_t0 = seg_end;
      seg_len = v.seg[s].len;
      start = v.seg[s].start;
      fresh = true;
    }
    load(tile + 1u);
  };
  for (uint32_t tile = t0; tile < t1; ++tile) {
    if (fresh) {
      const SegRec* const r = v.seg + s;
      map.load(*r GQS_CHECK_ONLY(, q));
      bins = r->bins;
      cursor = v.bin + r->bin0;
      out = dst + start;
      const uint32_t* const cell = v.cell + r->cell0;
      __syncthreads();
      for (uint32_t i = tid; i < map.used; i += kThreads) sm.tab[i] = KeyMap<T>::narrow(cell[i]);
      for (uint32_t i = tid; i < (map.kind & PART_COUNT); i += kThreads) sm.part[i] = static_cast<const Part<B>*>(v.part)[r->bin0 / 4u + i];
    }
    if (!bins) {  // equal keys only, which need not move
      advance(tile);
      continue;
    }
    for (uint32_t i = tid; i < bins; i += kThreads) sm.tile.cnt[i] = 0u;
    __syncthreads();
    const uint32_t here = len;
    B* const to = out;
    uint32_t* const cur = cursor;
    GQS_CHECK_ONLY(const uint32_t keys = seg_len;)
    by_kind<T>(map.kind, [&]<bool VALUE, bool PARTS_>() {
      scatter_tile<T, VALUE, PARTS_, false>(
          sm.tile, map, sm.tab, sm.part, bins, key, here, [&](uint32_t b, uint32_t c) { return atomicAdd(cur + b, c); },
          [&] { advance(tile); },
          [&](uint32_t, uint32_t at, B k) {
            if (GQS_OK(at < keys, q, 0xD20Bull)) to[at] = KeyOps<T>::raw(k);
          });
    });
  }
  if (tid == 0) atomicAdd(&q->chunks, (unsigned long long)(t1 - t0));
}

// ---- small plain sorts: map and scatter in one kernel, into ranges with room for kLocal keys each --------------
template <class B>
union SmallSmem {
  char all[sizeof(MapSmem<B>) + Sizes<B>::kSmallSample * sizeof(B)];
  MapSmem<B> map;
  struct {
    uint32_t tab[kMaxCells + kMaxSub];  // where the map leaves its tables
    Part<B> part[kMaxParts];
    TileSmem<B> tile;
  } s;
};

template <class T, uint32_t CL>
__global__ void __cluster_dims__(CL) __launch_bounds__(kThreads, kTileCtas) split_small(const BOf<T>* src, BOf<T>* area, uint32_t n, uint32_t k, Small* st, uint32_t tile_keys,
                                                                 Queue* q) {
  using B = BOf<T>;
  constexpr int ROWS = Sizes<B>::kTileRows;
  constexpr uint32_t LT = Sizes<B>::kLocal;
  extern __shared__ __align__(16) unsigned char split_dyn[];
  SmallSmem<B>& sm = *reinterpret_cast<SmallSmem<B>*>(split_dyn);
  const uint32_t tid = threadIdx.x;
  pdl_wait();
  pdl_trigger();
  const uint32_t tiles = (n + tile_keys - 1u) / tile_keys;
  KeyMap<T> map;
  uint32_t bins;
  if (blockIdx.x < tiles) {  // read while the map is made
    const uint32_t k0 = blockIdx.x * tile_keys, here = n - k0 < tile_keys ? n - k0 : tile_keys;
    prefetch_l2(src + k0, here, tid, kThreads);
  }
  // (there are two tiles at least, so there is a CTA 1)
  if (blockIdx.x == 0) clear(st->eq, bin_room(k) * 4);
  if (blockIdx.x == 1) clear(q, sizeof(Queue));
  make_map<T, CL>(sm.map, src, n, k, 0u, kSmallOver, Sizes<B>::kSmallSample, map, bins, [&](uint32_t b, B x) {
    if (blockIdx.x == 0 && GQS_OK(b < bin_room(k), q, 0xD208ull)) {
      st->eq[b] = 1u;
      st->value[b] = x;
    }
  });
#ifdef GQS_CHECK
  map.q = q;
  map.bins = bins;
  map.check(cell_count(k) + sub_room(k), k);
  bins = map.bins;
#endif
  if (blockIdx.x == 0 && tid == 0) {
    st->bins = bins;
    st->left = 0ull;
  }
  if (blockIdx.x == 1 && tid == 0) {
    q->part_keys = n;
    q->part_jobs = 1u;
    q->chunks = tiles;
#ifdef GQS_PROFILE
    q->lvl_start = (unsigned long long)global_timer_ns();
    level_note(q, 0, 0, n);
#endif
  }
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const uint32_t k0 = tile * tile_keys, here = n - k0 < tile_keys ? n - k0 : tile_keys;
    B key[ROWS];
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      const uint32_t i = (uint32_t)j * kThreads + tid;
      if (i < here) key[j] = KeyOps<T>::key(src[k0 + i]);
    }
    for (uint32_t i = tid; i < bins; i += kThreads) sm.s.tile.cnt[i] = 0u;
    __syncthreads();
    by_kind<T>(map.kind, [&]<bool VALUE, bool PARTS_>() {
      scatter_tile<T, VALUE, PARTS_, PARTS_>(
          sm.s.tile, map, sm.s.tab, sm.s.part, bins, key, here,
          [&](uint32_t b, uint32_t c) { return atomicAdd(&st->cursor[b], c); }, [] {},
          [&](uint32_t b, uint32_t at, B x) {
            // keys past the room are dropped: local_small sees that the range is too long and leaves the sort (its keys are
            // still in d) to the persistent kernel
            if (at < LT && GQS_OK(b < bin_room(k), q, 0xD20Cull)) area[(size_t)b * LT + at] = KeyOps<T>::raw(x);
          });
    });
    __syncthreads();
  }
}

// ---- the on-chip sort of a range ------------------------------------------------------------------
// Sorting networks over registers (Batcher's odd-even merge).
template <class K>
__device__ __forceinline__ void order2(K& a, K& b) {
  const K lo = a < b ? a : b, hi = a < b ? b : a;
  a = lo;
  b = hi;
}
template <class K>
__device__ __forceinline__ void sort4(K* v) {
  order2(v[0], v[1]); order2(v[2], v[3]);
  order2(v[0], v[2]); order2(v[1], v[3]);
  order2(v[1], v[2]);
}
template <class K>
__device__ __forceinline__ void merge8(K* v) {  // v[0, 4) and v[4, 8) are sorted
#pragma unroll
  for (int i = 0; i < 4; ++i) order2(v[i], v[i + 4]);
  order2(v[2], v[4]); order2(v[3], v[5]);
  order2(v[1], v[2]); order2(v[3], v[4]); order2(v[5], v[6]);
}
template <class K>
__device__ __forceinline__ void merge16(K* v) {  // v[0, 8) and v[8, 16) are sorted
#pragma unroll
  for (int i = 0; i < 8; ++i) order2(v[i], v[i + 8]);
#pragma unroll
  for (int i = 4; i < 8; ++i) order2(v[i], v[i + 4]);
#pragma unroll
  for (int i = 2; i < 12; i += 4) {
    order2(v[i], v[i + 2]);
    order2(v[i + 1], v[i + 3]);
  }
#pragma unroll
  for (int i = 1; i < 15; i += 2) order2(v[i], v[i + 1]);
}
template <int W, class K>
__device__ __forceinline__ void merge_block(K* v) {
  static_assert(W == 8 || W == 16, "networks of 8 and 16 keys");
  if constexpr (W == 8) merge8(v);
  else merge16(v);
}
template <int W, class K>
__device__ __forceinline__ void sort_block(K* v) {
#pragma unroll
  for (int h = 0; h < W; h += 8) {
    sort4(v + h);
    sort4(v + h + 4);
    merge8(v + h);
  }
  if constexpr (W == 16) merge16(v);
}

template <class B>
struct LocalSmem {
  // Blocks of kBlock keys. The 16-byte pieces of each are permuted by its number, so that eight lanes that read the same piece of
  // neighbouring blocks meet different banks.
  alignas(128) B keys[Sizes<B>::kLocal];
  alignas(16) uint32_t cur[Sizes<B>::kLocal / 2];  // the bins' counters, two in each word
  B wmin[Sizes<B>::kSortThreads / 32], wmax[Sizes<B>::kSortThreads / 32];
  uint32_t wsum[Sizes<B>::kSortThreads / 32];
  uint32_t most;
  static constexpr uint32_t kTodos = Sizes<B>::kLocal / (Sizes<B>::kShortBin + 1) + 2, kBigs = Sizes<B>::kLocal / (kWarpBin + 1) + 1;
  uint32_t todos;            // bins for a warp each
  uint16_t todo[kTodos];
  uint32_t bigs, big[kBigs];  // bins for the CTA, later: (first key << 16) | keys
  static constexpr uint32_t V = 16 / sizeof(B), kPieces = Sizes<B>::kBlock / V;  // keys of a piece, pieces of a block
  static __device__ __forceinline__ uint32_t slot(uint32_t i) { return i ^ ((i / V >> 3 & (kPieces - 1u)) * V); }
  __device__ __forceinline__ uint4* piece(uint32_t b, uint32_t i) {
    return reinterpret_cast<uint4*>(keys) + (b * kPieces + i ^ (b * kPieces >> 3 & (kPieces - 1u)));
  }
};

// f(j) for every row j, of NT keys each, in which this thread has one of `len` keys: four full rows at a time need no test for each.
// (Recursion, not a loop: around a loop that ends early the compiler kept the keys in local memory.)
template <int ROWS, uint32_t NT, int J = 0, class F>
__device__ __forceinline__ void for_rows(uint32_t len, F&& f) {
  static_assert(ROWS % 4 == 0, "whole groups");
  if constexpr (J < ROWS) {
    if ((uint32_t)(J + 4) * NT <= len) {
      f(J);
      f(J + 1);
      f(J + 2);
      f(J + 3);
      for_rows<ROWS, NT, J + 4>(len, f);
    } else {
      const uint32_t i = (uint32_t)J * NT + threadIdx.x;
      if (i < len) f(J);
      if (i + NT < len) f(J + 1);
      if (i + 2u * NT < len) f(J + 2);
      if (i + 3u * NT < len) f(J + 3);
    }
  }
}

// The keys of a range while it is sorted: less its least, mn. The words of a pair sort are a key above a value, and the values
// seldom fill their 32 bits: the bits that no value of the range has are left out, so that equal steps of the result do not leave
// the bins between two keys empty.
template <class T>
struct Near {
  using B = BOf<T>;
  static constexpr bool kWords = KeyOps<T>::kIdentity && sizeof(B) == 8;
  B mn;
  uint32_t width;  // of the values
  __device__ __forceinline__ B in(B x) const {
    if constexpr (kWords) return (((x >> 32) - (mn >> 32)) << width | (uint32_t)x) - (uint32_t)mn;
    else return x - mn;
  }
  __device__ __forceinline__ B out(B y) const {
    if constexpr (kWords) {
      y += (uint32_t)mn;
      return ((y >> width) + (mn >> 32)) << 32 | (y & ((B(1) << width) - 1u));
    } else {
      return y + mn;
    }
  }
};

// How a range's keys (less its least, mn) fall into bins: equal steps of the integer, or of the value.
template <class T>
struct BinMap {
  using B = BOf<T>;
  B mn;
  uint32_t bins, sh, mult;  // (x >> sh) * mult / 2^32, or x itself (mult 0)
  float flo, scale;
  bool by_value;
  // `range`: hi, less lo. `key`: one of the range's keys, if `has`.
  __device__ __forceinline__ BinMap(B lo, B hi, B range, uint32_t n, bool first, B key, bool has) : mn(lo), bins(n), flo(0.f), scale(0.f), by_value(false) {
    const int over = bits_of(range) - 32;
    sh = over > 0 ? (uint32_t)over : 0u;
    const uint32_t top = (uint32_t)(range >> sh);
    // rounded down far enough that no bin is past the last
    mult = top < bins ? 0u : __float2uint_rz(__fmul_rn(__fdiv_rn((float)bins, __fadd_rn((float)top, 1.f)), 4294963200.f));
    if constexpr (kFloating<T>) {
      // keys on both sides of zero, or of many exponents: equal steps of the integer would leave most bins empty
      constexpr int kExpShift = sizeof(B) == 8 ? 52 : 23;
      const B zero = B(1) << (sizeof(B) * 8 - 1);
      if (first && ((lo < zero && hi >= zero) || (range >> kExpShift) > 3u)) {
        flo = as_float<T>(lo);
        const float b = as_float<T>(hi), w = __fsub_rn(b, flo);
        scale = __fdiv_rn((float)bins * 0.99999f, w);
        by_value = finite_span(flo, b, w) && scale < 3e38f;
        if (by_value) {
          // the one that has nearer to a half of these keys in the middle half of its bins
          auto off = [&](uint32_t bin) {
            const int in = __syncthreads_count(has && bin >= n / 4u && bin < n / 4u * 3u);
            return 2 * in;
          };
          const int all = __syncthreads_count(has);
          by_value = abs(off(of<true>(key - lo)) - all) <= abs(off(of<false>(key - lo)) - all);
        }
      }
    }
  }
  template <bool VALUE>
  __device__ __forceinline__ uint32_t of(B x) const {
    if constexpr (VALUE) {
      const uint32_t u = __float2uint_rz(__fmul_rn(__fsub_rn(as_float<T>(x + mn), flo), scale));
      return u < bins ? u : bins - 1u;
    } else {
      const uint32_t y = (uint32_t)(x >> sh);
      return mult ? __umulhi(y, mult) : y;
    }
  }
  __device__ __forceinline__ uint32_t any(B x) const {
    if (kFloating<T> && by_value) return of<kFloating<T>>(x);
    return of<false>(x);
  }
};

// Bound by shared-memory wavefronts and issue slots together (21 wavefronts and 84 instructions a row of 32 keys, 59 % and 56 % of their rates at 2^25 u32): count 2.5,
// place 2.8 and write 3.5 of them, networks 4, counters 2. Two counters share a word, eight are scanned with one 16-byte access, and
// blocks are permuted, not padded: 30 to 21 wavefronts, 101 to 84 instructions, 2^28 u32 3.62 to 3.37 ms, 2^20 43.6 to 35.3 us.
// 64-bit keys use networks of eight and two bins a key (a comparison is six instructions): 2^26 f64 2.00 to 1.87 ms.
// Sorts `len` keys (row j, thread tid: key j * NT + tid, as the map orders them) into dst[off, off + len). Calls between() once
// the keys have left their registers. Every bin holds about one key, so after one counting pass each key is close to its place, and
// networks over neighbouring blocks finish the order without knowing the bins.
template <class T, class Between>
__device__ __forceinline__ void sort_bins(LocalSmem<BOf<T>>& sm, BOf<T> (&key)[Sizes<BOf<T>>::kLocalRows], uint32_t len, BOf<T>* dst,
                                          uint32_t off, bool first, Queue* q, Between&& between) {
  using B = BOf<T>;
  using S = LocalSmem<B>;
  constexpr int ROWS = Sizes<B>::kLocalRows;
  constexpr uint32_t NT = Sizes<B>::kSortThreads, LT = Sizes<B>::kLocal, kShortBin = Sizes<B>::kShortBin;
  constexpr int W = Sizes<B>::kBlock;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  dst += off;
  B mn = kmax<B>(), mx = B(0);
  uint32_t values = 0u;
  for_rows<ROWS, NT>(len, [&](int j) {
    mn = key[j] < mn ? key[j] : mn;
    mx = key[j] > mx ? key[j] : mx;
    if (Near<T>::kWords) values |= (uint32_t)key[j];
  });
  mn = warp_min<B>(mn);
  mx = warp_max<B>(mx);
  if (Near<T>::kWords) values = __reduce_or_sync(0xffffffffu, values);
  __syncthreads();  // the range before has left shared memory
  if (lane == 0) {
    sm.wmin[warp] = mn;
    sm.wmax[warp] = mx;
    if (Near<T>::kWords) sm.wsum[warp] = values;
  }
  // bins: a power of two, at least as many as keys
  constexpr uint32_t kMinBins = 8u * NT < LT ? 8u * NT : LT;
  const uint32_t some = 16u / W * len;
  const uint32_t bins = 1u << ceil_log2(some < kMinBins ? kMinBins : some < LT ? some : LT);
  for (uint32_t i = tid; i < bins / 8u; i += NT) reinterpret_cast<uint4*>(sm.cur)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (tid == 0) {
    sm.most = 0u;
    sm.todos = 0u;
  }
  __syncthreads();
  mn = warp_min<B>(sm.wmin[lane & (NT / 32 - 1)]);
  mx = warp_max<B>(sm.wmax[lane & (NT / 32 - 1)]);
  Near<T> near{mn, 0u};
  if (Near<T>::kWords) near.width = (uint32_t)bits_of(__reduce_or_sync(0xffffffffu, sm.wsum[lane & (NT / 32 - 1)]));
  const BinMap<T> map(mn, mx, near.in(mx), bins, first, key[0], tid < len);
  auto count = [&]<bool VALUE>() {
    for_rows<ROWS, NT>(len, [&](int j) {
      key[j] = near.in(key[j]);
      const uint32_t b = map.template of<VALUE>(key[j]);
      if (GQS_OK(b < bins, q, 0xD20Dull)) atomicAdd(&sm.cur[b >> 1], b & 1u ? 0x10000u : 1u);
    });
  };
  if (kFloating<T> && map.by_value) count.template operator()<kFloating<T>>();
  else count.template operator()<false>();
  __syncthreads();
  {
    // exclusive scan in place: a warp has bins / (NT / 32) consecutive counters, 256 at a time (8 a lane, in one 16-byte word)
    constexpr uint32_t CH = LT / (8u * NT);
    uint4* const mine = reinterpret_cast<uint4*>(sm.cur) + warp * (bins / NT * 4u) + lane;
    const uint32_t ch = bins / (8u * NT);
    uint32_t before[CH], run = 0u, most = 0u;
    // halves of x: c0 and c1; of pair(x): c0 and c0 + c1
    auto pair = [](uint32_t x) { return x * 0x10001u; };
#pragma unroll
    for (uint32_t i = 0; i < CH; ++i) {
      if (i >= ch) break;
      const uint4 w = mine[i * 32u];
      most = __vmaxu2(most, __vmaxu2(__vmaxu2(w.x, w.y), __vmaxu2(w.z, w.w)));
      const uint32_t sum = pair(w.x + w.y + w.z + w.w) >> 16;  // (at most kLocal: no half carries into the other)
      uint32_t inc = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if ((int)lane >= o) inc += u;
      }
      before[i] = run + inc - sum;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    most = __reduce_max_sync(0xffffffffu, max(most >> 16, most & 0xffffu));
    if (lane == 0) {
      sm.wsum[warp] = run;
      if (most > kShortBin) atomicMax(&sm.most, most);
    }
    __syncthreads();
    const uint32_t up = __reduce_add_sync(0xffffffffu, lane < warp ? sm.wsum[lane] : 0u);
#pragma unroll
    for (uint32_t i = 0; i < CH; ++i) {
      if (i >= ch) break;
      uint32_t e = pair(up + before[i]);  // in both halves
      auto next = [&](uint32_t x) {
        const uint32_t v = e + (x << 16);
        e += pair(pair(x) >> 16);
        return v;
      };
      const uint4 w = mine[i * 32u];
      uint4 v;
      v.x = next(w.x);
      v.y = next(w.y);
      v.z = next(w.z);
      v.w = next(w.w);
      mine[i * 32u] = v;
    }
  }
  __syncthreads();
  auto place = [&]<bool VALUE>() {
    for_rows<ROWS, NT>(len, [&](int j) {
      const uint32_t b = map.template of<VALUE>(key[j]);
      if (!GQS_OK(b < bins, q, 0xD20Dull)) return;
      const uint32_t old = atomicAdd(&sm.cur[b >> 1], b & 1u ? 0x10000u : 1u);
      if (!GQS_OK((b & 1u ? old >> 16 : old & 0xffffu) < len, q, 0xD20Eull)) return;
      sm.keys[S::slot(b & 1u ? old >> 16 : old & 0xffffu)] = key[j];
    });
  };
  if (kFloating<T> && map.by_value) place.template operator()<kFloating<T>>();
  else place.template operator()<false>();
  const uint32_t blocks = (len + W - 1u) / W;
  if (tid < blocks * W - len) sm.keys[S::slot(len + tid)] = kmax<B>();
  const bool longs = sm.most > kShortBin;
  between();
  __syncthreads();
  // cur[b] is now the end of bin b
  if (longs) {
    // Long bins: those of equal keys are in order as they are, the others are sorted by a warp each.
    constexpr uint32_t kMixed = 0x8000u;
    static_assert(LT < kMixed, "a counter's bits below the mark");
    volatile uint16_t* const ends = reinterpret_cast<volatile uint16_t*>(sm.cur);
    auto end_of = [&](uint32_t b) { return ends[b] & (kMixed - 1u); };
    auto first_of = [&](uint32_t b) { return b ? end_of(b - 1u) : 0u; };
    auto mark = [&](uint32_t b) {  // whether it was marked before
      const uint32_t m = kMixed << (16u * (b & 1u));
      return (atomicOr(&sm.cur[b >> 1], m) & m) != 0u;
    };
    for (uint32_t i = tid; i < len; i += NT) {
      const B k = sm.keys[S::slot(i)];
      const uint32_t b = map.any(k), s = first_of(b);
      if (end_of(b) - s > kShortBin && k != sm.keys[S::slot(s)] && !mark(b)) {
        const uint32_t n = end_of(b) - s;
        if (!GQS_OK(s + n <= len, q, 0xD20Full)) continue;
        const uint32_t to = atomicAdd(n <= kWarpBin ? &sm.todos : &sm.bigs, 1u);
        if (!GQS_OK(to < (n <= kWarpBin ? S::kTodos : S::kBigs), q, 0xD20Full)) continue;
        if (n <= kWarpBin) sm.todo[to] = (uint16_t)b;
        else sm.big[to] = ((off + s) << 16) | n;
      }
    }
    __syncthreads();
    const uint32_t m = GQS_OK(sm.todos <= S::kTodos, q, 0xD20Full) ? sm.todos : 0u;
    for (uint32_t t = warp; t < m; t += NT / 32) {
      const uint32_t b = sm.todo[t], s = first_of(b), n = end_of(b) - s;
      auto sort_bin = [&]<int R>() {
        B v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = r * 32u + lane < n ? sm.keys[S::slot(s + r * 32u + lane)] : kmax<B>();
        warp_bitonic<R>(v);
        __syncwarp();
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (lane * R + r < n) sm.keys[S::slot(s + lane * R + r)] = v[r];
      };
      if (n <= 32u) sort_bin.template operator()<1>();
      else if (n <= 64u) sort_bin.template operator()<2>();
      else if (n <= 128u) sort_bin.template operator()<4>();
      else sort_bin.template operator()<8>();
    }
    __syncthreads();
  }
  // Every other key is within W / 2 places of its own: blocks of W, then the halves that meet between them.
  constexpr int V = S::V, P = W / V;
  for (uint32_t b = tid; b < blocks; b += NT) {
    B v[W];
#pragma unroll
    for (int i = 0; i < P; ++i) *reinterpret_cast<uint4*>(&v[i * V]) = *sm.piece(b, i);
    sort_block<W>(v);
#pragma unroll
    for (int i = 0; i < P; ++i) *sm.piece(b, i) = *reinterpret_cast<const uint4*>(&v[i * V]);
  }
  __syncthreads();
  for (uint32_t b = tid; b + 1u < blocks; b += NT) {
    B v[W];
#pragma unroll
    for (int i = 0; i < P / 2; ++i) {
      *reinterpret_cast<uint4*>(&v[i * V]) = *sm.piece(b, P / 2 + i);
      *reinterpret_cast<uint4*>(&v[W / 2 + i * V]) = *sm.piece(b + 1u, i);
    }
    merge_block<W>(v);
#pragma unroll
    for (int i = 0; i < P / 2; ++i) {
      *sm.piece(b, P / 2 + i) = *reinterpret_cast<const uint4*>(&v[i * V]);
      *sm.piece(b + 1u, i) = *reinterpret_cast<const uint4*>(&v[W / 2 + i * V]);
    }
  }
  __syncthreads();
  const B* const mine = &sm.keys[S::slot(tid)];
  static_assert(NT % 128u == 0u, "slot(i + NT) is slot(i) + NT");
  B* const to = dst + tid;
  for_rows<ROWS, NT>(len, [&](int j) { to[j * NT] = KeyOps<T>::raw(near.out(mine[j * NT])); });
}

// v = *p where `use`: as inline code, so that the loads stay one behind the other with nothing between them.
__device__ __forceinline__ void load_if(uint32_t& v, const uint32_t* p, bool use) {
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q ld.global.u32 %0, [%1];\n}" : "+r"(v) : "l"(p), "r"((uint32_t)use) : "memory");
}
__device__ __forceinline__ void load_if(uint64_t& v, const uint64_t* p, bool use) {
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q ld.global.u64 %0, [%1];\n}" : "+l"(v) : "l"(p), "r"((uint32_t)use) : "memory");
}

template <class B>
__device__ __forceinline__ void load_range(const B* p, uint32_t len, B (&raw)[Sizes<B>::kLocalRows]) {
  const B* const mine = p + threadIdx.x;
#pragma unroll
  for (int j = 0; j < Sizes<B>::kLocalRows; j += 4) {
    if ((uint32_t)j * Sizes<B>::kSortThreads >= len) break;
#pragma unroll
    for (int u = j; u < j + 4; ++u)
      load_if(raw[u], mine + u * Sizes<B>::kSortThreads, (uint32_t)u * Sizes<B>::kSortThreads + threadIdx.x < len);
  }
}

// Sorts a range of `len` keys into dst (see sort_bins), with the longest bins that it leaves, each as a range of its own: its
// two extremes fall into different bins then, of keys 2^11 times closer together, so there are at most six rounds.
// Returns whether there were any (the keys that between() loaded are then lost).
template <class T, class Between>
__device__ __forceinline__ bool sort_range(LocalSmem<BOf<T>>& sm, BOf<T> (&key)[Sizes<BOf<T>>::kLocalRows], uint32_t len, BOf<T>* dst,
                                           Queue* q, Between&& between) {
  using B = BOf<T>;
  if (threadIdx.x == 0) sm.bigs = 0u;
  sort_bins<T>(sm, key, len, dst, 0u, true, q, between);
  if (sm.most <= kWarpBin) return false;
  bool again = false;
  while (true) {
    __syncthreads();  // every thread has read what changes below, and sees the keys in dst
    const uint32_t m = GQS_OK(sm.bigs <= LocalSmem<B>::kBigs, q, 0xD20Full) ? sm.bigs : 0u;
    if (!m) return again;
    again = true;
    const uint32_t e = sm.big[m - 1u];
    __syncthreads();
    if (threadIdx.x == 0) sm.bigs = m - 1u;
    if (!GQS_OK((e >> 16) + (e & 0xffffu) <= len, q, 0xD210ull)) continue;
    load_range<B>(dst + (e >> 16), e & 0xffffu, key);
    for_rows<Sizes<B>::kLocalRows, Sizes<B>::kSortThreads>(e & 0xffffu, [&](int j) { key[j] = KeyOps<T>::key(key[j]); });
    sort_bins<T>(sm, key, e & 0xffffu, dst, e >> 16, false, q, [] {});
  }
}

// p[0, len) = x, by nt threads
template <class B>
__device__ __forceinline__ void fill_range(B* p, uint32_t len, B x, uint32_t tid, uint32_t nt) {
  constexpr uint32_t V = 16 / sizeof(B);
  const uint32_t over = (uint32_t)(-(reinterpret_cast<uintptr_t>(p) / sizeof(B)) & (V - 1u)), head = over < len ? over : len;
  const uint32_t vecs = (len - head) / V;
  if (tid < head) p[tid] = x;
  uint4 w;
  if constexpr (sizeof(B) == 8) w = make_uint4((uint32_t)x, (uint32_t)(x >> 32), (uint32_t)x, (uint32_t)(x >> 32));
  else w = make_uint4(x, x, x, x);
  uint4* const v = reinterpret_cast<uint4*>(p + head);
  for (uint32_t i = tid; i < vecs; i += nt) v[i] = w;
  for (uint32_t i = head + vecs * V + tid; i < len; i += nt) p[i] = x;
}

template <class T>
__global__ void __launch_bounds__((int)Sizes<BOf<T>>::kSortThreads, (int)Sizes<BOf<T>>::kSortCtas) local_sort(BOf<T>* d, BOf<T>* dn, unsigned long long n, Tables t, uint32_t plain_n, Queue* q) {
  using B = BOf<T>;
  constexpr int ROWS = Sizes<B>::kLocalRows;
  constexpr uint32_t NT = Sizes<B>::kSortThreads, LT = Sizes<B>::kLocal;
  extern __shared__ __align__(16) unsigned char split_dyn[];
  LocalSmem<B>& sm = *reinterpret_cast<LocalSmem<B>*>(split_dyn);
  const uint32_t tid = threadIdx.x;
  pdl_wait();
  pdl_trigger();
  if (plain_n) {  // the whole sort, by one CTA
    clear(q, sizeof(Queue));
    __threadfence();
    __syncthreads();
  } else if (ld_relaxed(&q->error)) {
    return;
  }
#ifdef GQS_PROFILE
  if (tid == 0) atomicCAS(&q->lvl_start, 0ull, (unsigned long long)global_timer_ns());
#endif
  const uint32_t nb = plain_n ? 1u : t.ctl->buckets;
  unsigned long long sorted = 0ull, moved = 0ull;
  uint32_t jobs = 0u;
  B key[ROWS];
  auto fetch = [&](const Bucket& k) {
    if ((k.flags & EQUAL) || k.len > LT) return;
    prefetch_l2(((k.flags & IN_DN) ? dn : d) + k.start, k.len, tid, NT);
  };
  uint32_t at = blockIdx.x;
  Bucket coming{};
  if (at < nb) {
    coming = plain_n ? Bucket{0ull, plain_n, 0u} : t.bucket[at];
    fetch(coming);
  }
  for (; at < nb; at += gridDim.x) {
    const Bucket bk = coming;
    const bool more = at + gridDim.x < nb;
    if (more) coming = t.bucket[at + gridDim.x];  // its keys are loaded once this range's have left the registers
    if (!GQS_OK(bk.start + bk.len <= n, q, 0xD201ull)) break;
    const B* const src = ((bk.flags & IN_DN) ? dn : d) + bk.start;
    B* const dst = d + bk.start;
    const uint32_t len = bk.len;
    if ((bk.flags & EQUAL) || len > LT) {
      bool same = (bk.flags & EQUAL) != 0u;
      B x = KeyOps<T>::raw((B)bk.value);
      // longer than the map's sample made likely: many equal keys, or keys too close together for it
      if (!same && len <= 8u * kCopyChunk) {
        x = src[0];
        same = true;
        for (uint32_t i0 = 0; i0 < len && same; i0 += 8u * NT) {
          bool eq = true;
#pragma unroll
          for (uint32_t u = 0; u < 8u; ++u) {
            const uint32_t i = i0 + u * NT + tid;
            if (i < len) eq &= src[i] == x;
          }
          same = !__syncthreads_or(!eq);
        }
      }
      if (same) {
        fill_range<B>(dst, len, x, tid, NT);
        moved += len;
      } else if (tid == 0) {
        const unsigned long long to = atomicAdd(&t.ctl->leftovers, 1ull);
        if (!GQS_OK(to < t.lefts, q, 0xD211ull)) break;
        t.left[2 * to] = bk.start;
        t.left[2 * to + 1] = bk.start + len;
        atomicAdd(&q->left, 1u);
      }
      if (more) fetch(coming);
      continue;
    }
    sorted += len;
    ++jobs;
#ifdef GQS_PROFILE
    if (tid == 0) level_note(q, 2u, 2, len);
#endif
    load_range<B>(src, len, key);
    if (!KeyOps<T>::kIdentity) for_rows<ROWS, NT>(len, [&](int j) { key[j] = KeyOps<T>::key(key[j]); });
    sort_range<T>(sm, key, len, dst, q, [&] {
      if (more) fetch(coming);
    });
  }
  if (tid == 0 && (sorted || moved)) {
    atomicAdd(&q->total, sorted + moved);
    atomicAdd(&q->done, sorted + moved);
    if (jobs) {
      atomicAdd(&q->local_keys, sorted);
      atomicAdd(&q->local_jobs, jobs);
    }
  }
}

constexpr uint32_t kOwnRanges = 32;  // of one CTA of local_small
struct Extent {
  uint32_t bin, start, len, equal;
};
template <class B>
struct SmallSortSmem {
  LocalSmem<B> local;
  Extent own[kOwnRanges];
  uint32_t wsum[Sizes<B>::kSortThreads / 32];
  uint32_t fills;
  Extent fill[Sizes<B>::kSmallMax / kCopyChunk + 1];  // long ranges of equal keys
};

// Every CTA of local_small takes a turn when it has read the cursors; the last one zeroes them, as its last work, so that no CTA
// waits for its turn's answer.
__device__ __forceinline__ uint32_t take_turn(Small* st) {
  __threadfence();
  return atomicAdd(&st->done, 1u);
}
__device__ __forceinline__ void leave_small(Small* st, uint32_t bins, uint32_t turn) {  // thread 0's turn
  if (__syncthreads_or(threadIdx.x == 0 && turn == gridDim.x - 1u)) {
    for (uint32_t i = threadIdx.x; i < bins; i += blockDim.x) st->cursor[i] = 0u;
    if (threadIdx.x == 0) st->done = 0u;
  }
}

// Latency: a chain of reads (ranges, counts) and one range's sort a CTA, 9 us of the 29 at 2^20 keys. Each CTA reads what it needs of
// all ranges in one round, its turn's answer is not waited for, and long ranges of equal keys are shared by all CTAs.
// The ranges of a small sort: their starts are the scan of their counts, which every CTA makes for itself.
template <class T>
__global__ void __launch_bounds__((int)Sizes<BOf<T>>::kSortThreads, (int)Sizes<BOf<T>>::kSortCtas) local_small(BOf<T>* d, const BOf<T>* area, uint32_t n, unsigned long long bound, Small* st, Queue* q) {
  using B = BOf<T>;
  constexpr int ROWS = Sizes<B>::kLocalRows;
  constexpr uint32_t NT = Sizes<B>::kSortThreads, LT = Sizes<B>::kLocal;
  constexpr uint32_t R = (kBinSlots + NT - 1) / NT;
  extern __shared__ __align__(16) unsigned char split_dyn[];
  SmallSortSmem<B>& sm = *reinterpret_cast<SmallSortSmem<B>*>(split_dyn);
  const uint32_t tid = threadIdx.x;
  pdl_wait();
  pdl_trigger();
  const uint32_t bins = st->bins;
  uint32_t c[R], sum = 0u, total;
  uint32_t equal = 0u;  // bit i: c[i] is of a range of equal keys, to be written by this CTA
  bool full = false;    // a range ran out of room
  const uint32_t per = (bins + NT - 1u) / NT;
  if (tid == 0) sm.fills = 0u;
#pragma unroll
  for (uint32_t i = 0; i < R; ++i) {
    const uint32_t b = tid * per + i;
    c[i] = 0u;
    if (i < per && b < bins) {
      c[i] = st->cursor[b];
      if (b % gridDim.x == blockIdx.x && st->eq[b]) equal |= 1u << i;
    }
  }
#pragma unroll
  for (uint32_t i = 0; i < R; ++i) {
    if (c[i] > LT && !st->eq[tid * per + i]) full = true;
    sum += c[i];
  }
  full = __syncthreads_or(full);  // (and every thread has its counts)
  const uint32_t turn = tid == 0 ? take_turn(st) : 0u;
  uint32_t at = block_scan<NT>(sum, sm.wsum, total);
  if (full || total != n) {
    if (blockIdx.x == 0 && tid == 0) {
      if (full) {  // d is as it was: all of it is left to the persistent kernel
        st->table[0] = 0ull;
        st->table[1] = n;
        st->left = 1ull;
        q->left = 1u;
      } else {  // the counters were not zero when the sort began: no start below can be relied on
        set_error(q, ST_INTERNAL, total);
      }
    }
    leave_small(st, bins, turn);
    return;
  }
#pragma unroll
  for (uint32_t i = 0; i < R; ++i) {
    const uint32_t b = tid * per + i;
    if (i < per && b < bins && b % gridDim.x == blockIdx.x && GQS_OK(b / gridDim.x < kOwnRanges, q, 0xD212ull))
      sm.own[b / gridDim.x] = Extent{b, at, c[i], equal >> i & 1u};
    if (c[i] > kCopyChunk) {
      const uint32_t to = atomicAdd(&sm.fills, 1u);
      if (GQS_OK(to < sizeof(sm.fill) / sizeof(sm.fill[0]), q, 0xD213ull)) sm.fill[to] = Extent{b, at, c[i], 1u};
    }
    at += c[i];
  }
  __syncthreads();
  unsigned long long sorted = 0ull, moved = 0ull;
  uint32_t jobs = 0u;
  for (uint32_t o = 0; o * gridDim.x + blockIdx.x < bins; ++o) {
    const uint32_t b = sm.own[o].bin, start = sm.own[o].start, len = sm.own[o].len;
    if (!len || !GQS_OK((unsigned long long)start + len <= bound, q, 0xD202ull)) continue;
    if (sm.own[o].equal) {
      if (len <= kCopyChunk) {
        const B x = KeyOps<T>::raw((B)st->value[b]);
        fill_range<B>(d + start, len, x, tid, NT);
      }
      moved += len;  // longer ones below
      continue;
    }
    sorted += len;
    ++jobs;
#ifdef GQS_PROFILE
    if (tid == 0) level_note(q, 1u, 2, len);
#endif
    B key[ROWS];
    load_range<B>(area + (size_t)b * LT, len, key);
    if (!KeyOps<T>::kIdentity) for_rows<ROWS, NT>(len, [&](int j) { key[j] = KeyOps<T>::key(key[j]); });
    sort_range<T>(sm.local, key, len, d + start, q, [] {});
  }
  // long ranges of equal keys: every CTA writes a part of each
  for (uint32_t f = 0; f < sm.fills GQS_CHECK_ONLY(&& f < sizeof(sm.fill) / sizeof(sm.fill[0])); ++f) {
    const uint32_t b = sm.fill[f].bin, start = sm.fill[f].start, len = sm.fill[f].len;
    if (!GQS_OK((unsigned long long)start + len <= bound, q, 0xD202ull)) continue;
    const B x = KeyOps<T>::raw((B)st->value[b]);
    const uint32_t i0 = (uint32_t)((unsigned long long)len * blockIdx.x / gridDim.x);
    const uint32_t i1 = (uint32_t)((unsigned long long)len * (blockIdx.x + 1u) / gridDim.x);
    fill_range<B>(d + start + i0, i1 - i0, x, tid, NT);
  }
  leave_small(st, bins, turn);
  if (tid == 0 && (sorted || moved)) {
    atomicAdd(&q->total, sorted + moved);
    atomicAdd(&q->done, sorted + moved);
    if (jobs) {
      atomicAdd(&q->local_keys, sorted);
      atomicAdd(&q->local_jobs, jobs);
    }
  }
}

// ---- host ----------------------------------------------------------------------------------------
// Ranges of a small sort: few enough for one on each CTA of local_small where that leaves them short.
template <class B>
uint32_t small_count(size_t n, int sms) {
  const size_t least = n / (Sizes<B>::kLocal / 10 * 3) + 1, most = n / 1024 + 1, want = (size_t)sms * Sizes<B>::kSortCtas;
  const size_t k = want < least ? least : want > most ? most : want;
  return k < 2 ? 2u : k > kMaxBins ? kMaxBins : (uint32_t)k;
}

template <class B>
bool is_small(size_t n, bool plain) {
  return plain && n > Sizes<B>::kLocal && n <= Sizes<B>::kSmallMax;
}

template <class B>
struct Layout {
  size_t segs[2], bins[2], cells[2], parts[2], buckets, left;
  size_t ctl_at, seg_at[2], bin_at[2], eq_at[2], value_at[2], cell_at[2], part_at[2], bucket_at, left_at, small_at, area_at, bytes;
  Layout(size_t n, size_t nseg, bool plain, int sms) {
    const size_t L = Sizes<B>::kLocal, G = Sizes<B>::kTarget;
    size_t at = 0;
    auto put = [&at](size_t b) {
      const size_t r = at;
      at += (b + 255) / 256 * 256;
      return r;
    };
    small_at = put(sizeof(Small));  // first, whatever n is: it has to stay as small sorts leave it
    ctl_at = put(sizeof(Ctl));
    left = n / L + 1;
    left_at = put(left * 16);
    if (is_small<B>(n, plain)) {
      area_at = put((size_t)bin_room(small_count<B>(n, sms)) * L * sizeof(B));
      bytes = at;
      return;
    }
    segs[0] = plain ? 1 : n / L + 1;
    segs[1] = n / L + 1;
    for (int l = 0; l < 2; ++l) {
      bins[l] = 5 * (n / G) / 2 + 9 * segs[l] + 8;
      parts[l] = bins[l] / 4 + 1;
      cells[l] = 16 * (n / G) + 312 * segs[l];
      seg_at[l] = put(segs[l] * sizeof(SegRec));
      bin_at[l] = put(bins[l] * 4);
      eq_at[l] = put(bins[l] * 4);
      value_at[l] = put(bins[l] * 8);
      cell_at[l] = put(cells[l] * 4);
      part_at[l] = put(parts[l] * sizeof(Part<B>));
    }
    buckets = bins[0] + bins[1] + n / kCopyChunk + (plain ? 0 : nseg) + 8;
    bucket_at = put(buckets * sizeof(Bucket));
    bytes = at;
  }
  Level level(void* scratch, int l) const {
    char* p = static_cast<char*>(scratch);
    return Level{reinterpret_cast<SegRec*>(p + seg_at[l]), reinterpret_cast<uint32_t*>(p + bin_at[l]),
                 reinterpret_cast<unsigned long long*>(p + value_at[l]), reinterpret_cast<uint32_t*>(p + eq_at[l]), reinterpret_cast<uint32_t*>(p + cell_at[l]),
                 p + part_at[l],
                 (uint32_t)segs[l], (uint32_t)bins[l], (uint32_t)cells[l], (uint32_t)l};
  }
  Tables tables(void* scratch, uint32_t tile_keys, unsigned long long bound) const {
    char* p = static_cast<char*>(scratch);
    return Tables{reinterpret_cast<Ctl*>(p + ctl_at), reinterpret_cast<Bucket*>(p + bucket_at),
                  reinterpret_cast<unsigned long long*>(p + left_at), (uint32_t)buckets, tile_keys, (uint32_t)left, bound};
  }
};

template <class K>
cudaError_t allow_smem(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <class T>
cudaError_t prepare_t() {
  using B = BOf<T>;
  cudaError_t e = allow_smem(split_scatter<T>, sizeof(ScatterSmem<B>));
  if (e == cudaSuccess) e = allow_smem(split_map<T>, sizeof(MapSmem<B>) + Sizes<B>::kMaxSample * sizeof(B));
  if (e == cudaSuccess) e = allow_smem(split_small<T, 1>, sizeof(SmallSmem<B>));
  if (e == cudaSuccess) e = allow_smem(split_small<T, kCluster>, sizeof(SmallSmem<B>));
  if (e == cudaSuccess) e = allow_smem(local_sort<T>, sizeof(LocalSmem<B>));
  if (e == cudaSuccess) e = allow_smem(local_small<T>, sizeof(SmallSortSmem<B>));
  return e;
}

template <class T>
cudaError_t launch_t(const SplitArgs& a, SplitResult* out) {
  using B = BOf<T>;
  const bool plain = a.offsets == nullptr;
  const Layout<B> lay(a.n, a.nseg, plain, a.sms);
  char* const base = static_cast<char*>(a.scratch);
  B* d = static_cast<B*>(a.d);
  B* dn = static_cast<B*>(a.dn);
  cudaStream_t s = a.stream;
  const uint32_t sms = (uint32_t)a.sms;
  auto least = [](uint32_t x, size_t y) { return (size_t)x < y ? x : (uint32_t)y; };
  cudaError_t e = cudaSuccess;
  bool early = false;
  auto go = [&](auto kernel, uint32_t grid, uint32_t block, size_t smem, auto... args) {
    if (e == cudaSuccess) e = launch_kernel(early, kernel, dim3(grid), dim3(block), smem, s, args...);
    early = true;
  };
  unsigned long long* const left = reinterpret_cast<unsigned long long*>(base + lay.left_at);
  // tiles: large ones write longer runs; a small sort needs one for every SM
  uint32_t tile_keys = Sizes<B>::kTile;
  if (is_small<B>(a.n, plain)) {
    while (tile_keys > 4u * kThreads && a.n / tile_keys < sms) tile_keys -= 2u * kThreads;
    Small* st = reinterpret_cast<Small*>(base + lay.small_at);
    B* area = reinterpret_cast<B*>(base + lay.area_at);
    const uint32_t n = (uint32_t)a.n, tiles = (n + tile_keys - 1u) / tile_keys, k = small_count<B>(a.n, a.sms);
    // Once every SM has two CTAs that read the whole sample, L2 is busy with it: a cluster reads it once (2^20 u32 33.0 to 29.3 us,
    // 2^21 44.7 to 39.3). With fewer CTAs a cluster's share SMs while others stay idle (300007 f64 28.4 to 33.3 us).
    if (tiles > sms) {
      const uint32_t ctas = (least(sms * kTileCtas, tiles) + kCluster - 1u) / kCluster * kCluster;
      go(split_small<T, kCluster>, ctas, kThreads, sizeof(SmallSmem<B>), (const B*)d, area, n, k, st, tile_keys, a.q);
    } else {
      go(split_small<T, 1>, tiles, kThreads, sizeof(SmallSmem<B>), (const B*)d, area, n, k, st, tile_keys, a.q);
    }
    const uint32_t ranges = bin_room(k), few = sms * Sizes<B>::kSortCtas, enough = (ranges + kOwnRanges - 1u) / kOwnRanges;
    go(local_small<T>, few > ranges ? ranges : few > enough ? few : enough, Sizes<B>::kSortThreads, sizeof(SmallSortSmem<B>), d, (const B*)area, n, a.bound, st, a.q);
    out->table = reinterpret_cast<const unsigned long long*>(base + lay.small_at + offsetof(Small, table));
    out->count = reinterpret_cast<const unsigned long long*>(base + lay.small_at + offsetof(Small, left));
    out->most = 1u;
    out->from_dn = 0u;
    return e;
  }
  // One level reaches ranges that fit on chip up to kMaxBins of them. A plain sort past 2^21 keys takes two levels even so: fewer,
  // larger ranges a level write longer runs.
  const uint32_t levels = a.n > (size_t)kMaxBins * Sizes<B>::kTarget || (plain && a.n > (1u << 21)) ? 2u : a.n > Sizes<B>::kLocal ? 1u : 0u;
  while (tile_keys > 4u * kThreads && a.n / tile_keys < 2u * sms) tile_keys -= 2u * kThreads;
  const Tables t = lay.tables(a.scratch, tile_keys, a.bound);
  const Level lv[2] = {lay.level(a.scratch, 0), lay.level(a.scratch, 1)};
  if (!plain) {  // the first kernel of a plain sort clears them
    e = cudaMemsetAsync(a.q, 0, sizeof(Queue), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(t.ctl, 0, sizeof(Ctl), s);
    SortArgs<T> sa{};
    sa.d = d;
    sa.dn = dn;
    sa.q = a.q;
    sa.n = a.bound;
    go(split_plan_segments<T>, (uint32_t)((a.nseg + 7) / 8), 256, 0, sa, t, lv[0], a.offsets, a.nseg_dev, (uint32_t)a.nseg, a.bound, a.pairs,
       levels);
  }
  for (uint32_t l = 0; l < levels; ++l) {
    const B* src = l ? dn : d;
    B* dst = l ? d : dn;
    const uint32_t gs = least(sms * 3u, lay.segs[l]);
    const uint32_t tiles = (uint32_t)(a.n / tile_keys + lay.segs[l]);
    const uint32_t sample = plain && !l ? Sizes<B>::kMaxSample : Sizes<B>::kMaxSample2;
    go(split_map<T>, gs, kThreads, sizeof(MapSmem<B>) + sample * sizeof(B), src, t, lv[l], plain && !l ? (uint32_t)a.n : 0u, levels, sample, a.q);
    go(split_count<T>, least(sms * 3u, tiles), kThreads, 0, src, t, lv[l], a.q);
    go(split_starts<T>, gs, kThreads, 0, t, lv[l], lv[1], levels, a.q);
    go(split_scatter<T>, least(sms * kTileCtas, tiles), kThreads, sizeof(ScatterSmem<B>), src, dst, t, lv[l], a.q);
  }
  const bool one = plain && !levels;
  go(local_sort<T>, one ? 1u : least(sms * Sizes<B>::kSortCtas, lay.buckets), Sizes<B>::kSortThreads, sizeof(LocalSmem<B>), d, dn, a.bound, t, one ? (uint32_t)a.n : 0u, a.q);
  out->table = left;
  out->count = &t.ctl->leftovers;
  out->most = levels ? (uint32_t)lay.left : 0u;
  out->from_dn = levels == 1u ? 1u : 0u;
  return e;
}

}  // namespace

size_t split_scratch_bytes(int dtype, size_t n, size_t nseg, bool plain, int sms) {
  auto bytes = [&]<class B>() {
    // never less than a smaller plain sort takes: the roomy ranges of the longest small one need more than somewhat longer sorts
    const size_t all = Layout<B>(n, nseg, plain, sms).bytes, most = Sizes<B>::kSmallMax;
    const size_t small = plain && n > most ? Layout<B>(most, 1, true, sms).bytes : 0;
    return all > small ? all : small;
  };
  return kDtypeBytes(dtype) == 4 ? bytes.template operator()<uint32_t>() : bytes.template operator()<uint64_t>();
}

size_t split_clear_bytes() { return sizeof(Small); }

size_t split_keep_bytes(int dtype, size_t n, size_t nseg, int sms) {
  return kDtypeBytes(dtype) == 4 ? Layout<uint32_t>(n, nseg, false, sms).seg_at[0] : Layout<uint64_t>(n, nseg, false, sms).seg_at[0];
}

cudaError_t split_prepare(int dtype) {
  switch (dtype) {
    case DT_U32: return prepare_t<uint32_t>();
    case DT_F32: return prepare_t<float>();
    case DT_F64: return prepare_t<double>();
    default: return prepare_t<uint64_t>();
  }
}

cudaError_t split_launch(int dtype, const SplitArgs& a, SplitResult* out) {
  switch (dtype) {
    case DT_U32: return launch_t<uint32_t>(a, out);
    case DT_F32: return launch_t<float>(a, out);
    case DT_F64: return launch_t<double>(a, out);
    default: return launch_t<uint64_t>(a, out);
  }
}

}  // namespace gqs
