// Partition sort for one B200 (sm_100a): the engine's plain device sort
// (thrust::sort -> CUB DeviceRadixSort in the reference, src/tanasic_sort.cuh:
// 264-266). Keys alone carry no identity: equal integers are the same bytes in
// any order, so the passes that move keys need not be stable, and the work can
// go from the most significant bits down:
//   P0 part_start     : a sample of the keys gives a monotone map key -> cell
//                       (at most 1024 cells of about equal size); other blocks
//                       clear the counters.
//   P1 part_histogram : one read counts the cells exactly. The last block turns
//                       the counts into cell starts and a work list.
//   P2 part_scatter   : moves every key to its cell (other buffer). A key's
//                       rank in its tile is what one shared-memory atomic
//                       returns; a tile reserves its place in each cell with
//                       one global atomic. No ballots, masks or look-back.
//   part_map, P1, part_plan, P2 on every cell that is still larger than one
//                       block can sort, as a second level.
//   P3 part_local     : one block sorts one unit (a cell, or neighbouring small
//                       cells) in shared memory and stores it to the caller's
//                       buffer.
//   P4 part_tail      : one cooperative launch for the rest, mostly nothing:
//                       units that the common way left out of order or that are
//                       too large for it, cells that hold one value,
//                       and, through the same steps once more, cells that two
//                       levels left too large (keys clustered at several
//                       scales); the zeros' signs.
// Inputs that one block can hold take a single launch (part_small).
//
// HBM traffic of one level: read + (read + write) + (read + write) = 5 n w;
// two levels: 8 n w. The stable 8-bit passes move (2 w + 1) n w: 9 n w for
// 4-byte keys and 17 n w for 8-byte keys, and rank every key w times. Measured
// on a B200 (B200 copy peak 6.45 TB/s), against the 8-bit passes: 2^30 uniform
// uint32 15.5 -> 12.2 ms; with a copy of the input before the sort, 10^8 normal
// float64 4.93 -> 2.64 ms, 2^20 int64 below 10^6 87 -> 52.5 us, 50021 normal
// float32 with 0.1 % zeros and NaN 65.5 -> 50.5 us, 1000 uint32 54.7 -> 18.2 us.
// part_histogram reads at 6.4 TB/s. part_scatter (22 SM cycles per 32 keys) and
// part_local (32) are bound by the shared-memory pipe and its latency: a scatter
// issues 14 shared wavefronts and 37-40 instructions per 32 keys, where the
// stable ranking of the 8-bit passes issues 24 and 63.
//
// IEEE zeros: -0.0 and +0.0 are equal keys with different bytes and keep their
// input order. The kernels turn -0.0 into +0.0 on the way in; when both occur,
// the first scatter records the zeros' signs in input order, and the signs are
// written over the sorted zeros at the end.
#include <algorithm>
#include <mutex>

#include "device_common.cuh"
#include "dispatch.cuh"
#include "partition_sort.cuh"
#include "engine_types.h"

namespace mgs {
namespace {

using u32 = uint32_t;
using u64 = unsigned long long;

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr u32 kMaxCells = 1024;        // cells of one segment, the two out-of-range cells included
constexpr u32 kHistWords = 4096;       // shared counters of the histogram: cells x copies
constexpr u32 kCounterWords = 2048;    // ... of a scatter tile
constexpr u32 kCoarse = kThreads;      // coarse intervals of the sampled map
constexpr u32 kSamples = 4096;         // keys a map is made from
constexpr int kFixBits = 20;           // fraction bits of the map's cell positions
constexpr u32 kBarrierSpins = 1u << 25;

// Shapes per key width. A unit is at most kLocalThreads * kLocalItems keys,
// sorted by one block in shared memory, kLocalBlocks such blocks per SM; 4 mod 8
// (4-byte) and 2 mod 4 (8-byte) items make the 16-byte shared loads of a
// thread's consecutive keys free of bank conflicts. Small blocks, because the
// steps of a unit are short and separated by barriers: 2^28 uint32, part_local
// with 512 x 20 keys and two blocks per SM 1.39 ms, 256 x 28 and three 1.37 ms,
// 384 x 20 and three 1.39 ms, 256 x 20 and four 1.27 ms (same code, with a
// call for crowded bins in it).
// kTileItems keys per thread make a scatter tile, kTileBlocks blocks per SM: a
// larger tile has longer runs per cell and fewer global atomics per key, until
// its keys spill. 2^28 uint32, both scatters: 16 items and two blocks 1.43 ms,
// 18 and two 1.43, 20 and two 1.64, 24 and two 2.08, 12 and three 1.83. 8-byte
// keys, whole sorts of 2^20 int64 / 10^8 float64 / 2^28 uint64: 8 items 54 us /
// 2.63 / 5.11 ms, 10 items 56 us / 2.62 / 5.00 ms.
// 256 x 20 keys and four blocks against 512 x 20 and two in part_local, whole
// sorts: 2^24 uint32 237 / 239 us, 2^26 float32 0.945 / 1.03 ms, 2^28 uint32
// 2.85 / 2.88 ms, 2^30 uint32 12.15 / 11.74 ms: only the largest would gain.
template <int W>
struct Shape;
template <>
struct Shape<4> {
  static constexpr int kLocalThreads = 256, kLocalItems = 20, kLocalBlocks = 4;
  static constexpr int kTileItems = 16, kTileBlocks = 2;
  static constexpr int kWideItems = 20;  // per thread, where 512 or 1024 threads sort a unit
};
template <>
struct Shape<8> {
  static constexpr int kLocalThreads = 256, kLocalItems = 14, kLocalBlocks = 4;
  static constexpr int kTileItems = 8, kTileBlocks = 2;
  static constexpr int kWideItems = 14;
};
template <typename B>
constexpr u32 kTile = u32(kThreads) * Shape<sizeof(B)>::kTileItems;
// Parts of `per` keys in len keys, the last one shorter. (len + per - 1) / per
// would wrap for the largest sorts: len may be any number below 2^32.
__host__ __device__ constexpr u32 parts_of(u32 len, u32 per) { return len / per + (len % per != 0u ? 1u : 0u); }
static_assert(parts_of(~0u, 8192u) == 524288u && parts_of(~0u, ~0u) == 1u && parts_of(0u, 8u) == 0u, "no wrap");
template <typename B>
constexpr u32 kCap = u32(Shape<sizeof(B)>::kLocalThreads) * Shape<sizeof(B)>::kLocalItems;
template <typename B>
constexpr u32 kWideCap = u32(kThreads) * Shape<sizeof(B)>::kWideItems;  // what 512 threads sort in one block
// Keys per cell a map aims at: 7/10 of a unit where the sample looks uniform
// (cell sizes then vary by sqrt only), half a unit where it does not (a coarse
// interval's share is known to about 18 %).
template <typename B>
constexpr u32 kCellUniform = kCap<B> / 10 * 7;
template <typename B>
constexpr u32 kCellSampled = kCap<B> / 2;
// Cell slots of a segment: 8 + kCellsPerTile per tile covers 2 ceil(len / kCellSampled) + 3 (a split map's cells).
template <typename B>
constexpr u32 kCellsPerTile = (2 * kTile<B> + kCellSampled<B> - 1) / kCellSampled<B>;

// ---------------------------------------------------------------- keys ------
// Total order of the raw bits: the engine's order, except that -0.0 comes
// right before +0.0.
template <typename B, int KIND>
__device__ __forceinline__ B to_ordered(B b) {
  constexpr B sign = B(1) << (sizeof(B) * 8 - 1);
  if (KIND == kUnsignedKey) return b;
  if (KIND == kSignedKey) return b ^ sign;
  return b ^ ((B(0) - (b >> (sizeof(B) * 8 - 1))) | sign);
}
template <typename B, int KIND>
__device__ __forceinline__ B from_ordered(B o) {
  constexpr B sign = B(1) << (sizeof(B) * 8 - 1);
  if (KIND == kUnsignedKey) return o;
  if (KIND == kSignedKey) return o ^ sign;
  return (o & sign) ? (o ^ sign) : ~o;
}
template <typename B>
constexpr B kNegZero = (B(1) << (sizeof(B) * 8 - 1)) - 1;  // ordered -0.0; +0.0 is one more
// The order the sort works in: IEEE -0.0 counts as +0.0.
template <typename B, int KIND>
__device__ __forceinline__ B one_zero(B o) {
  return KIND == kFloatKey && o == kNegZero<B> ? o + 1 : o;
}

__device__ __forceinline__ int leading_zeros(u64 v) { return __clzll((long long)v); }

// ---------------------------------------------------------------- map -------
// Monotone map of ordered keys to cells [0, ncells), of one of three kinds:
//   kLinear: equal cells over the sampled range (keys outside it in the first
//            and the last one), where the sample looks uniform;
//   kTable : equal intervals over the sampled range, each cut into equal cells,
//            as many as its share of the sample asks for (per interval the
//            position of its start and its width in cells, kFixBits fraction
//            bits); cells of their own for smaller (0) and larger keys
//            (ncells - 1): densities that are smooth within an interval;
//   kSplit : quantiles of the sorted sample (edges; a key's cell is the number
//            of edges <= key), whatever the keys are. A value that takes up
//            more than one cell's share gets a cell of its own. Costs a binary
//            search per key, so it is taken where a table's cells would be far
//            from equal.
// Linear maps and tables reduce a key to 32 bits first, x: a 4-byte key itself;
// of an 8-byte key the high word, when the range spans at least 2^16 of them
// (kPlain), else the offset from the smallest key, shifted into 31 bits, plus
// one, with 0 and ~0 for keys outside the range (kOffset); or, for tables of
// values crowded towards the smallest one over many scales, exponent and
// leading bits of the offset plus one, likewise (kLog).
enum MapKind : u32 { kLinear = 0, kTable = 1, kSplit = 2 };
enum MapX : u32 { kPlain = 0, kOffset = 1, kLog = 2 };
template <typename B>
struct alignas(16) Map {
  B lo, range;
  u32 x_lo, x_hi;
  u32 scale;  // linear: cell = umulhi(x - x_lo, scale); table: interval, likewise (0: interval = x - x_lo)
  u32 shift, ncells, kind, xmode;
  u32 pad[5];
};

__device__ __forceinline__ u32 log_x(u32 d) {
  const u32 z = u32(__clz(int(d)));
  return ((32u - z) << 26) | ((d << min(z, 31u) << 1) >> 6);
}
__device__ __forceinline__ u32 log_x(u64 d) {
  const u32 z = u32(__clzll((long long)d));
  return ((64u - z) << 25) | u32((d << min(z, 63u) << 1) >> 39);
}

template <u32 X, typename B>
__device__ __forceinline__ u32 x_of(const Map<B>& m, B key) {
  if constexpr (X == kPlain) {
    if constexpr (sizeof(B) == 4) {
      return key;
    } else {
      return u32(key >> 32);
    }
  } else {
    const B d = key - m.lo;
    const u32 x = (X == kLog ? log_x(d) : u32(d >> m.shift)) + 1u;
    return d <= m.range ? x : (key < m.lo ? 0u : ~0u);
  }
}

// The interval that holds x - x_lo, and the position within it (a 32-bit
// fraction).
__device__ __forceinline__ u32 interval_of(u32 d, u32 scale, u32& part) {
  const u64 p = u64(d) * scale;
  part = u32(p);
  return scale ? u32(p >> 32) : d;  // scale 0: fewer values than intervals
}

// The shared memory that a map of any kind needs beside it.
template <typename B>
union alignas(16) MapTable {
  uint2 interval[kCoarse];
  B edge[kMaxCells];  // ncells - 1 edges, ascending
};

template <u32 KIND, u32 X, typename B>
__device__ __forceinline__ u32 cell_of(const Map<B>& m, const MapTable<B>& tab, B key) {
  if constexpr (KIND == kSplit) {
    const u32 edges = m.ncells - 1u;
    u32 c = 0;
    for (u32 b = m.scale; b; b >>= 1)  // the largest power of two <= edges
      if (c + b <= edges && tab.edge[c + b - 1u] <= key) c += b;
    return c;
  } else {
    const u32 x = x_of<X, B>(m, key);
    const u32 t = min(max(x, m.x_lo), m.x_hi);
    if (KIND == kLinear) return __umulhi(t - m.x_lo, m.scale);
    u32 part;
    const uint2 e = tab.interval[interval_of(t - m.x_lo, m.scale, part)];
    u32 c = 1u + ((e.x + __umulhi(part, e.y)) >> kFixBits);
    c = x >= m.x_hi ? m.ncells - (x == m.x_hi ? 2u : 1u) : c;  // the largest x never shares the smallest one's cell
    return x < m.x_lo ? 0u : c;
  }
}

// The cells of N keys of a split map: the keys' searches go side by side.
template <typename B, int N>
__device__ __forceinline__ void split_cells(const Map<B>& m, const MapTable<B>& tab, const B (&k)[N], u32 (&c)[N]) {
  const u32 edges = m.ncells - 1u;
#pragma unroll
  for (int i = 0; i < N; ++i) c[i] = 0;
  for (u32 b = m.scale; b; b >>= 1) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const u32 t = c[i] + b;
      if (tab.edge[min(t, edges) - 1u] <= k[i] && t <= edges) c[i] = t;
    }
  }
}

template <u32 V>
struct Const {
  static constexpr u32 value = V;
};
// f(kind, x) with the map's kind as compile-time values (the same in every
// thread of the block).
template <typename B, class F>
__device__ __forceinline__ void with_kind(const Map<B>& m, F&& f) {
  if (m.kind == kSplit) {
    f(Const<kSplit>{}, Const<kPlain>{});
    return;
  }
  if (m.xmode == kLog) {
    f(Const<kTable>{}, Const<kLog>{});
    return;
  }
  if constexpr (sizeof(B) == 8) {
    if (m.xmode == kOffset) {
      if (m.kind == kTable) {
        f(Const<kTable>{}, Const<kOffset>{});
      } else {
        f(Const<kLinear>{}, Const<kOffset>{});
      }
      return;
    }
  }
  if (m.kind == kTable) {
    f(Const<kTable>{}, Const<kPlain>{});
  } else {
    f(Const<kLinear>{}, Const<kPlain>{});
  }
}
// The same without compile-time values, for where speed does not matter.
template <typename B>
__device__ u32 any_cell_of(const Map<B>& m, const MapTable<B>& tab, B key) {
  u32 c = 0;
  with_kind<B>(m, [&](auto kind, auto x) { c = cell_of<decltype(kind)::value, decltype(x)::value, B>(m, tab, key); });
  return c;
}

// One value for every key of a cell? True only where the map proves it for every
// key, sampled or not: such a cell's keys are copied as they are, and nothing
// looks at them again.
//   kSplit : keys of a cell between two edges lie in [edge, next edge).
//   kTable : offsets and logarithms send every key outside the sampled range to
//            the first or the last cell, and so do 4-byte keys themselves: the
//            other cells are made of offsets in [0, range], searched below.
//            High words (8-byte kPlain) bound neither end of the sample, and a
//            cell that takes a high word takes all 2^32 keys that have it.
//   kLinear: the end cells take what lies outside, and every cell spans four
//            values or more (a linear map needs 4 * kMaxCells of them).
template <typename B>
__device__ __noinline__ bool cell_is_one_value(const Map<B>& m, const MapTable<B>& tab, u32 cell) {
  if (cell == 0u || cell == m.ncells - 1u) return false;  // may hold keys outside the sampled range
  if (m.kind == kSplit) return tab.edge[cell] - tab.edge[cell - 1u] == 1;
  if (m.kind == kLinear || (sizeof(B) == 8 && m.xmode == kPlain)) return false;
  auto cell_at = [&](B d) { return any_cell_of<B>(m, tab, m.lo + d); };
  B first[2];
  for (u32 q = 0; q < 2; ++q) {  // the smallest offset with a cell >= cell + q
    B a = 0, b = m.range;
    while (a < b) {
      const B mid = a + (b - a) / 2;
      if (cell_at(mid) >= cell + q) {
        b = mid;
      } else {
        a = mid + 1;
      }
    }
    first[q] = a;
  }
  if (cell_at(first[1]) < cell + 1u) return first[0] == m.range;  // no larger cell inside the range
  return first[1] - first[0] == 1;
}

// ---------------------------------------------------------------- state -----
// A range of keys still to be split: [start, start + len) of buffer src (0: the
// caller's keys, 1: the scratch buffer), its tiles and its cells.
struct alignas(16) Segment {
  u32 start, len, tile_base, cell_base;
  u32 src;
  u32 identity;  // one value: its keys stay where they are
  u32 done;      // nothing is left to do for it (until a probe finds a second value)
  u32 pad;
};

struct State {
  u64 list[2];        // per segment list: segments << 32 | tiles
  u32 units, next_unit, left;
  u32 hist_done;
  u32 neg_zeros, pos_zeros, below_zeros;  // IEEE keys: -0.0, +0.0, keys that sort before them
  u32 barrier;
  u32 dirty;  // segments found to hold several values
  u32 in_place;  // the caller's array holds one value (zeros of either sign count as one)
  u32 pad;
};

// A unit: start, len (30 bits), bit 30 = buffer it sits in, bit 31 = already in order (store it only).
constexpr u32 kUnitSrc = 1u << 30, kUnitCopy = 1u << 31, kUnitLen = kUnitSrc - 1;

template <typename B>
struct Sort {
  B* keys;  // the caller's keys
  B* tmp;   // the scratch buffer
  __device__ __forceinline__ B* buf(u32 which) const { return which ? tmp : keys; }
  State* st;
  Segment* seg0;  // the two segment lists
  Segment* seg1;
  u32* count0;  // cell counts of the segments of a list (one each for the two levels that are launched apart)
  u32* count1;
  __device__ __forceinline__ Segment* segs(u32 list) const { return list ? seg1 : seg0; }
  u32* cursor;     // next free position of each cell of the level being scattered
  Map<B>* maps;    // per segment of the level being scattered
  MapTable<B>* tables;  // likewise
  uint4* tiles;    // per tile of a list: first key, keys, segment, buffer
  uint2* units;
  uint2* left;  // units for the tail: of more than kCap keys, or not in order after the common way
  u32* tile_zeros;  // root tiles: zeros of both signs; then their exclusive prefix
  u32* zero_signs;  // bit i: the i-th zero of the input is -0.0
  u32* status;
  u32 n;
  u32 last_list;  // the list that the levels launched apart leave behind
};

template <typename B>
__device__ __forceinline__ Map<B> load_map(const Map<B>* p) {
  static_assert(sizeof(Map<B>) % 16 == 0, "whole 16-byte words");
  Map<B> m;
#pragma unroll
  for (int i = 0; i < int(sizeof(m) / 16); ++i)
    reinterpret_cast<uint4*>(&m)[i] = __ldcg(reinterpret_cast<const uint4*>(p) + i);
  return m;
}

// ---------------------------------------------------------------- blocks ----
// Exclusive scan over the block (any multiple of 32 threads up to 1024); total
// out. Ends without a barrier after the last read of `tmp`: callers separate
// uses with a barrier of their own.
template <int THREADS>
__device__ __forceinline__ u32 block_scan(u32 v, u32* tmp, u32* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  u32 incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) tmp[warp] = incl;
  __syncthreads();
  u32 w = lane < THREADS / 32 ? tmp[lane] : 0u;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 t = __shfl_up_sync(0xffffffffu, w, o);
    if (lane >= o) w += t;
  }
  *total = __shfl_sync(0xffffffffu, w, 31);
  const u32 before = __shfl_sync(0xffffffffu, w, warp ? warp - 1 : 0);
  return incl - v + (warp ? before : 0u);
}

__device__ __forceinline__ u32 warp_min(u32 v) { return __reduce_min_sync(0xffffffffu, v); }
__device__ __forceinline__ u32 warp_max(u32 v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ __forceinline__ u64 warp_min(u64 v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const u64 t = __shfl_xor_sync(0xffffffffu, v, o);
    v = t < v ? t : v;
  }
  return v;
}
__device__ __forceinline__ u64 warp_max(u64 v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const u64 t = __shfl_xor_sync(0xffffffffu, v, o);
    v = t > v ? t : v;
  }
  return v;
}
// Block minimum and maximum in every thread; mm: 64 elements of shared memory.
// One barrier inside; the caller's next barrier ends the use of mm.
template <int THREADS, typename B>
__device__ __forceinline__ void block_min_max(B& lo, B& hi, B* mm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  lo = warp_min(lo);
  hi = warp_max(hi);
  if (lane == 0) {
    mm[warp] = lo;
    mm[32 + warp] = hi;
  }
  __syncthreads();
  const bool in = lane < THREADS / 32;
  lo = warp_min(in ? mm[lane] : ~B(0));
  hi = warp_max(in ? mm[32 + lane] : B(0));
}

// Polls of the grid barrier (set_barrier_spins).
__device__ u32 g_barrier_spins = kBarrierSpins;

// Blocks that wait on one another (cooperative launch): all arrive, bounded
// wait. A block whose bound runs out reports it at once and must leave: the
// others then cannot pass the next barrier, so no block works on a later step
// than one past what every block has finished.
__device__ __forceinline__ bool grid_barrier(State* st, u32 target, u32 spins, u32* status) {
  __shared__ u32 s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&st->barrier, 1u);
    u32 ok = 0;
    for (u32 i = 0; i < spins; ++i) {
      if (ld_volatile_u32(&st->barrier) >= target) {
        ok = 1;
        break;
      }
      if (i > 16) __nanosleep(64);
    }
    __threadfence();
    if (!ok && status != nullptr) atomicOr(status, kStatusQueueTimeout);
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// ---------------------------------------------------------------- sampling --
template <typename B>
struct MapSmem {
  MapTable<B> tab;
  u32 hist[kCoarse];
  B mm[64];
  u32 tmp[33];
  float chi[kWarps];
  u32 dense[kWarps];
};

// Keys that one level can still split into units.
template <typename B>
constexpr u32 kOneLevel = (kMaxCells - 2u) * kCellUniform<B>;

// Cells a segment of len keys is split into when a cell should hold `per`:
// all of them if one level can, else the square root, so that two levels
// split evenly, times `more` (of a table's cells many hold few keys or none).
template <typename B>
__device__ __forceinline__ u32 inner_cells(u32 len, u32 per, u32 more) {
  u32 need = parts_of(len, per);
  if (need > kMaxCells - 2u)
    need = len <= kOneLevel<B> ? kMaxCells - 2u : min(kMaxCells - 2u, more * u32(sqrtf(float(need)) + 1.f));
  return max(need, 4u);  // the smallest and the largest sampled key get different cells
}

// The part of a map that the range of the keys decides.
template <typename B>
__device__ __forceinline__ void set_range(Map<B>& m, B lo, B hi) {
  m.lo = lo;
  m.range = hi - lo;
  m.shift = 0;
  m.xmode = kPlain;
  if constexpr (sizeof(B) == 4) {
    m.x_lo = lo;
    m.x_hi = hi;
  } else if ((hi >> 32) - (lo >> 32) < 65536u) {
    const int lz = leading_zeros(m.range);  // 64 for a range of one value
    m.xmode = kOffset;
    m.shift = lz < 33 ? u32(33 - lz) : 0u;
    m.x_lo = 1u;
    m.x_hi = u32(m.range >> m.shift) + 1u;
  } else {
    m.x_lo = u32(lo >> 32);
    m.x_hi = u32(hi >> 32);
  }
}
// scale for equal intervals over [x_lo, x_hi]
template <typename B>
__device__ __forceinline__ u32 interval_scale(const Map<B>& m) {
  const u32 xr = m.x_hi - m.x_lo;
  return xr >= kCoarse ? u32((u64(kCoarse) << 32) / (u64(xr) + 1u)) : 0u;
}

template <typename B, int KIND>
__device__ Map<B> build_map(const B* __restrict__ src, u32 len, MapSmem<B>& sm, u32* scratch) {
  constexpr u32 kPer = kSamples / kThreads;
  const u32 tid = threadIdx.x;
  u32 per = min(len < (1u << 19) ? kPer / 4u : kPer, max(1u, len / (8u * kThreads)));
  per = 1u << (31u - u32(__clz(int(per))));
  const u32 samples = per * kThreads;  // a power of two
  const u32 stride = len / samples;
  B x[kPer];
  B lo = ~B(0), hi = B(0);
#pragma unroll
  for (u32 i = 0; i < kPer; ++i) {
    const u32 q = i * kThreads + tid;
    const u32 h = (q * 2654435761u) >> 8;  // a place of its own within its stride
    if (i < per) x[i] = __ldcg(src + size_t(q) * stride + h % stride);
  }
#pragma unroll
  for (u32 i = 0; i < kPer; ++i) {
    if (i < per) {
      x[i] = one_zero<B, KIND>(to_ordered<B, KIND>(x[i]));
      lo = x[i] < lo ? x[i] : lo;
      hi = x[i] > hi ? x[i] : hi;
    }
  }
  __syncthreads();  // the caller's last use of sm
  sm.hist[tid] = 0u;
  block_min_max<kThreads, B>(lo, hi, sm.mm);
  Map<B> m;
  set_range<B>(m, lo, hi);
  u32 xr = m.x_hi - m.x_lo;
  m.scale = interval_scale<B>(m);
  auto sample_intervals = [&] {
#pragma unroll
    for (u32 i = 0; i < kPer; ++i) {
      if (i < per) {
        u32 part;
        const u32 v = m.xmode == kLog ? x_of<kLog, B>(m, x[i])
                                      : (m.xmode == kOffset ? x_of<kOffset, B>(m, x[i]) : x_of<kPlain, B>(m, x[i]));
        atomicAdd(&sm.hist[interval_of(v - m.x_lo, m.scale, part)], 1u);
      }
    }
    __syncthreads();
  };
  sample_intervals();
  // Is the sample uniform over the range? Chi-squared over the coarse intervals.
  static_assert(kCoarse == kThreads, "an interval per thread");
  u32 c = sm.hist[tid];
  float chi;
  const float width = m.scale ? 4294967296.f / float(m.scale) : 1.f, whole = float(xr) + 1.f;
  {
    const float want = float(samples) * fminf(fmaxf(whole - float(tid) * width, 0.f), width) / whole;
    const float diff = float(c) - want;
    chi = diff * diff / fmaxf(want, 0.5f);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) chi += __shfl_xor_sync(0xffffffffu, chi, o);
  if ((tid & 31) == 0) sm.chi[tid >> 5] = chi;
  // No stretch of 32 intervals may be much denser than the whole either.
  const float in_warp = float(__reduce_add_sync(0xffffffffu, c));
  if ((tid & 31u) == 0u)
    sm.dense[tid >> 5] = in_warp * whole > 1.3f * float(samples) * fminf(32.f * width, whole) + 64.f * whole;
  u32 total;
  u32 cum = block_scan<kThreads>(c, sm.tmp, &total);  // its barrier also publishes sm.chi
  chi = 0.f;
  u32 dense = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    chi += sm.chi[w];
    dense |= sm.dense[w];
  }
  const bool uniform = xr >= 4u * kMaxCells && !dense && chi < float(kCoarse) + 2.5f * sqrtf(2.f * float(kCoarse));
  if (uniform) {
    m.kind = kLinear;
    m.ncells = inner_cells<B>(len, kCellUniform<B>, 1u);
    // The true range reaches beyond the sample's by about a sample's distance on either side: widened by six of
    // them, the first and the last cell are not overfull.
    const B beyond = m.range / samples * 6u;
    lo -= lo < beyond ? lo : beyond;
    hi += ~hi < beyond ? B(~hi) : beyond;
    set_range<B>(m, lo, hi);
    xr = m.x_hi - m.x_lo;
    m.scale = u32((u64(m.ncells) << 32) / (u64(xr) + 1u));
    __syncthreads();
    return m;
  }
  m.kind = kTable;
  // Over an eighth of the keys in one interval: a logarithmic x, if that cuts the fullest interval to half.
  auto fullest_of = [&](u32 v) {
    v = __reduce_max_sync(0xffffffffu, v);
    __syncthreads();
    if ((tid & 31u) == 0u) sm.dense[tid >> 5] = v;
    __syncthreads();
    return __reduce_max_sync(0xffffffffu, sm.dense[tid & (kWarps - 1u)]);
  };
  const u32 fullest = fullest_of(c);
  if (xr >= 2u * kCoarse && fullest > samples / 8u) {
    const Map<B> equal = m;
    m.xmode = kLog;
    m.x_lo = 1u;
    m.x_hi = log_x(m.range) + 1u;
    m.scale = interval_scale<B>(m);
    sm.hist[tid] = 0u;
    __syncthreads();
    sample_intervals();
    const u32 c_log = sm.hist[tid];
    const u32 cum_log = block_scan<kThreads>(c_log, sm.tmp, &total);
    if (2u * fullest_of(c_log) <= fullest) {
      c = c_log;
      cum = cum_log;
    } else {
      m = equal;
    }
  }
  const u32 want = inner_cells<B>(len, kCellSampled<B>, 2u);
  // Twice as many where one level has room for them: fewer cells are then above a unit, which only the tail sorts
  // (neighbouring small cells make a unit together). 10^6 normal float32 with 0.1 % zeros and NaN: 97 -> 79 us.
  u32 ni = len <= kOneLevel<B> ? min(2u * want, kMaxCells - 2u) : want;
  m.ncells = ni + 2u;
  {
    const u64 all = u64(ni) << kFixBits;
    const u32 base = u32(u64(cum) * all / samples), end = u32(u64(cum + c) * all / samples);
    sm.tab.interval[tid] = make_uint2(base, end - base);
  }
  // How well do these cells split the sample? Keys in cells that hold more than three times their share, or than
  // the next level can split, and more than one value.
  u32* const cell_count = scratch;
  u32* const cell_min = scratch + kMaxCells;
  u32* const cell_max = scratch + 2u * kMaxCells;
  static_assert(3u * kMaxCells <= kHistWords && kMaxCells == 2u * kThreads, "scratch");
  for (u32 q = tid; q < kMaxCells; q += kThreads) {
    cell_count[q] = 0u;
    cell_min[q] = ~0u;
    cell_max[q] = 0u;
  }
  __syncthreads();
  with_kind<B>(m, [&](auto kind, auto xk) {
    constexpr u32 kKind = decltype(kind)::value, kX = decltype(xk)::value;
    if constexpr (kKind == kTable) {
#pragma unroll
      for (u32 i = 0; i < kPer; ++i) {
        if (i < per) {
          const u32 q = cell_of<kKind, kX, B>(m, sm.tab, x[i]);
          const u32 v = u32(x[i]) ^ u32(u64(x[i]) >> 32);
          atomicAdd(cell_count + q, 1u);
          atomicMin(cell_min + q, v);
          atomicMax(cell_max + q, v);
        }
      }
    }
  });
  __syncthreads();
  const bool last_level = len <= kOneLevel<B>;
  const u32 most =
      last_level ? 3u * samples / want + 8u : u32(0.6f * float(kMaxCells) * float(kCellSampled<B>) * float(samples) / float(len)) + 8u;
  u32 over = 0;
  for (u32 q = tid; q < m.ncells; q += kThreads)
    if (cell_count[q] > most && cell_min[q] != cell_max[q]) over += cell_count[q];
  block_scan<kThreads>(over, sm.tmp, &over);
  __syncthreads();
  if (over <= samples / 8u) return m;
  // No: the quantiles of the sample, sorted in the scratch: of every second key where it does not hold them all
  // (not of the first half: samples are in the order of the keys, which may be sorted).
  constexpr u32 kSorted = kHistWords * 4u / u32(sizeof(B));
  B* const sorted = reinterpret_cast<B*>(scratch);
  const u32 count = min(samples, kSorted), every = samples / count;  // powers of two all
  __syncthreads();
#pragma unroll
  for (u32 i = 0; i < kPer; ++i)
    if (i < per && (tid & (every - 1u)) == 0u) sorted[(i * kThreads + tid) / every] = x[i];
  for (u32 size = 2; size <= count; size <<= 1) {
    for (u32 d = size >> 1; d > 0; d >>= 1) {
      __syncthreads();
      for (u32 i = tid; i < count / 2u; i += kThreads) {
        const u32 p = 2u * i - (i & (d - 1u));
        const B u = sorted[p], v = sorted[p + d];
        if ((v < u) == ((p & size) == 0u)) {
          sorted[p] = v;
          sorted[p + d] = u;
        }
      }
    }
  }
  __syncthreads();
  ni = min(2u * want, kMaxCells - 2u);  // quantiles of a sample are rough: more of them
  m.kind = kSplit;
  m.ncells = ni + 1u;  // edges: the smallest key, then ni - 1 quantiles
  m.scale = 1u << (31u - u32(__clz(int(ni))));
  for (u32 q = tid; q < ni; q += kThreads) {
    B e = sorted[q * count / ni];
    if (q && e == sorted[(q - 1u) * count / ni] && e != ~B(0)) e += 1;  // a value's second quantile ends its cell
    sm.tab.edge[q] = e;
  }
  __syncthreads();
  return m;
}

template <typename B>
__device__ __forceinline__ void load_table(MapTable<B>& to, const MapTable<B>* from) {
  for (u32 i = threadIdx.x; i < u32(sizeof(to) / 16); i += kThreads)
    reinterpret_cast<uint4*>(&to)[i] = __ldcg(reinterpret_cast<const uint4*>(from) + i);
}

template <typename B>
__device__ __forceinline__ void store_map(const Sort<B>& a, u32 s, const Map<B>& m, const MapSmem<B>& sm) {
  if (threadIdx.x == 0) a.maps[s] = m;
  if (m.kind != kLinear) {
    for (u32 i = threadIdx.x; i < u32(sizeof(sm.tab) / 16); i += kThreads)
      reinterpret_cast<uint4*>(a.tables + s)[i] = reinterpret_cast<const uint4*>(&sm.tab)[i];
  }
}

// Copies of each counter: as many as fit into `words` words, at most one per lane.
__device__ __forceinline__ u32 copy_shift(u32 ncells, u32 words) {
  const u32 bits = 32u - u32(__clz(int(ncells - 1u)));  // cells rounded up to 2^bits
  return min(5u, 31u - u32(__clz(int(words))) - bits);
}

// ---------------------------------------------------------------- P1 --------
template <typename B>
struct HistSmem {
  alignas(16) u32 cnt[kHistWords];
  MapTable<B> tab;
  Map<B> map;
  u32 last;
};

struct ZeroCounts {
  u32 zeros, neg, below;  // IEEE keys of the caller's: zeros of both signs, -0.0, keys that sort before them
};

// Counts the cells of p[0..n), a map of one kind: 16-byte loads, and single keys
// at the ends. Not inlined: each kind then has registers of its own.
template <typename B, int KIND, bool ROOT, u32 MAP, u32 X>
__device__ __noinline__ ZeroCounts count_range(const B* __restrict__ p, u32 n, const HistSmem<B>& sm,
                                               unsigned char* cnt_bytes, u32 step) {
  constexpr int kBatch = 4;  // loads in flight per thread
  constexpr u32 kPerVec = 16 / sizeof(B);
  const u32 tid = threadIdx.x;
  const Map<B> m = sm.map;
  ZeroCounts z{0, 0, 0};
  auto see = [&](B key) {
    key = to_ordered<B, KIND>(key);
    if (ROOT && KIND == kFloatKey) {
      z.zeros += (key - kNegZero<B>) < B(2) ? 1u : 0u;
      z.neg += key == kNegZero<B> ? 1u : 0u;
      z.below += key < kNegZero<B> ? 1u : 0u;
    }
    return one_zero<B, KIND>(key);
  };
  auto count = [&](u32 cell) { atomicAdd(reinterpret_cast<u32*>(cnt_bytes + cell * step), 1u); };
  const u32 head = min(n, u32((16u - (u32(reinterpret_cast<uintptr_t>(p)) & 15u)) & 15u) / u32(sizeof(B)));
  const u32 vecs = (n - head) / kPerVec, tail = head + vecs * kPerVec;
  if (tid < head) count(cell_of<MAP, X, B>(m, sm.tab, see(__ldcg(p + tid))));
  if (tid < n - tail) count(cell_of<MAP, X, B>(m, sm.tab, see(__ldcg(p + tail + tid))));
  auto count_vec = [&](const uint4& q) {
    B k[kPerVec];
    if constexpr (sizeof(B) == 4) {
      k[0] = q.x;
      k[1] = q.y;
      k[2] = q.z;
      k[3] = q.w;
    } else {
      k[0] = (u64(q.y) << 32) | q.x;
      k[1] = (u64(q.w) << 32) | q.z;
    }
    u32 c[kPerVec];
#pragma unroll
    for (u32 e = 0; e < kPerVec; ++e) k[e] = see(k[e]);
    if constexpr (MAP == kSplit) {
      split_cells<B, int(kPerVec)>(m, sm.tab, k, c);
    } else {
#pragma unroll
      for (u32 e = 0; e < kPerVec; ++e) c[e] = cell_of<MAP, X, B>(m, sm.tab, k[e]);
    }
#pragma unroll
    for (u32 e = 0; e < kPerVec; ++e) count(c[e]);
  };
  const uint4* v = reinterpret_cast<const uint4*>(p + head);
  u32 i = tid;
#pragma unroll 1
  for (; i + (kBatch - 1) * kThreads < vecs; i += kBatch * kThreads) {
    uint4 q[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) q[b] = ld_stream_v4(v + i + b * kThreads);
#pragma unroll
    for (int b = 0; b < kBatch; ++b) count_vec(q[b]);
  }
#pragma unroll 1
  for (; i < vecs; i += kThreads) count_vec(ld_stream_v4(v + i));
  return z;
}

// The segment of a tile: the largest s with tile_base <= t.
__device__ __forceinline__ u32 segment_of(const Segment* segs, u32 nseg, u32 t) {
  u32 s = 0, hi = nseg;
  while (hi - s > 1u) {
    const u32 mid = (s + hi) / 2u;
    if (__ldcg(&segs[mid].tile_base) <= t) {
      s = mid;
    } else {
      hi = mid;
    }
  }
  return s;
}

// Counts the cells of the tiles [t0, t1) of a segment list into counts. The
// segments' maps are ready.
template <typename B, int KIND, bool ROOT>
__device__ void histogram_tiles(const Sort<B>& a, const Segment* segs, u32 nseg, u32* counts, u32 t0, u32 t1,
                                HistSmem<B>& sm) {
  const u32 tid = threadIdx.x;
  if (t0 >= t1) return;
  u32 s = segment_of(segs, ROOT ? 1u : nseg, t0);
  ZeroCounts z{0, 0, 0};
  for (u32 t = t0; t < t1; ++s) {
    const uint4 head = ROOT ? make_uint4(0u, a.n, 0u, 0u) : __ldcg(reinterpret_cast<const uint4*>(segs + s));
    const u32 start = head.x, len = head.y, tile_base = head.z, cell_base = head.w;
    const u32 buf = ROOT ? 0u : __ldcg(&segs[s].src);
    const u32 e = min(t1, tile_base + parts_of(len, kTile<B>));
    if (!ROOT) {
      for (u32 x = t + tid; x < e; x += kThreads) {
        const u32 first = (x - tile_base) * kTile<B>;
        a.tiles[x] = make_uint4(start + first, min(kTile<B>, len - first), s, buf);
      }
      if (__ldcg(&segs[s].done)) {
        t = e;
        continue;
      }
    }
    __syncthreads();  // the last segment's map and counts are read
    if (tid == 0) sm.map = load_map<B>(a.maps + s);
    load_table<B>(sm.tab, a.tables + s);  // unused by linear maps
    __syncthreads();
    const u32 ncells = sm.map.ncells, cs = copy_shift(ncells, kHistWords);
    const u32 step = 4u << cs, sub = (tid & ((1u << cs) - 1u)) * 4u;
    for (u32 i = tid; i < (ncells << cs); i += kThreads) sm.cnt[i] = 0u;
    __syncthreads();
    const B* src = a.buf(buf) + start;
    unsigned char* const cnt_bytes = reinterpret_cast<unsigned char*>(sm.cnt) + sub;
    with_kind<B>(sm.map, [&](auto kind, auto x) {
      constexpr u32 kKind = decltype(kind)::value, kX = decltype(x)::value;
      if (ROOT && KIND == kFloatKey) {  // zeros are counted tile by tile
        for (; t < e; ++t) {
          const ZeroCounts y = count_range<B, KIND, ROOT, kKind, kX>(src + size_t(t) * kTile<B>,
                                                                      min(kTile<B>, len - t * kTile<B>), sm, cnt_bytes, step);
          z.zeros += y.zeros;
          z.neg += y.neg;
          z.below += y.below;
          const u32 zeros = __reduce_add_sync(0xffffffffu, y.zeros);
          if ((tid & 31u) == 0u && zeros) atomicAdd(&a.tile_zeros[t], zeros);
        }
      } else {
        const u32 first = (t - tile_base) * kTile<B>;
        const u64 end = min(u64(len), u64(e - tile_base) * kTile<B>);
        count_range<B, KIND, ROOT, kKind, kX>(src + first, u32(end - first), sm, cnt_bytes, step);
        t = e;
      }
    });
    __syncthreads();
    for (u32 c = tid; c < ncells; c += kThreads) {
      u32 sum = 0;
      for (u32 q = 0; q < (1u << cs); ++q) sum += sm.cnt[(c << cs) | ((q + tid) & ((1u << cs) - 1u))];
      if (sum) atomicAdd(&counts[cell_base + c], sum);
    }
  }
  if (ROOT && KIND == kFloatKey) {
    const u32 neg = __reduce_add_sync(0xffffffffu, z.neg);
    const u32 pos = __reduce_add_sync(0xffffffffu, z.zeros) - neg;
    const u32 below = __reduce_add_sync(0xffffffffu, z.below);
    if ((tid & 31u) == 0u) {
      if (below) atomicAdd(&a.st->below_zeros, below);
      if (neg) atomicAdd(&a.st->neg_zeros, neg);
      if (pos) atomicAdd(&a.st->pos_zeros, pos);
    }
  }
}

// ---------------------------------------------------------------- plan ------
struct PlanSmem {
  u32 start[kMaxCells + 1];  // starts of the runs of cells that become one unit or one segment
  u32 cell[kMaxCells];       // the run's cell, ~0 for a run of small cells
  u32 tmp[33], tmp2[33];
  u32 emitted, base, identity;
};

// From a segment's cell counts: the cells' first positions (cursor), the units
// and the next list's segments. to: the list that takes cells that are still
// too large; raw: the segment is the caller's, not yet moved;
// last: the tail comes next and probes those cells for a second value.
template <typename B>
__device__ void plan_segment(const Sort<B>& a, Segment* seg, const Map<B>& m, const MapTable<B>& tab, u32 to, bool raw,
                             bool last, const u32* counts, PlanSmem& sm) {
  constexpr u32 cap = kCap<B>, half = cap / 2;
  const u32 tid = threadIdx.x;
  const uint4 head = __ldcg(reinterpret_cast<const uint4*>(seg));
  const u32 start = head.x, len = head.y, cell_base = head.w;
  const u32 src = __ldcg(&seg->src);
  __syncthreads();
  if (tid == 0) {
    sm.emitted = 0;
    sm.identity = 0;
  }
  const u32 c0 = 2 * tid;
  u32 c[2];
  c[0] = c0 < m.ncells ? __ldcg(counts + cell_base + c0) : 0u;
  c[1] = c0 + 1 < m.ncells ? __ldcg(counts + cell_base + c0 + 1) : 0u;
  u32 total;
  u32 at[2];
  at[0] = block_scan<kThreads>(c[0] + c[1], sm.tmp, &total);
  at[1] = at[0] + c[0];
  // A run breaks at every cell above half a unit, after it, and where the
  // start of a small cell enters another half-unit window: a run of small
  // cells then holds at most two halves.
  auto small = [&](u32 n) { return n <= half; };
  // the cell before this thread's first one
  u32 pc = __shfl_up_sync(0xffffffffu, c[1], 1), pa = __shfl_up_sync(0xffffffffu, at[1], 1);
  if ((tid & 31u) == 0u && tid) {
    pc = c0 - 1 < m.ncells ? __ldcg(counts + cell_base + c0 - 1) : 0u;
    pa = at[0] - pc;
  }
  bool brk[2];
  brk[0] = c0 < m.ncells && (c0 == 0 || !small(c[0]) || !small(pc) || at[0] / half != pa / half);
  brk[1] = c0 + 1 < m.ncells && (!small(c[1]) || !small(c[0]) || at[1] / half != at[0] / half);
  u32 runs;
  u32 r = block_scan<kThreads>(u32(brk[0]) + u32(brk[1]), sm.tmp2, &runs);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    if (c0 + q < m.ncells) {
      if (c[q] == len) sm.identity = 1u;
      a.cursor[cell_base + c0 + q] = start + at[q];
    }
    if (brk[q]) {
      sm.start[r] = at[q];
      sm.cell[r] = small(c[q]) ? ~0u : c0 + q;
      ++r;
    }
  }
  if (tid == 0) sm.start[runs] = len;
  __syncthreads();
  // Every key in one cell: it holds one value. Were there two, the smallest and the largest sampled key would differ
  // and have different cells (a table gives x_lo cell 1 and x_hi cell ncells - 2; equal cells over more than 4096
  // values part them; the second edge of a split lies above the first and not above its largest sample); and if all
  // samples are one value, every map of a range of one value sends the keys below and above it to other cells.
  const bool identity = sm.identity != 0;
  if (tid == 0) seg->identity = identity ? 1u : 0u;
  if (identity && raw) {  // one value: the caller's keys are sorted as they are
    if (tid == 0) a.st->in_place = 1u;
    return;
  }
  const u32 in = identity ? src : src ^ 1u;
  u32 slot[2], unit_len[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const u32 i = tid + u32(q) * kThreads;
    slot[q] = ~0u;
    if (i >= runs) continue;
    const u32 n = sm.start[i + 1] - sm.start[i];
    if (n == 0) continue;
    unit_len[q] = n;
    if (n <= cap) {
      slot[q] = atomicAdd(&sm.emitted, 1u);
      continue;
    }
    const u32 at0 = start + sm.start[i];
    if (n <= kWideCap<B>) {  // what 512 threads sort in one block: the tail does it
      a.left[atomicAdd(&a.st->left, 1u)] = make_uint2(at0, n | (in ? kUnitSrc : 0u));
    } else if (identity || cell_is_one_value<B>(m, tab, sm.cell[i])) {
      const u32 chunk = max(cap, parts_of(n, 256u)), chunks = parts_of(n, chunk);
      const u32 u = atomicAdd(&a.st->units, chunks);
      for (u32 x = 0; x < chunks; ++x)
        a.units[u + x] = make_uint2(at0 + x * chunk, min(chunk, n - x * chunk) | (in ? kUnitSrc : 0u) | kUnitCopy);
    } else {
      const u32 tiles = parts_of(n, kTile<B>);
      const u64 got = atomicAdd(&a.st->list[to], (u64(1) << 32) | tiles);
      const u32 id = u32(got >> 32), tb = u32(got);
      Segment* o = a.segs(to) + id;
      o->start = at0;
      o->len = n;
      o->tile_base = tb;
      o->cell_base = id * 8u + tb * kCellsPerTile<B>;
      o->src = in;
      o->identity = o->done = last ? 1u : 0u;
    }
  }
  __syncthreads();
  if (tid == 0) sm.base = sm.emitted ? atomicAdd(&a.st->units, sm.emitted) : 0u;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const u32 i = tid + u32(q) * kThreads;
    if (slot[q] != ~0u)
      a.units[sm.base + slot[q]] = make_uint2(start + sm.start[i], unit_len[q] | (in ? kUnitSrc : 0u));
  }
}

// Root only, IEEE keys with zeros of both signs: the zeros before each root
// tile, and room for their signs.
template <typename B>
__device__ void plan_zeros(const Sort<B>& a, u32* tmp) {
  const u32 neg = __ldcg(&a.st->neg_zeros), pos = __ldcg(&a.st->pos_zeros);
  if (neg == 0 || pos == 0) return;
  const u32 tiles = parts_of(a.n, kTile<B>);
  const u32 words = u32((u64(neg) + pos + 31) / 32);
  for (u32 i = threadIdx.x; i < words; i += kThreads) a.zero_signs[i] = 0u;
  u32 carry = 0;
  for (u32 t0 = 0; t0 < tiles; t0 += kThreads) {
    const u32 t = t0 + threadIdx.x;
    u32 total;
    __syncthreads();
    const u32 before = block_scan<kThreads>(t < tiles ? __ldcg(a.tile_zeros + t) : 0u, tmp, &total);
    if (t < tiles) a.tile_zeros[t] = carry + before;
    carry += total;
  }
}

// Block 0 makes the whole array's map; the others clear what a sort counts in.
template <typename B, int KIND>
__global__ __launch_bounds__(kThreads) void part_start_kernel(Sort<B> a, uint4* clear, u32 clear_vecs) {
  __shared__ MapSmem<B> sm;
  __shared__ __align__(16) u32 scratch[kHistWords];
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) {
      Segment* o = a.segs(0);
      o->start = 0;
      o->len = a.n;
      o->tile_base = 0;
      o->cell_base = 0;
      o->src = 0;
      o->done = 0;
    }
    const Map<B> m = build_map<B, KIND>(a.keys, a.n, sm, scratch);
    store_map<B>(a, 0u, m, sm);
    return;
  }
  for (u32 i = (blockIdx.x - 1u) * kThreads + threadIdx.x; i < clear_vecs; i += (gridDim.x - 1u) * kThreads)
    clear[i] = make_uint4(0u, 0u, 0u, 0u);
}

// The whole array: counts its cells; the last block to finish plans the level.
template <typename B, int KIND>
__global__ __launch_bounds__(kThreads, 2) void part_histogram_root_kernel(Sort<B> a) {
  __shared__ HistSmem<B> sm;
  __shared__ PlanSmem plan;
  const u32 tiles = parts_of(a.n, kTile<B>);
  const u32 t0 = u32(u64(tiles) * blockIdx.x / gridDim.x), t1 = u32(u64(tiles) * (blockIdx.x + 1) / gridDim.x);
  histogram_tiles<B, KIND, true>(a, a.segs(0), 1u, a.count0, t0, t1, sm);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) sm.last = atomicAdd(&a.st->hist_done, 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!sm.last) return;
  __threadfence();
  plan_segment<B>(a, a.segs(0), sm.map, sm.tab, 1u, true, a.last_list == 1u, a.count0, plan);
  if (KIND == kFloatKey) plan_zeros<B>(a, plan.tmp);
}

// The maps of the segments s0, s0 + step, ... of a list.
template <typename B, int KIND>
__device__ void map_segments(const Sort<B>& a, const Segment* segs, u32 s0, u32 step, u32 nseg, MapSmem<B>& sm,
                             u32* scratch) {
  for (u32 s = s0; s < nseg; s += step) {
    const uint4 q = __ldcg(reinterpret_cast<const uint4*>(segs + s));
    if (__ldcg(&segs[s].done)) continue;
    const B* src = a.buf(__ldcg(&segs[s].src)) + q.x;
    const Map<B> m = build_map<B, KIND>(src, q.y, sm, scratch);
    store_map<B>(a, s, m, sm);
  }
}

template <typename B, int KIND>
__global__ __launch_bounds__(kThreads) void part_map_kernel(Sort<B> a) {
  __shared__ MapSmem<B> sm;
  __shared__ __align__(16) u32 scratch[kHistWords];
  map_segments<B, KIND>(a, a.segs(1), blockIdx.x, gridDim.x, u32(__ldcg(&a.st->list[1]) >> 32), sm, scratch);
}

// Segmented sort: its large segments as list 1. One block, 1024 segments a
// round. A segment that starts before the end of an earlier large one (the
// offsets are out of order) is left out and reported: disjoint segments of the
// array are what the lists' capacities are computed for (layout).
template <typename B>
__global__ __launch_bounds__(1024) void part_segments_kernel(Sort<B> a, const u64* __restrict__ offsets,
                                                             const u32* __restrict__ ids, const u32* __restrict__ count) {
  __shared__ u32 tmp[33], last_end[32];
  const u32 segs = *count, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  u32 taken = 0, base = 0, end = 0;  // of the rounds so far: segments and tiles in the list, the largest end
  bool left_out = false;
  for (u32 r = 0; r < segs; r += 1024u) {
    const u32 i = r + threadIdx.x;
    u32 first = 0, len = 0;
    if (i < segs) {
      const u32 id = ids[i];
      first = u32(offsets[id]);
      len = u32(offsets[id + 1u] - offsets[id]);
    }
    u32 reach = first + len;  // the largest end up to this segment
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 t = __shfl_up_sync(0xffffffffu, reach, o);
      if (lane >= u32(o)) reach = max(reach, t);
    }
    if (lane == 31u) last_end[warp] = reach;
    __syncthreads();
    u32 before = __shfl_up_sync(0xffffffffu, reach, 1);  // ... up to the one before it
    if (lane == 0) before = 0;
    before = max(max(before, end), warp_max(lane < warp ? last_end[lane] : 0u));
    end = max(end, warp_max(last_end[lane]));
    const bool ok = i < segs && first >= before;
    left_out |= i < segs && !ok;
    const u32 tiles = parts_of(len, kTile<B>);
    // Segments and tiles in one scan: a round's disjoint segments have at most 2^20 full tiles and 1024 shorter ones.
    static_assert(kTile<B> >= 4096u, "a round's tiles fit 21 bits");
    u32 total;
    const u32 at = block_scan<1024>(ok ? (1u << 21) | tiles : 0u, tmp, &total);
    if (ok) {
      const u32 id = taken + (at >> 21);
      Segment s;
      s.start = first;
      s.len = len;
      s.tile_base = base + (at & ((1u << 21) - 1u));
      s.cell_base = id * 8u + s.tile_base * kCellsPerTile<B>;
      s.src = s.identity = s.done = s.pad = 0u;
      a.seg1[id] = s;
    }
    taken += total >> 21;
    base += total & ((1u << 21) - 1u);
    __syncthreads();  // tmp and last_end are read
  }
  if (threadIdx.x == 0 && taken) a.st->list[1] = (u64(taken) << 32) | base;
  if (__syncthreads_or(left_out) && threadIdx.x == 0 && a.status != nullptr) atomicOr(a.status, kStatusBadInput);
}

// Every segment of list 1.
template <typename B, int KIND>
__global__ __launch_bounds__(kThreads, 2) void part_histogram_kernel(Sort<B> a) {
  __shared__ HistSmem<B> sm;
  const u64 list = __ldcg(&a.st->list[1]);
  const u32 nseg = u32(list >> 32), tiles = u32(list);
  const u32 t0 = u32(u64(tiles) * blockIdx.x / gridDim.x), t1 = u32(u64(tiles) * (blockIdx.x + 1) / gridDim.x);
  histogram_tiles<B, KIND, false>(a, a.segs(1), nseg, a.count1, t0, t1, sm);
}

template <typename B>
__global__ __launch_bounds__(kThreads) void part_plan_kernel(Sort<B> a, bool raw) {
  __shared__ PlanSmem sm;
  __shared__ MapTable<B> tab;
  const u32 nseg = u32(__ldcg(&a.st->list[1]) >> 32);
  for (u32 s = blockIdx.x; s < nseg; s += gridDim.x) {
    __syncthreads();
    load_table<B>(tab, a.tables + s);
    plan_segment<B>(a, a.segs(1) + s, load_map<B>(a.maps + s), tab, 0u, raw, true, a.count1, sm);
  }
}

// ---------------------------------------------------------------- P2 --------
template <typename B>
struct ScatterSmem {
  B keys[kTile<B>];
  u32 cnt[2][kCounterWords];  // of this tile and the next one (zero)
  u32 gbase[kMaxCells];
  MapTable<B> tab;
  Map<B> map;  // of the current segment; read from here where it is used (registers are short)
  u32 cell_base, identity;
  u32 tmp[33];
  uint16_t cells[kTile<B>];  // of the keys, where the map is a split
  u32 zeros[kThreads];  // zeros per item and warp, then their exclusive prefix
};

// A tile's keys, thread t's are t, t + kThreads, ...
template <typename B>
__device__ __forceinline__ void load_tile(B (&k)[Shape<sizeof(B)>::kTileItems], const B* __restrict__ src, u32 cnt) {
  constexpr int kItems = Shape<sizeof(B)>::kTileItems;
  src += threadIdx.x;
  if (cnt == kTile<B>) {
#pragma unroll
    for (int i = 0; i < kItems; ++i) k[i] = __ldcg(src + i * kThreads);
  } else {
    const int left = int(cnt) - int(threadIdx.x);
#pragma unroll
    for (int i = 0; i < kItems; ++i)
      if (i * kThreads < left) k[i] = __ldcg(src + i * kThreads);
  }
}

// One tile of keys (in k, raw) into the cells of its segment; k then holds the
// next tile's keys. Counters, ranks and places
// are in bytes of keys, so that a key's shared address is one addition.
template <typename B, int KIND, bool ROOT, bool WHOLE, u32 MAP, u32 X>
__device__ __forceinline__ void scatter_tile(const Sort<B>& a, B (&k)[Shape<sizeof(B)>::kTileItems],
                                             B* __restrict__ dst, u32 cnt, const B* __restrict__ next, u32 next_cnt,
                                             u32 tile, bool signs, u32 which, ScatterSmem<B>& sm) {
  constexpr int kItems = Shape<sizeof(B)>::kTileItems;
  const u32 tid = threadIdx.x;
  const int left = int(cnt) - int(tid);
  const u32 ncells = sm.map.ncells, cs = copy_shift(ncells, kCounterWords);
  const u32 step = 4u << cs, sub = (tid & ((1u << cs) - 1u)) * 4u;
  u32* const counters = sm.cnt[which];
  unsigned char* const cnt_bytes = reinterpret_cast<unsigned char*>(counters);
  unsigned char* const key_bytes = reinterpret_cast<unsigned char*>(sm.keys);
  u32 zeros_before = 0;
  if (ROOT && KIND == kFloatKey && signs) zeros_before = __ldcg(a.tile_zeros + tile);  // on its way meanwhile
  u32 pk[kItems];  // the key's counter (byte offset) | its rank there << 16
  u32 neg_mask = 0;  // the items that are -0.0
  if (KIND != kUnsignedKey) {
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      k[i] = to_ordered<B, KIND>(k[i]);
      if (KIND == kFloatKey) neg_mask |= k[i] == kNegZero<B> ? 1u << i : 0u;
      k[i] = one_zero<B, KIND>(k[i]);
    }
  }
  Map<B> m = sm.map;
  if constexpr (MAP == kSplit) {
    split_cells<B, kItems>(m, sm.tab, k, pk);
  }
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    if (WHOLE || i * kThreads < left) {
      const u32 at = (MAP == kSplit ? pk[i] : cell_of<MAP, X, B>(m, sm.tab, k[i])) * step + sub;
      pk[i] = at | (atomicAdd(reinterpret_cast<u32*>(cnt_bytes + at), u32(sizeof(B))) << 16);
    }
  }
  if (ROOT && KIND == kFloatKey) {
    // Signs of the zeros, in input order (item, then thread).
    if (signs) {
      static_assert(kItems * kWarps <= kThreads, "a count per warp and item");
      u32 zero_mask = 0;
#pragma unroll
      for (int i = 0; i < kItems; ++i) {
        const bool z = (WHOLE || i * kThreads < left) && k[i] == kNegZero<B> + 1;
        const u32 mask = __ballot_sync(0xffffffffu, z);
        if ((tid & 31u) == 0u) sm.zeros[i * kWarps + (tid >> 5)] = __popc(mask);
        zero_mask |= z ? 1u << i : 0u;
      }
      __syncthreads();
      u32 total;
      const u32 count = tid < kItems * kWarps ? sm.zeros[tid] : 0u;
      const u32 before = block_scan<kThreads>(count, sm.tmp, &total);
      if (total) {  // the same in every thread
        if (tid < kItems * kWarps) sm.zeros[tid] = zeros_before + before;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
          const u32 mask = __ballot_sync(0xffffffffu, (zero_mask >> i) & 1u);
          if ((neg_mask & zero_mask) >> i & 1u) {
            const u32 r = sm.zeros[i * kWarps + (tid >> 5)] + __popc(mask & lanemask_lt());
            atomicOr(&a.zero_signs[r >> 5], 1u << (r & 31u));
          }
        }
      }
    }
  }
  __syncthreads();
  // Exclusive scan of the counters, four consecutive words per thread; the other set is cleared meanwhile.
  static_assert(kCounterWords == 4 * kThreads, "one 16-byte word per thread");
  reinterpret_cast<uint4*>(sm.cnt[which ^ 1u])[tid] = make_uint4(0u, 0u, 0u, 0u);
  uint4* const v = reinterpret_cast<uint4*>(counters) + tid;
  uint4 x = *v;
  u32 total;
  u32 run = block_scan<kThreads>(x.x + x.y + x.z + x.w, sm.tmp, &total), t;
  t = x.x; x.x = run; run += t;
  t = x.y; x.y = run; run += t;
  t = x.z; x.z = run; run += t;
  x.w = run;
  *v = x;
  __syncthreads();
  for (u32 c = tid; c < ncells; c += kThreads) {
    const u32 s = counters[c << cs] / u32(sizeof(B));
    const u32 e = ((c + 1u) << cs) < kCounterWords ? counters[(c + 1u) << cs] / u32(sizeof(B)) : cnt;
    if (e != s) sm.gbase[c] = atomicAdd(a.cursor + sm.cell_base + c, e - s) - s;
  }
#pragma unroll
  for (int i = 0; i < kItems; ++i)
    if (WHOLE || i * kThreads < left)
    {
      const u32 to = *reinterpret_cast<const u32*>(cnt_bytes + (pk[i] & 0xFFFFu)) + (pk[i] >> 16);
      *reinterpret_cast<B*>(key_bytes + to) = k[i];
      if (MAP == kSplit) sm.cells[to / u32(sizeof(B))] = uint16_t((pk[i] & 0xFFFFu) >> (cs + 2u));
    }
  load_tile<B>(k, next, next_cnt);  // in flight while this tile is stored
  __syncthreads();
  m = sm.map;  // not kept in registers across the barriers
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    if (WHOLE || i * kThreads < left) {
      const B key = sm.keys[i * kThreads + tid];
      const u32 c = MAP == kSplit ? u32(sm.cells[i * kThreads + tid]) : cell_of<MAP, X, B>(m, sm.tab, key);
      const u32 to = sm.gbase[c] + u32(i * kThreads) + tid;
      if (to < a.n) dst[to] = key;  // always, if the counts are those of these keys
    }
  }
}

// The tiles [t0, t1) of a level. Each block takes consecutive tiles (all tiles
// cost the same), so a segment's map is read once per block and segment.
template <typename B, int KIND, bool ROOT>
__device__ void scatter_tiles(const Sort<B>& a, const Segment* segs, u32 t0, u32 t1, ScatterSmem<B>& sm) {
  if (t0 >= t1) return;
  const u32 tid = threadIdx.x;
  auto tile_at = [&](u32 t) {  // first key, keys, segment, buffer
    return ROOT ? make_uint4(t * kTile<B>, min(kTile<B>, a.n - t * kTile<B>), 0u, 0u) : __ldcg(a.tiles + t);
  };
  B k[Shape<sizeof(B)>::kTileItems];
  uint4 cur = tile_at(t0);
  load_tile<B>(k, a.buf(cur.w) + cur.x, cur.y);
  u32 have = ~0u, which = 0;
  const bool signs = ROOT && KIND == kFloatKey && __ldcg(&a.st->neg_zeros) && __ldcg(&a.st->pos_zeros);
  reinterpret_cast<uint4*>(sm.cnt[0])[tid] = make_uint4(0u, 0u, 0u, 0u);
  for (u32 t = t0; t < t1; ++t) {
    uint4 next = cur;
    next.y = 0;
    if (t + 1 < t1) next = tile_at(t + 1);
    const B* ahead = a.buf(next.w) + next.x;
    if (cur.z != have) {
      __syncthreads();  // the map's last use
      if (tid == 0) {
        sm.map = load_map<B>(a.maps + cur.z);
        sm.cell_base = ROOT ? 0u : __ldcg(&segs[cur.z].cell_base);
        sm.identity = __ldcg(&segs[cur.z].identity);
      }
      load_table<B>(sm.tab, a.tables + cur.z);  // unused by linear maps
      have = cur.z;
      __syncthreads();
    }
    if (sm.identity) {  // the segment stays where it is
      load_tile<B>(k, ahead, next.y);
    } else {
      B* dst = a.buf(cur.w ^ 1u);
      with_kind<B>(sm.map, [&](auto kind, auto x) {
        constexpr u32 kKind = decltype(kind)::value, kX = decltype(x)::value;
        if (cur.y == kTile<B>) {
          scatter_tile<B, KIND, ROOT, true, kKind, kX>(a, k, dst, cur.y, ahead, next.y, t, signs, which, sm);
        } else {
          scatter_tile<B, KIND, ROOT, false, kKind, kX>(a, k, dst, cur.y, ahead, next.y, t, signs, which, sm);
        }
      });
      which ^= 1u;
    }
    cur = next;
  }
}

template <typename B, int KIND, bool ROOT>
__global__ __launch_bounds__(kThreads, Shape<sizeof(B)>::kTileBlocks) void part_scatter_kernel(Sort<B> a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  ScatterSmem<B>& sm = *reinterpret_cast<ScatterSmem<B>*>(smem_raw);
  const Segment* segs = a.segs(ROOT ? 0u : 1u);
  if (ROOT && __ldcg(&segs->identity)) return;
  const u32 tiles = ROOT ? parts_of(a.n, kTile<B>) : u32(__ldcg(&a.st->list[1]));
  const u32 t0 = u32(u64(tiles) * blockIdx.x / gridDim.x), t1 = u32(u64(tiles) * (blockIdx.x + 1) / gridDim.x);
  scatter_tiles<B, KIND, ROOT>(a, segs, t0, t1, sm);
}

// ---------------------------------------------------------------- P3 --------
// One block sorts up to THREADS * ITEMS keys. The keys' range is cut into about
// one bin per key; a key's place is its bin's start plus the rank that the
// counting atomic returned. If a bin holds more than kBinLimit keys, the bins
// are cut once more, each into as many parts as it holds keys, which evens out
// any density that is smooth within a bin. Then every bin or part is mostly at
// most kBinLimit long, and odd-even transposition in registers over each
// thread's consecutive keys, and over windows across the threads' borders,
// finishes the order: as many rounds as the fullest bin has keys. What is still
// out of order after that (keys clustered at several scales) is merge sorted:
// the same cost whatever the keys are.
template <typename B>
constexpr u32 kBinLimit = sizeof(B) == 4 ? 8 : 7;
// Keys on either side of a border between two threads' keys that a bin across it can reach (a multiple of 16
// bytes; the windows of neighbouring borders must not overlap).
template <typename B>
constexpr u32 kBorder = sizeof(B) == 4 ? 8 : 6;
constexpr u32 kExactBits = 15;  // Bins gives every value a bin of its own for ranges below 2^kExactBits

template <typename B, int THREADS, int ITEMS>
struct LocalSmem {
  static constexpr u32 kKeys = u32(THREADS) * ITEMS;
  static constexpr u32 kBins = u32(ITEMS + 3) / 4u * 4u * THREADS;  // a bin per key
  static_assert(kBins <= 1u << kExactBits, "a range below the bins' number must fit the exact bins");
  alignas(16) B keys[kKeys + 16];
  alignas(16) u32 bins[kBins + 4];
  B mm[64];
  u32 tmp[4][33], most[33];
  u32 nbins;
};

// Exclusive scan in place of `groups` * 4 * THREADS counters (16-bit totals) in
// their natural order; thread t holds words 4t..4t+3 of each group of 4 *
// THREADS (16-byte accesses without bank conflicts). Returns the largest
// counter. One barrier inside; the caller's next barrier publishes the starts.
template <int THREADS, int MAX_GROUPS>
__device__ __forceinline__ u32 scan_counters(u32* c, u32 groups, u32 (&tmp)[4][33], u32* most) {
  constexpr int kPairs = (MAX_GROUPS + 1) / 2;
  static_assert(kPairs <= 4, "tmp rows");
  const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  u32 pair[kPairs], incl[kPairs];
  u32 mx = 0;
#pragma unroll
  for (int p = 0; p < kPairs; ++p) pair[p] = 0;
#pragma unroll
  for (int g = 0; g < MAX_GROUPS; ++g) {
    if (u32(g) < groups) {
      const uint4 v = reinterpret_cast<const uint4*>(c)[g * THREADS + tid];
      mx = max(max(mx, max(v.x, v.y)), max(v.z, v.w));
      pair[g / 2] += (v.x + v.y + v.z + v.w) << (g & 1 ? 16 : 0);
    }
  }
  mx = warp_max(mx);
#pragma unroll
  for (int p = 0; p < kPairs; ++p) {
    incl[p] = pair[p];
    if (u32(2 * p) < groups) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u32 t = __shfl_up_sync(0xffffffffu, incl[p], o);
        if (lane >= u32(o)) incl[p] += t;
      }
      if (lane == 31u) tmp[p][warp] = incl[p];
    }
  }
  if (lane == 0) most[warp] = mx;
  __syncthreads();
  u32 offset = 0;
#pragma unroll
  for (int p = 0; p < kPairs; ++p) {
    if (u32(2 * p) < groups) {
      u32 w = lane < u32(THREADS / 32) ? tmp[p][lane] : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u32 t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= u32(o)) w += t;
      }
      const u32 total = __shfl_sync(0xffffffffu, w, 31);
      const u32 before = __shfl_sync(0xffffffffu, w, warp ? warp - 1u : 0u);
      const u32 ex = incl[p] - pair[p] + (warp ? before : 0u);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int g = 2 * p + h;
        if (g < MAX_GROUPS && u32(g) < groups) {
          u32 run = offset + (h ? ex >> 16 : ex & 0xFFFFu);
          uint4 v, q;  // read again (volatile: not kept from above): registers are short
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                       : "r"(smem_u32(c) + (g * THREADS + tid) * 16u)
                       : "memory");
          q.x = run;
          run += v.x;
          q.y = run;
          run += v.y;
          q.z = run;
          run += v.z;
          q.w = run;
          reinterpret_cast<uint4*>(c)[g * THREADS + tid] = q;
          offset += h ? total >> 16 : total & 0xFFFFu;
        }
      }
    }
  }
  return warp_max(lane < u32(THREADS / 32) ? most[lane] : 0u);
}

// Two rounds of odd-even transposition over N registers.
template <typename B, int N>
__device__ __forceinline__ void transpose_twice(B (&x)[N]) {
#pragma unroll
  for (int i = 0; i + 1 < N; i += 2) {
    const B lo = x[i] < x[i + 1] ? x[i] : x[i + 1], hi = x[i] < x[i + 1] ? x[i + 1] : x[i];
    x[i] = lo;
    x[i + 1] = hi;
  }
#pragma unroll
  for (int i = 1; i + 1 < N; i += 2) {
    const B lo = x[i] < x[i + 1] ? x[i] : x[i + 1], hi = x[i] < x[i + 1] ? x[i + 1] : x[i];
    x[i] = lo;
    x[i + 1] = hi;
  }
}

// At least `rounds` rounds of odd-even transposition over N registers.
template <typename B, int N>
__device__ __forceinline__ void transpose_rounds(B (&x)[N], u32 rounds) {
#pragma unroll
  for (int r = 0; r < int(kBinLimit<B>); r += 2) {
    if (u32(r) >= rounds) break;
    transpose_twice<B, N>(x);
  }
}

template <typename B, int N>
__device__ __forceinline__ void load_run(const B* p, B (&x)[N]) {
  static_assert((N * sizeof(B)) % 16 == 0, "whole 16-byte words");
#pragma unroll
  for (int i = 0; i < int(N * sizeof(B) / 16); ++i) {
    const uint4 q = reinterpret_cast<const uint4*>(p)[i];
    if constexpr (sizeof(B) == 4) {
      x[4 * i] = q.x;
      x[4 * i + 1] = q.y;
      x[4 * i + 2] = q.z;
      x[4 * i + 3] = q.w;
    } else {
      x[2 * i] = (u64(q.y) << 32) | q.x;
      x[2 * i + 1] = (u64(q.w) << 32) | q.z;
    }
  }
}
template <typename B, int N>
__device__ __forceinline__ void store_run(B* p, const B (&x)[N]) {
#pragma unroll
  for (int i = 0; i < int(N * sizeof(B) / 16); ++i) {
    uint4 q;
    if constexpr (sizeof(B) == 4) {
      q = make_uint4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
    } else {
      q = make_uint4(u32(x[2 * i]), u32(x[2 * i] >> 32), u32(x[2 * i + 1]), u32(x[2 * i + 1] >> 32));
    }
    reinterpret_cast<uint4*>(p)[i] = q;
  }
}

// The bins of one part of the keys: bin(key) = floor(offset * nbins / range),
// the offset from the smallest key taken to 32 bits; one bin per value when
// there are few enough values.
template <typename B>
struct Bins {
  B lo;
  u32 shift, mul, scale;
  bool exact;
  __device__ __forceinline__ Bins(B lo_, B range, u32 nbins) : lo(lo_) {
    shift = 0;
    if constexpr (sizeof(B) == 8) {
      const int lz = leading_zeros(range);
      shift = lz < 32 ? u32(32 - lz) : 0u;
    }
    exact = range < B(nbins);
    // Exact: d * 2^17 * 2^15 / 2^32 = d. Both products must fit: d < nbins <= 2^15 (checked in LocalSmem).
    mul = exact ? 1u << (32 - kExactBits) : 1u;
    scale = exact ? 1u << kExactBits
                  : u32(float(nbins) * (4294967296.f * 0.9999995f) / (float(u32(range >> shift)) + 1.f));
  }
  // bin in the high word, position within the bin (a 32-bit fraction) in the low word
  __device__ __forceinline__ u64 product(B key) const {
    u32 dn;
    if constexpr (sizeof(B) == 4) {
      dn = key - lo;
    } else {
      dn = u32((key - lo) >> shift);
    }
    return u64(dn * mul) * scale;
  }
};

// Writes the zeros with their signs, in input order (src, the caller's bits, is
// still unsorted), over the sorted zeros in sm.keys. Ends with a barrier.
template <typename B, int KIND, int THREADS, int ITEMS>
__device__ __noinline__ void order_zeros(const B* src, u32 len, LocalSmem<B, THREADS, ITEMS>& sm) {
  u32 a0 = 0, b0 = len;  // first key >= -0.0
  while (a0 < b0) {
    const u32 mid = (a0 + b0) / 2;
    if (sm.keys[mid] < kNegZero<B>) {
      a0 = mid + 1;
    } else {
      b0 = mid;
    }
  }
  __syncthreads();
  for (u32 i = 0; i * THREADS < len; ++i) {
    const u32 idx = i * THREADS + threadIdx.x;
    const B key = idx < len ? to_ordered<B, KIND>(__ldcg(src + idx)) : B(0);
    const bool z = (key - kNegZero<B>) < B(2);
    u32 total;
    const u32 at = block_scan<THREADS>(z ? 1u : 0u, sm.tmp[0], &total);
    if (z) sm.keys[a0 + at] = key;
    a0 += total;
    __syncthreads();
  }
}

// A unit's keys, thread t's are t, t + THREADS, ...
template <typename B, int THREADS, int ITEMS>
__device__ __forceinline__ void load_unit(B (&k)[ITEMS], const B* __restrict__ src, u32 n) {
  src += threadIdx.x;
  const int left = int(n) - int(threadIdx.x);
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    if (i * THREADS < left) k[i] = __ldcg(src + i * THREADS);
}

constexpr u32 kOneValue = ~0u;

// The fast way to place NI items per thread (the last four of them perhaps
// not there; the others are, so their latencies overlap): n ordered keys k into
// sm.keys by their bins. Returns the fullest bin's keys, kOneValue when all
// keys are equal, or kBinLimit + 1 when a bin holds more (nothing is placed
// then; the bins' starts, lo, hi and nbins are left in sm for place_by_parts).
template <typename B, int THREADS, int ITEMS, int NI>
__device__ __forceinline__ u32 place_by_bins(const B (&k)[ITEMS], u32 n, LocalSmem<B, THREADS, ITEMS>& sm) {
  constexpr u32 kLimit = kBinLimit<B>;
  constexpr u32 kGroup = 4u * THREADS;  // bins of one scan group
  constexpr int kSure = NI > 4 ? (NI % 4 ? NI / 4 * 4 : NI - 4) : 0;
  constexpr u32 groups = (NI + 3) / 4;
  constexpr u32 nbins = groups * kGroup;  // about one bin per key
  static_assert(nbins <= LocalSmem<B, THREADS, ITEMS>::kBins, "bins fit");
  const u32 tid = threadIdx.x;
  const int left = int(n) - int(tid);
  u32 ranks[(NI + 7) / 8];  // 4 bits per key: enough when no bin is crowded
#pragma unroll
  for (int i = 0; i < (NI + 7) / 8; ++i) ranks[i] = 0u;
#pragma unroll
  for (u32 g = 0; g < groups; ++g) reinterpret_cast<uint4*>(sm.bins)[g * THREADS + tid] = make_uint4(0u, 0u, 0u, 0u);
  B lo = ~B(0), hi = B(0);
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    if (i < kSure || i * THREADS < left) {
      lo = k[i] < lo ? k[i] : lo;
      hi = k[i] > hi ? k[i] : hi;
    }
  }
  block_min_max<THREADS, B>(lo, hi, sm.mm);
  if (lo == hi) return kOneValue;
  const Bins<B> bins(lo, hi - lo, nbins);
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    if (i < kSure || i * THREADS < left) {
      const u32 b = u32(bins.product(k[i]) >> 32);
      ranks[i / 8] += atomicAdd(sm.bins + b, 1u) << (4 * (i % 8));
    }
  }
  __syncthreads();
  const u32 most = scan_counters<THREADS, int(groups)>(sm.bins, groups, sm.tmp, sm.most);
  __syncthreads();
  if (!bins.exact && most > kLimit) {
    if (tid == 0) {
      sm.bins[nbins] = n;
      sm.mm[0] = lo;
      sm.mm[1] = hi;
      sm.nbins = nbins;
    }
    return kLimit + 1u;
  }
  if (most > 15u) {  // a bin per value: many equal keys, in any order
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (i < kSure || i * THREADS < left) sm.keys[atomicAdd(sm.bins + u32(bins.product(k[i]) >> 32), 1u)] = k[i];
    return 0u;
  }
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    if (i < kSure || i * THREADS < left) {
      const u32 b = u32(bins.product(k[i]) >> 32);
      sm.keys[sm.bins[b] + ((ranks[i / 8] >> (4 * (i % 8))) & 15u)] = k[i];
    }
  }
  return bins.exact ? 0u : most;
}

// The same after place_by_bins found a bin too full: each bin [s, e) is cut into
// e - s equal parts, numbered like the positions, which evens out a density that
// is smooth within the bins. Returns the fullest part's keys, at most
// kBinLimit + 1: if such a part's keys are equal, as they mostly are, or only a
// few too many, kBinLimit rounds, once or a few times, still finish the order
// (in_order tells). Begins with a barrier.
template <typename B, int THREADS, int ITEMS>
__device__ __forceinline__ u32 place_by_parts(const B (&k)[ITEMS], u32 n, LocalSmem<B, THREADS, ITEMS>& sm) {
  constexpr u32 kGroup = 4u * THREADS;
  constexpr int kGroups = (ITEMS + 3) / 4;
  static_assert(kGroups * kGroup * 4 <= sizeof(sm.keys), "the parts' counters lie over the keys");
  const u32 tid = threadIdx.x;
  const int left = int(n) - int(tid);
  u32* const parts = reinterpret_cast<u32*>(sm.keys);
  const u32 groups = (n + kGroup - 1) / kGroup;
  for (u32 g = 0; g < groups; ++g) reinterpret_cast<uint4*>(parts)[g * THREADS + tid] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const Bins<B> bins(sm.mm[0], sm.mm[1] - sm.mm[0], sm.nbins);
  auto part_of = [&](B key) {
    const u64 p = bins.product(key);
    const u32 b = u32(p >> 32), s = sm.bins[b], e = sm.bins[b + 1u];
    return s + __umulhi(u32(p), e - s);
  };
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    if (i * THREADS < left) atomicAdd(parts + part_of(k[i]), 1u);
  __syncthreads();
  const u32 most = scan_counters<THREADS, kGroups>(parts, groups, sm.tmp, sm.most);
  __syncthreads();
  u32 at[(ITEMS + 1) / 2];  // two 16-bit positions a word
#pragma unroll
  for (int i = 0; i < (ITEMS + 1) / 2; ++i) at[i] = 0u;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    if (i * THREADS < left) at[i / 2] |= atomicAdd(parts + part_of(k[i]), 1u) << (16 * (i & 1));
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    if (i * THREADS < left) sm.keys[(at[i / 2] >> (16 * (i & 1))) & 0xFFFFu] = k[i];
  return min(most, kBinLimit<B> + 1u);
}

// place_by_bins for the items that n takes. No barrier at the end.
template <typename B, int THREADS, int ITEMS>
__device__ __forceinline__ u32 place_keys(const B (&k)[ITEMS], u32 n, LocalSmem<B, THREADS, ITEMS>& sm) {
  const u32 fours = (n + 4u * THREADS - 1u) / (4u * THREADS);
  u32 rounds = 0;
  // The cases below ITEMS, then all items.
#define MGS_PLACE(F)                                                                             \
  if (4 * F < ITEMS && fours <= F) {                                                             \
    rounds = place_by_bins<B, THREADS, ITEMS, (4 * F < ITEMS ? 4 * F : ITEMS)>(k, n, sm);        \
  } else
  MGS_PLACE(1)
  MGS_PLACE(2)
  MGS_PLACE(3)
  MGS_PLACE(4)
  MGS_PLACE(5)
  MGS_PLACE(6) { rounds = place_by_bins<B, THREADS, ITEMS, ITEMS>(k, n, sm); }
#undef MGS_PLACE
  if (rounds != kOneValue && rounds > kBinLimit<B>) rounds = place_by_parts<B, THREADS, ITEMS>(k, n, sm);
  return rounds;
}

// Whether the n placed keys are in order; the same in every thread. Ends with a barrier.
template <typename B, int THREADS, int ITEMS>
__device__ __forceinline__ bool in_order(u32 n, LocalSmem<B, THREADS, ITEMS>& sm) {
  const u32 at = threadIdx.x * u32(ITEMS);
  bool bad = false;
  if (at < n) {
    B x[ITEMS];
    load_run<B, ITEMS>(sm.keys + at, x);
#pragma unroll
    for (int i = 0; i + 1 < ITEMS; ++i) bad |= x[i + 1] < x[i];
    bad |= at + u32(ITEMS) < n && sm.keys[at + u32(ITEMS)] < x[ITEMS - 1];
  }
  return __syncthreads_or(bad) == 0;
}

// Orders the placed keys within their bins. Begins and ends with a barrier.
template <typename B, int THREADS, int ITEMS>
__device__ __forceinline__ void finish_order(u32 n, u32 rounds, LocalSmem<B, THREADS, ITEMS>& sm) {
  const u32 tid = threadIdx.x;
  // After the last key, keys that sort last: the windows below may read them.
  if (tid < u32(ITEMS) + 16u && n + tid < u32(THREADS) * ITEMS + 16u) sm.keys[n + tid] = ~B(0);
  __syncthreads();
  if (rounds > 1u) {  // kBinLimit + 1 means kBinLimit
    if (tid * u32(ITEMS) < n) {
      B x[ITEMS];
      load_run<B, ITEMS>(sm.keys + tid * ITEMS, x);
      transpose_rounds<B, ITEMS>(x, rounds);
      store_run<B, ITEMS>(sm.keys + tid * ITEMS, x);
    }
    __syncthreads();
    // Bins that cross into the next thread's keys: the keys around the border.
    constexpr u32 border = kBorder<B>;
    static_assert(2 * border <= u32(ITEMS) && kBinLimit<B> - 1 <= border, "windows are disjoint and wide enough");
    const u32 w0 = (tid + 1u) * u32(ITEMS) - border;
    if (tid + 1u < u32(THREADS) && w0 + border < n) {
      B x[2 * border];
      load_run<B, 2 * border>(sm.keys + w0, x);
      transpose_rounds<B, 2 * border>(x, rounds);
      store_run<B, 2 * border>(sm.keys + w0, x);
    }
    __syncthreads();
  }
}

// Merge sort of the n keys in shared memory: each thread's consecutive keys by
// transposition in registers, then rounds of pairwise merges, a thread per ITEMS
// consecutive outputs. Pairs that are in order already (most are: the bins came
// out in order) are left as they are. Begins after and ends with a barrier.
// Bound by the latency of shared memory (a chain of ITEMS reads per round). It
// took the place of binning crowded parts again, one after the other, and of
// networks of one warp, whose cost grew with the number of clusters. B200, whole
// sorts of 2000 clusters of int64: 10^6 187 -> 150 us, 3 * 10^6 310 -> 240,
// 10^7 724 -> 554.
template <typename B, int THREADS, int ITEMS>
__device__ __forceinline__ void merge_order(u32 n, LocalSmem<B, THREADS, ITEMS>& sm) {
  const u32 at = threadIdx.x * u32(ITEMS);
  B x[ITEMS];
  if (at < n) {
    load_run<B, ITEMS>(sm.keys + at, x);
#pragma unroll 1
    for (int r = 0; r < ITEMS; r += 2) transpose_twice<B, ITEMS>(x);
    store_run<B, ITEMS>(sm.keys + at, x);  // what lies after the last key sorts last (finish_order)
  }
  __syncthreads();
#pragma unroll 1
  for (u32 w = ITEMS; w < n; w *= 2u) {  // runs of w keys
    const u32 a0 = at - at % (2u * w), b0 = a0 + w, b1 = min(b0 + w, n);
    const bool merge = at < n && b0 < n && sm.keys[b0] < sm.keys[b0 - 1u];
    if (merge) {
      const u32 d = at - a0;  // outputs of this pair before this thread's
      u32 lo = d > b1 - b0 ? d - (b1 - b0) : 0u, hi = min(d, w);  // how many of them are the first run's
      while (lo < hi) {
        const u32 mid = (lo + hi) / 2u;
        if (sm.keys[b0 + (d - 1u - mid)] < sm.keys[a0 + mid]) {
          hi = mid;
        } else {
          lo = mid + 1u;
        }
      }
      u32 i = a0 + lo, j = b0 + (d - lo);
      B u = sm.keys[i], v = sm.keys[j];
#pragma unroll
      for (int t = 0; t < ITEMS; ++t) {  // after the last output both runs are used up: the padding follows
        const bool first = i < b0 && (j >= b1 || !(v < u));
        x[t] = first ? u : v;
        if (first) {
          u = sm.keys[++i];
        } else {
          v = sm.keys[++j];
        }
      }
    }
    __syncthreads();
    if (merge) store_run<B, ITEMS>(sm.keys + at, x);
    __syncthreads();
  }
}

// Whether the keys are in order after finish_order and, when a bin held more
// than kBinLimit keys, a few more of its rounds: they do for bins that are only
// a little too full. merge_order is for the others.
template <typename B, int THREADS, int ITEMS>
__device__ __forceinline__ bool finished(u32 n, u32 rounds, LocalSmem<B, THREADS, ITEMS>& sm) {
  if (rounds <= kBinLimit<B>) return true;
  for (u32 tries = 0; !in_order<B, THREADS, ITEMS>(n, sm); ++tries) {
    if (tries == 2u) return false;
    finish_order<B, THREADS, ITEMS>(n, rounds, sm);
  }
  return true;
}

template <typename B, int KIND, int THREADS, int ITEMS>
__device__ __forceinline__ void store_unit(B* __restrict__ dst, u32 n, LocalSmem<B, THREADS, ITEMS>& sm) {
  dst += threadIdx.x;
  const int left = int(n) - int(threadIdx.x);
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    if (i * THREADS < left) dst[i * THREADS] = from_ordered<B, KIND>(sm.keys[i * THREADS + threadIdx.x]);
}

template <typename B>
__device__ __forceinline__ const B* unit_keys(const Sort<B>& a, uint2 unit) {
  return a.buf((unit.y & kUnitSrc) ? 1u : 0u) + unit.x;
}
// Keys of a unit that are loaded to be sorted.
__device__ __forceinline__ u32 unit_load(uint2 unit) { return (unit.y & kUnitCopy) ? 0u : unit.y & kUnitLen; }

// A unit whose keys are in k. ahead() runs once k is no longer needed. False
// when bins were crowded with different keys: nothing is stored then, and the
// keys are left in shared memory, not in order (merge_order is not called here,
// because in part_local's loop it costs registers that the common way needs).
template <typename B, int KIND, int THREADS, int ITEMS, class Ahead>
__device__ __forceinline__ bool sort_unit(const Sort<B>& a, uint2 unit, const B (&k)[ITEMS],
                                          LocalSmem<B, THREADS, ITEMS>& sm, Ahead&& ahead) {
  const u32 len = unit.y & kUnitLen;
  B* dst = a.keys + unit.x;
  if (unit.y & kUnitCopy) {
    ahead();
    const B* src = unit_keys(a, unit);
#pragma unroll 4
    for (u32 i = threadIdx.x; i < len; i += THREADS) dst[i] = from_ordered<B, KIND>(__ldcg(src + i));
    return true;
  }
  const u32 rounds = place_keys<B, THREADS, ITEMS>(k, len, sm);
  if (rounds == kOneValue) {
    const B key = from_ordered<B, KIND>(k[0]);
    for (u32 i = threadIdx.x; i < len; i += THREADS) dst[i] = key;
    ahead();
    return true;
  }
  ahead();
  finish_order<B, THREADS, ITEMS>(len, rounds, sm);
  if (!finished<B, THREADS, ITEMS>(len, rounds, sm)) return false;
  store_unit<B, KIND, THREADS, ITEMS>(dst, len, sm);
  return true;
}

// A unit by itself; crowded: the common way failed on it before. Not inlined: the tail calls it in three places.
template <typename B, int KIND, int THREADS, int ITEMS>
__device__ __noinline__ void sort_any_unit(const Sort<B>& a, uint2 unit, bool crowded, LocalSmem<B, THREADS, ITEMS>& sm) {
  const u32 len = unit.y & kUnitLen;
  B k[ITEMS];
  load_unit<B, THREADS, ITEMS>(k, unit_keys(a, unit), unit_load(unit));
  __syncthreads();  // the last use of sm
  if (crowded) {
    const int left = int(len) - int(threadIdx.x);
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) sm.keys[i * THREADS + threadIdx.x] = i * THREADS < left ? k[i] : ~B(0);
    __syncthreads();
  } else if (sort_unit<B, KIND, THREADS, ITEMS>(a, unit, k, sm, [] {})) {
    return;
  }
  merge_order<B, THREADS, ITEMS>(len, sm);
  store_unit<B, KIND, THREADS, ITEMS>(a.keys + unit.x, len, sm);
}

template <typename B, int KIND>
__global__ __launch_bounds__(Shape<sizeof(B)>::kLocalThreads, Shape<sizeof(B)>::kLocalBlocks) void part_local_kernel(Sort<B> a) {
  constexpr int THREADS = Shape<sizeof(B)>::kLocalThreads, ITEMS = Shape<sizeof(B)>::kLocalItems;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  auto& sm = *reinterpret_cast<LocalSmem<B, THREADS, ITEMS>*>(smem_raw);
  __shared__ uint2 s_next[2];  // the next unit, by the parity of the one being sorted
  const u32 units = __ldcg(&a.st->units);
  if (blockIdx.x >= units) return;
  uint2 cur = __ldcg(a.units + blockIdx.x);
  B k[ITEMS];
  load_unit<B, THREADS, ITEMS>(k, unit_keys(a, cur), unit_load(cur));
  for (u32 turn = 0;; turn ^= 1u) {
    // One thread of the last warp claims the next unit while this one is placed; its keys are loaded while this
    // one is brought into order and stored.
    if (threadIdx.x == THREADS - 32) {
      const u32 u = gridDim.x + atomicAdd(&a.st->next_unit, 1u);
      s_next[turn] = u < units ? __ldcg(a.units + u) : make_uint2(0u, 0u);
    }
    if (cur.y & kUnitCopy) __syncthreads();  // else place_keys has barriers
    uint2 next;
    const bool done = sort_unit<B, KIND, THREADS, ITEMS>(a, cur, k, sm, [&] {
      next = s_next[turn];
      load_unit<B, THREADS, ITEMS>(k, unit_keys(a, next), unit_load(next));
    });
    if (!done && threadIdx.x == 0) a.left[atomicAdd(&a.st->left, 1u)] = cur;  // the tail's
    if (next.y == 0u) break;
    cur = next;
    __syncthreads();
  }
}

// The whole input in one block.
template <typename B, int KIND, int THREADS>
__global__ __launch_bounds__(THREADS, 1) void part_small_kernel(B* keys, u32 n) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  auto& sm = *reinterpret_cast<LocalSmem<B, THREADS, Shape<sizeof(B)>::kWideItems>*>(smem_raw);
  constexpr int ITEMS = Shape<sizeof(B)>::kWideItems;
  B k[ITEMS];
  bool neg = false;
  load_unit<B, THREADS, ITEMS>(k, keys, n);
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    k[i] = to_ordered<B, KIND>(k[i]);
    if (KIND == kFloatKey && u32(i * THREADS) + threadIdx.x < n) neg |= k[i] == kNegZero<B>;
    k[i] = one_zero<B, KIND>(k[i]);
  }
  const u32 rounds = place_keys<B, THREADS, ITEMS>(k, n, sm);
  if (rounds == kOneValue) return;
  finish_order<B, THREADS, ITEMS>(n, rounds, sm);
  if (!finished<B, THREADS, ITEMS>(n, rounds, sm)) merge_order<B, THREADS, ITEMS>(n, sm);
  if (KIND == kFloatKey) {
    if (__syncthreads_or(neg)) order_zeros<B, KIND, THREADS, ITEMS>(keys, n, sm);
  }
  store_unit<B, KIND, THREADS, ITEMS>(keys, n, sm);
}

// ---------------------------------------------------------------- merge -----
// One output tile of a k-way merge of integer keys: the tile's slice of every
// run (from the split matrix) is read in run order and sorted like a unit; equal
// keys are the same bytes, so the merge's order among them does not show.
// Tiles of kWideCap keys: half as many splits to find as with the units' blocks.
// 2^28 uint32, 16 runs: 1.19 ms against 1.96 ms of four merge rounds.
template <typename B, int KIND>
__global__ __launch_bounds__(kThreads, 2) void kway_unit_tile_kernel(const B* const* __restrict__ runs, int k,
                                                                     const u64* __restrict__ splits,
                                                                     B* __restrict__ out, u64 total, u64 tile0) {
  constexpr int ITEMS = Shape<sizeof(B)>::kWideItems;
  using Smem = LocalSmem<B, kThreads, ITEMS>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const B** sptr = reinterpret_cast<const B**>(smem_raw + (sizeof(Smem) + 15) / 16 * 16);  // slice r's first key - seg0[r]
  u32* seg0 = reinterpret_cast<u32*>(sptr + k);  // slice offsets in the tile (k + 1)
  const u32 tid = threadIdx.x;
  const u64 j = tile0 + blockIdx.x;
  const u64 d0 = j * u64(kWideCap<B>);
  const u32 cnt = u32(min(u64(kWideCap<B>), total - d0));
  const u32 per_thread = (u32(k) + kThreads - 1u) / kThreads;
  u32 local = 0;
  for (u32 i = 0; i < per_thread; ++i) {
    const u32 r = tid * per_thread + i;
    if (r < u32(k)) local += u32(splits[(j + 1) * k + r] - splits[j * k + r]);
  }
  u32 tot;
  u32 at = block_scan<kThreads>(local, sm.tmp[0], &tot);
  for (u32 i = 0; i < per_thread; ++i) {
    const u32 r = tid * per_thread + i;
    if (r < u32(k)) {
      const u64 s = splits[j * k + r];
      seg0[r] = at;
      sptr[r] = runs[r] + s - at;
      at += u32(splits[(j + 1) * k + r] - s);
    }
  }
  if (tid == 0) seg0[k] = cnt;
  __syncthreads();
  // Consecutive threads read consecutive keys; a thread's slice only moves forward (its keys are kThreads apart).
  B key[ITEMS];
  {
    u32 r = 0, hi = u32(k);  // the largest r with seg0[r] <= tid
    while (hi - r > 1u) {
      const u32 mid = (r + hi) >> 1;
      if (seg0[mid] <= tid) {
        r = mid;
      } else {
        hi = mid;
      }
    }
    u32 end = seg0[r + 1u];
    const B* base = sptr[r];
#pragma unroll
    for (int t = 0; t < ITEMS; ++t) {
      const u32 i = u32(t) * kThreads + tid;
      if (i < cnt) {
        if (i >= end) {
          do {
            ++r;
          } while (seg0[r + 1u] <= i);  // seg0[k] = cnt > i ends the walk
          end = seg0[r + 1u];
          base = sptr[r];
        }
        key[t] = __ldg(base + i);
      }
    }
  }
#pragma unroll
  for (int t = 0; t < ITEMS; ++t) key[t] = to_ordered<B, KIND>(key[t]);
  const u32 rounds = place_keys<B, kThreads, ITEMS>(key, cnt, sm);
  if (rounds == kOneValue) {
    const B one = from_ordered<B, KIND>(key[0]);
    for (u32 i = tid; i < cnt; i += kThreads) out[d0 + i] = one;
    return;
  }
  finish_order<B, kThreads, ITEMS>(cnt, rounds, sm);
  if (!finished<B, kThreads, ITEMS>(cnt, rounds, sm)) merge_order<B, kThreads, ITEMS>(cnt, sm);
  store_unit<B, KIND, kThreads, ITEMS>(out + d0, cnt, sm);
}

// ---------------------------------------------------------------- P4 --------
template <typename B>
union TailSmem {
  struct {
    MapSmem<B> map;
    alignas(16) u32 scratch[kHistWords];
  } map;
  HistSmem<B> hist;
  PlanSmem plan;
  ScatterSmem<B> scatter;
  LocalSmem<B, kThreads, Shape<sizeof(B)>::kWideItems> local;
};

// The segments that are left: most hold one value many times (their cell was
// not known to). Compares every key with its segment's first one, and meanwhile
// stores it where the segment sits in the scratch buffer; segments in the
// caller's buffer are only read.
template <typename B, int KIND>
__device__ void probe_segments(const Sort<B>& a) {
  Segment* const segs = a.segs(a.last_list);
  const u64 list = __ldcg(&a.st->list[a.last_list]);
  const u32 nseg = u32(list >> 32), tiles = u32(list);
  for (u32 t = blockIdx.x; t < tiles; t += gridDim.x) {
    const u32 s = segment_of(segs, nseg, t);
    const u32 start = __ldcg(&segs[s].start), len = __ldcg(&segs[s].len), src = __ldcg(&segs[s].src);
    const u32 first = (t - __ldcg(&segs[s].tile_base)) * kTile<B>;
    const u32 cnt = min(kTile<B>, len - first);
    const B* p = a.buf(src) + start;
    const B key = __ldcg(p);
    if (__syncthreads_or(ld_volatile_u32(&segs[s].done) == 0u)) continue;
    bool other = false;
#pragma unroll 4
    for (u32 i = threadIdx.x; i < cnt; i += kThreads) {
      other |= __ldcg(p + first + i) != key;
      if (src) a.keys[start + first + i] = from_ordered<B, KIND>(key);
    }
    if (__syncthreads_or(other) && threadIdx.x == 0 && atomicExch(&segs[s].done, 0u) != 0u) {
      segs[s].identity = 0u;
      atomicAdd(&a.st->dirty, 1u);
    }
  }
}

// Cooperative launch. Sorts the units that are left, then goes on with the
// segments of list `cur`, if any are left; last, the zeros' signs.
template <typename B, int KIND>
__global__ __launch_bounds__(kThreads, 2) void part_tail_kernel(Sort<B> a, u32 cur) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  TailSmem<B>& sm = *reinterpret_cast<TailSmem<B>*>(smem_raw);
  __shared__ MapTable<B> tab;
  const u32 tid = threadIdx.x, G = gridDim.x, b = blockIdx.x;
  const u32 spins = g_barrier_spins;
  u32 waits = 0;
  bool ok = true;
  constexpr int ITEMS = Shape<sizeof(B)>::kWideItems;
  u32 left = __ldcg(&a.st->left);  // the list up to here is done
  // From the last block on: the first ones probe, meanwhile.
  for (u32 u = G - 1u - b; u < left; u += G) {
    const uint2 unit = __ldcg(a.left + u);
    sort_any_unit<B, KIND, kThreads, ITEMS>(a, unit, (unit.y & kUnitLen) <= kCap<B>, sm.local);
  }
  if (__ldcg(&a.st->list[cur]) != 0u) {
    probe_segments<B, KIND>(a);
    ok = grid_barrier(a.st, ++waits * G, spins, a.status);
  }
  // Probed segments of one value that sit in the caller's buffer: to the caller's bits. Tile by tile: a loop over the
  // segments in every block was a chain of dependent reads, 1.3 us per segment (27 segments, 3 * 10^6 float64 with a
  // heavy tail: 240 -> 206 us).
  if (KIND != kUnsignedKey && ok) {
    const Segment* segs = a.segs(cur);
    const u64 list = __ldcg(&a.st->list[cur]);
    for (u32 t = b; t < u32(list); t += G) {
      const Segment* seg = segs + segment_of(segs, u32(list >> 32), t);
      if (!__ldcg(&seg->done) || __ldcg(&seg->src)) continue;
      const u32 first = (t - __ldcg(&seg->tile_base)) * kTile<B>;
      const u32 cnt = min(kTile<B>, __ldcg(&seg->len) - first);
      B* p = a.keys + __ldcg(&seg->start) + first;
#pragma unroll 4
      for (u32 i = tid; i < cnt; i += kThreads) p[i] = from_ordered<B, KIND>(__ldcg(p + i));
    }
  }
  for (bool first = true; ok; first = false) {
    const u64 list = __ldcg(&a.st->list[cur]);
    const u32 nseg = u32(list >> 32), tiles = u32(list);
    if (nseg == 0 || (first && __ldcg(&a.st->dirty) == 0u)) break;
    const u32 t0 = u32(u64(tiles) * b / G), t1 = u32(u64(tiles) * (b + 1) / G);
    const u32 cells = nseg * 8u + tiles * kCellsPerTile<B>;
    for (u32 i = b * kThreads + tid; i < cells; i += G * kThreads) a.count0[i] = 0u;
    if (!(ok = grid_barrier(a.st, ++waits * G, spins, a.status))) break;
    if (b == 0 && tid == 0) {
      a.st->units = 0;
      a.st->list[cur ^ 1u] = 0;
    }
    map_segments<B, kUnsignedKey>(a, a.segs(cur), b, G, nseg, sm.map.map, sm.map.scratch);
    if (!(ok = grid_barrier(a.st, ++waits * G, spins, a.status))) break;
    histogram_tiles<B, kUnsignedKey, false>(a, a.segs(cur), nseg, a.count0, t0, t1, sm.hist);
    if (!(ok = grid_barrier(a.st, ++waits * G, spins, a.status))) break;
    for (u32 s = b; s < nseg; s += G) {
      if (__ldcg(&a.segs(cur)[s].done)) continue;
      __syncthreads();
      load_table<B>(tab, a.tables + s);
      plan_segment<B>(a, a.segs(cur) + s, load_map<B>(a.maps + s), tab, cur ^ 1u, false, false, a.count0, sm.plan);
    }
    if (!(ok = grid_barrier(a.st, ++waits * G, spins, a.status))) break;
    scatter_tiles<B, kUnsignedKey, false>(a, a.segs(cur), t0, t1, sm.scatter);
    if (!(ok = grid_barrier(a.st, ++waits * G, spins, a.status))) break;
    const u32 units = __ldcg(&a.st->units);
    for (u32 u = b; u < units; u += G) sort_any_unit<B, KIND, kThreads, ITEMS>(a, __ldcg(a.units + u), false, sm.local);
    const u32 more = __ldcg(&a.st->left);
    for (u32 u = left + b; u < more; u += G) sort_any_unit<B, KIND, kThreads, ITEMS>(a, __ldcg(a.left + u), false, sm.local);
    left = more;
    cur ^= 1u;
    // The lists and units of this level are read before any block starts the next one's first step (the
    // next level's first barrier comes before its first write to them).
  }
  if (KIND == kFloatKey && ok) {
    const u32 neg = __ldcg(&a.st->neg_zeros), pos = __ldcg(&a.st->pos_zeros);
    if (neg && !__ldcg(&a.st->in_place)) {
      if ((waits || left) && !grid_barrier(a.st, ++waits * G, spins, a.status)) return;  // every key is in its place
      constexpr B sign = B(1) << (sizeof(B) * 8 - 1);
      const u32 lo = __ldcg(&a.st->below_zeros);
      const u32 zeros = neg + pos;
#pragma unroll 4
      for (u64 i = b * kThreads + tid; i < zeros; i += G * kThreads)  // 64 bits: a step past 2^32 must not wrap
        a.keys[lo + i] = !pos || ((__ldcg(a.zero_signs + (i >> 5)) >> (i & 31u)) & 1u) ? sign : B(0);
    }
  }
}

// ---------------------------------------------------------------- host ------
size_t align_up(size_t x, size_t to) { return (x + to - 1) / to * to; }

struct Layout {
  size_t segs_off[2], counts_off[2], cursor_off, maps_off, tables_off, tiles_off, units_off, left_off, zeros_off, signs_off, keys_off,
      total, clear_bytes;
  size_t max_segs, max_tiles;
  bool small, two_levels;
};

// Scratch for n keys; segments > 0: of a segmented sort with that many large segments at most.
//
// Capacities of the lists (the kernels append without a check). The segments of
// a list are disjoint parts of the array, and a level's cells are disjoint
// parts of its segments, because a segment's counts sum to its length (its
// histogram counts every key once, whatever the keys are):
//   segments: list 1 of a segmented sort has `segments` at most; every other
//             segment has more than kWideCap keys, so n / (kWideCap + 1).
//   tiles   : a full tile per kTile keys and a shorter one per segment.
//   cells   : 8 per segment and kCellsPerTile per tile (see there).
//   units   : with h = kCap / 2: a segment of len keys breaks into at most
//             len / h windows, 2 runs more per cell above h, and 2 at its ends:
//             3 len / h + 2 runs; cells of one value go in chunks of kCap keys or
//             more, and one shorter one. Two levels before the units are sorted,
//             on disjoint keys (a key of the second level has no unit of the
//             first): 3 n / h + 2 segments of list 1 + 3 n / h + 2 n / kWideCap
//             + n / kCap, below 8 n / h + 2 segments + 4096.
//   left    : disjoint runs of more than kCap keys, and units; the list is not
//             emptied between levels, whose keys are disjoint too.
template <typename B, int KIND>
Layout layout(size_t n, size_t segments) {
  Layout L{};
  L.small = segments == 0 && n <= size_t(2 * kThreads) * Shape<sizeof(B)>::kWideItems;
  if (L.small) return L;
  L.two_levels = segments > 0 || n > kOneLevel<B>;
  L.max_segs = std::max(n / (kWideCap<B> + 1) + 1, segments);
  L.max_tiles = n / kTile<B> + L.max_segs + 1;
  const size_t cells = std::max<size_t>(kMaxCells, L.max_segs * 8 + L.max_tiles * kCellsPerTile<B>);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off += align_up(bytes, 256);
    return at;
  };
  // Cleared before every sort: the state, the counts, the tiles' zero counts.
  take(sizeof(State));
  L.counts_off[0] = take(cells * 4);
  L.counts_off[1] = L.two_levels ? take(cells * 4) : L.counts_off[0];
  L.zeros_off = KIND == kFloatKey ? take((n / kTile<B> + 1) * 4) : 0;
  L.clear_bytes = off;
  L.segs_off[0] = take(L.max_segs * sizeof(Segment));
  L.segs_off[1] = take(L.max_segs * sizeof(Segment));
  L.cursor_off = take(cells * 4);
  L.maps_off = take(L.max_segs * sizeof(Map<B>));
  L.tables_off = take(L.max_segs * sizeof(MapTable<B>));
  L.tiles_off = take(L.max_tiles * sizeof(uint4));
  L.units_off = take((8 * (n / (kCap<B> / 2)) + 2 * segments + 4096) * sizeof(uint2));
  L.left_off = take((8 * (n / (kCap<B> / 2)) + 2 * segments + 4096) * sizeof(uint2));
  L.signs_off = KIND == kFloatKey ? take(n / 8 + 8) : 0;
  L.keys_off = take(n * sizeof(B));
  L.total = off;
  return L;
}

template <typename B>
Sort<B> make_sort(const Layout& L, B* keys, size_t n, char* tb, uint32_t* d_status) {
  Sort<B> a;
  a.keys = keys;
  a.tmp = reinterpret_cast<B*>(tb + L.keys_off);
  a.st = reinterpret_cast<State*>(tb);
  a.seg0 = reinterpret_cast<Segment*>(tb + L.segs_off[0]);
  a.seg1 = reinterpret_cast<Segment*>(tb + L.segs_off[1]);
  a.count0 = reinterpret_cast<u32*>(tb + L.counts_off[0]);
  a.count1 = reinterpret_cast<u32*>(tb + L.counts_off[1]);
  a.cursor = reinterpret_cast<u32*>(tb + L.cursor_off);
  a.maps = reinterpret_cast<Map<B>*>(tb + L.maps_off);
  a.tables = reinterpret_cast<MapTable<B>*>(tb + L.tables_off);
  a.tiles = reinterpret_cast<uint4*>(tb + L.tiles_off);
  a.units = reinterpret_cast<uint2*>(tb + L.units_off);
  a.left = reinterpret_cast<uint2*>(tb + L.left_off);
  a.tile_zeros = reinterpret_cast<u32*>(tb + L.zeros_off);
  a.zero_signs = reinterpret_cast<u32*>(tb + L.signs_off);
  a.status = d_status;
  a.n = u32(n);
  a.last_list = L.two_levels ? 0u : 1u;
  return a;
}

struct Device {
  int sms = 148;
};
Device current_device() {
  Device d;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) == cudaSuccess &&
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0)
    d.sms = sms;
  return d;
}

template <typename B, int KIND, int THREADS>
cudaError_t launch_small(B* keys, size_t n, cudaStream_t stream, LaunchRecorder* rec) {
  auto kernel = part_small_kernel<B, KIND, THREADS>;
  constexpr size_t smem = sizeof(LocalSmem<B, THREADS, Shape<sizeof(B)>::kWideItems>);
  static SmemLimitOnce attr;
  cudaError_t e = attr.ensure(kernel, smem);
  if (e != cudaSuccess) return e;
  return launch_kernel(rec, "part_small", kernel, dim3(1), dim3(THREADS), smem, stream, keys, u32(n));
}

template <typename B, int KIND, bool ROOT>
cudaError_t launch_scatter(const Sort<B>& a, unsigned grid, cudaStream_t stream, LaunchRecorder* rec) {
  auto kernel = part_scatter_kernel<B, KIND, ROOT>;
  static SmemLimitOnce attr;
  cudaError_t e = attr.ensure(kernel, sizeof(ScatterSmem<B>));
  if (e != cudaSuccess) return e;
  return launch_kernel(rec, "part_scatter", kernel, dim3(grid), dim3(kThreads), sizeof(ScatterSmem<B>), stream, a);
}

// The level of list 1: KIND and raw as in part_histogram_kernel and plan_segment.
template <typename B, int KIND>
cudaError_t launch_level(const Sort<B>& a, size_t seg_blocks, bool raw, unsigned sms, cudaStream_t stream,
                         LaunchRecorder* rec) {
  cudaError_t e = launch_kernel(rec, "part_map", part_map_kernel<B, KIND>, dim3(unsigned(seg_blocks)), dim3(kThreads), 0,
                                stream, a);
  if (e != cudaSuccess) return e;
  e = launch_kernel(rec, "part_histogram", part_histogram_kernel<B, KIND>, dim3(sms * 2), dim3(kThreads), 0, stream, a);
  if (e != cudaSuccess) return e;
  e = launch_kernel(rec, "part_plan", part_plan_kernel<B>, dim3(unsigned(seg_blocks)), dim3(kThreads), 0, stream, a, raw);
  if (e != cudaSuccess) return e;
  return launch_scatter<B, KIND, false>(a, sms * Shape<sizeof(B)>::kTileBlocks, stream, rec);
}

// The units, then whatever is left.
template <typename B, int KIND>
cudaError_t launch_units(const Sort<B>& a, size_t max_units, unsigned sms, cudaStream_t stream, LaunchRecorder* rec) {
  using LShape = Shape<sizeof(B)>;
  constexpr size_t local_smem = sizeof(LocalSmem<B, LShape::kLocalThreads, LShape::kLocalItems>);
  auto local = part_local_kernel<B, KIND>;
  static SmemLimitOnce local_attr;
  cudaError_t e = local_attr.ensure(local, local_smem);
  if (e != cudaSuccess) return e;
  e = launch_kernel(rec, "part_local", local, dim3(unsigned(std::min<size_t>(max_units, size_t(sms) * LShape::kLocalBlocks))),
                    dim3(LShape::kLocalThreads), local_smem, stream, a);
  if (e != cudaSuccess) return e;
  auto tail = part_tail_kernel<B, KIND>;
  static SmemLimitOnce tail_attr;
  e = tail_attr.ensure(tail, sizeof(TailSmem<B>));
  if (e != cudaSuccess) return e;
  Sort<B> copy = a;
  u32 cur = a.last_list;
  void* args[] = {&copy, &cur};
  // A cooperative grid starts when all its blocks can be resident. With 2 * sms blocks, all that fit, that was when
  // the chip was empty, and kernels of other streams waited meanwhile: the serving loop on four streams came to 3.7
  // Gkeys/s (requests of 2^10..2^18 keys) and 35 (2^10..2^26). With 64, 96, 128, 148, 222 or 256 blocks it came to
  // 5.1-5.3 and 48-49; without this kernel the former to 5.5. A block per SM is also faster than two for the little
  // that is mostly left (3 * 10^6 float64 heavy tail 249 / 280 us); from 2^24 keys on half as many more are (3.3 *
  // 10^7 float32, a third zeros, infinities and NaN: 659 us with 148, 642 with 222; 5 * 10^7 in clusters 2.14 / 2.08 ms).
  const unsigned tail_grid = a.n < (1u << 24) ? sms : sms + sms / 2;
  if (rec) rec->before("part_tail", stream);
  e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(tail), dim3(tail_grid), dim3(kThreads), args,
                                  sizeof(TailSmem<B>), stream);
  if (rec) rec->after("part_tail", stream);
  return e;
}

template <typename B, int KIND>
cudaError_t sort_typed(B* keys, size_t n, void* temp, size_t temp_bytes, cudaStream_t stream, uint32_t* d_status,
                       LaunchRecorder* rec) {
  if (n <= 1) return cudaSuccess;
  constexpr size_t half = size_t(kThreads) * Shape<sizeof(B)>::kWideItems;
  if (n <= half) return launch_small<B, KIND, kThreads>(keys, n, stream, rec);
  if (n <= 2 * half) return launch_small<B, KIND, 2 * kThreads>(keys, n, stream, rec);
  const Layout L = layout<B, KIND>(n, 0);
  if (temp == nullptr || temp_bytes < L.total) return cudaErrorInvalidValue;
  char* tb = static_cast<char*>(temp);
  const Sort<B> a = make_sort<B>(L, keys, n, tb, d_status);
  const unsigned sms = unsigned(current_device().sms);
  const size_t tiles = (n + kTile<B> - 1) / kTile<B>;
  const size_t clear_vecs = L.clear_bytes / 16;
  const size_t clear_blocks = std::min<size_t>((clear_vecs + 4 * kThreads - 1) / (4 * kThreads), size_t(sms) * 2);
  cudaError_t e = launch_kernel(rec, "part_start", part_start_kernel<B, KIND>, dim3(unsigned(1 + clear_blocks)),
                                dim3(kThreads), 0, stream, a, reinterpret_cast<uint4*>(tb), u32(clear_vecs));
  if (e != cudaSuccess) return e;
  const unsigned hist_grid = unsigned(std::min<size_t>(tiles, size_t(sms) * 2));
  e = launch_kernel(rec, "part_histogram", part_histogram_root_kernel<B, KIND>, dim3(hist_grid), dim3(kThreads), 0,
                    stream, a);
  if (e != cudaSuccess) return e;
  e = launch_scatter<B, KIND, true>(a, unsigned(std::min<size_t>(tiles, size_t(sms) * Shape<sizeof(B)>::kTileBlocks)),
                                    stream, rec);
  if (e != cudaSuccess) return e;
  if (L.two_levels) {
    e = launch_level<B, kUnsignedKey>(a, std::min<size_t>(L.max_segs, kMaxCells), false, sms, stream, rec);
    if (e != cudaSuccess) return e;
  }
  return launch_units<B, KIND>(a, 2 * (n / (kCap<B> / 2)) + 1, sms, stream, rec);
}

// The large segments of a segmented sort: one level apart, what it leaves in the tail.
template <typename B, int KIND>
cudaError_t segments_typed(B* keys, size_t n, const u64* offsets, const u32* ids, const u32* count, size_t max_count,
                           void* temp, size_t temp_bytes, cudaStream_t stream, uint32_t* d_status,
                           LaunchRecorder* rec) {
  const Layout L = layout<B, KIND>(n, max_count);
  if (temp == nullptr || temp_bytes < L.total) return cudaErrorInvalidValue;
  char* tb = static_cast<char*>(temp);
  const Sort<B> a = make_sort<B>(L, keys, n, tb, d_status);
  const unsigned sms = unsigned(current_device().sms);
  cudaError_t e = cudaMemsetAsync(tb, 0, L.clear_bytes, stream);
  if (e != cudaSuccess) return e;
  e = launch_kernel(rec, "part_segments", part_segments_kernel<B>, dim3(1), dim3(1024), 0, stream, a, offsets, ids,
                    count);
  if (e != cudaSuccess) return e;
  e = launch_level<B, KIND>(a, std::min<size_t>(max_count, size_t(sms) * 4), true, sms, stream, rec);
  if (e != cudaSuccess) return e;
  return launch_units<B, KIND>(a, 2 * (n / (kCap<B> / 2)) + 1, sms, stream, rec);
}

}  // namespace

size_t partition_sort_temp_bytes(int dtype, size_t n) {
  size_t bytes = 0;
  dispatch_dtype(dtype, [&](auto tr) {
    using Tr = decltype(tr);
    bytes = layout<typename Tr::Bits, Tr::kKind>(n, 0).total;
  });
  return bytes;
}

cudaError_t partition_sort(int dtype, void* d_keys, size_t n, void* d_temp, size_t temp_bytes, cudaStream_t stream,
                           uint32_t* d_status, LaunchRecorder* rec) {
  if (n >= (size_t(1) << 32)) return cudaErrorInvalidValue;
  cudaError_t result = cudaErrorInvalidValue;
  dispatch_dtype(dtype, [&](auto tr) {
    using Tr = decltype(tr);
    result = sort_typed<typename Tr::Bits, Tr::kKind>(static_cast<typename Tr::Bits*>(d_keys), n, d_temp, temp_bytes,
                                                      stream, d_status, rec);
  });
  return result;
}

size_t partition_segments_temp_bytes(int dtype, size_t n, size_t max_segments) {
  size_t bytes = 0;
  dispatch_dtype(dtype, [&](auto tr) {
    using Tr = decltype(tr);
    if constexpr (Tr::kKind != kFloatKey) bytes = layout<typename Tr::Bits, Tr::kKind>(n, max_segments).total;
  });
  return bytes;
}

cudaError_t partition_segments(int dtype, void* d_keys, size_t n, const unsigned long long* d_offsets,
                               const uint32_t* d_ids, const uint32_t* d_count, size_t max_segments, void* d_temp,
                               size_t temp_bytes, cudaStream_t stream, uint32_t* d_status, LaunchRecorder* rec) {
  cudaError_t result = cudaErrorInvalidValue;
  dispatch_dtype(dtype, [&](auto tr) {
    using Tr = decltype(tr);
    if constexpr (Tr::kKind != kFloatKey)
      result = segments_typed<typename Tr::Bits, Tr::kKind>(static_cast<typename Tr::Bits*>(d_keys), n, d_offsets, d_ids,
                                                            d_count, max_segments, d_temp, temp_bytes, stream, d_status,
                                                            rec);
  });
  return result;
}

cudaError_t set_barrier_spins(uint32_t spins) {
  const u32 v = spins ? spins : kBarrierSpins;
  return cudaMemcpyToSymbol(g_barrier_spins, &v, sizeof(v));
}

size_t kway_unit_tile_keys(int dtype) {
  size_t keys = 0;
  dispatch_dtype(dtype, [&](auto tr) {
    using Tr = decltype(tr);
    if constexpr (Tr::kKind != kFloatKey) keys = kWideCap<typename Tr::Bits>;
  });
  return keys;
}

cudaError_t kway_unit_tiles(int dtype, const void* d_runs, int k, const uint64_t* d_splits, void* out, uint64_t total,
                            uint64_t tile0, uint64_t tiles, cudaStream_t stream, LaunchRecorder* rec) {
  cudaError_t result = cudaErrorInvalidValue;
  if (k < 1 || k > kMaxUnitTileRuns || tiles == 0 || tiles > 0x7FFFFFFFull) return result;
  dispatch_dtype(dtype, [&](auto tr) {
    using Tr = decltype(tr);
    using B = typename Tr::Bits;
    if constexpr (Tr::kKind != kFloatKey) {
      auto kernel = kway_unit_tile_kernel<B, Tr::kKind>;
      constexpr size_t base = (sizeof(LocalSmem<B, kThreads, Shape<sizeof(B)>::kWideItems>) + 15) / 16 * 16;
      static SmemLimitOnce attr;
      result = attr.ensure(kernel, base + size_t(kMaxUnitTileRuns) * 12 + 4);
      if (result != cudaSuccess) return;
      result = launch_kernel(rec, "kway_unit_tiles", kernel, dim3(unsigned(tiles)), dim3(kThreads),
                             base + size_t(k) * 12 + 4, stream, static_cast<const B* const*>(d_runs), k,
                             reinterpret_cast<const u64*>(d_splits), static_cast<B*>(out), u64(total), u64(tile0));
    }
  });
  return result;
}

}  // namespace mgs
