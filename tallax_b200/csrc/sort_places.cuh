// Stable row-wise argsort by estimated places, rows of up to 131072 elements in the shared memory of a CTA or of a cluster
// of CTAs.  Included by sort.cu.
//
// A radix sort moves every element once per digit, at 128 warp instructions per 32 elements each time.  Here every element is
// moved once, to a place that is estimated from its key, and is then put right among the few that were sent to the same place:
//   * The keys, less the row's least one, are counted in 2048 equal ranges of their bits; inside a range the elements are
//     taken to lie evenly.  That gives every key an estimated place in 0..n-1 which never falls as the key rises.  (Float keys:
//     four ranges an octave, so the density inside one hardly varies.)  16-bit keys take the position as their low bits.
//   * Elements with the same place are a group: they are counted, the counts are summed up, and every element goes to its
//     group, one shared-memory atomic each.  The order inside a group is left to chance.
//   * An element's rank in its group is the number of lesser (key, position) pairs in it: a group has two elements on average.
//   In a cluster every CTA owns a share of the places.  The elements first go to their owners, each once, over distributed
// shared memory and in the order of their positions; everything after that is the owner's alone (four cluster barriers a row,
// where four radix passes took fourteen).
//
// What does not fit takes the radix passes of sort_radix.cuh, with the same result:
//   * rows whose keys differ in two digits at most (16-bit keys: in one), or of which many elements are equal, by a sample:
//     before anything else is done;
//   * rows of which an owner would get more than it has room for: in the cluster, from the elements as they were read;
//   * owners whose groups are large: each its own share, without the cluster, the elements it received being in the order of
//     their positions.
//
// What bounds it: latency and barriers, then instruction issue (about 200 per 32 elements).
// us, radix passes (up to 1024 elements: the bitonic network) / this, normal keys: f32 [128, 65536] 329 / 138, [128, 12000]
// 53 / 17, [1024, 4096] 79 / 32, [64, 4097] 19.4 / 7.8, [1000, 700] 22 / 10.5, [1, 131072] 88 / 38; bf16, of two passes,
// [128, 65536] 178 / 141, [1024, 4096] 46 / 34, [64, 4097] 11.4 / 8.1.
//   Rows that fall back take fewer passes than their digits where their keys have a shorter form: less the least one and without
// the bits that are the same in all of them, or, of few different keys, their numbers, which are one digit.  us, a radix sort of all
// digits / the passes of this kernel on the keys as they are / on the shorter form: rounded keys (27 values) bf16 [128, 65536] 170 / 191 / 140,
// [1024, 4096] 46 / 50 / 41, [64, 4097] 11.2 / 12.0 / 10.0, [1000, 1500] 23.3 / 26.6 / 23.1, f16 [300, 20000] 109 / 120 / 92, f32 [128, 65536] 290 / 186 /
// 136, [1024, 4096] 78 / 46 / 37; the same times a million, i32 [128, 65536] 295 / 303 / 249, [300, 20000] 179 / 199 / 160; two keys of which the first
// has 50 values, bf16 [128, 65536] 456 / 420 / 367.
//   Tried: two places an element (groups of 1.5 elements) made nothing faster and a sort through in_perm a fifth slower, because
// the shared memory it takes is the L1 that the reads through in_perm need.
#pragma once
#include "sort_radix.cuh"

namespace tlx {

constexpr int kPlaceRanges = 2048;
constexpr int kPlacePosBits = 17;             // positions; the group's number in its CTA lies above them
constexpr uint32_t kPlacePosMask = (1u << kPlacePosBits) - 1;
static_assert(kRadixMaxRow <= 1 << kPlacePosBits, "a position fits its bits");
constexpr uint32_t kPlaceMaxGroup = 512;      // elements of a group at most, and ...
constexpr uint32_t kPlaceMaxMean = 24;        // ... of an element's group on average: at seven instructions an element of the group
                                              // a rank then costs what two radix passes do
constexpr int kPlaceWindow = 6;               // elements of a group that every element is compared with before any test
                                              // (six: one element in 1700 is in a larger group, one warp in fifty)

constexpr int kMaxValues = 256;              // different keys of a row whose numbers are one digit
// Entries of the table that numbers them, a byte each, at most: with more of them a pass over the CTA's `cap` elements is the cheaper one
// (f32, with / without: 0..199, 17223 entries, [64, 4097], 4352 elements, 12.7 us / 11.7; [128, 65536], 16384 elements, 154 / 190; 0..49, 4241
// entries, [1000, 1500], 2048 elements, 23.5 / 26.2).
__host__ __device__ constexpr uint32_t value_table_max(uint32_t cap) { return cap < 4096 ? 8192 : 2 * cap; }

struct __align__(16) PlaceShared {
  RadixShared radix;
  uint32_t red[4][32];     // of every warp: least key, greatest key, differing bits; groups' squares
  uint32_t row[4];         // this CTA's: least key, greatest key, differing bits
  union {
    uint32_t to[32][8];            // of every warp: elements for every CTA of the cluster
    uint32_t value[kMaxValues];    // a row of few keys: the keys by their numbers
  };
  uint32_t count[8];       // of this CTA: the same
  struct {
    int encode;              // a row that is sorted by digits: it may have a shorter form
    uint32_t base, most;     // its least and greatest key; shorter form: the base
    uint32_t bits;           // of a key whose first bit is set, those that are the same in all keys
    int shift, numbered;     // shorter form: (key >> shift) - base, or these keys' numbers (before: it may be a row of few keys)
  } coded;
};
static_assert(sizeof(PlaceShared) % 16 == 0, "the counters behind it are cleared 16 bytes at a time");

// Elements that a CTA of a cluster has room for: a sixteenth more than it reads.
template <int IPT, bool CL> constexpr int kPlaceRoom = CL ? IPT + IPT / 16 : IPT;

// Counters a thread: one for every place, or the radix passes' [warps][256].
template <int IPT> constexpr int kPlaceCounters = IPT > 8 ? IPT : 8;

// Dynamic shared memory: PlaceShared, counters [threads * kPlaceCounters] u16, key and
// position pairs and kPlaceWindow more (before them, in the same place: sums of the ranges [2048 + 4] u32, counts of the
// ranges [2048] u16).
template <int IPT, bool CL>
__host__ __device__ __forceinline__ size_t place_smem(int threads) {
  constexpr size_t ranges = (kPlaceRanges + 4) * 4 + kPlaceRanges * 2;
  const size_t pairs = ((size_t)threads * kPlaceRoom<IPT, CL> + kPlaceWindow) * 8;
  static_assert(IPT == 4 || value_table_max(256 * IPT) <= 256 * IPT * 8, "the table of a row of few keys lies in the pairs' place");
  return sizeof(PlaceShared) + (size_t)threads * kPlaceCounters<IPT> * 2 + (pairs > ranges ? pairs : ranges);
}

// Digits that the passes take of keys which differ in the bits `diff`.
__device__ __forceinline__ int differing_digits(uint32_t diff) {
  return (int)((diff & 0xFFu) != 0) + (int)((diff & 0xFF00u) != 0) + (int)((diff & 0xFF0000u) != 0) + (int)((diff >> 24) != 0);
}

// Rows of few different keys, of which every key has marked its entry of `table` [range] u8, the last one's among them: the marks become
// the numbers of the keys in their order, and s.value[number] the key.  False if there are more than kMaxValues.
//   In a cluster every CTA adds the others' marks to its own; the marks are summed up.  No atomics: a mark is the same whoever sets it.
template <bool CL>
static __device__ __forceinline__ bool number_marks(unsigned char* table, uint32_t range, int rank, int cluster, PlaceShared& s) {
  const int nt = blockDim.x, vectors = (int)(range + 15) / 16;
  uint4* t4 = reinterpret_cast<uint4*>(table);
  if constexpr (CL) {
    cl_sync();
    for (int i = threadIdx.x; i < vectors; i += nt) {
      uint4 q = t4[i];
      for (int o = 1; o < cluster; ++o) {   // (what another one may have added by now are marks too)
        const uint4 e = cl_ld_v4(cl_map(t4 + i, (uint32_t)(rank + o < cluster ? rank + o : rank + o - cluster)));
        q.x |= e.x; q.y |= e.y; q.z |= e.z; q.w |= e.w;
      }
      t4[i] = q;
    }
    cl_sync();
  } else {
    __syncthreads();
  }
  // thread t < 256: `per` vectors from t * per on.  Marks -> marks before them (beyond the last mark the bytes may run over).
  const int per = (vectors + 255) / 256, i0 = threadIdx.x * per, i1 = threadIdx.x < 256 ? min(i0 + per, vectors) : 0;
  uint32_t marks = 0;
  for (int i = i0; i < i1; ++i) {
    const uint4 q = t4[i];
    marks += __popc(q.x) + __popc(q.y) + __popc(q.z) + __popc(q.w);
  }
  uint32_t before = radix_scan256(marks, s.radix.warp);
  if (threadIdx.x == 255) s.count[0] = before + marks;
  for (int i = i0; i < i1; ++i) {
    uint4 q = t4[i];
    auto sums = [&](uint32_t& w) {
      const uint32_t at = w * 0x01010101u;
      w = before * 0x01010101u + (at << 8);
      before += at >> 24;
    };
    sums(q.x); sums(q.y); sums(q.z); sums(q.w);
    t4[i] = q;
  }
  __syncthreads();
  if (s.count[0] > kMaxValues) return false;
  // an entry is marked if the next one's number is another one (the last entry is)
  const uint32_t* words = reinterpret_cast<const uint32_t*>(table);
  for (uint32_t i = threadIdx.x; 4 * i < range - 1; i += nt) {
    const uint32_t w = words[i], next = w >> 8 | words[i + 1] << 24;
#pragma unroll
    for (uint32_t b = 0; b < 4; ++b)
      if (((w ^ next) >> 8 * b & 255u) && 4 * i + b < range - 1) s.value[w >> 8 * b & 255u] = 4 * i + b;
  }
  if (threadIdx.x == 0) s.value[s.count[0] - 1] = range - 1;
  return true;
}

template <int DT, int IPT, bool CL, bool PAST>
__global__ void __launch_bounds__(kRadixMaxThreads) sort_places_kernel(
    const typename Elem<DT>::type* __restrict__ keys, const int32_t* __restrict__ in_perm, int64_t n64, int descending,
    typename Elem<DT>::type* __restrict__ out_keys, int32_t* __restrict__ out_perm, int cluster,
    const __grid_constant__ SortCarry carry) {
  using RK = RadixKey<DT>;
  using T = typename Elem<DT>::type;
  constexpr bool kHalf = RK::kBits == 16;
  constexpr int kRoom = kPlaceRoom<IPT, CL>;
  constexpr bool kShorter = IPT > 4;   // (four elements a thread: a pass costs little more than the search for a shorter form)
  extern __shared__ __align__(16) unsigned char place_raw[];
  const int nt = blockDim.x, nw = nt >> 5, cap = nt * IPT, n = (int)n64;
  const int lane = lane_id(), w = warp_id();
  PlaceShared& s = *reinterpret_cast<PlaceShared*>(place_raw);
  uint32_t* group = reinterpret_cast<uint32_t*>(place_raw + sizeof(PlaceShared));   // two counters a word
  unsigned short* group_half = reinterpret_cast<unsigned short*>(group);
  uint2* pair = reinterpret_cast<uint2*>(group + nt * kPlaceCounters<IPT> / 2);
  uint32_t* sum = reinterpret_cast<uint32_t*>(pair);                                // elements in the ranges before
  uint32_t* range = sum + kPlaceRanges + 4;                                         // two counters a word
  const int rank = CL ? (int)cl_rank() : 0;
  const int64_t row = CL ? blockIdx.x / cluster : blockIdx.x;
  const int c0 = rank * cap;
  const T* krow = keys + row * n64;
  const int32_t* prow = in_perm ? in_perm + row * n64 : nullptr;
  const uint32_t flip = descending ? (kHalf ? 0xFFFFu : 0xFFFFFFFFu) : 0u;
  // 16-bit keys: the position, as 65536ths of the row, in the low bits, so that equal keys lie evenly too
  const uint32_t pos_scale = kHalf ? 2 * (0xFFFFFFFFu / (uint32_t)n) : 0u;
  // the element of key `key` and position `pos` goes to place `at` of the row
  auto emit = [&](int at, uint32_t key, uint32_t pos) {
    const int64_t to = row * n64 + at;
    if (out_keys) out_keys[to] = RK::back((kHalf ? key >> 16 : key) ^ flip);
    if (prow) pos = (uint32_t)prow[pos];
    if (out_perm) out_perm[to] = (int32_t)pos;
    carry_one(carry, row * n64 + pos, to);
  };

  grid_wait();
  // element w * 32 * IPT + 32 j + lane of the CTA
  const int i0 = w * 32 * IPT + lane, left = n - (c0 + i0);   // element j is there if 32 j < left
  uint32_t k[kRoom], p[kRoom];
  {
    T raw[IPT];
    if (prow) {
      int32_t at[IPT];
#pragma unroll
      for (int j = 0; j < IPT; ++j) at[j] = 32 * j < left ? prow[c0 + i0 + 32 * j] : 0;
#pragma unroll
      for (int j = 0; j < IPT; ++j) raw[j] = krow[at[j]];
    } else {
#pragma unroll
      for (int j = 0; j < IPT; ++j) raw[j] = krow[32 * j < left ? c0 + i0 + 32 * j : 0];
    }
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      k[j] = RK::make(raw[j]) ^ flip;
      if (kHalf) k[j] = k[j] << 16 | (32 * j < left ? __umulhi((uint32_t)(c0 + i0 + 32 * j) << 15, pos_scale) : 0u);
    }
  }
  for (int i = threadIdx.x; i < kPlaceRanges / 2; i += nt) range[i] = 0;
  // (what was read in the place of elements past the row's end is the row's first element)
  uint32_t least = k[0], greatest = k[0], diff = 0, equal = 0;
  uint32_t first = RK::make(krow[prow ? prow[0] : 0]) ^ flip;
  if (kHalf) first <<= 16;
  // Float keys: of negative numbers all bits are turned round.  A bit that is the same in all of them once that is undone is the
  // same in all keys of one sign, and the last pass parts the signs (f32 of few digits, of both signs: two passes, not four).
  auto upright = [&](uint32_t key) { return DT == TLX_I32 || DT == TLX_U32 ? key : key ^ (~(uint32_t)((int32_t)key >> 31) & 0x7FFFFFFFu); };
  first = upright(first);
#pragma unroll
  for (int j = 0; j < IPT; ++j) {
    least = min(least, k[j]);
    greatest = max(greatest, k[j]);
    diff |= upright(k[j]) ^ first;
  }
  if (kHalf) diff &= 0xFFFF0000u;
  {
    // how often two elements are equal, from a sample of 32 a warp
    const uint32_t there = __ballot_sync(0xFFFFFFFFu, left > 0), like = __match_any_sync(0xFFFFFFFFu, kHalf ? k[0] >> 16 : k[0]) & there;
    equal = __reduce_add_sync(0xFFFFFFFFu, left > 0 ? (uint32_t)__popc(like) - 1u : 0u);
  }
  least = __reduce_min_sync(0xFFFFFFFFu, least);
  greatest = __reduce_max_sync(0xFFFFFFFFu, greatest);
  diff = __reduce_or_sync(0xFFFFFFFFu, diff);
  if (lane == 0) { s.red[0][w] = least; s.red[1][w] = greatest; s.red[2][w] = diff; s.red[3][w] = equal; }
  __syncthreads();
  least = __reduce_min_sync(0xFFFFFFFFu, s.red[0][lane < nw ? lane : 0]);
  greatest = __reduce_max_sync(0xFFFFFFFFu, s.red[1][lane < nw ? lane : 0]);
  diff = __reduce_or_sync(0xFFFFFFFFu, s.red[2][lane < nw ? lane : 0]);
  equal = __reduce_add_sync(0xFFFFFFFFu, lane < nw ? s.red[3][lane] : 0u);
  if constexpr (CL) {
    if (threadIdx.x == 0) { s.row[0] = least; s.row[1] = greatest; s.row[2] = diff; s.row[3] = equal; }
    cl_sync();
    const uint32_t of = (uint32_t)(lane < cluster ? lane : 0);
    least = __reduce_min_sync(0xFFFFFFFFu, cl_ld_u32(cl_map(&s.row[0], of)));
    greatest = __reduce_max_sync(0xFFFFFFFFu, cl_ld_u32(cl_map(&s.row[1], of)));
    diff = __reduce_or_sync(0xFFFFFFFFu, cl_ld_u32(cl_map(&s.row[2], of)));
    equal = __reduce_add_sync(0xFFFFFFFFu, lane < cluster ? cl_ld_u32(cl_map(&s.row[3], of)) : 0u);
  }

  // The radix passes of the whole row.  Rows that need two of them at most are done sooner that way.
  auto whole_row_by_digits = [&](uint32_t passes, bool coded) {
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      p[j] = (uint32_t)(c0 + i0 + 32 * j);
      if (32 * j >= left) k[j] = 0xFFFFFFFFu;
    }
    const bool scattered = radix_by_digits<IPT, CL, PAST>(
        reinterpret_cast<uint32_t(&)[IPT]>(k), reinterpret_cast<uint32_t(&)[IPT]>(p), passes, n, rank, cluster, s.radix, group_half,
        reinterpret_cast<uint32_t*>(pair), reinterpret_cast<uint32_t*>(pair) + cap);
    if constexpr (CL) cl_sync();   // (nobody leaves while another one may still read its counts)
    if (coded) {
      const int shift = s.coded.shift;
      const uint32_t base = s.coded.base, bits = s.coded.bits, low = (1u << shift) - 1u;
      const bool numbered = s.coded.numbered;
#pragma unroll
      for (int j = 0; j < IPT; ++j) {
        const uint32_t top = ((numbered ? s.value[k[j] & 255u] : k[j]) + base) << shift;
        k[j] = top | ((upright(top) == top ? bits : ~bits) & low);
      }
    }
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      const int c = c0 + (scattered ? (int)threadIdx.x + j * nt : i0 + 32 * j);
      if (c < n) emit(c, k[j], p[j]);
    }
  };
  const int digits = differing_digits(diff);
  // Of 992 ordered pairs a warp, n / (32 IPT) warps, these are equal if an element's equals, with itself, are kPlaceMaxMean.
  // 16-bit keys, whose equals lie evenly: if one pair in 64 is, which are keys of a few dozen values.
  const uint32_t many = kHalf ? (uint32_t)n / (2 * IPT) : kPlaceMaxMean * 31 / IPT;
  bool by_digits = digits <= (kHalf ? 1 : 2) || equal > many;
  // (what such a row needs later is left in shared memory: in registers it costs the rest of the kernel spilled ones)
  if (kShorter && threadIdx.x == 0) {
    s.coded.encode = by_digits && digits > 1;
    s.coded.base = least;
    s.coded.most = greatest;
    s.coded.bits = first;
    s.coded.numbered = equal * (8 * IPT) >= (uint32_t)n;   // one pair in 256 is equal, by the sample, as of 256 keys that are equally frequent
  }

  int m = n, out0 = 0;   // CTA: elements that it puts right, and their first place in the row
  if (!by_digits) {
    for (int i = threadIdx.x; i < cap / 8; i += nt) reinterpret_cast<uint4*>(group)[i] = make_uint4(0, 0, 0, 0);
    // counts of the ranges, of the whole row in every CTA, and their sums
    const int bits = 32 - __clz(greatest - least), sh = bits > 11 ? bits - 11 : 0;
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      const uint32_t b = (k[j] - least) >> sh;
      if (32 * j < left && TLX_IN_BOUNDS(b, kPlaceRanges, 37)) atomicAdd(&range[b >> 1], (b & 1) ? 0x10000u : 1u);
    }
    if constexpr (CL) cl_sync();
    else __syncthreads();
    uint32_t c[8] = {}, total = 0;
    if (threadIdx.x < kPlaceRanges / 8) {
      const uint4* mine = reinterpret_cast<const uint4*>(range) + threadIdx.x;
      for (int r = 0; r < (CL ? cluster : 1); ++r) {
        const uint4 q = CL ? cl_ld_v4(cl_map(mine, (uint32_t)r)) : *mine;
        const uint32_t e[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { c[2 * i] += e[i] & 0xFFFFu; c[2 * i + 1] += e[i] >> 16; }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) total += c[i];
    }
    uint32_t before = radix_scan256(total, s.radix.warp);
    if (threadIdx.x < kPlaceRanges / 8) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        sum[8 * threadIdx.x + i] = before;
        before += c[i];
      }
      if (threadIdx.x == kPlaceRanges / 8 - 1) sum[kPlaceRanges] = before;
    }
    __syncthreads();
    // estimated places
    auto place = [&](uint32_t key) {
      const uint32_t o = key - least, b = o >> sh, at = sum[b];
      return at + __umulhi((o << 1) << (31 - sh), sum[b + 1] - at);
    };

    if constexpr (CL) {
      // To the owners: CTA d owns places d * per .. of the row.  e[j]: place, and above its bits the element's rank among
      // the warp's elements for the same CTA.
      const int per = (n + cluster - 1) / cluster;
      const uint32_t inv = 0xFFFFFFFFu / (uint32_t)per + 1;   // place / per: exact while the product of the two is below 2^32
      auto owner = [&](uint32_t at) { return __umulhi(at, inv); };
      uint32_t e[IPT], run = 0;                               // run, lane d: elements for CTA d & 7 so far
      const uint32_t x0 = (lane & 1) ? 0u : ~0u, x1 = (lane & 2) ? 0u : ~0u, x2 = (lane & 4) ? 0u : ~0u;
#pragma unroll
      for (int j = 0; j < IPT; ++j) {
        const bool there = 32 * j < left;
        const uint32_t at = there ? place(k[j]) : 0u, d = owner(at);
        const uint32_t v = __ballot_sync(0xFFFFFFFFu, there);
        const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, d & 1), b1 = __ballot_sync(0xFFFFFFFFu, d & 2), b2 = __ballot_sync(0xFFFFFFFFu, d & 4);
        const uint32_t peers = v & ((d & 1) ? b0 : ~b0) & ((d & 2) ? b1 : ~b1) & ((d & 4) ? b2 : ~b2);
        const uint32_t old = __shfl_sync(0xFFFFFFFFu, run, d);
        e[j] = at | (old + __popc(peers & ((1u << lane) - 1u))) << kPlacePosBits;
        run += __popc(v & (b0 ^ x0) & (b1 ^ x1) & (b2 ^ x2));
      }
      if (lane < 8) s.to[w][lane] = run;
      __syncthreads();
      uint32_t offset = 0, all = 0;   // for CTA lane & 7: of the warps before this one, of the CTA
      for (int i = 0; i < nw; ++i) {
        const uint32_t t = s.to[i][lane & 7];
        if (i < w) offset += t;
        all += t;
      }
      if (threadIdx.x < 8) s.count[lane] = all;
      cl_sync();
      // CTAs r and r + 4, r = lane / 8, give CTA lane & 7 so many elements
      uint32_t got = 0, earlier = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = (lane >> 3) + 4 * h;
        const uint32_t t = r < cluster ? cl_ld_u32(cl_map(&s.count[lane & 7], (uint32_t)r)) : 0u;
        got += t;
        if (r < rank) earlier += t;
      }
      got += __shfl_xor_sync(0xFFFFFFFFu, got, 8);
      got += __shfl_xor_sync(0xFFFFFFFFu, got, 16);
      earlier += __shfl_xor_sync(0xFFFFFFFFu, earlier, 8);
      earlier += __shfl_xor_sync(0xFFFFFFFFu, earlier, 16);
      if (__any_sync(0xFFFFFFFFu, got > (uint32_t)(nt * kRoom))) {
        by_digits = true;   // (every warp of every CTA sees the same numbers)
      } else {
        m = (int)__shfl_sync(0xFFFFFFFFu, got, rank);
        out0 = (int)__reduce_add_sync(0xFFFFFFFFu, lane < rank ? got : 0u);
        const uint32_t mine = cl_map(pair, (uint32_t)(lane & 7) < (uint32_t)cluster ? lane & 7 : 0) + 8u * (offset + earlier);
#pragma unroll
        for (int j = 0; j < IPT; ++j) {
          const uint32_t at = e[j] & kPlacePosMask, d = owner(at);
          const uint32_t to = __shfl_sync(0xFFFFFFFFu, mine, d) + 8u * (e[j] >> kPlacePosBits);
          if (32 * j < left && TLX_IN_BOUNDS(to - cl_map(pair, d), nt * kRoom * 8, 30)) cl_st_u64(to, k[j], (uint32_t)(c0 + i0 + 32 * j) | (at - d * per) << kPlacePosBits);
        }
        cl_sync();   // the last: from here on every CTA is on its own
        // in the order of their positions: element w * 32 * kRoom + 32 j + lane
#pragma unroll
        for (int j = 0; j < kRoom; ++j) {
          const int i = w * 32 * kRoom + 32 * j + lane;
          const uint2 q = i < m ? pair[i] : make_uint2(0xFFFFFFFFu, kPlacePosMask);
          k[j] = q.x;
          p[j] = q.y;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < IPT; ++j) {
        p[j] = (uint32_t)(i0 + 32 * j);
        if (32 * j < left) p[j] |= place(k[j]) << kPlacePosBits;
      }
    }
  }
  if (by_digits) {
    __syncthreads();
    uint32_t passes = diff;
    bool coded = false;
    if (kShorter && s.coded.encode) {
      const int low = __ffs(diff) - 1;
      const uint32_t base = s.coded.base >> low, most = (s.coded.most >> low) - base;
      const bool few = s.coded.numbered && most > 255 && most < value_table_max(cap);
      bool numbered = false;
      if (few || (39 - __clz(most)) / 8 < differing_digits(diff)) {
#pragma unroll
        for (int j = 0; j < IPT; ++j) k[j] = (k[j] >> low) - base;
        if (few) {
          unsigned char* table = reinterpret_cast<unsigned char*>(pair);
          for (uint32_t i = threadIdx.x; i < most / 16 + 1; i += nt) reinterpret_cast<uint4*>(table)[i] = make_uint4(0, 0, 0, 0);
          __syncthreads();
#pragma unroll
          for (int j = 0; j < IPT; ++j)
            if (TLX_IN_BOUNDS(k[j], most + 1, 38)) table[k[j]] = 1;
          numbered = number_marks<CL>(table, most + 1, rank, cluster, s);
          if (numbered) {
#pragma unroll
            for (int j = 0; j < IPT; ++j) k[j] = table[k[j]];
          }
        }
        passes = numbered ? 255 : 0xFFFFFFFFu >> __clz(most);
        __syncthreads();   // (what is read above is overwritten)
        if (threadIdx.x == 0) {
          s.coded.base = base;
          s.coded.shift = low;
          s.coded.numbered = numbered;
        }
        // (passes of their own: where they meet the others' the kernel spills 70 bytes of registers, f32 [1024, 8192] 62.9 us against 61.6)
        if constexpr (!CL) {
          whole_row_by_digits(passes, true);
          return;
        }
        coded = true;
      }
    }
    whole_row_by_digits(passes, CL && coded);
    return;
  }

  const int r0 = w * 32 * kRoom + lane;
#pragma unroll
  for (int j = 0; j < kRoom; ++j) {
    const uint32_t b = p[j] >> kPlacePosBits;
    if (r0 + 32 * j < m && TLX_IN_BOUNDS(b, cap, 31)) atomicAdd(&group[b >> 1], (b & 1) ? 0x10000u : 1u);
  }
  __syncthreads();
  // counts -> first places; how large the groups are
  uint32_t squares = 0, large = 0;
  {
    constexpr int kWords = IPT / 2, kVec = kWords < 4 ? kWords : 4;
    static_assert(kWords % kVec == 0 && (kVec == 2 || kVec == 4), "a thread's counters are whole vectors");
    using Vec = typename std::conditional<kVec == 4, uint4, uint2>::type;
    Vec* mine = reinterpret_cast<Vec*>(group) + threadIdx.x * (kWords / kVec);
    uint32_t q[kWords], total = 0;
#pragma unroll
    for (int i = 0; i < kWords / kVec; ++i) {
      const Vec v = mine[i];
      memcpy(q + kVec * i, &v, sizeof(v));
    }
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
      const uint32_t a = q[i] & 0xFFFFu, b = q[i] >> 16;
      squares += min(a, kPlaceMaxGroup) * min(a, kPlaceMaxGroup) + min(b, kPlaceMaxGroup) * min(b, kPlaceMaxGroup);
      large |= a > kPlaceMaxGroup || b > kPlaceMaxGroup;
      q[i] = total | (total + a) << 16;
      total += a + b;
    }
    uint32_t incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += up;
    }
    squares = __reduce_add_sync(0xFFFFFFFFu, squares);
    large = __any_sync(0xFFFFFFFFu, large);
    if (lane == 31) s.red[0][w] = incl;
    if (lane == 0) { s.red[1][w] = squares; s.red[2][w] = large; }
    __syncthreads();
    uint32_t base = incl - total + __reduce_add_sync(0xFFFFFFFFu, lane < w ? s.red[0][lane] : 0u);
    squares = __reduce_add_sync(0xFFFFFFFFu, lane < nw ? s.red[1][lane] : 0u);
    large = __any_sync(0xFFFFFFFFu, lane < nw && s.red[2][lane]);
    base |= base << 16;
#pragma unroll
    for (int i = 0; i < kWords; ++i) q[i] += base;
#pragma unroll
    for (int i = 0; i < kWords / kVec; ++i) {
      Vec v;
      memcpy(&v, q + kVec * i, sizeof(v));
      mine[i] = v;
    }
  }
  __syncthreads();

  if (large || squares > kPlaceMaxMean * (uint32_t)m) {
    // the CTA's own elements by digits
#pragma unroll
    for (int j = 0; j < kRoom; ++j) {
      p[j] &= kPlacePosMask;
      if (r0 + 32 * j >= m) k[j] = 0xFFFFFFFFu;
    }
    uint32_t* sk = reinterpret_cast<uint32_t*>(pair);
    const bool scattered = radix_by_digits<kRoom, false, false>(k, p, diff, m, 0, 1, s.radix, group_half, sk, sk + nt * kRoom);
#pragma unroll
    for (int j = 0; j < kRoom; ++j) {
      const int i = scattered ? (int)threadIdx.x + j * nt : r0 + 32 * j;
      if (i < m) emit(out0 + i, k[j], p[j]);
    }
    return;
  }
  // to the groups: a counter ends where the next group begins
#pragma unroll
  for (int j = 0; j < kRoom; ++j) {
    const uint32_t b = p[j] >> kPlacePosBits;
    if (r0 + 32 * j < m && TLX_IN_BOUNDS(b, cap, 32)) {
      const uint32_t old = atomicAdd(&group[b >> 1], (b & 1) ? 0x10000u : 1u), at = (b & 1) ? old >> 16 : old & 0xFFFFu;
      if (TLX_IN_BOUNDS(at, nt * kRoom, 33)) pair[at] = make_uint2(k[j], p[j]);
    }
  }
  if (threadIdx.x < kPlaceWindow) pair[m + threadIdx.x] = make_uint2(0xFFFFFFFFu, 0xFFFFFFFFu);
  __syncthreads();
  // ranks in the groups.  What follows a group is greater than anything in it, so a window may reach past its end.
  // (Eight elements a turn, with the reads of what is carried in flight together: f32 [128, 65536] with a payload 190 us against
  // 173.  The lines of more reads in flight than two a thread don't fit the L1 that the shared memory leaves.)
#pragma unroll 2
  for (int i = threadIdx.x; i < m; i += nt) {
    const uint2 q = pair[i];
    const uint32_t b = q.y >> kPlacePosBits;
    const int from = b ? group_half[b - 1] : 0, end = group_half[b];
    const uint64_t mine = (uint64_t)q.x << 32 | q.y;
    int at = from;
#pragma unroll
    for (int t = 0; t < kPlaceWindow; ++t) {
      const uint2 o = pair[from + t];
      at += ((uint64_t)o.x << 32 | o.y) < mine;
    }
    for (int t = from + kPlaceWindow; t < end; ++t) {
      const uint2 o = pair[t];
      at += ((uint64_t)o.x << 32 | o.y) < mine;
    }
    emit(out0 + at, q.x, q.y & kPlacePosMask);
  }
}

}  // namespace tlx
