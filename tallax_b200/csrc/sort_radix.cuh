// Radix passes over a row's keys and positions, least significant digit first, eight bits a pass, in the shared memory of one
// CTA or of a cluster of CTAs: what sort_places.cuh falls back to.
//
// What bounds them: barriers and shared-memory latency, then integer instructions that issue at half rate, 128 per 32 elements
// and pass.  Every pass keeps the order of equal digits, so the position need not be compared: it travels beside the key.
//
// A pass.  A warp owns consecutive elements, 32 at a time; lanes with the same digit find each other with one ballot per
// digit bit (__match_any_sync took half as long again), their number goes into the warp's own counter of the digit and
// gives every lane its rank among the warp's equal digits.  The counters of all warps are turned into places (digit
// first, then warp), the elements are scattered to them and read again in order.
//   In a cluster the scatter first goes to the CTA's own shared memory, so that runs of equal digits lie together; then
// the CTAs exchange their digit counts and every run is copied to where it belongs in the row, in whichever CTA that
// is: the copies over distributed shared memory are contiguous.
// Digits in which all keys of the row agree (small integers) are skipped.
#pragma once
#include "row_cluster.cuh"

namespace tlx {

constexpr int kRadixMaxThreads = 1024;
constexpr int kRadixMaxRow = 131072;   // elements per row at most

// Order-preserving key of a type in its own number of bits, and back (-0 comes back as +0, NaN as the one NaN).
template <int DT> struct RadixKey {
  static constexpr int kBits = 32;
  using T = typename Elem<DT>::type;
  static __device__ __forceinline__ uint32_t make(T v) { return Elem<DT>::key(v); }
  static __device__ __forceinline__ T back(uint32_t k) { return Elem<DT>::from_key(k); }
};
__device__ __forceinline__ uint32_t radix_key_half(uint32_t b, uint32_t inf) {
  uint32_t k = (b & 0x8000u) ? (~b & 0xFFFFu) : (b | 0x8000u);
  if (b == 0x8000u) k = 0x8000u;
  return (b & 0x7FFFu) > inf ? 0xFFFFu : k;
}
__device__ __forceinline__ unsigned short radix_half_back(uint32_t k) {
  return (unsigned short)(k == 0xFFFFu ? 0x7FFFu : (k & 0x8000u) ? (k & 0x7FFFu) : (~k & 0xFFFFu));
}
template <> struct RadixKey<TLX_BF16> {
  static constexpr int kBits = 16;
  static __device__ __forceinline__ uint32_t make(__nv_bfloat16 v) { return radix_key_half(__bfloat16_as_ushort(v), 0x7F80u); }
  static __device__ __forceinline__ __nv_bfloat16 back(uint32_t k) { return __ushort_as_bfloat16(radix_half_back(k)); }
};
template <> struct RadixKey<TLX_F16> {
  static constexpr int kBits = 16;
  static __device__ __forceinline__ uint32_t make(__half v) { return radix_key_half(__half_as_ushort(v), 0x7C00u); }
  static __device__ __forceinline__ __half back(uint32_t k) { return __ushort_as_half(radix_half_back(k)); }
};

// What is brought into the keys' order: payloads, and further keys, which leave in canonical form.
struct SortCarry {
  const void* in[TLX_SORT_MAX_CARRIED];
  void* out[TLX_SORT_MAX_CARRIED];
  int bytes[TLX_SORT_MAX_CARRIED];
  int key_dtype[TLX_SORT_MAX_CARRIED];   // -1: not a key
  int count;
};
// Element `from` of the arrays to their element `to`.
__device__ __forceinline__ void carry_one(const SortCarry& c, int64_t from, int64_t to) {
#pragma unroll
  for (int i = 0; i < TLX_SORT_MAX_CARRIED; ++i) {
    if (i >= c.count) break;
    const int key = c.key_dtype[i];
    if (c.bytes[i] == 4) {
      const uint32_t v = __ldg(reinterpret_cast<const uint32_t*>(c.in[i]) + from);
      reinterpret_cast<uint32_t*>(c.out[i])[to] = key == TLX_F32 ? __float_as_uint(key_f32(f32_key(__uint_as_float(v)))) : v;
    } else {
      const uint32_t v = __ldg(reinterpret_cast<const unsigned short*>(c.in[i]) + from), inf = key == TLX_BF16 ? 0x7F80u : 0x7C00u;
      reinterpret_cast<unsigned short*>(c.out[i])[to] = key >= 0 ? radix_half_back(radix_key_half(v, inf)) : (unsigned short)v;
    }
  }
}

struct __align__(16) RadixShared {
  uint32_t total[256];    // elements of every digit in this CTA
  int shift_by[256];      // cluster: place in the row - place in the CTA
  uint32_t warp[32];
};

static_assert(sizeof(RadixShared) % 16 == 0, "the counters behind it are cleared 16 bytes at a time");

// Exclusive sum over the 256 digits of one value each (thread d < 256 holds digit d's), all threads call.
__device__ __forceinline__ uint32_t radix_scan256(uint32_t v, uint32_t* warp_sum) {
  uint32_t incl = v;
  if (threadIdx.x < 256) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane_id() >= o) incl += up;
    }
    if (lane_id() == 31) warp_sum[warp_id()] = incl;
  }
  __syncthreads();
  uint32_t base = 0;
  if (threadIdx.x < 256) {
#pragma unroll
    for (int i = 0; i < 8; ++i) base += i < warp_id() ? warp_sum[i] : 0u;
  }
  return base + incl - v;
}

// By digits.  k, p: element w * 32 * IPT + 32 j + lane of the CTA in k[j], p[j]; diff: the bits in which the row's keys
// differ.  Leaves the CTA's part of the sorted row in k, p: element threadIdx.x + j * blockDim.x of it in k[j], p[j].
//   The places past the row's end hold the greatest key and the last positions, so every pass leaves them where they are.
// PAST: warps that have no other, beyond the row's n elements, are passed over (f32 [1024, 1025] 45 us against 52).  Not
// where every warp has elements: the branch costs 3 %.  A test per group of 32 elements keeps a warp's groups from
// overlapping: f32 [1024, 4096] 105 us against 90.
template <int IPT, bool CL, bool PAST>
__device__ __forceinline__ bool radix_by_digits(uint32_t (&k)[IPT], uint32_t (&p)[IPT], uint32_t diff, int n, int rank, int cluster,
                                                RadixShared& s, unsigned short* count, uint32_t* sk, uint32_t* sp) {
  const int nt = blockDim.x, cap = nt * IPT;
  const int lane = lane_id(), w = warp_id();
  const int nw = PAST ? (n + 32 * IPT - 1) / (32 * IPT) : nt >> 5;   // warps that have elements
  const bool mine_exist = !PAST || w < nw;
  uint2* pair = reinterpret_cast<uint2*>(sk);   // cluster: key and position side by side, one access for both
  auto get = [&](int i, uint32_t& key, uint32_t& pos) {
    if constexpr (CL) {
      const uint2 e = pair[i];
      key = e.x;
      pos = e.y;
    } else {
      key = sk[i];
      pos = sp[i];
    }
  };
  // place / cap without an integer division: (place + 0.5) / cap is at least 0.5 / cap away from a whole number, and a place
  // is below 2^17, far more than the product's rounding error
  const float inv_cap = 1.0f / (float)cap;
  bool scattered = false;
#pragma unroll 1
  for (int sh = 0; sh < 32; sh += 8) {
    if (((diff >> sh) & 255u) == 0) continue;
    if (scattered && mine_exist) {
#pragma unroll
      for (int j = 0; j < IPT; ++j) get(w * 32 * IPT + 32 * j + lane, k[j], p[j]);
    }
    // ranks among the warp's equal digits
    unsigned short* mine = count + w * 256;
    unsigned short at[IPT];
    if (mine_exist) {
      reinterpret_cast<uint4*>(mine)[lane] = make_uint4(0, 0, 0, 0);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < IPT; ++j) {
        const uint32_t d = (k[j] >> sh) & 255u;
        uint32_t peers = 0xFFFFFFFFu;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const bool one = (d >> b) & 1u;
          const uint32_t v = __ballot_sync(0xFFFFFFFFu, one);
          peers &= one ? v : ~v;
        }
        const int before = __popc(peers & ((1u << lane) - 1u));
        const uint32_t old = mine[d];
        __syncwarp();
        if (before == 0) mine[d] = (unsigned short)(old + __popc(peers));
        __syncwarp();
        at[j] = (unsigned short)(old + before);
      }
    }
    __syncthreads();
    // counters -> places: digit first, then warp.  Groups of 256 threads take the warps in equal shares.
    {
      const int groups = nt >> 8, g = threadIdx.x >> 8, d = threadIdx.x & 255;
      const int share = (nw + groups - 1) / groups, w0 = g * share, w1 = min(w0 + share, nw);
      uint32_t sum = 0;
      if (g < groups)
        for (int i = w0; i < w1; ++i) sum += count[i * 256 + d];
      if (groups > 1) {
        // the groups' totals meet in the scatter area, which nobody reads now
        if (g < groups) sk[g * 256 + d] = sum;
        __syncthreads();
      }
      uint32_t total = sum, before = 0;
      if (groups > 1 && g < groups) {
        total = 0;
        for (int i = 0; i < groups; ++i) {
          const uint32_t t = sk[i * 256 + d];
          if (i < g) before += t;
          total += t;
        }
      }
      const uint32_t base = radix_scan256(total, s.warp);
      if (threadIdx.x < 256) { s.total[d] = total; s.shift_by[d] = (int)base; }
      __syncthreads();
      if (g < groups) {
        uint32_t run = (uint32_t)s.shift_by[d] + before;
        for (int i = w0; i < w1; ++i) {
          const uint32_t c = count[i * 256 + d];
          count[i * 256 + d] = (unsigned short)run;
          run += c;
        }
      }
      __syncthreads();
    }
    if (mine_exist) {
#pragma unroll
      for (int j = 0; j < IPT; ++j) {
        const int to = mine[(k[j] >> sh) & 255u] + at[j];
        if constexpr (CL) {
          pair[to] = make_uint2(k[j], p[j]);
        } else {
          sk[to] = k[j];
          sp[to] = p[j];
        }
      }
    }
    __syncthreads();
    if constexpr (CL) {
      // read back in the CTA's order; then (nobody's area is needed any more) every element to its place in the row
#pragma unroll
      for (int j = 0; j < IPT; ++j) {
        get(threadIdx.x + j * nt, k[j], p[j]);
      }
      cl_sync();
      uint32_t all = 0, before = 0;
      if (threadIdx.x < 256) {
#pragma unroll 8
        for (int r = 0; r < cluster; ++r) {
          const uint32_t t = cl_ld_u32(cl_map(&s.total[threadIdx.x], (uint32_t)r));
          if (r < rank) before += t;
          all += t;
        }
      }
      const uint32_t base = radix_scan256(all, s.warp);
      if (threadIdx.x < 256) s.shift_by[threadIdx.x] = (int)(base + before) - s.shift_by[threadIdx.x];
      __syncthreads();
#pragma unroll
      for (int j = 0; j < IPT; ++j) {
        const int to = threadIdx.x + j * nt + s.shift_by[(k[j] >> sh) & 255u];
        const int r = (int)(((float)to + 0.5f) * inv_cap), i = to - r * cap;
        cl_st_u64(cl_map(pair + i, (uint32_t)r), k[j], p[j]);
      }
      cl_sync();
    }
    scattered = true;
  }
  if (scattered) {   // (PAST: what was never scattered to the last places is not written out either)
#pragma unroll
    for (int j = 0; j < IPT; ++j) get(threadIdx.x + j * nt, k[j], p[j]);
  }
  return scattered;
}

}  // namespace tlx
