// A row spread over the CTAs of a thread-block cluster, resident in their shared memory.
//
// Every CTA copies its contiguous part of the row in once (16-byte asynchronous copies; a row may start at any
// element), and whatever is then asked about the row is answered from shared memory, with the cluster's
// hardware barrier and distributed shared memory between the parts: no second pass over HBM, no workspace, no
// kernel boundary between the stages.  A row's latency is one HBM round trip and a few cluster barriers, and it
// hardly depends on the row's length: the cluster grows with the row.
//
// The bound: every thread keeps running maxima of disjoint groups of its elements (packed maxima over the slots
// of its 16-byte vectors), each of them an element of the row.  The K-th largest of the cluster's group maxima
// (about 2048 of them, shared as bf16 rounded towards -inf) is a lower bound of the row's K-th largest element,
// whatever the order of the elements, and a tight one: with G groups about -G ln(1 - K/G) elements lie at or
// above it, 51 for K = 50 and 1420 for K = 1024.
#pragma once
#include "select.cuh"

namespace tlx {

constexpr int kRcThreads = 256;
constexpr int kRcWarps = kRcThreads / 32;
constexpr int kRcListCap = 2048;         // candidates of one CTA, and of the whole row
constexpr int kRcMaxK = 1024;            // largest top-k of the candidate path (1420 +- 40 candidates)
constexpr int kRcBoundWords = 1024;      // packed pairs of group maxima that the bound is taken from
constexpr int kRcMaxCluster = 16;
constexpr int kRcMaxPart = 49152;        // elements of a part (positions are 16 bits; its bytes fit shared memory)

// ---- cluster primitives -----------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cl_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_sync() { cl_arrive(); cl_wait(); }
// address of `p` (a shared variable of this CTA) in the shared memory of CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cl_map(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ uint32_t cl_ld_u32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t cl_ld_u16(uint32_t a) {
  unsigned short v;
  asm volatile("ld.shared::cluster.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void cl_st_u64(uint32_t addr, uint32_t lo, uint32_t hi) {
  asm volatile("st.shared::cluster.v2.u32 [%0], {%1, %2};" :: "r"(addr), "r"(lo), "r"(hi) : "memory");
}
__device__ __forceinline__ void cl_st_u32(uint32_t a, uint32_t v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void cl_st_f32(uint32_t a, float v) { cl_st_u32(a, __float_as_uint(v)); }
__device__ __forceinline__ void cl_st_f64(uint32_t a, double v) { asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }
__device__ __forceinline__ float cl_ld_f32(uint32_t a) { return __uint_as_float(cl_ld_u32(a)); }
__device__ __forceinline__ double cl_ld_f64(uint32_t a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint4 cl_ld_v4(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}

// ---- running maxima of the slots of 16-byte vectors (NaNs are skipped: they stay out of the maxima) ----------
template <int DT> struct GroupMax;
template <> struct GroupMax<TLX_BF16> {
  static constexpr int kSlots = 8;
  __nv_bfloat162 m[4];
  __device__ __forceinline__ void init() {
    const __nv_bfloat16 ninf = __float2bfloat16_rn(-INFINITY);
#pragma unroll
    for (int j = 0; j < 4; ++j) m[j] = __halves2bfloat162(ninf, ninf);
  }
  __device__ __forceinline__ void add(const uint4& v) {
    const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) m[j] = __hmax2(m[j], e[j]);
  }
  __device__ __forceinline__ void add_one(__nv_bfloat16 x) { m[0] = __hmax2(m[0], __halves2bfloat162(x, m[0].y)); }
  __device__ __forceinline__ float slot(int j) const {
    return (j & 1) ? __high2float(m[j >> 1]) : __low2float(m[j >> 1]);
  }
};
template <> struct GroupMax<TLX_F16> {
  static constexpr int kSlots = 8;
  __half2 m[4];
  __device__ __forceinline__ void init() {
    const __half ninf = __float2half_rn(-INFINITY);
#pragma unroll
    for (int j = 0; j < 4; ++j) m[j] = __halves2half2(ninf, ninf);
  }
  __device__ __forceinline__ void add(const uint4& v) {
    const __half2* e = reinterpret_cast<const __half2*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) m[j] = __hmax2(m[j], e[j]);
  }
  __device__ __forceinline__ void add_one(__half x) { m[0] = __hmax2(m[0], __halves2half2(x, __high2half(m[0]))); }
  __device__ __forceinline__ float slot(int j) const {
    return (j & 1) ? __high2float(m[j >> 1]) : __low2float(m[j >> 1]);
  }
};
template <> struct GroupMax<TLX_F32> {
  static constexpr int kSlots = 4;
  float m[4];
  __device__ __forceinline__ void init() {
#pragma unroll
    for (int j = 0; j < 4; ++j) m[j] = -INFINITY;
  }
  __device__ __forceinline__ void add(const uint4& v) {
    const float* e = reinterpret_cast<const float*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) m[j] = fmaxf(m[j], e[j]);
  }
  __device__ __forceinline__ void add_one(float x) { m[0] = fmaxf(m[0], x); }
  __device__ __forceinline__ float slot(int j) const { return m[j]; }
};

// ---- per-CTA state in shared memory -------------------------------------------------------------------------
struct __align__(16) RcShared {
  uint32_t red_u32[4][kRcWarps];        // block reductions alternate between two sets (0, 1; out-of-line routines
  double red_f64[4][2][kRcWarps];       // 2, 3), which makes one barrier each enough
  uint32_t hist[256];
  int pick[4];
  int n_list;                           // candidates of this CTA (may exceed kRcListCap: overflow)
  // rows without top-k
  float dom_x[2 * kRcMaxCluster], dom_s[2 * kRcMaxCluster];   // per CTA: its greatest element and its best-scored one
  float cut_x[14], cut_s[14];           // an element is out if one of these has at least its value and a greater score
  int n_cut;
  float bin_mass[16];                   // softmax mass of this CTA's elements, by their distance from the row's greatest one
  double z_part;                        // ... of all of them; later of those above a value
  float query[4];                       // values whose mass above the leader asks for
  int n_query;
  int query_tok[4];                     // leader: their tokens
  // leader: what the CTAs have sent
  int sent[kRcMaxCluster];
  double z[kRcMaxCluster], msum[kRcMaxCluster][4];
  int first[kRcMaxCluster + 1];         // leader: first candidate of every CTA in the gathered list
  uint32_t key_lo, key_hi;              // range of the candidates' keys (from the bound's search)
  int n_near;
  unsigned long long win;               // winner of a round of the decision
};

// The dynamic shared memory of a CTA: state, the bound's words, the candidate list (position inside the part, value,
// score), the part.  Four CTAs with parts of 32 KB fit an SM.
struct RcLayout {
  int bound_words;
  uint32_t off_bound, off_pos, off_x, off_s, off_part;
  __host__ __device__ __forceinline__ RcLayout(int cluster, bool scores) {
    bound_words = kRcBoundWords / cluster;
    off_bound = (uint32_t)((sizeof(RcShared) + 127) & ~size_t(127));
    off_pos = off_bound + (uint32_t)bound_words * 4;
    off_x = off_pos + kRcListCap * 2;
    off_s = off_x + kRcListCap * 4;
    off_part = off_s + (scores ? kRcListCap * 4 : 0);
  }
};
constexpr int kRcBins = 2048;            // bins of the leader's selection, in the place of its part
constexpr int kRcMinPartBytes = kRcBins * 4;

// ---- block reductions ------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t rc_max_u32(uint32_t v, RcShared& s, int& tog) {
  v = __reduce_max_sync(0xFFFFFFFFu, v);
  if (lane_id() == 0) s.red_u32[tog][warp_id()] = v;
  __syncthreads();
  v = __reduce_max_sync(0xFFFFFFFFu, s.red_u32[tog][lane_id() & (kRcWarps - 1)]);
  tog ^= 1;
  return v;
}
// Two sums at a time, in a fixed order.
__device__ __forceinline__ void rc_sum2_f64(double& a, double& b, RcShared& s, int& tog) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) { a += shfl_xor_f64(a, o); b += shfl_xor_f64(b, o); }
  if (lane_id() == 0) { s.red_f64[tog][0][warp_id()] = a; s.red_f64[tog][1][warp_id()] = b; }
  __syncthreads();
  a = s.red_f64[tog][0][0];
  b = s.red_f64[tog][1][0];
#pragma unroll
  for (int w = 1; w < kRcWarps; ++w) { a += s.red_f64[tog][0][w]; b += s.red_f64[tog][1][w]; }
  tog ^= 1;
}

// ---- a CTA's part of the row -------------------------------------------------------------------------------------
template <int DT>
struct RcPart {
  using T = typename Elem<DT>::type;
  static constexpr int VEC = 16 / (int)sizeof(T);
  const T* g;      // first element of the part in global memory
  int n;           // elements
  int off;         // elements between the 16-byte boundary before it and the first one
  int nvec;        // 16-byte vectors that hold the part
  uint4* vec;      // the vectors in shared memory; what lies outside the part holds -inf
  __device__ __forceinline__ RcPart(const T* row, int64_t row_len, int64_t part_len, uint32_t rank, unsigned char* smem) {
    const int64_t c0 = (int64_t)rank * part_len;
    int64_t m = row_len - c0;
    m = m < 0 ? 0 : (m < part_len ? m : part_len);
    g = row + c0;
    n = (int)m;
    off = (int)((reinterpret_cast<uintptr_t>(g) & 15) / sizeof(T));
    nvec = n > 0 ? (off + n + VEC - 1) / VEC : 0;
    vec = reinterpret_cast<uint4*>(smem);
  }
  __device__ __forceinline__ T elem(int i) const { return reinterpret_cast<const T*>(vec)[off + i]; }
  // Every thread copies the vectors it will look at itself: tid, tid + 256, ...  The first and the last one may
  // reach outside the part; they are copied element by element.
  __device__ __forceinline__ void copy_in() const {
    const unsigned char* base = reinterpret_cast<const unsigned char*>(g - off);
#pragma unroll 4
    for (int v = threadIdx.x; v < nvec; v += kRcThreads) {
      if ((v > 0 || off == 0) && (v + 1) * VEC <= off + n) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(vec + v)),
                     "l"(base + (size_t)v * 16) : "memory");
      } else {
        T* d = reinterpret_cast<T*>(vec + v);
        for (int j = 0; j < VEC; ++j) {
          const int i = v * VEC + j - off;
          T x;
          if constexpr (DT == TLX_F32) x = -INFINITY;
          else if constexpr (DT == TLX_BF16) x = __float2bfloat16_rn(-INFINITY);
          else x = __float2half_rn(-INFINITY);
          if (i >= 0 && i < n) x = g[i];
          d[j] = x;
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  __device__ __forceinline__ void copy_wait() const { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
};

// f32 -> bf16 bits rounded towards -inf (no NaN comes here)
__device__ __forceinline__ uint32_t bf16_floor_bits(float x) {
  const uint32_t b = __float_as_uint(x);
  return (b & 0x80000000u ? b + 0xFFFFu : b) >> 16;
}
__device__ __forceinline__ __nv_bfloat162 rc_bf162(uint32_t w) {
  __nv_bfloat162 r;
  memcpy(&r, &w, 4);
  return r;
}
__device__ __forceinline__ uint32_t rc_bits(__nv_bfloat162 v) {
  uint32_t w;
  memcpy(&w, &v, 4);
  return w;
}

// This CTA's share of the bound's words: the thread's group maxima, folded until the cluster has about
// kRcBoundWords packed pairs in all.
template <int DT>
__device__ __forceinline__ void rc_publish_maxima(const GroupMax<DT>& gm, int words, uint32_t* bound) {
  uint32_t w[4];
  int have;
  if constexpr (DT == TLX_BF16) {
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = rc_bits(gm.m[j]);
    have = 4;
  } else {
    constexpr int kPairs = GroupMax<DT>::kSlots / 2;
    have = kPairs;
#pragma unroll
    for (int j = 0; j < kPairs; ++j) w[j] = bf16_floor_bits(gm.slot(2 * j)) | (bf16_floor_bits(gm.slot(2 * j + 1)) << 16);
#pragma unroll
    for (int j = kPairs; j < 4; ++j) w[j] = 0xFF80FF80u;
  }
  if (words >= 4 * kRcThreads) {          // one CTA: all of them
    reinterpret_cast<uint4*>(bound)[threadIdx.x] = make_uint4(w[0], w[1], w[2], w[3]);
    return;
  }
  if (have == 4) { w[0] = rc_bits(__hmax2(rc_bf162(w[0]), rc_bf162(w[2]))); w[1] = rc_bits(__hmax2(rc_bf162(w[1]), rc_bf162(w[3]))); }
  if (words >= 2 * kRcThreads) {
    reinterpret_cast<uint2*>(bound)[threadIdx.x] = make_uint2(w[0], w[1]);
    return;
  }
  __nv_bfloat162 m = __hmax2(rc_bf162(w[0]), rc_bf162(w[1]));
  int fold = kRcThreads / words;          // 1, 2 or 4 lanes share a word
  for (int o = 1; o < fold; o <<= 1) m = __hmax2(m, rc_bf162(__shfl_xor_sync(0xFFFFFFFFu, rc_bits(m), o)));
  if ((threadIdx.x & (fold - 1)) == 0) bound[threadIdx.x / fold] = rc_bits(m);
}

// The K-th largest of the cluster's group maxima as a 16-bit key (0x80, every finite element, if there are fewer than
// K).  Warp 0 holds all of them, 32 packed words a lane, and searches the key bits in which they differ, one warp
// reduction a bit and no barrier: nine or ten rounds of about 100 cycles.  Spread over the CTA's warps, with a barrier
// a round, the same search took 2.3 us instead of 0.8; a histogram would be serialised by the few bins that the
// maxima share.
__device__ __forceinline__ __nv_bfloat162 rc_key_pair(uint32_t key) {
  const uint32_t b = key & 0x8000u ? key & 0x7FFFu : ~key & 0xFFFFu;
  return rc_bf162(b | (b << 16));
}
__device__ __forceinline__ uint32_t rc_key16(float x) { return f32_key(x) >> 16; }
__device__ __forceinline__ uint32_t rc_bound_key16(const uint32_t* bound, int words, int K, RcShared& s) {
  if (warp_id() == 0) {
    uint32_t w[32];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int at = (lane_id() + 32 * j) * 4;
      const uint4 q = cl_ld_v4(cl_map(bound + at % words, (uint32_t)(at / words)));
      w[4 * j] = q.x; w[4 * j + 1] = q.y; w[4 * j + 2] = q.z; w[4 * j + 3] = q.w;
    }
    __nv_bfloat162 hi = rc_bf162(w[0]), lo = hi;
#pragma unroll
    for (int j = 1; j < 32; ++j) { hi = __hmax2(hi, rc_bf162(w[j])); lo = __hmin2(lo, rc_bf162(w[j])); }
    const uint32_t kmax = __reduce_max_sync(0xFFFFFFFFu, rc_key16(fmaxf(__low2float(hi), __high2float(hi))));
    const uint32_t kmin = __reduce_min_sync(0xFFFFFFFFu, rc_key16(fminf(__low2float(lo), __high2float(lo))));
    // a few of many: fewer and larger groups give as tight a bound (512 groups: 53 elements for K = 50)
    const int n = K <= 64 ? 8 : K <= 256 ? 16 : 32;
    if (n <= 16) {
#pragma unroll
      for (int j = 0; j < 16; ++j) w[j] = rc_bits(__hmax2(rc_bf162(w[j]), rc_bf162(w[j + 16])));
      if (n <= 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = rc_bits(__hmax2(rc_bf162(w[j]), rc_bf162(w[j + 8])));
      }
    }
    uint32_t t = kmin;
    if (kmax > kmin) {
      int bit = 31 - __clz(kmax ^ kmin);
      t = kmax & ~((2u << bit) - 1u);
#pragma unroll 1
      for (; bit >= 0; --bit) {
        const __nv_bfloat162 p = rc_key_pair(t | (1u << bit));
        __nv_bfloat162 c0 = __hge2(rc_bf162(w[0]), p), c1 = __hge2(rc_bf162(w[1]), p);
#pragma unroll
        for (int j = 2; j < 32; j += 2) {
          if ((j == 8 && n == 8) || (j == 16 && n == 16)) break;
          c0 = __hadd2(c0, __hge2(rc_bf162(w[j]), p));
          c1 = __hadd2(c1, __hge2(rc_bf162(w[j + 1]), p));
        }
        c0 = __hadd2(c0, c1);
        const int c = __reduce_add_sync(0xFFFFFFFFu, (int)(__low2float(c0) + __high2float(c0)));
        if (c >= K) t |= 1u << bit;
      }
    }
    if (lane_id() == 0) { s.pick[0] = (int)(t < 0x80u ? 0x80u : t); s.key_lo = (uint32_t)s.pick[0] << 16; s.key_hi = (kmax << 16) | 0xFFFFu; }
  }
  __syncthreads();
  return (uint32_t)s.pick[0];
}

// The part's elements that are not below `thr` (NaNs among them) join the CTA's list.
template <int DT>
__device__ __forceinline__ bool rc_any_at_least(const uint4& v, float thr) {
  if constexpr (DT == TLX_BF16) {
    const __nv_bfloat16 tb = __ushort_as_bfloat16((unsigned short)bf16_floor_bits(thr));
    const __nv_bfloat162 t2 = __halves2bfloat162(tb, tb);
    const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&v);
    return !(__hblt2(e[0], t2) && __hblt2(e[1], t2) && __hblt2(e[2], t2) && __hblt2(e[3], t2));
  } else if constexpr (DT == TLX_F16) {
    const __half2* e = reinterpret_cast<const __half2*>(&v);
    bool any = false;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __half22float2(e[j]);
      any = any || !(f.x < thr) || !(f.y < thr);
    }
    return any;
  } else {
    const float* e = reinterpret_cast<const float*>(&v);
    return !(e[0] < thr) || !(e[1] < thr) || !(e[2] < thr) || !(e[3] < thr);
  }
}

template <int DT>
__device__ __forceinline__ void rc_filter(const RcPart<DT>& part, float thr, RcShared& s, float* lx, unsigned short* lpos) {
  using T = typename Elem<DT>::type;
  constexpr int VEC = RcPart<DT>::VEC;
#pragma unroll 1
  for (int v = threadIdx.x; v < part.nvec; v += kRcThreads) {
    const uint4 w = part.vec[v];
    if (!rc_any_at_least<DT>(w, thr)) continue;
    const T* e = reinterpret_cast<const T*>(&w);
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      const float x = elem_as_float<DT>(e[j]);
      const int i = v * VEC + j - part.off;
      if (!(x < thr) && (unsigned)i < (unsigned)part.n) {
        const int slot = atomicAdd(&s.n_list, 1);
        if (slot < kRcListCap) { lx[slot] = x; lpos[slot] = (unsigned short)i; }
      }
    }
  }
}

// Prefix of the CTAs' counts (s.first); whether a list or the whole overflowed, which every CTA that asks sees alike.
__device__ __forceinline__ bool rc_count(RcShared& s, int cluster) {
  if (threadIdx.x < 32) {
    const int lane = lane_id();
    int c = lane < cluster ? (int)cl_ld_u32(cl_map(&s.n_list, (uint32_t)lane)) : 0;
    const unsigned over = __ballot_sync(0xFFFFFFFFu, c > kRcListCap);
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane < cluster) s.first[lane + 1] = incl;
    if (lane == 0) { s.first[0] = 0; s.pick[0] = over != 0; }
  }
  __syncthreads();
  return s.pick[0] || s.first[cluster] > kRcListCap;
}
// Leader, lists that did not overflow: the other CTAs' candidates behind its own ones in its own list.  Returns their number.
__device__ __forceinline__ int rc_collect(RcShared& s, int cluster, float* lx, float* ls, unsigned short* lpos) {
  const int m = s.first[cluster];
#pragma unroll 1
  for (int i = s.first[1] + threadIdx.x; i < m; i += kRcThreads) {
    int r = 1;
    while (i >= s.first[r + 1]) ++r;
    const int k = i - s.first[r];
    const float x = cl_ld_f32(cl_map(lx + k, (uint32_t)r));
    const uint32_t pos = cl_ld_u16(cl_map(lpos + k, (uint32_t)r));
    if (ls) ls[i] = cl_ld_f32(cl_map(ls + k, (uint32_t)r));
    lx[i] = x;
    lpos[i] = (unsigned short)pos;
  }
  __syncthreads();
  return m;
}
// column of candidate i of the gathered list
__device__ __forceinline__ int64_t rc_column(const RcShared& s, const unsigned short* lpos, int i, int64_t part_len) {
  int r = 0;
  while (i >= s.first[r + 1]) ++r;
  return (int64_t)r * part_len + lpos[i];
}

// CTAs per row: parts of at most 40 KB (three or four CTAs fit an SM), eight CTAs at most: clusters of sixteen find
// their place on the GPU so much later that they are only worth it for a few rows, where the shorter parts count.
// A few rows take more and smaller parts, down to 8 KB, while there is an SM for every two CTAs.
inline int rc_cluster_size(int64_t rows, int64_t n, int elem_bytes) {
  const int64_t row_bytes = n * elem_bytes;
  int c = n > kRcListCap ? 2 : 1;
  while (c < 8 && row_bytes > (int64_t)c * 40960) c *= 2;
  while (c < kRcMaxCluster && rows * c * 2 <= 296 && row_bytes > (int64_t)c * 8192) c *= 2;
  if (c < kRcMaxCluster && n > (int64_t)c * kRcMaxPart) c = kRcMaxCluster;
  return c;
}
// Elements of a part, a multiple of a 16-byte vector.
inline int64_t rc_part_len(int64_t n, int cluster, int elem_bytes) {
  const int vec = 16 / elem_bytes;
  return ((n + cluster - 1) / cluster + vec - 1) / vec * vec;
}

}  // namespace tlx
