// Row-wise exact / single-pass top-k and the per-shard candidate stage of the
// vocab-sharded sampler.  One CTA per row: the streaming collector leaves a superset of
// the top-k in shared memory, a bitonic network orders it by (value desc, index asc).
#include "row_cluster.cuh"
#include "exchange.cuh"

#include <cstdlib>
#include <cstring>
#include <mutex>

namespace tlx {

constexpr int kTopkThreads = 512;

struct TopkParams {
  const void* x;
  int64_t rows, n, row_stride;
  int k_max;
  const int32_t* k_per_row;
  int use_replace;
  double replace_val;
  int mode;
  void* out_vals;
  int32_t* out_idx;
  int32_t* out_valid;
  int32_t* out_depths;
  void* out_cutoff;
  // candidate stage of the vocab-sharded sampler (all null / zero for plain top-k)
  float* cand_vals;
  int32_t* cand_idx;
  float* cand_noise;
  int64_t col_offset;
  int64_t dim0_offset;
  NoiseSrc noise;
  ExchangeTargets ex;   // ex.world > 0: the candidates go to every rank's exchange buffer instead
};

template <int DT>
__device__ __forceinline__ typename Elem<DT>::type cast_replace(double v) {
  if constexpr (DT == TLX_F32) return (float)v;
  else if constexpr (DT == TLX_BF16) return __float2bfloat16_rn((float)v);
  else if constexpr (DT == TLX_F16) return __float2half_rn((float)v);
  else if constexpr (DT == TLX_I32) return (int32_t)v;
  else return (uint32_t)v;
}

// What the exchange buffer's header says to a step: bit 0, which of its two sets the step uses; bit 1, whether the call's extents are
// the buffer's.  It changes between steps only, when no candidate kernel runs.
__device__ __forceinline__ uint32_t exchange_state(const TopkParams& p) {
  const volatile ExchangeHeader* h = reinterpret_cast<const volatile ExchangeHeader*>(p.ex.peer[p.ex.rank]);
  const uint32_t step = h->step, rows = h->rows, k = h->k_cand, world = h->world;
  return (step & 1u) | (rows == (uint32_t)p.rows && k == (uint32_t)p.k_max && world == (uint32_t)p.ex.world ? 2u : 0u);
}
// Candidate stage: the noise of the row's element `col`.
__device__ __forceinline__ float candidate_noise(const TopkParams& p, int64_t r, int32_t col) {
  return p.noise.dense ? __ldg(p.noise.dense + r * p.noise.stride + col) : p.noise.at(r + p.dim0_offset, (int64_t)col + p.col_offset);
}
struct PlacedRow {         // a short list in order; candidate stage: with what was read while it was put in order
  uint64_t cand[96];
  float value[96], noise[96];
  uint32_t state;          // exchange_state
};

// Writes a row's results from its sorted candidate list (m valid entries, the first K are the answer).
// kStage: as the candidate stage (-1: as the call says).  kPlaced: `cand` is a PlacedRow's.
template <int DT, int kStage = -1, bool kPlaced = false>
__device__ __forceinline__ void emit_row(const TopkParams& p, int64_t r, const typename Elem<DT>::type* __restrict__ row,
                                         const uint64_t* cand, int m, int refinements = 0, int bin = 0) {
  const PlacedRow* known = kPlaced ? reinterpret_cast<const PlacedRow*>(cand) : nullptr;
  using T = typename Elem<DT>::type;
  const int K = p.k_max;
  const int k_row = p.k_per_row ? p.k_per_row[r] : K;
  uint32_t par = 0;   // which of the exchange buffer's two sets this step uses
  const bool exchange = kStage != 0 && p.ex.world > 0;
  bool deliver = exchange;
  if (exchange) {
    // a call whose extents are not the buffer's stores nothing anywhere and leaves a mark
    const uint32_t state = kPlaced ? known->state : exchange_state(p);
    par = state & 1u;
    deliver = (state & 2u) != 0;
    if (!deliver && threadIdx.x == 0) reinterpret_cast<volatile ExchangeHeader*>(p.ex.peer[p.ex.rank])->error = 2u;
  }
  for (int j = threadIdx.x; j < K; j += blockDim.x) {
    const uint64_t c = cand[j];
    const int32_t col = (int32_t)cand_low(c);
    const bool have = j < m;
    if (kStage < 0 ? p.cand_vals || exchange : kStage == 1) {
      // candidate stage: f32 value, global token id, noise at that token
      const float v = !have ? -INFINITY : kPlaced ? known->value[j] : elem_as_float<DT>(row[col]);
      const int64_t tok = (int64_t)col + p.col_offset;
      const float u = !have ? 0.5f : kPlaced ? known->noise[j] : candidate_noise(p, r, col);
      if (exchange) {
        if (!deliver) continue;
        // slot `rank` of every rank's buffer, this rank's own included, starting with the next rank
        const size_t plane = (size_t)p.rows * K;
        for (int i = 0; i < p.ex.world; ++i) {
          int peer = p.ex.rank + 1 + i;
          if (peer >= p.ex.world) peer -= p.ex.world;
          float* blk = reinterpret_cast<float*>(p.ex.peer[peer] + p.ex.off_cand[par]) + (size_t)p.ex.rank * 3 * plane;
          blk[r * K + j] = v;
          reinterpret_cast<int32_t*>(blk)[plane + r * K + j] = have ? (int32_t)tok : -1;
          blk[2 * plane + r * K + j] = u;
        }
      } else {
        p.cand_vals[r * K + j] = v;
        p.cand_idx[r * K + j] = have ? (int32_t)tok : -1;
        p.cand_noise[r * K + j] = u;
      }
    } else {
      T v = have ? row[col] : cast_replace<DT>(0.0);
      if (p.use_replace && j >= k_row) v = cast_replace<DT>(p.replace_val);
      reinterpret_cast<T*>(p.out_vals)[r * K + j] = v;
      p.out_idx[r * K + j] = have ? col : 0;
    }
  }
  if (exchange) {
    // the row's block is on its way to every rank: one arrival count each, released after the stores
    __syncthreads();
    if (deliver && (int)threadIdx.x < p.ex.world) {
      __threadfence_system();
      atomicAdd_system(reinterpret_cast<uint32_t*>(p.ex.peer[threadIdx.x] + p.ex.off_flags[par]) + r, 1u);
    }
  }
  if (threadIdx.x == 0) {
    if (p.out_depths) p.out_depths[r] = refinements;
    if (p.out_cutoff) {
      if constexpr (DT == TLX_I32 || DT == TLX_U32)
        reinterpret_cast<int32_t*>(p.out_cutoff)[r] = (int32_t)Elem<TLX_I32>::from_key((uint32_t)bin << kHistShift);
      else
        reinterpret_cast<float*>(p.out_cutoff)[r] = bin_lower_value(bin);
    }
  }
}

// What every kernel here begins with.  Exchange mode (in which they are launched in plain order: 1024 rows of 18992, k = 50, with the
// merge kernel 36.7 us, as dependents of the merge kernel before them 37.4): the merge kernel that follows waits for the rows' arrival counts, not for
// this kernel, and may be scheduled now.
__device__ __forceinline__ void topk_start(const TopkParams& p) {
  grid_wait();
  if (p.ex.world > 0) grid_release();
}

template <int DT, int CAP>
__global__ void __launch_bounds__(kTopkThreads) topk_kernel(TopkParams p) {
  using T = typename Elem<DT>::type;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SelectShared& s = *reinterpret_cast<SelectShared*>(smem_raw);
  uint64_t* cand = reinterpret_cast<uint64_t*>(smem_raw + ((sizeof(SelectShared) + 15) & ~size_t(15)));
  const int64_t r = blockIdx.x;
  const T* row = reinterpret_cast<const T*>(p.x) + r * p.row_stride;
  const int K = p.k_max;
  topk_start(p);

  bool ok = collect_row<DT, CAP>(row, p.n, K, s, cand);
  if (!ok) {
    if (p.mode == 0) {
      exact_select_row<DT>(row, p.n, K, s, cand);
    } else {
      if (threadIdx.x == 0) { if (p.out_valid) atomicExch(p.out_valid, 0); s.fill = CAP; }
      __syncthreads();
    }
  }
  const int m = min(s.fill, CAP);
  sort_candidates(cand, m);

  emit_row<DT>(p, r, row, cand, m, s.refinements, s.bin);
}

// ---- many short rows ---------------------------------------------------------------------------------
// A CTA of 128 threads per row, eight of them per SM, two passes over the row (the second one finds the
// row in L2).  Pass 1 keeps, per thread, the running maximum of every slot of its 16-byte vectors: 128 x
// kSlots group maxima, each an element of the row.  The K-th largest of them (K <= number of groups) is
// a lower bound of the row's K-th largest element, and with groups of a few dozen elements it is a tight
// one: for K = 50 of 19 000 elements about K + 1 elements lie at or above it.  Pass 2 collects those, a
// bitonic network orders them.  The bound is taken on the top 16 key bits.  NaNs have the greatest key:
// the maxima skip them (so they stay elements of the row), pass 2 admits them by its negated compare.
constexpr int kShortThreads = 128;
constexpr int kShortCap = 1024;
constexpr int kShortMaxK = 128;

// Row traversal by 16-byte vectors: fv(vector, first column) in the aligned body, of which one piece of a vector per thread
// in `sub` is read, kU loads in flight per thread; fs(element, column) for the unaligned head and tail.
template <int DT, int kU, typename FV, typename FS>
__device__ __forceinline__ void for_each_vec(const typename Elem<DT>::type* __restrict__ row, int64_t n, int sub, FV&& fv,
                                             FS&& fs) {
  using T = typename Elem<DT>::type;
  constexpr int VEC = 16 / (int)sizeof(T);
  const uintptr_t addr = reinterpret_cast<uintptr_t>(row);
  int64_t head = (int64_t)(((16 - (addr & 15)) & 15) / sizeof(T));
  if (head > n) head = n;
  for (int64_t c = threadIdx.x; c < head; c += blockDim.x) fs(row[c], c);
  const int64_t nvec = (n - head) / VEC;
  const uint4* vp = reinterpret_cast<const uint4*>(row + head);
  const int64_t step = (int64_t)blockDim.x * sub;
  int64_t i = threadIdx.x;
  for (; i + (int64_t)(kU - 1) * step < nvec; i += (int64_t)kU * step) {
    uint4 v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) v[u] = __ldg(vp + i + (int64_t)u * step);
#pragma unroll
    for (int u = 0; u < kU; ++u) fv(v[u], head + (i + (int64_t)u * step) * VEC);
  }
#pragma unroll 1
  for (; i < nvec; i += step) fv(__ldg(vp + i), head + i * VEC);
#pragma unroll 1
  for (int64_t c = head + nvec * VEC + threadIdx.x; c < n; c += blockDim.x) fs(row[c], c);
}

// The elements of one vector that lie at or above the bound join the candidate list.
template <int DT>
static __device__ __noinline__ void push_vector(uint4 v, int64_t cb, uint32_t t16, float thr, int* fill, uint64_t* cand,
                                            int cap) {
  using T = typename Elem<DT>::type;
  const T* x = reinterpret_cast<const T*>(&v);
#pragma unroll
  for (int j = 0; j < 16 / (int)sizeof(T); ++j) {
    if (!(elem_as_float<DT>(x[j]) < thr)) {
      const uint32_t key = Elem<DT>::key(x[j]);
      if ((key >> 16) >= t16) {
        const int slot = atomicAdd(fill, 1);
        if (slot < cap) cand[slot] = cand_make(key, (uint32_t)(cb + j));
      }
    }
  }
}

// The K-th largest of the G 16-bit keys in shared memory (1 <= K <= G): two counting passes of 8 bits.
// hist: 512 words (one histogram per pass), pick: 4 words, both in shared memory.  All threads call.  The
// bin that holds the `need`-th largest is found by warp 0 alone (eight bins per lane, one shuffle scan):
// five CTA barriers in all.
__device__ __forceinline__ void warp_pick_bin(const uint32_t* h, int need, int* out) {
  const int lane = lane_id();
  const int hi = 255 - 8 * lane;   // lane l owns bins hi, hi-1, ..., hi-7 (descending)
  uint32_t local = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) local += h[hi - j];
  uint32_t incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += up;
  }
  const uint32_t excl = incl - local;
  if (excl < (uint32_t)need && incl >= (uint32_t)need) {
    uint32_t run = excl;
    for (int j = 0; j < 8; ++j) {
      const uint32_t c = h[hi - j];
      if (run + c >= (uint32_t)need) { out[0] = hi - j; out[1] = (int)run; break; }
      run += c;
    }
  }
}

static __device__ __noinline__ uint32_t kth_largest_u16(const uint16_t* keys, int G, int K, uint32_t* hist, int* pick) {
  for (int i = threadIdx.x; i < 512; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < G; i += blockDim.x) atomicAdd(&hist[keys[i] >> 8], 1u);
  __syncthreads();
  if (warp_id() == 0) warp_pick_bin(hist, K, pick);
  __syncthreads();
  const uint32_t top = (uint32_t)pick[0];
  const int need = K - pick[1];
  for (int i = threadIdx.x; i < G; i += blockDim.x) {
    const uint32_t k = keys[i];
    if ((k >> 8) == top) atomicAdd(&hist[256 + (k & 255u)], 1u);
  }
  __syncthreads();
  if (warp_id() == 0) warp_pick_bin(hist + 256, need, pick + 2);
  __syncthreads();
  return (top << 8) | (uint32_t)pick[2];
}

// 16-bit key of the greatest element of a vector (a NaN has the greatest key).
template <int DT>
__device__ __forceinline__ uint32_t vector_key16(const uint4& v) {
  if constexpr (DT == TLX_BF16) {
    const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&v);
    const __nv_bfloat162 a = __hmax2_nan(__hmax2_nan(e[0], e[1]), __hmax2_nan(e[2], e[3]));
    return f32_key(__bfloat162float(__hmax_nan(__low2bfloat16(a), __high2bfloat16(a)))) >> 16;
  } else {
    using T = typename Elem<DT>::type;
    const T* e = reinterpret_cast<const T*>(&v);
    uint32_t k = 0;
#pragma unroll
    for (int j = 0; j < 16 / (int)sizeof(T); ++j) k = max(k, Elem<DT>::key(e[j]));
    return k >> 16;
  }
}

// Orders m distinct composites: four lanes count the ones below a composite, which is its place.
__device__ __forceinline__ void order_by_count(const uint64_t* cand, int m, uint64_t* placed) {
  const int part = threadIdx.x & 3;
  for (int i0 = 0; i0 < m; i0 += blockDim.x / 4) {
    const int i = i0 + threadIdx.x / 4;
    const uint64_t c = cand[min(i, m - 1)];
    int below = 0;
#pragma unroll 4
    for (int j = part; j < m; j += 4) below += cand[j] < c ? 1 : 0;
    below += __shfl_xor_sync(0xFFFFFFFFu, below, 1);
    below += __shfl_xor_sync(0xFFFFFFFFu, below, 2);
    if (part == 0 && i < m) placed[below] = c;
  }
}

// ---- long rows -----------------------------------------------------------------------------------------------------------
// A CTA per row, for rows that L2 would not keep between two passes: the bound comes from every eighth of the row's pieces
// of a vector per thread, whose vectors leave the 16-bit keys of their greatest elements in shared memory, so that every byte of the
// row is read once.  An eighth of the row bounds loosely (about 1200 vectors hold an element at or above the bound for
// K = 128): the vectors are noted with their keys, a list per warp, the K-th greatest of these keys is a second, tight
// bound (K vectors hold an element at or above it), and only the vectors that reach it are looked into.
// HBM-bound; f32 [1024, 262144], k = 128: 285 us with the bound from a quarter of the row and the whole row read again,
// 234 us with one list of noted vectors per CTA of 128 threads, 205 us with a list per warp of a CTA of 256 threads, 171 us
// with no more shared memory taken from L1 than it needs (the bytes alone: 164 us).
constexpr int kSampledSub = 8;
constexpr int kSampledNotes = 256;   // noted vectors of a warp
constexpr int64_t kSampledVecs = 65536;   // vectors of a row at most: their numbers have 16 bits
template <int DT>
__device__ __forceinline__ bool vector_reaches(const uint4& v, float thr) {   // (true also for vectors somewhat below)
  if constexpr (DT == TLX_F16) {
    const __half2 t2 = __half2half2(__float2half_rd(thr));
    const __half2* e = reinterpret_cast<const __half2*>(&v);
    return !(__hblt2(e[0], t2) && __hblt2(e[1], t2) && __hblt2(e[2], t2) && __hblt2(e[3], t2));
  } else {
    return rc_any_at_least<DT>(v, thr);
  }
}
template <int DT, int TH>
__global__ void __launch_bounds__(TH, 1024 / TH) topk_sampled_kernel(TopkParams p) {
  using T = typename Elem<DT>::type;
  constexpr int kSlots = GroupMax<DT>::kSlots, G = TH * kSlots, VEC = 16 / (int)sizeof(T);
  constexpr int kGroup = TH * kSampledSub;   // vectors of eight pieces; the first piece is sampled
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SelectShared& s = *reinterpret_cast<SelectShared*>(smem_raw);
  uint64_t* cand = reinterpret_cast<uint64_t*>(smem_raw + ((sizeof(SelectShared) + 15) & ~size_t(15)));
  uint16_t* vkeys = reinterpret_cast<uint16_t*>(s.hist);            // the sampled vectors' keys; later
  uint64_t* list = reinterpret_cast<uint64_t*>(s.hist);             // the candidates, and behind them
  uint32_t* hist8 = s.hist + kShortCap * 2;                         // the second bound's histogram
  uint16_t* sel = reinterpret_cast<uint16_t*>(hist8 + 256);         // the vectors to look into
  uint16_t* gkeys = reinterpret_cast<uint16_t*>(cand);              // the groups' maxima and a histogram; later the noted vectors, TH * 32 bytes
  static_assert(kSampledVecs / kSampledSub * 2 <= sizeof(s.hist) && kShortCap * 3 + 256 <= kHistBins && G * 2 + 2048 <= TH * 32, "");
  const int64_t r = blockIdx.x;
  const T* row = reinterpret_cast<const T*>(p.x) + r * p.row_stride;
  const int K = p.k_max, n = (int)p.n, tid = threadIdx.x;
  topk_start(p);
  const int head = (int)(((16 - (reinterpret_cast<uintptr_t>(row) & 15)) & 15) / sizeof(T));
  const int nvec = (n - head) / VEC;
  const uint4* vp = reinterpret_cast<const uint4*>(row + head);
  GroupMax<DT> gm;
  gm.init();
#pragma unroll 1
  for (int g0 = 0; g0 * kGroup < nvec; g0 += 8) {
    uint4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if ((g0 + u) * kGroup + tid < nvec) v[u] = __ldcs(vp + (g0 + u) * kGroup + tid);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if ((g0 + u) * kGroup + tid < nvec) {
        gm.add(v[u]);
        vkeys[(g0 + u) * TH + tid] = (uint16_t)vector_key16<DT>(v[u]);
      }
  }
#pragma unroll
  for (int j = 0; j < kSlots; ++j) gkeys[tid * kSlots + j] = (uint16_t)(f32_key(gm.slot(j)) >> 16);
  // while the bound is found, what is streamed next comes into L2
#pragma unroll
  for (int g = 0; g < 2; ++g)
    if (tid < TH - TH / kSampledSub && (g + 1) * kGroup <= nvec)
      asm volatile("prefetch.global.L2 [%0];" :: "l"(vp + g * kGroup + TH + tid * 8));
  if (tid == 0) { s.fill = 0; s.bin = 0; s.above = 0; s.refinements = 0; }
  __syncthreads();
  const uint32_t t16 = kth_largest_u16(gkeys, G, K, reinterpret_cast<uint32_t*>(gkeys + G), s.tmp_i);
  const float thr = key_f32(t16 << 16);   // (a NaN pattern, the bin of -inf, admits everything)

  // (key, number) of the vectors that may hold an element at or above the bound, in the warp's list
  uint32_t* noted = reinterpret_cast<uint32_t*>(cand) + warp_id() * kSampledNotes;
  const unsigned below_me = (1u << lane_id()) - 1;
  int nn = 0;
  auto look = [&](bool reaches, auto key16, int i) {
    const unsigned b = __ballot_sync(0xFFFFFFFFu, reaches);
    if (b) {
      const int slot = nn + __popc(b & below_me);
      if (reaches && slot < kSampledNotes) noted[slot] = (key16() << 16) | (uint32_t)i;
      nn += __popc(b);
    }
  };
#pragma unroll 1
  for (int g = 0; g * kGroup < nvec; ++g) {
    const int i = g * kGroup + tid;
    const uint32_t k = i < nvec ? vkeys[g * TH + tid] : 0u;
    look(i < nvec && k >= t16, [&] { return k; }, i);
  }
#pragma unroll 1
  for (int g = 0; g * kGroup < nvec; ++g) {
    const int i0 = g * kGroup + tid;
    uint4 v[kSampledSub];
    if ((g + 1) * kGroup <= nvec) {
#pragma unroll
      for (int u = 1; u < kSampledSub; ++u) v[u] = __ldcs(vp + i0 + u * TH);
#pragma unroll
      for (int u = 1; u < kSampledSub; ++u)
        look(vector_reaches<DT>(v[u], thr), [&] { return vector_key16<DT>(v[u]); }, i0 + u * TH);
    } else {
#pragma unroll 1
      for (int u = 1; u < kSampledSub; ++u) {
        const int i = i0 + u * TH;
        const uint4 w = i < nvec ? __ldcs(vp + i) : make_uint4(0, 0, 0, 0);
        look(i < nvec && vector_reaches<DT>(w, thr), [&] { return vector_key16<DT>(w); }, i);
      }
    }
  }
  if (lane_id() == 0) s.scan_u32[warp_id()] = (uint32_t)nn;
  __syncthreads();   // the sampled vectors' keys have been used: their space is free
  int most = 0, total = 0;
#pragma unroll
  for (int w = 0; w < TH / 32; ++w) {
    most = max(most, (int)s.scan_u32[w]);
    total += (int)s.scan_u32[w];
  }
  auto push_one = [&](int c) {
    const T x = row[c];
    const uint32_t key = Elem<DT>::key(x);
    if ((key >> 16) >= t16) list[atomicAdd(&s.fill, 1)] = cand_make(key, (uint32_t)c);
  };
  if (tid < head) push_one(tid);
  if (tid >= 32 && head + nvec * VEC + tid - 32 < n) push_one(head + nvec * VEC + tid - 32);
  bool exact = most > kSampledNotes;   // more vectors than a list holds
  if (!exact) {
    uint32_t t2 = t16;
    if (total > K) {
      // the keys lie close above the bound as a rule: one histogram of their distances from it, and only if the K-th
      // greatest key is 255 or more away (two octaves) a second, coarse one of the keys from there on
      for (int shift = 0;; shift = 8) {
        for (int i = tid; i < 256; i += TH) hist8[i] = 0;
        __syncthreads();
        for (int l = lane_id(); l < nn; l += 32) {
          const uint32_t key = max(noted[l] >> 16, t16);
          if (key >= t2) atomicAdd(&hist8[min((key - t2) >> shift, 255u)], 1u);
        }
        __syncthreads();
        if (warp_id() == 0) warp_pick_bin(hist8, K, s.tmp_i);
        __syncthreads();
        t2 += (uint32_t)s.tmp_i[0] << shift;
        if (shift != 0 || s.tmp_i[0] < 255) break;
      }
    }
    for (int l = lane_id(); l < nn; l += 32)
      if ((noted[l] >> 16) >= t2) {
        const int slot = atomicAdd(&s.above, 1);
        if (slot < kShortCap * 2) sel[slot] = (uint16_t)noted[l];
      }
    __syncthreads();
    exact = s.above > kShortCap * 2;
    const float thr2 = key_f32(t2 << 16);
    for (int l = tid; !exact && l < s.above; l += TH) {
      const int i = sel[l];
      push_vector<DT>(__ldg(vp + i), head + (int64_t)i * VEC, t2, thr2, &s.fill, list, kShortCap);
    }
  }
  __syncthreads();
  exact = exact || s.fill > kShortCap;   // huge groups of equal values, or keys far above the bound
  if (exact) {
    __syncthreads();
    exact_select_row<DT>(row, n, K, s, cand);
    const int m = min(s.fill, kShortCap);
    sort_candidates(cand, m);
    emit_row<DT>(p, r, row, cand, m);
  } else if (s.fill <= 256) {
    const int m = s.fill;
    order_by_count(list, m, cand);
    __syncthreads();
    emit_row<DT>(p, r, row, cand, m);
  } else {
    const int m = s.fill;
    sort_candidates(list, m);
    emit_row<DT>(p, r, row, list, m);
  }
}

// SUB: the bound comes from one piece in SUB of the row.  kStage: 1 the candidate stage, whose values, noise and exchange header are
// read while the composites are counted, not one after the other behind it (1024 shard rows of 18 992, k = 50, with the merge: bf16
// 36.1 -> 32.9 us, f16 38.2 -> 35.1, f32 41.5 -> 38.6); 0 not the stage; -1 as the call says.
template <int DT, int SUB, int kStage>
__global__ void __launch_bounds__(kShortThreads, 8) topk_short_kernel(TopkParams p) {
  using T = typename Elem<DT>::type;
  constexpr int kSlots = GroupMax<DT>::kSlots;
  constexpr int G = kShortThreads * kSlots;
  constexpr int kU = DT == TLX_F32 ? 9 : 10;   // loads in flight per thread (of f32 the tenth would spill)
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SelectShared& s = *reinterpret_cast<SelectShared*>(smem_raw);
  // all of it lives in the big histogram's space, which only the fallback uses (its candidates, too, are written when the
  // histogram has been read): 4 KB for the group keys and the small histogram, and later the noted vectors, and later the
  // ordered candidates; 8 KB for the candidates
  uint64_t* cand = reinterpret_cast<uint64_t*>(s.hist + 1024);
  uint16_t* gkeys = reinterpret_cast<uint16_t*>(s.hist);            // G * 2 bytes <= 2 KB
  uint32_t* hist8 = s.hist + 512;                                     // 512 words
  const int64_t r = blockIdx.x;
  const T* row = reinterpret_cast<const T*>(p.x) + r * p.row_stride;
  const int K = p.k_max;
  const int64_t n = p.n;
  topk_start(p);

  // bf16 rows of up to 4096 vectors (64 KB) read in full by pass 1: pass 1 also leaves every vector's greatest
  // element (NaN if it holds one) in shared memory, in the candidate list's space, and pass 2 reads those
  // 2 bytes per vector instead of the row
  constexpr int VEC = 16 / (int)sizeof(T);
  int64_t head = (int64_t)(((16 - (reinterpret_cast<uintptr_t>(row) & 15)) & 15) / sizeof(T));
  if (head > n) head = n;
  const int64_t nvec = (n - head) / VEC;
  bool vec_maxima = false;
  if constexpr (DT == TLX_BF16 && SUB == 1) vec_maxima = nvec <= kShortCap * 4;
  __nv_bfloat16* vmax = reinterpret_cast<__nv_bfloat16*>(cand);
  GroupMax<DT> gm;
  gm.init();
  if constexpr (DT == TLX_BF16 && SUB == 1) {
    if (vec_maxima) {
      const __nv_bfloat16 ninf = __float2bfloat16_rn(-INFINITY);
      for (int64_t i = nvec + threadIdx.x; i < ((nvec + 7) & ~(int64_t)7); i += blockDim.x) vmax[i] = ninf;
      for_each_vec<DT, kU>(row, n, 1,
        [&](const uint4& v, int64_t cb) {
          gm.add(v);
          const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&v);
          const __nv_bfloat162 a = __hmax2_nan(__hmax2_nan(e[0], e[1]), __hmax2_nan(e[2], e[3]));
          vmax[(cb - head) >> 3] = __hmax_nan(__low2bfloat16(a), __high2bfloat16(a));
        },
        [&](T x, int64_t) { gm.add_one(x); });
    }
  }
  if (!vec_maxima)
    for_each_vec<DT, kU>(row, n, SUB, [&](const uint4& v, int64_t) { gm.add(v); }, [&](T x, int64_t) { gm.add_one(x); });
#pragma unroll
  for (int j = 0; j < kSlots; ++j) gkeys[threadIdx.x * kSlots + j] = (uint16_t)(f32_key(gm.slot(j)) >> 16);
  if (threadIdx.x == 0) { s.fill = 0; s.bin = 0; s.above = 0; s.refinements = 0; }
  __syncthreads();
  const uint32_t t16 = kth_largest_u16(gkeys, G, K, hist8, s.tmp_i);
  // lower edge of the bound's 16-bit bin as a value; a NaN pattern (the bin of -inf) admits everything
  const float thr = key_f32(t16 << 16);

  auto push_one = [&](T x, int64_t c) {
    if (!(elem_as_float<DT>(x) < thr)) {
      const uint32_t key = Elem<DT>::key(x);
      if ((key >> 16) >= t16) {
        const int slot = atomicAdd(&s.fill, 1);
        if (slot < kShortCap) cand[slot] = cand_make(key, (uint32_t)c);
      }
    }
  };
  // The streaming loop only notes which vectors hold an element at or above the bound (about one per
  // candidate); the noted vectors are then read again, one per thread, and their elements pushed.
  uint32_t* noted = s.hist;                 // up to kShortCap first columns
  int* nnoted = &s.above;                   // (tmp_i holds the bound's picks, which threads may still be reading)
  if (threadIdx.x == 0) *nnoted = 0;
  __syncthreads();
  auto note = [&](int64_t cb) {
    const int slot = atomicAdd(nnoted, 1);
    if (slot < kShortCap) noted[slot] = (uint32_t)cb;
  };
  if constexpr (DT == TLX_BF16) {
    const __nv_bfloat16 tb = __ushort_as_bfloat16((unsigned short)(__float_as_uint(thr) >> 16));
    const __nv_bfloat162 t2 = __halves2bfloat162(tb, tb);
    if (vec_maxima) {
      // eight vectors' maxima per 16-byte load; the few elements before and after the aligned body are
      // pushed after the barrier below (the candidate list shares its space with the maxima)
      const uint4* vm4 = reinterpret_cast<const uint4*>(vmax);
      const int groups = (int)((nvec + 7) >> 3);
      for (int g = threadIdx.x; g < groups; g += blockDim.x) {
        const uint4 w = vm4[g];
        const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&w);
        if (!(__hblt2(e[0], t2) && __hblt2(e[1], t2) && __hblt2(e[2], t2) && __hblt2(e[3], t2))) {
          const __nv_bfloat16* x = reinterpret_cast<const __nv_bfloat16*>(&w);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (g * 8 + j < nvec && !__hlt(x[j], tb)) note(head + ((int64_t)g * 8 + j) * VEC);   // not the padding
        }
      }
    } else {
      for_each_vec<DT, kU>(row, n, 1,
        [&](const uint4& v, int64_t cb) {
          const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&v);
          // __hblt2: both halves less than the bound (false when either is a NaN)
          if (!(__hblt2(e[0], t2) && __hblt2(e[1], t2) && __hblt2(e[2], t2) && __hblt2(e[3], t2))) note(cb);
        },
        push_one);
    }
  } else if constexpr (DT == TLX_F16) {
    for_each_vec<DT, kU>(row, n, 1,
      [&](const uint4& v, int64_t cb) {
        const __half2* e = reinterpret_cast<const __half2*>(&v);
        bool any = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __half22float2(e[j]);
          any = any || !(f.x < thr) || !(f.y < thr);
        }
        if (any) note(cb);
      },
      push_one);
  } else {
    for_each_vec<DT, kU>(row, n, 1,
      [&](const uint4& v, int64_t cb) {
        const float* e = reinterpret_cast<const float*>(&v);
        if (!(e[0] < thr) || !(e[1] < thr) || !(e[2] < thr) || !(e[3] < thr)) note(cb);
      },
      push_one);
  }
  __syncthreads();
  if (vec_maxima) {
    for (int64_t c = threadIdx.x; c < head; c += blockDim.x) push_one(row[c], c);
    for (int64_t c = head + nvec * VEC + threadIdx.x; c < n; c += blockDim.x) push_one(row[c], c);
  }
  if (*nnoted > kShortCap) {
    if (threadIdx.x == 0) s.fill = kShortCap + 1;   // more vectors than the list holds: the exact fallback
  } else {
    for (int l = threadIdx.x; l < *nnoted; l += blockDim.x) {
      const int64_t cb = noted[l];
      push_vector<DT>(__ldg(reinterpret_cast<const uint4*>(row + cb)), cb, t16, thr, &s.fill, cand, kShortCap);
    }
  }
  __syncthreads();
  if (s.fill > kShortCap) exact_select_row<DT>(row, n, K, s, cand);   // huge groups of equal values
  const int m = min(s.fill, kShortCap);
  if (m <= 96) {
    // a handful of candidates: every thread counts the composites below its own (they are distinct) and
    // puts it at that place; no network, no barriers in between
    static_assert(sizeof(PlacedRow) <= sizeof(s.hist));
    PlacedRow& placed = *reinterpret_cast<PlacedRow*>(s.hist);
    if (kStage == 1 && p.ex.world > 0 && threadIdx.x == blockDim.x - 1) placed.state = exchange_state(p);
    if ((int)threadIdx.x < m) {
      const uint64_t c = cand[threadIdx.x];
      float v = 0.f, u = 0.f;
      if constexpr (kStage == 1) {
        v = elem_as_float<DT>(row[cand_low(c)]);
        u = candidate_noise(p, r, (int32_t)cand_low(c));
      }
      int below = 0;
      for (int i = 0; i < m; ++i) below += cand[i] < c ? 1 : 0;
      placed.cand[below] = c;
      if constexpr (kStage == 1) {
        placed.value[below] = v;
        placed.noise[below] = u;
      }
    }
    __syncthreads();
    emit_row<DT, kStage, kStage == 1>(p, r, row, placed.cand, m);
  } else {
    sort_candidates(cand, m);
    emit_row<DT, kStage>(p, r, row, cand, m);
  }
}

// ---- fewer rows: a row over the CTAs of a cluster -------------------------------------------------------------------------
// (row_cluster.cuh)  The cluster's bound leaves a few more than K candidates, which the leader gathers and orders: up to
// 256 by counting the greater ones of each, more by the bitonic network.  Too many candidates (huge groups of equal
// values) or fewer than K finite elements: the exact radix select.  One CTA per row, or a row cut into "rows" with a
// second call over their results, took three launches and 18 us for f32 [8, 32768], k = 64.
template <int DT>
__global__ void __launch_bounds__(kRcThreads, 4) topk_cluster_kernel(const __grid_constant__ TopkParams p, int cluster, int64_t part_len) {
  using T = typename Elem<DT>::type;
  extern __shared__ __align__(128) unsigned char smem[];
  RcShared& s = *reinterpret_cast<RcShared*>(smem);
  const RcLayout l(cluster, false);
  const uint32_t rank = cl_rank();
  const int64_t r = blockIdx.x / cluster;
  const T* row = reinterpret_cast<const T*>(p.x) + r * p.row_stride;
  const RcPart<DT> part(row, p.n, part_len, rank, smem + l.off_part);
  topk_start(p);
  part.copy_in();
  const int K = p.k_max;
  float* lx = reinterpret_cast<float*>(smem + l.off_x);
  unsigned short* lpos = reinterpret_cast<unsigned short*>(smem + l.off_pos);
  if (threadIdx.x == 0) s.n_list = 0;
  part.copy_wait();
  __syncthreads();
  float thr = -INFINITY;
  if (p.n > kRcListCap) {
    uint32_t* bound = reinterpret_cast<uint32_t*>(smem + l.off_bound);
    GroupMax<DT> gm;
    gm.init();
#pragma unroll 2
    for (int v = threadIdx.x; v < part.nvec; v += kRcThreads) gm.add(part.vec[v]);
    rc_publish_maxima<DT>(gm, l.bound_words, bound);
    cl_sync();
    thr = key_f32(rc_bound_key16(bound, l.bound_words, K, s) << 16);
  } else {
    cl_sync();
  }
  rc_filter<DT>(part, thr, s, lx, lpos);
  cl_sync();
  if (rank != 0) {
    cl_sync();
    return;
  }
  int m = rc_count(s, cluster) ? -1 : rc_collect(s, cluster, lx, nullptr, lpos);
  cl_arrive();   // the other CTAs may leave
  uint64_t* cand = reinterpret_cast<uint64_t*>(smem + l.off_part);   // the part is not needed any more
  if (m < K) {   // (or -1)
    SelectShared& sel = *reinterpret_cast<SelectShared*>(smem + l.off_part + (size_t)kRcListCap * 8);
    exact_select_row<DT>(row, p.n, K, sel, cand);
    m = K;
    sort_candidates(cand, m);
  } else {
#pragma unroll 1
    for (int i = threadIdx.x; i < m; i += kRcThreads) cand[i] = cand_make(f32_key(lx[i]), (uint32_t)rc_column(s, lpos, i, part_len));
    if (m <= kRcThreads) {
      uint64_t* placed = cand + kRcThreads;
      if ((int)threadIdx.x >= m) cand[threadIdx.x] = ~0ull;
      __syncthreads();
      if ((int)threadIdx.x < m) {
        const uint64_t mine = cand[threadIdx.x];
        const ulonglong2* c2 = reinterpret_cast<const ulonglong2*>(cand);
        int below = 0;
#pragma unroll 4
        for (int j = 0; j < (m + 1) / 2; ++j) {
          const ulonglong2 c = c2[j];
          below += (c.x < mine ? 1 : 0) + (c.y < mine ? 1 : 0);
        }
        placed[below] = mine;
      }
      __syncthreads();
      cand = placed;
    } else {
      __syncthreads();
      sort_candidates(cand, m);
    }
  }
  emit_row<DT>(p, r, row, cand, m);
  cl_wait();
}

// Exact mode of floating-point rows without the diagnostics of the one-pass kernel, and not a comparison run of that one.
static bool float_rows(int dtype, const TopkParams& p) {
  return (dtype == TLX_F32 || dtype == TLX_BF16 || dtype == TLX_F16) && p.mode == 0 && !p.out_valid && !p.out_depths && !p.out_cutoff;
}
static const char* forced_path() {   // "short" / "long": comparison runs of the two-pass and of the one-pass kernel
  static const char* force = getenv("TLX_TOPK_PATH");
  return force;
}

// Whether the long-row kernel serves a call: rows whose vectors have 16-bit numbers, and either
// - fewer than 256 rows of more bytes in all than the shared memory of the clusters that run at the same time holds, about
//   14 MB: beyond it the cluster form takes several waves (f32 [148, 33000] 18 us against 12, [100, 131072] 43 against 18,
//   [148, 262144] 57 against 30; below it f32 [100, 33000] 11.4 against 11.5, [20, 131072] 11.8 against 16.6); or
// - rows of more than 80 KB, more than 30 MB in all, whose second reading by the two-pass kernel L2 no longer serves (f32
//   [1024, 24500] 51 us against 40, [450, 24500] 26 against 22, [300, 24500] 16.8 against 18.2; of 64 KB [1024, 16384] 27
//   against 28); 70 MB where 592 CTAs of 256 threads do not run all the rows at once ([600, 24000]
//   25 us both, [600, 30000] 31 against 27).
static bool long_rows_apply(int dtype, const TopkParams& p) {
  const int64_t row = p.n * dtype_bytes(dtype), all = row * p.rows;
  if (!float_rows(dtype, p) || p.k_max > kShortMaxK || row / 16 > kSampledVecs || forced_path()) return false;
  if (p.rows < 256) return all > (14ll << 20);
  return row > (80 << 10) && all > ((p.rows > 4 * 148 ? 70ll : 30ll) << 20);
}

// Whether the cluster form is faster than the one-pass kernel, by the number of candidates that the leader has to order and by how
// many waves of clusters there are.  Few rows leave the one-pass kernel's SMs idle, so their clusters may take several waves (us
// cluster / one-pass, f32, k = 256: [16, 300000] 31/71, [50, 262144] 61/66, [64, 262144] 74/66).
// - k <= 128, or a row of which all elements are counted: not more than 64 MB
// - k <= 200 (up to 256 candidates, ordered by counting): few rows, or not more than 40 MB (k = 200: [255, 32768] 32/35,
//   [255, 65536] 53/47)
// - k <= 440 (512 in the bitonic network): rows of at least 12000 elements, and few, or not more than 16 MB, 40 MB of 16-bit ones
//   (k = 300: [1, 8192] 14.0/12.7, [255, 8192] 22/17, [1, 12000] 14.4/16.8, [255, 16384] 26/27, [148, 32768] 30/29; bf16, k = 256:
//   [255, 65536] 43/47)
// - above: few rows that are long enough for the leader's network not to matter (k = 1024: [1, 16384] 31/30, [1, 32768] 33/38,
//   [32, 32768] 42/39, [32, 65536] 45/52, [64, 65536] 71/53, [50, 131072] 64/70; k = 512: [1, 12000] 20/20, [32, 32768] 24/29, [148, 32768] 39/33)
static bool cluster_order_pays(int64_t rows, int64_t n, int k, int elem_bytes) {
  const int64_t mb = (rows * n * elem_bytes + (1 << 20) - 1) >> 20;
  const bool few = mb <= 64 && (rows <= 50 || (rows <= 64 && mb <= 40) || (rows <= 100 && elem_bytes == 2 && k <= 440));
  if (k <= kShortMaxK || n <= kRcThreads) return mb <= 64;
  if (k <= 200) return few || mb <= 40;
  if (k <= 440) return n >= 12000 && (few || mb <= (elem_bytes == 2 ? 40 : 16));
  return few && n >= (rows <= 8 ? 20ll : rows <= 32 ? 40ll : 120ll) * k;
}
// Whether the cluster form serves a call: fewer rows than the kernels with a CTA per row want, rows that a cluster holds and that
// are longer than a candidate list (all elements of a shorter row are candidates: up to 256 are ordered by counting, f32 [60, 208]
// 5.7 us against 9.0 of the one-pass kernel, but more would be sorted, f16 [95, 1365], k = 4 25 against 7).
static bool cluster_rows_apply(int dtype, const TopkParams& p) {
  if (!float_rows(dtype, p) || p.k_max > kRcMaxK || forced_path() || long_rows_apply(dtype, p)) return false;
  return p.rows < 256 && (p.n <= kRcThreads || p.n > kRcListCap) && p.n <= (int64_t)kRcMaxCluster * kRcMaxPart &&
         cluster_order_pays(p.rows, p.n, p.k_max, dtype_bytes(dtype));
}

template <int DT>
static int launch_topk_cluster(cudaStream_t st, const TopkParams& p) {
  const int es = (int)sizeof(typename Elem<DT>::type);
  const int cluster = rc_cluster_size(p.rows, p.n, es);
  const int64_t part_len = rc_part_len(p.n, cluster, es);
  size_t part_bytes = (size_t)part_len * es + 32;
  const size_t least = (size_t)kRcListCap * 8 + sizeof(SelectShared);   // of the exact select
  if (part_bytes < least) part_bytes = least;
  const size_t smem = RcLayout(cluster, false).off_part + part_bytes;
  {
    static std::mutex mu;
    static size_t raised[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 0 || dev >= 64 || raised[dev] < smem) {
      const void* f = (const void*)topk_cluster_kernel<DT>;
      cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
      if (e != cudaSuccess) return set_error(TLX_ERR_CUDA, "top_k: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      if (dev >= 0 && dev < 64) raised[dev] = smem;
    }
  }
  return launch_dependent(topk_cluster_kernel<DT>, {(unsigned)(p.rows * cluster), kRcThreads, smem, cluster, -1, p.ex.world > 0}, st, "top_k", p, cluster, part_len);
}

// Whether the two-pass kernel serves a call: K <= 128, enough rows to fill the eight CTAs per SM, and
// - rows of up to 128 KB; or
// - 16-bit rows of more vectors than the long-row kernel numbers (1 MB), if they are more than the two per SM that the one-pass
//   kernel reads at once.  us two-pass / one-pass, k = 20: bf16 [300, 524296] 97/160, [1024, 600000] 228/397, [592, 1200000]
//   269/364; f16 [592, 600000] 152/215, [256, 600000] 117/108.  32-bit rows, with half the elements a byte, gain only while they
//   are short and no whole waves (f32 [300, 300000] 94/121, [592, 327680] 160/155, [592, 1000000] 418/371).
static bool short_rows_apply(int dtype, const TopkParams& p) {
  if (!float_rows(dtype, p) || p.k_max > kShortMaxK) return false;
  if (forced_path()) return !strcmp(forced_path(), "short");
  const int64_t row = p.n * dtype_bytes(dtype);
  if (row / 16 > kSampledVecs) return p.rows > 2 * 148 && dtype != TLX_F32;
  return p.rows >= 256 && p.n >= 2048 && row <= (128 << 10);
}

// The shared memory that `ctas` CTAs of an SM need (1 KB each is the system's), asked for once per device, and not more: what
// is left is L1, without which fewer loads are in flight (f32 [1024, 262144], k = 128: 171 us, and 205 us with all
// of it shared memory).
template <typename F>
static cudaError_t ask_shared_memory(std::mutex& mu, bool (&asked)[64], F* kernel, size_t smem, int ctas) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  if (dev >= 0 && dev < 64 && asked[dev]) return cudaSuccess;
  const size_t percent = ((smem + 1024) * ctas * 100 + (228 << 10) - 1) / (228 << 10);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)(percent < 100 ? percent : 100));
  if (e == cudaSuccess && smem > (48 << 10)) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess && dev >= 0 && dev < 64) asked[dev] = true;
  return e;
}

template <int DT, int SUB, int kStage>
static int launch_topk_short_from(cudaStream_t st, const TopkParams& p) {
  const size_t smem = sizeof(SelectShared);
  static std::mutex mu;
  static bool asked[64] = {};
  cudaError_t e = ask_shared_memory(mu, asked, topk_short_kernel<DT, SUB, kStage>, smem, 1024 / kShortThreads);
  if (e != cudaSuccess) return set_error(TLX_ERR_CUDA, "top_k: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  return launch_dependent(topk_short_kernel<DT, SUB, kStage>, {(unsigned)p.rows, kShortThreads, smem, 1, -1, p.ex.world > 0}, st, "top_k (short rows)", p);
}
// 16-bit rows of more than 1 MB, which L2 does not keep between the passes: the bound from a quarter of the row (bf16 [1024, 600000],
// k = 20: 228 us against 355)
// Without the stage's code the compiler fits bf16 rows into the 64 registers without a spill (bf16 [256, 30000], k = 64: 17.1 -> 16.3
// us, [4096, 8192] 47.7 -> 46.7), the other forms only with it (f16 [1024, 18992], k = 50: 20.0 against 20.6, bf16 [592, 600000],
// k = 20: 146 against 156).
template <int DT>
static int launch_topk_short(cudaStream_t st, const TopkParams& p) {
  if constexpr (DT != TLX_F32)
    if (p.n * (int64_t)sizeof(typename Elem<DT>::type) / 16 > kSampledVecs) return launch_topk_short_from<DT, 4, -1>(st, p);
  if (p.cand_vals || p.ex.world > 0) return launch_topk_short_from<DT, 1, 1>(st, p);
  return launch_topk_short_from<DT, 1, DT == TLX_BF16 ? 0 : -1>(st, p);
}

template <int DT, int TH>
static int launch_topk_sampled_threads(cudaStream_t st, const TopkParams& p) {
  const size_t smem = ((sizeof(SelectShared) + 15) & ~size_t(15)) + TH * 32;
  static std::mutex mu;
  static bool asked[64] = {};
  cudaError_t e = ask_shared_memory(mu, asked, topk_sampled_kernel<DT, TH>, smem, 1024 / TH);
  if (e != cudaSuccess) return set_error(TLX_ERR_CUDA, "top_k: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  return launch_dependent(topk_sampled_kernel<DT, TH>, {(unsigned)p.rows, TH, smem, 1, -1, p.ex.world > 0}, st, "top_k (long rows)", p);
}
// 1024 threads per SM in any case: one, two, four or eight rows at a time, by which of them has every row running at once (f32
// [128, 262144]: 27.4 us with CTAs of 1024 threads, 31 of 512, 49 of 256; [200, 100000]: 32, 24, 30; [500, 100000]: 65, 47,
// 42; bf16 [800, 60000]: 34 us of 256, 27.5 us of 128).  CTAs of 128 threads have lists for twice the vectors that reach the
// bound as a rule only up to K = 64.
template <int DT>
static int launch_topk_sampled(cudaStream_t st, const TopkParams& p) {
  constexpr int sms = 148;
  if (p.rows <= sms) return launch_topk_sampled_threads<DT, 1024>(st, p);
  if (p.rows <= 2 * sms) return launch_topk_sampled_threads<DT, 512>(st, p);
  if (p.rows > 4 * sms && p.k_max <= 64) return launch_topk_sampled_threads<DT, 128>(st, p);
  return launch_topk_sampled_threads<DT, 256>(st, p);
}

template <int DT, int CAP>
static int launch_topk_cap(cudaStream_t st, const TopkParams& p) {
  const size_t smem = ((sizeof(SelectShared) + 15) & ~size_t(15)) + (size_t)CAP * 8;
  // the shared-memory limit of this instantiation is raised once per device, not per call
  static std::mutex mu;
  static bool raised[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 0 || dev >= 64 || !raised[dev]) {
      cudaError_t e = cudaFuncSetAttribute(topk_kernel<DT, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return set_error(TLX_ERR_CUDA, "top_k: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      if (dev >= 0 && dev < 64) raised[dev] = true;
    }
  }
  // out_valid starts as 1: a stream-ordered 4-byte copy node instead of a kernel of its own
  if (p.out_valid) {
    static const int32_t one = 1;
    cudaError_t e = cudaMemcpyAsync(p.out_valid, &one, sizeof(one), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return set_error(TLX_ERR_CUDA, "top_k: cudaMemcpyAsync: %s", cudaGetErrorString(e));
  }
  return launch_dependent(topk_kernel<DT, CAP>, {(unsigned)p.rows, kTopkThreads, smem, 1, -1, p.ex.world > 0}, st, "top_k", p);
}

template <int DT>
static int launch_topk(cudaStream_t st, const TopkParams& p) {
  if (p.k_max <= 256) return launch_topk_cap<DT, 1024>(st, p);
  if (p.k_max <= 1024) return launch_topk_cap<DT, 4096>(st, p);
  return launch_topk_cap<DT, 8192>(st, p);
}

static int dispatch_topk(cudaStream_t st, int dtype, const TopkParams& p, const char* what) {
  if (cluster_rows_apply(dtype, p)) {
    switch (dtype) {
      case TLX_F32: return launch_topk_cluster<TLX_F32>(st, p);
      case TLX_BF16: return launch_topk_cluster<TLX_BF16>(st, p);
      default: return launch_topk_cluster<TLX_F16>(st, p);
    }
  }
  if (long_rows_apply(dtype, p)) {
    switch (dtype) {
      case TLX_F32: return launch_topk_sampled<TLX_F32>(st, p);
      case TLX_BF16: return launch_topk_sampled<TLX_BF16>(st, p);
      default: return launch_topk_sampled<TLX_F16>(st, p);
    }
  }
  if (short_rows_apply(dtype, p)) {
    switch (dtype) {
      case TLX_F32: return launch_topk_short<TLX_F32>(st, p);
      case TLX_BF16: return launch_topk_short<TLX_BF16>(st, p);
      default: return launch_topk_short<TLX_F16>(st, p);
    }
  }
  switch (dtype) {
    case TLX_F32: return launch_topk<TLX_F32>(st, p);
    case TLX_BF16: return launch_topk<TLX_BF16>(st, p);
    case TLX_F16: return launch_topk<TLX_F16>(st, p);
    case TLX_I32: return launch_topk<TLX_I32>(st, p);
    case TLX_U32: return launch_topk<TLX_U32>(st, p);
    default: return set_error(TLX_ERR_UNSUPPORTED, "%s: dtype %d not supported", what, dtype);
  }
}

// ---- a handful of long rows: every row is cut into parts, each part's top-k is found by a CTA of its own
// (the same kernel on rows * parts "rows"), and a second pass takes the top-k of the parts' candidates.
// Among equal values the parts' order and, inside a part, the ascending index order of its candidates keep
// the lower original index first, as the one-pass kernel does.
struct SplitPlan {
  int parts = 0;          // 0: no split
  int64_t part_len = 0;
  size_t off_idx_a = 0, off_idx_b = 0, bytes = 0;
};

static SplitPlan split_plan(int64_t rows, int64_t n, int k_max, int elem_bytes) {
  SplitPlan sp;
  if (rows <= 0 || rows > 16 || n < 16384 || k_max > 256) return sp;   // more rows fill the GPU by themselves
  for (int parts = 16; parts >= 4; parts >>= 1) {
    if (n % parts) continue;
    const int64_t len = n / parts;
    if (len < 2048 || len < 4 * (int64_t)k_max || (len * elem_bytes) % 16) continue;
    sp.parts = parts;
    sp.part_len = len;
    break;
  }
  if (!sp.parts) return sp;
  auto align = [](size_t v) { return (v + 255) & ~size_t(255); };
  const size_t cand = (size_t)rows * sp.parts * k_max;
  sp.off_idx_a = align(cand * elem_bytes);
  sp.off_idx_b = sp.off_idx_a + align(cand * 4);
  sp.bytes = sp.off_idx_b + align((size_t)rows * k_max * 4);
  return sp;
}

// out_idx[r, j] = original column of the candidate that the second pass picked at position pos_b[r, j]
__global__ void topk_map_index_kernel(const int32_t* __restrict__ idx_a, const int32_t* __restrict__ pos_b,
                                      int32_t* __restrict__ out_idx, int64_t rows, int k, int parts, int64_t part_len) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= rows * k) return;
  const int64_t r = e / k;
  const int pos = pos_b[e];
  out_idx[e] = idx_a[r * (int64_t)parts * k + pos] + (int32_t)((pos / k) * part_len);
}

}  // namespace tlx

using namespace tlx;

extern "C" {

size_t tlx_top_k_workspace_bytes(int64_t rows, int64_t n, int k_max) { return split_plan(rows, n, k_max, 4).bytes; }

int tlx_top_k(void* stream, const void* x, int dtype, int64_t rows, int64_t n, int64_t row_stride, int k_max,
              const int32_t* k_per_row, int use_replace, double replace_val, int mode, void* out_vals,
              int32_t* out_idx, int32_t* out_valid, int32_t* out_depths, void* out_cutoff, void* workspace,
              size_t workspace_bytes) {
  cudaStream_t st = (cudaStream_t)stream;
  TLX_CHECK_ARG(rows >= 0 && n >= 0, "top_k: negative extent");
  TLX_CHECK_ARG(k_max >= 1, "top_k: k must be >= 1, got %d", k_max);
  if (k_max > TLX_TOPK_MAX_K)
    return set_error(TLX_ERR_UNSUPPORTED, "top_k: k=%d exceeds the supported maximum %d", k_max, TLX_TOPK_MAX_K);
  TLX_CHECK_ARG((int64_t)k_max <= n, "top_k: k=%d exceeds the row length %lld", k_max, (long long)n);
  TLX_CHECK_ARG(mode == 0 || mode == 1, "top_k: mode must be 0 or 1");
  TLX_CHECK_ARG(n < (1ll << 31) && rows < (1ll << 31), "top_k: extent too large");
  TLX_CHECK_ARG(row_stride >= n, "top_k: row stride smaller than the row");
  if (rows == 0) return TLX_OK;
  TLX_CHECK_ARG(x && out_vals && out_idx, "top_k: null pointer");
  // few long rows, exact mode, no diagnostics asked for, and scratch given: split the rows over CTAs
  const int es = dtype == TLX_BF16 || dtype == TLX_F16 ? 2 : 4;
  const SplitPlan sp = split_plan(rows, n, k_max, es);
  TopkParams p{};
  p.x = x; p.rows = rows; p.n = n; p.row_stride = row_stride; p.k_max = k_max; p.k_per_row = k_per_row;
  p.use_replace = use_replace; p.replace_val = replace_val; p.mode = mode; p.out_vals = out_vals;
  p.out_idx = out_idx; p.out_valid = out_valid; p.out_depths = out_depths; p.out_cutoff = out_cutoff;
  if (sp.parts && !cluster_rows_apply(dtype, p) && !long_rows_apply(dtype, p) && mode == 0 && !out_valid && !out_depths && !out_cutoff && row_stride == n && workspace &&
      workspace_bytes >= sp.bytes && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0 &&
      (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
    unsigned char* ws = (unsigned char*)workspace;
    TopkParams a{};
    a.x = x; a.rows = rows * sp.parts; a.n = sp.part_len; a.row_stride = sp.part_len; a.k_max = k_max;
    a.out_vals = ws; a.out_idx = (int32_t*)(ws + sp.off_idx_a);
    int rc = dispatch_topk(st, dtype, a, "top_k");
    if (rc != TLX_OK) return rc;
    TopkParams b{};
    b.x = ws; b.rows = rows; b.n = (int64_t)sp.parts * k_max; b.row_stride = b.n; b.k_max = k_max;
    b.k_per_row = k_per_row; b.use_replace = use_replace; b.replace_val = replace_val;
    b.out_vals = out_vals; b.out_idx = (int32_t*)(ws + sp.off_idx_b);
    if ((rc = dispatch_topk(st, dtype, b, "top_k")) != TLX_OK) return rc;
    const int64_t total = rows * k_max;
    topk_map_index_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>((const int32_t*)(ws + sp.off_idx_a),
                                                                          (const int32_t*)(ws + sp.off_idx_b), out_idx, rows,
                                                                          k_max, sp.parts, sp.part_len);
    TLX_CHECK_LAUNCH("top_k (index map)");
    return TLX_OK;
  }
  return dispatch_topk(st, dtype, p, "top_k");
}

size_t tlx_shard_candidates_workspace_bytes(int64_t, int64_t, int) { return 0; }

static int shard_candidates_impl(void* stream, const void* logits, int dtype, int64_t rows, int64_t v_local,
                                 int64_t row_stride, int64_t col_offset, int k_cand, const float* noise,
                                 int64_t noise_stride, uint32_t key0, uint32_t key1, const uint32_t* key_dev,
                                 int64_t vocab_total, int64_t dim0_offset, const int32_t* dim0_offset_dev,
                                 float* out_vals, int32_t* out_idx, float* out_noise,
                                 const ExchangeTargets* ex = nullptr) {
  cudaStream_t st = (cudaStream_t)stream;
  TLX_CHECK_ARG(rows >= 0 && v_local > 0, "shard_candidates: bad extent");
  TLX_CHECK_ARG(k_cand >= 1 && k_cand <= 1024, "shard_candidates: k_cand must be in [1, 1024], got %d", k_cand);
  TLX_CHECK_ARG((int64_t)k_cand <= v_local, "shard_candidates: k_cand exceeds the shard width");
  TLX_CHECK_ARG(dtype == TLX_F32 || dtype == TLX_BF16 || dtype == TLX_F16, "shard_candidates: float logits only");
  TLX_CHECK_ARG(row_stride >= v_local, "shard_candidates: row stride smaller than the row");
  TLX_CHECK_ARG(col_offset >= 0 && col_offset + v_local <= (1ll << 31), "shard_candidates: token ids exceed int32");
  if (rows == 0) return TLX_OK;
  TLX_CHECK_ARG(logits && (ex || (out_vals && out_idx && out_noise)), "shard_candidates: null pointer");
  TopkParams p{};
  if (ex) p.ex = *ex;
  p.x = logits; p.rows = rows; p.n = v_local; p.row_stride = row_stride; p.k_max = k_cand;
  p.cand_vals = out_vals; p.cand_idx = out_idx; p.cand_noise = out_noise; p.col_offset = col_offset;
  p.dim0_offset = dim0_offset;
  p.noise.dense = noise; p.noise.stride = noise_stride; p.noise.k0 = key0; p.noise.k1 = key1; p.noise.vocab = vocab_total;
  p.noise.key_dev = key_dev; p.noise.row_offset_dev = dim0_offset_dev;
  return dispatch_topk(st, dtype, p, "shard_candidates");
}

int tlx_shard_candidates(void* stream, const void* logits, int dtype, int64_t rows, int64_t v_local,
                         int64_t row_stride, int64_t col_offset, int k_cand, const float* noise, int64_t noise_stride,
                         uint32_t key0, uint32_t key1, int64_t vocab_total, int64_t dim0_offset, float* out_vals,
                         int32_t* out_idx, float* out_noise, void*, size_t) {
  return shard_candidates_impl(stream, logits, dtype, rows, v_local, row_stride, col_offset, k_cand, noise, noise_stride,
                               key0, key1, nullptr, vocab_total, dim0_offset, nullptr, out_vals, out_idx, out_noise);
}

int tlx_shard_candidates_dev(void* stream, const void* logits, int dtype, int64_t rows, int64_t v_local,
                             int64_t row_stride, int64_t col_offset, int k_cand, const float* noise,
                             int64_t noise_stride, const uint32_t* key_dev, int64_t vocab_total,
                             const int32_t* dim0_offset_dev, float* out_vals, int32_t* out_idx, float* out_noise,
                             void*, size_t) {
  if (!noise && !key_dev) return set_error(TLX_ERR_INVALID, "shard_candidates: neither noise nor a key given");
  return shard_candidates_impl(stream, logits, dtype, rows, v_local, row_stride, col_offset, k_cand, noise, noise_stride,
                               0u, 0u, key_dev, vocab_total, 0, dim0_offset_dev, out_vals, out_idx, out_noise);
}

int tlx_exchange_shard_candidates(void* stream, const void* logits, int dtype, int64_t rows, int64_t v_local,
                                  int64_t row_stride, int64_t col_offset, int k_cand, const float* noise,
                                  int64_t noise_stride, const uint32_t* key_dev, uint32_t key0, uint32_t key1,
                                  int64_t vocab_total, int64_t dim0_offset, const int32_t* dim0_offset_dev, int rank,
                                  int world, void* const* exchange_of_rank) {
  TLX_CHECK_ARG(world >= 1 && world <= kExchangeMaxWorld && rank >= 0 && rank < world,
                "exchange_shard_candidates: rank %d of %d", rank, world);
  TLX_CHECK_ARG(exchange_of_rank && rows >= 1 && k_cand >= 1, "exchange_shard_candidates: bad argument");
  ExchangeTargets ex{};
  ex.world = world;
  ex.rank = rank;
  const ExchangeLayout l = exchange_layout(rows, k_cand, world);
  for (int q = 0; q < 2; ++q) { ex.off_flags[q] = l.off_flags[q]; ex.off_cand[q] = l.off_cand[q]; }
  for (int i = 0; i < world; ++i) {
    TLX_CHECK_ARG(exchange_of_rank[i], "exchange_shard_candidates: buffer of rank %d is null", i);
    ex.peer[i] = (unsigned char*)exchange_of_rank[i];
  }
  return shard_candidates_impl(stream, logits, dtype, rows, v_local, row_stride, col_offset, k_cand, noise, noise_stride,
                               key0, key1, key_dev, vocab_total, dim0_offset, dim0_offset_dev, nullptr, nullptr, nullptr,
                               &ex);
}

}  // extern "C"
