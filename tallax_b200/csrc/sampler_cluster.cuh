// Fused sampler, one kernel: a row is spread over a thread-block cluster (row_cluster.cuh), included by sampler.cu.
//
// Rows with 1 <= top_k <= 1024 (greedy rows are top_k = 1): every CTA filters its part against the cluster's bound,
// scores its candidates (x / T + Gumbel of the noise there) and leaves them in its list; the leader gathers the
// lists over distributed shared memory, cuts them to the top-k set (radix descent over the keys) and decides.
//
// Decision.  A token is kept if the softmax mass of the greater values of the set is below top_p, so nothing has to
// be sorted: the best score of the set wins if the mass above its value is below top_p * Z; otherwise no lower
// value is kept either, and the best score among the greater values is tried.  One or two rounds as a rule.
//
// Rows without top-k of which top_p leaves a share: the softmax denominator and the mass at sixteen distances from the
// greatest element come first, and say from which value on elements can be kept; only those are scored (rc_pruned_row).
//   The others, and what that leaves open: every CTA publishes its greatest element and that element's score.  An element can only
// win if no greater (or equal) element has a greater score, because a greater value is kept whenever the smaller one is;
// so what the published pairs dominate is out, and before its noise is even looked at an element is out if its
// value plus the greatest Gumbel term there is would not do.  The survivors (a handful) go to the leader, and the
// mass above its best ones comes from one more pass over the parts, which are still in shared memory.
//
// Rows with 1024 < top_k < vocab, and rows whose lists overflow, are cut to their top-k set in shared memory (rc_cut_parts)
// and then taken as rows without.
//
// Rows without top-k whose survivors the lists cannot hold, greedy rows with huge groups of greatest values, rows without a
// finite maximum, and rows longer than a cluster holds take rc_slow_row: exact, any top-k, by passes over the row in global
// memory.
#pragma once
#include "row_cluster.cuh"

namespace tlx {

struct RcSampleParams {
  SampleParams sp;
  int cluster;
  int64_t part_len;   // elements of a part, a multiple of a 16-byte vector
};

// Warp 0: the bin of a 256-bin histogram that holds the need-th element counted from the top; out[0] = bin,
// out[1] = elements in higher bins, out[2] = elements in the bin.
__device__ __forceinline__ void rc_pick_bin(const uint32_t* h, int need, int* out) {
  const int lane = lane_id();
  const int hi = 255 - 8 * lane;
  uint32_t local = 0;
#pragma unroll 1
  for (int j = 0; j < 8; ++j) local += h[hi - j];
  uint32_t incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += up;
  }
  uint32_t run = incl - local;
  if (run < (uint32_t)need && incl >= (uint32_t)need) {
#pragma unroll 1
    for (int j = 0; j < 8; ++j) {
      const uint32_t c = h[hi - j];
      if (run + c >= (uint32_t)need) { out[0] = hi - j; out[1] = (int)run; out[2] = (int)c; break; }
      run += c;
    }
  }
}

// Key of a score for an unsigned maximum; NaN is below everything.
__device__ __forceinline__ uint32_t rc_score_key(float a) { return a == a ? f32_key(a) : 0u; }
__device__ __forceinline__ unsigned long long rc_win_make(float y, int64_t tok) {
  return ((unsigned long long)rc_score_key(y) << 32) | (uint32_t)(0x7FFFFFFF - (int32_t)tok);
}

// One row by passes over global memory, any top-k, ties or NaNs.  Returns the token.
template <int DT>
static __device__ __noinline__ int rc_slow_row(const typename Elem<DT>::type* __restrict__ row, int64_t n, int64_t K, float p,
                                               float T_, const NoiseSrc& noise, int64_t nrow, RcShared& s) {
  using T = typename Elem<DT>::type;
  int tog = 0;
  auto composite = [](T v, int64_t c) { return ((uint64_t)Elem<DT>::key(v) << 32) | (uint32_t)(0x7FFFFFFF - (int32_t)c); };
  auto block_max = [&](uint64_t v) {
    const uint32_t hi = rc_max_u32((uint32_t)(v >> 32), s, tog);
    const uint32_t lo = rc_max_u32((uint32_t)(v >> 32) == hi ? (uint32_t)v : 0u, s, tog);
    return ((uint64_t)hi << 32) | lo;
  };
  __syncthreads();
  uint64_t best = 0;
  for_each_elem<DT>(row, 0, n, [&](T v, int64_t c) { const uint64_t x = composite(v, c); best = x > best ? x : best; });
  const uint64_t top = block_max(best);
  const int top_col = 0x7FFFFFFF - (int)(uint32_t)top;
  if (T_ < kSamplingEps) return top_col;
  const float xmax = key_f32((uint32_t)(top >> 32));
  uint64_t least = 0;   // least composite of the top-k set
  if (K < n) {
    int need = (int)K;
#pragma unroll 1
    for (int sh = 56; sh >= 0; sh -= 8) {
      s.hist[threadIdx.x] = 0;
      __syncthreads();
      for_each_elem<DT>(row, 0, n, [&](T v, int64_t c) {
        const uint64_t x = composite(v, c);
        if (sh == 56 || ((x ^ least) >> (sh + 8)) == 0) atomicAdd(&s.hist[(x >> sh) & 255], 1u);
      });
      __syncthreads();
      if (warp_id() == 0) rc_pick_bin(s.hist, need, s.pick);
      __syncthreads();
      least |= (uint64_t)(uint32_t)s.pick[0] << sh;
      need -= s.pick[1];
      if (s.pick[2] == need) break;   // the whole bin belongs to the set
    }
  }
  double z = 0.0, unused = 0.0;
  for_each_elem<DT>(row, 0, n, [&](T v, int64_t c) {
    if (composite(v, c) >= least) z += (double)expf(elem_as_float<DT>(v) - xmax);
  });
  rc_sum2_f64(z, unused, s, tog);
  // softmax mass of the set's elements whose key is above `key`, and whether there is one
  bool none_above = false;
  auto mass_above = [&](uint32_t key) {
    double mass = 0.0, count = 0.0;
    for_each_elem<DT>(row, 0, n, [&](T v, int64_t c) {
      if (Elem<DT>::key(v) > key && composite(v, c) >= least) { mass += (double)expf(elem_as_float<DT>(v) - xmax); count += 1.0; }
    });
    rc_sum2_f64(mass, count, s, tog);
    none_above = count == 0.0;
    return mass;
  };
  uint32_t from = 0;   // least key still in question
#pragma unroll 1
  for (int round = 0; round < 8; ++round) {
    auto eligible = [&](T v, int64_t c) { return Elem<DT>::key(v) >= from && composite(v, c) >= least; };
    uint32_t a = 0;
    for_each_elem<DT>(row, 0, n, [&](T v, int64_t c) {
      if (eligible(v, c)) a = max(a, rc_score_key(__fdiv_rn(elem_as_float<DT>(v), T_) + gumbel_screen(noise.at(nrow, c))));
    });
    const uint32_t ak = rc_max_u32(a, s, tog);
    if (ak == 0) return top_col;   // nothing has a score
    const float cut = screen_cut(key_f32(ak));
    uint64_t w = 0;
    for_each_elem<DT>(row, 0, n, [&](T v, int64_t c) {
      if (eligible(v, c)) {
        const float u = noise.at(nrow, c), q = __fdiv_rn(elem_as_float<DT>(v), T_);
        if (q + gumbel_screen(u) >= cut) { const uint64_t x = rc_win_make(q + gumbel_exact(u), c); w = x > w ? x : w; }
      }
    });
    w = block_max(w);
    const int tok = 0x7FFFFFFF - (int)(uint32_t)w;
    const uint32_t wk = Elem<DT>::key(row[tok]);
    const double mass = mass_above(wk);
    if (none_above || !(mass / z >= (double)p)) return tok;
    from = wk + 1;
    if (round == 6) {
      // many records in a row: the least key that is kept, by bisection; the next round is then the last
      uint32_t hi = (uint32_t)(top >> 32);
#pragma unroll 1
      while (from < hi) {
        const uint32_t mid = from + (hi - from) / 2;
        const double m = mass_above(mid);
        if (none_above || !(m / z >= (double)p)) hi = mid; else from = mid + 1;
      }
    }
  }
  return top_col;
}

// Leader: cuts the gathered list to the top-K set.  Elements outside it lose their score (-inf) and their weight
// (value -inf).  K-th greatest key by radix descent from the first bit in which the keys differ; ties at the K-th
// key are admitted by ascending column.
static __device__ __noinline__ void rc_cut_to_k(RcShared& s, int m, int K, int64_t part_len, float* lx, float* ls,
                                                const unsigned short* lpos, uint32_t* bins) {
  int tog = 2;
  uint32_t kmin = s.key_lo, kmax = s.key_hi;   // (a NaN lies above: the top bin takes it)
  // One histogram of 2048 bins over the range of the keys; the K-th key's bin then holds a few elements, which are
  // ranked by counting.
  {
    const uint32_t range = kmax > kmin ? kmax - kmin : 0;
    const int shift = range >> 11 ? 21 - __clz(range) : 0;
    auto bin_of = [&](float x) { return (kRcBins - 1) - (int)min((f32_key(x) - kmin) >> shift, (uint32_t)kRcBins - 1); };
    uint4* b4 = reinterpret_cast<uint4*>(bins);
    b4[threadIdx.x] = make_uint4(0, 0, 0, 0);
    b4[threadIdx.x + kRcThreads] = make_uint4(0, 0, 0, 0);
    if (threadIdx.x == 0) s.pick[3] = 0;
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < m; i += kRcThreads) atomicAdd(&bins[bin_of(lx[i])], 1u);
    __syncthreads();
    const uint4 c0 = b4[2 * threadIdx.x], c1 = b4[2 * threadIdx.x + 1];
    const int sum = (int)(c0.x + c0.y + c0.z + c0.w + c1.x + c1.y + c1.z + c1.w);
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane_id() >= o) incl += up;
    }
    if (lane_id() == 31) s.red_u32[0][warp_id()] = (uint32_t)incl;
    __syncthreads();
#pragma unroll 1
    for (int w = 0; w < warp_id(); ++w) incl += (int)s.red_u32[0][w];
    if (incl - sum < K && incl >= K) {
      int run = incl - sum;
#pragma unroll 1
      for (int j = 0; j < 8; ++j) {
        const int c = (int)bins[8 * threadIdx.x + j];
        if (run + c >= K) { s.pick[0] = 8 * threadIdx.x + j; s.pick[1] = run; s.pick[2] = c; break; }
        run += c;
      }
    }
    __syncthreads();
    const int bin = s.pick[0], need = K - s.pick[1], in_bin = s.pick[2];
    if (in_bin <= 256) {
      uint64_t* list = reinterpret_cast<uint64_t*>(bins);   // (the histogram has been read)
      unsigned short* at = reinterpret_cast<unsigned short*>(list + 256);
      if ((int)threadIdx.x >= in_bin) list[threadIdx.x] = 0;
#pragma unroll 1
      for (int i = threadIdx.x; i < m; i += kRcThreads) {
        const int b = bin_of(lx[i]);
        if (b > bin) { lx[i] = -INFINITY; ls[i] = -INFINITY; }
        else if (b == bin) {
          const int slot = atomicAdd(&s.pick[3], 1);
          list[slot] = ((uint64_t)f32_key(lx[i]) << 32) | (uint32_t)(0x7FFFFFFF - (int32_t)rc_column(s, lpos, i, part_len));
          at[slot] = (unsigned short)i;
        }
      }
      __syncthreads();
      if ((int)threadIdx.x < in_bin) {
        const uint64_t c = list[threadIdx.x];
        const ulonglong2* l2 = reinterpret_cast<const ulonglong2*>(list);
        int before = 0;
#pragma unroll 4
        for (int j = 0; j < (in_bin + 1) / 2; ++j) {
          const ulonglong2 o = l2[j];
          before += (o.x > c ? 1 : 0) + (o.y > c ? 1 : 0);
        }
        if (before >= need) { lx[at[threadIdx.x]] = -INFINITY; ls[at[threadIdx.x]] = -INFINITY; }
      }
      __syncthreads();
      return;
    }
  }
  // keys so spread, or so many equal ones, that the bin holds more than that: digit by digit
  kmax = 0;
  uint32_t kmin_inv = 0;
#pragma unroll 1
  for (int i = threadIdx.x; i < m; i += kRcThreads) {
    const uint32_t k = f32_key(lx[i]);
    kmax = max(kmax, k);
    kmin_inv = max(kmin_inv, ~k);
  }
  kmax = rc_max_u32(kmax, s, tog);
  kmin = ~rc_max_u32(kmin_inv, s, tog);
  int need = K, ties = m;
  uint32_t vk = kmax;          // prefix of the K-th key; bits below `top` are still to be found
  int top = kmax == kmin ? 0 : 32 - __clz(kmax ^ kmin);
  if (top < 32) vk &= ~((1u << top) - 1u); else vk = 0;
#pragma unroll 1
  while (top > 0) {
    const int sh = top > 8 ? top - 8 : 0;
    s.hist[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < m; i += kRcThreads) {
      const uint32_t k = f32_key(lx[i]);
      if (top == 32 || ((k ^ vk) >> top) == 0) atomicAdd(&s.hist[(k >> sh) & ((1u << (top - sh)) - 1u)], 1u);
    }
    __syncthreads();
    if (warp_id() == 0) rc_pick_bin(s.hist, need, s.pick);
    __syncthreads();
    vk |= (uint32_t)s.pick[0] << sh;
    need -= s.pick[1];
    ties = s.pick[2];
    top = sh;
    __syncthreads();
    if (ties == need) break;   // everything in the bin belongs to the set: vk is its lower end
  }
  // ties at the K-th key (vk is complete then): the `need` lowest columns stay, found by the same descent over the columns
  // (distinct and below 2^24), inverted.  Comparing every tie with every other one took 1.2 ms for 1500 equal values.
  uint32_t from = 0;   // least inverted column that stays
  if (need < ties) {
    from = 0x7Fu << 24;
#pragma unroll 1
    for (int sh = 16; sh >= 0; sh -= 8) {
      s.hist[threadIdx.x] = 0;
      __syncthreads();
#pragma unroll 1
      for (int i = threadIdx.x; i < m; i += kRcThreads)
        if (f32_key(lx[i]) == vk) {
          const uint32_t c = 0x7FFFFFFFu - (uint32_t)rc_column(s, lpos, i, part_len);
          if (((c ^ from) >> (sh + 8)) == 0) atomicAdd(&s.hist[(c >> sh) & 255u], 1u);
        }
      __syncthreads();
      if (warp_id() == 0) rc_pick_bin(s.hist, need, s.pick);
      __syncthreads();
      from |= (uint32_t)s.pick[0] << sh;
      need -= s.pick[1];
      const bool whole = s.pick[2] == need;
      __syncthreads();
      if (whole) break;
    }
  }
#pragma unroll 1
  for (int i = threadIdx.x; i < m; i += kRcThreads) {
    const uint32_t k = f32_key(lx[i]);
    if (k < vk || (k == vk && from != 0 && 0x7FFFFFFFu - (uint32_t)rc_column(s, lpos, i, part_len) < from)) { ls[i] = -INFINITY; lx[i] = -INFINITY; }
  }
  __syncthreads();
}

// Leader: the decision (top of the file) over more than kRcSmall candidates, cut to the top-K set.  A round has three
// barriers.  Returns the token, -1 if no kept element has a score.
static __device__ __noinline__ int rc_decide_large(RcShared& s, int m, float pp, int64_t part_len, const float* lx,
                                                   const float* ls, const unsigned short* lpos, float T_, const NoiseSrc& noise,
                                                   int64_t nrow) {
  int tog = 2;
  float above = -INFINITY, x0 = 0.f;
  bool first = true;
#pragma unroll 1
  for (int round = 0; round < kRcListCap; ++round) {
    uint32_t a = 0, xk = 0;
#pragma unroll 1
    for (int i = threadIdx.x; i < m; i += kRcThreads) {
      const float x = lx[i];
      if (first) xk = max(xk, f32_key(x));
      if (first || x > above) a = max(a, rc_score_key(ls[i]));
    }
    a = __reduce_max_sync(0xFFFFFFFFu, a);
    if (first) xk = __reduce_max_sync(0xFFFFFFFFu, xk);
    if (lane_id() == 0) { s.red_u32[2][warp_id()] = a; s.red_u32[3][warp_id()] = xk; }
    if (threadIdx.x == 0) { s.win = 0; s.n_near = 0; }
    __syncthreads();
    a = __reduce_max_sync(0xFFFFFFFFu, s.red_u32[2][lane_id() & (kRcWarps - 1)]);
    if (first) x0 = key_f32(__reduce_max_sync(0xFFFFFFFFu, s.red_u32[3][lane_id() & (kRcWarps - 1)]));
    if (a <= 0x007FFFFFu) return -1;   // NaN or -inf
    const float cut = screen_cut(key_f32(a));
#pragma unroll 1
    for (int i = threadIdx.x; i < m; i += kRcThreads)
      if ((first || lx[i] > above) && ls[i] >= cut) {
        atomicAdd(&s.n_near, 1);
        s.win = (unsigned long long)i;
      }
    __syncthreads();
    int at = (int)s.win;
    if (s.n_near > 1) {   // several within the screening slack of the best: decided on the f64-evaluated noise
      __syncthreads();
      if (threadIdx.x == 0) s.win = 0;
      __syncthreads();
#pragma unroll 1
      for (int i = threadIdx.x; i < m; i += kRcThreads)
        if ((first || lx[i] > above) && ls[i] >= cut) {
          const int64_t col = rc_column(s, lpos, i, part_len);
          atomicMax(&s.win, rc_win_make(__fdiv_rn(lx[i], T_) + gumbel_exact(noise.at(nrow, col)), col));
        }
      __syncthreads();
      const int tok = 0x7FFFFFFF - (int)(uint32_t)s.win;
#pragma unroll 1
      for (int i = threadIdx.x; i < m; i += kRcThreads)
        if ((first || lx[i] > above) && ls[i] >= cut && rc_column(s, lpos, i, part_len) == tok) s.n_near = i;
      __syncthreads();
      at = s.n_near;
    }
    const float wx = lx[at];
    double mass = 0.0, z = 0.0;
#pragma unroll 1
    for (int i = threadIdx.x; i < m; i += kRcThreads) {
      const double w = (double)expf(lx[i] - x0);
      z += w;
      if (lx[i] > wx) mass += w;
    }
    rc_sum2_f64(mass, z, s, tog);
    if (mass == 0.0 || !(mass / z >= (double)pp)) return (int)rc_column(s, lpos, at, part_len);
    above = wx;
    first = false;
  }
  return -1;
}

// Leader: at most 256 candidates.  Every thread ranks one by counting, which sorts the top-K set; one warp then takes
// the softmax prefix, the top-p threshold and the best score among the kept ones.  Returns the token, -1 if no kept
// one has a score.
constexpr int kRcSmall = 256;
static __device__ __noinline__ int rc_decide_small(RcShared& s, int m, int K, float pp, int64_t part_len, const float* lx,
                                                   const float* ls, const unsigned short* lpos, unsigned char* scratch,
                                                   float T_, const NoiseSrc& noise, int64_t nrow) {
  uint64_t* comp = reinterpret_cast<uint64_t*>(scratch);
  float* sx = reinterpret_cast<float*>(comp + kRcSmall);
  float* ss = sx + kRcSmall;
  int* scol = reinterpret_cast<int*>(ss + kRcSmall);
  const int i = threadIdx.x;
  uint64_t mine = 0;
  float x = 0.f, a = 0.f;
  if (i < m) {
    x = lx[i];
    a = ls[i];
    mine = ((uint64_t)f32_key(x) << 32) | (uint32_t)(0x7FFFFFFF - (int32_t)rc_column(s, lpos, i, part_len));
  }
  comp[i] = mine;
  __syncthreads();
  if (i < m) {
    int rank = 0;
    const ulonglong2* c2 = reinterpret_cast<const ulonglong2*>(comp);
#pragma unroll 4
    for (int j = 0; j < (m + 1) / 2; ++j) {
      const ulonglong2 c = c2[j];
      rank += (c.x > mine ? 1 : 0) + (c.y > mine ? 1 : 0);
    }
    if (rank < K) {
      sx[rank] = x;
      ss[rank] = a;
      scol[rank] = 0x7FFFFFFF - (int)(uint32_t)mine;
    }
  }
  __syncthreads();
  if (warp_id() == 0) {
    const int lane = lane_id(), n = min(m, K), per = (n + 31) / 32;
    const int i0 = lane * per, i1 = min(i0 + per, n);
    const float x0 = sx[0];
    double acc = 0.0;
#pragma unroll 1
    for (int j = i0; j < i1; ++j) acc += (double)expf(sx[j] - x0);
    double incl = acc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = shfl_up_f64(incl, o);
      if (lane >= o) incl += up;
    }
    const double Z = __hiloint2double(__shfl_sync(0xFFFFFFFFu, __double2hiint(incl), 31),
                                      __shfl_sync(0xFFFFFFFFu, __double2loint(incl), 31));
    double run = incl - acc;
    int below = 0;
#pragma unroll 1
    for (int j = i0; j < i1; ++j) {
      run += (double)expf(sx[j] - x0);
      below += run / Z < (double)pp ? 1 : 0;
    }
    below = __reduce_add_sync(0xFFFFFFFFu, below);
    // a sum that is not a number keeps everything
    const float thr = Z == Z ? sx[min(below, n - 1)] : -INFINITY;
    uint32_t best = 0;
#pragma unroll 1
    for (int j = i0; j < i1; ++j)
      if (sx[j] >= thr) best = max(best, rc_score_key(ss[j]));
    best = __reduce_max_sync(0xFFFFFFFFu, best);
    int tok = -1;
    if (best > 0x007FFFFFu) {
      const float cut = screen_cut(key_f32(best));
      int near_ = 0;
      uint32_t hi = 0, lo = 0;
#pragma unroll 1
      for (int j = i0; j < i1; ++j)
        if (sx[j] >= thr && ss[j] >= cut) { ++near_; lo = max(lo, (uint32_t)(0x7FFFFFFF - scol[j])); }
      near_ = __reduce_add_sync(0xFFFFFFFFu, near_);
      if (near_ > 1) {   // several within the screening slack of the best: decided on the f64-evaluated noise
        lo = 0;
#pragma unroll 1
        for (int j = i0; j < i1; ++j)
          if (sx[j] >= thr && ss[j] >= cut) {
            const uint32_t k = rc_score_key(__fdiv_rn(sx[j], T_) + gumbel_exact(noise.at(nrow, scol[j])));
            const uint32_t c = (uint32_t)(0x7FFFFFFF - scol[j]);
            if (k > hi || (k == hi && c > lo)) { hi = k; lo = c; }
          }
        const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, hi);
        if (hi != top) lo = 0;
      }
      lo = __reduce_max_sync(0xFFFFFFFFu, lo);
      tok = 0x7FFFFFFF - (int)lo;
    }
    if (lane == 0) s.pick[0] = tok;
  }
  __syncthreads();
  return s.pick[0];
}

// ---- rows without top-k ------------------------------------------------------------------------------------------
constexpr int kRcWideCap = 512;     // survivors of a CTA
constexpr int kRcWideSend = 32;     // survivors a CTA may hand to the leader
constexpr int kRcQueue = 384;       // positions a warp has noted and not yet scored (up to 127 + 32 lanes x 8)
static_assert(kRcWarps * kRcQueue * 2 + kRcWideCap * 4 <= kRcListCap * 4, "the queues lie behind the scores");
static_assert(kRcMaxCluster * kRcWideSend == 512, "the leader's copies of the survivors");

// The places of the survivors in the list's space: this CTA's own ones, and (leader) those that the CTAs have sent,
// kRcWideSend places each.
struct RcWideLists {
  unsigned short *pos, *queue;
  float *x, *s, *all_x, *all_s;
  int* all_col;
  __device__ __forceinline__ RcWideLists(unsigned char* smem, const RcLayout& l) {
    pos = reinterpret_cast<unsigned short*>(smem + l.off_pos);
    all_s = reinterpret_cast<float*>(smem + l.off_pos + kRcWideCap * 2);
    x = reinterpret_cast<float*>(smem + l.off_x);
    all_x = x + kRcWideCap;
    all_col = reinterpret_cast<int*>(all_x + kRcMaxCluster * kRcWideSend);
    s = reinterpret_cast<float*>(smem + l.off_s);
    queue = reinterpret_cast<unsigned short*>(s + kRcWideCap);
  }
};

// What the passes over a row without top-k need of it.
struct RcWideRow {
  int64_t col0, nrow;
  float rt;                  // 1 / T
  const float* dense;        // the part's noise, or null: the key
  uint32_t k0, k1, ctr0;     // key; counter of the part's first element
};

// The least score of a survivor, by its value.
struct RcLow {
  float bx, bs, ms;   // at or below bx: bs; above it: ms
  __device__ __forceinline__ float of(float x) const { return x <= bx ? bs : ms; }
};
// Whether an element can reach the score `cut`: its Gumbel term -log(-log u) is at most -log(1 - u).
__device__ __forceinline__ bool rc_may_reach(float x, float u, float rt, float cut) {
  return 1.0f - u <= __expf(fmaf(x, rt, -cut)) * 1.0001f;
}
template <int DT>
__device__ __forceinline__ void rc_keep_survivor(float x, float u, int i, const RcWideRow& r, RcShared& s, const RcWideLists& w) {
  const float a = fmaf(x, r.rt, gumbel_screen(u));
  bool out = !(a > -INFINITY);
#pragma unroll 1
  for (int j = 0; j < s.n_cut; ++j) out = out || (x <= s.cut_x[j] && a < s.cut_s[j]);
  if (!out) {
    const int slot = atomicAdd(&s.n_list, 1);
    if (slot < kRcWideCap) { w.x[slot] = x; w.s[slot] = a; w.pos[slot] = (unsigned short)i; }
  }
}

// Noise from a key.  Scores `count` (at most 128) noted elements, four per lane: four interleaved chains of dependent
// rounds (with the two warps that a scheduler has here, one chain would leave it idle).
template <int DT>
__device__ __forceinline__ void rc_score_noted(const RcPart<DT>& part, const unsigned short* queue, int count, const RcLow& low,
                                               const RcWideRow& r, RcShared& s, const RcWideLists& w) {
  int at[4];
  float u[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int q = lane_id() + 32 * k;
    at[k] = q < count ? queue[q] : -1;
    u[k] = fmaxf(threefry_uniform01(r.k0, r.k1, r.ctr0 + (uint32_t)at[k]), kF32Tiny);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (at[k] < 0) continue;
    const float x = elem_as_float<DT>(part.elem(at[k]));
    if (rc_may_reach(x, u[k], r.rt, low.of(x))) rc_keep_survivor<DT>(x, u[k], at[k], r, s, w);
  }
}

// The part's survivors (see the top of the file) into the CTA's list.
//   From a key: a warp notes the positions whose value allows a survivor at all and makes their noise 128 at a time.
//   From a tensor: the noise is read beside the values, and a vector is looked into if its greatest value with its
//   greatest noise could survive.
template <int DT>
__device__ __forceinline__ void rc_survivors(const RcPart<DT>& part, const RcLow& low, float xcut, const RcWideRow& r,
                                               RcShared& s, const RcWideLists& l) {
  using T = typename Elem<DT>::type;
  constexpr int VEC = RcPart<DT>::VEC;
  const int lane = lane_id();
  unsigned short* queue = l.queue + warp_id() * kRcQueue;
  const bool aligned = r.dense && (reinterpret_cast<uintptr_t>(r.dense - part.off) & 15) == 0;
  int waiting = 0;
#pragma unroll 1
  for (int v0 = 0; v0 < part.nvec; v0 += kRcThreads) {
    const int v = v0 + threadIdx.x;
    const bool last = v0 + kRcThreads >= part.nvec;
    uint32_t mask = 0;
    float u[VEC];
    if (v < part.nvec) {
      const uint4 w = part.vec[v];
      const T* e = reinterpret_cast<const T*>(&w);
      const int i0 = v * VEC - part.off;
      if (r.dense) {
        if (aligned && i0 >= 0 && i0 + VEC <= part.n) {
#pragma unroll
          for (int j = 0; j < VEC; j += 4) {
            const float4 q = __ldcs(reinterpret_cast<const float4*>(r.dense + i0 + j));
            u[j] = q.x; u[j + 1] = q.y; u[j + 2] = q.z; u[j + 3] = q.w;
          }
        } else {
#pragma unroll
          for (int j = 0; j < VEC; ++j) u[j] = i0 + j >= 0 && i0 + j < part.n ? __ldg(r.dense + i0 + j) : 0.f;
        }
      }
      if (r.dense) {
        float xm = elem_as_float<DT>(e[0]), um = u[0];
#pragma unroll
        for (int j = 1; j < VEC; ++j) { xm = fmaxf(xm, elem_as_float<DT>(e[j])); um = fmaxf(um, u[j]); }
        if (rc_may_reach(xm, um, r.rt, low.of(xm))) {
#pragma unroll
          for (int j = 0; j < VEC; ++j) {
            const float x = elem_as_float<DT>(e[j]);
            if (x > -INFINITY && rc_may_reach(x, u[j], r.rt, low.of(x))) rc_keep_survivor<DT>(x, u[j], i0 + j, r, s, l);
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < VEC; ++j) mask |= elem_as_float<DT>(e[j]) >= xcut ? 1u << j : 0u;
        if (xcut == -INFINITY) {   // nothing is ruled out by its value: leave out what lies outside the part
          for (int j = 0; j < VEC; ++j)
            if (i0 + j < 0 || i0 + j >= part.n) mask &= ~(1u << j);
        }
      }
    }
    if (r.dense) continue;
    if (__ballot_sync(0xFFFFFFFFu, mask != 0)) {
      int incl = __popc(mask);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += up;
      }
      int at = waiting + incl - __popc(mask);
      while (mask) {
        const int j = __ffs(mask) - 1;
        mask &= mask - 1;
        queue[at++] = (unsigned short)(v * VEC + j - part.off);
      }
      waiting += __shfl_sync(0xFFFFFFFFu, incl, 31);
      __syncwarp();
    }
    while (waiting >= 128 || (last && waiting > 0)) {
      const int count = min(waiting, 128);
      waiting -= count;
      rc_score_noted<DT>(part, queue + waiting, count, low, r, s, l);
    }
    __syncwarp();
  }
}

// Leader, warp 0: the best of the survivors that the CTAs have sent, among those above `above` (all of them if `first`):
// its place, -1 if none has a score.  `most`: the greatest number that a CTA has sent.
__device__ __forceinline__ int rc_best_sent(int most, bool first, float above, const RcWideLists& l, float T_,
                                            const NoiseSrc& noise, int64_t nrow) {
  const int i0 = (lane_id() & 15) * kRcWideSend + (lane_id() >> 4), i1 = i0 + (most + 1) / 2 * 2;   // every other place
  uint32_t a = 0;
#pragma unroll 1
  for (int i = i0; i < i1; i += 2)
    if (first || l.all_x[i] > above) a = max(a, rc_score_key(l.all_s[i]));
  a = __reduce_max_sync(0xFFFFFFFFu, a);
  if (a <= 0x007FFFFFu) return -1;
  const float cut = screen_cut(key_f32(a));
  int near_ = 0, at = -1;
#pragma unroll 1
  for (int i = i0; i < i1; i += 2)
    if ((first || l.all_x[i] > above) && l.all_s[i] >= cut) { ++near_; at = i; }
  near_ = __reduce_add_sync(0xFFFFFFFFu, near_);
  if (near_ > 1) {   // several within the screening slack: decided on the f64-evaluated noise
    uint32_t hi = 0, lo = 0;
    at = -1;
#pragma unroll 1
    for (int i = i0; i < i1; i += 2)
      if ((first || l.all_x[i] > above) && l.all_s[i] >= cut) {
        const int col = l.all_col[i];
        const uint32_t k = rc_score_key(__fdiv_rn(l.all_x[i], T_) + gumbel_exact(noise.at(nrow, col)));
        const uint32_t c = (uint32_t)(0x7FFFFFFF - col);
        if (k > hi || (k == hi && c > lo)) { hi = k; lo = c; at = i; }
      }
    const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, hi);
    const uint32_t low = __reduce_max_sync(0xFFFFFFFFu, hi == top ? lo : 0u);
    if (hi != top || lo != low) at = -1;
  }
  return __reduce_max_sync(0xFFFFFFFFu, at);
}

// Warp 0: more than kRcWideSend survivors: drops those that another one dominates, in place.
__device__ __forceinline__ int rc_thin_out(int m, float* lx, float* ls, unsigned short* lpos) {
  const int lane = lane_id();
  float above = -INFINITY;
  bool first = true;
  // marks are collected in the scores' sign of life: a dominated entry gets the score -inf
#pragma unroll 1
  for (int round = 0; round < 2 * kRcWideSend; ++round) {
    uint32_t a = 0;
#pragma unroll 1
    for (int i = lane; i < m; i += 32) if (first || lx[i] > above) a = max(a, rc_score_key(ls[i]));
    a = __reduce_max_sync(0xFFFFFFFFu, a);
    if (a <= 0x007FFFFFu) break;
    uint32_t xk = 0;
#pragma unroll 1
    for (int i = lane; i < m; i += 32)
      if ((first || lx[i] > above) && rc_score_key(ls[i]) == a) xk = max(xk, f32_key(lx[i]));
    const float x = key_f32(__reduce_max_sync(0xFFFFFFFFu, xk)), cut = screen_cut(key_f32(a));
#pragma unroll 1
    for (int i = lane; i < m; i += 32)
      if ((first || lx[i] > above) && lx[i] <= x && ls[i] < cut) ls[i] = -INFINITY;
    __syncwarp();
    above = x;
    first = false;
  }
  int kept = 0;
#pragma unroll 1
  for (int i0 = 0; i0 < m; i0 += 32) {
    const int i = i0 + lane;
    const float x = i < m ? lx[i] : 0.f, a = i < m ? ls[i] : -INFINITY;
    const unsigned short q = i < m ? lpos[i] : 0;
    const unsigned live = __ballot_sync(0xFFFFFFFFu, a > -INFINITY);
    const int to = kept + __popc(live & ((1u << lane) - 1u));
    if (a > -INFINITY) { lx[to] = x; ls[to] = a; lpos[to] = q; }
    kept += __popc(live);
    __syncwarp();
  }
  return kept;
}

// The thread's share of the softmax denominator and of the mass above two values (q0 <= q1).  Four sums of each: f64
// additions are a chain of latencies.
template <int DT>
__device__ __forceinline__ void rc_masses(const RcPart<DT>& part, float xmax, float q0, float q1, double& z, double& m0, double& m1) {
  using T = typename Elem<DT>::type;
  constexpr int VEC = RcPart<DT>::VEC;
  double zs[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
  for (int v = threadIdx.x; v < part.nvec; v += kRcThreads) {
    const uint4 w = part.vec[v];
    const T* e = reinterpret_cast<const T*>(&w);
    const bool any = rc_any_at_least<DT>(w, q0);
    double y[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      y[j] = (double)expf(elem_as_float<DT>(e[j]) - xmax);
      zs[j & 3] += y[j];
    }
    if (any) {
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        const float x = elem_as_float<DT>(e[j]);
        if (x > q0) m0 += y[j];
        if (x > q1) m1 += y[j];
      }
    }
  }
  z = (zs[0] + zs[1]) + (zs[2] + zs[3]);
}

// The thread's share of the mass above a value alone.
template <int DT>
__device__ __forceinline__ void rc_masses_above(const RcPart<DT>& part, float xmax, float q, double& mass) {
  using T = typename Elem<DT>::type;
  constexpr int VEC = RcPart<DT>::VEC;
#pragma unroll 1
  for (int v = threadIdx.x; v < part.nvec; v += kRcThreads) {
    const uint4 w = part.vec[v];
    if (!rc_any_at_least<DT>(w, q)) continue;
#pragma unroll 1
    for (int j = 0; j < VEC; ++j) {
      const float x = elem_as_float<DT>(reinterpret_cast<const T*>(part.vec + v)[j]);
      if (x > q) mass += (double)expf(x - xmax);
    }
  }
}

// Rows with 1024 < top_k < vocab and rows whose lists overflowed: cuts the row, which lies in the parts, to its top-K set.  What is outside the set becomes
// -inf, and the row is then one without top-k.
//   The K-th greatest key comes from histograms of 2048 bins, eleven bits of the key at a time (two for bf16, three for f32, in
// `bins`); the leader adds the CTAs' bins up and tells them which one holds the K-th key.  Of keys equal to it the lowest
// columns belong to the set: the CTAs' own counts say how many of each part.
//   Bound by latency: three reads of the part and four or six cluster barriers, about 15 us a row.  top_k 2000, a call: bf16
// [8, 128256] 44 us, f32 [32, 128256] 70 us (by rc_slow_row, one CTA a row over global memory, 699 and 809 us).
template <int DT>
static __device__ __noinline__ void rc_cut_parts(uint4* vec, int off, int n, int nvec, int K, int cluster, uint32_t rank,
                                                 RcShared& s, uint32_t* bins) {
  using T = typename Elem<DT>::type;
  constexpr int VEC = 16 / (int)sizeof(T), kBits = 8 * (int)sizeof(T), kDigit = 11;
  static_assert(1 << kDigit == kRcBins && kRcBins == 8 * kRcThreads, "eight bins a thread");
  auto key_of = [](T v) { return Elem<DT>::key(v) >> (32 - kBits); };   // (a bf16 is told by the upper half)
  int need = K, in_bin = 0, bin = 0, top = kBits;
  uint32_t vk = 0;   // the K-th key's bits from `top` on
#pragma unroll 1
  do {
    const int sh = top > kDigit ? top - kDigit : 0;
    const uint32_t least = vk, width_mask = top == 32 ? 0xFFFFFFFFu : (1u << top) - 1u;
    uint4* b4 = reinterpret_cast<uint4*>(bins);
    b4[threadIdx.x] = make_uint4(0, 0, 0, 0);
    b4[threadIdx.x + kRcThreads] = make_uint4(0, 0, 0, 0);
    __syncthreads();
#pragma unroll 1
    for (int v = threadIdx.x; v < nvec; v += kRcThreads) {
      const uint4 w = vec[v];
      const T* e = reinterpret_cast<const T*>(&w);
      uint32_t at = 0;
      uint32_t run = 0;   // equal neighbours are added at once
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        const uint32_t d = key_of(e[j]) - least;   // (below `least`: wraps to a distance beyond the range)
        if (d <= width_mask && (unsigned)(v * VEC + j - off) < (unsigned)n) {
          if (run && (d >> sh) != at) { atomicAdd(&bins[at], run); run = 0; }
          at = d >> sh;
          ++run;
        }
      }
      if (run) atomicAdd(&bins[at], run);
    }
    cl_sync();
    if (rank == 0) {
      // thread t: the bins 8 t' .. 8 t' + 7, t' = 255 - t, of all CTAs
      const int t = kRcThreads - 1 - (int)threadIdx.x;
      uint32_t c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 2
      for (int r = 0; r < cluster; ++r) {
        const uint32_t a = cl_map(bins + 8 * t, (uint32_t)r);
        const uint4 x = cl_ld_v4(a), y = cl_ld_v4(a + 16);
        c[0] += x.x; c[1] += x.y; c[2] += x.z; c[3] += x.w;
        c[4] += y.x; c[5] += y.y; c[6] += y.z; c[7] += y.w;
      }
      int sum = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) sum += (int)c[j];
      int incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane_id() >= o) incl += up;
      }
      if (lane_id() == 31) s.red_u32[0][warp_id()] = (uint32_t)incl;
      __syncthreads();
#pragma unroll 1
      for (int w = 0; w < warp_id(); ++w) incl += (int)s.red_u32[0][w];
      if (incl - sum < need && incl >= need) {
        int run = incl - sum, found = 0, above = 0, count = 0;
#pragma unroll
        for (int j = 7; j >= 0; --j) {
          if (run < need && run + (int)c[j] >= need) { found = 8 * t + j; above = run; count = (int)c[j]; }
          run += (int)c[j];
        }
#pragma unroll 1
        for (int r = 0; r < cluster; ++r) {
          cl_st_u32(cl_map(&s.pick[0], (uint32_t)r), (uint32_t)found);
          cl_st_u32(cl_map(&s.pick[1], (uint32_t)r), (uint32_t)above);
          cl_st_u32(cl_map(&s.pick[2], (uint32_t)r), (uint32_t)count);
        }
      }
    }
    cl_sync();
    bin = s.pick[0];
    need -= s.pick[1];
    in_bin = s.pick[2];
    vk |= (uint32_t)bin << sh;
    top = sh;
  } while (top > 0 && in_bin != need);   // (a bin that belongs to the set as a whole needs no finer look)

  // elements of this part among the `need` of the last bin: `allowed` of its `mine`, those of the lowest columns
  int mine = 0, allowed = 0;
  if (in_bin != need) {
    const int lane = lane_id();
    mine = (int)bins[bin];
    const int c = lane < cluster && lane < (int)rank ? (int)cl_ld_u32(cl_map(bins + bin, (uint32_t)lane)) : 0;
    allowed = min(max(need - (int)__reduce_add_sync(0xFFFFFFFFu, (unsigned)c), 0), mine);
  }
  const bool in_order = allowed > 0 && allowed < mine;
  const bool above_only = in_bin != need && allowed == 0;
  int seen = 0, tog = 2;
#pragma unroll 1
  for (int v0 = 0; v0 < nvec; v0 += kRcThreads) {
    const int v = v0 + threadIdx.x;
    uint32_t keep = 0, ties = 0;
    if (v < nvec) {
      const uint4 w = vec[v];
      const T* e = reinterpret_cast<const T*>(&w);
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        const uint32_t k = key_of(e[j]);
        if (above_only ? k > vk : k >= vk) keep |= 1u << j;
        if (in_order && k == vk && (unsigned)(v * VEC + j - off) < (unsigned)n) ties |= 1u << j;
      }
    }
    if (in_order) {
      int incl = __popc(ties);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane_id() >= o) incl += up;
      }
      if (lane_id() == 31) s.red_u32[tog][warp_id()] = (uint32_t)incl;
      __syncthreads();
      int before = seen + incl - __popc(ties);
#pragma unroll
      for (int u = 0; u < kRcWarps; ++u) {
        const int c = (int)s.red_u32[tog][u];
        before += u < warp_id() ? c : 0;
        seen += c;
      }
      tog ^= 1;
      for (uint32_t m = ties; m; m &= m - 1, ++before)
        if (before >= allowed) keep &= ~(m & (0u - m));
    }
    if (v < nvec && keep != (1u << VEC) - 1u) {
      T* e = reinterpret_cast<T*>(vec + v);
#pragma unroll
      for (int j = 0; j < VEC; ++j)
        if (!(keep >> j & 1u)) {
          if constexpr (DT == TLX_F32) e[j] = -INFINITY;
          else e[j] = __float2bfloat16_rn(-INFINITY);
        }
    }
  }
  __syncthreads();
}

// Rows with 1 <= top_k <= 1024 and greedy rows.  Returns the token in the leader (rank 0), -1 if the row has to be
// answered by rc_slow_row; the other CTAs return -1 when they may leave.  kRcOver, in every CTA alike: the lists overflowed
// (huge groups of equal values; fewer finite groups than top_k), and the row has to be cut in the parts.
constexpr int kRcOver = -2;
template <int DT>
__device__ __forceinline__ int rc_normal_row(const RcSampleParams& p, const RcPart<DT>& part, int64_t col0, uint32_t rank, int K,
                                             float pp, float T_, int64_t nrow, RcShared& s, const RcLayout& l,
                                             unsigned char* smem) {
  float* lx = reinterpret_cast<float*>(smem + l.off_x);
  float* ls = reinterpret_cast<float*>(smem + l.off_s);
  unsigned short* lpos = reinterpret_cast<unsigned short*>(smem + l.off_pos);
  uint32_t* bound = reinterpret_cast<uint32_t*>(smem + l.off_bound);
  const bool greedy = T_ < kSamplingEps;
  float thr = key_f32(0x80u << 16);
  if (p.sp.vocab > kRcListCap) {
    GroupMax<DT> gm;
    gm.init();
#pragma unroll 2
    for (int v = threadIdx.x; v < part.nvec; v += kRcThreads) gm.add(part.vec[v]);
    rc_publish_maxima<DT>(gm, l.bound_words, bound);
    cl_sync();
    TLX_STAMP(p.sp, 2);
    thr = key_f32(rc_bound_key16(bound, l.bound_words, K, s) << 16);
  } else {
    if (threadIdx.x == 0) { s.key_lo = 0x80u << 16; s.key_hi = 0xFFFFFFFFu; }
    cl_sync();
  }
  TLX_STAMP(p.sp, 3);
  rc_filter<DT>(part, thr, s, lx, lpos);
  __syncthreads();
  TLX_STAMP(p.sp, 4);
  const int nl = min(s.n_list, kRcListCap);
#pragma unroll 1
  for (int i = threadIdx.x; i < nl; i += kRcThreads) {
    float a = 0.f;
    if (!greedy) a = __fdiv_rn(lx[i], T_) + gumbel_screen(p.sp.noise.at(nrow, col0 + lpos[i]));
    ls[i] = a;
  }
  TLX_STAMP(p.sp, 5);
  cl_sync();
  TLX_STAMP(p.sp, 6);
  const bool full = rc_count(s, p.cluster);
  if (full && !greedy) return kRcOver;
  if (rank != 0) {
    cl_sync();
    return -1;
  }
  const int m = full ? -1 : rc_collect(s, p.cluster, lx, ls, lpos);
  cl_arrive();   // the other CTAs may leave
  TLX_STAMP(p.sp, 7);
  int tok = -1;
  if (m > 0 && greedy) {
    if (threadIdx.x == 0) s.win = 0;
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < m; i += kRcThreads)
      atomicMax(&s.win, ((unsigned long long)f32_key(lx[i]) << 32) |
                            (uint32_t)(0x7FFFFFFF - (int32_t)rc_column(s, lpos, i, p.part_len)));
    __syncthreads();
    tok = 0x7FFFFFFF - (int)(uint32_t)s.win;
  } else if (m > 0 && m <= kRcSmall) {
    tok = rc_decide_small(s, m, K, pp, p.part_len, lx, ls, lpos, smem + l.off_part, T_, p.sp.noise, nrow);
  } else if (m > 0) {
    if (m > K) rc_cut_to_k(s, m, K, p.part_len, lx, ls, lpos, reinterpret_cast<uint32_t*>(smem + l.off_part));
    TLX_STAMP(p.sp, 8);
    tok = rc_decide_large(s, m, pp, p.part_len, lx, ls, lpos, T_, p.sp.noise, nrow);
  }
  cl_wait();
  TLX_STAMP(p.sp, 9);
  return tok;
}

// ---- rows without top-k of which top-p leaves a share -----------------------------------------------------------------
constexpr float kRcPruneBelow = 0.9999f;   // top_p from which on hardly anything is ruled out by it
// Elements of a part from which on it is worth it; with noise from a tensor all it saves is the tensor's reading.  us without / with,
// no top-k: tensor f32 [8, 32000] (parts of 2000) 13.8 / 15.7, [64, 50257] (6283) 28.8 / 25.4, [8, 151936] (9496) 23.6 / 22.1; key f32
// [8, 32000] 15.5 / 15.9, bf16 [1, 128256] (8016) 16.0 / 14.1, f32 [64, 50257] 37.8 / 29.3, bf16 [32, 128256] 45 / 31.
constexpr int kRcPruneTensorPart = 6000, kRcPruneKeyPart = 3000;
constexpr int kRcMassBins = 16;
constexpr int kRcScan = -3;                // rc_pruned_row: not settled here

// A normal f32 that is not negative as f64, by integer operations (the conversion is an eighth-rate instruction).  Zero becomes
// 2^-127, which no sum with an addend of 1 notices.
__device__ __forceinline__ double rc_widen(float y) {
  const uint32_t b = __float_as_uint(y);
  return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}

// The thread's share of the softmax denominator, and of the mass at the distances [i, i + 1), i < 16, below the greatest
// element: bin i in acc[256 i + thread].  The bins only rule elements out, with a margin; they are f32.  A NaN makes the
// denominator one.
template <int DT>
__device__ __forceinline__ double rc_mass_bins(const RcPart<DT>& part, float xmax, float* acc) {
  using T = typename Elem<DT>::type;
  constexpr int VEC = RcPart<DT>::VEC;
  float* mine = acc + threadIdx.x;
#pragma unroll
  for (int i = 0; i < kRcMassBins; ++i) mine[kRcThreads * i] = 0.f;
  double zs[4] = {0.0, 0.0, 0.0, 0.0};
  bool nan = false;
#pragma unroll 1
  for (int v = threadIdx.x; v < part.nvec; v += kRcThreads) {
    const uint4 w = part.vec[v];
    const T* e = reinterpret_cast<const T*>(&w);
    const bool any = rc_any_at_least<DT>(w, xmax - (float)kRcMassBins);
    float y[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      y[j] = expf(elem_as_float<DT>(e[j]) - xmax);
      nan = nan || y[j] != y[j];
      zs[j & 3] += rc_widen(y[j]);
    }
    if (any) {
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        const float d = xmax - elem_as_float<DT>(e[j]);
        // (int)d without a conversion: the low bits of d + 2^23, rounded towards zero
        if (d < (float)kRcMassBins) mine[kRcThreads * (__float_as_int(__fadd_rz(d, 8388608.0f)) & (kRcMassBins - 1))] += y[j];
      }
    }
  }
  const double z = (zs[0] + zs[1]) + (zs[2] + zs[3]);
  return nan ? __longlong_as_double(0x7FF8000000000000ll) : z;
}

// The best screened score of the part's elements from `lo` on, per thread: score, place, and the second best score.  A warp
// notes their positions and scores them 128 at a time, four interleaved chains a lane; what cannot reach the warp's best score so
// far, less the screening slack, is passed over.
struct RcTop {
  float a1, a2;
  int at;
};
template <int DT>
__device__ __forceinline__ RcTop rc_best_from(const RcPart<DT>& part, float lo, const RcWideRow& r, unsigned short* queue) {
  using T = typename Elem<DT>::type;
  constexpr int VEC = RcPart<DT>::VEC;
  const int lane = lane_id();
  const uint32_t lt = (1u << lane) - 1u;
  RcTop best{-INFINITY, -INFINITY, 0};
  float reach = -INFINITY;
  int waiting = 0;
#pragma unroll 1
  for (int v0 = 0; v0 < part.nvec; v0 += kRcThreads) {
    const int v = v0 + threadIdx.x;
    const bool last = v0 + kRcThreads >= part.nvec;
    uint32_t mask = 0;
    if (v < part.nvec) {
      const uint4 w = part.vec[v];
      const T* e = reinterpret_cast<const T*>(&w);
#pragma unroll
      for (int j = 0; j < VEC; ++j) mask |= elem_as_float<DT>(e[j]) >= lo ? 1u << j : 0u;   // (outside the part: -inf)
    }
    // every lane's first element, every lane's second one, ...
    for (uint32_t some = __ballot_sync(0xFFFFFFFFu, mask != 0); some; some = __ballot_sync(0xFFFFFFFFu, mask != 0)) {
      if (mask) queue[waiting + __popc(some & lt)] = (unsigned short)(v * VEC + __ffs(mask) - 1 - part.off);
      mask &= mask - 1;
      waiting += __popc(some);
    }
    __syncwarp();
    while (waiting >= 128 || (last && waiting > 0)) {
      const int count = min(waiting, 128);
      waiting -= count;
      int at[4];
      float u[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        at[k] = lane + 32 * k < count ? queue[waiting + lane + 32 * k] : -1;
        if (r.dense) u[k] = at[k] >= 0 ? __ldg(r.dense + at[k]) : 0.f;
      }
      if (!r.dense) {
#pragma unroll
        for (int k = 0; k < 4; ++k) u[k] = fmaxf(threefry_uniform01(r.k0, r.k1, r.ctr0 + (uint32_t)at[k]), kF32Tiny);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (at[k] < 0) continue;
        const float x = elem_as_float<DT>(part.elem(at[k]));
        if (!rc_may_reach(x, u[k], r.rt, reach)) continue;
        const float a = fmaf(x, r.rt, gumbel_screen(u[k]));
        if (a > best.a1) { best.a2 = best.a1; best.a1 = a; best.at = at[k]; }
        else if (a > best.a2) best.a2 = a;
      }
      const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, rc_score_key(best.a1));
      if (top > 0x007FFFFFu) reach = screen_cut(key_f32(top));
    }
    __syncwarp();
  }
  return best;
}

// Top-p first: the denominator and the mass at sixteen distances from the greatest element say, in every CTA alike, from which
// value on elements can be kept at all, within one unit of the logits; those are scored, and the best of them wins if the mass
// above it is below top_p * Z.  If not, the best of the greater ones is next.  `x`: the thread's greatest element.
//   Returns the token (in every CTA), -1 if there is no finite maximum, kRcScan if the row is left to the way without
// bounds on the values: nothing is ruled out, no score, several scores within the screening slack of the best, or groups whose
// greatest elements are all equal (`least`: the least of the thread's), as a rule a constant row.
//   Four cluster barriers and three short loops over the part.  What bounds it: the denominator (5 of 20 us a row of bf16 [32, 128256]:
// 24 instructions an element, two of them eighth-rate) and the scores (6 us).  us a call, without / with it: noise from a
// key, bf16 [32, 128256] mixed parameters 32.5 / 23.3, no top-k 41 / 28.5, [40, 179328] 64 / 46; f32 [64, 50257] 34 / 25; tensor
// bf16 [32, 128256] mixed 25.3 / 23.5, [40, 179328] 34 / 29; flat rows 134 / 74.
//   Tried: the bins as 2^-23ths by integer atomics 6.6 us instead of 5.7; noise of a tensor read beside the values, two vectors a turn,
// 9 us instead of 6 (the queue has 128 reads in flight a warp).
template <int DT>
__device__ __forceinline__ int rc_pruned_row(const RcSampleParams& p, const RcPart<DT>& part, int64_t col0, float x, float least, float pp,
                                             const RcWideRow& r, RcShared& s, const RcLayout& layout, unsigned char* smem, int& tog) {
  const int lane = lane_id(), of = lane < p.cluster ? lane : 0;
  const bool asks = lane < p.cluster;
  const uint32_t xm = rc_max_u32(f32_key(x), s, tog), lm = ~rc_max_u32(~f32_key(least), s, tog);
  if (threadIdx.x == 0) { s.dom_x[0] = key_f32(xm); s.dom_x[1] = key_f32(lm); }
  cl_sync();
  TLX_STAMP(p.sp, 2);
  const uint32_t at_x = cl_map(s.dom_x, (uint32_t)of);
  const float xmax = key_f32(__reduce_max_sync(0xFFFFFFFFu, f32_key(cl_ld_f32(at_x))));
  const float xleast = key_f32(__reduce_min_sync(0xFFFFFFFFu, f32_key(cl_ld_f32(at_x + 4))));
  if (!(fabsf(xmax) < INFINITY) || xleast == xmax) {
    cl_sync();
    return xleast == xmax && fabsf(xmax) < INFINITY ? kRcScan : -1;
  }
  float* acc = reinterpret_cast<float*>(smem + layout.off_x);
  double z = rc_mass_bins<DT>(part, xmax, acc), unused = 0.0;
  rc_sum2_f64(z, unused, s, tog);
  static_assert(kRcMassBins == 2 * kRcWarps && kRcMassBins * kRcThreads * 4 <= kRcListCap * 8, "two bins a warp, in the lists' space");
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int bin = 2 * warp_id() + h;
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < kRcThreads / 32; ++i) m += acc[kRcThreads * bin + 32 * i + lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xFFFFFFFFu, m, o);
    if (lane == 0) s.bin_mass[bin] = m;
  }
  if (threadIdx.x == 0) s.z_part = z;
  cl_sync();
  TLX_STAMP(p.sp, 3);
  double Z = asks ? cl_ld_f64(cl_map(&s.z_part, (uint32_t)of)) : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) Z += shfl_xor_f64(Z, o);
  float mass = 0.f;
#pragma unroll 1
  for (int i = 0; i < p.cluster; ++i) mass += cl_ld_f32(cl_map(&s.bin_mass[lane & (kRcMassBins - 1)], (uint32_t)i));
#pragma unroll
  for (int o = 1; o < kRcMassBins; o <<= 1) {
    const float up = __shfl_up_sync(0xFFFFFFFFu, mass, o);
    if (lane >= o) mass += up;
  }
  // an element is out if what is nearer to the greatest one than its unit's upper end has a share of top_p already
  const unsigned enough = __ballot_sync(0xFFFFFFFFu, lane < kRcMassBins && (double)mass >= (double)pp * 1.0001 * Z);
  int tok = kRcScan;
  if (enough) {
    float lo = xmax - (float)__ffs(enough);
    lo -= 1e-5f * fmaxf(fabsf(lo), fabsf(xmax));   // (the distances are rounded)
    lo = fmaxf(lo, -FLT_MAX);                      // (finite also next to the type's least value: what lies outside the part is -inf)
    unsigned short* queue = reinterpret_cast<unsigned short*>(smem + layout.off_s) + warp_id() * kRcQueue;
#pragma unroll 1
    for (int round = 0; round < 8; ++round) {
      const RcTop best = rc_best_from<DT>(part, lo, r, queue);
      if (round == 0) { TLX_STAMP(p.sp, 10); }
      // of the CTA: the best score, its element, and the second best score
      const uint32_t mine = rc_score_key(best.a1), ak = rc_max_u32(mine, s, tog);
      if (mine == ak) s.pick[3] = (int)threadIdx.x;
      __syncthreads();
      const bool chosen = s.pick[3] == (int)threadIdx.x;
      const uint32_t ak2 = rc_max_u32(rc_score_key(chosen ? best.a2 : best.a1), s, tog);
      if (chosen) {
        s.query[0] = key_f32(ak);
        s.query[1] = elem_as_float<DT>(part.elem(best.at));
        s.query[2] = key_f32(ak2);
        s.query_tok[0] = (int)(col0 + best.at);
      }
      if (round == 0) { TLX_STAMP(p.sp, 5); }
      cl_sync();
      const uint32_t q = cl_map(s.query, (uint32_t)of);
      const float a = asks ? cl_ld_f32(q) : -INFINITY, xa = cl_ld_f32(q + 4), a2 = asks ? cl_ld_f32(q + 8) : -INFINITY;
      const int ta = (int)cl_ld_u32(cl_map(s.query_tok, (uint32_t)of));
      const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, rc_score_key(a));
      if (top <= 0x007FFFFFu) break;   // no score
      const float cut = screen_cut(key_f32(top));
      const unsigned near_ = __ballot_sync(0xFFFFFFFFu, a >= cut);
      if (__popc(near_) > 1 || __any_sync(0xFFFFFFFFu, a2 >= cut)) break;
      const int winner = __ffs(near_) - 1;
      const float x1 = __shfl_sync(0xFFFFFFFFu, xa, winner);
      const int t1 = __shfl_sync(0xFFFFFFFFu, ta, winner);
      if (x1 == xmax) { tok = t1; break; }   // nothing lies above it: kept whatever top_p is
      // the mass down to the lower end of its unit is below top_p, which settles it; else the mass above it is summed up
      const float upto = __shfl_sync(0xFFFFFFFFu, mass, min((int)(xmax - x1), kRcMassBins - 1));
      if ((double)upto < (double)pp * 0.9999 * Z) { tok = t1; break; }
      double above = 0.0, none = 0.0;
      rc_masses_above<DT>(part, xmax, x1, above);
      rc_sum2_f64(above, none, s, tog);
      if (threadIdx.x == 0) s.z_part = above;   // (the denominator's parts were read before the last barrier of the cluster)
      if (round == 0) { TLX_STAMP(p.sp, 13); }
      cl_sync();
      double m = asks ? cl_ld_f64(cl_map(&s.z_part, (uint32_t)of)) : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m += shfl_xor_f64(m, o);
      if (m == 0.0 || !(m / Z >= (double)pp)) { tok = t1; break; }
      lo = key_f32(f32_key(x1) + 1u);
    }
  }
  cl_sync();   // nobody leaves, or goes on, while its words may still be read
  return tok;
}

// Rows without top-k.  Returns the token in the leader, -1 if the row has to be answered by rc_slow_row.
template <int DT>
__device__ __forceinline__ int rc_wide_row(const RcSampleParams& p, const RcPart<DT>& part, int64_t col0, uint32_t rank, float pp,
                                           float T_, int64_t nrow, RcShared& s, const RcLayout& layout, unsigned char* smem,
                                           int& tog) {
  using T = typename Elem<DT>::type;
  constexpr int VEC = RcPart<DT>::VEC;
  const RcWideLists l(smem, layout);
  const NoiseSrc& noise = p.sp.noise;
  RcWideRow r;
  r.col0 = col0;
  r.nrow = nrow;
  r.rt = __frcp_rn(T_);
  r.dense = noise.dense ? noise.dense_row(nrow) + col0 : nullptr;
  r.k0 = r.k1 = r.ctr0 = 0;
  if (!r.dense) {
    r.k0 = noise.key_dev ? __ldg(noise.key_dev) : noise.k0;
    r.k1 = noise.key_dev ? __ldg(noise.key_dev + 1) : noise.k1;
    r.ctr0 = (uint32_t)(noise.row_of(nrow) * noise.vocab + col0);
  }
  // every thread's greatest element
  GroupMax<DT> gm;
  gm.init();
#pragma unroll 2
  for (int v = threadIdx.x; v < part.nvec; v += kRcThreads) gm.add(part.vec[v]);
  float x = -INFINITY, least = INFINITY;   // (groups without a finite element are left out of the least)
#pragma unroll
  for (int j = 0; j < GroupMax<DT>::kSlots; ++j) {
    const float g = gm.slot(j);
    x = fmaxf(x, g);
    if (g > -INFINITY) least = fminf(least, g);
  }
  if (pp < kRcPruneBelow && p.part_len >= (r.dense ? kRcPruneTensorPart : kRcPruneKeyPart)) {
    const int tok = rc_pruned_row<DT>(p, part, col0, x, least, pp, r, s, layout, smem, tog);
    if (tok != kRcScan) return tok;
  }
  // its score; of the CTA: the greatest element and the best-scored one of these
  float a = -INFINITY;
  if (x > -INFINITY) {
    int at = 0;
#pragma unroll 1
    for (int v = threadIdx.x; v < part.nvec; v += kRcThreads) {
      if (!rc_any_at_least<DT>(part.vec[v], x)) continue;
      const T* e = reinterpret_cast<const T*>(part.vec + v);
#pragma unroll 1
      for (int j = 0; j < VEC; ++j)
        if (elem_as_float<DT>(e[j]) == x) at = v * VEC + j - part.off;
    }
    const float u = r.dense ? __ldg(r.dense + at) : fmaxf(threefry_uniform01(r.k0, r.k1, r.ctr0 + (uint32_t)at), kF32Tiny);
    a = fmaf(x, r.rt, gumbel_screen(u));
    if (!(a == a)) a = -INFINITY;
  }
  {
    const uint32_t xk = f32_key(x), ak = rc_score_key(a);
    const uint32_t xm = rc_max_u32(xk, s, tog), am = rc_max_u32(ak, s, tog);
    const uint32_t xa = rc_max_u32(xk == xm ? ak : 0u, s, tog), ax = rc_max_u32(ak == am ? xk : 0u, s, tog);
    if (threadIdx.x == 0) {
      s.query[0] = key_f32(xm); s.query[1] = key_f32(xa);   // (the queries' place, not used yet)
      s.query[2] = key_f32(ax); s.query[3] = key_f32(am);
    }
    if (rank == 0) {
#pragma unroll 1
      for (int i = threadIdx.x; i < kRcMaxCluster * kRcWideSend; i += kRcThreads) l.all_s[i] = -INFINITY;
    }
  }
  cl_sync();
  TLX_STAMP(p.sp, 2);
  if ((int)threadIdx.x < p.cluster) {
    const uint32_t q = cl_map(s.query, threadIdx.x);
    const float v0 = cl_ld_f32(q), v1 = cl_ld_f32(q + 4), v2 = cl_ld_f32(q + 8), v3 = cl_ld_f32(q + 12);
    s.dom_x[2 * threadIdx.x] = v0; s.dom_s[2 * threadIdx.x] = v1;
    s.dom_x[2 * threadIdx.x + 1] = v2; s.dom_s[2 * threadIdx.x + 1] = v3;
  }
  __syncthreads();
  float xmax = -INFINITY, ms = -INFINITY, bx = -INFINITY, bs = -INFINITY;
#pragma unroll 1
  for (int i = 0; i < 2 * p.cluster; ++i) {
    const float dx = s.dom_x[i], ds = s.dom_s[i];
    if (dx > xmax) { xmax = dx; ms = ds; }
    else if (dx == xmax) ms = fmaxf(ms, ds);
    if (ds > bs || (ds == bs && dx > bx)) { bs = ds; bx = dx; }
  }
  // the same in every CTA: no finite maximum, or no score for it
  const bool lost = !(fabsf(xmax) < INFINITY) || !(fabsf(ms) < INFINITY) || !(fabsf(bs) < INFINITY);
  if (!lost) {
    // [0]: the published element with the best score; [1]: the row's greatest element; the rest: filled below
    if (threadIdx.x < 2) {
      s.cut_x[threadIdx.x] = threadIdx.x == 0 ? bx : xmax;
      s.cut_s[threadIdx.x] = screen_cut(threadIdx.x == 0 ? bs : ms);
    }
    if (threadIdx.x == 0) s.n_cut = 2;
    __syncthreads();
    RcLow low{bx, screen_cut(bs), screen_cut(ms)};
    float above = -INFINITY;
#pragma unroll 1
    for (int attempt = 0;; ++attempt) {
      // from a key the greatest Gumbel term is that of 1 - 2^-23: 15.943
      rc_survivors<DT>(part, low, (low.bs - 15.95f) * T_, r, s, l);
      __syncthreads();
      if (attempt == 0) { TLX_STAMP(p.sp, 10); }
      if (s.n_list <= kRcWideCap || attempt == 4) break;
      // too many (a flat row): the best of those that were kept, the best among the greater ones and the best
      // among those that are greater again dominate nearly all of them, as a rule; where the three lie close together,
      // the next attempt goes on from the last of them
      int cuts = s.n_cut;
#pragma unroll 1
      for (int j = 0; j < 3; ++j) {
        const bool first = attempt == 0 && j == 0;
        uint32_t bk = 0, xk = 0;
#pragma unroll 1
        for (int i = threadIdx.x; i < kRcWideCap; i += kRcThreads) if (first || l.x[i] > above) bk = max(bk, rc_score_key(l.s[i]));
        bk = rc_max_u32(bk, s, tog);
        if (bk == 0) break;
#pragma unroll 1
        for (int i = threadIdx.x; i < kRcWideCap; i += kRcThreads)
          if ((first || l.x[i] > above) && rc_score_key(l.s[i]) == bk) xk = max(xk, f32_key(l.x[i]));
        above = key_f32(rc_max_u32(xk, s, tog));
        const float cut = screen_cut(key_f32(bk));
        if (threadIdx.x == 0) { s.cut_x[cuts] = above; s.cut_s[cuts] = cut; }
        ++cuts;
        if (first && cut > low.bs) { low.bs = cut; low.bx = above; }
      }
      __syncthreads();
      if (threadIdx.x == 0) { s.n_list = 0; s.n_cut = cuts; }
      __syncthreads();
    }
    if (warp_id() == 0) {
      // to the leader: the survivors (those that others dominate are left out if there are many)
      const int lane = lane_id();
      int k = s.n_list;
      if (k > kRcWideCap) k = kRcWideSend + 1;   // given up: rc_slow_row
      else if (k > kRcWideSend) k = rc_thin_out(k, l.x, l.s, l.pos);
      if (lane < k && k <= kRcWideSend) {
        const int i = rank * kRcWideSend + lane;
        cl_st_f32(cl_map(l.all_x + i, 0), l.x[lane]);
        cl_st_f32(cl_map(l.all_s + i, 0), l.s[lane]);
        cl_st_u32(cl_map(l.all_col + i, 0), (uint32_t)(col0 + l.pos[lane]));
      }
      if (lane == 0) cl_st_u32(cl_map(s.sent + rank, 0), (uint32_t)k);
    }
  }
  TLX_STAMP(p.sp, 5);
  cl_sync();
  TLX_STAMP(p.sp, 6);
  if (lost) return -1;
  int tok = -1, most = 0;
  float above = -INFINITY;
  bool first = true, going = true;
  if (rank == 0 && warp_id() == 0) {
    const int lane = lane_id();
    going = !__any_sync(0xFFFFFFFFu, lane < p.cluster && s.sent[lane] > kRcWideSend);
    most = __reduce_max_sync(0xFFFFFFFFu, lane < p.cluster ? s.sent[lane] : 0);
  }
#pragma unroll 1
  for (int round = 0; round < kRcListCap; ++round) {
    if (rank == 0 && warp_id() == 0) {
      // the tokens in question: the best score, and the best score among greater values
      const int lane = lane_id();
      int nq = 0;
      float q[2] = {INFINITY, INFINITY};
#pragma unroll 1
      while (going && nq < 2) {
        const int i = rc_best_sent(most, first, above, l, T_, noise, nrow);
        if (i < 0) { going = false; break; }
        above = l.all_x[i];
        first = false;
        if (lane == 0) s.query_tok[nq] = l.all_col[i];
        if (nq == 0) q[0] = above; else q[1] = above;
        ++nq;
        if (above == xmax) going = false;   // nothing lies above it: kept whatever top_p is
      }
      __syncwarp();
      if (nq > 0 && tok < 0 && q[0] == xmax) { tok = s.query_tok[0]; nq = 0; }
      if (lane < p.cluster) {
        cl_st_f32(cl_map(s.query, lane), q[0]);
        cl_st_f32(cl_map(s.query + 1, lane), q[1]);
        cl_st_u32(cl_map(&s.n_query, lane), (uint32_t)nq);
      }
    }
    if (round == 0) { TLX_STAMP(p.sp, 12); }
    cl_sync();
    const int nq = s.n_query;
    if (nq == 0) break;
    double z = 0.0, unused = 0.0, m0 = 0.0, m1 = 0.0;
    rc_masses<DT>(part, xmax, s.query[0], s.query[1], z, m0, m1);
    rc_sum2_f64(m0, m1, s, tog);
    rc_sum2_f64(z, unused, s, tog);
    if (threadIdx.x == 0) {
      cl_st_f64(cl_map(&s.z[rank], 0), z);
      cl_st_f64(cl_map(&s.msum[rank][0], 0), m0);
      cl_st_f64(cl_map(&s.msum[rank][1], 0), m1);
    }
    if (round == 0) { TLX_STAMP(p.sp, 13); }
    cl_sync();
    if (round == 0) { TLX_STAMP(p.sp, 14); }
    if (rank == 0 && warp_id() == 0) {
      double Z = lane_id() < p.cluster ? s.z[lane_id()] : 0.0;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) Z += shfl_xor_f64(Z, o);
#pragma unroll 1
      for (int j = 0; j < nq && tok < 0; ++j) {
        double mass = lane_id() < p.cluster ? s.msum[lane_id()][j] : 0.0;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) mass += shfl_xor_f64(mass, o);
        if (mass == 0.0 || !(mass / Z >= (double)pp)) tok = s.query_tok[j];
        tok = __shfl_sync(0xFFFFFFFFu, tok, 0);
      }
      if (tok >= 0) going = false;
    }
  }
  if (threadIdx.x == 0) s.pick[0] = tok;
  __syncthreads();
  TLX_STAMP(p.sp, 9);
  return s.pick[0];
}

// One cluster per row.
template <int DT>
__global__ void __launch_bounds__(kRcThreads, 4) sample_cluster_kernel(const __grid_constant__ RcSampleParams p) {
  using T = typename Elem<DT>::type;
  extern __shared__ __align__(128) unsigned char smem[];
  RcShared& s = *reinterpret_cast<RcShared*>(smem);
  const RcLayout l(p.cluster, true);
  const uint32_t rank = cl_rank();
  const int64_t row = blockIdx.x / p.cluster;
  const int64_t n = p.sp.vocab;
  const T* rowp = reinterpret_cast<const T*>(p.sp.logits) + row * p.sp.row_stride;
  const RcPart<DT> part(rowp, n, p.part_len, rank, smem + l.off_part);
  grid_wait();
  part.copy_in();
  TLX_STAMP(p.sp, 0);
  const float T_ = p.sp.temperature[row], pp = p.sp.top_p[row];
  int64_t K = p.sp.top_k[row];
  if (K <= 0 || K > n) K = n;
  if (T_ < kSamplingEps) K = 1;
  const bool resident = p.part_len > 0, wide = resident && n > 1 && (K >= n || K > kRcMaxK);
  if (threadIdx.x == 0) s.n_list = 0;
  part.copy_wait();
  __syncthreads();
  TLX_STAMP(p.sp, 1);
  const int64_t col0 = (int64_t)rank * p.part_len, nrow = row + p.sp.dim0_offset;
  int tok = -1, tog = 0;
  if (resident && !wide) tok = rc_normal_row<DT>(p, part, col0, rank, (int)K, pp, T_, nrow, s, l, smem);
  const bool over = tok == kRcOver;
  if (wide || over) {
    if (K < n) {
      rc_cut_parts<DT>(part.vec, part.off, part.n, part.nvec, (int)K, p.cluster, rank, s, reinterpret_cast<uint32_t*>(smem + l.off_x));
      if (threadIdx.x == 0) s.n_list = 0;   // (read by the other CTAs before the barriers of the cut)
    }
    tok = rc_wide_row<DT>(p, part, col0, rank, pp, T_, nrow, s, l, smem, tog);
  }
  if (rank != 0) return;
  int status = (wide || !resident ? kStatusGeneral : 0) | (over ? kStatusRedone : 0);
  if (tok < 0) {
    tok = rc_slow_row<DT>(rowp, n, K, pp, T_, p.sp.noise, nrow, s);
    status |= resident ? kStatusRedone : 0;
  }
  if (threadIdx.x == 0) {
    p.sp.out_tokens[row] = tok;
    if (p.sp.out_status) p.sp.out_status[row] = status;
  }
}

}  // namespace tlx
