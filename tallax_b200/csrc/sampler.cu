// Fused temperature / top-k / top-p / noise sampler on [rows, vocab] logits, the candidate-level sampler, and the
// merge stage of the vocab-sharded sampler.
//
// Two forms of the fused sampler share this file's parameter block and small helpers:
//   sampler_cluster.cuh  one kernel; a row is resident in the shared memory of a thread-block cluster.  Any alignment,
//                        f32 and bf16, any top-k.
//   sampler_stream.cuh   three chained kernels; rows are cut into parts that persistent CTAs stream.  Large batches of
//                        16-byte aligned bf16 rows, where the clusters' turnover is slower than the stream.
#include <atomic>
#include <cstdlib>
#include <mutex>

#include "sampler_general.cuh"
#include "exchange.cuh"

namespace tlx {

constexpr int kMergeCap = 4096;      // candidates (u64) held in shared memory
constexpr int kWin = 2048;           // bf16 histogram window: 16 binades of 16-bit keys below the maximum

enum StatusBits : int { kStatusGeneral = 1, kStatusTimeout = 2, kStatusRedone = 4 };

constexpr size_t kSharedHeader = (sizeof(SelectShared) + 15) & ~size_t(15);
constexpr size_t kUnionBytes = 32768;  // kMergeCap candidates (u64) == kHistBins f64 mass bins

struct SampleParams {
  const void* logits;
  int64_t rows, vocab, row_stride;
  const int32_t* top_k;
  const float* top_p;
  const float* temperature;
  NoiseSrc noise;
  int64_t dim0_offset;
  int32_t* out_tokens;
  int32_t* out_status;
  long long* timeline; // timeline builds only: 16 global-timer stamps per CTA (see TLX_STAMP)
};

// Timeline builds (python -m tallax_b200.build --timeline, a library of its own) record the global timer
// at marked points of the streaming path's kernels, 16 slots per CTA; other builds compile the marks away.
#ifdef TLX_TIMELINE
__device__ __forceinline__ long long global_timer_ns() {
  long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
#define TLX_STAMP(sp, k)                                                                              \
  do {                                                                                                \
    if (threadIdx.x == 0 && (sp).timeline) (sp).timeline[(size_t)blockIdx.x * 16 + (k)] = global_timer_ns(); \
  } while (0)
#else
#define TLX_STAMP(sp, k) do {} while (0)
#endif

// ---- PTX wrappers ---------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst_smem, const void* src_gmem, uint32_t bytes,
                                          unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst_smem)),
               "l"(src_gmem), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ __nv_bfloat162 bf162_bits(uint32_t w) {
  __nv_bfloat162 r;
  memcpy(&r, &w, sizeof(r));
  return r;
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Block-wide max / min of one u32 per thread: one redux per warp, one shared-memory round.
__device__ __forceinline__ uint32_t block_max_u32(uint32_t v, uint32_t* scratch) {
  v = __reduce_max_sync(0xFFFFFFFFu, v);
  if (lane_id() == 0) scratch[warp_id()] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  uint32_t r = __reduce_max_sync(0xFFFFFFFFu, scratch[lane_id() < nw ? lane_id() : 0]);
  __syncthreads();
  return r;
}
__device__ __forceinline__ uint32_t block_min_u32(uint32_t v, uint32_t* scratch) {
  return ~block_max_u32(~v, scratch);
}

// Number of the `n` listed tokens below `tok`.
static __device__ __noinline__ uint32_t tie_rank(const uint32_t* tie_tok, int n, uint32_t tok) {
  uint32_t rank = 0;
  for (int j = 0; j < n; ++j) rank += tie_tok[j] < tok ? 1u : 0u;
  return rank;
}

// Sampler tail on unsorted bf16 candidates, without sorting them: a histogram over the
// candidates' 16-bit keys gives the top-k boundary (key and admitted ties), the softmax
// denominator and the top-p threshold exactly as in the whole-row path (the mass of a value
// group is count * exp(value - max)); the Gumbel arg-max then runs over the kept candidates.
// Needs the keys to span at most kHistBins values; returns -1 otherwise (caller sorts).
static __device__ __noinline__ int tail_bf16_hist(const SampleParams& p, int64_t row, int K, float pp, float T_, int m,
                                              SelectShared& s, const uint64_t* cand) {
  uint32_t kmx = 0, kmn = 0xFFFFFFFFu;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    const uint32_t k16 = cand_key(cand[i]) >> 16;
    kmx = k16 > kmx ? k16 : kmx;
    kmn = k16 < kmn ? k16 : kmn;
  }
  const int kmax = (int)block_max_u32(kmx, s.scan_u32);
  const int kmin = (int)block_min_u32(kmn, s.scan_u32);
  const int W = kmax - kmin + 1;
  if (W > kHistBins) return -1;
  TLX_STAMP(p, 3);
  uint32_t* win = s.hist;   // win[kmax - key16]
  for (int i = threadIdx.x; i < W; i += blockDim.x) win[i] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < m; i += blockDim.x) atomicAdd(&win[kmax - (int)(cand_key(cand[i]) >> 16)], 1u);
  __syncthreads();
  const float xmax = key16_value(kmax);
  const int per = (W + (int)blockDim.x - 1) / (int)blockDim.x;
  const int i0 = threadIdx.x * per;

  // top-k boundary: first bin (descending key) at which the running count reaches K
  uint32_t local = 0;
  for (int j = 0; j < per; ++j) if (i0 + j < W) local += win[i0 + j];
  uint32_t total;
  const uint32_t incl = block_scan_incl<uint32_t>(local, s.scan_u32, &total, ShflUpU32());
  const uint32_t before = incl - local;
  if (before < (uint32_t)K && incl >= (uint32_t)K) {
    uint32_t run = before;
    for (int j = 0; j < per; ++j) {
      const uint32_t c = win[i0 + j];
      if (run + c >= (uint32_t)K) { s.tmp_i[0] = i0 + j; s.tmp_i[1] = (int)((uint32_t)K - run); s.tmp_i[2] = (int)c; break; }
      run += c;
    }
  }
  __syncthreads();
  const int vk_idx = s.tmp_i[0];
  const uint32_t ties_admitted = (uint32_t)s.tmp_i[1], ties_total = (uint32_t)s.tmp_i[2];
  TLX_STAMP(p, 4);
  // denominator and top-p threshold over the top-k set
  double mass = 0.0;
  for (int j = 0; j < per; ++j) {
    const int idx = i0 + j;
    if (idx < W && idx <= vk_idx) {
      const uint32_t c = idx == vk_idx ? ties_admitted : win[idx];
      if (c) mass += (double)c * (double)expf(key16_value(kmax - idx) - xmax);
    }
  }
  double Z;
  const double mincl = block_scan_incl<double>(mass, s.scan_f64, &Z, ShflUpF64());
  const double target = (double)pp * Z;
  if (threadIdx.x == 0) s.tmp_i[3] = vk_idx;   // default: keep the whole top-k set
  __syncthreads();
  if (mincl - mass < target && mincl >= target) {
    double run = mincl - mass;
    for (int j = 0; j < per; ++j) {
      const int idx = i0 + j;
      if (idx < W && idx <= vk_idx) {
        const uint32_t c = idx == vk_idx ? ties_admitted : win[idx];
        if (c) {
          run += (double)c * (double)expf(key16_value(kmax - idx) - xmax);
          if (run >= target) { s.tmp_i[3] = idx; break; }
        }
      }
    }
  }
  __syncthreads();
  const int vstar_idx = s.tmp_i[3];
  const bool cut_ties = vstar_idx == vk_idx && ties_admitted < ties_total;
  __syncthreads();
  TLX_STAMP(p, 5);
  // the lowest tokens of the boundary group are the admitted ones: list the group's tokens
  uint32_t* tie_tok = s.hist;   // the histogram is no longer needed
  if (cut_ties) {
    if (threadIdx.x == 0) s.fill = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
      const uint64_t c = cand[i];
      if (kmax - (int)(cand_key(c) >> 16) == vk_idx) tie_tok[atomicAdd(&s.fill, 1)] = cand_low(c);
    }
    __syncthreads();
  }
  const int n_ties = cut_ties ? s.fill : 0;
  // Gumbel arg-max over the kept candidates, screened in f32 (see final_argmax)
  const int64_t nrow = row + p.dim0_offset;
  float a1 = -INFINITY, a2 = -INFINITY, q1 = 0.f, u1 = 0.5f;
  int c1 = 0x7FFFFFFF;
  auto kept = [&](uint64_t c) {
    const int idx = kmax - (int)(cand_key(c) >> 16);
    if (idx > vstar_idx) return false;
    if (idx < vk_idx || !cut_ties) return true;
    // idx == vk_idx: admitted if fewer than ties_admitted group members have a lower token
    return tie_rank(tie_tok, n_ties, cand_low(c)) < ties_admitted;
  };
  {
    // decide which of the thread's candidates are kept and start their noise loads, four at a time
    constexpr int kBatch = 4;
#pragma unroll 1
    for (int i0b = threadIdx.x; i0b < m; i0b += kBatch * (int)blockDim.x) {
      uint32_t keep_mask = 0;
      float uu[kBatch];
      uint64_t cc[kBatch];
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const int i = i0b + j * (int)blockDim.x;
        uu[j] = 0.5f;
        cc[j] = 0;
        if (i < m) {
          cc[j] = cand[i];
          if (kept(cc[j])) { keep_mask |= 1u << j; uu[j] = p.noise.at(nrow, (int64_t)cand_low(cc[j])); }
        }
      }
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        if (keep_mask & (1u << j)) {
          const float q = __fdiv_rn(key_f32(cand_key(cc[j])), T_);
          const float a = q + gumbel_screen(uu[j]);
          if (a > a1) { a2 = a1; a1 = a; q1 = q; u1 = uu[j]; c1 = (int)cand_low(cc[j]); }
          else if (a > a2) a2 = a;
        }
      }
    }
  }
  TLX_STAMP(p, 6);
  const Best top = block_best(Best{a1, c1}, s);
  const float cut = screen_cut(top.y);
  const int leaders = __syncthreads_count(a1 >= cut);
  const int crowded = __syncthreads_or(a2 >= cut);
  TLX_STAMP(p, 7);
  // nothing else comes within the slack of the best screened score: it is the winner as it stands
  if (leaders == 1 && !crowded) return top.tok;
  Best best{-INFINITY, 0x7FFFFFFF};
  if (!crowded) {
    if (a1 >= cut) best = Best{q1 + gumbel_exact(u1), c1};
  } else {
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
      const uint64_t c = cand[i];
      if (kept(c)) {
        const float u = p.noise.at(nrow, (int64_t)cand_low(c));
        const float q = __fdiv_rn(key_f32(cand_key(c)), T_);
        if (q + gumbel_screen(u) >= cut) best = best_of(best, Best{q + gumbel_exact(u), (int)cand_low(c)});
      }
    }
  }
  const int result = block_best(best, s).tok;
  return result;
}

}  // namespace tlx
#include "sampler_stream.cuh"
#include "sampler_cluster.cuh"
namespace tlx {

// ---- the kernels --------------------------------------------------------------------------
template <int DT>
__global__ void __launch_bounds__(256) top_p_and_sample_kernel(const typename Elem<DT>::type* __restrict__ logits,
                                                               const int32_t* __restrict__ idx, int k,
                                                               const float* __restrict__ top_p,
                                                               const float* __restrict__ temperature, NoiseSrc noise,
                                                               typename Elem<DT>::type replace, int64_t dim0_offset,
                                                               int32_t* __restrict__ out) {
  using T = typename Elem<DT>::type;
  __shared__ SelectShared s;
  const int64_t r = blockIdx.x;
  const T* x = logits + r * k;
  const int32_t* id = idx + r * k;
  const float T_ = temperature[r];
  if (T_ < kSamplingEps) {
    if (threadIdx.x == 0) out[r] = id[0];
    return;
  }
  // the top-k set is the prefix of entries that were not overwritten with the replace value
  uint32_t valid = 0;
  const float rep = elem_as_float<DT>(replace);
  for (int i = threadIdx.x; i < k; i += blockDim.x) valid += (elem_as_float<DT>(x[i]) != rep) ? 1u : 0u;
  uint32_t nv;
  block_scan_incl<uint32_t>(valid, s.scan_u32, &nv, ShflUpU32());
  const int K = nv ? (int)nv : 1;
  const int64_t nrow = r + dim0_offset;
  const int tok = sample_tail<4>(
      K, top_p[r], T_, s, [&](int i) { return elem_as_float<DT>(x[i]); }, [&](int i) { return (int)id[i]; },
      [&](int i) { return noise.at(nrow, (int64_t)id[i]); });
  if (threadIdx.x == 0) out[r] = tok;
}

// ---------------------------------------------------------------------------------
// merge stage of the vocab-sharded sampler
// ---------------------------------------------------------------------------------
constexpr int kMergeThreads = 512;
constexpr int kMergeMaxCand = 8192;

struct MergeParams {
  const float* cand_vals;
  const int32_t* cand_idx;
  const float* cand_noise;
  int n_cand, k_per_block;
  int64_t block_stride, row_stride;
  const int32_t* top_k;
  const float* top_p;
  const float* temperature;
  int32_t* out;
  // exchange mode (xbuf non-null): the candidates are read from this rank's exchange buffer, set by set
  unsigned char* xbuf;
  size_t off_flags[2], off_cand[2];
  int world;
  int64_t rows;
  int32_t* status;
};

__device__ __forceinline__ uint32_t ld_acquire_sys_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long exchange_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Number of entries of the ascending list blk[0..len) whose high word is smaller than `target`.  The high
// word is the inverted key; it never reaches 0xFFFFFFFF (no key is 0), so target may be a high word plus one.
__device__ __forceinline__ int count_high_below(const uint64_t* blk, int len, uint32_t target) {
  const uint32_t* hi = reinterpret_cast<const uint32_t*>(blk) + 1;
  int lo = 0;
  while (len > 0) {
    const int half = len >> 1;
    if (hi[2 * (lo + half)] < target) { lo += half + 1; len -= half + 1; }
    else len = half;
  }
  return lo;
}

// One CTA per row.  The shards' blocks arrive sorted (value desc, token asc), which the kernel checks: a
// candidate's place in the merged order is then its place in its own block plus, for every other block,
// the number of entries that precede it there (a binary search), and only places below K are filled; one
// comparison per block rules most candidates out before any search.
// Unsorted blocks take the bitonic network over all candidates instead.
__global__ void __launch_bounds__(kMergeThreads) merge_and_sample_kernel(MergeParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SelectShared& s = *reinterpret_cast<SelectShared*>(smem_raw);
  uint64_t* cand = reinterpret_cast<uint64_t*>(smem_raw + ((sizeof(SelectShared) + 15) & ~size_t(15)));
  const int n_cand = p.n_cand, kpb = p.k_per_block;
  int P = 2;
  while (P < n_cand) P <<= 1;
  uint64_t* merged = cand + P;
  const int64_t r = blockIdx.x;
  // (there before the candidates are; from L2: this kernel has not waited for anything yet)
  const float T_ = __ldcg(p.temperature + r), pp = __ldcg(p.top_p + r);
  int K = __ldcg(p.top_k + r);
  if (K <= 0 || K > n_cand) K = n_cand;

  const float* v = p.cand_vals;
  const int32_t* id = p.cand_idx;
  const float* un = p.cand_noise;
  ExchangeHeader* xh = reinterpret_cast<ExchangeHeader*>(p.xbuf);
  uint32_t* flag = nullptr;
  if (xh) {
    const uint32_t par = *reinterpret_cast<volatile const uint32_t*>(&xh->step) & 1u;
    const size_t plane = (size_t)p.rows * kpb;
    v = reinterpret_cast<const float*>(p.xbuf + p.off_cand[par]);
    id = reinterpret_cast<const int32_t*>(v) + plane;
    un = v + 2 * plane;
    flag = reinterpret_cast<uint32_t*>(p.xbuf + p.off_flags[par]) + r;
    // a call whose extents are not the buffer's reads nothing: token -1, status 2
    if (xh->rows != (uint32_t)p.rows || xh->k_cand != (uint32_t)kpb || xh->world != (uint32_t)p.world) {
      if (threadIdx.x == 0) {
        atomicExch(&xh->error, 2u);
        if (p.status) atomicExch(p.status, 2);
        p.out[r] = -1;
      }
      if (blockIdx.x == gridDim.x - 1) grid_wait();
      return;
    }
    if (threadIdx.x == 0) {
      // every rank's block of this row has arrived when the word reads `world`; two seconds at most
      const unsigned long long t0 = exchange_timer_ns();
      bool ok = false;
      for (int it = 0; it < (1 << 24); ++it) {
        if (ld_acquire_sys_u32(flag) >= (uint32_t)p.world) { ok = true; break; }
        if (exchange_timer_ns() - t0 > 2000000000ull) break;
        __nanosleep(100);
      }
      if (!ok) {
        atomicExch(&xh->error, 1u);
        if (p.status) atomicExch(p.status, 1);
      }
    }
    __syncthreads();
  }
  v += r * p.row_stride;
  id += r * p.row_stride;
  un += r * p.row_stride;
  // block of candidate i without an integer division: (i + 0.5) / kpb is at least 0.5 / kpb away from an
  // integer and i < 8192, far more than the product's rounding error
  const float inv_kpb = 1.0f / (float)kpb;
  auto block_of = [&](uint32_t i) { return (int)(((float)i + 0.5f) * inv_kpb); };
  auto at = [&](uint32_t i) {
    const int b = block_of(i);
    return (int64_t)b * p.block_stride + (int64_t)((int)i - b * kpb);
  };
  // low word = position in the gathered list: shards are laid side by side in ascending
  // token order, so position order equals token order among equal values
  int unsorted = 0;
  for (int i = threadIdx.x; i < n_cand; i += blockDim.x) {
    const float x = xh ? __ldcg(v + at(i)) : v[at(i)];
    cand[i] = cand_make(f32_key(x), (uint32_t)i);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n_cand; i += blockDim.x)
    if (i != block_of(i) * kpb && cand[i - 1] > cand[i]) unsorted = 1;
  unsorted = __syncthreads_or(unsorted);
  const uint64_t* top = cand;
  if (unsorted) {
    sort_candidates(cand, n_cand);
  } else if (n_cand > kpb) {
    // Step 1, every candidate: q entries of its own block precede it; if entry K-1-q of another block does
    // too, so do that block's first K-q entries and its place is K or more.  The others (K and a few more
    // per block) are listed.  Step 2, one listed candidate per thread: a binary search per other block.
    const int blocks = n_cand / kpb;
    uint32_t* listed = reinterpret_cast<uint32_t*>(merged + n_cand);
    if (threadIdx.x == 0) s.fill = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n_cand; i += blockDim.x) {
      const int b = block_of(i);
      const int q = i - b * kpb;
      if (q >= K) continue;
      const uint64_t c = cand[i];
      const int probe = K - 1 - q;
      bool out = false;
      if (probe < kpb)
        for (int o = 0; o < blocks && !out; ++o) out = o != b && cand[o * kpb + probe] < c;
      if (!out) {
        // the same with the places shared out evenly: if entry d-1 of EVERY other block precedes it, with
        // d * (blocks - 1) >= K - q, its place is K or more as well
        const int d = (K - q + blocks - 2) / (blocks - 1);
        if (d - 1 < kpb) {
          bool all = true;
          for (int o = 0; o < blocks && all; ++o) all = o == b || cand[o * kpb + d - 1] < c;
          out = all;
        }
      }
      if (!out) listed[atomicAdd(&s.fill, 1)] = (uint32_t)i;
    }
    __syncthreads();
    const int nlisted = s.fill;
    for (int l = threadIdx.x; l < nlisted; l += blockDim.x) {
      const int i = (int)listed[l];
      const int b = block_of(i);
      const int q = i - b * kpb;
      const uint64_t c = cand[i];
      int place = q;
      const int span = min(kpb, K - q);   // a block's entries from `span` on cannot change the verdict
      // entries of another block that precede c: a smaller high word (the inverted key), or an equal one in a
      // block before c's own (positions, the low words, grow with the block) -- a search on the high words
      const uint32_t chi = (uint32_t)(c >> 32);
      for (int o = 0; o < blocks && place < K; ++o)
        if (o != b) place += count_high_below(cand + o * kpb, span, chi + (o < b ? 1u : 0u));
      if (place < K) merged[place] = c;
    }
    __syncthreads();
    top = merged;
  }
  int tok = 0;
  const auto value_of = [&](int i) { return key_f32(cand_key(top[i])); };
  const auto token_of = [&](int i) { return (int)id[at(cand_low(top[i]))]; };
  const auto noise_of = [&](int i) { return un[at(cand_low(top[i]))]; };
  if (T_ < kSamplingEps) tok = token_of(0);
  else if (K > 128) tok = sample_tail<2>(K, pp, T_, s, value_of, token_of, noise_of);
  else if (warp_id() == 0) tok = sample_tail_warp<4>(K, pp, T_, value_of, token_of, noise_of);
  if (threadIdx.x == 0) {
    p.out[r] = tok;
    if (xh) {
      // the row is consumed: clear its arrival word; the last row's CTA of the step advances the step
      *reinterpret_cast<volatile uint32_t*>(flag) = 0u;
      __threadfence();
      if (atomicAdd(&xh->done, 1u) == gridDim.x - 1) {
        *reinterpret_cast<volatile uint32_t*>(&xh->done) = 0u;
        __threadfence();
        atomicAdd(&xh->step, 1u);
      }
    }
  }
  // (exchange mode: this kernel is not complete before the candidate kernel is, for what follows on the stream)
  if (xh && blockIdx.x == gridDim.x - 1) grid_wait();
}

// ---------------------------------------------------------------------------------
// top-p mask on the reference's (k, B) layout: column b holds row b's candidates,
// sorted descending along axis 0.  Literal semantics, including the quirk that a
// threshold index equal to k reads as 0.0.
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) top_p_mask_kernel(const float* __restrict__ x, const float* __restrict__ p,
                                                         int k, int64_t B, float replace, float* __restrict__ out) {
  __shared__ double scan_f64[40];
  __shared__ uint32_t scan_u32[40];
  constexpr int kMaxItems = 8;
  const int64_t b = blockIdx.x;
  const int per = (k + blockDim.x - 1) / blockDim.x;
  const int i0 = threadIdx.x * per;
  const float x0 = x[b];
  double run[kMaxItems];
  float xv[kMaxItems];
  double acc = 0.0;
#pragma unroll
  for (int j = 0; j < kMaxItems; ++j) {
    const int i = i0 + j;
    if (j < per && i < k) {
      xv[j] = x[(int64_t)i * B + b];
      acc += (double)expf(xv[j] - x0);
      run[j] = acc;
    }
  }
  double Z;
  const double base = block_scan_incl<double>(acc, scan_f64, &Z, ShflUpF64()) - acc;
  uint32_t below = 0;
  const double pd = (double)p[b];
#pragma unroll
  for (int j = 0; j < kMaxItems; ++j) {
    const int i = i0 + j;
    if (j < per && i < k) below += ((base + run[j]) / Z < pd) ? 1u : 0u;
  }
  uint32_t t;
  block_scan_incl<uint32_t>(below, scan_u32, &t, ShflUpU32());
  const float thr = ((int)t < k) ? x[(int64_t)t * B + b] : 0.0f;
#pragma unroll
  for (int j = 0; j < kMaxItems; ++j) {
    const int i = i0 + j;
    if (j < per && i < k) out[(int64_t)i * B + b] = (xv[j] >= thr) ? xv[j] : replace;
  }
}

// ---------------------------------------------------------------------------------
// Gumbel arg-max with noise indexed by (idx0, idx1): position of the winner along `axis`
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) gumbel_argmax_kernel(const float* __restrict__ logits,
                                                            const int32_t* __restrict__ idx0,
                                                            const int32_t* __restrict__ idx1, int64_t rows,
                                                            int64_t cols, uint32_t k0, uint32_t k1,
                                                            const uint32_t* __restrict__ key_dev, int64_t dim1,
                                                            int axis, int32_t* __restrict__ out) {
  __shared__ float sy[8];
  __shared__ int sp[8];
  if (key_dev) { k0 = __ldg(key_dev); k1 = __ldg(key_dev + 1); }
  const int64_t line = blockIdx.x;                    // row (axis 1) or column (axis 0)
  const int64_t len = axis == 1 ? cols : rows;
  const int64_t step = axis == 1 ? 1 : cols;
  const int64_t start = axis == 1 ? line * cols : line;
  Best best{-INFINITY, 0x7FFFFFFF};
  for (int64_t i = threadIdx.x; i < len; i += blockDim.x) {
    const int64_t e = start + i * step;
    const float f = threefry_uniform01(k0, k1, (uint32_t)((int64_t)idx0[e] * dim1 + (int64_t)idx1[e]));
    const float u = fmaxf(f, kF32Tiny);
    const float l = logits[e];
    const float a = l + gumbel_screen(u);
    if (a >= best.y - (kGumbelSlack + 1e-5f * fabsf(best.y)) || best.y == -INFINITY)
      best = best_of(best, Best{l + gumbel_exact(u), (int)i});
  }
  best = warp_best(best);
  if (lane_id() == 0) { sy[warp_id()] = best.y; sp[warp_id()] = best.tok; }
  __syncthreads();
  if (threadIdx.x == 0) {
    Best b{-INFINITY, 0x7FFFFFFF};
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) b = best_of(b, Best{sy[w], sp[w]});
    out[line] = b.tok != 0x7FFFFFFF ? b.tok : 0;   // nothing has a score: the line's first position
  }
}

static int device_sm_count() {
  static int cached[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

// ---- streaming path (sampler_stream.cuh): workspace layout and launches ---------------------------
struct StreamLayout {
  int P, part_chunks, nchunks, nfin;
  size_t off_desc, off_counts, off_lump, off_wbest, off_flag, off_rowdone, off_state, off_records, off_hist, off_cands, off_timeline = 0, bytes;
};
static size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
static StreamLayout stream_layout(int64_t rows, int64_t vocab) {
  StreamLayout l;
  l.nchunks = (int)((vocab * 2 + kStChunk - 1) / kStChunk);
  l.part_chunks = (l.nchunks + kStMaxParts - 1) / kStMaxParts;
  if (l.part_chunks < 2) l.part_chunks = 2;
  l.P = (l.nchunks + l.part_chunks - 1) / l.part_chunks;
  l.nfin = (int)((vocab * 2 + kFinChunk - 1) / kFinChunk);
  size_t o = 256;   // [0]: error flag, [1]: item counter
  l.off_desc = o;    o = align256(o + (size_t)rows * sizeof(StreamDesc));
  l.off_counts = o;  o = align256(o + (size_t)rows * l.P * kStWarps * sizeof(int));
  l.off_lump = o;    o = align256(o + (size_t)rows * l.P * sizeof(double));
  l.off_wbest = o;   o = align256(o + (size_t)rows * sizeof(unsigned long long));
  l.off_flag = o;    o = align256(o + (size_t)rows * sizeof(int));
  l.off_rowdone = o; o = align256(o + (size_t)rows * sizeof(int));
  l.off_state = o;   o = align256(o + (size_t)rows * sizeof(WideState));
  l.off_records = o; o = align256(o + (size_t)rows * l.nfin * sizeof(FinRecord));
  l.off_hist = o;    o = align256(o + (size_t)rows * kStWin * sizeof(uint32_t));
  l.off_cands = o;   o = align256(o + (size_t)rows * l.P * kStWarps * kStWarpCap * sizeof(uint32_t));
#ifdef TLX_TIMELINE
  l.off_timeline = o; o = align256(o + (size_t)4 * 8192 * 16 * sizeof(long long));
#endif
  l.bytes = o;
  return l;
}
// bf16 rows that bulk copies can address, long enough for the prologue's sample, few enough for the
// kernels' per-row tables in shared memory, short enough for 16 parts of at most ten chunks
static bool stream_path_serves(int dtype, int64_t rows, int64_t vocab, int64_t row_stride, const void* logits) {
  if (dtype != TLX_BF16 || vocab < kStMinVocab || rows > kStMaxRows) return false;
  if ((reinterpret_cast<uintptr_t>(logits) & 15) != 0 || ((row_stride * 2) & 15) != 0 || ((vocab * 2) & 15) != 0) return false;
  return stream_layout(rows, vocab).part_chunks <= kStMaxPartChunks;
}

// Whether it is the faster one for a call that both forms serve.  The clusters' time grows with the bytes (four CTAs an SM
// take turns of about 10 us); the stream starts from the 20 to 25 us of its three kernels and then moves more bytes per second.
// Where they meet depends on the parameters, which the host does not know.  us stream / cluster, requests with mixed
// parameters, with one usual top_k and without top-k:
//                      a noise tensor                     a key
//   [32, 128256]   28/23  16/12  33/30            30/23  17/12  36/29
//   [48, 151936]   30/28  21/14  38/39            33/28  22/14  40/40
//   [64, 128256]   31/29  22/15  39/36            33/28  21/15  41/38
//   [256, 32000]   33/39  34/25  41/38            34/38  28/23  44/40
//   [72, 128256]   32/32  23/21  45/40            35/29  22/20  48/40
//   [80, 128256]   33/35  23/22  46/40            37/32  25/21  50/42
// Up to 16 MB the cluster form saves more on the one usual setting than it loses on mixed ones; beyond, it runs in several waves.
// One line for both kinds of noise.  With a key it lies low for long rows (the last two lines: 9 to 17 % would be gained up to there at least)
// and right for many short ones; the workspace is sized for the stream from 16 MB on in either case.
static bool stream_path_wanted(int64_t rows, int64_t vocab) { return rows * vocab * 2 > (16ll << 20); }

// Diagnostic switch for timing the stages of the streaming path one by one (environment variable
// TLX_SAMPLE_STAGES = 1..3: launch only the first n kernels; +16: the stream kernel only takes the
// chunks, the streaming floor; +32 / +64: the final pass without its scoring / without its records).
// Unset in normal use: all three kernels run.
static int debug_stages() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("TLX_SAMPLE_STAGES");
    v = e ? atoi(e) : 3;
    if (v <= 0) v = 3;
  }
  return v;
}

// ---- cluster path (sampler_cluster.cuh) -----------------------------------------------------------------------
template <int DT>
static int launch_cluster_path(cudaStream_t st, const SampleParams& sp) {
  const int es = (int)sizeof(typename Elem<DT>::type);
  RcSampleParams p{};
  p.sp = sp;
  p.cluster = rc_cluster_size(sp.rows, sp.vocab, es);
  p.part_len = rc_part_len(sp.vocab, p.cluster, es);
  if (p.part_len > kRcMaxPart) { p.cluster = 1; p.part_len = 0; }   // longer than a cluster holds: rc_slow_row
  size_t part_bytes = (size_t)p.part_len * es + 32;
  if (part_bytes < kRcMinPartBytes) part_bytes = kRcMinPartBytes;
  const size_t smem = RcLayout(p.cluster, true).off_part + part_bytes;
  static SmemLimit limit;
  int rc;
  if ((rc = raise_smem(limit, (const void*)sample_cluster_kernel<DT>, smem, "sample")) != TLX_OK) return rc;
  {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 0 || dev >= 64 || !done[dev]) {
      cudaError_t e = cudaFuncSetAttribute((const void*)sample_cluster_kernel<DT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e == cudaSuccess) e = cudaFuncSetAttribute((const void*)sample_cluster_kernel<DT>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
      if (e != cudaSuccess) return set_error(TLX_ERR_CUDA, "sample: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      if (dev >= 0 && dev < 64) done[dev] = true;
    }
  }
  return launch_dependent(sample_cluster_kernel<DT>, {(unsigned)(sp.rows * p.cluster), kRcThreads, smem, p.cluster}, st, "sample", p);
}

static int launch_stream_path(cudaStream_t st, const SampleParams& sp, void* workspace) {
  const StreamLayout l = stream_layout(sp.rows, sp.vocab);
  const int stages = debug_stages() & 15;
  unsigned char* ws = (unsigned char*)workspace;
  const int sms = device_sm_count();
  StreamParams p{};
  p.sp = sp;
  p.P = l.P; p.part_chunks = l.part_chunks; p.nchunks = l.nchunks; p.nfin = l.nfin; p.row_bytes = sp.vocab * 2;
  // the noise tensor can be streamed next to the logits if its rows start on 16-byte boundaries
  const bool dense = sp.noise.dense && (reinterpret_cast<uintptr_t>(sp.noise.dense) & 15) == 0 && (sp.noise.stride & 3) == 0;
  // Wide rows' arg-max over their kept elements: the stream kernel does it (final items, one record each), but
  // for a noise tensor that cannot be streamed, for which the finish kernel makes a final pass with the CTAs that three per SM leave
  // beside one per row.  (With noise from a key it made that pass too, after the whole stream kernel: bf16 [256, 151936] mixed
  // parameters 63 us, [256, 128256] without top-k 149; as final items 48 and 95.)
  const int64_t fin_elems = sp.noise.dense ? StFinal<false>::kElems : StFinal<true>::kElems;
  const bool final_in_stream = dense || !sp.noise.dense;
  p.fin_items = final_in_stream ? (int)((sp.vocab + fin_elems - 1) / fin_elems) : 0;
  p.fin_ctas = final_in_stream ? 0 : (3 * sms - (int)sp.rows < sms ? sms : 3 * sms - (int)sp.rows);
  p.error_flag = (int*)ws;
  p.item_counter = (int*)ws + 1;
  p.row_signals = (int*)ws + 2;
  p.unit_counter = (int*)ws + 3;
  p.desc = (StreamDesc*)(ws + l.off_desc);
  p.counts = (int*)(ws + l.off_counts);
  p.wlump = (double*)(ws + l.off_lump);
  p.wbest = (unsigned long long*)(ws + l.off_wbest);
  p.wflag = (int*)(ws + l.off_flag);
  p.rowdone = (int*)(ws + l.off_rowdone);
  p.wstate = (WideState*)(ws + l.off_state);
  p.records = (FinRecord*)(ws + l.off_records);
  p.whist = (uint32_t*)(ws + l.off_hist);
  p.cands = (uint32_t*)(ws + l.off_cands);
  p.debug = (debug_stages() >> 4) & 31;
  const int64_t items = sp.rows * (int64_t)l.P;
  const size_t st_smem = kStFixedSmem + (size_t)sp.rows * 6;   // descriptor word and order entry per row
  const size_t fin_smem = kStFinishFixedSmem + (size_t)sp.rows * sizeof(int);
  static SmemLimit stream_limits[2], finish_limits[2];
  int rc;
  const bool from_key = !sp.noise.dense;
  const auto stream = from_key ? sample_stream_kernel<true> : sample_stream_kernel<false>;
  if ((rc = raise_smem(stream_limits[from_key], (const void*)stream, st_smem, "sample")) != TLX_OK) return rc;
  const auto finish = p.fin_ctas > 0 ? sample_finish_kernel<true> : sample_finish_kernel<false>;
  if ((rc = raise_smem(finish_limits[p.fin_ctas > 0], (const void*)finish, fin_smem, "sample")) != TLX_OK) return rc;
  // An SM changes its split between L1 and shared memory only while idle: the three kernels ask for the same
  // split, so that each one's CTAs can move in beside those of the one before.
  {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 0 && dev < 64 && !done[dev]) {
      cudaFuncSetAttribute((const void*)sample_prologue_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
      cudaFuncSetAttribute((const void*)sample_stream_kernel<true>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
      cudaFuncSetAttribute((const void*)sample_stream_kernel<false>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
      cudaFuncSetAttribute((const void*)sample_finish_kernel<true>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
      cudaFuncSetAttribute((const void*)sample_finish_kernel<false>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
      done[dev] = true;
    }
  }
#ifdef TLX_TIMELINE
  long long* tl = (long long*)(ws + l.off_timeline);
  p.sp.timeline = tl;
#define TLX_TIMELINE_KERNEL(k) p.sp.timeline = tl + (size_t)(k) * 8192 * 16
#else
#define TLX_TIMELINE_KERNEL(k) do {} while (0)
#endif
  if ((rc = launch_dependent(sample_prologue_kernel, {(unsigned)sp.rows, kStProThreads}, st, "sample (prologue)", p)) != TLX_OK) return rc;
  if (stages < 2) return TLX_OK;
  const int64_t sgrid = items < 4ll * sms ? items : 4ll * sms;
  TLX_TIMELINE_KERNEL(1);
  if ((rc = launch_dependent(stream, {(unsigned)sgrid, kStThreads, st_smem}, st, "sample (stream)", p)) != TLX_OK) return rc;
  if (stages < 3) return TLX_OK;
  TLX_TIMELINE_KERNEL(2);
  return launch_dependent(finish, {(unsigned)(p.fin_ctas + sp.rows), kStThreads, fin_smem}, st, "sample (finish)", p);
}

}  // namespace tlx

using namespace tlx;

extern "C" {

size_t tlx_sample_workspace_bytes(int64_t rows, int64_t vocab) {
  if (rows <= 0 || vocab <= 0) return 0;
  return stream_path_wanted(rows, vocab) ? stream_layout(rows, vocab).bytes : 256;
}

// Key and row offset of a call: host values or device operands (see NoiseSrc).
struct CallOperands {
  uint32_t key0 = 0, key1 = 0;
  int64_t dim0_offset = 0;
  const uint32_t* key_dev = nullptr;
  const int32_t* dim0_offset_dev = nullptr;
};

static int sample_impl(void* stream, const void* logits, int dtype, int64_t rows, int64_t vocab, int64_t row_stride,
                       const int32_t* top_k, const float* top_p, const float* temperature, const float* noise,
                       int64_t noise_stride, const CallOperands& op, int32_t* out_tokens, int32_t* out_status,
                       void* workspace, size_t workspace_bytes) {
  cudaStream_t st = (cudaStream_t)stream;
  const uint32_t key0 = op.key0, key1 = op.key1;
  const int64_t dim0_offset = op.dim0_offset;
  TLX_CHECK_ARG(rows >= 0 && vocab >= 1, "sample: bad extent");
  TLX_CHECK_ARG(vocab < (1ll << 31) && rows < (1ll << 31), "sample: extent too large");
  TLX_CHECK_ARG(row_stride >= vocab, "sample: row stride smaller than the row");
  if (dtype != TLX_F32 && dtype != TLX_BF16)
    return set_error(TLX_ERR_UNSUPPORTED, "sample: logits dtype %d not supported (f32, bf16)", dtype);
  if (rows == 0) return TLX_OK;
  TLX_CHECK_ARG(logits && top_k && top_p && temperature && out_tokens, "sample: null pointer");
  TLX_CHECK_ARG(!noise || noise_stride >= vocab, "sample: noise stride smaller than the row");
  SampleParams p{};
  p.logits = logits; p.rows = rows; p.vocab = vocab; p.row_stride = row_stride;
  p.top_k = top_k; p.top_p = top_p; p.temperature = temperature;
  p.noise.dense = noise; p.noise.stride = noise_stride; p.noise.k0 = key0; p.noise.k1 = key1; p.noise.vocab = vocab;
  p.noise.key_dev = op.key_dev; p.noise.row_offset_dev = op.dim0_offset_dev;
  p.dim0_offset = dim0_offset; p.out_tokens = out_tokens; p.out_status = out_status;
  if (stream_path_serves(dtype, rows, vocab, row_stride, logits) && stream_path_wanted(rows, vocab) &&
      workspace && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0 && workspace_bytes >= stream_layout(rows, vocab).bytes)
    return launch_stream_path(st, p, workspace);
#ifdef TLX_TIMELINE
  // timeline builds: the caller's workspace receives the stamps, if it is large enough
  if (workspace && workspace_bytes >= (size_t)rows * kRcMaxCluster * 128) p.timeline = (long long*)workspace;
#endif
  return dtype == TLX_BF16 ? launch_cluster_path<TLX_BF16>(st, p) : launch_cluster_path<TLX_F32>(st, p);
}

int tlx_debug_check_status(int32_t* out4) {
#ifdef TLX_CHECKED
  int32_t w[4] = {0, 0, 0, 0};
  if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpyFromSymbol(w, g_tlx_check_word, sizeof(w)) != cudaSuccess)
    return set_error(TLX_ERR_CUDA, "debug_check_status: could not read the check word");
  const int32_t zero[4] = {0, 0, 0, 0};
  cudaMemcpyToSymbol(g_tlx_check_word, zero, sizeof(zero));
  if (out4) for (int i = 0; i < 4; ++i) out4[i] = w[i];
  return w[0] ? 1 : 0;
#else
  if (out4) for (int i = 0; i < 4; ++i) out4[i] = 0;
  return set_error(TLX_ERR_UNSUPPORTED, "debug_check_status: not a checked build (python -m tallax_b200.build --checked)");
#endif
}

int tlx_init(int device, unsigned flags) {
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count)
    return set_error(TLX_ERR_INVALID, "init: no CUDA device %d", device);
  int prev = 0;
  cudaGetDevice(&prev);
  if (cudaSetDevice(device) != cudaSuccess) return set_error(TLX_ERR_CUDA, "init: cudaSetDevice(%d) failed", device);
  device_sm_count();
  int rc = TLX_OK;
  (void)flags;   // TLX_INIT_SIDE_STREAM: accepted; no path forks a stream any more
  cudaSetDevice(prev);
  return rc;
}

int tlx_sample(void* stream, const void* logits, int dtype, int64_t rows, int64_t vocab, int64_t row_stride,
               const int32_t* top_k, const float* top_p, const float* temperature, const float* noise,
               int64_t noise_stride, uint32_t key0, uint32_t key1, int64_t dim0_offset, int32_t* out_tokens,
               int32_t* out_status, void* workspace, size_t workspace_bytes) {
  CallOperands op;
  op.key0 = key0; op.key1 = key1; op.dim0_offset = dim0_offset;
  return sample_impl(stream, logits, dtype, rows, vocab, row_stride, top_k, top_p, temperature, noise, noise_stride, op,
                     out_tokens, out_status, workspace, workspace_bytes);
}

int tlx_sample_dev(void* stream, const void* logits, int dtype, int64_t rows, int64_t vocab, int64_t row_stride,
                   const int32_t* top_k, const float* top_p, const float* temperature, const float* noise,
                   int64_t noise_stride, const uint32_t* key_dev, const int32_t* dim0_offset_dev, int32_t* out_tokens,
                   int32_t* out_status, void* workspace, size_t workspace_bytes) {
  if (!noise && !key_dev) return set_error(TLX_ERR_INVALID, "sample: neither noise nor a key given");
  CallOperands op;
  op.key_dev = key_dev; op.dim0_offset_dev = dim0_offset_dev;
  return sample_impl(stream, logits, dtype, rows, vocab, row_stride, top_k, top_p, temperature, noise, noise_stride, op,
                     out_tokens, out_status, workspace, workspace_bytes);
}

static int top_p_and_sample_impl(void* stream, const void* topk_logits, int dtype, const int32_t* topk_idx, int64_t rows,
                                 int k, const float* top_p, const float* temperature, const float* noise,
                                 int64_t noise_stride, const CallOperands& op, int64_t vocab_size, double replace_val,
                                 int32_t* out_tokens) {
  const uint32_t key0 = op.key0, key1 = op.key1;
  const int64_t dim0_offset = op.dim0_offset;
  cudaStream_t st = (cudaStream_t)stream;
  TLX_CHECK_ARG(rows >= 0 && k >= 1, "top_p_and_sample: bad extent");
  if (k > 1024) return set_error(TLX_ERR_UNSUPPORTED, "top_p_and_sample: k=%d exceeds 1024", k);
  TLX_CHECK_ARG(vocab_size >= 1, "top_p_and_sample: vocab_size must be positive");
  if (rows == 0) return TLX_OK;
  TLX_CHECK_ARG(topk_logits && topk_idx && top_p && temperature && out_tokens, "top_p_and_sample: null pointer");
  NoiseSrc ns{noise, noise_stride, key0, key1, vocab_size, op.key_dev, op.dim0_offset_dev};
  if (dtype == TLX_F32) {
    top_p_and_sample_kernel<TLX_F32><<<(unsigned)rows, 256, 0, st>>>((const float*)topk_logits, topk_idx, k, top_p,
                                                                      temperature, ns, (float)replace_val, dim0_offset,
                                                                      out_tokens);
  } else if (dtype == TLX_BF16) {
    top_p_and_sample_kernel<TLX_BF16><<<(unsigned)rows, 256, 0, st>>>(
        (const __nv_bfloat16*)topk_logits, topk_idx, k, top_p, temperature, ns,
        __float2bfloat16_rn((float)replace_val), dim0_offset, out_tokens);
  } else {
    return set_error(TLX_ERR_UNSUPPORTED, "top_p_and_sample: dtype %d not supported (f32, bf16)", dtype);
  }
  TLX_CHECK_LAUNCH("top_p_and_sample");
  return TLX_OK;
}

int tlx_top_p_and_sample(void* stream, const void* topk_logits, int dtype, const int32_t* topk_idx, int64_t rows,
                         int k, const float* top_p, const float* temperature, const float* noise,
                         int64_t noise_stride, uint32_t key0, uint32_t key1, int64_t vocab_size, double replace_val,
                         int64_t dim0_offset, int32_t* out_tokens) {
  CallOperands op;
  op.key0 = key0; op.key1 = key1; op.dim0_offset = dim0_offset;
  return top_p_and_sample_impl(stream, topk_logits, dtype, topk_idx, rows, k, top_p, temperature, noise, noise_stride, op,
                               vocab_size, replace_val, out_tokens);
}

int tlx_top_p_and_sample_dev(void* stream, const void* topk_logits, int dtype, const int32_t* topk_idx, int64_t rows,
                             int k, const float* top_p, const float* temperature, const float* noise,
                             int64_t noise_stride, const uint32_t* key_dev, int64_t vocab_size, double replace_val,
                             const int32_t* dim0_offset_dev, int32_t* out_tokens) {
  if (!noise && !key_dev) return set_error(TLX_ERR_INVALID, "top_p_and_sample: neither noise nor a key given");
  CallOperands op;
  op.key_dev = key_dev; op.dim0_offset_dev = dim0_offset_dev;
  return top_p_and_sample_impl(stream, topk_logits, dtype, topk_idx, rows, k, top_p, temperature, noise, noise_stride, op,
                               vocab_size, replace_val, out_tokens);
}

int tlx_top_p_mask(void* stream, const float* topk_logits, const float* p, int k, int64_t batch, double replace_val,
                   float* out) {
  cudaStream_t st = (cudaStream_t)stream;
  TLX_CHECK_ARG(k >= 1 && batch >= 0, "top_p_mask: bad extent");
  if (k > 1024) return set_error(TLX_ERR_UNSUPPORTED, "top_p_mask: k=%d exceeds 1024", k);
  if (batch == 0) return TLX_OK;
  TLX_CHECK_ARG(topk_logits && p && out, "top_p_mask: null pointer");
  top_p_mask_kernel<<<(unsigned)batch, 128, 0, st>>>(topk_logits, p, k, batch, (float)replace_val, out);
  TLX_CHECK_LAUNCH("top_p_mask");
  return TLX_OK;
}

static int gumbel_argmax_impl(void* stream, const float* logits, const int32_t* idx0, const int32_t* idx1, int64_t rows,
                              int64_t cols, uint32_t key0, uint32_t key1, const uint32_t* key_dev, int64_t dim1_size,
                              int axis, int32_t* out_pos) {
  cudaStream_t st = (cudaStream_t)stream;
  TLX_CHECK_ARG(axis == 0 || axis == 1, "gumbel_argmax: axis must be 0 or 1, got %d", axis);
  TLX_CHECK_ARG(rows > 0 && cols > 0 && dim1_size > 0, "gumbel_argmax: bad extent");
  TLX_CHECK_ARG(logits && idx0 && idx1 && out_pos, "gumbel_argmax: null pointer");
  const int64_t lines = axis == 1 ? rows : cols;
  gumbel_argmax_kernel<<<(unsigned)lines, 256, 0, st>>>(logits, idx0, idx1, rows, cols, key0, key1, key_dev, dim1_size,
                                                       axis, out_pos);
  TLX_CHECK_LAUNCH("gumbel_argmax");
  return TLX_OK;
}

int tlx_gumbel_argmax(void* stream, const float* logits, const int32_t* idx0, const int32_t* idx1, int64_t rows,
                      int64_t cols, uint32_t key0, uint32_t key1, int64_t dim1_size, int axis, int32_t* out_pos) {
  return gumbel_argmax_impl(stream, logits, idx0, idx1, rows, cols, key0, key1, nullptr, dim1_size, axis, out_pos);
}

int tlx_gumbel_argmax_dev(void* stream, const float* logits, const int32_t* idx0, const int32_t* idx1, int64_t rows,
                          int64_t cols, const uint32_t* key_dev, int64_t dim1_size, int axis, int32_t* out_pos) {
  if (!key_dev) return set_error(TLX_ERR_INVALID, "gumbel_argmax: null key");
  return gumbel_argmax_impl(stream, logits, idx0, idx1, rows, cols, 0u, 0u, key_dev, dim1_size, axis, out_pos);
}

static int launch_merge(cudaStream_t st, const MergeParams& p, int64_t rows) {
  int P = 2;
  while (P < p.n_cand) P <<= 1;
  const size_t smem = kSharedHeader + (size_t)P * 8 + (size_t)p.n_cand * 12;   // candidates, merged order, list
  static SmemLimit limit;
  int rc;
  if ((rc = raise_smem(limit, (const void*)merge_and_sample_kernel, smem, "merge_and_sample")) != TLX_OK) return rc;
  // one thread per two (padded) candidates: the sort's stages pair them up, the tail takes two items per thread
  int threads = P / 2;
  threads = threads < 64 ? 64 : (threads > kMergeThreads ? kMergeThreads : threads);
  // many rows of few candidates: CTAs of 128 threads, eight per SM, so that a thousand rows are one wave
  if (rows >= 256 && P <= 1024 && threads > 128) threads = 128;
  if (p.xbuf) {
    // exchange mode: the rows' arrival counts order this kernel after the candidate kernels, so it may be
    // scheduled while this rank's candidate kernel still runs (its CTAs have all started by then) and has
    // its launch latency behind it when the first rows arrive
    // ... and does run beside it only on SMs that need not change the size of their shared memory in between: the
    // candidate kernels' sizes are all of it for fewer than 256 rows and 64 % for more (1024 rows of 18992, k = 50, with
    // their candidate kernel: 37.0 us, with the default 39.5 us)
    const size_t need = (smem + 1024) * (size_t)((rows + 147) / 148 < 8 ? (rows + 147) / 148 : 8) * 100 / (228 << 10) + 1;
    const int carveout = rows < 256 || need > 100 ? 100 : need < 64 ? 64 : (int)need;
    return launch_dependent(merge_and_sample_kernel, {(unsigned)rows, (unsigned)threads, smem, 1, carveout}, st, "merge_and_sample", p);
  }
  merge_and_sample_kernel<<<(unsigned)rows, threads, smem, st>>>(p);
  TLX_CHECK_LAUNCH("merge_and_sample");
  return TLX_OK;
}

int tlx_merge_and_sample(void* stream, const float* cand_vals, const int32_t* cand_idx, const float* cand_noise,
                         int64_t rows, int n_cand, int k_per_block, int64_t block_stride, int64_t row_stride,
                         const int32_t* top_k, const float* top_p, const float* temperature, int32_t* out_tokens) {
  cudaStream_t st = (cudaStream_t)stream;
  TLX_CHECK_ARG(rows >= 0 && n_cand >= 1, "merge_and_sample: bad extent");
  TLX_CHECK_ARG(k_per_block >= 1 && n_cand % k_per_block == 0, "merge_and_sample: n_cand must be a multiple of k_per_block");
  TLX_CHECK_ARG(row_stride >= k_per_block && block_stride >= 0, "merge_and_sample: bad strides");
  if (n_cand > kMergeMaxCand)
    return set_error(TLX_ERR_UNSUPPORTED, "merge_and_sample: %d candidates exceed %d", n_cand, kMergeMaxCand);
  if (rows == 0) return TLX_OK;
  TLX_CHECK_ARG(cand_vals && cand_idx && cand_noise && top_k && top_p && temperature && out_tokens,
                "merge_and_sample: null pointer");
  MergeParams p{};
  p.cand_vals = cand_vals; p.cand_idx = cand_idx; p.cand_noise = cand_noise; p.n_cand = n_cand;
  p.k_per_block = k_per_block; p.block_stride = block_stride; p.row_stride = row_stride; p.top_k = top_k;
  p.top_p = top_p; p.temperature = temperature; p.out = out_tokens;
  return launch_merge(st, p, rows);
}

int tlx_exchange_merge_and_sample(void* stream, void* exchange, int64_t rows, int k_cand, int world,
                                  const int32_t* top_k, const float* top_p, const float* temperature,
                                  int32_t* out_tokens, int32_t* out_status) {
  cudaStream_t st = (cudaStream_t)stream;
  TLX_CHECK_ARG(rows >= 1 && k_cand >= 1 && world >= 1 && world <= kExchangeMaxWorld, "exchange_merge_and_sample: bad extent");
  if ((int64_t)world * k_cand > kMergeMaxCand)
    return set_error(TLX_ERR_UNSUPPORTED, "exchange_merge_and_sample: %lld candidates exceed %d",
                     (long long)world * k_cand, kMergeMaxCand);
  TLX_CHECK_ARG(exchange && top_k && top_p && temperature && out_tokens, "exchange_merge_and_sample: null pointer");
  const ExchangeLayout l = exchange_layout(rows, k_cand, world);
  MergeParams p{};
  p.n_cand = world * k_cand; p.k_per_block = k_cand; p.block_stride = (int64_t)l.block_elems; p.row_stride = k_cand;
  p.top_k = top_k; p.top_p = top_p; p.temperature = temperature; p.out = out_tokens;
  p.xbuf = (unsigned char*)exchange; p.world = world; p.rows = rows; p.status = out_status;
  for (int q = 0; q < 2; ++q) { p.off_flags[q] = l.off_flags[q]; p.off_cand[q] = l.off_cand[q]; }
  return launch_merge(st, p, rows);
}

}  // extern "C"
