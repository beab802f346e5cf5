// Gather (take_along_axis), cumsum, arg-max and counter-based uniform noise.
// All four are HBM-bound; all but the gather's random reads are coalesced.
#include "row_cluster.cuh"

#include <atomic>

namespace tlx {

static thread_local char g_err[512] = "";

int set_error(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

static std::atomic<unsigned long long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

// ---------------------------------------------------------------------------------
// gather
// ---------------------------------------------------------------------------------
// Eight consecutive outputs per thread: two 16-byte index loads, eight independent random reads in flight,
// 16-byte stores.  Bound by DRAM bandwidth on random columns of a large matrix: every 4-byte element costs about 100 bytes of
// DRAM traffic (f32 [1024, 4096] out of [1024, 262144]: 460 MB in 79 us, 89 % of the copy bandwidth).
__device__ __forceinline__ uint32_t ld_no_l1(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
template <typename T, bool kNoL1>
__global__ void __launch_bounds__(256) gather_axis1_kernel(const T* __restrict__ values, const int32_t* __restrict__ idx,
                                                           T* __restrict__ out, int64_t rows, int64_t vcols, int64_t icols) {
  constexpr int kPer = 8;
  grid_wait();
  const int64_t groups_per_row = (icols + kPer - 1) / kPer;
  const int64_t total = rows * groups_per_row;
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < total; g += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = g / groups_per_row;
    const int64_t c0 = (g - r * groups_per_row) * kPer;
    const int32_t* ip = idx + r * icols + c0;
    const T* vrow = values + r * vcols;
    T* op = out + r * icols + c0;
    int32_t ii[kPer];
    const int n = (int)min((int64_t)kPer, icols - c0);
    if (n == kPer && ((reinterpret_cast<uintptr_t>(ip) & 15) == 0)) {
      const int4 a = __ldcs(reinterpret_cast<const int4*>(ip));
      const int4 b = __ldcs(reinterpret_cast<const int4*>(ip) + 1);
      ii[0] = a.x; ii[1] = a.y; ii[2] = a.z; ii[3] = a.w;
      ii[4] = b.x; ii[5] = b.y; ii[6] = b.z; ii[7] = b.w;
    } else {
#pragma unroll
      for (int j = 0; j < kPer; ++j) ii[j] = (j < n) ? __ldg(ip + j) : -1;
    }
    T o[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const bool ok = (j < n) && ii[j] >= 0 && (int64_t)ii[j] < vcols;
      if constexpr (kNoL1) o[j] = ok ? ld_no_l1(vrow + ii[j]) : T(0);
      else o[j] = ok ? __ldg(vrow + ii[j]) : T(0);
    }
    if (n == kPer && sizeof(T) == 4 && ((reinterpret_cast<uintptr_t>(op) & 15) == 0)) {
      uint4 w0, w1;
      memcpy(&w0, &o[0], 16);
      memcpy(&w1, &o[4], 16);
      __stcs(reinterpret_cast<uint4*>(op), w0);
      __stcs(reinterpret_cast<uint4*>(op) + 1, w1);
    } else {
#pragma unroll
      for (int j = 0; j < kPer; ++j) if (j < n) op[j] = o[j];
    }
  }
}

template <typename T>
__global__ void gather_axis0_kernel(const T* __restrict__ values, const int32_t* __restrict__ idx,
                                    T* __restrict__ out, int64_t vrows, int64_t cols, int64_t irows) {
  grid_wait();
  const int64_t total = irows * cols;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = e % cols;
    const int32_t i = __ldg(idx + e);
    const bool ok = i >= 0 && (int64_t)i < vrows;
    out[e] = ok ? __ldg(values + (int64_t)i * cols + c) : T(0);
  }
}

template <typename T>
static int launch_gather(cudaStream_t st, const void* values, const int32_t* idx, void* out, int64_t vr,
                         int64_t vc, int64_t ir, int64_t ic, int axis) {
  const int threads = 256;
  if (axis == 1) {
    const int64_t total = ir * ((ic + 7) >> 3);
    if (total == 0) return TLX_OK;
    const int64_t want = (total + threads - 1) / threads;
    const LaunchShape shape{(unsigned)(want < 148 * 64 ? want : 148 * 64), (unsigned)threads};
    // Many outputs out of rows of which hardly a line is read twice: the lines are not kept in L1.  us kept / not, rotating inputs,
    // and with a cold L2: f32 [1024, 1000] out of [1024, 262144] 25.6/23.6, 39/33; [256, 4096] 22.2/21.5, 33/31.  A line's second
    // reading, or a matrix that lies in L2, wants L1: [1024, 4096] out of [1024, 65537] 44.0/45.1, 59/74; [1024, 100] out of
    // [1024, 262144] 4.1/5.8.
    if constexpr (sizeof(T) == 4) {
      if (vc > (64 << 10) && ic * 32 <= vc && ir * ic >= (1 << 18)) {
        return launch_dependent(gather_axis1_kernel<T, true>, shape, st, "take_along_axis", (const T*)values, idx, (T*)out, ir, vc, ic);
      }
    }
    return launch_dependent(gather_axis1_kernel<T, false>, shape, st, "take_along_axis", (const T*)values, idx, (T*)out, ir, vc, ic);
  } else {
    const int64_t total = ir * ic;
    if (total == 0) return TLX_OK;
    const int64_t want = (total + threads - 1) / threads;
    const LaunchShape shape{(unsigned)(want < 148 * 32 ? want : 148 * 32), (unsigned)threads};
    return launch_dependent(gather_axis0_kernel<T>, shape, st, "take_along_axis", (const T*)values, idx, (T*)out, vr, vc, ir);
  }
}

// ---------------------------------------------------------------------------------
// cumsum
// ---------------------------------------------------------------------------------
// Along rows.  HBM-bound: one read, one write.  A CTA sums tiles of 256 threads x V vectors of four; a row's tiles go
// round the CTAs of a cluster (as many CTAs as it takes to fill the GPU) and every turn carries the sum on.  What
// keeps the memory system busy is a ring of kStages tiles per CTA, filled by asynchronous copies that run ahead of
// the scans, the barriers and the stores: without it the cluster's barrier of every turn was paid in full (f32
// [256, 128256] 81 us).  A thread copies and reads the same vectors, so the ring needs no barrier of its own.
//   A warp owns V runs of 32 vectors, scanned independently and chained afterwards; warp totals meet in shared memory,
// CTA totals in distributed shared memory, and the sums go out from registers.  Reversed sums walk the same vectors
// from the end.  f32 [64, 128256]: 143 us with one CTA per row and a block scan per 1024 elements.
constexpr int kCumsumThreads = 256;
template <typename T, typename Idx, int V, int kStages, int kThreads>
__global__ void __launch_bounds__(kThreads)
cumsum_axis1_kernel(const T* __restrict__ in, T* __restrict__ out, Idx cols, int reverse, int cluster, int same_phase) {
  constexpr int kWarps = kThreads / 32, kPer = kThreads * V;
  __shared__ __align__(16) uint4 ring[kStages][kPer];
  __shared__ T warp_total[2][kWarps];
  __shared__ T cta_total[2];           // alternating, so that a slow reader of the last turn is not overtaken
  const int rank = cluster > 1 ? (int)cl_rank() : 0;
  const int64_t row = blockIdx.x / cluster;
  const T* src = in + row * (int64_t)cols;
  T* dst = out + row * (int64_t)cols;
  const int off = (int)((reinterpret_cast<uintptr_t>(src) & 15) / sizeof(T));
  const Idx nvec = (off + cols + 3) / 4;
  const int lane = lane_id(), w = warp_id();
  const int slot0 = w * 32 * V + lane;
  const Idx stride = (Idx)kPer * cluster;
  auto fetch = [&](Idx v0, int stage) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const Idx v = v0 + 32 * k;
      if (v < nvec) {
        const Idx c = (reverse ? nvec - 1 - v : v) * 4 - off;
        uint4* d = &ring[stage][slot0 + 32 * k];
        if (c >= 0 && c + 4 <= cols) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(d)), "l"(src + c) : "memory");
        } else {
          T e[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) e[j] = c + j >= 0 && c + j < cols ? src[c + j] : T(0);
          memcpy(d, e, 16);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  grid_wait();
  Idx v0 = (Idx)rank * kPer + slot0;   // in the order of summation
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) fetch(v0 + i * stride, i);
  T carry = T(0);
  int turn = 0, stage = 0;
  for (Idx base = 0; base < nvec; base += stride, v0 += stride, turn ^= 1) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    T x[V][4];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      T e[4] = {T(0), T(0), T(0), T(0)};
      if (v0 + 32 * k < nvec) memcpy(e, &ring[stage][slot0 + 32 * k], 16);
#pragma unroll
      for (int j = 0; j < 4; ++j) x[k][j] = reverse ? e[3 - j] : e[j];
    }
    fetch(v0 + (kStages - 1) * stride, stage == 0 ? kStages - 1 : stage - 1);   // the slot that was read a turn ago
    stage = stage + 1 == kStages ? 0 : stage + 1;
    T incl[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
#pragma unroll
      for (int j = 1; j < 4; ++j) x[k][j] += x[k][j - 1];
      incl[k] = x[k][3];
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const T up = __shfl_up_sync(0xFFFFFFFFu, incl[k], o);
        if (lane >= o) incl[k] += up;
      }
    }
    T run = T(0);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const T total = __shfl_sync(0xFFFFFFFFu, incl[k], 31);
      incl[k] = run + (incl[k] - x[k][3]);    // sum before this vector, inside the warp
      run += total;
    }
    if (lane == 0) warp_total[turn][w] = run;
    __syncthreads();
    T before = T(0), cta = T(0);
#pragma unroll
    for (int i = 0; i < kWarps; ++i) {
      const T t = warp_total[turn][i];
      if (i < w) before += t;
      cta += t;
    }
    T all = cta;
    if (cluster > 1) {
      if (threadIdx.x == 0) cta_total[turn] = cta;
      cl_sync();
      all = T(0);
      T mine = T(0);
      const uint32_t bits = lane < cluster ? cl_ld_u32(cl_map(&cta_total[turn], (uint32_t)lane)) : 0u;
      T t;
      memcpy(&t, &bits, 4);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const T ti = __shfl_sync(0xFFFFFFFFu, t, i);
        if (i < cluster) {
          if (i < rank) mine += ti;
          all += ti;
        }
      }
      before += mine;
    }
    before += carry;
    carry += all;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const Idx v = v0 + 32 * k, c = (reverse ? nvec - 1 - v : v) * 4 - off;
      if (v >= nvec) continue;
      const T add = before + incl[k];
      T e[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) e[j] = x[k][reverse ? 3 - j : j] + add;
      if (same_phase && c >= 0 && c + 4 <= cols) {
        uint4 q;
        memcpy(&q, e, 16);
        __stcs(reinterpret_cast<uint4*>(dst + c), q);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) if (c + j >= 0 && c + j < cols) dst[c + j] = e[j];
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (cluster > 1) cl_sync();   // nobody leaves while its total may still be read
}

// The same over the CTAs of a cluster, one turn ahead: the next tile is read and summed up inside the CTA between arriving at the
// cluster's barrier with a tile's total and waiting there, which hides most of the barrier (us, with the wait directly behind the arrival /
// this: f32 [64, 128256] 17.3 / 16.4, [16, 128256] 11.6 / 10.3, [1, 128256] 9.5 / 8.0, [64, 10000] 4.5 / 3.6).  A tile's sums inside the CTA stay in registers meanwhile: four CTAs an SM.
template <typename T>
__global__ void __launch_bounds__(kCumsumThreads, 4)
cumsum_cluster_kernel(const T* __restrict__ in, T* __restrict__ out, int cols, int reverse, int cluster, int same_phase) {
  constexpr int kWarps = kCumsumThreads / 32, V = 4, kPer = kCumsumThreads * V, kStages = 2;
  __shared__ __align__(16) uint4 ring[kStages][kPer];
  __shared__ T warp_total[2][kWarps];
  __shared__ T cta_total[2];
  const int rank = (int)cl_rank();
  const int64_t row = blockIdx.x / cluster;
  const T* src = in + row * (int64_t)cols;
  T* dst = out + row * (int64_t)cols;
  const int off = (int)((reinterpret_cast<uintptr_t>(src) & 15) / sizeof(T));
  const int nvec = (off + cols + 3) / 4;
  const int lane = lane_id(), w = warp_id(), slot0 = w * 32 * V + lane;
  const int stride = kPer * cluster, turns = (nvec + stride - 1) / stride;
  auto column = [&](int v) { return (reverse ? nvec - 1 - v : v) * 4 - off; };
  auto fetch = [&](int v0, int stage) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int v = v0 + 32 * k;
      if (v < nvec) {
        const int c = column(v);
        uint4* d = &ring[stage][slot0 + 32 * k];
        if (c >= 0 && c + 4 <= cols) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(d)), "l"(src + c) : "memory");
        } else {
          T e[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) e[j] = c + j >= 0 && c + j < cols ? src[c + j] : T(0);
          memcpy(d, e, 16);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // tile `turn`: sums inside the CTA, in the order of summation; returns the CTA's total
  auto sum_tile = [&](int v0, int turn, T (&x)[V][4]) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    T incl[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      T e[4] = {T(0), T(0), T(0), T(0)};
      if (v0 + 32 * k < nvec) memcpy(e, &ring[turn & 1][slot0 + 32 * k], 16);
#pragma unroll
      for (int j = 0; j < 4; ++j) x[k][j] = reverse ? e[3 - j] : e[j];
    }
    fetch(v0 + stride, (turn + 1) & 1);   // (the slot that was read a turn ago, by this thread)
#pragma unroll
    for (int k = 0; k < V; ++k) {
#pragma unroll
      for (int j = 1; j < 4; ++j) x[k][j] += x[k][j - 1];
      incl[k] = x[k][3];
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const T up = __shfl_up_sync(0xFFFFFFFFu, incl[k], o);
        if (lane >= o) incl[k] += up;
      }
    }
    T run = T(0);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const T total = __shfl_sync(0xFFFFFFFFu, incl[k], 31);
      incl[k] = run + (incl[k] - x[k][3]);
      run += total;
    }
    if (lane == 0) warp_total[turn & 1][w] = run;
    __syncthreads();
    T before = T(0), cta = T(0);
#pragma unroll
    for (int i = 0; i < kWarps; ++i) {
      const T t = warp_total[turn & 1][i];
      if (i < w) before += t;
      cta += t;
    }
#pragma unroll
    for (int k = 0; k < V; ++k) {
#pragma unroll
      for (int j = 0; j < 4; ++j) x[k][j] += before + incl[k];
    }
    return cta;
  };
  auto publish = [&](int turn, T cta) {
    if (threadIdx.x == 0) cta_total[turn & 1] = cta;
    cl_arrive();
  };
  grid_wait();
  int v0 = rank * kPer + slot0;
  T x[V][4], next[V][4], carry = T(0);
  fetch(v0, 0);
  publish(0, sum_tile(v0, 0, x));
#pragma unroll 1
  for (int turn = 0; turn < turns; ++turn, v0 += stride) {
    const bool more = turn + 1 < turns;
    T cta = T(0);
    if (more) cta = sum_tile(v0 + stride, turn + 1, next);
    cl_wait();
    const uint32_t bits = lane < cluster ? cl_ld_u32(cl_map(&cta_total[turn & 1], (uint32_t)lane)) : 0u;
    T t, mine = T(0), all = T(0);
    memcpy(&t, &bits, 4);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const T ti = __shfl_sync(0xFFFFFFFFu, t, i);
      if (i < rank) mine += ti;
      if (i < cluster) all += ti;
    }
    // (a total is overwritten two turns on, when every CTA has arrived at the turn between with what it read)
    publish(turn + 1, cta);   // (after the last turn: nobody leaves while its total may still be read)
    const T add = carry + mine;
    carry += all;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int v = v0 + 32 * k, c = column(v);
      if (v < nvec) {
        T e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = x[k][reverse ? 3 - j : j] + add;
        if (same_phase && c >= 0 && c + 4 <= cols) {
          uint4 q;
          memcpy(&q, e, 16);
          __stcs(reinterpret_cast<uint4*>(dst + c), q);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) if (c + j >= 0 && c + j < cols) dst[c + j] = e[j];
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) x[k][j] = next[k][j];
    }
  }
  cl_wait();
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Along columns.  A CTA takes 32 columns (128-byte rows of the matrix per warp) and kAxis0Warps x kAxis0Rows rows at a
// time: every warp sums its own consecutive rows, the totals meet in shared memory, the sums go out from registers.
// Few columns: the rows of a turn are cut over the CTAs of a cluster, whose totals meet in distributed shared memory.
// One thread per column with one load in flight took 130 us for f32 [1024, 500].
constexpr int kAxis0Warps = 16, kAxis0Rows = 16, kAxis0Turn = kAxis0Warps * kAxis0Rows;
template <typename T>
__global__ void __launch_bounds__(kAxis0Warps * 32) cumsum_axis0_kernel(const T* __restrict__ in, T* __restrict__ out, int64_t rows,
                                                                         int64_t cols, int reverse, int cluster) {
  __shared__ T total[2][kAxis0Warps][32];
  __shared__ T cta_total[2][32];
  const int rank = cluster > 1 ? (int)cl_rank() : 0;
  const int lane = lane_id(), w = warp_id();
  const int64_t c = blockIdx.x / cluster * 32ll + lane;
  const bool live = c < cols;
  T carry = T(0);
  int turn = 0;
  grid_wait();
  for (int64_t base = 0; base < rows; base += (int64_t)kAxis0Turn * cluster, turn ^= 1) {
    const int64_t r0 = base + rank * kAxis0Turn + w * kAxis0Rows;
    T x[kAxis0Rows];
#pragma unroll
    for (int k = 0; k < kAxis0Rows; ++k) {
      const int64_t r = r0 + k;
      x[k] = live && r < rows ? __ldcs(in + (reverse ? rows - 1 - r : r) * cols + c) : T(0);
    }
#pragma unroll
    for (int k = 1; k < kAxis0Rows; ++k) x[k] += x[k - 1];
    total[turn][w][lane] = x[kAxis0Rows - 1];
    __syncthreads();
    T before = carry, cta = T(0);
#pragma unroll
    for (int i = 0; i < kAxis0Warps; ++i) {
      const T t = total[turn][i][lane];
      if (i < w) before += t;
      cta += t;
    }
    T all = cta;
    if (cluster > 1) {
      if (w == 0) cta_total[turn][lane] = cta;
      cl_sync();
      all = T(0);
      for (int i = 0; i < cluster; ++i) {
        const uint32_t bits = cl_ld_u32(cl_map(&cta_total[turn][lane], (uint32_t)i));
        T t;
        memcpy(&t, &bits, 4);
        if (i < rank) before += t;
        all += t;
      }
    }
    carry += all;
#pragma unroll
    for (int k = 0; k < kAxis0Rows; ++k) {
      const int64_t r = r0 + k;
      if (live && r < rows) __stcs(out + (reverse ? rows - 1 - r : r) * cols + c, x[k] + before);
    }
  }
  if (cluster > 1) cl_sync();   // nobody leaves while its totals may still be read
}

// The same for a few rows: a thread per column, a short loop.  The kernel above is straight-line code for sixteen rows a warp
// and most of its time is then instruction fetch and idle warps.
//   Eight rows at a time are summed up on their own and added to the sum of those before: rounding errors gather over 8 + rows / 8
// additions, not over all rows (128 rows of uniform numbers, relative error of the sums 5.8e-8; one running sum 1.4e-7, the kernel
// above 5.1e-8), and sixteen loads are in flight (f32 [128, 70000] 24.2 us with the running sum, 16.8 so).
template <typename T>
__global__ void __launch_bounds__(128) cumsum_axis0_few_kernel(const T* __restrict__ in, T* __restrict__ out, int64_t rows, int64_t cols,
                                                               int reverse) {
  constexpr int kRows = 8;
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  grid_wait();
  if (c >= cols) return;
  const int64_t step = reverse ? -cols : cols;
  int64_t at = (reverse ? rows - 1 : 0) * cols + c;
  T before = T(0);
  int64_t r = 0;
#pragma unroll 2
  for (; r + kRows <= rows; r += kRows, at += kRows * step) {
    T x[kRows];
#pragma unroll
    for (int k = 0; k < kRows; ++k) x[k] = in[at + k * step];
#pragma unroll
    for (int k = 1; k < kRows; ++k) x[k] += x[k - 1];
#pragma unroll
    for (int k = 0; k < kRows; ++k) out[at + k * step] = before + x[k];
    before += x[kRows - 1];
  }
  // the rest: four, then at most three
  T sum = T(0);
  if (r + 4 <= rows) {
    T x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = in[at + k * step];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      sum += x[k];
      out[at + k * step] = before + sum;
    }
    r += 4;
    at += 4 * step;
  }
  const int left = (int)(rows - r);
  T x[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) x[k] = k < left ? in[at + k * step] : T(0);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    sum += x[k];
    if (k < left) out[at + k * step] = before + sum;
  }
}

template <typename T, typename Idx, int V, int kStages, int kThreads = kCumsumThreads>
static int launch_cumsum_rows(cudaStream_t st, const T* in, T* out, int64_t rows, int64_t cols, int reverse, int cluster) {
  const int same = ((reinterpret_cast<uintptr_t>(in) ^ reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  return launch_dependent(cumsum_axis1_kernel<T, Idx, V, kStages, kThreads>, {(unsigned)(rows * cluster), kThreads, 0, cluster}, st, "cumsum",
                          in, out, cols, reverse, cluster, same);
}

// One vector a thread for rows of up to 1024 elements, and a single warp for up to 128 (f32 [6000, 60] 4.7 us, with eight warps
// 10.0); beyond that two tiles of 4096 elements (32 KB: six CTAs fit an SM)
// and as many CTAs per row, up to eight and up to its tiles, as give 740 in all (five per SM): a barrier across CTAs
// every turn costs more than it brings once the rows fill the GPU.  Measured, f32, with the ring: [64, 128256] 15.7 us,
// [167, 27252] 10.1, [256, 128256] 54, [1024, 31000] 48 (5.3 TB/s).
template <typename T>
static int launch_cumsum(cudaStream_t st, const void* in, void* out, int64_t rows, int64_t cols, int axis, int reverse) {
  const T* x = (const T*)in;
  T* y = (T*)out;
  if (axis == 0) {
    // A thread per column where both types gain.  us a thread per column / sixteen warps per 32 columns, f32 and i32: [16, 500] 1.5/3.2
    // 1.6/3.2, [40, 4096] 2.1/3.2 2.5/3.3, [64, 4096] 2.7/3.2 3.5/3.4, [48, 16384] 3.2/8.3 4.0/8.5, [64, 16384] 5.8/8.5 8.5/8.8, [64, 32768]
    // 7.3/13.5 10.2/13.9, [96, 32768] 9.9/14.3 14.4/14.7, [128, 70000] 16.9/29 20.8/30, [256, 70000] 31/37 39/37
    if (rows <= (cols < 8192 ? 40 : cols < 32768 ? 48 : cols < 65536 ? 64 : 128)) {
      return launch_dependent(cumsum_axis0_few_kernel<T>, {(unsigned)((cols + 127) / 128), 128}, st, "cumsum", x, y, rows, cols, reverse);
    }
    const int64_t strips = (cols + 31) / 32;
    int cluster = 1;
    while (cluster < 8 && strips * cluster * 2 <= 592 && (int64_t)cluster * kAxis0Turn < rows) cluster *= 2;
    return launch_dependent(cumsum_axis0_kernel<T>, {(unsigned)(strips * cluster), kAxis0Warps * 32, 0, cluster}, st, "cumsum", x, y, rows,
                            cols, reverse, cluster);
  }
  const int64_t n = cols + 3;   // the first vector may be a partial one
  if (n <= 128) return launch_cumsum_rows<T, int, 1, 2, 32>(st, x, y, rows, cols, reverse, 1);
  if (n <= 1024) return launch_cumsum_rows<T, int, 1, 2>(st, x, y, rows, cols, reverse, 1);
  int cluster = 1;
  while (cluster < 8 && rows * cluster * 2 <= 740 && cluster * 4096ll < n) cluster *= 2;
  // one turn ahead while all clusters of CTAs that hold a tile more in registers, four an SM, surely run at once (us ahead / not: f32
  // [64, 128256], 512 CTAs, 16.4 / 17.2, [140, 20000], 560, 9.5 / 9.5, [72, 128256], 576, 22.8 / 18.8, [150, 30000], 600, 13.1 / 10.9)
  if (cluster > 1 && rows * cluster <= 520 && cols < (1ll << 30)) {
    const int same = ((reinterpret_cast<uintptr_t>(x) ^ reinterpret_cast<uintptr_t>(y)) & 15) == 0;
    return launch_dependent(cumsum_cluster_kernel<T>, {(unsigned)(rows * cluster), kCumsumThreads, 0, cluster}, st, "cumsum", x, y, (int)cols,
                            reverse, cluster, same);
  }
  if (cols < (1ll << 30)) return launch_cumsum_rows<T, int, 4, 2>(st, x, y, rows, cols, reverse, cluster);
  return launch_cumsum_rows<T, int64_t, 4, 2>(st, x, y, rows, cols, reverse, cluster);
}

// ---------------------------------------------------------------------------------
// arg-max, lowest index on ties
// ---------------------------------------------------------------------------------
template <int DT>
__global__ void argmax_axis1_kernel(const typename Elem<DT>::type* __restrict__ x, int64_t cols,
                                    int32_t* __restrict__ out) {
  __shared__ uint64_t sbest[32];
  const typename Elem<DT>::type* row = x + blockIdx.x * cols;
  // composite: key in the high word, inverted column in the low word -> one u64 max
  uint64_t best = 0;
  for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) {
    uint64_t v = ((uint64_t)Elem<DT>::key(row[c]) << 32) | (uint32_t)(0x7FFFFFFF - (int32_t)c);
    best = v > best ? v : best;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    uint64_t n = shfl_xor_u64(best, o);
    best = n > best ? n : best;
  }
  if (lane_id() == 0) sbest[warp_id()] = best;
  __syncthreads();
  if (warp_id() == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    best = lane_id() < nw ? sbest[lane_id()] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      uint64_t n = shfl_xor_u64(best, o);
      best = n > best ? n : best;
    }
    if (lane_id() == 0) out[blockIdx.x] = 0x7FFFFFFF - (int32_t)(uint32_t)best;
  }
}

template <int DT>
__global__ void argmax_axis0_kernel(const typename Elem<DT>::type* __restrict__ x, int64_t rows, int64_t cols,
                                    int32_t* __restrict__ out) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= cols) return;
  uint32_t bk = 0;
  int32_t bi = 0;
  for (int64_t r = 0; r < rows; ++r) {
    uint32_t k = Elem<DT>::key(x[r * cols + c]);
    if (r == 0 || k > bk) { bk = k; bi = (int32_t)r; }
  }
  out[c] = bi;
}

template <int DT>
static int launch_argmax(cudaStream_t st, const void* keys, int64_t rows, int64_t cols, int axis, int32_t* out) {
  using T = typename Elem<DT>::type;
  if (axis == 1) {
    argmax_axis1_kernel<DT><<<(unsigned)rows, 256, 0, st>>>((const T*)keys, cols, out);
  } else {
    argmax_axis0_kernel<DT><<<(unsigned)((cols + 127) / 128), 128, 0, st>>>((const T*)keys, rows, cols, out);
  }
  TLX_CHECK_LAUNCH("argmax");
  return TLX_OK;
}

// ---------------------------------------------------------------------------------
// counter-based uniform noise at arbitrary (i0, i1)
// ---------------------------------------------------------------------------------
__global__ void sparse_uniform_kernel(uint32_t k0, uint32_t k1, const uint32_t* __restrict__ key_dev,
                                      const int32_t* __restrict__ i0, const int32_t* __restrict__ i1, int64_t count,
                                      int64_t dim1, float minval, float maxval, float* __restrict__ out) {
  if (key_dev) { k0 = __ldg(key_dev); k1 = __ldg(key_dev + 1); }   // the key as a device operand
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < count;
       e += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t ctr = (uint32_t)((int64_t)i0[e] * dim1 + (int64_t)i1[e]);
    const float f = threefry_uniform01(k0, k1, ctr);
    // separate multiply and add, as the reference computes them
    out[e] = fmaxf(minval, __fadd_rn(__fmul_rn(f, __fsub_rn(maxval, minval)), minval));
  }
}

// ---------------------------------------------------------------------------------
// key outputs in canonical form: what a float looks like after the round trip through the
// order-preserving key (-0 -> +0, every NaN -> the one canonical NaN), in place
// ---------------------------------------------------------------------------------
template <int DT>
__global__ void canonicalize_kernel(typename Elem<DT>::type* __restrict__ x, int64_t count) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < count; e += (int64_t)gridDim.x * blockDim.x)
    x[e] = Elem<DT>::from_key(Elem<DT>::key(x[e]));
}

}  // namespace tlx

using namespace tlx;

extern "C" {

int tlx_abi_version(void) { return TLX_ABI_VERSION; }
const char* tlx_last_error(void) { return tlx::g_err; }
unsigned long long tlx_kernel_launches(void) { return tlx::g_launches.load(std::memory_order_relaxed); }

int tlx_take_along_axis(void* stream, const void* values, const int32_t* indices, void* out, int64_t val_rows,
                        int64_t val_cols, int64_t idx_rows, int64_t idx_cols, int elem_bytes, int axis) {
  cudaStream_t st = (cudaStream_t)stream;
  TLX_CHECK_ARG(axis == 0 || axis == 1, "take_along_axis: axis must be 0 or 1, got %d", axis);
  TLX_CHECK_ARG(val_rows >= 0 && val_cols >= 0 && idx_rows >= 0 && idx_cols >= 0, "take_along_axis: negative extent");
  if (axis == 1)
    TLX_CHECK_ARG(val_rows == idx_rows, "take_along_axis: batch extents differ (%lld vs %lld)", (long long)val_rows,
                  (long long)idx_rows);
  else
    TLX_CHECK_ARG(val_cols == idx_cols, "take_along_axis: batch extents differ (%lld vs %lld)", (long long)val_cols,
                  (long long)idx_cols);
  if (idx_rows * idx_cols == 0) return TLX_OK;
  TLX_CHECK_ARG(values && indices && out, "take_along_axis: null pointer");
  switch (elem_bytes) {
    case 1: return launch_gather<uint8_t>(st, values, indices, out, val_rows, val_cols, idx_rows, idx_cols, axis);
    case 2: return launch_gather<uint16_t>(st, values, indices, out, val_rows, val_cols, idx_rows, idx_cols, axis);
    case 4: return launch_gather<uint32_t>(st, values, indices, out, val_rows, val_cols, idx_rows, idx_cols, axis);
    case 8: return launch_gather<uint64_t>(st, values, indices, out, val_rows, val_cols, idx_rows, idx_cols, axis);
    default: return set_error(TLX_ERR_UNSUPPORTED, "take_along_axis: element size %d not supported", elem_bytes);
  }
}

int tlx_cumsum(void* stream, const void* in, void* out, int64_t rows, int64_t cols, int dtype, int axis,
               int reverse) {
  cudaStream_t st = (cudaStream_t)stream;
  TLX_CHECK_ARG(axis == 0 || axis == 1, "cumsum: axis must be 0 or 1, got %d", axis);
  TLX_CHECK_ARG(rows >= 0 && cols >= 0, "cumsum: negative extent");
  if (rows * cols == 0) return TLX_OK;
  TLX_CHECK_ARG(in && out, "cumsum: null pointer");
  if (dtype != TLX_F32 && dtype != TLX_I32)
    return set_error(TLX_ERR_UNSUPPORTED, "cumsum: dtype %d not supported (f32, i32)", dtype);
  return dtype == TLX_F32 ? launch_cumsum<float>(st, in, out, rows, cols, axis, reverse)
                          : launch_cumsum<int>(st, in, out, rows, cols, axis, reverse);
}

int tlx_argmax(void* stream, const void* keys, int dtype, int64_t rows, int64_t cols, int axis, int32_t* out_idx) {
  cudaStream_t st = (cudaStream_t)stream;
  TLX_CHECK_ARG(axis == 0 || axis == 1, "argmax: axis must be 0 or 1, got %d", axis);
  TLX_CHECK_ARG(rows > 0 && cols > 0, "argmax: empty input");
  TLX_CHECK_ARG(keys && out_idx, "argmax: null pointer");
  TLX_CHECK_ARG(rows < (1ll << 31) && cols < (1ll << 31), "argmax: extent too large");
  switch (dtype) {
    case TLX_F32: return launch_argmax<TLX_F32>(st, keys, rows, cols, axis, out_idx);
    case TLX_BF16: return launch_argmax<TLX_BF16>(st, keys, rows, cols, axis, out_idx);
    case TLX_F16: return launch_argmax<TLX_F16>(st, keys, rows, cols, axis, out_idx);
    case TLX_I32: return launch_argmax<TLX_I32>(st, keys, rows, cols, axis, out_idx);
    case TLX_U32: return launch_argmax<TLX_U32>(st, keys, rows, cols, axis, out_idx);
    default: return set_error(TLX_ERR_UNSUPPORTED, "argmax: dtype %d not supported", dtype);
  }
}

static int sparse_random_uniform_impl(void* stream, uint32_t key0, uint32_t key1, const uint32_t* key_dev,
                                      const int32_t* idx0, const int32_t* idx1, int64_t count, int64_t dim1_size,
                                      float minval, float maxval, float* out) {
  cudaStream_t st = (cudaStream_t)stream;
  TLX_CHECK_ARG(count >= 0 && dim1_size > 0, "sparse_random_uniform: bad extent");
  if (count == 0) return TLX_OK;
  TLX_CHECK_ARG(idx0 && idx1 && out, "sparse_random_uniform: null pointer");
  const int64_t want = (count + 255) / 256;
  const int blocks = (int)(want < 148 * 16 ? want : 148 * 16);
  sparse_uniform_kernel<<<blocks, 256, 0, st>>>(key0, key1, key_dev, idx0, idx1, count, dim1_size, minval, maxval, out);
  TLX_CHECK_LAUNCH("sparse_random_uniform");
  return TLX_OK;
}

int tlx_canonicalize_keys(void* stream, void* x, int dtype, int64_t count) {
  cudaStream_t st = (cudaStream_t)stream;
  TLX_CHECK_ARG(count >= 0, "canonicalize_keys: negative extent");
  if (count == 0 || dtype == TLX_I32 || dtype == TLX_U32) return TLX_OK;   // integers are their own canonical form
  TLX_CHECK_ARG(x, "canonicalize_keys: null pointer");
  const int64_t want = (count + 255) / 256;
  const int blocks = (int)(want < 148 * 16 ? want : 148 * 16);
  switch (dtype) {
    case TLX_F32: canonicalize_kernel<TLX_F32><<<blocks, 256, 0, st>>>((float*)x, count); break;
    case TLX_BF16: canonicalize_kernel<TLX_BF16><<<blocks, 256, 0, st>>>((__nv_bfloat16*)x, count); break;
    case TLX_F16: canonicalize_kernel<TLX_F16><<<blocks, 256, 0, st>>>((__half*)x, count); break;
    default: return set_error(TLX_ERR_UNSUPPORTED, "canonicalize_keys: dtype %d not supported", dtype);
  }
  TLX_CHECK_LAUNCH("canonicalize_keys");
  return TLX_OK;
}

int tlx_sparse_random_uniform(void* stream, uint32_t key0, uint32_t key1, const int32_t* idx0, const int32_t* idx1,
                              int64_t count, int64_t dim1_size, float minval, float maxval, float* out) {
  return sparse_random_uniform_impl(stream, key0, key1, nullptr, idx0, idx1, count, dim1_size, minval, maxval, out);
}

int tlx_sparse_random_uniform_dev(void* stream, const uint32_t* key_dev, const int32_t* idx0, const int32_t* idx1,
                                  int64_t count, int64_t dim1_size, float minval, float maxval, float* out) {
  if (!key_dev) return set_error(TLX_ERR_INVALID, "sparse_random_uniform: null key");
  return sparse_random_uniform_impl(stream, 0u, 0u, key_dev, idx0, idx1, count, dim1_size, minval, maxval, out);
}

}  // extern "C"
