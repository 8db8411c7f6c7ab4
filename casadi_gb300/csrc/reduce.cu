// Reductions over instances (MapSum). See reduce.cuh for the two summation orders.
//
// The instance-order sums give each row to a CTA, or, where rows are many or short, to a thread
// (in_chains); the tree kernel runs one warp per work item with coalesced loads along the instance
// axis (rows are instance-minor) and is bound by HBM (one read of the block).
#include <algorithm>

#include "reduce.cuh"

namespace cgb {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarpsPerCta = 8;
constexpr int kChainThreads = 128;

// ---- instance-order sums ------------------------------------------------------------------------
// ((0 + x0) + x1) + ... rounds at every step, so the order of the additions cannot change; but
// within one binade of the running sum s = m u (u its ulp, 2^52 < m < 2^53) a step adds a whole
// number of ulps, round(x/u), and a tie goes to the even of two neighbours: the step's increment
// of m depends on s only through m's parity. A step is therefore a pair of integers (the increment
// from an even and from an odd m), pairs compose associatively, and a run of steps is a parallel
// scan, exact as long as every intermediate m stays inside the binade. A CTA takes a chunk of
// 4096 elements of a row: scan, then every thread replays its eight steps from its own start and
// looks for the first m outside (2^52, 2^53). Up to there the result is the sequential one; that
// element is added in FP64, and the scan goes on after it: by one warp, 128 elements at a time,
// since failures come in clusters (a sum about a power of two crosses it every third element or
// so), until four windows have passed without one; a window that ends early is followed by 8, 16,
// ... 64 elements in FP64 (sums that stay near zero, infinities and NaN: all of them).
//
// A dependent FP64 addition takes about 70 cycles, a warp's window as much as eight of them. The
// rollout's cost and 20 shared controls' gradients summed over 131072 instances (21 rows, one launch)
// take 9.0 ms as plain chains and 0.28 to 0.55 ms here, by how long a gradient's sum stays about a
// power of two; 2.33 ms where one is near zero throughout (5063 crossings). With the CTA's scan after
// every failure these were 0.32 to 0.72 and 3.39 ms.
constexpr int kOrdThreads = 512;
constexpr int kOrdPer = 8;
constexpr int kOrdChunk = kOrdThreads * kOrdPer;
constexpr int kOrdLane = 4, kOrdWindow = 32 * kOrdLane;  // elements of a lane and of a warp's scan
constexpr int kOrdClean = 4;        // windows without a failure before the CTA scans again
constexpr int kOrdMinSerial = 8, kOrdMaxSerial = 64;  // a warp's scan costs as much as 8 additions
constexpr long long kM52 = 1ll << 52, kM53 = 1ll << 53;

// Increments of m over a run of steps that starts at an even (i0) or odd (i1) m.
struct Inc {
  long long i0, i1;
};
__device__ __forceinline__ Inc compose(const Inc& a, const Inc& b) {
  return Inc{a.i0 + ((a.i0 & 1) ? b.i1 : b.i0), a.i1 + ((a.i1 & 1) ? b.i0 : b.i1)};
}
__device__ __forceinline__ Inc shfl_up(const Inc& a, int d) {
  return Inc{__shfl_up_sync(kFull, a.i0, d), __shfl_up_sync(kFull, a.i1, d)};
}

// The step of x for a sum with exponent field es >= 2 and sign bit sneg: m += round(x/u).
// False when x alone leaves the binade (or is not finite).
__device__ __forceinline__ bool step_of(double x, int es, bool sneg, Inc* out) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(x));
  const int ex = static_cast<int>((b >> 52) & 0x7ff);
  const long long mx = static_cast<long long>(b & (kM52 - 1)) + (ex ? kM52 : 0);
  const int d = es - (ex ? ex : 1);  // |x| / u = mx >> d
  const int sh = d < 0 ? 0 : (d > 54 ? 54 : d);
  long long k = mx >> sh;
  const long long rem = mx - (k << sh), half = sh ? 1ll << (sh - 1) : kM53;
  const int tie = rem == half ? 1 : 0, odd = static_cast<int>(k & 1);
  k += rem > half ? 1 : 0;
  const long long a0 = k + (tie & odd), a1 = k + (tie & (odd ^ 1));
  const bool neg = (static_cast<long long>(b) < 0) != sneg;
  *out = Inc{neg ? -a0 : a0, neg ? -a1 : a1};
  return d >= 0 && ex != 2047;
}

__device__ __forceinline__ int ord_pad(int i) { return i + (i >> 3); }  // conflict-free by eights

// Adds elements [i, i + w) to *s by one warp (w <= kOrdWindow), up to the first that needs a step in
// FP64; how many were added.
__device__ __forceinline__ int sum_window(const double* buf, int i, int w, int lane, double* s) {
  const long long sb = __double_as_longlong(*s);
  const int es = static_cast<int>((sb >> 52) & 0x7ff);
  const bool sneg = sb < 0;
  if (es < 2 || es == 2047) return 0;
  const long long m0 = (sb & (kM52 - 1)) | kM52;
  const long long top = (sneg ? kM52 << 11 : 0) | (static_cast<long long>(es) << 52);
  Inc step[kOrdLane], inc{0, 0};
  bool out[kOrdLane];
#pragma unroll
  for (int j = 0; j < kOrdLane; ++j) {
    const int k = lane * kOrdLane + j;
    const bool in = k < w;
    out[j] = !step_of(in ? buf[ord_pad(i + k)] : 0.0, es, sneg, &step[j]);
    if (out[j]) step[j] = Inc{0, 0};
    inc = compose(inc, step[j]);
  }
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const Inc up = shfl_up(inc, d);
    if (lane >= d) inc = compose(up, inc);
  }
  Inc pre = shfl_up(inc, 1);
  if (lane == 0) pre = Inc{0, 0};
  long long m = m0 + ((m0 & 1) ? pre.i1 : pre.i0), m_fail = m;
  int f = kOrdLane;
#pragma unroll
  for (int j = 0; j < kOrdLane; ++j) {
    const long long mj = m + ((m & 1) ? step[j].i1 : step[j].i0);
    if (f == kOrdLane && lane * kOrdLane + j < w && (out[j] || mj <= kM52 || mj >= kM53)) {
      f = j;
      m_fail = m;
    }
    m = mj;
  }
  const unsigned failed = __ballot_sync(kFull, f < kOrdLane);
  const int at = failed ? __ffs(failed) - 1 : 31;
  const long long end = __shfl_sync(kFull, failed ? m_fail : m, at);
  const int got = failed ? at * kOrdLane + __shfl_sync(kFull, f, at) : w;
  *s = __longlong_as_double(top | (end & (kM52 - 1)));
  return got;
}

struct SumRowsArgs {
  SumRows g[kMaxSumGroups];
  int count;
};

__global__ void __launch_bounds__(kOrdThreads)
    k_sum_instance_order(const __grid_constant__ SumRowsArgs a, long long total, long long n) {
  __shared__ double buf[kOrdChunk + kOrdChunk / 8];
  __shared__ Inc warp_inc[kOrdThreads / 32];
  __shared__ int fail_at;
  __shared__ double sum_at;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (long long rr = blockIdx.x; rr < total; rr += gridDim.x) {
    long long r = rr;
    int g = 0;
    while (r >= a.g[g].rows) r -= a.g[g++].rows;
    const double* row = a.g[g].src + r * a.g[g].ld;
    double s = 0.0, next[kOrdPer];
    auto fetch = [&](long long pos) {
#pragma unroll
      for (int j = 0; j < kOrdPer; ++j) {
        const long long i = pos + t + kOrdThreads * j;
        next[j] = i < n ? __ldg(row + i) : 0.0;  // past the end: adds nothing
      }
    };
    fetch(0);
    int serial = kOrdMinSerial;
    for (long long pos = 0; pos < n; pos += kOrdChunk) {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < kOrdPer; ++j) buf[ord_pad(t + kOrdThreads * j)] = next[j];
      fetch(pos + kOrdChunk);
      const int cnt = static_cast<int>(n - pos < kOrdChunk ? n - pos : kOrdChunk);
      for (int off = 0; off < cnt;) {  // elements [off, cnt) of the chunk are left
        if (t == 0) fail_at = kOrdChunk;
        __syncthreads();
        const long long sb = __double_as_longlong(s);
        const int es = static_cast<int>((sb >> 52) & 0x7ff);
        const bool sneg = sb < 0;
        const long long m0 = (sb & (kM52 - 1)) | kM52;
        int fail = off;
        if (es >= 2 && es < 2047) {
          Inc step[kOrdPer], run{0, 0};
          int bad = kOrdPer;  // first of this thread's elements that leaves the binade by itself
#pragma unroll
          for (int j = kOrdPer - 1; j >= 0; --j) {
            const int i = t * kOrdPer + j;
            if (!step_of(buf[ord_pad(i)], es, sneg, &step[j])) {
              bad = i >= off ? j : bad;
              step[j] = Inc{0, 0};
            }
            if (i < off) step[j] = Inc{0, 0};
          }
#pragma unroll
          for (int j = 0; j < kOrdPer; ++j) run = compose(run, step[j]);
          // scan over the warp, then over the warps
          Inc inc = run;
#pragma unroll
          for (int d = 1; d < 32; d <<= 1) {
            const Inc up = shfl_up(inc, d);
            if (lane >= d) inc = compose(up, inc);
          }
          if (lane == 31) warp_inc[warp] = inc;
          Inc pre = shfl_up(inc, 1);
          if (lane == 0) pre = Inc{0, 0};
          __syncthreads();
          Inc all = lane < kOrdThreads / 32 ? warp_inc[lane] : Inc{0, 0};
#pragma unroll
          for (int d = 1; d < kOrdThreads / 32; d <<= 1) {
            const Inc up = shfl_up(all, d);
            if (lane >= d) all = compose(up, all);
          }
          const int w1 = warp ? warp - 1 : 0, wl = kOrdThreads / 32 - 1;
          Inc before{__shfl_sync(kFull, all.i0, w1), __shfl_sync(kFull, all.i1, w1)};
          if (warp == 0) before = Inc{0, 0};
          const long long tot0 = __shfl_sync(kFull, all.i0, wl);
          const long long tot1 = __shfl_sync(kFull, all.i1, wl);
          pre = compose(before, pre);
          // this thread's steps from its own start
          long long m = m0 + ((m0 & 1) ? pre.i1 : pre.i0), m_fail = m;
          int f = kOrdPer;
#pragma unroll
          for (int j = 0; j < kOrdPer; ++j) {
            const long long mj = m + ((m & 1) ? step[j].i1 : step[j].i0);
            if (f == kOrdPer && (j == bad || mj <= kM52 || mj >= kM53) &&
                t * kOrdPer + j >= off) {
              f = j;
              m_fail = m;
            }
            m = mj;
          }
          const int mine = f < kOrdPer ? t * kOrdPer + f : kOrdChunk;
          const int first = __reduce_min_sync(kFull, mine);
          if (lane == 0 && first < kOrdChunk) atomicMin(&fail_at, first);
          __syncthreads();
          fail = fail_at;
          const long long top = (sneg ? kM52 << 11 : 0) | (static_cast<long long>(es) << 52);
          if (fail >= cnt) {
            s = __longlong_as_double(top | ((m0 + ((m0 & 1) ? tot1 : tot0)) & (kM52 - 1)));
            break;
          }
          if (mine == fail) sum_at = __longlong_as_double(top | (m_fail & (kM52 - 1)));
        } else if (t == 0) {
          sum_at = s;
        }
        __syncthreads();
        if (warp == 0) {
          double acc = sum_at;
          int i = fail;
          for (int clean = 0; i < cnt && clean < kOrdClean;) {
            // the failing element in FP64 (in a stretch of failures: some more)
            const int end = min(i + serial, cnt);
            for (; i + 8 <= end; i += 8) {
              double v[8];
#pragma unroll
              for (int k = 0; k < 8; ++k) v[k] = buf[ord_pad(i + k)];
#pragma unroll
              for (int k = 0; k < 8; ++k) acc = __dadd_rn(acc, v[k]);
            }
            for (; i < end; ++i) acc = __dadd_rn(acc, buf[ord_pad(i)]);
            for (clean = 0; i < cnt && clean < kOrdClean; ++clean) {
              const int w = min(kOrdWindow, cnt - i), got = sum_window(buf, i, w, lane, &acc);
              i += got;
              if (got < w) {
                serial = got < 2 * kOrdMinSerial ? min(2 * serial, kOrdMaxSerial) : kOrdMinSerial;
                break;
              }
            }
          }
          if (lane == 0) {
            sum_at = acc;
            fail_at = i;
          }
        }
        __syncthreads();
        s = sum_at;
        off = fail_at;
        __syncthreads();
      }
    }
    if (t == 0) a.g[g].dst[r] = s;
  }
}

// The same sums with one thread per row running its chain of additions: 43 ns an element whatever
// else runs (a dependent FP64 addition), a row beside the others as long as the pipe has room. For
// many rows or few instances (in_chains).
__global__ void __launch_bounds__(kChainThreads)
    k_sum_instance_chain(const __grid_constant__ SumRowsArgs a, long long n) {
  long long r = static_cast<long long>(blockIdx.x) * kChainThreads + threadIdx.x;
  int g = 0;
  while (g < a.count && r >= a.g[g].rows) r -= a.g[g++].rows;
  if (g >= a.count) return;
  const double* row = a.g[g].src + r * a.g[g].ld;
  double acc = 0.0;
  long long i = 0;
  for (; i + 8 <= n; i += 8) {
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __ldg(row + i + j);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc = __dadd_rn(acc, v[j]);
  }
  for (; i < n; ++i) acc = __dadd_rn(acc, __ldg(row + i));
  a.g[g].dst[r] = acc;
}

// One level of the blocked tree: item (r, b) sums x[r][b*256 .. b*256+255] into y[r][b].
__global__ void __launch_bounds__(kWarpsPerCta * 32)
    k_sum_tree_level(long long rows, long long m, const double* __restrict__ src, long long ld,
                     double* __restrict__ dst, long long dst_ld) {
  const int lane = threadIdx.x & 31;
  const long long nb = (m + kTreeBlock - 1) / kTreeBlock;
  const long long item = static_cast<long long>(blockIdx.x) * kWarpsPerCta + (threadIdx.x >> 5);
  if (item >= rows * nb) return;
  const long long r = item / nb, b = item - r * nb;
  const double* x = src + r * ld + b * kTreeBlock;
  const long long left = m - b * kTreeBlock;
  double acc = 0.0;
#pragma unroll
  for (int k = 0; k < kTreeBlock / 32; ++k) {
    const int i = k * 32 + lane;
    if (i < left) acc = __dadd_rn(acc, __ldg(x + i));
  }
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) acc = __dadd_rn(acc, __shfl_xor_sync(kFull, acc, s));
  if (lane == 0) dst[r * dst_ld + b] = acc;
}

__global__ void __launch_bounds__(kWarpsPerCta * 32)
    k_or_rows(long long rows, long long n, const unsigned long long* __restrict__ src,
              long long ld, unsigned long long* __restrict__ dst, bool accumulate) {
  const int lane = threadIdx.x & 31;
  const long long r = static_cast<long long>(blockIdx.x) * kWarpsPerCta + (threadIdx.x >> 5);
  if (r >= rows) return;
  const unsigned long long* row = src + r * ld;
  unsigned long long acc = 0;
  for (long long i = lane; i < n; i += 32) acc |= __ldg(row + i);
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) acc |= __shfl_xor_sync(kFull, acc, s);
  if (lane == 0) dst[r] = accumulate ? (dst[r] | acc) : acc;
}

__global__ void k_broadcast_rows(long long rows, long long n,
                                 const unsigned long long* __restrict__ src,
                                 unsigned long long* __restrict__ dst, long long ld) {
  const long long total = rows * n;
  for (long long k = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; k < total;
       k += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = k / n, i = k - r * n;
    dst[r * ld + i] = __ldg(src + r);
  }
}

__global__ void k_add_blocks(long long ndir, long long nnz, long long n,
                             const double* __restrict__ a, long long a_nz, long long a_dir,
                             const double* __restrict__ b, double* __restrict__ dst) {
  const long long total = ndir * nnz * n;
  for (long long q = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; q < total;
       q += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long i = q % n, r = q / n, k = r % nnz, d = r / nnz;
    const double* pa = a ? a + d * a_dir + k * a_nz + i : nullptr;
    double v;
    if (pa && b) v = __dadd_rn(__ldg(pa), __ldg(b + q));
    else if (pa) v = __ldg(pa);
    else if (b) v = __ldg(b + q);
    else v = 0.0;
    dst[q] = v;
  }
}

unsigned blocks_for(long long items) {
  const long long b = (items + kWarpsPerCta - 1) / kWarpsPerCta;
  return static_cast<unsigned>(std::max<long long>(1, b));
}

}  // namespace

size_t reduce_scratch_bytes(long long rows, long long n, int order) {
  if (order != kOrderTree) return 0;
  // two ping-pong level buffers; the first level's output is the largest
  const long long nb = (n + kTreeBlock - 1) / kTreeBlock;
  if (nb <= 1) return 0;
  const long long nb2 = (nb + kTreeBlock - 1) / kTreeBlock;
  return static_cast<size_t>(rows) * static_cast<size_t>(nb + nb2) * sizeof(double);
}

cudaError_t reduce_sum(long long rows, long long n, const double* src, long long ld, double* dst,
                       int order, double* scratch, cudaStream_t s) {
  if (rows <= 0) return cudaSuccess;
  if (order == kOrderInstance || n == 0) {  // no instances: +0, as the instance-order sum
    const SumRows one{src, ld, dst, rows};
    return reduce_sum_instance_multi(&one, 1, n, s);
  }
  // tree: levels until one value per row; at least one level (n <= 256 included)
  long long m = n;
  const double* x = src;
  long long x_ld = ld;
  const long long nb1 = (n + kTreeBlock - 1) / kTreeBlock;
  double* buf[2] = {scratch, scratch ? scratch + rows * nb1 : nullptr};
  int which = 0;
  for (;;) {
    const long long nb = (m + kTreeBlock - 1) / kTreeBlock;
    const bool last = nb <= 1;
    double* y = last ? dst : buf[which];
    const long long y_ld = last ? 1 : nb;
    if (!y) return cudaErrorInvalidValue;
    k_sum_tree_level<<<blocks_for(rows * std::max<long long>(nb, 1)), kWarpsPerCta * 32, 0, s>>>(
        rows, m, x, x_ld, y, y_ld);
    if (cudaError_t e = cudaGetLastError()) return e;
    if (last) return cudaSuccess;
    x = y;
    x_ld = y_ld;
    m = nb;
    which ^= 1;
  }
}

// Whether `rows` sums over n instances run as chains of additions, a thread per row, or as scans, a
// CTA per row. A scan costs more the more CTAs share an SM and the longer a sum stays near zero or
// about a power of two, a chain costs its length; with q rows per SM the scan starts where what it
// saves on terms of one sign makes up for what it loses on terms that cancel: from 512 instances at q
// = 1, 1024 q up to q = 16, nowhere past that. In us, chain and scan of terms of one sign (terms that
// cancel): 21 rows, 256 instances 16, 20 (25), 1024: 50, 27 (65), 8192: 360, 56 (410); 304 rows, 2048:
// 143, 46 (123); 608 rows, 4096: 282, 103 (405); 1000 rows, 1024: 76, 83 (205), 8192: 570, 220 (1040);
// 2000 rows, 4096: 285, 303 (1070), 16384: 1730, 570 (3170); 4000 rows, 1024: 76, 269 (690), 16384:
// 1630, 1090 (5980); 64000 rows, 64: 23, 1720 (1890).
bool in_chains(long long rows, long long n) {
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    sms = 1;
  const long long q = (rows + sms - 1) / sms;
  return q > 16 || n < (q == 1 ? 512 : 1024 * q);
}

cudaError_t reduce_sum_instance_multi(const SumRows* groups, int count, long long n,
                                      cudaStream_t s) {
  // at most kMaxSumGroups groups per launch (the launch's parameter block holds them); more
  // groups take more launches, each row's chain being the same
  for (int k0 = 0; k0 < count; k0 += kMaxSumGroups) {
    const int c = std::min(kMaxSumGroups, count - k0);
    SumRowsArgs a;
    long long total = 0;
    for (int k = 0; k < c; ++k) {
      a.g[k] = groups[k0 + k];
      total += groups[k0 + k].rows;
    }
    a.count = c;
    if (total == 0) continue;
    if (in_chains(total, n)) {
      const long long grid = (total + kChainThreads - 1) / kChainThreads;
      k_sum_instance_chain<<<static_cast<unsigned>(grid), kChainThreads, 0, s>>>(a, n);
    } else {
      const unsigned grid = static_cast<unsigned>(std::min<long long>(total, 1 << 20));
      k_sum_instance_order<<<grid, kOrdThreads, 0, s>>>(a, total, n);
    }
    if (cudaError_t e = cudaGetLastError()) return e;
  }
  return cudaSuccess;
}

cudaError_t reduce_or(long long rows, long long n, const unsigned long long* src, long long ld,
                      unsigned long long* dst, bool accumulate, cudaStream_t s) {
  if (rows <= 0) return cudaSuccess;
  k_or_rows<<<blocks_for(rows), kWarpsPerCta * 32, 0, s>>>(rows, n, src, ld, dst, accumulate);
  return cudaGetLastError();
}

cudaError_t broadcast_rows(long long rows, long long n, const unsigned long long* src,
                           unsigned long long* dst, long long ld, cudaStream_t s) {
  if (rows <= 0 || n <= 0) return cudaSuccess;
  const long long total = rows * n;
  const unsigned grid = static_cast<unsigned>(std::min<long long>((total + 255) / 256, 4096));
  k_broadcast_rows<<<grid, 256, 0, s>>>(rows, n, src, dst, ld);
  return cudaGetLastError();
}

cudaError_t add_blocks(long long ndir, long long nnz, long long n, const double* a, long long a_nz,
                       long long a_dir, const double* b, double* dst, cudaStream_t s) {
  const long long total = ndir * nnz * n;
  if (total <= 0) return cudaSuccess;
  const unsigned grid = static_cast<unsigned>(std::min<long long>((total + 255) / 256, 8192));
  k_add_blocks<<<grid, 256, 0, s>>>(ndir, nnz, n, a, a_nz, a_dir, b, dst);
  return cudaGetLastError();
}

}  // namespace cgb
