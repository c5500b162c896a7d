// Variable-length token selection: how many tokens a query group needs to cover a probability mass.
//
// For every row of fp32 scores (the normalised mass of one query group over all key tokens, sink tokens
// excluded) the kernel returns
//     count = #{ i : sum of all scores ranked strictly before i  <  topp },   ranking by descending score,
// i.e. the length of the shortest prefix of the descending order whose mass reaches topp (everything if the
// whole row stays below it, at least one).  That is the reference's top-p rule
// (mcsparse/kernels/flash_mcsa/token_sparse.py:842-876: sort, cumulative sum, mask cumsum_before < topp, count),
// without sorting: three histogram passes over the order-preserving 32-bit image of the scores (11, 11 and 10 bits,
// most significant first) narrow down the key at which the mass of the keys above it passes topp; ties on that key enter
// one by one until the mass is reached.  The selection itself (which tokens) is done by the top-k kernel with this
// count as the row's budget.
//
// A histogram bin holds its number of scores and their exact mass: the 11 bits of the first pass contain sign and
// exponent, so all scores of a bin are whole multiples of one power of two, and their 24-bit significands are added
// as integers (two halves of 12 bits in 32-bit words: no overflow up to 2^20 scores, 64-bit words beyond).  Integer sums do
// not depend on the order of the atomics, so the result is reproducible; bins are combined in fp64.
//
// What bounds it: the atomics of the first pass (three per score).  Two copies of the histogram (even and odd lanes)
// halve the collisions inside a warp; one 64-bit add per score in their place is a loop in shared memory and twice as slow
// (168 us against 96 in a loop of launches).  1,024 rows of 16,380 scores: 125 us (the bisection that came before, seventeen
// sweeps with three compares per score, took 644 us; one read of the scores at the copy rate: 10 us).
#include <type_traits>

#include "kernels.cuh"
#include "ptx.cuh"

namespace mcs {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kDigits = 2048;

__device__ __forceinline__ uint32_t prob_key(float s) {
  uint32_t u = __float_as_uint(s);
  if (s != s) return 0u;                                   // NaN carries no mass and ranks last
  if (s == 0.f) u = 0u;
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);       // order-preserving
}
__device__ __forceinline__ uint32_t key_bits(uint32_t k) { return (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k; }

// kBig: rows of more than 2^20 scores
template <bool kBig>
struct Shared {
  using Acc = typename std::conditional<kBig, unsigned long long, unsigned int>::type;
  static constexpr int kCopies = kBig ? 1 : 2;
  unsigned int cnt[kCopies][kDigits];
  Acc lo[kCopies][kDigits], hi[kCopies][kDigits];          // sums of the lower and upper 12 bits of the significands
  double warp_sum[kWarps];
  unsigned int warp_cnt[kWarps];
  int best, lowest;
  double s_above;
  unsigned int n_above, n_eq;
};

template <bool kBig>
__global__ void __launch_bounds__(kThreads) topp_count_kernel(const float* __restrict__ scores, const int32_t* __restrict__ sinks,
                                                             const __grid_constant__ SinkList sink_list, int n_sink, long long rows, int L,
                                                             float topp, int32_t* __restrict__ counts) {
  using S = Shared<kBig>;
  using Acc = typename S::Acc;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  S& sh = *reinterpret_cast<S*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int copy = lane & (S::kCopies - 1);
  for (int i = tid; i < S::kCopies * kDigits; i += kThreads) {
    sh.cnt[0][i] = 0u;                                     // (the copies are contiguous)
    sh.lo[0][i] = 0;
    sh.hi[0][i] = 0;
  }
  if (tid == 0) { sh.best = -1; sh.lowest = kDigits; }
  __syncthreads();
#pragma unroll 1
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float* sc = scores + row * (long long)L;
    uint32_t prefix = 0u, mask = 0u;
    double s_base = 0.0;                                   // mass and number of the scores above the current prefix
    unsigned int n_base = 0u, n_eq = 0u;
    bool all = false;
#pragma unroll 1
    for (int pass = 0; pass < 3; ++pass) {
      const int shift = pass == 0 ? 21 : (pass == 1 ? 10 : 0);
      const uint32_t dm = pass == 2 ? 1023u : 2047u;
      // sign: +1 adds a score, -1 (modulo 2^32 or 2^64) takes it out again
      auto count = [&](float v, unsigned int sign) {
        const uint32_t key = prob_key(v);
        if ((key & mask) != prefix) return;
        const uint32_t d = (key >> shift) & dm;
        const uint32_t u = __float_as_uint(v);
        uint32_t m = (u & 0x7FFFFFu) | ((u & 0x7F800000u) != 0u ? 0x800000u : 0u);
        if (v != v) m = 0u;
        atomicAdd(&sh.cnt[copy][d], sign);
        if (m != 0u) {
          atomicAdd(&sh.lo[copy][d], sign == 1u ? (Acc)(m & 0xFFFu) : (Acc)0 - (Acc)(m & 0xFFFu));
          atomicAdd(&sh.hi[copy][d], sign == 1u ? (Acc)(m >> 12) : (Acc)0 - (Acc)(m >> 12));
        }
      };
#pragma unroll 8
      for (int j = tid; j < L; j += kThreads) count(__ldg(sc + j), 1u);
      for (int i = tid; i < n_sink; i += kThreads) count(__ldg(sc + (sinks != nullptr ? sinks[i] : sink_list.idx[i])), 0xFFFFFFFFu);   // not ranked
      __syncthreads();
      // thread t owns digits 4 t .. 4 t + 3: their counts and masses, then the totals above them
      unsigned int c[4], c_sum = 0u;
      double s[4], s_sum = 0.0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int d = 4 * tid + i;
        unsigned int cc = 0u;
        Acc lo = 0, hi = 0;
#pragma unroll
        for (int q = 0; q < S::kCopies; ++q) {
          cc += sh.cnt[q][d]; lo += sh.lo[q][d]; hi += sh.hi[q][d];
          sh.cnt[q][d] = 0u; sh.lo[q][d] = 0; sh.hi[q][d] = 0;
        }
        c[i] = cc;
        const double m = (double)lo + 4096.0 * (double)hi;               // exact: below 2^53
        const uint32_t u = key_bits(prefix | ((uint32_t)d << shift));    // any key of the bin has its sign and exponent
        const int e = (int)((u >> 23) & 0xFFu);
        double v = 0.0;
        if (m != 0.0) v = e == 255 ? (double)INFINITY : scalbn(m, (e == 0 ? 1 : e) - 150);
        s[i] = (u & 0x80000000u) ? -v : v;
        c_sum += c[i];
        s_sum += s[i];
      }
      unsigned int c_incl = c_sum;
      double s_incl = s_sum;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned int cn = __shfl_down_sync(0xffffffffu, c_incl, off);
        const double sn = __shfl_down_sync(0xffffffffu, s_incl, off);
        if (lane + off < 32) { c_incl += cn; s_incl += sn; }
      }
      // exclusive totals of the lanes above
      unsigned int c_gt = __shfl_down_sync(0xffffffffu, c_incl, 1);
      double s_gt = __shfl_down_sync(0xffffffffu, s_incl, 1);
      if (lane == 31) { c_gt = 0u; s_gt = 0.0; }
      if (lane == 0) { sh.warp_cnt[warp] = c_incl; sh.warp_sum[warp] = s_incl; }
      __syncthreads();
      double s_hi = 0.0;
      for (int w = kWarps - 1; w > warp; --w) { c_gt += sh.warp_cnt[w]; s_hi += sh.warp_sum[w]; }
      s_gt += s_hi + s_base;
      c_gt += n_base;
      // the highest digit at which the mass reaches topp
      int mine = -1, low = kDigits;
      double s_mine = 0.0, s_run = s_gt;
      unsigned int n_mine = 0u, eq_mine = 0u, n_run = c_gt, n_low = 0u, eq_low = 0u;
      double s_low = 0.0;
#pragma unroll
      for (int i = 3; i >= 0; --i) {
        if (c[i] != 0u) { low = 4 * tid + i; s_low = s_run; n_low = n_run; eq_low = c[i]; }
        if (mine < 0 && c[i] != 0u && s_run + s[i] >= (double)topp) { mine = 4 * tid + i; s_mine = s_run; n_mine = n_run; eq_mine = c[i]; }
        s_run += s[i];
        n_run += c[i];
      }
      if (mine >= 0) atomicMax(&sh.best, mine);
      if (low < kDigits) atomicMin(&sh.lowest, low);
      __syncthreads();
      const int best = sh.best, lowest = sh.lowest;
      all = pass == 0 && best < 0;                         // the whole row stays below topp
      // (after the first pass the mass is known to be reached inside the prefix; if the last bit of an fp64 sum says
      // otherwise, it is at the lowest key)
      if (best >= 0 ? mine == best : low == lowest) {
        sh.s_above = best >= 0 ? s_mine : s_low;
        sh.n_above = best >= 0 ? n_mine : n_low;
        sh.n_eq = best >= 0 ? eq_mine : eq_low;
      }
      __syncthreads();
      if (tid == 0) { sh.best = -1; sh.lowest = kDigits; }
      s_base = sh.s_above;
      n_base = sh.n_above;
      n_eq = sh.n_eq;
      __syncthreads();
      if (all) break;
      prefix |= (uint32_t)(best >= 0 ? best : lowest) << shift;
      mask |= dm << shift;
    }
    if (tid == 0) {
      const unsigned int cap = (unsigned int)(L - n_sink);
      unsigned int n = cap;
      if (!all) {
        const double v = (double)__uint_as_float(key_bits(prefix));
        unsigned int take = n_eq;                          // ties enter one by one while the mass before them is below topp
        if (v > 0.0) {
          const double cn = ceil(((double)topp - s_base) / v);
          take = cn < 1.0 ? 1u : (cn > (double)n_eq ? n_eq : (unsigned int)cn);
        }
        n = n_base + take;
        if (n < 1u) n = 1u;
        if (n > cap) n = cap;
      }
      counts[row] = (int32_t)n;
    }
  }
}

template <bool kBig>
int launch(const float* scores, const int32_t* sinks, const SinkList& sink_list, int n_sink, long long rows, int L, float topp,
           int32_t* counts, cudaStream_t stream) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int smem = (int)sizeof(Shared<kBig>);
  if (cudaFuncSetAttribute(topp_count_kernel<kBig>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -8;
  const long long grid = rows < (long long)sms * 4 ? rows : (long long)sms * 4;
  topp_count_kernel<kBig><<<(unsigned)grid, kThreads, smem, stream>>>(scores, sinks, sink_list, n_sink, rows, L, topp, counts);
  return cudaGetLastError() == cudaSuccess ? 0 : -8;
}

}  // namespace

int launch_topp_count(const float* scores, const int32_t* sinks, const SinkList& sink_list, int n_sink, long long rows, int L, float topp,
                      int32_t* counts, cudaStream_t stream) {
  if (rows == 0) return 0;
  return L <= (1 << 20) ? launch<false>(scores, sinks, sink_list, n_sink, rows, L, topp, counts, stream)
                        : launch<true>(scores, sinks, sink_list, n_sink, rows, L, topp, counts, stream);
}

namespace {

// Budgets of the variable-length modes from the ranked counts (token_sparse.py:811-823, :902-923): whole tiles of ranked
// tokens, plus the sinks, to whole tiles again.  One CTA: the largest count of all rows bounds every row, and the rows are
// few (one per query group).  As elementwise torch operations this was fifteen launches and two waits of the host.
__global__ void __launch_bounds__(1024) selection_budgets_kernel(const int32_t* base, const int32_t* floor_rows, int floor_all, long long rows,
                                                                 int L, int n_sink, int tile, int32_t* budgets, int32_t* tiles, int32_t* k_max) {
  __shared__ int warp_max[32];
  const int tid = threadIdx.x;
  auto up = [&](long long v) { return (v + tile - 1) / tile * tile; };
  auto ranked = [&](long long i) -> long long {
    const int c = max(max(base[i], floor_rows != nullptr ? floor_rows[i] : floor_all), 1);
    return min(up(c), (long long)L);
  };
  int m = 0;
  for (long long i = tid; i < rows; i += 1024) m = max(m, (int)ranked(i));
  m = __reduce_max_sync(0xffffffffu, m);
  if ((tid & 31) == 0) warp_max[tid >> 5] = m;
  __syncthreads();
  m = 0;
  for (int w = 0; w < 32; ++w) m = max(m, warp_max[w]);
  const long long avail = (long long)m + n_sink;            // length of [sinks, longest ranked prefix]
  const long long cap = max((long long)tile, min(up(L), avail / tile * tile));
  auto budget = [&](long long c) {
    if (n_sink > 0) c = min(up(c + n_sink), avail);
    c = min(max(c, (long long)tile), cap);
    return (int)min(c / tile * tile, (long long)L);
  };
  for (long long i = tid; i < rows; i += 1024) {
    const int b = budget(ranked(i));
    budgets[i] = b;
    tiles[i] = b / tile;
  }
  if (tid == 0) *k_max = budget(m);                          // budgets grow with the count
}

}  // namespace

int launch_selection_budgets(const int32_t* base, const int32_t* floor_rows, int floor_all, long long rows, int L, int n_sink, int tile,
                             int32_t* budgets, int32_t* tiles, int32_t* k_max, cudaStream_t stream) {
  selection_budgets_kernel<<<1, 1024, 0, stream>>>(base, floor_rows, floor_all, rows, L, n_sink, tile, budgets, tiles, k_max);
  return cudaGetLastError() == cudaSuccess ? 0 : -8;
}

}  // namespace mcs
