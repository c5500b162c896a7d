// Exact top-k token selection with forced sink tokens, one score row per CTA.
//
// For every row of fp32 scores (one query group of one head) the kernel returns, in ascending
// index order, the sink tokens plus the (k_total - n_sink) non-sink tokens with the highest score;
// among equal scores the lowest indices win.  The result depends only on the fp32 scores, so it is
// bit-reproducible and can be compared exactly with a stable sort on the host.
//
// Tightens the reference's selection (mcsparse/kernels/flash_mcsa/token_sparse.py:755-945, topk
// mode with sink ranges): that code calls torch.topk(sorted=False) and then truncates the
// concatenation [sinks, topk] to a multiple of 128, which drops an implementation-defined subset;
// here the dropped entries are the lowest-ranked ones and the output is sorted.
//
// Two kernels, chosen by launch_topk_select: the streaming kernel (one sweep over the row, candidates above a sampled
// bound), and for budgets whose candidates do not fit in shared memory the general one described here.
//
// Algorithm of the general kernel, per row (1024 threads):
//   1. map scores to order-preserving 32-bit keys (NaN highest; sinks get key 0, below every real
//      key) and stage the row in shared memory when it fits (<= ~200 KB), else re-read it from L2;
//   2. MSB-first radix select, four 8-bit passes with warp-aggregated shared-memory histograms,
//      finds the key T of the k-th largest element and how many elements equal to T are needed;
//   3. one counting sweep and one writing sweep compact the selected indices in index order with
//      warp ballots: element j is taken if it is a sink, or key > T, or key == T and fewer than
//      `need` equal keys precede it.
#include "kernels.cuh"
#include "ptx.cuh"

namespace mcs {

namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kHistCopies = 8;

__device__ __forceinline__ uint32_t score_key(float s) {
  uint32_t u = __float_as_uint(s);
  if (s != s) return 0xFFFFFFFFu;                         // NaN: above every number, as torch.topk ranks it
  if (s == 0.f) u = 0u;                                   // -0 and +0 rank equal
  u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);          // order-preserving
  return u < 2u ? 2u : u;                                  // keep 0 (sink) and 1 (padding) reserved
}

__device__ __forceinline__ int sink_at(const TopkParams& p, int i) { return p.sinks != nullptr ? p.sinks[i] : p.sink_list.idx[i]; }

struct Shared {
  uint32_t hist[kHistCopies][256];
  uint32_t suffix[256];
  int sinks[kMaxSinks];
  int warp_sel[kWarps], warp_eq[kWarps];
  uint32_t prefix;
  int k_rem;
};

template <bool kStage>
__global__ void __launch_bounds__(kThreads, 1) topk_select_kernel(const __grid_constant__ TopkParams p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  Shared& sh = *reinterpret_cast<Shared*>(smem_raw);
  uint32_t* skeys = reinterpret_cast<uint32_t*>(smem_raw + sizeof(Shared));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int L = p.L, n_sink = p.n_sink;

  if (tid < n_sink) sh.sinks[tid] = sink_at(p, tid);
  __syncthreads();

#pragma unroll 1
  for (long long row = blockIdx.x; row < p.rows; row += gridDim.x) {
    const float* sc = p.scores + row * (long long)L;
    int32_t* out = p.out + row * (long long)p.k_total;
    // this row's budget (sinks included): the common k_total, or its own entry of k_rows
    const int k_row = p.k_rows != nullptr ? min(max(p.k_rows[row], n_sink), p.k_total) : p.k_total;
    const int k = k_row - n_sink;                         // non-sink tokens to pick (>= 0, <= L - n_sink)

    auto is_sink = [&](int j) {
      bool s = false;
      for (int i = 0; i < n_sink; ++i) s |= (sh.sinks[i] == j);
      return s;
    };
    auto key_at = [&](int j) -> uint32_t {
      if (kStage) return skeys[j];
      return is_sink(j) ? 0u : score_key(__ldg(sc + j));
    };

    if (kStage) {
      for (int j = tid; j < L; j += kThreads) skeys[j] = score_key(__ldcs(sc + j));
      __syncthreads();
      if (tid < n_sink) skeys[sh.sinks[tid]] = 0u;
    }
    if (tid == 0) { sh.prefix = 0u; sh.k_rem = k; }
    __syncthreads();

    // ---- radix select: key T of the k-th largest non-sink element
    if (k > 0) {
#pragma unroll 1
      for (int pass = 0; pass < 4; ++pass) {
        const int shift = 24 - 8 * pass;
        for (int i = tid; i < kHistCopies * 256; i += kThreads) (&sh.hist[0][0])[i] = 0u;
        __syncthreads();
        const uint32_t prefix = sh.prefix;
        const uint32_t hi_mask = pass == 0 ? 0u : (0xFFFFFFFFu << (shift + 8));
        uint32_t* hist = sh.hist[warp % kHistCopies];
        for (int j0 = warp * 32; j0 < L; j0 += kThreads) {
          const int j = j0 + lane;
          uint32_t key = 0u;
          if (j < L) key = key_at(j);
          const bool live = (j < L) && key != 0u && ((key & hi_mask) == prefix);
          const uint32_t digit = (key >> shift) & 0xFFu;
          // warp-aggregated histogram update: one atomic per distinct digit in the warp
          const uint32_t livemask = __ballot_sync(0xffffffffu, live);
          if (live) {
            const uint32_t peers = __match_any_sync(livemask, digit);
            if ((peers & ((1u << lane) - 1u)) == 0u) atomicAdd(&hist[digit], (uint32_t)__popc(peers));
          }
        }
        __syncthreads();
        // suffix counts over digits: suffix[d] = number of live keys with digit >= d
        if (tid < 256) {
          uint32_t c = 0;
          for (int i = 0; i < kHistCopies; ++i) c += sh.hist[i][tid];
          sh.suffix[tid] = c;
        }
        __syncthreads();
        for (int off = 1; off < 256; off <<= 1) {
          uint32_t v = 0;
          if (tid < 256 && tid + off < 256) v = sh.suffix[tid + off];
          __syncthreads();
          if (tid < 256) sh.suffix[tid] += v;
          __syncthreads();
        }
        if (tid < 256) {
          const uint32_t ge = sh.suffix[tid];
          const uint32_t gt = tid < 255 ? sh.suffix[tid + 1] : 0u;
          const uint32_t kr = (uint32_t)sh.k_rem;
          if (gt < kr && kr <= ge) {                      // exactly one digit satisfies this
            sh.prefix = prefix | ((uint32_t)tid << shift);
            sh.k_rem = (int)(kr - gt);
          }
        }
        __syncthreads();
      }
    }
    const uint32_t T = sh.prefix;
    const int need = k > 0 ? sh.k_rem : 0;                // how many keys == T to take (lowest indices first)

    // ---- counting sweep: per warp span, how many are certainly selected (sink or > T) and how many equal T
    const int span = ((L + kWarps - 1) / kWarps + 31) & ~31;     // contiguous elements per warp, multiple of 32
    const int lo = warp * span, hi = min(lo + span, L);
    int c_sel = 0, c_eq = 0;
    for (int j0 = lo; j0 < hi; j0 += 32) {
      const int j = j0 + lane;
      uint32_t key = 1u;
      if (j < hi) key = key_at(j);
      const bool in = j < hi;
      c_sel += __popc(__ballot_sync(0xffffffffu, in && (key == 0u || (k > 0 && key > T))));
      c_eq += __popc(__ballot_sync(0xffffffffu, in && k > 0 && key == T && key != 0u));
    }
    if (lane == 0) { sh.warp_sel[warp] = c_sel; sh.warp_eq[warp] = c_eq; }
    __syncthreads();
    int eq_before = 0, out_before = 0, n_out = need;       // (repeated sinks, which the contract excludes: fewer than k_row)
    for (int w = 0; w < kWarps; ++w) {                     // 32 entries: a serial prefix is cheapest
      const int e = sh.warp_eq[w];
      n_out += sh.warp_sel[w];
      if (w >= warp) continue;
      out_before += sh.warp_sel[w] + min(max(need - eq_before, 0), e);
      eq_before += e;
    }
    // ---- writing sweep
    for (int j0 = lo; j0 < hi; j0 += 32) {
      const int j = j0 + lane;
      uint32_t key = 1u;
      if (j < hi) key = key_at(j);
      const bool in = j < hi;
      const bool eq = in && k > 0 && key == T && key != 0u;
      const uint32_t eq_b = __ballot_sync(0xffffffffu, eq);
      const int eq_rank = eq_before + __popc(eq_b & ((1u << lane) - 1u));
      const bool sel = in && (key == 0u || (k > 0 && key > T) || (eq && eq_rank < need));
      const uint32_t sel_b = __ballot_sync(0xffffffffu, sel);
      if (sel) {
        const int pos = out_before + __popc(sel_b & ((1u << lane) - 1u));
        if (pos < k_row) out[pos] = j;
      }
      eq_before += __popc(eq_b);
      out_before += __popc(sel_b);
    }
    for (int i = min(k_row, n_out) + tid; i < p.k_total; i += kThreads) out[i] = 0;      // beyond the row's own budget: padding
    __syncthreads();                                       // shared state is reused by the next row
  }
}


// ------------------------------------------------------------------------------------------
// Streaming kernel: the row is read once, and only candidates are kept.
//
// What bounds the selection is instructions per key, not bytes: a key that goes through a histogram pass costs some
// fifteen of them, and the kernels above take every key through several.  Here a sample of the row (one key in L / 4096)
// gives a lower bound t below the k-th largest key; one sweep over the row then costs a compare and a conditional add
// per key and keeps the (key, index) pairs above t - about 1.4 k of them at k = 4096, L = 98,280.  The exact k-th key is
// found among those by histogram passes of 11 bits, and the ascending output comes from a bitmap of the
// row: one bit per selected index, a scan over the words' population counts, and a staging buffer, so that the order in
// which warps append candidates does not matter.  A row on which the sample misjudges (fewer than k keys above t and
// not the tie group at t itself, or more candidates than fit) is selected by the same passes over global memory: the
// sample decides the time only, never the result.
// Measured (one B200, a loop of calls with four sinks): 3,840 rows of 98,280 keys, k = 4,096: 8,058 -> 640 us (1.57 GB, floor
// 240 us at the measured copy rate).  The sweep itself runs at 5.5 TB/s; the other half of a row's time are the sample and histogram passes.
// ------------------------------------------------------------------------------------------
constexpr int kST = 512;                  // threads of the streaming kernel
constexpr int kSW = kST / 32;
constexpr int kSample = 4096;
constexpr int kSampleAll = 8192;          // rows of up to this length: every key is a candidate, no sample
constexpr int kDigits = 2048;
constexpr int kPrefetch = 128 * 1024;     // bytes of the next row
constexpr int kStreamMaxL = 131072;       // word prefixes are kept as 16-bit numbers in the histogram's space

struct SharedStream {
  uint32_t hist[kDigits];
  uint32_t warp_tot[kSW];
  uint32_t digit, rem, n_eq;              // result of the last histogram search
  uint32_t n_cand, n_dead, n_tie;
  uint32_t key_lo, key_hi;                // smallest and largest candidate key
};

// rank in the sample that lies below rank k of the row by 4.5 standard deviations of the sampling noise
__host__ __device__ inline int sample_rank(int k, int L) {
  const float e = (float)(((long long)k * kSample + L - 1) / L);
  return (int)(e + 4.5f * sqrtf(e) + 4.f);
}

// Finds the digit that holds the kr-th largest of the counted keys (1 <= kr <= their number), how many keys of that
// digit are needed and how many there are; clears the histogram.  All threads; two barriers.
__device__ __forceinline__ void hist_find(SharedStream& sh, uint32_t kr) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint4* h4 = reinterpret_cast<uint4*>(sh.hist);
  const uint4 c = h4[tid];                                   // digits 4 tid .. 4 tid + 3
  h4[tid] = make_uint4(0u, 0u, 0u, 0u);
  const uint32_t s = c.x + c.y + c.z + c.w;
  uint32_t incl = s;                                         // this lane and the lanes above it
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t n = __shfl_down_sync(0xffffffffu, incl, off);
    if (lane + off < 32) incl += n;
  }
  if (lane == 0) sh.warp_tot[warp] = incl;
  __syncthreads();
  const uint32_t w = (lane < kSW && lane > warp) ? sh.warp_tot[lane] : 0u;
  uint32_t gt = __reduce_add_sync(0xffffffffu, w) + incl - s;   // keys with a higher digit than this thread's
  const uint32_t cc[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
  for (int d = 3; d >= 0; --d) {
    const uint32_t ge = gt + cc[d];
    if (gt < kr && kr <= ge) { sh.digit = 4 * tid + d; sh.rem = kr - gt; sh.n_eq = cc[d]; }   // exactly one digit
    gt = ge;
  }
  __syncthreads();
}

// Key of the k-th largest key among those that visit(f) hands to f (key 0: not counted; the others lie in [lo, hi]);
// `need` of the `n_eq` keys equal to it belong to the k largest.  Passes of 11 bits over the bits in which the keys
// differ at all, so that the first histogram already spreads over its bins; at most max_passes (the result is then
// a lower bound: its remaining bits are zero).  Needs a cleared histogram.  (Equal keys cost no more than others: the
// hardware counts the lanes of an increment that hit one bin together.)
template <typename Visit>
__device__ __forceinline__ void kth_key(SharedStream& sh, uint32_t k, uint32_t lo, uint32_t hi, int max_passes, Visit visit, uint32_t& T,
                                        uint32_t& need, uint32_t& n_eq) {
  const int bits = 32 - __clz((int)(hi - lo));
  int above = 32;                                            // bits from here up are decided (32: all keys match)
  int shift = bits > 11 ? bits - 11 : 0;
  uint32_t prefix = 0u;
#pragma unroll 1
  for (int pass = 0; pass < max_passes; ++pass) {
    visit([&](uint32_t key) {
      const uint32_t x = key - lo;
      const bool live = key != 0u && (above == 32 || (x >> above) == prefix);
      const uint32_t digit = above == 32 ? x >> shift : (x >> shift) & ((1u << (above - shift)) - 1u);
      if (live) atomicAdd(&sh.hist[digit], 1u);
    });
    __syncthreads();
    hist_find(sh, k);
    prefix = (above == 32 ? 0u : prefix << (above - shift)) | sh.digit;
    k = sh.rem;
    above = shift;
    if (shift == 0) break;
    shift = shift > 11 ? shift - 11 : 0;
  }
  T = lo + (prefix << above);
  need = k;
  n_eq = sh.n_eq;
}

// Exclusive block-wide scan; two barriers (the second keeps warp_tot stable until everyone has read it).
__device__ __forceinline__ uint32_t stream_scan_excl(SharedStream& sh, uint32_t v) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t n = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += n;
  }
  if (lane == 31) sh.warp_tot[warp] = incl;
  __syncthreads();
  const uint32_t w = lane < warp ? sh.warp_tot[lane] : 0u;      // warp < kSW
  const uint32_t base = __reduce_add_sync(0xffffffffu, w);
  __syncthreads();
  return base + incl - v;
}

// kCtas CTAs per SM with kSU 16-byte loads per thread in flight (and as many being processed): 3 with 2 or, where a
// row's candidates take more than a third of shared memory, 2 with 4.
template <int kCtas, int kSU>
__global__ void __launch_bounds__(kST, kCtas) topk_stream_kernel(const __grid_constant__ TopkParams p, int cap, int words) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  SharedStream& sh = *reinterpret_cast<SharedStream*>(smem_raw);
  uint32_t* ckeys = reinterpret_cast<uint32_t*>(smem_raw + sizeof(SharedStream));   // [cap] candidates; later the output
  int* cidx = reinterpret_cast<int*>(ckeys + cap);                                  // [cap]
  uint32_t* bm = reinterpret_cast<uint32_t*>(cidx + cap);                           // [words] one bit per key of the row
  uint16_t* prefix16 = reinterpret_cast<uint16_t*>(sh.hist);                        // [words] during the write-out
  const int tid = threadIdx.x, lane = tid & 31;
  const int L = p.L, n_sink = p.n_sink;
  const int wpt = (words + kST - 1) / kST;                       // contiguous bitmap words per thread in the scans
  auto set_bit = [&](int j) { atomicOr(&bm[j >> 5], 1u << (j & 31)); };

#pragma unroll 1
  for (long long row = blockIdx.x; row < p.rows; row += gridDim.x) {
    const float* sc = p.scores + row * (long long)L;
    int32_t* out = p.out + row * (long long)p.k_total;
    const int k_row = p.k_rows != nullptr ? min(max(p.k_rows[row], n_sink), p.k_total) : p.k_total;
    const int k = k_row - n_sink;
    for (int i = tid; i < kDigits; i += kST) sh.hist[i] = 0u;
    for (int i = tid; i < words; i += kST) bm[i] = 0u;
    if (tid == 0) { sh.n_cand = 0u; sh.n_dead = 0u; sh.n_tie = 0u; sh.key_lo = 0xFFFFFFFFu; sh.key_hi = 0u; }
    __syncthreads();
    if (tid < n_sink) set_bit(sink_at(p, tid));                  // until the end of the row: bit set == sink
    __syncthreads();
    auto is_sink = [&](int j) { return ((bm[j >> 5] >> (j & 31)) & 1u) != 0u; };

    if (k > 0) {
      // ---- 1. lower bound t: candidates are the keys above it (NaN included)
      uint32_t t_key = 0u;
      float t = -INFINITY;
      const int r_s = sample_rank(k, L);
      bool sampled = L > kSampleAll && r_s < kSample;
      if (sampled) {
        uint32_t s[kSample / kST];
#pragma unroll
        for (int u = 0; u < kSample / kST; ++u) s[u] = __float_as_uint(__ldg(sc + (int)(((long long)(u * kST + tid) * L) >> 12)));
#pragma unroll
        for (int u = 0; u < kSample / kST; ++u) {
          const uint32_t key = score_key(__uint_as_float(s[u]));
          s[u] = is_sink((int)(((long long)(u * kST + tid) * L) >> 12)) ? 2u : key;
        }
        uint32_t need, n_eq;
        kth_key(sh, (uint32_t)r_s, 0u, 0xFFFFFFFFu, 2, [&](auto f) {
#pragma unroll
          for (int u = 0; u < kSample / kST; ++u) f(s[u]);
        }, t_key, need, n_eq);
        t = __uint_as_float((t_key & 0x80000000u) ? (t_key & 0x7FFFFFFFu) : ~t_key);
        if (t != t) { t = -INFINITY; sampled = false; }          // the bound fell among the NaNs: no bound
      }
      // ---- 2. one sweep over the row: aligned 16-byte loads (the row may start at any element; the chunks that reach
      // beyond it are read element by element), the next kSU loads in flight while the current ones are processed
      const int o = (int)((reinterpret_cast<uintptr_t>(sc) >> 2) & 3);
      const int nch = (o + L + 3) >> 2;
      auto load = [&](int c) -> float4 {
        if (4 * c >= o && 4 * c + 4 <= o + L) return __ldcs(reinterpret_cast<const float4*>(sc - o) + c);
        float4 f = make_float4(t, t, t, t);                      // t itself is no candidate
        const int j = 4 * c - o;
        if (j >= 0 && j < L) f.x = sc[j];
        if (j + 1 >= 0 && j + 1 < L) f.y = sc[j + 1];
        if (j + 2 >= 0 && j + 2 < L) f.z = sc[j + 2];
        if (j + 3 >= 0 && j + 3 < L) f.w = sc[j + 3];
        return f;
      };
      float4 nx[kSU];
#pragma unroll
      for (int u = 0; u < kSU; ++u) nx[u] = load(u * kST + tid);
#pragma unroll 1
      for (int c0 = 0; c0 < nch; c0 += kST * kSU) {
        float4 v[kSU];
#pragma unroll
        for (int u = 0; u < kSU; ++u) v[u] = nx[u];
        if (c0 + kST * kSU < nch) {
#pragma unroll
          for (int u = 0; u < kSU; ++u) nx[u] = load(c0 + kST * kSU + u * kST + tid);
        }
        uint32_t cnt = 0;
#pragma unroll
        for (int u = 0; u < kSU; ++u)
          cnt += (v[u].x <= t ? 0u : 1u) + (v[u].y <= t ? 0u : 1u) + (v[u].z <= t ? 0u : 1u) + (v[u].w <= t ? 0u : 1u);
        uint32_t incl = cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const uint32_t n = __shfl_up_sync(0xffffffffu, incl, off);
          if (lane >= off) incl += n;
        }
        uint32_t base = 0;
        if (lane == 31) base = atomicAdd(&sh.n_cand, incl);
        uint32_t pos = __shfl_sync(0xffffffffu, base, 31) + incl - cnt;
        if (cnt != 0u && pos + cnt <= (uint32_t)cap) {           // (an overflow shows in n_cand)
#pragma unroll
          for (int u = 0; u < kSU; ++u) {
            const int j = 4 * (c0 + u * kST + tid) - o;
            const float f[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (!(f[e] <= t)) { ckeys[pos] = __float_as_uint(f[e]); cidx[pos] = j + e; ++pos; }
          }
        }
      }
      // the start of this CTA's next row comes into L2 while this one is worked on in shared memory
      if (row + gridDim.x < p.rows) {
        const uint8_t* nr = reinterpret_cast<const uint8_t*>(sc + (long long)gridDim.x * L);
        for (int i = tid * 128; i < min(4 * L, kPrefetch); i += kST * 128) prefetch_l2(nr + i);
      }
      __syncthreads();
      // ---- 3. the exact k-th key
      const uint32_t C = sh.n_cand;
      uint32_t T = 0u, need = 0u, n_eq = 0u;
      bool from_row = false, tie = false;
      uint32_t live = 0;
      if (C <= (uint32_t)cap) {
        uint32_t lo = 0xFFFFFFFFu, hi = 0u;
        for (int i = tid; i < (int)C; i += kST) {                // sinks are no candidates; the others get their key
          if (is_sink(cidx[i])) {
            ckeys[i] = 0u;
            atomicAdd(&sh.n_dead, 1u);
          } else {
            const uint32_t key = score_key(__uint_as_float(ckeys[i]));
            ckeys[i] = key;
            lo = min(lo, key);
            hi = max(hi, key);
          }
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) { atomicMin(&sh.key_lo, lo); atomicMax(&sh.key_hi, hi); }
        __syncthreads();
        live = C - sh.n_dead;
      }
      // f(index, key) for the whole row, by whole warps (key 0 beyond its end), four loads of a thread in flight: what bounds these
      // passes is the latency of L2
      auto visit_row = [&](auto f) {
#pragma unroll 1
        for (int j0 = tid & ~31; j0 < L; j0 += 4 * kST) {
          float v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) { const int j = j0 + u * kST + lane; v[u] = j < L ? __ldg(sc + j) : 0.f; }
#pragma unroll
          for (int u = 0; u < 4; ++u) { const int j = j0 + u * kST + lane; f(j, j < L ? score_key(v[u]) : 0u); }
        }
      };
      auto ranked = [&](int j, uint32_t key) { return key == 0u || is_sink(j) ? 0u : key; };
      if (live >= (uint32_t)k) {
        kth_key(sh, (uint32_t)k, sh.key_lo, sh.key_hi, 3, [&](auto f) { for (int i = tid; i < (int)C; i += kST) f(ckeys[i]); }, T, need, n_eq);
      } else {
        from_row = true;
        if (sampled && C <= (uint32_t)cap) {
          // a tie group on the bound itself (masses that underflow to zero): the k-th key is t
          uint32_t n = 0;
          visit_row([&](int j, uint32_t key) { n += (key == t_key && !is_sink(j)) ? 1u : 0u; });
          n = __reduce_add_sync(0xffffffffu, n);
          if (lane == 0) atomicAdd(&sh.n_tie, n);
          __syncthreads();
          n_eq = sh.n_tie;
          tie = live + n_eq >= (uint32_t)k;
          T = t_key;
          need = (uint32_t)k - live;
        }
        if (!tie)
          kth_key(sh, (uint32_t)k, 0u, 0xFFFFFFFFu, 3, [&](auto f) { visit_row([&](int j, uint32_t key) { f(ranked(j, key)); }); }, T, need, n_eq);
      }
      // ---- 4. bitmap of the selected keys: above T, and the `need` lowest indices among those equal to T
      auto mark = [&](bool above, bool equal) {
        // (keys of the row are compared without the sink test, whose bits may be gone: a sink belongs to the result; a tie
        // group on the bound: the keys above it are the candidates)
        if (from_row && (equal || !tie))
          visit_row([&](int j, uint32_t key) {                   // one word of the bitmap per warp and step
            const uint32_t word = __ballot_sync(0xffffffffu, (above && key > T) || (equal && key == T));
            if (lane == 0 && word != 0u) atomicOr(&bm[j >> 5], word);
          });
        if (!from_row || (tie && above)) {
          for (int i = tid; i < (int)C; i += kST) {
            const uint32_t key = ckeys[i];
            if ((above && key > T) || (equal && key == T)) set_bit(cidx[i]);
          }
        }
      };
      if (need == n_eq) {
        mark(true, true);
      } else {
        __syncthreads();
        for (int i = tid; i < words; i += kST) bm[i] = 0u;
        __syncthreads();
        mark(false, true);
        __syncthreads();
        if (from_row) {                                          // a sink that equals T takes no part in the ranking
          if (tid < n_sink) atomicAnd(&bm[sink_at(p, tid) >> 5], ~(1u << (sink_at(p, tid) & 31)));
          __syncthreads();
        }
        uint32_t n = 0;
        for (int i = 0; i < wpt; ++i) { const int w = tid * wpt + i; if (w < words) n += __popc(bm[w]); }
        uint32_t before = stream_scan_excl(sh, n);
        for (int i = 0; i < wpt; ++i) {
          const int w = tid * wpt + i;
          if (w >= words) break;
          uint32_t b = bm[w];
          const uint32_t c = __popc(b);
          uint32_t keep = before >= need ? 0u : min(need - before, c);
          uint32_t r = 0u;
          for (; keep > 0u; --keep) { const uint32_t low = b & (0u - b); r |= low; b ^= low; }
          bm[w] = r;
          before += c;
        }
        __syncthreads();
        mark(true, false);
        if (tid < n_sink) set_bit(sink_at(p, tid));
      }
      __syncthreads();
    }
    // ---- 5. write-out: output position of every bitmap word's first bit, then one word per lane, staged so that the
    // global stores are consecutive
    {
      uint32_t n = 0;
      for (int i = 0; i < wpt; ++i) { const int w = tid * wpt + i; if (w < words) n += __popc(bm[w]); }
      uint32_t before = stream_scan_excl(sh, n);
      for (int i = 0; i < wpt; ++i) {
        const int w = tid * wpt + i;
        if (w >= words) break;
        prefix16[w] = (uint16_t)before;
        before += __popc(bm[w]);
      }
      if (tid == kST - 1) sh.rem = before;                         // indices in all
      __syncthreads();
      const int n_out = min(k_row, (int)sh.rem);                   // (repeated sinks, which the contract excludes: fewer than k_row)
      for (int w = tid; w < words; w += kST) {
        uint32_t b = bm[w];
        int pos = prefix16[w];
        while (b != 0u) {
          if (pos < n_out) ckeys[pos] = (uint32_t)(w * 32 + __ffs((int)b) - 1);
          ++pos;
          b &= b - 1u;
        }
      }
      __syncthreads();
      for (int i = tid; i < p.k_total; i += kST) out[i] = i < n_out ? (int)ckeys[i] : 0;   // beyond the row's budget: padding
    }
  }
}

}  // namespace

constexpr size_t kStreamSmemLimit = 224 * 1024;

size_t topk_stage_limit_bytes() { return 200 * 1024; }

int launch_topk_select(const TopkParams& p, cudaStream_t stream) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // Streaming path whenever the candidates that the sampled bound lets through fit in shared memory beside the bitmap, even
  // if only one CTA fits.  Against the kernels it replaced (general above 32,768 keys, a register-resident one below), masses
  // with a tenth of zeros, no sinks, device time of a replayed graph in us:
  //   rows x keys, k          before   streaming        rows x keys, k          before   streaming
  //   3,840 x 98,280, 4,096    6,353     637            6,144 x 32,760, 2,048     882     457
  //   2,000 x 98,280, 8,192    3,447     561            6,144 x 32,760, 8,192   4,575     759
  //   1,500 x 60,000, 13,000   1,680     431            3,000 x 32,760, 20,000  2,350     861
  //   444 x 4,700, 1,280          67      23            1,024 x 16,380, 1,664     143      59
  // (three CTAs per SM with two loads each against two with four, in an earlier loop of calls: 480 / 491 at 32,760 keys, 58 / 65
  // at 4,700; where only two fit, four loads win: 673 / 723 at 98,280).  Beyond it the general kernel: 2,000 x 32,760,
  // k = 28,000 in 638.  What the sample cannot help with is dearer than on the staged row of the general kernel where one CTA
  // fits: 600 x 40,000, k = 20,000 on rows of one single value 468 (273 there), of values 1e-5 apart 435 (373), on ramps 275 (244).
  if (p.L <= kStreamMaxL) {
    const int k = p.k_total - p.n_sink;
    const bool all = p.L <= kSampleAll;
    const int r_s = sample_rank(k > 0 ? k : 1, p.L);
    long long cap = p.L;
    if (!all) {
      // five standard deviations above the expected number, and 6% for the bound's truncation to 22 bits
      const double c = (r_s + 5.0 * sqrt((double)r_s) + 8.0) * p.L / kSample * 1.06 + 64.0;
      cap = (long long)c < p.L ? (long long)c : p.L;
    }
    cap = (cap + 3) & ~3ll;
    const int words = (p.L + 31) / 32;
    const size_t smem = sizeof(SharedStream) + (size_t)cap * 8 + (size_t)words * 4;
    if ((all || r_s < kSample) && smem <= kStreamSmemLimit) {
      const bool three = smem <= kStreamSmemLimit / 3;
      auto kern = three ? topk_stream_kernel<3, 2> : topk_stream_kernel<2, 4>;
      // (the limit, not this launch's size: another thread may launch the same kernel with another size in between)
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStreamSmemLimit) != cudaSuccess) return -8;
      const long long slots = (long long)(three ? 3 : smem <= kStreamSmemLimit / 2 ? 2 : 1) * sms;
      kern<<<(unsigned)(p.rows < slots ? p.rows : slots), kST, smem, stream>>>(p, (int)cap, words);
      return cudaGetLastError() == cudaSuccess ? 0 : -8;
    }
  }
  const size_t row_bytes = (size_t)p.L * 4;
  const bool stage = row_bytes <= topk_stage_limit_bytes();
  const size_t smem = sizeof(Shared) + (stage ? row_bytes : 0);
  const int grid = (int)(p.rows < (long long)sms ? p.rows : sms);
  if (stage) {
    if (cudaFuncSetAttribute(topk_select_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(Shared) + topk_stage_limit_bytes())) != cudaSuccess)
      return -8;
    topk_select_kernel<true><<<grid, kThreads, smem, stream>>>(p);
  } else {
    topk_select_kernel<false><<<grid, kThreads, smem, stream>>>(p);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -8;
}

}  // namespace mcs
