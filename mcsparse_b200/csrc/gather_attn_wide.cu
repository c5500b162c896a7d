// Gather-KV sparse flash-attention forward for the head dimensions the main kernel has no instantiation for:
// any multiple of 8 up to 256 other than 64 and 128 (96, 144, 160, 192, 256 ...) for bf16 / fp16, and any multiple
// of 16 up to 256 other than 128 for e4m3 (the reference's FP8 kernel lists 128 and 160).
//
// The reference pads 144 to 160 in its wrapper and keeps one compiled kernel per padded size
// (mcsparse/kernels/flash_mcsa/ops/flash_sparse_attn/cute/interface.py:45-74, :138-159).  Here the padding happens
// on the way into shared memory: a row is copied in 16-byte chunks into NB = ceil(row bytes / 128) swizzled column
// blocks and the chunks beyond the row are zero-filled, so no padded copy of Q, K or V exists in global memory.
//
// Same math and the same argument block as the main kernel (gather_attn.cu); less room: with D = 256 a K or V tile is 64 KB
// and the output accumulator takes 256 of the 512 tensor-memory columns.  One CTA per work item (one query group of one
// (batch, head)), 13 warps:
//   warps 0-7   softmax and epilogue: thread == query row == tensor-memory lane, warps w and w + 4 share their rows and take
//               the column halves 0-63 and 64-127 of every tile; they agree on one running maximum by a two-warp
//               barrier-with-OR per tile, as in the main kernel (e4m3: a second barrier hands the lower half's row sums to the
//               upper half)
//   warps 8-11  producers: 16-byte cp.async row gathers of Q, then K(0), K(1), V(0), K(2), V(1), ... into a ring
//               of 2-5 tile slots
//   warp 12     issues S = Q K^T (SS) and O += P V (P from tensor memory, V as an MN-major operand) in the order
//               QK(0), QK(1), PV(0), QK(2), PV(1), ...
// Tensor memory: two score buffers of 128 columns, O up to 256.  P overwrites the scores it was computed from (each half in
// its own columns); products execute in order, so Q K^T of tile g+2 may be issued right behind the P V of tile g that reads P
// out of the same buffer.  The softmax of tile g+1 thus finds its scores ready and never waits for a product.
// What bounds it: the softmax of a tile (two warps per sub-partition) and the row gather, 256 rows of 2 D bytes per tile.
// With four softmax warps over whole rows and one score buffer a tile took 4,900 cycles at every head dimension.
// Measured (8 heads x 20,475 tokens, 3,072 selected, permutation and residual; device time of a replayed graph): D = 144
// 535 -> 420 us (290 GFLOP; 176 us at the measured burst rate), 32 287 -> 253, 96 375 -> 325, 160 533 -> 482, 192 541 -> 515,
// 256 660 -> 641; e4m3 16 265 -> 263, 96 334 -> 305, 160 394 -> 354, 256 426 -> 388 (two less at 160 with the reference point
// by half rows, which gives other outputs).
// Every mbarrier wait is bounded and reports through the status word; a role whose wait expires leaves its loop, the others
// follow through their own bounded waits.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "kernels.cuh"
#include "ptx.cuh"

namespace mcs {

namespace {

constexpr int kTileN = 128;
constexpr int kThreadsW = 416;
constexpr int kProducerWarp0W = 8;
constexpr int kProducerThreadsW = 128;
constexpr int kMmaWarpW = 12;
constexpr uint32_t kColSW = 0, kColOW = 256;      // S[buf] at 128 * buf; P of half x in S[buf] at 64 * x

enum {
  WB_FULL = 0,              // [5] producers -> issuer
  WB_EMPTY = 5,             // [5] issuer -> producers
  WB_Q_FULL = 10,
  WB_S_FULL,                // [2] scores of a tile complete
  WB_P_READY = WB_S_FULL + 2,   // [2] probabilities of a tile stored
  WB_PV_DONE = WB_P_READY + 2,  // P V of a tile complete: O stable
  WB_O_FULL,                    // the last P V complete
  WB_DRAIN,
  WB_COUNT
};

template <int NB>
struct SmemW {
  static constexpr int kTileBytes = NB * 16384;                // 128 rows x NB column blocks of 128 bytes
  static constexpr int kRing = NB <= 2 ? 5 : (NB == 3 ? 3 : 2);
  static constexpr int kQ = 0;
  static constexpr int kRingOff = kTileBytes;
  static constexpr int kBars = kRingOff + kRing * kTileBytes;
  static constexpr int kXch = kBars + WB_COUNT * 8;            // float [2 halves][128]: tile maxima, exchanged on a raise
  static constexpr int kChain = kXch + 1024;                   // float4 [128]: the four running sums of the lower half (e4m3)
  static constexpr int kRow = kChain + 2048;                   // float [128]: the row's sum so far, exchanged with the maxima (e4m3)
  static constexpr int kSum = kRow + 512;                      // float [2][128]: row sums
  static constexpr int kTmemSlot = kSum + 1024;
  static constexpr int kTotal = kTmemSlot + 16;
  static constexpr int kDynamic = kTotal + 1024;
};

// One warp copies tile rows row0..row0+31: lane r holds the source row of tile row row0 + r (negative: zero row).
// kCh > 0: rows of exactly kCh 16-byte chunks; the warp walks the 32 x kCh chunks in order, 32 at a time, so that every
// lane of every request copies.  kCh == 0: eight lanes cover 128 contiguous bytes of a row, four rows per request;
// chunks at or beyond d_chunks (the padding up to the next multiple of 64 elements) are zero-filled.
template <int NB, int kCh>
__device__ __forceinline__ void warp_gather_rows_w(uint32_t s_tile, int row0, int my_row_idx, const uint8_t* base,
                                                   size_t row_bytes, int d_chunks, int lane) {
  if constexpr (kCh > 0) {
#pragma unroll
    for (int i = 0; i < kCh; ++i) {
      const int r = (i * 32 + lane) / kCh, c = (i * 32 + lane) % kCh;
      const int id = __shfl_sync(0xffffffffu, my_row_idx, r);
      const uint32_t dst = s_tile + (c >> 3) * 16384 + (row0 + r) * 128 + (((c & 7) ^ (r & 7)) << 4);
      if (id >= 0) cp_async16(dst, base + (size_t)id * row_bytes + c * 16);
      else cp_async16_zfill(dst, base, 0);
    }
  } else {
    const int c8 = lane & 7, sub = lane >> 3;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int rl = i * 4 + sub;
      const int id = __shfl_sync(0xffffffffu, my_row_idx, rl);
      const int row = row0 + rl;
      const uint32_t dst = s_tile + row * 128 + ((c8 ^ (row & 7)) << 4);
#pragma unroll
      for (int blk = 0; blk < NB; ++blk) {
        const int c = blk * 8 + c8;
        if (id >= 0 && c < d_chunks) cp_async16(dst + blk * 16384, base + (size_t)id * row_bytes + c * 16);
        else cp_async16_zfill(dst + blk * 16384, base, 0);
      }
    }
  }
}

// kType: 0 = bf16, 1 = fp16, 2 = e4m3 (Q/K/V 8-bit, logits scaled by scale_qk_log2[b,h,m], P quantised to e4m3 with a
// bias of 2^4, O scaled by scale_v[b,h], bf16 out: the contract of the main kernel's e4m3 instantiation)
template <int NB, int kType, int kCh>
__global__ void __launch_bounds__(kThreadsW, 1) gather_attn_wide_kernel(const GatherAttnParams p) {
  constexpr bool kFp16 = kType == 1;
  constexpr bool kFp8 = kType == 2;
  constexpr int kEs = kFp8 ? 1 : 2;                   // bytes per Q/K/V element
  using L = SmemW<NB>;
  constexpr int R = L::kRing;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t s_base = smem_u32(smem);
  const uint32_t bars = s_base + L::kBars;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kTmemSlot);
  auto bar = [&](int i) { return bars + 8u * i; };
  auto sRing = [&](int slot) { return s_base + L::kRingOff + slot * L::kTileBytes; };
  const uint32_t sQ = s_base + L::kQ;

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

  // ---- the work item of this CTA
  const int item = blockIdx.x;
  const int m = item % p.M, bh = item / p.M, h = bh % p.H, b = bh / p.H;
  const int row_base = m * p.group_rows;
  const int rows_valid = min(p.group_rows, p.Sq - row_base);
  int T = p.gather_len / kTileN;
  if (p.gl != nullptr) T = min(max(p.gl[item], 1), T);
  const int d_chunks = p.D * kEs / 16;            // 16-byte chunks of a Q/K/V row
  const int ksteps = (p.D * kEs + 31) / 32;       // k-steps of Q K^T (32 bytes of every row each)
  const int n_pv = (p.D + 15) / 16 * 16;          // output columns the P V product computes
  const int o_chunks = p.D / 8;                   // 16-byte chunks of an output row (16-bit elements)

  if (tid == 0) {
    for (int i = 0; i < R; ++i) {
      mbar_init(bar(WB_FULL + i), kProducerThreadsW);
      mbar_init(bar(WB_EMPTY + i), 1);
    }
    mbar_init(bar(WB_Q_FULL), kProducerThreadsW);
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(WB_S_FULL + i), 1);
      mbar_init(bar(WB_P_READY + i), 8);
    }
    mbar_init(bar(WB_PV_DONE), 1);
    mbar_init(bar(WB_O_FULL), 1);
    mbar_init(bar(WB_DRAIN), 1);
    mbar_fence_init();
  }
  constexpr uint32_t kTmemColsW = 512;
  if (warp == kMmaWarpW) {
    tmem_alloc(smem_u32(tmem_slot), kTmemColsW);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp < 8) {
    // ===================================================================== softmax and epilogue
    auto warp_arrive = [&](uint32_t bb) {
      __syncwarp();
      if (lane == 0) mbar_arrive(bb);
    };
    const int x = warp >> 2;                            // column half
    const int r_in = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = (static_cast<uint32_t>(warp & 3) * 32u) << 16;
    const int pair_bar = 1 + (warp & 3);                // named barriers of this row block's two warps
    const int sum_bar = 5 + (warp & 3);                 // (e4m3: from the lower half to the upper)
    float* xch = reinterpret_cast<float*>(smem + L::kXch);
    float4* chain = reinterpret_cast<float4*>(smem + L::kChain);
    float* row_sum = reinterpret_cast<float*>(smem + L::kRow);
    const float scale_log2 = kFp8 ? p.scale_qk_log2[item] : p.scale_log2;
    const unsigned long long scale2 = f2_pack(scale_log2, scale_log2);
    // lazy raise of the running maximum with the thresholds of the main kernel; e4m3 P is biased by 2^4 so that the
    // largest probability of a row lies in [2^4, 2^8]
    constexpr float kRescale = kFp8 ? 4.0f : (kFp16 ? 12.0f : 24.0f);
    constexpr float kBias = kFp8 ? 4.0f : 0.0f;
    // the output columns that this thread rescales and writes: 16-byte output chunks (8 columns) [c_lo, c_hi)
    const int half_chunks = (n_pv / 8 + 1) / 2;
    const int c_lo = x * half_chunks, c_hi = x == 0 ? half_chunks : n_pv / 8;
    const uint32_t tO = tmem + kColOW + lane_addr;
    // running maximum (the same in both halves); row sum of this half, for e4m3 that of the whole row (upper half) or a bound
    // below it (lower half: the whole row's at the last exchange, its own half's since)
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    int fail_g = 0;
    bool fail_bar_done = false;
#pragma unroll 1
    for (int g = 0; g < T; ++g) {
      const int buf = g & 1;
      ok = mbar_wait(bar(WB_S_FULL + buf), (g >> 1) & 1, p.status, 60);
      if (!ok) { fail_g = g; break; }
      tc_fence_after();
      const uint32_t tS = tmem + kColSW + buf * 128 + x * 64 + lane_addr;
      uint32_t sc[64];
      tmem_ld32(tS, *reinterpret_cast<uint32_t(*)[32]>(&sc[0]));
      tmem_ld32(tS + 32, *reinterpret_cast<uint32_t(*)[32]>(&sc[32]));
      tmem_wait_ld();
      if (p.dense && g == T - 1) {
        const int rem = p.Sk - g * kTileN - x * 64;       // valid key columns of this half of the last tile
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (i >= rem) sc[i] = 0xff800000u;
      }
      float mx[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) mx[q] = fmaxf(__uint_as_float(sc[2 * q]), __uint_as_float(sc[2 * q + 1]));
#pragma unroll
      for (int i = 8; i < 64; i += 8)
#pragma unroll
        for (int q = 0; q < 4; ++q) mx[q] = fmax3(mx[q], __uint_as_float(sc[i + 2 * q]), __uint_as_float(sc[i + 2 * q + 1]));
      const float m_loc = fmaxf(fmax3(mx[0], mx[1], mx[2]), mx[3]) * scale_log2;
      float alpha = 1.f;
      bool want = (m_loc - m_run) > kRescale;
      // e4m3: a new maximum that would hold more than an eighth of the row's mass so far becomes the reference point at once:
      // its probability is then exact (see the main kernel).  The rule goes by the mass of the whole row: by the mass of a half
      // the reference would move sooner and round every probability behind it at another scale.  The upper half's thread has
      // that mass, the lower half's a bound below it (with a margin for the rounding of its sums) and so may want an exchange
      // that then raises nothing.
      if constexpr (kFp8) want = want || ((m_loc > m_run) && (ex2_approx(m_loc - m_run + kBias) > (x == 0 ? 0.124f : 0.125f) * l_run));
      if (named_bar_red_or(pair_bar, 64, want)) {
        xch[x * 128 + r_in] = m_loc;
        if (kFp8 && x == 1) row_sum[r_in] = l_run;
        named_bar_sync(pair_bar, 64);
        const float m_new = fmaxf(m_loc, xch[(x ^ 1) * 128 + r_in]);
        bool raise = (m_new - m_run) > kRescale;            // the same decision in both threads of the row
        if constexpr (kFp8) {
          if (x == 0) l_run = row_sum[r_in];
          raise = raise || ((m_new > m_run) && (ex2_approx(m_new - m_run + kBias) > 0.125f * l_run));
        }
        if (raise) { alpha = ex2_approx(m_run - m_new); m_run = m_new; }
        if (!kFp8 || x == 0) l_run *= alpha;
        if (g > 0 && (!kFp8 || __any_sync(0xffffffffu, raise))) {
          // O is stable once P V of the previous tile has completed (this tile's P V waits for the stores below)
          ok = mbar_wait(bar(WB_PV_DONE), (g - 1) & 1, p.status, 61);
          if (!ok) { fail_g = g; fail_bar_done = true; break; }
          tc_fence_after();
#pragma unroll 1
          for (int c = c_lo; c < c_hi; ++c) {
            uint32_t r[8];
            tmem_ld8(tO + c * 8, r);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            tmem_st8(tO + c * 8, r);
          }
        }
        // (the partner has read this thread's entries before it arrives at the next tile's barrier)
      }
      const float neg_m = kBias - m_run;
      const unsigned long long neg2 = f2_pack(neg_m, neg_m);
      unsigned long long ls[2] = {0ull, 0ull};             // e4m3: four sums, over the columns of each residue modulo 4
#pragma unroll
      for (int c = 0; c < (kFp8 ? 2 : 4); ++c) {
        uint32_t pk[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if constexpr (kFp8) {
            const int e = c * 32 + 4 * i;
            const float2 ya = f2_unpack(f2_fma(f2_pack(__uint_as_float(sc[e]), __uint_as_float(sc[e + 1])), scale2, neg2));
            const float2 yb = f2_unpack(f2_fma(f2_pack(__uint_as_float(sc[e + 2]), __uint_as_float(sc[e + 3])), scale2, neg2));
            const float p0 = ex2_approx(ya.x), p1 = ex2_approx(ya.y), p2 = ex2_approx(yb.x), p3 = ex2_approx(yb.y);
            ls[0] = f2_add(ls[0], f2_pack(p0, p1));
            ls[1] = f2_add(ls[1], f2_pack(p2, p3));
            sc[e] = __float_as_uint(p0); sc[e + 1] = __float_as_uint(p1); sc[e + 2] = __float_as_uint(p2); sc[e + 3] = __float_as_uint(p3);
            pk[i] = pack_e4m3x4(p0, p1, p2, p3);
          } else {
            const int e = c * 16 + 2 * i;
            const float2 y = f2_unpack(f2_fma(f2_pack(__uint_as_float(sc[e]), __uint_as_float(sc[e + 1])), scale2, neg2));
            const float p0 = ex2_approx(y.x), p1 = ex2_approx(y.y);
            ls[i & 1] = f2_add(ls[i & 1], f2_pack(p0, p1));
            pk[i] = kFp16 ? pack_f16x2(p0, p1) : pack_bf16x2(p0, p1);
          }
        }
        tmem_st8(tS + c * 8, pk);
      }
      const float2 l0 = f2_unpack(ls[0]), l1 = f2_unpack(ls[1]);
      if (!kFp8 || x == 0) l_run += (l0.x + l0.y) + (l1.x + l1.y);
      if (kFp8 && x == 0) chain[r_in] = make_float4(l0.x, l0.y, l1.x, l1.y);
      tmem_wait_st();
      tc_fence_before();
      warp_arrive(bar(WB_P_READY + buf));
      if constexpr (kFp8) {
        // The upper half continues the four sums of the lower half in the order of the columns, so that the row's sum, and with
        // it the rule above, does not depend on how the row is split.  This runs under the tile's P V.  (The lower half only
        // announces its sums; it overwrites them behind the next tile's barrier.)
        if (x == 0) {
          named_bar_arrive(sum_bar, 64);
        } else {
          named_bar_sync(sum_bar, 64);
          const float4 s = chain[r_in];
          unsigned long long sa = f2_pack(s.x, s.y), sb = f2_pack(s.z, s.w);
#pragma unroll
          for (int i = 0; i < 64; i += 4) {
            sa = f2_add(sa, f2_pack(__uint_as_float(sc[i]), __uint_as_float(sc[i + 1])));
            sb = f2_add(sb, f2_pack(__uint_as_float(sc[i + 2]), __uint_as_float(sc[i + 3])));
          }
          const float2 a = f2_unpack(sa), c = f2_unpack(sb);
          l_run = l_run * alpha + ((a.x + a.y) + (c.x + c.y));
        }
      }
    }
    if (!ok) {
      // failure path: a bounded wait expired (the status word says where).  The partner warp may still be running; a named
      // barrier has no bounded wait, so this warp keeps meeting it once per remaining tile until it ends the same way.
      bool done = fail_bar_done;
      for (int g = fail_g; g < T; ++g) {
        if (!done && named_bar_red_or(pair_bar, 64, false)) named_bar_sync(pair_bar, 64);
        done = false;
        if constexpr (kFp8) {
          if (x == 0) named_bar_arrive(sum_bar, 64); else named_bar_sync(sum_bar, 64);
        }
      }
    }
    // ---- the row's sum: both halves, relative to the same maximum (e4m3: the upper half's thread has it all)
    float* sums = reinterpret_cast<float*>(smem + L::kSum);
    sums[x * 128 + r_in] = kFp8 && x == 0 ? 0.f : l_run;
    ok = !named_bar_red_or(pair_bar, 64, !ok);
    const float l_all = sums[r_in] + sums[128 + r_in];
    if (ok) ok = mbar_wait(bar(WB_O_FULL), 0, p.status, 62);
    if (ok) {
      tc_fence_after();
      // ---- epilogue: out = sign * O / l + residual, one rounding; the row goes to its original position
      const bool valid = r_in < rows_valid;
      const int row = row_base + r_in;
      long long orow = row;
      if (valid && p.perm != nullptr && !p.out_group_order) orow = p.perm[(size_t)bh * p.Sq + row];
      uint8_t* obase = reinterpret_cast<uint8_t*>(p.out);
      long long lrow = orow;
      if (p.n_out_peers > 0) {
        const int peer = valid ? static_cast<int>(orow / p.out_rows_per_peer) : 0;
        lrow = orow - (long long)peer * p.out_rows_per_peer;
        obase = reinterpret_cast<uint8_t*>(p.out_peer[peer]);
      }
      uint8_t* optr = obase + 2 * ((size_t)b * p.o_stride[0] + (size_t)lrow * p.o_stride[1] + (size_t)h * p.o_stride[2]);
      const uint8_t* rptr = p.residual == nullptr ? nullptr
          : reinterpret_cast<const uint8_t*>(p.residual) + 2 * ((size_t)b * p.r_stride[0] + (size_t)h * p.r_stride[1] + (size_t)row * p.r_stride[2]);
      const float w = p.out_sign * (kFp8 ? p.scale_v[bh] : 1.f) / l_all;
      const int c_end = min(c_hi, o_chunks);
#pragma unroll 2
      for (int c = c_lo; c < c_end; ++c) {
        uint4 res = make_uint4(0, 0, 0, 0);
        if (valid && rptr != nullptr) res = *reinterpret_cast<const uint4*>(rptr + c * 16);
        uint32_t ra[8];
        tmem_ld8(tO + c * 8, ra);
        tmem_wait_ld();
        const uint32_t rw[4] = {res.x, res.y, res.z, res.w};
        uint32_t ow[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float2 rr;
          if constexpr (kFp16) rr = __half22float2(*reinterpret_cast<const __half2*>(&rw[j]));
          else rr = make_float2(bf16_lo(rw[j]), bf16_hi(rw[j]));
          const float o0 = fmaf(__uint_as_float(ra[2 * j]), w, rr.x);
          const float o1 = fmaf(__uint_as_float(ra[2 * j + 1]), w, rr.y);
          ow[j] = kFp16 ? pack_f16x2(o0, o1) : pack_bf16x2(o0, o1);
        }
        if (valid) *reinterpret_cast<uint4*>(optr + c * 16) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
      }
      if (x == 0 && valid && p.lse != nullptr) p.lse[(size_t)bh * p.Sq + orow] = (m_run + lg2_approx(l_all) - kBias) * 0.6931471805599453f;
    }
    tc_fence_before();
  } else if (warp < kMmaWarpW) {
    // ===================================================================== producers
    const int pw = warp - kProducerWarp0W;
    const int row0 = pw * 32;
    const int my_row = row0 + lane;
    const size_t q_row = kEs * (size_t)p.q_stride[1], k_row = kEs * (size_t)p.k_stride[1], v_row = kEs * (size_t)p.v_stride[1];
    const uint8_t* qb = reinterpret_cast<const uint8_t*>(p.q) + kEs * ((size_t)b * p.q_stride[0] + (size_t)h * p.q_stride[2]);
    const uint8_t* kb = reinterpret_cast<const uint8_t*>(p.k) + kEs * ((size_t)b * p.k_stride[0] + (size_t)h * p.k_stride[2]);
    const uint8_t* vb = reinterpret_cast<const uint8_t*>(p.v) + kEs * ((size_t)b * p.v_stride[0] + (size_t)h * p.v_stride[2]);
    {
      int src_row = -1;
      if (my_row < rows_valid) {
        src_row = row_base + my_row;
        if (p.perm != nullptr) src_row = static_cast<int>(p.perm[(size_t)bh * p.Sq + src_row]);
      }
      warp_gather_rows_w<NB, kCh>(sQ, row0, src_row, qb, q_row, d_chunks, lane);
      cp_async_arrive_noinc(bar(WB_Q_FULL));
    }
    const size_t ioff = (size_t)item * p.gather_len + my_row;
    auto load_idx = [&](int g) -> int {
      int idx;
      if (p.dense) {
        idx = g * kTileN + my_row;
      } else if (p.gi16 != nullptr) {
        const size_t o = ioff + (size_t)g * kTileN;
        const uint32_t lo = __ldg(p.gi16 + o), hi = (__ldg(p.gi_hi + (o >> 5)) >> (o & 31)) & 1u;
        idx = static_cast<int>(lo | (hi << 16));
      } else {
        idx = __ldg(p.gi + ioff + (size_t)g * kTileN);
      }
      return min(max(idx, 0), p.Sk - 1);
    };
    int held0 = 0, held1 = 0;        // indices of the two key tiles whose V tile is still to come
    int idx_next = load_idx(0);
    bool ok = true;
#pragma unroll 1
    for (int e = 0; e < 2 * T && ok; ++e) {
      // ring entries in the issuer's consumption order: K(0), K(1), V(0), K(2), V(1), ..., K(T-1), V(T-2), V(T-1)
      bool is_v;
      int g;
      if (e == 0) { is_v = false; g = 0; }
      else if (e == 2 * T - 1) { is_v = true; g = T - 1; }
      else if (e & 1) { is_v = false; g = (e + 1) >> 1; }
      else { is_v = true; g = (e >> 1) - 1; }
      const int slot = e % R, use = e / R;
      if (use > 0) ok = mbar_wait(bar(WB_EMPTY + slot), (use - 1) & 1, p.status, 63);
      if (!ok) break;
      int idx;
      if (is_v) {
        idx = (g & 1) ? held1 : held0;
      } else {
        idx = idx_next;
        if (g & 1) held1 = idx; else held0 = idx;
        if (g + 1 < T) idx_next = load_idx(g + 1);     // in flight while this tile's copies are issued
      }
      warp_gather_rows_w<NB, kCh>(sRing(slot), row0, idx, is_v ? vb : kb, is_v ? v_row : k_row, d_chunks, lane);
      cp_async_arrive_noinc(bar(WB_FULL + slot));
    }
    cp_async_wait_all();
    tc_fence_before();
  } else {
    // ===================================================================== issuer of both products
    constexpr uint32_t kFmt = (kFp16 || kFp8) ? 0u : 1u;   // kind::f16: 0 f16, 1 bf16; kind::f8f6f4: 0 e4m3
    constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);   // SBO 1024, version 1, 128-byte swizzle
    auto desc = [&](uint32_t lo) { return (static_cast<uint64_t>(kDescHi) << 32) | lo; };
    constexpr uint32_t kLboK = (16u >> 4) << 16;
    constexpr uint32_t kLboV = (16384u >> 4) << 16;        // MN-major V: 16 KB between 64-element column blocks
    const uint32_t idesc_qk = mma_idesc(kFmt, kFmt, 0, 0, 128, kTileN);
    const uint32_t idesc_pv = mma_idesc(kFmt, kFmt, 0, 1, 128, static_cast<uint32_t>(n_pv));
    const bool leader = elect_one();
    bool ok = true;
    auto issue_qk = [&](int g) {
      const int e = g == 0 ? 0 : 2 * g - 1;
      const int slot = e % R, use = e / R;
      if (g == 0) ok = mbar_wait(bar(WB_Q_FULL), 0, p.status, 64);
      ok = ok && mbar_wait(bar(WB_FULL + slot), use & 1, p.status, 65);
      if (!ok) return;
      const uint32_t tS = tmem + kColSW + (g & 1) * 128;     // free: P V of tile g - 2, which read P out of it, was issued before
      fence_proxy_async_smem();
      tc_fence_after();
      const uint32_t qlo = ((sQ & 0x3FFFFu) >> 4) | kLboK;
      const uint32_t klo = ((sRing(slot) & 0x3FFFFu) >> 4) | kLboK;
#pragma unroll 1
      for (int j = 0; j < ksteps; ++j) {
        const uint32_t koff = (j >> 2) * (16384 >> 4) + (j & 3) * 2;
        if (leader) {
          if constexpr (kFp8) mma_f8_ss(tS, desc(qlo + koff), desc(klo + koff), idesc_qk, j > 0);
          else mma_f16_ss(tS, desc(qlo + koff), desc(klo + koff), idesc_qk, j > 0);
        }
      }
      if (leader) {
        tc_commit(bar(WB_EMPTY + slot));
        tc_commit(bar(WB_S_FULL + (g & 1)));
      }
    };
    auto issue_pv = [&](int g) {
      const int e = g < T - 1 ? 2 * g + 2 : 2 * T - 1;
      const int slot = e % R, use = e / R;
      ok = mbar_wait(bar(WB_FULL + slot), use & 1, p.status, 67) && mbar_wait(bar(WB_P_READY + (g & 1)), (g >> 1) & 1, p.status, 68);
      if (!ok) return;
      fence_proxy_async_smem();
      tc_fence_after();
      const uint32_t vlo = ((sRing(slot) & 0x3FFFFu) >> 4) | kLboV;
      const uint32_t tP = tmem + kColSW + (g & 1) * 128;     // k-steps of half x at columns 64 x
      if constexpr (kFp8) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // A: 32 e4m3 probabilities = 8 tensor-memory columns per k-step; B: 32 key rows = 4096 bytes
          if (leader) mma_f8_ts(tmem + kColOW, tP + (j >> 1) * 64 + (j & 1) * 8, desc(vlo + j * (4096 >> 4)), idesc_pv, (g > 0) || (j > 0));
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          // A: 16 packed probabilities = 8 tensor-memory columns per k-step; B: 16 key rows = 2048 bytes
          if (leader) mma_f16_ts(tmem + kColOW, tP + (j >> 2) * 64 + (j & 3) * 8, desc(vlo + j * (2048 >> 4)), idesc_pv, (g > 0) || (j > 0));
        }
      }
      if (leader) {
        tc_commit(bar(WB_EMPTY + slot));
        tc_commit(bar(WB_PV_DONE));
        if (g == T - 1) tc_commit(bar(WB_O_FULL));
      }
    };
    issue_qk(0);
    if (ok && T > 1) issue_qk(1);
#pragma unroll 1
    for (int g = 0; g < T && ok; ++g) {
      issue_pv(g);
      if (ok && g + 2 < T) issue_qk(g + 2);
    }
    if (!ok) {
      // error path: let outstanding products retire before tensor memory is released
      if (leader) tc_commit(bar(WB_DRAIN));
      mbar_wait_quiet(bar(WB_DRAIN), 0, 1 << 20);
    }
    __syncwarp();
    tc_fence_before();
  }

  __syncthreads();
  if (warp == kMmaWarpW) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemColsW);
  }
}

template <int NB, int kType, int kCh = 0>
int launch_wide(const GatherAttnParams& p, cudaStream_t stream) {
  using L = SmemW<NB>;
  auto kern = gather_attn_wide_kernel<NB, kType, kCh>;
  // a CTA needs all of tensor memory: ask for enough shared memory that only one is resident per SM
  const int smem = L::kDynamic < 120 * 1024 ? 120 * 1024 : L::kDynamic;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -8;
  const long long items = (long long)p.B * p.H * p.M;
  kern<<<static_cast<unsigned>(items), kThreadsW, smem, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : -8;
}

}  // namespace

int launch_gather_attn_wide(const GatherAttnParams& p, bool fp16, cudaStream_t stream) {
  if (p.D < 8 || p.D > 256 || p.D % 8 != 0 || p.group_rows > 128) return -3;
  // 144 and 160: a quarter and a sixth of the copies of the block-wise gather would be padding (144: 471 us against 548;
  // 160: 522 against 548, in a loop of calls).  At 96 the block-wise gather wins (371 against 389), as for the 160-byte rows of
  // e4m3 (389 / 402).
  if (p.D == 144) return fp16 ? launch_wide<3, 1, 18>(p, stream) : launch_wide<3, 0, 18>(p, stream);
  if (p.D == 160) return fp16 ? launch_wide<3, 1, 20>(p, stream) : launch_wide<3, 0, 20>(p, stream);
  const int nb = (p.D + 63) / 64;
  switch (nb) {
    case 1: return fp16 ? launch_wide<1, 1>(p, stream) : launch_wide<1, 0>(p, stream);
    case 2: return fp16 ? launch_wide<2, 1>(p, stream) : launch_wide<2, 0>(p, stream);
    case 3: return fp16 ? launch_wide<3, 1>(p, stream) : launch_wide<3, 0>(p, stream);
    default: return fp16 ? launch_wide<4, 1>(p, stream) : launch_wide<4, 0>(p, stream);
  }
}

int launch_gather_attn_wide_e4m3(const GatherAttnParams& p, cudaStream_t stream) {
  if (p.D < 16 || p.D > 256 || p.D % 16 != 0 || p.group_rows > 128) return -3;
  return p.D <= 128 ? launch_wide<1, 2>(p, stream) : launch_wide<2, 2>(p, stream);
}

}  // namespace mcs
