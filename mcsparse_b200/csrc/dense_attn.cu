// Dense flash-attention forward (bf16 / fp16, head dimension 64 or 128) for sm_100a: the dense mode of the package's
// attention, two query tiles per CTA.
//
// Persistent kernel, one CTA per SM.  A work item is 256 consecutive rows of the (optionally permuted) query
// sequence of one (batch, head), handled as two streams of 128 rows that share every K and V tile.  The kernel that
// gathers selected rows (gather_attn.cu) cannot share tiles between query groups, works on one group of 128 rows at a
// time and splits its 128 score columns over two warps per sub-partition; every tile then waits for the round trip
// scores -> softmax -> P V -> next scores, which left the tensor pipe idle for half of the time.  Here one stream's
// products run under the other stream's softmax:
//     issue order   P V A(t), Q K^T A(t+1), P V B(t), Q K^T B(t+1), ...
// and a softmax thread owns a whole row, so that no barrier, exchange or second running maximum exists.
//
// Roles (384 threads, 12 warps, three per sub-partition: 168 registers each):
//   warps 0-3, 4-7   softmax of streams A, B (thread == row == tensor-memory lane, all 128 columns in registers) and
//                    the epilogue of their rows
//   warp 8           K/V tiles by TMA into a ring, one elected thread
//   warp 9           issues every product
//   warps 10, 11     copy the Q tiles of streams A, B (rows through the permutation) with cp.async
//
// Tensor memory: S_A, S_B (128 columns each), O_A, O_B (D columns each).  P overwrites the scores it was computed from.
// Products of one thread execute in order, so Q K^T of tile t+1 may overwrite S right behind the P V of tile t that
// reads P out of it, and a completed Q K^T of tile t+1 implies that P V of tile t is complete: O may then be rescaled.
//
// What bounds it: per pair of tiles the tensor pipe needs 2,048 cycles and the special-function unit the same
// (32,768 exponentials at 16 per clock); under a long load the GPU's power limit lowers the clock.  Measured at 24 heads x
// 32,760 x 128 bf16 (13.2 TFLOP; 8.0 ms at the measured burst rate, 9.4 at the sustained one): 11.24 -> 10.14 ms in short
// bursts, 12.85 -> 11.28 ms in a loop of calls (3,146 cycles per pair of tiles; 1.77 GHz in a burst, 1.51 GHz in the loop).
// The exponentials are not what is left: without any (results wrong, timing only) a pair takes 3,225 cycles against 3,260
// before P V started early.  Shared memory is as busy as the tensor pipe: Q K^T reads both operands from it at 128 bytes
// per cycle, its full rate, while the next tiles are written.  Measured and not kept: an eighth / a quarter of the
// exponentials as polynomials on the FMA pipe (12.18 / 12.19 ms against 11.67 measured beside them in a loop: issue slots and energy), scalar
// instead of two-wide fused multiply-adds (12.13), P V started at half of the tile (11.60 against 11.54 at three quarters).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "kernels.cuh"
#include "ptx.cuh"

namespace mcs {

namespace {

constexpr int kTileN = 128;
constexpr int kThreadsD = 384;
constexpr int kTmaWarp = 8, kIssueWarp = 9, kQWarp0 = 10;
constexpr uint32_t kColS = 0, kColO = 256;
constexpr int kEarly = 6;       // P V of a tile starts when the probabilities of its first kEarly k-steps (of 8) are stored

template <int D>
struct SmemD {
  static constexpr int kTileBytes = (D / 64) * 16384;
  static constexpr int kRing = D == 128 ? 5 : 8;
  static constexpr int kQ = 0;                             // one tile per stream
  static constexpr int kRingOff = 2 * kTileBytes;
  static constexpr int kBars = kRingOff + kRing * kTileBytes;
  // barriers
  static constexpr int kFull = 0, kEmpty = kRing;          // [kRing]
  static constexpr int kQFull = 2 * kRing, kQEmpty = kQFull + 2, kSFull = kQEmpty + 2, kPReady = kSFull + 2, kOFull = kPReady + 2,
                       kOFree = kOFull + 2, kPEarly = kOFree + 2, kDrain = kPEarly + 2, kCount = kDrain + 1;
  static constexpr int kSlot = kBars + kCount * 8;
  static constexpr int kDynamic = kSlot + 16 + 1024;
};
static_assert(SmemD<128>::kDynamic <= 232448, "must fit 227 KB");

template <int D, bool kFp16>
__global__ void __launch_bounds__(kThreadsD, 1) dense_attn_kernel(const GatherAttnParams p, const __grid_constant__ DenseTileMaps maps,
                                                                  int pairs) {
  using L = SmemD<D>;
  constexpr int R = L::kRing;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t s_base = smem_u32(smem);
  const uint32_t bars = s_base + L::kBars;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kSlot);
  auto bar = [&](int i) { return bars + 8u * i; };
  auto sQ = [&](int x) { return s_base + L::kQ + x * L::kTileBytes; };
  auto sRing = [&](int slot) { return s_base + L::kRingOff + slot * L::kTileBytes; };
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int n_items = p.B * p.H * pairs;
  const int T = (p.Sk + kTileN - 1) / kTileN;
  // rows of stream x of an item; an item at the end of the sequence may have none in stream B
  auto first_row = [&](int item, int x) { return (item % pairs) * 256 + x * 128; };
  auto has_b = [&](int item) { return first_row(item, 1) < p.Sq; };

  if (tid == 0) {
    for (int i = 0; i < R; ++i) { mbar_init(bar(L::kFull + i), 1); mbar_init(bar(L::kEmpty + i), 1); }
    for (int x = 0; x < 2; ++x) {
      mbar_init(bar(L::kQFull + x), 32);
      mbar_init(bar(L::kQEmpty + x), 1);
      mbar_init(bar(L::kSFull + x), 1);
      mbar_init(bar(L::kPEarly + x), 4);
      mbar_init(bar(L::kPReady + x), 4);
      mbar_init(bar(L::kOFull + x), 1);
      mbar_init(bar(L::kOFree + x), 4);
    }
    mbar_init(bar(L::kDrain), 1);
    mbar_fence_init();
  }
  if (warp == kIssueWarp) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp < 8) {
    // ===================================================================== softmax and epilogue
    auto warp_arrive = [&](uint32_t b) {
      __syncwarp();
      if (lane == 0) mbar_arrive(b);
    };
    const int x = warp >> 2;
    const int r_in = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = (static_cast<uint32_t>(warp & 3) * 32u) << 16;
    const uint32_t tS = tmem + kColS + x * 128 + lane_addr, tO = tmem + kColO + x * D + lane_addr;
    // lazy raise of the running maximum: P stays below 2^kRescale (fp16: 65504)
    constexpr float kRescale = kFp16 ? 12.0f : 24.0f;
    const float scale = p.scale_log2;
    const unsigned long long scale2 = f2_pack(scale, scale);
    int g = 0, ic = 0;
    bool ok = true;
#pragma unroll 1
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      if (x == 1 && !has_b(item)) continue;
      // the sums of the two column halves are kept apart: the order of additions of the gathering kernel, and with it its bits
      float m_run = -INFINITY, l_run[2] = {0.f, 0.f};
#pragma unroll 1
      for (int t = 0; t < T; ++t, ++g) {
        ok = mbar_wait(bar(L::kSFull + x), g & 1, p.status, 110);
        if (!ok) break;
        tc_fence_after();
        uint32_t sc[128];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(tS + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&sc[c * 32]));
        tmem_wait_ld();
        if (t == T - 1) {
          // key positions beyond the sequence end (zero rows of the last tile) get -inf
          const int rem = p.Sk - t * kTileN;
          if (rem < kTileN) {
#pragma unroll
            for (int i = 0; i < 128; ++i)
              if (i >= rem) sc[i] = 0xff800000u;
          }
        }
        float mx[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) mx[q] = fmaxf(__uint_as_float(sc[2 * q]), __uint_as_float(sc[2 * q + 1]));
#pragma unroll
        for (int i = 8; i < 128; i += 8)
#pragma unroll
          for (int q = 0; q < 4; ++q) mx[q] = fmax3(mx[q], __uint_as_float(sc[i + 2 * q]), __uint_as_float(sc[i + 2 * q + 1]));
        const float m_loc = fmaxf(fmax3(mx[0], mx[1], mx[2]), mx[3]) * scale;
        const bool raise = (m_loc - m_run) > kRescale;
        if (__any_sync(0xffffffffu, raise)) {
          const float alpha = raise ? ex2_approx(m_run - m_loc) : 1.f;
          if (raise) m_run = m_loc;
          l_run[0] *= alpha;
          l_run[1] *= alpha;
          if (t > 0) {
#pragma unroll 1
            for (int c = 0; c < D / 8; ++c) {
              uint32_t r[8];
              tmem_ld8(tO + c * 8, r);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 8; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
              tmem_st8(tO + c * 8, r);
            }
          }
        }
        const unsigned long long neg2 = f2_pack(-m_run, -m_run);
        unsigned long long ls[2][2] = {};                    // [column half][chain] packed partial sums
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint32_t pk[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int e = c * 16 + 2 * i;
            const float2 y = f2_unpack(f2_fma(f2_pack(__uint_as_float(sc[e]), __uint_as_float(sc[e + 1])), scale2, neg2));
            const float p0 = ex2_approx(y.x), p1 = ex2_approx(y.y);
            ls[c / 4][i & 1] = f2_add(ls[c / 4][i & 1], f2_pack(p0, p1));
            pk[i] = kFp16 ? pack_f16x2(p0, p1) : pack_bf16x2(p0, p1);
          }
          tmem_st8(tS + c * 8, pk);
          if (c == kEarly - 1) {
            tmem_wait_st();
            tc_fence_before();
            warp_arrive(bar(L::kPEarly + x));
          }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float2 a0 = f2_unpack(ls[q][0]), a1 = f2_unpack(ls[q][1]);
          l_run[q] += (a0.x + a0.y) + (a1.x + a1.y);
        }
        tmem_wait_st();
        tc_fence_before();
        warp_arrive(bar(L::kPReady + x));
      }
      if (!ok) break;
      // ---- epilogue: out = sign * O / l + residual, one rounding; the row goes to its original position
      const int row = first_row(item, x) + r_in;
      const int bh = item / pairs, h = bh % p.H, b = bh / p.H;
      const bool valid = row < p.Sq;
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
      ok = mbar_wait(bar(L::kOFull + x), ic & 1, p.status, 111);
      if (!ok) break;
      tc_fence_after();
      const float l_all = l_run[0] + l_run[1], w = p.out_sign / l_all;
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        uint32_t ra[32];
        tmem_ld32(tO + c * 32, ra);
        tmem_wait_ld();
        if (c == D / 32 - 1) {
          tc_fence_before();
          warp_arrive(bar(L::kOFree + x));                   // the next item's first P V may overwrite O
        }
        if (valid) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 res = make_uint4(0, 0, 0, 0);
            if (rptr != nullptr) res = *reinterpret_cast<const uint4*>(rptr + c * 64 + q * 16);
            const uint32_t rw[4] = {res.x, res.y, res.z, res.w};
            uint32_t ow[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float rx, ry;
              if constexpr (kFp16) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&rw[j]));
                rx = f.x; ry = f.y;
              } else {
                rx = bf16_lo(rw[j]); ry = bf16_hi(rw[j]);
              }
              const float o0 = fmaf(__uint_as_float(ra[q * 8 + 2 * j]), w, rx);
              const float o1 = fmaf(__uint_as_float(ra[q * 8 + 2 * j + 1]), w, ry);
              ow[j] = kFp16 ? pack_f16x2(o0, o1) : pack_bf16x2(o0, o1);
            }
            *reinterpret_cast<uint4*>(optr + c * 64 + q * 16) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
          }
        }
      }
      if (valid && p.lse != nullptr) p.lse[(size_t)bh * p.Sq + orow] = (m_run + lg2_approx(l_all)) * 0.6931471805599453f;
      ++ic;
    }
    tc_fence_before();
  } else if (warp == kTmaWarp) {
    // ===================================================================== K/V tiles: K(0), V(0), K(1), V(1), ... over all items
    const bool leader = elect_one();
    int slot = 0, phase = 0;
    bool wrapped = false, ok = true;
#pragma unroll 1
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      const int bh = item / pairs, h = bh % p.H, b = bh / p.H;
      int ck[4] = {0, 0, 0, 0}, cv[4] = {0, 0, 0, 0};
      ck[maps.k_pos_h] = h; ck[maps.k_pos_b] = b;
      cv[maps.v_pos_h] = h; cv[maps.v_pos_b] = b;
#pragma unroll 1
      for (int e = 0; e < 2 * T && ok; ++e) {
        const bool is_v = e & 1;
        if (wrapped) ok = mbar_wait(bar(L::kEmpty + slot), phase ^ 1, p.status, 112);
        if (!ok) break;
        if (leader) {
          mbar_arrive_expect_tx(bar(L::kFull + slot), L::kTileBytes);
          const void* map = is_v ? static_cast<const void*>(maps.v) : static_cast<const void*>(maps.k);
          int co[4] = {0, is_v ? cv[1] : ck[1], is_v ? cv[2] : ck[2], is_v ? cv[3] : ck[3]};
          co[is_v ? maps.v_pos_row : maps.k_pos_row] = (e >> 1) * kTileN;
#pragma unroll
          for (int cb = 0; cb < D / 64; ++cb)
            tma_load_4d(sRing(slot) + cb * 16384, map, cb * 64, co[1], co[2], co[3], bar(L::kFull + slot));
        }
        if (++slot == R) { slot = 0; phase ^= 1; wrapped = true; }
      }
    }
    tc_fence_before();
  } else if (warp == kIssueWarp) {
    // ===================================================================== issuer of every product
    constexpr uint32_t kFmt = kFp16 ? 0u : 1u;
    constexpr uint32_t idesc_qk = mma_idesc(kFmt, kFmt, 0, 0, 128, kTileN);
    constexpr uint32_t idesc_pv = mma_idesc(kFmt, kFmt, 0, 1, 128, D);
    constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);    // SBO 1024, version 1, 128-byte swizzle
    constexpr uint32_t kLboK = (16u >> 4) << 16;
    constexpr uint32_t kLboV = (16384u >> 4) << 16;                         // MN-major V: 16 KB between column blocks
    auto desc = [&](uint32_t lo) { return (static_cast<uint64_t>(kDescHi) << 32) | lo; };
    const bool leader = elect_one();
    bool ok = true;
    int slot = 0, phase = 0;
    auto advance = [&]() { if (++slot == R) { slot = 0; phase ^= 1; } };
    int g[2] = {0, 0}, ic[2] = {0, 0};               // tiles and items of each stream whose P V (Q K^T) has been issued
    int iq[2] = {0, 0};
    const bool telemetry = p.clock_out != nullptr && blockIdx.x == 0;
    long long clk_c0 = 0, tiles = 0;
    unsigned long long clk_g0 = 0;
    if (telemetry) { clk_c0 = clock64(); clk_g0 = globaltimer_ns(); }
    auto qk = [&](int x, int kslot, bool first, bool last) {
      if (first) {
        ok = ok && mbar_wait(bar(L::kQFull + x), iq[x] & 1, p.status, 113);
        if (!ok) return;
        fence_proxy_async_smem();
        tc_fence_after();
      }
      const uint32_t qlo = ((sQ(x) & 0x3FFFFu) >> 4) | kLboK;
      const uint32_t klo = ((sRing(kslot) & 0x3FFFFu) >> 4) | kLboK;
#pragma unroll
      for (int j = 0; j < D / 16; ++j) {
        const uint32_t koff = (j >> 2) * (16384 >> 4) + (j & 3) * 2;
        if (leader) mma_f16_ss(tmem + kColS + x * 128, desc(qlo + koff), desc(klo + koff), idesc_qk, j > 0);
      }
      if (leader) {
        tc_commit(bar(L::kSFull + x));
        if (last) tc_commit(bar(L::kQEmpty + x));
      }
      if (last) ++iq[x];
    };
    auto pv = [&](int x, int vslot, bool first, bool last) {
      ok = ok && mbar_wait(bar(L::kPEarly + x), g[x] & 1, p.status, 114);
      if (first && ic[x] > 0) ok = ok && mbar_wait(bar(L::kOFree + x), (ic[x] - 1) & 1, p.status, 115);
      if (!ok) return;
      tc_fence_after();
      const uint32_t vlo = ((sRing(vslot) & 0x3FFFFu) >> 4) | kLboV;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j == kEarly) {
          ok = mbar_wait(bar(L::kPReady + x), g[x] & 1, p.status, 120);
          if (!ok) return;
          tc_fence_after();
        }
        if (leader)
          mma_f16_ts(tmem + kColO + x * D, tmem + kColS + x * 128 + j * 8, desc(vlo + j * (2048 >> 4)), idesc_pv, !first || j > 0);
      }
      if (leader && last) tc_commit(bar(L::kOFull + x));
      ++g[x];
      if (last) ++ic[x];
    };
    int item = blockIdx.x, t = 0;
    if (item < n_items) {
      ok = mbar_wait(bar(L::kFull + slot), phase, p.status, 116);
      if (ok) {
        qk(0, slot, true, T == 1);
        if (ok && has_b(item)) qk(1, slot, true, T == 1);
        if (ok && leader) tc_commit(bar(L::kEmpty + slot));
        advance();
      }
#pragma unroll 1
      while (ok) {
        const bool first = t == 0, last = t == T - 1;
        const int nt = last ? 0 : t + 1, nitem = last ? item + static_cast<int>(gridDim.x) : item;
        const bool more = nitem < n_items;
        const bool b_now = has_b(item), b_next = more && has_b(nitem);
        const int vslot = slot;
        ok = mbar_wait(bar(L::kFull + vslot), phase, p.status, 117);
        if (!ok) break;
        advance();
        const int kslot = slot, kphase = phase;
        pv(0, vslot, first, last);
        if (!ok) break;
        if (!last) {
          ok = mbar_wait(bar(L::kFull + kslot), kphase, p.status, 118);
          if (!ok) break;
          qk(0, kslot, false, nt == T - 1);
        }
        if (b_now) pv(1, vslot, first, last);
        if (!ok) break;
        if (leader) tc_commit(bar(L::kEmpty + vslot));
        if (last && more) {
          // (the last P V of both streams is in flight before the next item's Q is waited for)
          ok = mbar_wait(bar(L::kFull + kslot), kphase, p.status, 118);
          if (!ok) break;
          qk(0, kslot, true, T == 1);
        }
        if (b_next && ok) qk(1, kslot, last, nt == T - 1);
        ++tiles;
        if (!more || !ok) break;
        if (leader) tc_commit(bar(L::kEmpty + kslot));
        advance();
        t = nt;
        item = nitem;
      }
    }
    if (telemetry && lane == 0) {
      p.clock_out[0] = clock64() - clk_c0;
      p.clock_out[1] = static_cast<long long>(globaltimer_ns() - clk_g0);
      p.clock_out[2] = tiles;
    }
    if (!ok) {
      // error path: let outstanding products retire before tensor memory is released
      if (leader) tc_commit(bar(L::kDrain));
      mbar_wait_quiet(bar(L::kDrain), 0, 1 << 20);
    }
    __syncwarp();
    tc_fence_before();
  } else {
    // ===================================================================== Q tiles
    const int x = warp - kQWarp0;
    constexpr int kChunks = D / 8, kRpi = 32 / kChunks;
    const int sub = lane / kChunks, c = lane % kChunks;
    const size_t q_row = 2 * (size_t)p.q_stride[1];
    int ic = 0;
    bool ok = true;
#pragma unroll 1
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      if (x == 1 && !has_b(item)) continue;
      const int bh = item / pairs, h = bh % p.H, b = bh / p.H, row0 = first_row(item, x);
      const uint8_t* qb = reinterpret_cast<const uint8_t*>(p.q) + 2 * ((size_t)b * p.q_stride[0] + (size_t)h * p.q_stride[2]) + c * 16;
      int src[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int row = row0 + q * 32 + lane;
        src[q] = row < p.Sq ? (p.perm != nullptr ? static_cast<int>(p.perm[(size_t)bh * p.Sq + row]) : row) : -1;
      }
      if (ic > 0) ok = mbar_wait(bar(L::kQEmpty + x), (ic - 1) & 1, p.status, 119);
      if (!ok) break;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int i = 0; i < 32 / kRpi; ++i) {
          const int rl = i * kRpi + sub;
          const int id = __shfl_sync(0xffffffffu, src[q], rl);
          const int r = q * 32 + rl;
          const uint32_t dst = sQ(x) + (c >> 3) * 16384 + r * 128 + (((c & 7) ^ (r & 7)) << 4);
          if (id >= 0) cp_async16(dst, qb + (size_t)id * q_row);
          else cp_async16_zfill(dst, p.q, 0);
        }
      }
      cp_async_arrive_noinc(bar(L::kQFull + x));
      ++ic;
    }
    cp_async_wait_all();
    tc_fence_before();
  }

  __syncthreads();
  if (warp == kIssueWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <int D, bool kFp16>
int launch_d(const GatherAttnParams& p, const DenseTileMaps& maps, cudaStream_t stream) {
  using L = SmemD<D>;
  auto kern = dense_attn_kernel<D, kFp16>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynamic) != cudaSuccess) return -8;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int pairs = (p.Sq + 255) / 256;
  const long long items = (long long)p.B * p.H * pairs;
  kern<<<(unsigned)(items < sms ? items : sms), kThreadsD, L::kDynamic, stream>>>(p, maps, pairs);
  return cudaGetLastError() == cudaSuccess ? 0 : -8;
}

}  // namespace

bool dense_tile_maps(const GatherAttnParams& p, DenseTileMaps& maps) {
  maps.valid = encode_tile_map(p.k, p.k_stride, p.B, p.Sk, p.H, p.D, maps.k, maps.k_pos_h, maps.k_pos_row, maps.k_pos_b) &&
               encode_tile_map(p.v, p.v_stride, p.B, p.Sk, p.H, p.D, maps.v, maps.v_pos_h, maps.v_pos_row, maps.v_pos_b);
  return maps.valid != 0;
}

int launch_dense_attn(const GatherAttnParams& p, const DenseTileMaps& maps, bool fp16, cudaStream_t stream) {
  if (p.D == 128) return fp16 ? launch_d<128, true>(p, maps, stream) : launch_d<128, false>(p, maps, stream);
  if (p.D == 64) return fp16 ? launch_d<64, true>(p, maps, stream) : launch_d<64, false>(p, maps, stream);
  return -3;
}

}  // namespace mcs
