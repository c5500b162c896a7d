// Anchor-step group mass for sm_100a:
//
//   mass[b,h,m,j] = sum_{i in query group m} exp(scale * q_i . k_j - lse_i)        (fp32)
//
// i.e. the exact attention probability mass that query group m puts on key token j, given
// the log-sum-exp of every query row from a dense attention pass.  Optionally divided by
// the number of rows in the group (the reference's "mean" convention).
//
// Restates the reference's Triton kernel
// (mcsparse/kernels/flash_mcsa/ops/triton/block_probs.py:27-89), with an fp32 result instead
// of one rounded to bf16.
//
// One CTA per (batch*head, group), or per two neighbouring groups and a stretch of the key tiles (launch_group_mass).  The
// query rows stay resident in shared memory; the CTA streams its key tiles of the head.  The product is computed TRANSPOSED,
// S^T = K_tile Q^T, so that a TMEM lane is a key token and the sum over the group's queries
// runs along the columns inside one thread: no cross-thread reduction at all.
//
// "- lse_i" is folded into the MMA: the contraction is extended by one 16-wide k-step whose K
// columns are (1, 1, 1, 0, ...) and whose Q columns are (-hi, -mid, -lo, 0, ...), a three-term
// bf16 split of lse_i / scale, exact to fp32 precision.  The tensor core then delivers
// q_i . k_j - lse_i / scale and each element costs one multiply, one ex2 and one add.
// The SFU delivers 16 ex2 per clock and SM; a quarter of the exponentials are therefore evaluated by a polynomial on the FMA
// pipe.  With two query groups per CTA the SFU is busy 74% of the time, the tensor pipe 56%, and the products read both
// operands from shared memory at its full rate.
//
// Roles: warps 0-15 exponentiate and sum, in two groups of eight for the even and the odd key tiles, or for the two query
// groups (two threads per key token: warps w and w+4 of a group share a TMEM lane group and take 64 query columns each; the two partial sums meet in
// shared memory).  Four warps per SM sub-partition feed its SFU, and each group has two score buffers of its own, so one
// group's waits and tensor-memory loads lie under the other's exponentials: with a single group and two buffers the SFU
// was 64% busy (7,100 -> 6,517 us at 24 heads x 32,760 x 128, 655 -> 573 us at 8 x 16,380; floors 5,900 / 500 us of ex2
// alone, 4,400 / 370 with a quarter of them on the FMA pipe).  The first four (two query
// groups: eight) of them prepare the query operand before their first tile.  Warp 16 issues the MMAs (converged, one elected
// lane executes the tcgen05 instructions), warps 17-19 stream the key tiles into a 3-slot ring: by TMA (one elected thread,
// boxes of 128 rows x 128 bytes) when a tensor map can describe K's strides, else with cp.async.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "kernels.cuh"
#include "ptx.cuh"

namespace mcs {

namespace {

constexpr int kTile = 128;
constexpr int kThreads = 640;          // five warps per SM sub-partition: 96 registers each
constexpr int kExpWarps = 16;          // two groups of eight: even and odd key tiles
constexpr int kBufs = 4;               // score buffers of 128 columns in tensor memory
constexpr int kProducerWarps = 3;
constexpr int kProducerThreads = kProducerWarps * 32;
constexpr int kMmaWarp = 16;
constexpr int kProducerWarp0 = 17;
constexpr int kRing = 3;
constexpr uint32_t kTmemCols = 128 * kBufs;

enum { BAR_FULL = 0, BAR_EMPTY = BAR_FULL + kRing, BAR_Q_FULL = BAR_EMPTY + kRing, BAR_S_FULL, BAR_S_FREE = BAR_S_FULL + kBufs,
       BAR_PART = BAR_S_FREE + kBufs,  // [4 lane groups][kBufs]: partial sums of the upper column half are in shared memory
       BAR_DRAIN = BAR_PART + 4 * kBufs, BAR_COUNT };

// D is the head dimension rounded up to the tile layouts this kernel has: 64, 128, 192 or 256 (the true head
// dimension, any multiple of 8 up to 256, is a run-time value; rows are zero-padded on their way into shared memory)
template <int D, int G>
struct Smem {
  static constexpr int kBlocks = D / 64;
  static constexpr int kTileBytes = kBlocks * 16384;
  static constexpr int kQRows = 128 * G;                     // G query groups per CTA, see launch_group_mass
  static constexpr int kRingN = D == 256 ? 2 : kRing;        // key-tile slots that fit beside the query tile
  static constexpr int kQ = 0;                              // the groups' query rows (B operand)
  static constexpr int kX = G * kTileBytes;                 // extra k-steps, kQRows rows x 128 B: chunks 0-1 K's constant
                                                            // (1,1,1,0...), chunks 2-3 Q's, the rest unused
  static constexpr int kRingOff = kX + kQRows * 128;
  static constexpr int kBars = kRingOff + kRingN * kTileBytes;
  static constexpr int kPart = kBars + BAR_COUNT * 8;       // float [kBufs][128]: partial sums of the upper column half
  static constexpr int kTmemSlot = kPart + kBufs * 128 * 4;
  static constexpr int kTotal = kTmemSlot + 16;
  static constexpr int kDynamic = kTotal + 1024;
};

static_assert(Smem<128, 2>::kDynamic <= 232448 && Smem<192, 1>::kDynamic <= 232448 && Smem<256, 1>::kDynamic <= 232448, "padded layouts must fit 227 KB");

// 16-byte chunk c of row, 128-byte swizzle, tiles of kRows rows
template <int kRows = 128>
__device__ __forceinline__ uint32_t swz(int row, int c) {
  return static_cast<uint32_t>((c >> 3) * (kRows * 128) + row * 128 + (((c & 7) ^ (row & 7)) << 4));
}

// Constant extra K block, extra Q block and Q rows of tile rows row0 .. row0 + 31, by one warp.  (A function of its own: inlined
// into the kernel, the same code costs the exponentiating loop 1%: 6,920 us against 6,840 at 24 heads x 32,760 x 128.)
template <int D, bool kFp16, int G>
__device__ __noinline__ void prepare_queries(uint8_t* smem, const float* lse, const int64_t* perm, const uint8_t* qb, size_t q_row, int m0,
                                             int M, int group_rows, int Lq, float inv_scale, int d_chunks, int row0) {
  using L = Smem<D, G>;
  constexpr bool kWide = D > 128;
  constexpr int kChunks = kWide ? 32 : D / 8;
  constexpr int kRowsPerInstr = 32 / kChunks;
  const int lane = threadIdx.x & 31, sub = lane / kChunks, cch = lane % kChunks;
  const bool c_in_tile = !kWide || cch < D / 8;
  const bool c_live = !kWide || cch < d_chunks;
  const uint32_t s_base = smem_u32(smem);
  // K extra: every row (1, 1, 1, 0, ...); Q extra: (-hi, -mid, -lo, 0, ...) of lse / scale
  const uint32_t one = kFp16 ? 0x3C00u : 0x3F80u;
  uint8_t* xt = smem + L::kX;
  const int r = row0 + lane;
  uint4 kv0 = make_uint4(one | (one << 16), one, 0, 0);
  float x = 3.0e38f;                                 // padding rows: exp(-huge) = 0
  if (kFp16) x = 60000.f;
  const int m = m0 + (r >> 7), rr = r & 127, q_row0 = m * group_rows;
  const int rows_valid = m < M ? min(group_rows, Lq - q_row0) : 0;
  if (rr < rows_valid) x = lse[q_row0 + rr] * inv_scale;
  uint32_t w0, w1;
  if (kFp16) {
    const __half hi = __float2half_rn(x);
    const float r1 = x - __half2float(hi);
    const __half mid = __float2half_rn(r1);
    const __half lo = __float2half_rn(r1 - __half2float(mid));
    w0 = (uint32_t)__half_as_ushort(__hneg(hi)) | ((uint32_t)__half_as_ushort(__hneg(mid)) << 16);
    w1 = (uint32_t)__half_as_ushort(__hneg(lo));
  } else {
    const __nv_bfloat16 hi = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(hi);
    const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
    const __nv_bfloat16 lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
    w0 = (uint32_t)__bfloat16_as_ushort(__hneg(hi)) | ((uint32_t)__bfloat16_as_ushort(__hneg(mid)) << 16);
    w1 = (uint32_t)__bfloat16_as_ushort(__hneg(lo));
  }
  // two chunks of the row carry the 16 columns of a k-step
  *reinterpret_cast<uint4*>(xt + swz(r, 0)) = kv0;
  *reinterpret_cast<uint4*>(xt + swz(r, 1)) = make_uint4(0, 0, 0, 0);
  *reinterpret_cast<uint4*>(xt + swz(r, 2)) = make_uint4(w0, w1, 0, 0);
  *reinterpret_cast<uint4*>(xt + swz(r, 3)) = make_uint4(0, 0, 0, 0);
  // Q rows (through the permutation if given)
  int src = -1;
  if (rr < rows_valid) {
    src = q_row0 + rr;
    if (perm != nullptr) src = static_cast<int>(perm[src]);
  }
#pragma unroll
  for (int i = 0; i < 32 / kRowsPerInstr; ++i) {
    const int rl = i * kRowsPerInstr + sub;
    const int id = __shfl_sync(0xffffffffu, src, rl);
    const uint32_t dst = s_base + L::kQ + swz<L::kQRows>(row0 + rl, cch);
    if (c_in_tile) {
      if (id >= 0 && c_live) cp_async16(dst, qb + cch * 16 + (size_t)id * q_row);
      else cp_async16_zfill(dst, qb, 0);
    }
  }
}

template <int D, bool kFp16, int G>
__global__ void __launch_bounds__(kThreads, 1) group_mass_kernel(const GroupMassParams p, const __grid_constant__ KeyTileMap kmap, int splits) {
  // key tiles are 128 consecutive rows: with a valid tensor map one elected thread loads them by TMA
  const bool use_tma = kmap.valid != 0;
  using L = Smem<D, G>;
  constexpr bool kWide = D > 128;                       // padded layouts: the true head dimension is p.D < D
  constexpr int R = L::kRingN;
  const int d_chunks = p.D / 8;                          // 16-byte chunks of a real row
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t s_base = smem_u32(smem);
  const uint32_t bars = s_base + L::kBars;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kTmemSlot);
  auto bar = [&](int i) { return bars + 8u * i; };
  auto sRing = [&](int slot) { return s_base + L::kRingOff + slot * L::kTileBytes; };
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // provably warp-uniform

  // work item: a group (or two neighbouring ones) of one (batch, head) and one of `splits` stretches of its key tiles
  const int sets = (p.M + G - 1) / G;
  const int split = blockIdx.x % splits, set = blockIdx.x / splits;
  const int m0 = set % sets * G;
  const int bh = set / sets;
  const int h = bh % p.H, b = bh / p.H;
  const int all_tiles = (p.Lk + kTile - 1) / kTile;
  const int tile0 = static_cast<int>((long long)all_tiles * split / splits);
  const int n_tiles = static_cast<int>((long long)all_tiles * (split + 1) / splits) - tile0;
  auto rows_of = [&](int m) { return m < p.M ? min(p.group_rows, p.Lq - m * p.group_rows) : 0; };

  if (tid == 0) {
    for (int i = 0; i < R; ++i) {
      mbar_init(bar(BAR_FULL + i), use_tma ? 1 : kProducerThreads);
      mbar_init(bar(BAR_EMPTY + i), 1);
    }
    mbar_init(bar(BAR_Q_FULL), 2 * L::kQRows);          // per thread: its cp.async rows + its plain stores
    for (int i = 0; i < kBufs; ++i) {
      mbar_init(bar(BAR_S_FULL + i), 1);
      mbar_init(bar(BAR_S_FREE + i), G == 2 ? kExpWarps : kExpWarps / 2);
    }
    for (int i = 0; i < 4 * kBufs; ++i) mbar_init(bar(BAR_PART + i), 1);
    mbar_init(bar(BAR_DRAIN), 1);
    mbar_fence_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // The query operand: a block of 32 rows for each of the first exponentiating warps, which would wait for scores anyway; the
  // producers start on the keys at once.  (By the producers, before their first key tile: 9.3 us instead of 6.6 for one group
  // against one tile at D = 96 to 192.)
  if (warp < L::kQRows / 32) {
    prepare_queries<D, kFp16, G>(smem, p.lse + (size_t)bh * p.Lq, p.perm == nullptr ? nullptr : p.perm + (size_t)bh * p.Lq,
                                 reinterpret_cast<const uint8_t*>(p.q) + 2 * ((size_t)b * p.q_stride[0] + (size_t)h * p.q_stride[2]),
                                 2 * (size_t)p.q_stride[1], m0, p.M, p.group_rows, p.Lq, p.inv_scale, d_chunks, warp * 32);
    fence_proxy_async_smem();
    mbar_arrive(bar(BAR_Q_FULL));                        // release: the plain stores above
    cp_async_arrive_noinc(bar(BAR_Q_FULL));
  }

  if (warp < kExpWarps) {
    // ===================================================================== exp + column sum
    const int lg = warp & 3, x = (warp >> 2) & 1;      // TMEM lane group, column half
    const int j_in = lg * 32 + lane;                   // key token inside the tile == TMEM lane
    const uint32_t lane_addr = (static_cast<uint32_t>(lg) * 32u) << 16;
    const float c = p.scale_log2;
    const float xmin = -125.f / c;
    // two groups: each eight warps take one group's columns of every tile (two buffers of 256 columns); one group: the
    // even and the odd tiles (four buffers of 128)
    const int eg = warp >> 3, m = G == 2 ? m0 + eg : m0;
    const float norm = p.normalize ? 1.f / static_cast<float>(max(rows_of(m), 1)) : 1.f;
    float* out = p.mass + ((size_t)bh * p.M + min(m, p.M - 1)) * p.Lk;
    float* part = reinterpret_cast<float*>(smem + L::kPart);
    bool ok = true;
#pragma unroll 1
    for (int t = G == 2 ? 0 : eg; t < n_tiles && ok; t += G == 2 ? 1 : 2) {
      constexpr int kB = G == 2 ? 2 : kBufs;
      const int buf = t & (kB - 1), ph = (t / kB) & 1;
      const int pb = G == 2 ? 2 * eg + buf : buf;        // place of the partial sums
      const uint32_t tS = tmem + (G == 2 ? buf * 256 + eg * 128 : buf * 128) + x * 64 + lane_addr;
      ok = mbar_wait(bar(BAR_S_FULL + buf), ph, p.status, 40);
      if (!ok) break;
      tc_fence_after();
      float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t r[32];
        tmem_ld32(tS + q * 32, r);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          // Two of every eight exponentials are computed on the FMA pipe instead of the special-function unit
          // (see ex2_poly3_scaled); their positions are spread over the four partial sums.
          // Two measured best (6.52 ms against 6.69 / 6.88 ms with one / three at H=24, L=32,760: beyond a
          // quarter the extra instructions cost more issue slots than the unit gains).
          auto e = [&](int k) {
            const float v = __uint_as_float(r[i + k]);
            return k == 3 || k == 6 ? ex2_poly3_scaled(v, c, xmin) : ex2_approx(v * c);
          };
          a0 += e(0); a1 += e(1); a2 += e(2); a3 += e(3);
          a0 += e(4); a1 += e(5); a2 += e(6); a3 += e(7);
        }
      }
      tc_fence_before();
      const float sum = (a0 + a1) + (a2 + a3);
      // The two halves of a row meet in shared memory, in one place per score buffer, and are handed over
      // through an mbarrier (a bounded wait, unlike a named barrier).  The lower half releases the score
      // buffer only after it has read the partner's sums, so the partner's next write to that place (which
      // needs the release to get the buffer's next scores) cannot overtake the read.  (Copying all 64 values to
      // registers first and releasing the score buffer before the exponentials measured 10% slower.)
      if (x == 1) {
        part[pb * 128 + j_in] = sum;
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar(BAR_PART + kBufs * lg + pb));
          mbar_arrive(bar(BAR_S_FREE + buf));              // one arrival per warp
        }
      } else {
        ok = mbar_wait(bar(BAR_PART + kBufs * lg + pb), ph, p.status, 45);
        if (!ok) break;
        const int j = (tile0 + t) * kTile + j_in;
        if (j < p.Lk && m < p.M) out[j] = (sum + part[pb * 128 + j_in]) * norm;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(BAR_S_FREE + buf));
      }
    }
    cp_async_wait_all();
    tc_fence_before();
  } else if (warp == kMmaWarp) {
    // ===================================================================== MMA issuer
    {
      const bool leader = elect_one();
      constexpr uint32_t kFmt = kFp16 ? 0u : 1u;
      constexpr uint32_t idesc = mma_idesc(kFmt, kFmt, 0, 0, 128, 128 * G);
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
      constexpr uint32_t kLbo = (16u >> 4) << 16;
      auto desc = [&](uint32_t lo) { return (static_cast<uint64_t>(kDescHi) << 32) | lo; };
      const uint32_t qlo = (((s_base + L::kQ) & 0x3FFFFu) >> 4) | kLbo;
      const uint32_t kxlo = (((s_base + L::kX) & 0x3FFFFu) >> 4) | kLbo;
      const uint32_t qxlo = kxlo + 2;                    // second 32-byte k-step of the same rows
      bool ok = mbar_wait(bar(BAR_Q_FULL), 0, p.status, 41);
      int slot = 0, phase = 0;
#pragma unroll 1
      for (int t = 0; t < n_tiles && ok; ++t) {
        constexpr int kB = G == 2 ? 2 : kBufs;
        const int buf = t & (kB - 1);
        if (t >= kB) ok = mbar_wait(bar(BAR_S_FREE + buf), (t / kB - 1) & 1, p.status, 42);
        ok = ok && mbar_wait(bar(BAR_FULL + slot), phase, p.status, 43);
        if (!ok) break;
        fence_proxy_async_smem();
        tc_fence_after();
        const uint32_t tS = tmem + buf * 128 * G;
        const uint32_t klo = ((sRing(slot) & 0x3FFFFu) >> 4) | kLbo;
        if constexpr (kWide) {
          // the k-steps that hold real columns (the last one zero-padded to 16)
          const int ksteps = (p.D + 15) / 16;
#pragma unroll 1
          for (int j = 0; j < ksteps; ++j) {
            const uint32_t koff = (j >> 2) * (16384 >> 4) + (j & 3) * 2;
            if (leader) mma_f16_ss(tS, desc(klo + koff), desc(qlo + koff), idesc, j > 0);
          }
        } else {
#pragma unroll
          for (int j = 0; j < D / 16; ++j) {
            const uint32_t koff = (j >> 2) * (16384 >> 4) + (j & 3) * 2, qoff = (j >> 2) * (16384 * G >> 4) + (j & 3) * 2;
            if (leader) mma_f16_ss(tS, desc(klo + koff), desc(qlo + qoff), idesc, j > 0);     // A = K tile, B = query rows
          }
        }
        if (leader) {
          mma_f16_ss(tS, desc(kxlo), desc(qxlo), idesc, 1);                     // extra k-step: - lse / scale
          tc_commit(bar(BAR_EMPTY + slot));
          tc_commit(bar(BAR_S_FULL + buf));
        }
        if (++slot == R) { slot = 0; phase ^= 1; }
      }
      if (!ok) {
        if (leader) tc_commit(bar(BAR_DRAIN));
        mbar_wait_quiet(bar(BAR_DRAIN), 0, 1 << 20);
      }
    }
    __syncwarp();
    tc_fence_before();
  } else {
    // ===================================================================== producers
    const int pw = warp - kProducerWarp0;
    // one lane per 16-byte chunk of a row; the padded layouts give every lane one of 32 chunk positions, of which
    // D / 8 exist in the tile (the others idle) and p.D / 8 hold data (the rest is zero-filled)
    constexpr int kChunks = kWide ? 32 : D / 8;
    constexpr int kRowsPerInstr = 32 / kChunks;
    const int sub = lane / kChunks, cch = lane % kChunks;
    const bool c_in_tile = !kWide || cch < D / 8;
    const bool c_live = !kWide || cch < d_chunks;
    // ---- key tiles: contiguous rows t*128 .. t*128+127 of this head
    int n_tiles_cp = n_tiles;       // tiles copied with cp.async (none when TMA is used)
    const uint8_t* kb = reinterpret_cast<const uint8_t*>(p.k) + 2 * ((size_t)b * p.k_stride[0] + (size_t)h * p.k_stride[2]) + cch * 16;
    const size_t k_row = 2 * (size_t)p.k_stride[1];
    int slot = 0, phase = 0;
    bool wrapped = false, ok = true;
    const bool tma_leader = elect_one();
    if (use_tma) {
      // one thread of producer warp 0 issues every tile as D / 64 boxes of 128 rows x 128 bytes; rows beyond the
      // end of the sequence arrive as zeros
      if (pw == 0) {
        int co[4] = {0, 0, 0, 0};
        co[kmap.pos_h] = h;
        co[kmap.pos_b] = b;
#pragma unroll 1
        for (int t = 0; t < n_tiles && ok; ++t) {
          if (wrapped) ok = mbar_wait(bar(BAR_EMPTY + slot), phase ^ 1, p.status, 44);
          if (!ok) break;
          if (tma_leader) {
            mbar_arrive_expect_tx(bar(BAR_FULL + slot), L::kTileBytes);
            co[kmap.pos_row] = (tile0 + t) * kTile;
#pragma unroll
            for (int cb = 0; cb < L::kBlocks; ++cb)
              tma_load_4d(sRing(slot) + cb * 16384, kmap.k, cb * 64, co[1], co[2], co[3], bar(BAR_FULL + slot));
          }
          if (++slot == R) { slot = 0; phase ^= 1; wrapped = true; }
        }
      }
      n_tiles_cp = 0;
    }
#pragma unroll 1
    for (int t = 0; t < n_tiles_cp && ok; ++t) {
      if (wrapped) ok = mbar_wait(bar(BAR_EMPTY + slot), phase ^ 1, p.status, 44);
      if (!ok) break;
      const uint32_t dst0 = sRing(slot);
#pragma unroll 4
      for (int i = pw; i < 128 / kRowsPerInstr; i += kProducerWarps) {
        const int rl = i * kRowsPerInstr + sub;
        const int krow = (tile0 + t) * kTile + rl;
        const uint32_t dst = dst0 + swz(rl, cch);
        if (c_in_tile) {
          if (krow < p.Lk && c_live) cp_async16(dst, kb + (size_t)krow * k_row);
          else cp_async16_zfill(dst, p.k, 0);
        }
      }
      cp_async_arrive_noinc(bar(BAR_FULL + slot));
      if (++slot == R) { slot = 0; phase ^= 1; wrapped = true; }
    }
    cp_async_wait_all();
  }

  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

// (splits: for pairs of groups, see pair_splits; a single group takes all of its head's keys)
template <int D, bool kFp16, int G = 1>
int launch(const GroupMassParams& p, cudaStream_t stream, int splits = 1) {
  using L = Smem<D, G>;
  auto kern = group_mass_kernel<D, kFp16, G>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynamic) != cudaSuccess) return -8;
  const long long grid = (long long)p.B * p.H * ((p.M + G - 1) / G) * splits;
  KeyTileMap kmap{};
  // (the map carries the true head dimension: boxes that reach beyond it are zero-filled by the copy engine)
  kmap.valid = encode_tile_map(p.k, p.k_stride, p.B, p.Lk, p.H, p.D, kmap.k, kmap.pos_h, kmap.pos_row, kmap.pos_b);
  kern<<<(unsigned)grid, kThreads, L::kDynamic, stream>>>(p, kmap, splits);
  return cudaGetLastError() == cudaSuccess ? 0 : -8;
}

// Two groups per CTA (D = 128): one 128 x 256 product per key tile reads the keys once for both groups, where two 128 x 128
// products read both operands from shared memory at its full rate: 6,516 -> 6,125 us at 24 heads x 32,760, 556 -> 535 at
// 8 x 16,380.  But the items are twice as large: 24 heads x 4,680 (888 groups, six full waves) 178 -> 200 us.  Rows of the
// result do not depend on one another, so the key tiles of a pair may go to several CTAs.  Returns the number of CTAs per
// pair, or 0 for one group per CTA, by the length of the launch in key tiles of one group: a CTA's start (barriers, tensor
// memory, its query rows) is about four, a tile of two groups 1.9.  (At D = 64 the products are half as long: 96 us against
// 110 at 12 heads x 4,700; beside the wider tiles two groups do not fit.)
int pair_splits(const GroupMassParams& p) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long bh = (long long)p.B * p.H, tiles = ((long long)p.Lk + kTile - 1) / kTile;
  auto waves = [&](long long ctas) { return (double)((ctas + sms - 1) / sms); };
  double best = waves(bh * p.M) * ((double)tiles + 4.0);
  int splits = 0;
  for (int s = 1; s <= 8 && s <= tiles; ++s) {
    const long long ctas = bh * ((p.M + 1) / 2) * s;
    const double cost = waves(ctas) * ((double)((tiles + s - 1) / s) * 1.9 + 4.0);
    if (cost < best && ctas <= 0x7fffffffLL) { best = cost; splits = s; }
  }
  return splits;
}

}  // namespace

int launch_group_mass(const GroupMassParams& p, bool fp16, cudaStream_t stream) {
  if (p.D == 128) {
    const int splits = pair_splits(p);
    if (splits > 0) return fp16 ? launch<128, true, 2>(p, stream, splits) : launch<128, false, 2>(p, stream, splits);
    return fp16 ? launch<128, true>(p, stream) : launch<128, false>(p, stream);
  }
  if (p.D == 64) return fp16 ? launch<64, true>(p, stream) : launch<64, false>(p, stream);
  // every other multiple of 8 up to 256 (the reference's head-dimension table has 96, 144, 160, 192, 256): padded layouts
  if (p.D < 8 || p.D > 256 || p.D % 8 != 0) return -3;
  if (p.D <= 192) return fp16 ? launch<192, true>(p, stream) : launch<192, false>(p, stream);
  return fp16 ? launch<256, true>(p, stream) : launch<256, false>(p, stream);
}

}  // namespace mcs
