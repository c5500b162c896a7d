// Fast PDDP query grouping (recursive principal-direction bisection) for sm_100a.
//
// Restates mcsparse/kernels/flash_mcsa/pca_group.py:141-243.  Tokens of each (batch, head) are
// reordered so that every aligned block of C tokens holds similar vectors: at each level every
// node (a contiguous interval of the current order) computes the principal direction of its
// centred rows with a few power iterations on the Gram matrix X^T X - s s^T / n, sorts its rows
// by their projection on that direction and is split at the block-aligned midpoint.
//
// Per level, with no host synchronisation anywhere (the tree shape depends only on N and C):
//   node     tcgen05: G += X_tile^T X_tile over 128-row tiles gathered through the current permutation.  The SAME
//            shared-memory tile serves as both MMA operands (MN-major A and MN-major B); a second, 16-column MMA
//            against a tile of ones yields the column sums s.  A node of up to 2048 rows is finished by its CTA: centre,
//            normalise the start vector, iterate, project its rows (fp32), emit 64-bit sort keys (order-preserving
//            float bits << 32 | position inside the node: unique keys, so the sort is stable by construction).
//   power, project   the same for nodes of several 2048-row items, whose partial sums are added in a fixed order
//            (deterministic, no atomics).
//   sort     bitonic network over power-of-two padded segments, out of registers; global compare-exchange steps when a
//            segment exceeds one CTA's tile.  The last kernel writes the new order.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <vector>

#include "kernels.cuh"
#include "pddp_key.cuh"
#include "ptx.cuh"

namespace mcs {

namespace {

constexpr int kChunkRows = 2048;        // rows per gram work item
constexpr int kSortTile = 4096;         // keys per CTA in the shared-memory sort stages
constexpr int kMaxNodes = 4096;

// ------------------------------------------------------------------------------------------
// Tree shape (pure function of N, C): used identically on host (launch sizes) and device (tables).
// ------------------------------------------------------------------------------------------
struct LevelShape {
  int nodes;        // nodes at this level
  int items;        // gram work items (sum over nodes of ceil(size / kChunkRows))
  int pad;          // power of two >= largest node size
};

__host__ __device__ inline int next_pow2(int v) { int p = 1; while (p < v) p <<= 1; return p; }

// Fills block-interval arrays for successive levels.  lo/hi hold the current level (in blocks).
// Returns false when no interval has more than one block (no further level).
__host__ __device__ inline bool any_splittable(const int* lo, const int* hi, int n) {
  for (int i = 0; i < n; ++i) if (hi[i] - lo[i] > 1) return true;
  return false;
}
__host__ __device__ inline int split_level(const int* lo, const int* hi, int n, int* lo2, int* hi2) {
  int m = 0;
  for (int i = 0; i < n; ++i) {
    if (hi[i] - lo[i] <= 1) { lo2[m] = lo[i]; hi2[m] = hi[i]; ++m; }
    else {
      const int mid = lo[i] + (hi[i] - lo[i]) / 2;
      lo2[m] = lo[i]; hi2[m] = mid; ++m;
      lo2[m] = mid; hi2[m] = hi[i]; ++m;
    }
  }
  return m;
}

// Device tables of one level, laid out consecutively in the workspace.
struct LevelTables {
  int* node_start;   // [nodes] token start
  int* node_size;    // [nodes]
  int* node_item0;   // [nodes] first gram item of the node
  int* item_node;    // [items]
  int* item_row0;    // [items] first row (relative to node start)
};

// One CTA; a level's intervals are handled 1,024 at a time, with one scan for the positions of their work items and of
// their children (a single thread walking the lists took 73 us for 256 blocks).
constexpr int kTableThreads = 1024;
__global__ void __launch_bounds__(kTableThreads) pddp_tables_kernel(int N, int C, int* tab, int max_levels, int stride) {
  __shared__ unsigned long long warp_tot[kTableThreads / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int K = (N + C - 1) / C;
  // two scratch interval lists live at the end of the table area
  int* lo = tab + (size_t)max_levels * stride;
  int* hi = lo + kMaxNodes;
  int* lo2 = hi + kMaxNodes;
  int* hi2 = lo2 + kMaxNodes;
  if (tid == 0) { lo[0] = 0; hi[0] = K; }
  __syncthreads();
  int n = 1;
  for (int lv = 0; lv < max_levels; ++lv) {
    int* t = tab + (size_t)lv * stride;
    int* node_start = t, *node_size = t + kMaxNodes, *node_item0 = t + 2 * kMaxNodes;
    int* item_node = t + 3 * kMaxNodes, *item_row0 = item_node + (stride - 3 * kMaxNodes) / 2;
    unsigned long long run = 0ull;                       // (work items << 32 | children) of the intervals before this batch
    for (int i0 = 0; i0 < n; i0 += kTableThreads) {
      const int i = i0 + tid;
      int l = 0, h = 0, size = 0;
      unsigned long long v = 0ull;
      if (i < n) {
        l = lo[i]; h = hi[i];
        size = min(h * C, N) - l * C;
        v = ((unsigned long long)((size + kChunkRows - 1) / kChunkRows) << 32) | (h - l > 1 ? 2u : 1u);
      }
      unsigned long long incl = v;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long m = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += m;
      }
      if (lane == 31) warp_tot[warp] = incl;
      __syncthreads();
      unsigned long long before = run, all = run;
      for (int w = 0; w < kTableThreads / 32; ++w) {
        if (w < warp) before += warp_tot[w];
        all += warp_tot[w];
      }
      before += incl - v;
      if (i < n) {
        const int item0 = (int)(before >> 32), c0 = (int)(before & 0xFFFFFFFFull);
        node_start[i] = l * C; node_size[i] = size; node_item0[i] = item0;
        for (int r = 0, it = item0; r < size; r += kChunkRows, ++it) { item_node[it] = i; item_row0[it] = r; }
        if (h - l > 1) {
          const int mid = l + (h - l) / 2;
          lo2[c0] = l; hi2[c0] = mid; lo2[c0 + 1] = mid; hi2[c0 + 1] = h;
        } else {
          lo2[c0] = l; hi2[c0] = h;
        }
      }
      run = all;
      __syncthreads();
    }
    n = (int)(run & 0xFFFFFFFFull);
    int* x = lo; lo = lo2; lo2 = x;
    x = hi; hi = hi2; hi2 = x;
  }
}

__device__ __forceinline__ LevelTables level_tables(int* tab, int lv, int stride) {
  int* t = tab + (size_t)lv * stride;
  LevelTables T;
  T.node_start = t; T.node_size = t + kMaxNodes; T.node_item0 = t + 2 * kMaxNodes;
  T.item_node = t + 3 * kMaxNodes; T.item_row0 = T.item_node + (stride - 3 * kMaxNodes) / 2;
  return T;
}

__device__ __forceinline__ uint32_t swz(int row, int c) {
  return static_cast<uint32_t>((c >> 3) * 16384 + row * 128 + (((c & 7) ^ (row & 7)) << 4));
}

__device__ __forceinline__ uint32_t float_key(float f) {
  uint32_t u = __float_as_uint(f);
  if (f == 0.f) u = 0u;                                        // -0 == +0
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

constexpr int kProjRows = 8;            // (wide path) rows per warp: eight independent row loads in flight per lane
constexpr int kNodeThreads = 160;       // 4 gather / epilogue warps + 1 MMA warp
constexpr int kBufs = 3;                // 128-row tiles in flight per CTA
constexpr int kTileBytes = 32768;
constexpr int kPartialFloats = 128 * 128 + 128;

struct NodeSmem {
  static constexpr int kOnes = kBufs * kTileBytes;             // 16 rows x 128 B of ones
  static constexpr int kVec = kOnes + 2048;                    // float [128]
  static constexpr int kSum = kVec + 512;                      // float [128]
  static constexpr int kRed = kSum + 512;                      // float [4]
  static constexpr int kBars = kRed + 16;                      // kBufs full, kBufs empty, done, drain
  static constexpr int kSlot = kBars + (2 * kBufs + 2) * 8;
  static constexpr int kDynamic = kSlot + 16 + 1024;
};

// One warp copies rows 32 * warp .. + 31 of a tile of gathered rows; lane l holds the source row of tile row
// 32 * warp + l (negative: zero row).  D / 8 lanes cover one row, so every request is whole rows.
template <int D>
__device__ __forceinline__ void gather_tile_rows(uint32_t tile, int warp, int lane, int my_id, const uint8_t* xb, size_t row_bytes) {
  constexpr int kChunks = D / 8, kRpi = 32 / kChunks;
  const int sub = lane / kChunks, c = lane % kChunks;
#pragma unroll
  for (int i = 0; i < 32 / kRpi; ++i) {
    const int rl = i * kRpi + sub;
    const int id = __shfl_sync(0xffffffffu, my_id, rl);
    const uint32_t dst = tile + swz(warp * 32 + rl, c);
    if (id >= 0) cp_async16(dst, xb + (size_t)id * row_bytes + c * 16);
    else cp_async16_zfill(dst, xb, 0);
  }
}

// fp32 projection of tile row `row` on vec.  The additions are those of a warp that holds four elements per lane and
// reduces by butterflies from distance 16 down: element group l with group l + 16 first, then + 8, + 4, + 2, + 1.
template <int D, bool kFp16>
__device__ __forceinline__ float project_row(uint32_t tile, int row, const float* vec) {
  auto quad = [&](uint32_t w0, uint32_t w1, const float4 v) {
    float2 a, b;
    if (kFp16) {
      a = __half22float2(*reinterpret_cast<const __half2*>(&w0));
      b = __half22float2(*reinterpret_cast<const __half2*>(&w1));
    } else {
      a = make_float2(bf16_lo(w0), bf16_hi(w0));
      b = make_float2(bf16_lo(w1), bf16_hi(w1));
    }
    return fmaf(a.x, v.x, fmaf(a.y, v.y, fmaf(b.x, v.z, b.y * v.w)));
  };
  const float4* v4 = reinterpret_cast<const float4*>(vec);
  float s[16];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint4 w = lds_v4(tile + swz(row, c));
    s[2 * c] = quad(w.x, w.y, v4[2 * c]);
    s[2 * c + 1] = quad(w.z, w.w, v4[2 * c + 1]);
    if (D == 128) {
      const uint4 u = lds_v4(tile + swz(row, c + 8));
      s[2 * c] += quad(u.x, u.y, v4[2 * c + 16]);
      s[2 * c + 1] += quad(u.z, u.w, v4[2 * c + 17]);
    }
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1)
#pragma unroll
    for (int l = 0; l < o; ++l) s[l] += s[l + o];
  return s[0];
}

// Projects `rows` gathered rows (positions pos0 .. of head bh, which are r_first .. of their node) on vec and writes
// their sort keys.  128 threads, thread == row of a tile; a warp consumes only rows that it gathered itself, so the tiles
// need no barrier.  With `resident`, tile t already lies in buffer t.
template <int D, bool kFp16>
__device__ __forceinline__ void project_rows(uint32_t s_base, int warp, int lane, const uint8_t* xb, size_t row_bytes, const int* ids,
                                             int rows, int r_first, const float* vec, unsigned long long* keys, float* proj_out,
                                             bool resident) {
  const int n_tiles = (rows + 127) / 128, mine = warp * 32 + lane;
  auto load_id = [&](int t) { const int r = t * 128 + mine; return r < rows ? ids[r] : -1; };
  int id_next = 0;
  if (!resident) {
#pragma unroll
    for (int t = 0; t < kBufs - 1; ++t) {
      if (t < n_tiles) gather_tile_rows<D>(s_base + t * kTileBytes, warp, lane, load_id(t), xb, row_bytes);
      cp_async_commit_group();
    }
    id_next = load_id(kBufs - 1);
  }
  int buf = 0, fill = kBufs - 1;
#pragma unroll 1
  for (int t = 0; t < n_tiles; ++t) {
    if (!resident) {
      // tile t + kBufs - 1 goes where tile t - 1 was (read by this warp alone, one iteration ago)
      if (t + kBufs - 1 < n_tiles) gather_tile_rows<D>(s_base + fill * kTileBytes, warp, lane, id_next, xb, row_bytes);
      cp_async_commit_group();
      id_next = load_id(t + kBufs);
      cp_async_wait_group<kBufs - 1>();
      __syncwarp();
    }
    const float a = project_row<D, kFp16>(s_base + buf * kTileBytes, mine, vec);
    const int r = t * 128 + mine;
    if (r < rows) {
      keys[r_first + r] = sort_key(float_key(a), r_first + r);
      if (proj_out != nullptr) proj_out[r] = a;
    }
    __syncwarp();
    buf = buf + 1 == kBufs ? 0 : buf + 1;
    fill = fill + 1 == kBufs ? 0 : fill + 1;
  }
}

// ------------------------------------------------------------------------------------------
// node: Gram matrix of an item's rows; for a node that is one item also its principal direction and its sort keys
//
// Bound by the gathered reads of X (whole rows, 16 or 8 lanes each, kBufs tiles in flight per CTA and two CTAs per SM).
// A node of one item (up to kChunkRows rows: half of the levels and most of the nodes) never leaves its CTA: the Gram
// matrix stays in tensor memory, thread d holds row d, the power iterations are dot products of that row with a vector
// in shared memory, and the projections read the tiles that are still in shared memory (nodes of up to kBufs tiles) or
// gather them again out of L2.  Larger nodes write their partial sums for the power kernel; G is symmetric, so thread d
// writes column d and every store is one 128-byte line per warp.
// Same sums in the same order as a kernel per stage had: identical permutations.
// Measured (24 heads x 32,760 tokens x 128, 8 levels, kernel times of one call): Gram 1,140 + power 638 + project 556 us
// before; node 581 + power 63 + project 192 us now (X read twice per level at the measured copy rate: 490 us).  Of that,
// lanes that load whole rows instead of a row each, the transposed partial store and the fused power step are the most.
// ------------------------------------------------------------------------------------------
template <int D, bool kFp16>
__global__ void __launch_bounds__(kNodeThreads, 2) pddp_node_kernel(PddpParams p, int lv, int nodes, int pad, const int* perm_in,
                                                                    const float* v0, float* proj_out) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  using S = NodeSmem;
  const uint32_t s_base = smem_u32(smem);
  const uint32_t sOnes = s_base + S::kOnes;
  const uint32_t bars = s_base + S::kBars;
  float* vec = reinterpret_cast<float*>(smem + S::kVec);
  float* ssum = reinterpret_cast<float*>(smem + S::kSum);
  float* red = reinterpret_cast<float*>(smem + S::kRed);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + S::kSlot);
  enum { FULL = 0, EMPTY = kBufs, DONE = 2 * kBufs };
  auto bar = [&](int i) { return bars + 8u * i; };
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const LevelTables T = level_tables(p.tables, lv, p.table_stride);
  const int item = blockIdx.x, bh = blockIdx.y;
  const int node = T.item_node[item];
  const int row_begin = T.item_row0[item];
  const int size = T.node_size[node];
  const int rows = min(kChunkRows, size - row_begin);
  const int pos0 = T.node_start[node] + row_begin;
  const int n_tiles = (rows + 127) / 128;

  if (tid == 0) {
    for (int i = 0; i < kBufs; ++i) { mbar_init(bar(FULL + i), 128); mbar_init(bar(EMPTY + i), 1); }
    mbar_init(bar(DONE), 1);
    mbar_fence_init();
  }
  if (warp == 4) { tmem_alloc(smem_u32(tmem_slot), 256); tmem_relinquish(); }
  // ones tile: rows 0..15 (N = 16), 16 K-columns of 1.0 (K-major, 128-byte swizzled rows)
  if (tid < 16) {
    const uint32_t one2 = kFp16 ? 0x3C003C00u : 0x3F803F80u;
    *reinterpret_cast<uint4*>(smem + S::kOnes + swz(tid, 0)) = make_uint4(one2, one2, one2, one2);
    *reinterpret_cast<uint4*>(smem + S::kOnes + swz(tid, 1)) = make_uint4(one2, one2, one2, one2);
  }
  if (D == 64) {
    // features 64..127 of the 128-wide product do not exist: their column block is zero once and for all
    for (int i = tid; i < kBufs * 1024; i += kNodeThreads)
      *reinterpret_cast<uint4*>(smem + (i >> 10) * kTileBytes + 16384 + (i & 1023) * 16) = make_uint4(0u, 0u, 0u, 0u);
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp < 4) {
    // ---- gather rows of each tile through the permutation
    const uint8_t* xb = reinterpret_cast<const uint8_t*>(p.x) + 2 * (size_t)bh * p.x_stride_bh;
    const size_t row_bytes = 2 * (size_t)p.x_stride_row;
    const int* ids = perm_in + (size_t)bh * p.N + pos0;
    bool ok = true;
    // (in flight under the gather)
    const float v_start = (size <= kChunkRows && tid < D) ? v0[((size_t)bh * nodes + node) * D + tid] : 0.f;
    {
      int id_next = tid < rows ? ids[tid] : -1;
      int buf = 0, phase = 0;
#pragma unroll 1
      for (int t = 0; t < n_tiles && ok; ++t) {
        const int id = id_next, r1 = (t + 1) * 128 + tid;
        id_next = r1 < rows ? ids[r1] : -1;
        if (t >= kBufs) ok = mbar_wait(bar(EMPTY + buf), phase ^ 1, p.status, 60);
        if (!ok) break;
        gather_tile_rows<D>(s_base + buf * kTileBytes, warp, lane, id, xb, row_bytes);
        cp_async_arrive_noinc(bar(FULL + buf));
        if (++buf == kBufs) { buf = 0; phase ^= 1; }
      }
    }
    cp_async_wait_all();
    if (ok) ok = mbar_wait(bar(DONE), 0, p.status, 61);
    // (the four warps agree, so that none waits at the named barriers below for one that has given up)
    ok = !named_bar_red_or(1, 128, !ok);
    if (ok) {
      tc_fence_after();
      const int d = tid;                                       // feature row of G == TMEM lane
      const uint32_t lane_addr = (static_cast<uint32_t>(warp) * 32u) << 16;
      uint32_t r8[8];
      tmem_ld8(tmem + lane_addr + 128, r8);
      tmem_wait_ld();
      const float s_d = __uint_as_float(r8[0]);
      if (size > kChunkRows) {
        float* out = p.partial + ((size_t)bh * p.max_items + item) * kPartialFloats;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t r[32];
          tmem_ld32(tmem + lane_addr + c * 32, r);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) out[(size_t)(c * 32 + i) * 128 + d] = __uint_as_float(r[i]);
        }
        out[128 * 128 + d] = s_d;
      } else {
        // ---- centred Gram matrix, back in tensor memory
        ssum[d] = s_d;
        named_bar_sync(1, 128);
        const float inv_n = 1.f / (float)size;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t r[32];
          tmem_ld32(tmem + lane_addr + c * 32, r);
          tmem_wait_ld();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              r8[i] = __float_as_uint(__uint_as_float(r[q * 8 + i]) - ssum[c * 32 + q * 8 + i] * s_d * inv_n);
            tmem_st8(tmem + lane_addr + c * 32 + q * 8, r8);
          }
        }
        tmem_wait_st();
        // ---- power iterations
        auto sum_128 = [&](float x) {
          for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
          if (lane == 0) red[warp] = x;
          named_bar_sync(1, 128);
          return (red[0] + red[1]) + (red[2] + red[3]);
        };
        float v = v_start;
        float nrm = sqrtf(sum_128(v * v));
        v /= fmaxf(nrm, 1e-12f);
        for (int iter = 0; iter < p.pow_iters; ++iter) {
          vec[d] = v;
          named_bar_sync(1, 128);
          float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
          for (int c = 0; c < D / 32; ++c) {
            uint32_t r[32];
            tmem_ld32(tmem + lane_addr + c * 32, r);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float4 x = reinterpret_cast<const float4*>(vec)[c * 8 + i];
              a[0] += __uint_as_float(r[4 * i]) * x.x;
              a[1] += __uint_as_float(r[4 * i + 1]) * x.y;
              a[2] += __uint_as_float(r[4 * i + 2]) * x.z;
              a[3] += __uint_as_float(r[4 * i + 3]) * x.w;
            }
          }
          v = (a[0] + a[1]) + (a[2] + a[3]);
          nrm = sqrtf(sum_128(v * v));
          v /= fmaxf(nrm, 1e-12f);
        }
        vec[d] = v;                                            // (every thread is past its last read: sum_128's barrier)
        named_bar_sync(1, 128);
        // ---- projections and sort keys; slots beyond the node sort last
        unsigned long long* keys = p.keys + (size_t)bh * p.key_stride + (size_t)node * pad;
        project_rows<D, kFp16>(s_base, warp, lane, xb, row_bytes, ids, rows, 0, vec, keys,
                               proj_out != nullptr ? proj_out + (size_t)bh * p.N + pos0 : nullptr, n_tiles <= kBufs);
        for (int r = rows + tid; r < pad; r += 128) keys[r] = kPadKey;
        cp_async_wait_all();
      }
    } else if (size <= kChunkRows) {
      // a wait expired (the status word says where): the node keeps its order, so that the sort finds a key in every slot
      unsigned long long* keys = p.keys + (size_t)bh * p.key_stride + (size_t)node * pad;
      for (int r = tid; r < pad; r += 128) keys[r] = r < rows ? sort_key(0u, r) : kPadKey;
    }
    tc_fence_before();
  } else {
    {
      constexpr uint32_t kFmt = kFp16 ? 0u : 1u;
      constexpr uint32_t idesc_g = mma_idesc(kFmt, kFmt, 1, 1, 128, 128);   // A and B both MN-major
      constexpr uint32_t idesc_s = mma_idesc(kFmt, kFmt, 1, 0, 128, 16);    // B = ones, K-major
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
      auto desc = [&](uint32_t lo) { return (static_cast<uint64_t>(kDescHi) << 32) | lo; };
      const uint32_t ones_lo = ((sOnes & 0x3FFFFu) >> 4) | (1u << 16);
      const bool leader = elect_one();
      bool ok = true;
      int buf = 0, phase = 0;
#pragma unroll 1
      for (int t = 0; t < n_tiles && ok; ++t) {
        ok = mbar_wait(bar(FULL + buf), phase, p.status, 62);
        if (!ok) break;
        fence_proxy_async_smem();
        tc_fence_after();
        const uint32_t xlo = (((s_base + buf * kTileBytes) & 0x3FFFFu) >> 4) | ((16384u >> 4) << 16);
#pragma unroll
        for (int j = 0; j < 8; ++j) {             // 16 rows per k-step
          const uint64_t dx = desc(xlo + j * (2048 >> 4));
          if (leader) {
            mma_f16_ss(tmem, dx, dx, idesc_g, (t > 0) || (j > 0));
            mma_f16_ss(tmem + 128, dx, desc(ones_lo), idesc_s, (t > 0) || (j > 0));
          }
        }
        if (leader) tc_commit(bar(EMPTY + buf));
        if (++buf == kBufs) { buf = 0; phase ^= 1; }
      }
      if (leader) tc_commit(bar(DONE));
      if (!ok) mbar_wait_quiet(bar(DONE), 0, 1 << 20);     // outstanding products retire before tensor memory is released
    }
    __syncwarp();
    tc_fence_before();
  }
  __syncthreads();
  if (warp == 4) { tc_fence_after(); tmem_dealloc(tmem, 256); }
}

// ------------------------------------------------------------------------------------------
// power: dir[bh][node] = principal direction of a node of several items (pow_iters normalised mat-vecs)
// ------------------------------------------------------------------------------------------

// 512 threads: thread (d, q) = (tid & 127, tid >> 7) owns element d and the Gram rows e = q (mod 4); accumulators a_q
// over e = q, q+4, ... in increasing order, combined as (a0 + a1) + (a2 + a3).  A level has only 1 to 8 such nodes per
// head: the kernel is bound by the latency of summing the partials, so eight elements of a chunk and several chunks
// are loaded at once.
__global__ void __launch_bounds__(512, 1) pddp_power_kernel(PddpParams p, int lv, int nodes, const float* v0) {
  extern __shared__ __align__(16) float sm[];
  float* G = sm;                 // 128 x 128, symmetric
  float* vec = sm + 128 * 128;   // 128
  float* partial = vec + 128;    // 4 x 128
  float* red = partial + 512;    // 4
  const LevelTables T = level_tables(p.tables, lv, p.table_stride);
  const int node = blockIdx.x, bh = blockIdx.y, d = threadIdx.x & 127, q = threadIdx.x >> 7;
  const int size = T.node_size[node];
  if (size <= kChunkRows) return;                              // done by the node kernel
  const int item0 = T.node_item0[node];
  const int n_items = (size + kChunkRows - 1) / kChunkRows;
  const float* part = p.partial + ((size_t)bh * p.max_items + item0) * kPartialFloats;
  // fixed-order reduction of the partial Gram matrices
  float s_d = 0.f;
#pragma unroll 8
  for (int it = 0; it < n_items; ++it) s_d += part[(size_t)it * kPartialFloats + 128 * 128 + d];
  if (q == 0) vec[d] = s_d;
  __syncthreads();
  const float inv_n = 1.f / (float)size;
#pragma unroll 1
  for (int e0 = q; e0 < 128; e0 += 32) {
    float g[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int it = 0; it < n_items; ++it) {
#pragma unroll
      for (int j = 0; j < 8; ++j) g[j] += part[(size_t)it * kPartialFloats + (size_t)(e0 + 4 * j) * 128 + d];   // G[e][d], coalesced
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) G[(e0 + 4 * j) * 128 + d] = g[j] - vec[e0 + 4 * j] * s_d * inv_n;
  }
  __syncthreads();
  // sum over the 128 elements, identical in all four thread groups: warp sums, then (r0 + r1) + (r2 + r3)
  auto sum_128 = [&](float x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    __syncthreads();
    if (q == 0 && (threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    return (red[0] + red[1]) + (red[2] + red[3]);
  };
  const bool live = d < p.D;
  float v = live ? v0[((size_t)bh * nodes + node) * p.D + d] : 0.f;
  float nrm = sqrtf(sum_128(v * v));
  v /= fmaxf(nrm, 1e-12f);
  for (int iter = 0; iter < p.pow_iters; ++iter) {
    __syncthreads();
    if (q == 0) vec[d] = v;
    __syncthreads();
    float a = 0.f;
#pragma unroll 8
    for (int e = q; e < 128; e += 4) a += G[e * 128 + d] * vec[e];     // G symmetric: G[e][d], conflict-free
    partial[q * 128 + d] = a;
    __syncthreads();
    v = (partial[d] + partial[128 + d]) + (partial[256 + d] + partial[384 + d]);
    nrm = sqrtf(sum_128(v * v));
    v /= fmaxf(nrm, 1e-12f);
  }
  if (q == 0) p.dir[((size_t)bh * p.dir_nodes + node) * 128 + d] = v;
}

// ------------------------------------------------------------------------------------------
// project: sort keys of the items of nodes that are more than one item
// ------------------------------------------------------------------------------------------
template <int D, bool kFp16>
__global__ void __launch_bounds__(128) pddp_project_kernel(PddpParams p, int lv, int pad, const int* perm_in, float* proj_out) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ float vec[128];
  const LevelTables T = level_tables(p.tables, lv, p.table_stride);
  const int item = blockIdx.x, bh = blockIdx.y, tid = threadIdx.x;
  const int node = T.item_node[item], row_begin = T.item_row0[item], size = T.node_size[node];
  if (size <= kChunkRows) return;                              // done by the node kernel
  const int rows = min(kChunkRows, size - row_begin);
  const int pos0 = T.node_start[node] + row_begin;
  vec[tid] = p.dir[((size_t)bh * p.dir_nodes + node) * 128 + tid];
  __syncthreads();
  unsigned long long* keys = p.keys + (size_t)bh * p.key_stride + (size_t)node * pad;
  project_rows<D, kFp16>(smem_u32(smem), tid >> 5, tid & 31, reinterpret_cast<const uint8_t*>(p.x) + 2 * (size_t)bh * p.x_stride_bh,
                         2 * (size_t)p.x_stride_row, perm_in + (size_t)bh * p.N + pos0, rows, row_begin, vec, keys,
                         proj_out != nullptr ? proj_out + (size_t)bh * p.N + pos0 : nullptr, false);
  if (row_begin + rows == size)
    for (int r = size + tid; r < pad; r += 128) keys[r] = kPadKey;             // slots beyond the node sort last
  cp_async_wait_all();
}


// ------------------------------------------------------------------------------------------
// Head dimensions other than 64 and 128 (multiples of 8 up to 256): the principal direction by power iterations
// that never form the Gram matrix.  With t_r = x_r . v,
//     (X^T X - s s^T / n) v  =  sum_r x_r t_r  -  s (sum_r t_r) / n,
// so one pass over the node's rows per iteration gives the next vector.  The rows are read pow_iters times per level
// instead of once, which is the price of staying clear of a 256 x 256 Gram matrix per node; this path serves the
// uncommon head dimensions, the tensor-core Gram path above the common ones.  Partial sums of a node's chunks are
// combined in chunk order by the next kernel: deterministic, no atomics.
// ------------------------------------------------------------------------------------------
constexpr int kWideD = 256;
constexpr int kWideFloats = 2 * kWideD + 8;      // per chunk: sum_r x_r t_r [256], sum_r x_r [256], sum_r t_r

__device__ __forceinline__ float block_sum_256(float x, float* red) {
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) t += red[w];
  return t;
}

// v = v0 / |v0| for every node of the level (zeros beyond D)
__global__ void __launch_bounds__(256) pddp_wide_init_kernel(PddpParams p, int nodes, const float* v0, float* wdir) {
  __shared__ float red[8];
  const int node = blockIdx.x, bh = blockIdx.y, d = threadIdx.x;
  float v = d < p.D ? v0[((size_t)bh * nodes + node) * p.D + d] : 0.f;
  const float nrm = sqrtf(block_sum_256(v * v, red));
  wdir[((size_t)bh * p.dir_nodes + node) * kWideD + d] = v / fmaxf(nrm, 1e-12f);
}

template <bool kFp16>
__device__ __forceinline__ void unpack8(const uint4& w, float (&x)[8]) {
  const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (kFp16) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u[i]));
      x[2 * i] = f.x; x[2 * i + 1] = f.y;
    } else {
      x[2 * i] = bf16_lo(u[i]); x[2 * i + 1] = bf16_hi(u[i]);
    }
  }
}

// One CTA per chunk of up to kChunkRows rows of one node: lane l of every warp owns elements 8l .. 8l+7 of a row.
template <bool kFp16>
__global__ void __launch_bounds__(256) pddp_wide_matvec_kernel(PddpParams p, int lv, const int* perm_in, const float* wdir,
                                                               float* wpart) {
  __shared__ float acc_w[8][kWideD];
  __shared__ float acc_s[8][kWideD];
  __shared__ float acc_t[8];
  const LevelTables T = level_tables(p.tables, lv, p.table_stride);
  const int item = blockIdx.x, bh = blockIdx.y;
  const int node = T.item_node[item], row0 = T.item_row0[item];
  const int rows = min(kChunkRows, T.node_size[node] - row0);
  const int start = T.node_start[node] + row0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool live = lane * 8 < p.D;
  float v[8], w[8], sx[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] = live ? wdir[((size_t)bh * p.dir_nodes + node) * kWideD + lane * 8 + j] : 0.f;
    w[j] = 0.f; sx[j] = 0.f;
  }
  float st = 0.f;
  const uint8_t* xb = reinterpret_cast<const uint8_t*>(p.x) + 2 * (size_t)bh * p.x_stride_bh + lane * 16;
  constexpr int kIn = 4;                                         // rows in flight per warp
#pragma unroll 1
  for (int r = warp * kIn; r < rows; r += 8 * kIn) {
    uint4 raw[kIn];
#pragma unroll
    for (int i = 0; i < kIn; ++i) {
      raw[i] = make_uint4(0u, 0u, 0u, 0u);
      if (r + i < rows && live) {
        const int id = perm_in[(size_t)bh * p.N + start + r + i];
        raw[i] = *reinterpret_cast<const uint4*>(xb + 2 * (size_t)id * p.x_stride_row);
      }
    }
#pragma unroll
    for (int i = 0; i < kIn; ++i) {
      float x[8];
      unpack8<kFp16>(raw[i], x);
      float t = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) t = fmaf(x[j], v[j], t);
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
#pragma unroll
      for (int j = 0; j < 8; ++j) { w[j] = fmaf(x[j], t, w[j]); sx[j] += x[j]; }
      st += t;                                                   // (rows beyond the chunk are zero rows: t = 0)
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) { acc_w[warp][lane * 8 + j] = w[j]; acc_s[warp][lane * 8 + j] = sx[j]; }
  if (lane == 0) acc_t[warp] = st;
  __syncthreads();
  float* out = wpart + ((size_t)bh * p.max_items + item) * kWideFloats;
  const int d = threadIdx.x;
  float a = 0.f, b = 0.f;
#pragma unroll
  for (int q = 0; q < 8; ++q) { a += acc_w[q][d]; b += acc_s[q][d]; }          // warps in fixed order
  out[d] = a;
  out[kWideD + d] = b;
  if (d == 0) {
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += acc_t[q];
    out[2 * kWideD] = t;
  }
}

// next vector of every node: chunks combined in order, centred, normalised
__global__ void __launch_bounds__(256) pddp_wide_step_kernel(PddpParams p, int lv, float* wdir, const float* wpart) {
  __shared__ float red[8];
  const LevelTables T = level_tables(p.tables, lv, p.table_stride);
  const int node = blockIdx.x, bh = blockIdx.y, d = threadIdx.x;
  const int size = T.node_size[node];
  const int item0 = T.node_item0[node];
  const int n_items = (size + kChunkRows - 1) / kChunkRows;
  const float* part = wpart + ((size_t)bh * p.max_items + item0) * kWideFloats;
  float wr = 0.f, s = 0.f, t = 0.f;
  for (int it = 0; it < n_items; ++it) {
    wr += part[(size_t)it * kWideFloats + d];
    s += part[(size_t)it * kWideFloats + kWideD + d];
    t += part[(size_t)it * kWideFloats + 2 * kWideD];
  }
  float v = wr - s * (t / (float)size);
  const float nrm = sqrtf(block_sum_256(v * v, red));
  wdir[((size_t)bh * p.dir_nodes + node) * kWideD + d] = v / fmaxf(nrm, 1e-12f);
}

// projection of every row on its node's direction, eight elements per lane (the counterpart of pddp_project_kernel)
template <bool kFp16>
__global__ void __launch_bounds__(256) pddp_wide_project_kernel(PddpParams p, int lv, int nodes, int pad, const int* perm_in,
                                                                const float* wdir, float* proj_out) {
  const LevelTables T = level_tables(p.tables, lv, p.table_stride);
  const int bh = blockIdx.y;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long total = (long long)nodes * pad;
  const long long slot0 = warp * kProjRows;
  if (slot0 >= total) return;
  const int node = (int)(slot0 / pad), r0 = (int)(slot0 % pad);
  unsigned long long* keys = p.keys + (size_t)bh * p.key_stride;
  const int nsize = T.node_size[node];
  const int pos0 = T.node_start[node] + r0;
  const bool live = lane * 8 < p.D;
  float v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = live ? wdir[((size_t)bh * p.dir_nodes + node) * kWideD + lane * 8 + j] : 0.f;
  int my_id = -1;
  if (lane < kProjRows && r0 + lane < nsize) my_id = perm_in[(size_t)bh * p.N + pos0 + lane];
  uint4 raw[kProjRows];
#pragma unroll
  for (int i = 0; i < kProjRows; ++i) {
    const int id = __shfl_sync(0xffffffffu, my_id, i);
    raw[i] = make_uint4(0u, 0u, 0u, 0u);
    if (id >= 0 && live)
      raw[i] = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(p.x) +
                                              2 * ((size_t)bh * p.x_stride_bh + (size_t)id * p.x_stride_row) + lane * 16);
  }
#pragma unroll
  for (int i = 0; i < kProjRows; ++i) {
    float x[8];
    unpack8<kFp16>(raw[i], x);
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc = fmaf(x[j], v[j], acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      const int r = r0 + i;
      if (r >= nsize) {
        keys[slot0 + i] = kPadKey;
      } else {
        keys[slot0 + i] = sort_key(float_key(acc), r);
        if (proj_out != nullptr) proj_out[(size_t)bh * p.N + pos0 + i] = acc;
      }
    }
  }
}

// ------------------------------------------------------------------------------------------
// sort: bitonic network over segments of `pad` keys (power of two), ascending inside each segment
// ------------------------------------------------------------------------------------------
// A CTA of kT threads sorts 8 kT consecutive slots (several short segments or a part of a long one).  A thread holds eight
// slots whose positions differ in three neighbouring bits, b .. b + 2, and does the three compare distances of these bits in
// registers; between groups of three the slots change hands through shared memory (padded by one slot in eight, so that
// every layout is read and written without bank conflicts).  A full tile changes hands 27 times for its 78 steps; with the
// distances of 8 to 128 as lane exchanges (sixteen 32-bit shuffles per step) and the larger ones through shared memory one by
// one it took 47 us instead of 37.  Stages k_lo .. k_hi; distances above the tile are done by the global kernel.
// The kernel of a segment's last stage writes the new order itself: new_perm[start + r] = old_perm[start + position].
// Segments of up to 1,024 slots take CTAs of 128 threads and those of 2,048 of 256, so that a level's slots spread over more
// CTAs than SMs.
constexpr int kSortThreads = kSortTile / 8;

template <int kT>
__global__ void __launch_bounds__(kT) pddp_sort_kernel(PddpParams p, int lv, long long slots, int pad, int k_lo, int k_hi,
                                                      const int* perm_in, int* perm_out) {
  constexpr int kTile = 8 * kT;
  constexpr int kTileBits = kT == 128 ? 10 : (kT == 256 ? 11 : 12);
  static_assert((1 << kTileBits) == kTile, "tile size");
  __shared__ unsigned long long sk[kTile + kTile / 8];
  unsigned long long* keys = p.keys + (size_t)blockIdx.y * p.key_stride;
  const int tid = threadIdx.x;
  const long long slot0 = (long long)blockIdx.x * kTile + tid * 8;         // slots is a multiple of 8 (pad >= 8)
  const bool live = slot0 < slots;
  unsigned long long a[8];
  if (live) {
    const ulonglong2* src = reinterpret_cast<const ulonglong2*>(keys + slot0);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const ulonglong2 v = src[i]; a[2 * i] = v.x; a[2 * i + 1] = v.y; }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = kPadKey;
  }
  auto cmpx = [&](int i, int j, bool asc) {
    const bool swap = (a[i] > a[j]) == asc;
    const unsigned long long x = swap ? a[j] : a[i], y = swap ? a[i] : a[j];
    a[i] = x;
    a[j] = y;
  };
  // compare distances of bits b + 2 (if n == 3), b + 1 (if n >= 2) and b, all in one direction
  auto steps = [&](int n, bool asc) {
    if (n == 3) { cmpx(0, 4, asc); cmpx(1, 5, asc); cmpx(2, 6, asc); cmpx(3, 7, asc); }
    if (n >= 2) { cmpx(0, 2, asc); cmpx(1, 3, asc); cmpx(4, 6, asc); cmpx(5, 7, asc); }
    cmpx(0, 1, asc); cmpx(2, 3, asc); cmpx(4, 5, asc); cmpx(6, 7, asc);
  };
  // position in the tile of this thread's slot 0 when its slots differ in bits b .. b + 2
  auto first = [&](int b) { return ((tid >> b) << (b + 3)) | (tid & ((1 << b) - 1)); };
  int cur = 0;                                                             // the layout's b
  auto relayout = [&](int b) {
    const int f = first(cur), t = first(b);
#pragma unroll
    for (int i = 0; i < 8; ++i) { const int x = f + (i << cur); sk[x + (x >> 3)] = a[i]; }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) { const int x = t + (i << b); a[i] = sk[x + (x >> 3)]; }
    __syncthreads();
    cur = b;
  };
  if (k_lo == 2) {
    cmpx(0, 1, true); cmpx(2, 3, false); cmpx(4, 5, true); cmpx(6, 7, false);
    cmpx(0, 2, true); cmpx(1, 3, true); cmpx(4, 6, false); cmpx(5, 7, false);
    cmpx(0, 1, true); cmpx(2, 3, true); cmpx(4, 5, false); cmpx(6, 7, false);
  }
  const int tile0 = (int)(((long long)blockIdx.x * kTile) & (pad - 1));    // the tile's position inside its segment (0 if it holds several)
#pragma unroll 1
  for (int k = max(k_lo, 8); k <= k_hi; k <<= 1) {
    int left = min(31 - __clz(k), kTileBits);                              // compare distances of bits left - 1 .. 0 are to be done
#pragma unroll 1
    while (left > 3) {
      const int b = left - 3;
      relayout(b);
      steps(3, (k == pad) || (((tile0 + first(b)) & (pad - 1) & k) == 0)); // (bit k of the position is the same for all eight slots)
      left = b;
    }
    if (cur != 0) relayout(0);
    steps(left, (k == pad) || (((tile0 + tid * 8) & (pad - 1) & k) == 0));
  }
  if (!live) return;
  const int gi = (int)(slot0 & (pad - 1));                                 // position of this thread's first key in its segment
  if (k_hi == pad) {
    const LevelTables T = level_tables(p.tables, lv, p.table_stride);
    const int node = (int)(slot0 / pad);
    const int size = T.node_size[node];
    const size_t start = (size_t)blockIdx.y * p.N + T.node_start[node];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (gi + i < size) perm_out[start + gi + i] = perm_in[start + key_position(a[i], size)];
  } else {
    ulonglong2* dst = reinterpret_cast<ulonglong2*>(keys + slot0);
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[i] = make_ulonglong2(a[2 * i], a[2 * i + 1]);
  }
}

// One compare-exchange step at distance j >= tile of stage k.
__global__ void __launch_bounds__(256) pddp_sort_global_kernel(unsigned long long* keys_all, size_t key_stride, long long half_total,
                                                               int pad, int k, int j) {
  unsigned long long* keys = keys_all + (size_t)blockIdx.y * key_stride;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= half_total) return;
  const long long i = ((t & ~(long long)(j - 1)) << 1) | (t & (j - 1));
  const int gi = (int)(i & (pad - 1));
  const bool asc = (k == pad) || ((gi & k) == 0);
  unsigned long long a = keys[i], b = keys[i + j];
  if ((a > b) == asc) { keys[i] = b; keys[i + j] = a; }
}

__global__ void pddp_iota_kernel(int* perm, long long total, int N) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < total) perm[i] = (int)(i % N);
}
__global__ void pddp_widen_kernel(const int* perm, long long* out, long long total) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < total) out[i] = perm[i];
}

}  // namespace

// ------------------------------------------------------------------------------------------
// Host side: tree shape, workspace layout, per-level launches
// ------------------------------------------------------------------------------------------
namespace {

struct Plan {
  int levels = 0;
  int K = 0;
  std::vector<LevelShape> shape;
  int max_items = 0;
  size_t key_stride = 0;          // u64 keys per (batch*head)
  int table_stride = 0;
  // byte offsets inside the workspace
  size_t off_tables = 0, off_perm_a = 0, off_perm_b = 0, off_partial = 0, off_dir = 0, off_keys = 0, total = 0;
};

Plan make_plan(int BH, int N, int C) {
  Plan pl;
  pl.K = (N + C - 1) / C;
  std::vector<int> lo(1, 0), hi(1, pl.K), lo2, hi2;
  while (any_splittable(lo.data(), hi.data(), (int)lo.size())) {
    LevelShape ls{(int)lo.size(), 0, 1};
    int max_size = 1;
    for (size_t i = 0; i < lo.size(); ++i) {
      const int size = std::min(hi[i] * C, N) - lo[i] * C;
      ls.items += (size + kChunkRows - 1) / kChunkRows;
      max_size = std::max(max_size, size);
    }
    ls.pad = std::max(next_pow2(max_size), 8);   // the projection kernel works on whole groups of kProjRows = 8 slots
    pl.shape.push_back(ls);
    pl.max_items = std::max(pl.max_items, ls.items);
    pl.key_stride = std::max(pl.key_stride, (size_t)ls.nodes * ls.pad);
    lo2.assign(2 * lo.size(), 0); hi2.assign(2 * lo.size(), 0);
    const int m = split_level(lo.data(), hi.data(), (int)lo.size(), lo2.data(), hi2.data());
    lo.assign(lo2.begin(), lo2.begin() + m); hi.assign(hi2.begin(), hi2.begin() + m);
  }
  pl.levels = (int)pl.shape.size();
  pl.table_stride = 3 * kMaxNodes + 2 * (pl.max_items + 8);
  auto align = [](size_t v) { return (v + 255) & ~size_t(255); };
  size_t o = 0;
  pl.off_tables = o; o = align(o + ((size_t)std::max(pl.levels, 1) * pl.table_stride + 4 * kMaxNodes) * sizeof(int));
  pl.off_perm_a = o; o = align(o + (size_t)BH * N * sizeof(int));
  pl.off_perm_b = o; o = align(o + (size_t)BH * N * sizeof(int));
  pl.off_partial = o; o = align(o + (size_t)BH * std::max(pl.max_items, 1) * kPartialFloats * sizeof(float));
  pl.off_dir = o; o = align(o + (size_t)BH * pl.K * 128 * sizeof(float));
  pl.off_keys = o; o = align(o + (size_t)BH * std::max(pl.key_stride, (size_t)1) * sizeof(unsigned long long));
  pl.total = o;
  return pl;
}

}  // namespace

size_t pddp_workspace_bytes(int BH, int N, int C) {
  if (BH < 1 || N < 1 || C < 1 || (N + C - 1) / C > kMaxNodes) return 0;
  return make_plan(BH, N, C).total;
}

long long pddp_start_vector_rows(int BH, int N, int C) {
  const Plan pl = make_plan(BH, N, C);
  long long rows = 0;
  for (const auto& ls : pl.shape) rows += (long long)BH * ls.nodes;
  return rows;
}

int launch_pddp(const PddpArgs& a, cudaStream_t stream) {
  const int BH = a.BH, N = a.N, C = a.C;
  const long long total = (long long)BH * N;
  uint8_t* ws = reinterpret_cast<uint8_t*>(a.workspace);
  const Plan pl = make_plan(BH, N, C);
  if (pl.total > a.workspace_bytes) return -7;
  int* perm_a = reinterpret_cast<int*>(ws + pl.off_perm_a);
  int* perm_b = reinterpret_cast<int*>(ws + pl.off_perm_b);
  const int tb = 256;
  pddp_iota_kernel<<<(unsigned)((total + tb - 1) / tb), tb, 0, stream>>>(perm_a, total, N);
  if (pl.levels > 0) {
    PddpParams p{};
    p.x = a.x; p.x_stride_bh = a.x_stride_bh; p.x_stride_row = a.x_stride_row;
    p.N = N; p.D = a.D; p.BH = BH; p.pow_iters = a.pow_iters;
    p.tables = reinterpret_cast<int*>(ws + pl.off_tables); p.table_stride = pl.table_stride;
    p.max_items = std::max(pl.max_items, 1);
    p.partial = reinterpret_cast<float*>(ws + pl.off_partial);
    p.dir = reinterpret_cast<float*>(ws + pl.off_dir); p.dir_nodes = pl.K;
    p.keys = reinterpret_cast<unsigned long long*>(ws + pl.off_keys); p.key_stride = pl.key_stride;
    p.status = a.status;
    pddp_tables_kernel<<<1, kTableThreads, 0, stream>>>(N, C, p.tables, pl.levels, pl.table_stride);
    auto node = a.D == 64 ? (a.fp16 ? pddp_node_kernel<64, true> : pddp_node_kernel<64, false>)
                          : (a.fp16 ? pddp_node_kernel<128, true> : pddp_node_kernel<128, false>);
    auto project = a.D == 64 ? (a.fp16 ? pddp_project_kernel<64, true> : pddp_project_kernel<64, false>)
                             : (a.fp16 ? pddp_project_kernel<128, true> : pddp_project_kernel<128, false>);
    const int project_smem = kBufs * kTileBytes + 1024;
    const int power_smem = (128 * 128 + 128 + 512 + 8) * sizeof(float);
    if (cudaFuncSetAttribute(node, cudaFuncAttributeMaxDynamicSharedMemorySize, NodeSmem::kDynamic) != cudaSuccess ||
        cudaFuncSetAttribute(project, cudaFuncAttributeMaxDynamicSharedMemorySize, project_smem) != cudaSuccess ||
        cudaFuncSetAttribute(pddp_power_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, power_smem) != cudaSuccess)
      return -8;
    const float* v0 = a.start_vectors;
    const bool wide = a.D != 64 && a.D != 128;
    // wide path: per-chunk partial sums first, then the directions (256 floats per node), both inside the partial area
    float* wpart = p.partial;
    float* wdir = p.partial + (size_t)BH * p.max_items * kWideFloats;
    if (wide && ((size_t)BH * p.max_items * kWideFloats + (size_t)BH * pl.K * kWideD) >
                    (size_t)BH * p.max_items * kPartialFloats)
      return -7;
    for (int lv = 0; lv < pl.levels; ++lv) {
      const LevelShape& ls = pl.shape[lv];
      if (a.perm_levels != nullptr)
        cudaMemcpyAsync(a.perm_levels + (size_t)lv * total, perm_a, total * sizeof(int), cudaMemcpyDeviceToDevice, stream);
      const long long slots = (long long)ls.nodes * ls.pad;
      float* proj = a.proj_levels != nullptr ? a.proj_levels + (size_t)lv * total : nullptr;
      const unsigned pgrid = (unsigned)((slots / kProjRows * 32 + 255) / 256);
      if (wide) {
        // Gram-free power iterations (head dimensions other than 64 / 128); partial sums and directions live in the
        // area the Gram partials would use
        pddp_wide_init_kernel<<<dim3(ls.nodes, BH), 256, 0, stream>>>(p, ls.nodes, v0, wdir);
        for (int it = 0; it < a.pow_iters; ++it) {
          if (a.fp16) pddp_wide_matvec_kernel<true><<<dim3(ls.items, BH), 256, 0, stream>>>(p, lv, perm_a, wdir, wpart);
          else pddp_wide_matvec_kernel<false><<<dim3(ls.items, BH), 256, 0, stream>>>(p, lv, perm_a, wdir, wpart);
          pddp_wide_step_kernel<<<dim3(ls.nodes, BH), 256, 0, stream>>>(p, lv, wdir, wpart);
        }
        if (a.fp16) pddp_wide_project_kernel<true><<<dim3(pgrid, BH), 256, 0, stream>>>(p, lv, ls.nodes, ls.pad, perm_a, wdir, proj);
        else pddp_wide_project_kernel<false><<<dim3(pgrid, BH), 256, 0, stream>>>(p, lv, ls.nodes, ls.pad, perm_a, wdir, proj);
      } else {
        node<<<dim3(ls.items, BH), kNodeThreads, NodeSmem::kDynamic, stream>>>(p, lv, ls.nodes, ls.pad, perm_a, v0, proj);
        if (ls.items > ls.nodes) {               // some nodes are more than one item
          pddp_power_kernel<<<dim3(ls.nodes, BH), 512, power_smem, stream>>>(p, lv, ls.nodes, v0);
          project<<<dim3(ls.items, BH), 128, project_smem, stream>>>(p, lv, ls.pad, perm_a, proj);
        }
      }
      v0 += (size_t)BH * ls.nodes * a.D;
      // bitonic sort of every segment of `pad` keys; the last kernel writes the new order
      const int tile_k = std::min(ls.pad, kSortTile);
      auto sort = [&](auto kern, int threads, int k_lo, int k_hi) {
        kern<<<dim3((unsigned)((slots + 8 * threads - 1) / (8 * threads)), BH), threads, 0, stream>>>(p, lv, slots, ls.pad, k_lo, k_hi, perm_a, perm_b);
      };
      if (ls.pad <= 1024) sort(pddp_sort_kernel<128>, 128, 2, tile_k);
      else if (ls.pad <= 2048) sort(pddp_sort_kernel<256>, 256, 2, tile_k);
      else sort(pddp_sort_kernel<kSortThreads>, kSortThreads, 2, tile_k);
      for (int k = tile_k * 2; k <= ls.pad; k <<= 1) {
        for (int j = k >> 1; j >= kSortTile; j >>= 1)
          pddp_sort_global_kernel<<<dim3((unsigned)((slots / 2 + 255) / 256), BH), 256, 0, stream>>>(p.keys, p.key_stride, slots / 2, ls.pad, k, j);
        sort(pddp_sort_kernel<kSortThreads>, kSortThreads, k, k);
      }
      std::swap(perm_a, perm_b);
    }
  }
  if (a.perm_levels != nullptr)
    cudaMemcpyAsync(a.perm_levels + (size_t)pl.levels * total, perm_a, total * sizeof(int), cudaMemcpyDeviceToDevice, stream);
  pddp_widen_kernel<<<(unsigned)((total + tb - 1) / tb), tb, 0, stream>>>(perm_a, a.perm_out, total);
  return cudaGetLastError() == cudaSuccess ? 0 : -8;
}

int pddp_levels(int N, int C) { return make_plan(1, N, C).levels; }

// ------------------------------------------------------------------------------------------
// Built-in scratch for callers that cannot allocate device memory.
//
// Some hosts of this library have no way to hand over a workspace: an inference server that has
// given every free byte of the GPU to its own memory pool and forbids further allocations, or
// code on a latency-critical path where cudaMalloc is banned because it synchronises the whole
// device.  For them the library carries one fixed scratch array in its own device image.  It is
// part of the module, so each GPU that loads the library pays for it from load to exit: hence
// the small, fixed size.  In host code the array's name is only a handle, never an address a
// kernel could use; the usable device address comes from cudaGetSymbolAddress, asked once per
// device while that device is current.
// ------------------------------------------------------------------------------------------
constexpr size_t kStaticScratchBytes = 32u << 20;   // 32 MiB
static __device__ __align__(256) unsigned char g_pddp_static_scratch[kStaticScratchBytes];

size_t pddp_static_scratch_bytes() { return kStaticScratchBytes; }

// Device address of the built-in scratch on the CURRENT device (looked up on the first call per
// device, then cached).  Returns nullptr if the lookup fails.
void* pddp_static_scratch_address() {
  static void* cached[64] = {nullptr};
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (cached[dev] == nullptr) {
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_pddp_static_scratch) != cudaSuccess) return nullptr;
    cached[dev] = ptr;
  }
  return cached[dev];
}

}  // namespace mcs
