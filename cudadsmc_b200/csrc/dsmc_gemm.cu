// The warm-start surrogate's BF16 GEMM (sm_100a): C = A B with FP32
// accumulation, a bias / GELU epilogue, a split reduction, and the masked
// mean-square error of the field decoder fused behind its product.
//
// One persistent CTA per SM (or per tile where there are fewer):
//   warp 0     TMA: operand tiles of 64 k into a ring of kStages stages
//   warp 1     tcgen05.mma into one of two TMEM accumulators
//   warps 2-  epilogue of the other accumulator: tcgen05.ld, bias / GELU /
//              error, then 32 x 32 blocks through swizzled shared memory out
//              by TMA stores (or reductions)
// so that loads, products and stores of consecutive tiles overlap.
//
// What bounds it: the decoder (k = 256 against a field of 327,680 columns)
// moves 4 output bytes per 512 FLOP, so memory does; the hidden layers
// (512 x 512) are latency, one tile per CTA.  A form whose threads copied the
// operands between barriers, and whose epilogue lanes stored to 32 rows at
// once, took (us, before -> now; one B200, cold caches): 1 x 327680 x 256
// 270 -> 46, 100 rows 270 -> 50 (0.9 of the copy bandwidth), the decoder and
// error of 1024 rows 3105 + 1414 + 232 in three kernels -> 610 in one, its
// basis gradient (256 x 327680 x 1024) 1389 -> 220 and coefficient gradient
// (1024 x 256 x 327680, split 64) 958 -> 209, a 100 x 512 x 512 layer 45 -> 10.
// The two gradients run at 9 TB/s of operand traffic out of L2.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "dsmc_b200.h"
#include "dsmc_kernels.cuh"
#include "dsmc_umma.cuh"

// Set by a GEMM whose wait on its tensor-core work or copies ran out (a
// second); dsmc_gemm_check reports and clears it.
__device__ unsigned int g_gemm_failed = 0;

namespace {

using bf16 = __nv_bfloat16;
using namespace dsmcb;

struct GemmArgs {
  int m, n, k;
  int a_mn, b_mn;        // operand majors: 0 K, 1 M / N contiguous
  int tiles_m, tiles_n;  // output tiles
  int splits, kchunk;    // K range per split (a multiple of the K step)
  float* c;
  int ldc;
  float beta;
  const float* bias;
  int act;  // 0 none, 1 GELU
  bf16* cb;
  int ldcb;
  int tma_t;          // the targets come by TMA
  int tma_c, tma_cb;  // the output goes out by TMA (its rows 16-byte aligned)
  int b_early;        // B is not written by the kernel before this one: its first tiles may be
                      // fetched while that one finishes
  int beside;         // may run beside the kernel before this one (beside_entry)
  int part_rows;      // > 0: split z writes its own m x n product, part_rows rows further down per split
  // the fused error (MSE kernels): targets, scale, column sums, loss, count
  const bf16* t;
  int ldt;
  float scale;
  float* colsum;
  double* loss;
  unsigned long long* count;
};

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678f)); }

// Epilogue warps: four (one per quarter of the accumulator's lanes); one per
// 32 x 32 block of the tile where the tile is narrow (a layer's GELU, one tile
// per CTA, is then half as long), and for the error: sixteen, four per quarter taking every fourth block of 32 columns.
// Its 900 instructions per block are chains of short waits (accumulator,
// targets, FP64 sum, column sum), so its time falls with the warps that share
// a scheduler: 1024 x 327680 x 256 took 1026 us with four, 890 with eight, 610 with
// sixteen.
// To make room, their staging is single buffered and the gradient block takes
// the field block's place once that has left.
template <int BN, bool MSE>
struct Shape {
  static constexpr int kStages = BN == 256 || MSE ? 3 : BN == 128 ? 4 : 6;
  static constexpr int kEpiWarps = MSE || BN == 64 ? BN / 8 : 4;  // BN / 8: one per block of the tile
  static constexpr int kThreads = 64 + 32 * kEpiWarps;
  static constexpr bool kOneBlock = kEpiWarps == BN / 8;
  static constexpr int kStaging = kOneBlock ? 1 : 2;
  static constexpr int kABytes = umma::kBM * umma::kBK * 2;
  static constexpr int kBBytes = BN * umma::kBK * 2;
  static constexpr uint32_t kTmemCols = 2 * BN;
};

// The error's shared memory: per epilogue warp the targets of its next block
// (64-byte swizzle), and the running sum of every column, handed from warp to
// warp in row order.
template <int BN, bool MSE>
struct MseSmem {};
template <int BN>
struct __align__(128) MseSmem<BN, true> {
  unsigned char t[BN / 8][2048];
  float colsum[BN];
  unsigned long long tbar[BN / 8];
  unsigned long long chain[4][BN / 32];
};

// (a multiple of 1024 bytes up to the targets: every tile and block sits on its
// swizzle's period from a base on 1024)
template <int BN, bool MSE>
struct __align__(128) Smem {
  using Sh = Shape<BN, MSE>;
  unsigned char a[Sh::kStages][Sh::kABytes];
  unsigned char b[Sh::kStages][Sh::kBBytes];
  // 32 x 32 blocks on their way out, per epilogue warp: FP32
  // rows of 128 bytes (128-byte swizzle), BF16 rows of 64 (64-byte swizzle)
  unsigned char f[Sh::kEpiWarps][Sh::kStaging][4096];
  unsigned char h[Sh::kEpiWarps][Sh::kStaging][2048];
  MseSmem<BN, MSE> mse;
  alignas(16) float bias[Sh::kEpiWarps][Sh::kOneBlock ? 32 : BN];
  unsigned long long full[Sh::kStages], empty[Sh::kStages];
  unsigned long long tfull[2], tempty[2], drain;
  uint32_t tmem_base;
  uint32_t failed;
};

// Offset of 16-byte chunk c of row r in a 32-row block, rows of 128 or 64 bytes.
__device__ __forceinline__ int chunk128(int r, int c) { return 128 * r + 16 * (c ^ (r & 7)); }
__device__ __forceinline__ int chunk64(int r, int c) { return 64 * r + 16 * (c ^ ((r >> 1) & 3)); }

// A staged block out by plain stores, a row's 32 columns at a time: where the
// rows are not 16-byte aligned, and where C is read back (beta) or added to
// (splits).  Each lane storing its own row touched 32 rows at once (1 x 327680
// x 256 with beta 288 us, split four ways 426; now 82 and 191).  The rows' loads
// of C are in flight together; beta's sums go back to the block.
__device__ __forceinline__ void rows_out(const GemmArgs& g, unsigned char* blk, int row0, int c0) {
  const int lane = threadIdx.x & 31, rows = min(32, g.m - row0);
  if (c0 + lane >= g.n) return;
  float* cp = g.c + (size_t)row0 * g.ldc + c0 + lane;
  const bool back = g.beta != 0.f && g.splits == 1;
  float old[32];
#pragma unroll
  for (int r = 0; r < 32; r++) old[r] = back && r < rows ? cp[(size_t)r * g.ldc] : 0.f;
#pragma unroll
  for (int r = 0; r < 32; r++) {
    if (r >= rows) break;
    float* at = reinterpret_cast<float*>(blk + chunk128(r, lane >> 2) + 4 * (lane & 3));
    float x = *at;
    if (g.splits > 1) {
      atomicAdd(cp + (size_t)r * g.ldc, x);
    } else {
      if (back) {
        x += g.beta * old[r];
        *at = x;
      }
      cp[(size_t)r * g.ldc] = x;
    }
  }
}
__device__ __forceinline__ void rows_out_bf16(const GemmArgs& g, const unsigned char* blk, int row0, int c0) {
  const int lane = threadIdx.x & 31, rows = min(32, g.m - row0);
  if (c0 + lane >= g.n) return;
  bf16* cp = g.cb + (size_t)row0 * g.ldcb + c0 + lane;
#pragma unroll 8
  for (int r = 0; r < rows; r++)
    cp[(size_t)r * g.ldcb] = *reinterpret_cast<const bf16*>(blk + chunk64(r, lane >> 3) + 2 * (lane & 7));
}

// The tiles of CTA `b` of `g`.  Plain: all (m, n, split) items round robin, m
// fastest, so that the tiles that share a column block of B run side by side
// and B comes from memory once.  COLS: whole columns of tiles, m innermost,
// so that one CTA sums a column over all rows.
struct TileWalk {
  int tiles_m, tiles_n, splits, step, item, m;
  bool cols;
  __device__ __forceinline__ TileWalk(const GemmArgs& g, bool c)
      : tiles_m(g.tiles_m), tiles_n(g.tiles_n), splits(g.splits), step(gridDim.x), item(blockIdx.x), m(0), cols(c) {}
  __device__ __forceinline__ bool get(int& mt, int& nt, int& z) const {
    if (cols) {
      mt = m;
      nt = item;
      z = 0;
      return item < tiles_n;
    }
    mt = item % tiles_m;
    const int r = item / tiles_m;
    nt = r % tiles_n;
    z = r / tiles_n;
    return z < splits;
  }
  __device__ __forceinline__ void next() {
    if (cols && ++m < tiles_m) return;
    m = 0;
    item += step;
  }
};

__device__ __forceinline__ int k_tiles(const GemmArgs& g, int z) {
  return (min(g.k, (z + 1) * g.kchunk) - z * g.kchunk + umma::kBK - 1) / umma::kBK;
}

// Column sums of the error's gradient, every column added row by row from
// row 0 on in FP32, as dsmc_colsum adds it: the warp of rows [32 quad,
// 32 quad + nr) of tile `tile` takes the running sums of column block q from
// the warp of the rows before it (the first from the last warp of the tile
// before, whose sums it drops when a new column block starts) and hands them
// on.  The hand-over goes round the four warps in a ring, so no warp can be
// a whole phase ahead of the next.  False if the wait ran out.
template <int BN>
__device__ __forceinline__ bool column_chain(MseSmem<BN, true>& sm, const GemmArgs& g, const unsigned char* gr,
                                             int quad, int q, int tile, int mt, int c0, int nr) {
  const int lane = threadIdx.x & 31;
  bool ok = true;
  if (quad > 0) ok = dev::mbar_wait_bounded(&sm.chain[quad][q], tile & 1);
  else if (tile > 0) ok = dev::mbar_wait_bounded(&sm.chain[0][q], (tile - 1) & 1);
  float s = (quad == 0 && mt == 0) ? 0.f : sm.colsum[32 * q + lane];
  const unsigned char* rows = gr + 4 * (lane & 3);
  if (nr == 32) {
#pragma unroll
    for (int r = 0; r < 32; r++) s += *reinterpret_cast<const float*>(rows + chunk128(r, lane >> 2));
  } else {
    for (int r = 0; r < nr; r++) s += *reinterpret_cast<const float*>(rows + chunk128(r, lane >> 2));
  }
  sm.colsum[32 * q + lane] = s;
  if (quad == 3 && mt == g.tiles_m - 1 && c0 + lane < g.n) g.colsum[c0 + lane] = s;
  __syncwarp();
  if (lane == 0) umma::mbar_arrive(&sm.chain[(quad + 1) & 3][q]);
  return __all_sync(0xffffffffu, ok);
}

// The blocks of one epilogue warp that hold elements, in the order it works
// through them: the next one's targets are fetched while it works on one.
template <int BN>
struct TargetWalk {
  TileWalk w;
  int issued = 0, used = 0;
  __device__ __forceinline__ TargetWalk(const GemmArgs& g) : w(g, true) {}
  // one lane: the next block's copy
  __device__ __forceinline__ void issue(const GemmArgs& g, const CUtensorMap* map, MseSmem<BN, true>& sm, int ew,
                                        int quad, int q) {
    int mt, nt, z;
    while (w.get(mt, nt, z)) {
      const int row0 = mt * umma::kBM + 32 * quad, c0 = nt * BN + 32 * q;
      w.next();
      if (row0 >= g.m || c0 >= g.n) continue;
      dev::mbar_expect_tx(&sm.tbar[ew], 2048);
      umma::tma_load(sm.t[ew], map, c0, row0, &sm.tbar[ew]);
      issued++;
      break;
    }
  }
};

// PLAIN: some output does not go out by TMA (a form of its own: with that code
// in it the kernel takes 14 to 40 registers more, and a prediction of one
// condition 80 us instead of 73).
template <int BN, bool MSE, bool PLAIN>
__global__ void __launch_bounds__(Shape<BN, MSE>::kThreads, 1)
    k_gemm(const __grid_constant__ GemmArgs g, const __grid_constant__ CUtensorMap map_a,
           const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_c,
           const __grid_constant__ CUtensorMap map_cb, const __grid_constant__ CUtensorMap map_t) {
  using namespace umma;
  using namespace dev;
  using Sh = Shape<BN, MSE>;
  constexpr int S = Sh::kStages, E = Sh::kEpiWarps;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  Smem<BN, MSE>& sm = *reinterpret_cast<Smem<BN, MSE>*>(smem_raw);
  if (smem_u32(smem_raw) & 1023u) {  // the swizzles would not line up
    if (threadIdx.x == 0) atomicOr(&g_gemm_failed, 1u);
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(&sm.tfull[s], 1);
      mbar_init(&sm.tempty[s], E);
    }
    mbar_init(&sm.drain, 1);
    if constexpr (MSE) {
      for (int w = 0; w < 4; w++)
        for (int q = 0; q < BN / 32; q++) mbar_init(&sm.mse.chain[w][q], 1);
      for (int w = 0; w < E; w++) mbar_init(&sm.mse.tbar[w], 1);
    }
    sm.failed = 0;
    fence_mbar_init();
    tma_prefetch(&map_a);
    tma_prefetch(&map_b);
    if (g.tma_c) tma_prefetch(&map_c);
    if (g.tma_cb) tma_prefetch(&map_cb);
  }
  if (warp == 1) tmem_alloc(&sm.tmem_base, Sh::kTmemCols);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = sm.tmem_base;
  volatile uint32_t* failed = &sm.failed;
  auto load_b = [&](int s, int nt, int kx) {
    if (g.b_mn) {
#pragma unroll
      for (int q = 0; q < BN / 64; q++)
        tma_load(sm.b[s] + 8192 * q, &map_b, nt * BN + 64 * q, kx, &sm.full[s]);
    } else {
      tma_load(sm.b[s], &map_b, kx, nt * BN, &sm.full[s]);
    }
  };
  int early = 0;  // stages whose B is on its way already
  if (g.b_early && warp == 0 && lane == 0) {
    int mt, nt, z;
    if (TileWalk(g, MSE).get(mt, nt, z)) {
      early = min(S, k_tiles(g, z));
      for (int j = 0; j < early; j++) {
        mbar_expect_tx(&sm.full[j], Sh::kABytes + Sh::kBBytes);
        load_b(j, nt, z * g.kchunk + j * kBK);
      }
    }
  }
  // everything above ran beside the kernel before this one
  beside_entry(g.beside);

  if (warp == 0 && lane == 0) {
    int it = 0;  // tiles of k handed out so far
    bool ok = true;
    for (TileWalk w(g, MSE); ok; w.next()) {
      int mt, nt, z;
      if (!w.get(mt, nt, z)) break;
      const int kt = k_tiles(g, z), k0 = z * g.kchunk;
      for (int j = 0; j < kt; j++, it++) {
        const int s = it % S;
        if (it >= S && !mbar_wait_bounded(&sm.empty[s], ((it / S) - 1) & 1)) ok = false;
        if (!ok || *failed) {
          ok = false;
          break;
        }
        const int kx = k0 + j * kBK;
        if (it >= early) {
          mbar_expect_tx(&sm.full[s], Sh::kABytes + Sh::kBBytes);
          load_b(s, nt, kx);
        }
        if (g.a_mn) {
          tma_load(sm.a[s], &map_a, mt * kBM, kx, &sm.full[s]);
          tma_load(sm.a[s] + 8192, &map_a, mt * kBM + 64, kx, &sm.full[s]);
        } else {
          tma_load(sm.a[s], &map_a, kx, mt * kBM, &sm.full[s]);
        }
      }
    }
    // the copies in flight land before the shared memory goes away
    for (int i = max(0, it - S); i < it; i++)
      if (!mbar_wait_bounded(&sm.full[i % S], (i / S) & 1)) ok = false;
    if (!ok) *failed = 1;
  } else if (warp == 1 && lane == 0) {
    const uint32_t idesc = instr_desc(g.a_mn, g.b_mn, BN);
    const uint32_t a_lbo = g.a_mn ? 8192u : 16u, b_lbo = g.b_mn ? 8192u : 16u;
    const uint32_t a_step = g.a_mn ? 2048u : 32u, b_step = g.b_mn ? 2048u : 32u;
    int it = 0, tile = 0;
    bool ok = true;
    for (TileWalk w(g, MSE); ok; w.next(), tile++) {
      int mt, nt, z;
      if (!w.get(mt, nt, z)) break;
      const int acc = tile & 1;
      if (tile >= 2 && !mbar_wait_bounded(&sm.tempty[acc], ((tile >> 1) - 1) & 1)) ok = false;
      if (!ok || *failed) {
        ok = false;
        break;
      }
      fence_after_sync();
      const uint32_t d = tmem + (uint32_t)(acc * BN);
      const int kt = k_tiles(g, z);
      for (int j = 0; j < kt; j++, it++) {
        const int s = it % S;
        if (!mbar_wait_bounded(&sm.full[s], (it / S) & 1) || *failed) {
          ok = false;
          break;
        }
        fence_after_sync();
        const uint32_t a0 = smem_u32(sm.a[s]), b0 = smem_u32(sm.b[s]);
#pragma unroll
        for (int q = 0; q < kBK / 16; q++)
          mma(d, smem_desc(a0 + a_step * q, a_lbo), smem_desc(b0 + b_step * q, b_lbo), idesc,
              (j > 0 || q > 0) ? 1u : 0u);
        commit(&sm.empty[s]);
      }
      if (ok) commit(&sm.tfull[acc]);
    }
    // the products in flight finish before the tensor memory goes away
    commit(&sm.drain);
    if (!mbar_wait_bounded(&sm.drain, 0)) ok = false;
    if (!ok) *failed = 1;
  } else if (warp >= 2) {
    const int ew = warp - 2;
    const int quad = warp & 3;  // the TMEM lanes this warp may read
    unsigned char* fst = sm.f[ew][0];
    unsigned char* hst = sm.h[ew][0];
    float* sbias = sm.bias[ew];
    int tile = 0, buf = 0;
    bool ok = true;
    double loss = 0.0;
    unsigned long long count = 0;
    [[maybe_unused]] TargetWalk<BN> targets(g);
    if constexpr (MSE) {
      if (g.tma_t && lane == 0) targets.issue(g, &map_t, sm.mse, ew, quad, ew >> 2);
    }
    // the bias of a tile's columns, asked for one tile ahead
    constexpr int kBlocks = Sh::kOneBlock ? 1 : BN / 32;  // per warp and tile
    float bv[kBlocks];
    auto load_bias = [&](const TileWalk& w) {
      int mt, nt, z;
      const bool there = w.get(mt, nt, z);
#pragma unroll
      for (int q = 0; q < kBlocks; q++) {
        const int c = nt * BN + 32 * (Sh::kOneBlock ? ew >> 2 : q) + lane;
        bv[q] = there && c < g.n ? __ldg(g.bias + c) : 0.f;
      }
    };
    TileWalk w(g, MSE);
    if (g.bias) load_bias(w);
    for (; ok; tile++) {
      int mt, nt, z;
      if (!w.get(mt, nt, z)) break;
      w.next();
      if (g.bias) {
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kBlocks; q++) sbias[32 * q + lane] = bv[q];
        __syncwarp();
        load_bias(w);
      }
      const int acc = tile & 1;
      ok = mbar_wait_bounded(&sm.tfull[acc], (tile >> 1) & 1) && !*failed;
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      fence_after_sync();
      const int row0 = mt * kBM + 32 * quad, row = row0 + lane;
      const uint32_t t0 = tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)(acc * BN);
#pragma unroll 1
      for (int q = Sh::kOneBlock ? ew >> 2 : 0; q < BN / 32; q += Sh::kOneBlock ? BN / 32 : 1) {
        const int c0 = nt * BN + 32 * q;
        const bool any = row0 < g.m && c0 < g.n;  // the warp's block has elements
        float v[32];
        ld32(t0 + (uint32_t)(32 * q), v);
        if (Sh::kOneBlock || q == BN / 32 - 1) {  // the accumulator is read: the next tile but one may overwrite it
          fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.tempty[acc]);
        }
        if (!any) {
          // no rows here: the column sums pass through
          if constexpr (MSE)
            if (c0 < g.n) ok = column_chain(sm.mse, g, fst, quad, q, tile, mt, c0, 0) && ok;
          continue;
        }
        if (g.bias) {
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const float4 b = *reinterpret_cast<const float4*>(sbias + (Sh::kOneBlock ? 0 : 32 * q) + 4 * i);
            v[4 * i] += b.x; v[4 * i + 1] += b.y; v[4 * i + 2] += b.z; v[4 * i + 3] += b.w;
          }
        }
        // this warp's staging buffers are free again
        if (lane == 0) bulk_wait_read<Sh::kStaging - 1>();
        __syncwarp();
        if (MSE && !g.tma_c) {  // (a field off 16 bytes; as rows_out the kernel spills twice as much)
#pragma unroll
          for (int i = 0; i < 32; i++)
            if (row < g.m && c0 + i < g.n) g.c[(size_t)row * g.ldc + c0 + i] = v[i];
        } else if (g.c) {
#pragma unroll
          for (int i = 0; i < 8; i++)
            *reinterpret_cast<float4*>(fst + 4096 * buf + chunk128(lane, i)) =
                make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          if (PLAIN && !g.tma_c) {
            __syncwarp();
            rows_out(g, fst + 4096 * buf, row0, c0);
            __syncwarp();
            if (g.beta != 0.f) {  // the sum, for the BF16 copy
#pragma unroll
              for (int i = 0; i < 8; i++) {
                const float4 x = *reinterpret_cast<const float4*>(fst + 4096 * buf + chunk128(lane, i));
                v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
              }
            }
          }
        }
        if constexpr (MSE) {
          // the field goes out now, the gradient follows in its place
          if (g.tma_c) {
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
              tma_store(&map_c, fst, c0, row0);
              bulk_commit();
            }
          }
          // the block's targets, two per word; rows and columns past the end
          // count as targets that are not there
          uint32_t tw[16];
          if (g.tma_t) {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&sm.mse.tbar[ew], targets.used & 1)) && ok;
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const uint4 x = *reinterpret_cast<const uint4*>(sm.mse.t[ew] + chunk64(lane, i));
              tw[4 * i] = x.x; tw[4 * i + 1] = x.y; tw[4 * i + 2] = x.z; tw[4 * i + 3] = x.w;
            }
            targets.used++;
            __syncwarp();
            if (lane == 0 && ok) targets.issue(g, &map_t, sm.mse, ew, quad, q);
            if (row >= g.m || c0 + 32 > g.n) {
#pragma unroll
              for (int i = 0; i < 16; i++)
                if (row >= g.m || c0 + 2 * i >= g.n) tw[i] = 0x7fc07fc0u;  // n is even
            }
          } else {
            const unsigned short* tp = reinterpret_cast<const unsigned short*>(g.t) + (size_t)row * g.ldt + c0;
#pragma unroll
            for (int i = 0; i < 16; i++)
              tw[i] = row < g.m && c0 + 2 * i < g.n
                          ? (uint32_t)tp[2 * i] | ((uint32_t)tp[2 * i + 1] << 16) : 0x7fc07fc0u;
          }
          // v: the error's gradient from here on
          double ls[4] = {0.0, 0.0, 0.0, 0.0};
          uint32_t ct = 0;
#pragma unroll
          for (int i = 0; i < 32; i++) {
            const float tf = __uint_as_float((i & 1) ? (tw[i >> 1] & 0xffff0000u) : (tw[i >> 1] << 16));
            const bool there = tf == tf;
            const float e = there ? v[i] - tf : 0.f;
            const double d = (double)e;
            ls[i & 3] += d * d;
            ct += there;
            v[i] = there ? g.scale * 2.f * e : 0.f;
          }
          loss += (ls[0] + ls[1]) + (ls[2] + ls[3]);
          count += ct;
        } else if (g.act == 1) {
#pragma unroll
          for (int i = 0; i < 32; i++) v[i] = gelu(v[i]);
        }
        if (g.cb) {
          uint32_t p[16];
#pragma unroll
          for (int i = 0; i < 16; i++) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            p[i] = *reinterpret_cast<const uint32_t*>(&b);
          }
          if (MSE && !g.tma_cb) {
#pragma unroll
            for (int i = 0; i < 32; i++)
              if (row < g.m && c0 + i < g.n) g.cb[(size_t)row * g.ldcb + c0 + i] = __float2bfloat16(v[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
              *reinterpret_cast<uint4*>(hst + 2048 * buf + chunk64(lane, i)) =
                  make_uint4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]);
          }
          if (PLAIN && !g.tma_cb) {
            __syncwarp();
            rows_out_bf16(g, hst + 2048 * buf, row0, c0);
            __syncwarp();
          }
        }
        if constexpr (MSE) {
          if (g.tma_cb) {
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
              tma_store(&map_cb, hst, c0, row0);
              bulk_commit();
              bulk_wait_read<1>();
            }
          } else if (lane == 0) {
            bulk_wait_read<0>();
          }
          __syncwarp();  // the field block has left
#pragma unroll
          for (int i = 0; i < 8; i++)
            *reinterpret_cast<float4*>(fst + chunk128(lane, i)) =
                make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          __syncwarp();
          ok = column_chain(sm.mse, g, fst, quad, q, tile, mt, c0, min(32, g.m - row0)) && ok;
        } else if (g.tma_c || g.tma_cb) {
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            if (g.tma_c) {
              if (g.part_rows) tma_store(&map_c, fst + 4096 * buf, c0, z * g.part_rows + row0);
              else if (g.splits > 1) tma_reduce_add(&map_c, fst + 4096 * buf, c0, row0);
              else tma_store(&map_c, fst + 4096 * buf, c0, row0);
            }
            if (g.tma_cb) tma_store(&map_cb, hst + 2048 * buf, c0, row0);
            bulk_commit();
          }
          buf = (buf + 1) % Sh::kStaging;  // the other block, where the warp has two
        }
      }
    }
    if (lane == 0) bulk_wait_all();
    if constexpr (MSE) {
      // targets still on their way land before the shared memory goes away
      if (g.tma_t && lane == 0)
        for (int i = targets.used; i < targets.issued; i++)
          if (!mbar_wait_bounded(&sm.mse.tbar[ew], i & 1)) ok = false;
    }
    if (!ok) *failed = 1;
    if (MSE) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        loss += __shfl_xor_sync(0xffffffffu, loss, o);
        count += __shfl_xor_sync(0xffffffffu, count, o);
      }
      if (lane == 0) {
        atomicAdd(g.loss, loss);
        atomicAdd(g.count, count);
      }
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    fence_after_sync();
    tmem_dealloc(tmem, Sh::kTmemCols);
  }
  if (threadIdx.x == 0 && sm.failed) atomicOr(&g_gemm_failed, 1u);
  beside_exit(g.beside);
}

// The sum of the splits' products in FP64, rounded once: C in FP32 and BF16.
__global__ void __launch_bounds__(256) k_sum_splits(const float* __restrict__ part, int splits, size_t stride,
                                                    int m, int n, float* __restrict__ c, bf16* __restrict__ cb) {
  chained_entry();
  const size_t count = (size_t)m * n;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    int z = 0;
    for (; z + 16 <= splits; z += 16) {
      float v[16];
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] = __ldcs(part + (size_t)(z + j) * stride + i);
#pragma unroll
      for (int j = 0; j < 16; j++) s += (double)v[j];
    }
    for (; z < splits; z++) s += (double)__ldcs(part + (size_t)z * stride + i);
    const float f = (float)s;
    c[i] = f;
    if (cb) cb[i] = __float2bfloat16(f);
  }
}

// The network's inputs, handed over in the kernel's parameters (a copy from
// pageable host memory would first wait for the stream): BF16, rows padded
// with zeros to `pad`.
template <int N>
struct InputBlock {
  float v[N];
};
template <int N>
__global__ void __launch_bounds__(256) k_inputs(const __grid_constant__ InputBlock<N> x, int row0, int rows, int n_in,
                                                int pad, bf16* out) {
  chained_entry();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows * pad; i += gridDim.x * blockDim.x) {
    const int r = i / pad, c = i - r * pad;
    out[(size_t)(row0 + r) * pad + c] = __float2bfloat16(c < n_in ? x.v[r * n_in + c] : 0.f);
  }
}

// ------------------------------------------------------------------- host ----

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
  static EncodeFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<EncodeFn>(f);
  }();
  return fn;
}

// A row-major array (rows x cols, ld elements apart) in boxes of bx x by.
bool make_map(CUtensorMap* map, bool f32, const void* base, int rows, int cols, int ld, int bx, int by,
              CUtensorMapSwizzle swizzle) {
  const size_t el = f32 ? 4 : 2;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * el};
  const cuuint32_t box[2] = {(cuuint32_t)bx, (cuuint32_t)by};
  const cuuint32_t one[2] = {1, 1};
  const EncodeFn fn = encode_fn();
  return fn && fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                  const_cast<void*>(base), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, bool MSE, bool PLAIN>
cudaError_t launch_shape(const GemmArgs& g, const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& c,
                         const CUtensorMap& cb, const CUtensorMap& t, uint32_t items, cudaStream_t s) {
  static bool set[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const int smem = (int)sizeof(Smem<BN, MSE>);
  static_assert(sizeof(Smem<BN, MSE>) <= 227 * 1024, "shared memory of one CTA");
  if (!set[dev & 63]) {
    e = cudaFuncSetAttribute(k_gemm<BN, MSE, PLAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    set[dev & 63] = true;
  }
  return launch_chained(k_gemm<BN, MSE, PLAIN>, std::min<uint32_t>(items, (uint32_t)num_sms()), Shape<BN, MSE>::kThreads, smem, s, true, g,
                        a, b, c, cb, t);
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// The common part of the entry points: tile width, tensor maps, launch.
// a_trans / b_trans as dsmc_gemm_bf16.
template <bool MSE>
int run(GemmArgs g, const void* a, int lda, int a_trans, const void* b, int ldb, int b_trans, cudaStream_t s) {
  using umma::kBK;
  using umma::kBM;
  g.a_mn = a_trans;
  g.b_mn = !b_trans;
  g.tiles_m = (g.m + kBM - 1) / kBM;
  // The widest tile that still gives every SM one: 256 columns halve the
  // operand traffic of 128; where there are fewer such tiles than SMs, the
  // chain of one tile is what the call waits for, and narrow tiles spread it.
  const int sms = num_sms();
  auto items = [&](int bn) {
    const int tn = (g.n + bn - 1) / bn;
    return (int64_t)tn * (MSE ? 1 : (int64_t)g.tiles_m * g.splits);
  };
  const int bn = !MSE && items(256) >= sms ? 256 : items(128) >= sms ? 128 : 64;
  g.tiles_n = (g.n + bn - 1) / bn;
  const int64_t n_items = items(bn);
  if (n_items > 0x7fffffff) return DSMC_ERR_ARG;
  CUtensorMap ma, mb, mc{}, mcb{}, mt{};
  const CUtensorMapSwizzle s128 = CU_TENSOR_MAP_SWIZZLE_128B;
  if (!(a_trans ? make_map(&ma, false, a, g.k, g.m, lda, 64, kBK, s128)
                : make_map(&ma, false, a, g.m, g.k, lda, kBK, kBM, s128)))
    return DSMC_ERR_ARG;
  if (!(b_trans ? make_map(&mb, false, b, g.n, g.k, ldb, kBK, bn, s128)
                : make_map(&mb, false, b, g.k, g.n, ldb, 64, kBK, s128)))
    return DSMC_ERR_ARG;
  // outputs by TMA where their rows allow it and nothing is read back
  g.tma_c = g.c && aligned16(g.c) && g.ldc % 4 == 0 && g.ldc >= g.n && g.beta == 0.f &&
            make_map(&mc, true, g.c, g.part_rows ? g.part_rows * g.splits : g.m, g.n, g.ldc, 32, 32, s128);
  if (g.part_rows && !g.tma_c) return DSMC_ERR_ARG;
  g.tma_cb = g.cb && aligned16(g.cb) && g.ldcb % 8 == 0 && g.ldcb >= g.n &&
             make_map(&mcb, false, g.cb, g.m, g.n, g.ldcb, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B);
  g.tma_t = MSE && aligned16(g.t) && g.ldt % 8 == 0 &&
            make_map(&mt, false, g.t, g.m, g.n, g.ldt, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B);
  const uint32_t count = (uint32_t)n_items;
  cudaError_t e;
  if constexpr (MSE) {  // (its plain stores are in the one form)
    e = bn == 128 ? launch_shape<128, true, false>(g, ma, mb, mc, mcb, mt, count, s)
                  : launch_shape<64, true, false>(g, ma, mb, mc, mcb, mt, count, s);
  } else if ((g.c && !g.tma_c) || (g.cb && !g.tma_cb)) {
    e = bn == 256   ? launch_shape<256, false, true>(g, ma, mb, mc, mcb, mt, count, s)
        : bn == 128 ? launch_shape<128, false, true>(g, ma, mb, mc, mcb, mt, count, s)
                    : launch_shape<64, false, true>(g, ma, mb, mc, mcb, mt, count, s);
  } else {
    e = bn == 256   ? launch_shape<256, false, false>(g, ma, mb, mc, mcb, mt, count, s)
        : bn == 128 ? launch_shape<128, false, false>(g, ma, mb, mc, mcb, mt, count, s)
                    : launch_shape<64, false, false>(g, ma, mb, mc, mcb, mt, count, s);
  }
  return e == cudaSuccess ? DSMC_OK : DSMC_ERR_CUDA;
}

template <int N>
cudaError_t launch_inputs(const float* x, int row0, int rows, int n_in, int pad, bf16* out, cudaStream_t s) {
  InputBlock<N> b;
  std::memcpy(b.v, x + (size_t)row0 * n_in, (size_t)rows * n_in * sizeof(float));
  return launch_chained(k_inputs<N>, grid_for((uint64_t)rows * pad, 256, 1), 256, 0, s, true, b, row0, rows, n_in, pad,
                        out);
}

}  // namespace

extern "C" {

static int gemm(int m, int n, int k, const void* a, int lda, int a_trans, const void* b, int ldb, int b_trans,
                float* c, int ldc, float beta, const float* bias, int act, void* c_bf16, int ldcb, int split_k,
                bool b_early, bool beside, void* stream) {
  if (m <= 0 || n <= 0 || k <= 0 || !a || !b || (!c && !c_bf16)) return DSMC_ERR_ARG;
  // 16-byte rows along the contiguous dimension of each operand
  if (k % 8 || lda % 8 || ldb % 8 || !aligned16(a) || !aligned16(b)) return DSMC_ERR_ARG;
  if ((a_trans && m % 8) || (!b_trans && n % 8)) return DSMC_ERR_ARG;
  if (split_k < 1) split_k = 1;
  if (split_k > 1 && (!c || bias || act || c_bf16)) return DSMC_ERR_ARG;
  GemmArgs g{};
  g.m = m; g.n = n; g.k = k;
  g.c = c; g.ldc = ldc; g.beta = beta;
  g.bias = bias; g.act = act;
  g.cb = static_cast<bf16*>(c_bf16); g.ldcb = ldcb;
  const int ksteps = (k + umma::kBK - 1) / umma::kBK;
  const int per = (ksteps + split_k - 1) / split_k;
  g.kchunk = per * umma::kBK;
  g.splits = (k + g.kchunk - 1) / g.kchunk;
  g.b_early = b_early;
  g.beside = beside;
  return run<false>(g, a, lda, a_trans != 0, b, ldb, b_trans != 0, (cudaStream_t)stream);
}

int dsmc_gemm_bf16(int m, int n, int k, const void* a, int lda, int a_trans, const void* b, int ldb,
                   int b_trans, float* c, int ldc, float beta, const float* bias, int act, void* c_bf16,
                   int ldcb, int split_k, void* stream) {
  return gemm(m, n, k, a, lda, a_trans, b, ldb, b_trans, c, ldc, beta, bias, act, c_bf16, ldcb, split_k, false, false,
              stream);
}

int dsmc_gemm_split_bf16(int m, int n, int k, const void* a, int lda, int a_trans, const void* b, int ldb,
                         int b_trans, float* c, void* c_bf16, int split_k, float* workspace, void* stream) {
  if (m <= 0 || n <= 0 || k <= 0 || !a || !b || !c || !workspace || split_k < 1) return DSMC_ERR_ARG;
  if (k % 8 || lda % 8 || ldb % 8 || n % 4 || !aligned16(a) || !aligned16(b) || !aligned16(workspace))
    return DSMC_ERR_ARG;
  if ((a_trans && m % 8) || (!b_trans && n % 8)) return DSMC_ERR_ARG;
  GemmArgs g{};
  g.m = m; g.n = n; g.k = k;
  g.c = workspace; g.ldc = n;
  const int ksteps = (k + umma::kBK - 1) / umma::kBK;
  g.kchunk = (ksteps + split_k - 1) / split_k * umma::kBK;
  g.splits = (k + g.kchunk - 1) / g.kchunk;
  // whole 32-row blocks per split: a store of one never reaches the next's rows
  g.part_rows = (m + 31) / 32 * 32;
  const int st = run<false>(g, a, lda, a_trans != 0, b, ldb, b_trans != 0, (cudaStream_t)stream);
  if (st != DSMC_OK) return st;
  const cudaError_t e = launch_chained(k_sum_splits, grid_for((uint64_t)m * n, 256, 8), 256, 0, (cudaStream_t)stream,
                                       true, (const float*)workspace, g.splits, (size_t)g.part_rows * n, m, n, c,
                                       static_cast<bf16*>(c_bf16));
  return e == cudaSuccess ? DSMC_OK : DSMC_ERR_CUDA;
}

size_t dsmc_gemm_split_workspace(int m, int n, int split_k) {
  return m > 0 && n > 0 && split_k > 0 ? (size_t)split_k * ((m + 31) / 32 * 32) * n * sizeof(float) : 0;
}

int dsmc_decode_mse(int m, int n, int k, const void* a, const void* b, const float* bias, const void* t_bf16,
                    float scale, float* y, void* dy_bf16, float* dy_colsum, double* loss,
                    unsigned long long* count, void* stream) {
  if (m <= 0 || n <= 0 || k <= 0 || !a || !b || !t_bf16 || !y || !dy_bf16 || !dy_colsum || !loss || !count)
    return DSMC_ERR_ARG;
  if (k % 8 || n % 8 || !aligned16(a) || !aligned16(b)) return DSMC_ERR_ARG;
  GemmArgs g{};
  g.m = m; g.n = n; g.k = k;
  g.c = y; g.ldc = n;
  g.bias = bias;
  g.cb = static_cast<bf16*>(dy_bf16); g.ldcb = n;
  g.kchunk = (k + umma::kBK - 1) / umma::kBK * umma::kBK;
  g.splits = 1;
  g.t = static_cast<const bf16*>(t_bf16); g.ldt = n;
  g.scale = scale;
  g.colsum = dy_colsum;
  g.loss = loss;
  g.count = count;
  return run<true>(g, a, k, 0, b, n, 0, (cudaStream_t)stream);
}

int dsmc_mlp_forward(const dsmc_mlp* n, const float* x, int batch, void* xb, float* const* z, void* const* h, void* cb,
                     float* y, void* stream) {
  if (!n || !x || batch <= 0 || !xb || !h || !cb || n->depth < 0 || n->n_in <= 0 ||
      n->in_pad < n->n_in || n->n_in > 4096 || (n->depth == 0 && n->hidden != n->in_pad))
    return DSMC_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  // as many rows per launch as the parameters hold
  const int small = 1000, large = 4096;
  for (int r = 0; r < batch;) {
    const bool few = (batch - r) * (int64_t)n->n_in <= small;
    const int rows = std::min(batch - r, (few ? small : large) / n->n_in);
    const cudaError_t e = few ? launch_inputs<small>(x, r, rows, n->n_in, n->in_pad, static_cast<bf16*>(xb), s)
                              : launch_inputs<large>(x, r, rows, n->n_in, n->in_pad, static_cast<bf16*>(xb), s);
    if (e != cudaSuccess) return DSMC_ERR_CUDA;
    r += rows;
  }
  // the weights are nothing that the kernels of this pass write, and whatever
  // wrote them before the pass was complete before its first kernel's work
  const void* in = xb;
  int k = n->in_pad;
  for (int l = 0; l < n->depth; l++) {
    const int st = gemm(batch, n->hidden, k, in, k, 0, n->w[l], n->hidden, 0, z ? z[l] : nullptr, n->hidden, 0.f,
                        n->b[l], 1, h[l], n->hidden, 1, true, false, stream);
    if (st != DSMC_OK) return st;
    in = h[l];
    k = n->hidden;
  }
  int st = gemm(batch, n->modes, k, in, k, 0, n->w_out, n->modes, 0, nullptr, 0, 0.f, n->b_out, 0, cb, n->modes, 1,
                true, false, stream);
  if (st == DSMC_OK && y)
    st = gemm(batch, n->fields, n->modes, cb, n->modes, 0, n->basis, n->fields, 0, y, n->fields, 0.f, n->mean, 0,
              nullptr, 0, 1, true, false, stream);
  return st;
}

// Three results of a layer's gradient dz that do not depend on one another,
// each too small for the GPU (1024 x 512: 32, 16 and 64 blocks): the weights'
// GEMM waits for what is on the stream, the other two run beside it (one
// after the other 33 us a layer; with Adam's parameters beside one another too,
// a step on 1024 conditions 1692 -> 1586 us).
int dsmc_layer_backward(int batch, int din, int dout, const void* x, const float* dz, const void* dz_bf16,
                        const void* w, float* dw, float* db, float* dx, void* stream) {
  if (batch <= 0 || din <= 0 || dout <= 0 || !x || !dz || !dz_bf16 || !dw || !db || (dx && !w)) return DSMC_ERR_ARG;
  int st = gemm(din, dout, batch, x, din, 1, dz_bf16, dout, 0, dw, dout, 0.f, nullptr, 0, nullptr, 0, 1, false, false,
                stream);
  if (st != DSMC_OK) return st;
  if (launch_colsum_beside(dz, batch, dout, dout, db, (cudaStream_t)stream) != cudaSuccess) return DSMC_ERR_CUDA;
  if (dx)
    st = gemm(batch, din, dout, dz_bf16, dout, 0, w, dout, 1, dx, din, 0.f, nullptr, 0, nullptr, 0, 1, false, true, stream);
  return st;
}

int dsmc_gemm_check(void* stream) {
  if (cudaStreamSynchronize((cudaStream_t)stream) != cudaSuccess) return DSMC_ERR_CUDA;
  unsigned int f = 0;
  if (cudaMemcpyFromSymbol(&f, g_gemm_failed, sizeof(f)) != cudaSuccess) return DSMC_ERR_CUDA;
  if (!f) return DSMC_OK;
  f = 0;
  if (cudaMemcpyToSymbol(g_gemm_failed, &f, sizeof(f)) != cudaSuccess) return DSMC_ERR_CUDA;
  return DSMC_ERR_DEVICE;
}

}  // extern "C"
