// Kernels of the DSMC timestep other than the fused cell kernel (sm_100a):
// the cell-start scan, the scatter into sorted order, the initial keys, the
// stage kernels, the initial fill and the inflow injection.
//
// Memory plan per particle and step (SoA FP32 state, 24 B):
//   scatter: read key 4 B + state 24 B, write state 24 B + orig 4 B
//   cell:    read state 24 B + orig 4 B, write state 24 B + key 4 B
// Per-cell arrays (counts, starts, (sigma*g)max/remainder, RNG state) add a
// few bytes per particle.  All particle traffic is coalesced except the
// scatter's writes, which land near-sorted because most particles stay in or
// next to their cell between steps.
#include <algorithm>

#include "dsmc_step_dev.cuh"

namespace dsmcb {
namespace {

using namespace dev;

// Move stage: free flight and boundaries for n particles in place.  Without a
// body and from kMoveByFour particles on each thread flies four at a time,
// their loads in flight together (4.2M particles: 38 -> 34 us; 800,000 7.3 ->
// 7.7, and a call on 20,000 with diffuse faces 16 -> 19 us: the boundaries of a
// thread's particles come one after the other).
constexpr uint32_t kMoveByFour = 1500000;
template <bool BODY, int U>
__global__ void __launch_bounds__(256) k_move(const __grid_constant__ StepParams p, uint32_t n, uint32_t step) {
  for (uint32_t base = blockIdx.x * blockDim.x * U; base < n; base += gridDim.x * blockDim.x * U) {
    float3 pos[U], vel[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
      const uint32_t i = base + k * blockDim.x + threadIdx.x;
      if (i < n) {
        pos[k] = make_float3(p.out.x[i], p.out.y[i], p.out.z[i]);
        vel[k] = make_float3(p.out.u[i], p.out.v[i], p.out.w[i]);
      }
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      const uint32_t i = base + k * blockDim.x + threadIdx.x;
      if (i >= n) continue;
      const bool live = BODY ? move_particle(p, pos[k], vel[k], i, step) : move_free(p, pos[k], vel[k], i, step);
      p.out.x[i] = live ? pos[k].x : __int_as_float(0x7fc00000);
      p.out.y[i] = pos[k].y; p.out.z[i] = pos[k].z;
      p.out.u[i] = vel[k].x; p.out.v[i] = vel[k].y; p.out.w[i] = vel[k].z;
    }
  }
}

__global__ void __launch_bounds__(256) k_cell_ids(GridGeom g, const float* __restrict__ x,
                                                  const float* __restrict__ y,
                                                  const float* __restrict__ z, uint32_t n,
                                                  uint32_t* __restrict__ keys,
                                                  uint32_t* __restrict__ idx) {
  constexpr int U = 4;  // positions in flight per thread
  for (uint32_t base = blockIdx.x * blockDim.x * U; base < n; base += gridDim.x * blockDim.x * U) {
    float3 q[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
      const uint32_t i = base + k * blockDim.x + threadIdx.x;
      if (i < n) q[k] = make_float3(x[i], y[i], z[i]);
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      const uint32_t i = base + k * blockDim.x + threadIdx.x;
      if (i >= n) continue;
      keys[i] = cell_id3d(g, q[k].x, q[k].y, q[k].z);
      if (idx) idx[i] = i;
    }
  }
}

// Keys and counts of a freshly uploaded state (particles outside the box are
// dead when the faces are in use).
__global__ void k_index(GridGeom g, const float* __restrict__ x, const float* __restrict__ y,
                        const float* __restrict__ z, uint32_t n, uint32_t* __restrict__ keys,
                        uint32_t* count, uint32_t* tile_sum, uint32_t n_scan_tiles, int face_mode) {
  extern __shared__ uint32_t s_tile[];
  for (uint32_t t = threadIdx.x; t < n_scan_tiles; t += blockDim.x) s_tile[t] = 0;
  __syncthreads();
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    const bool active = i < n;
    bool live = false;
    uint32_t key = kDeadKey;
    if (active) {
      const float px = x[i], py = y[i], pz = z[i];
      live = !(face_mode != 0 && (px < g.gmin.x || px > g.gmax.x || py < g.gmin.y ||
                                   py > g.gmax.y || pz < g.gmin.z || pz > g.gmax.z));
      if (live) key = cell_id3d(g, px, py, pz);
      keys[i] = key;
    }
    if (active && live) warp_count_key(count, key, s_tile);
  }
  __syncthreads();
  flush_tile_hist(s_tile, tile_sum, n_scan_tiles);
}

// Exclusive scan of per-cell counts.  Block b owns cells [b*2048, (b+1)*2048);
// its offset is the sum of the per-tile totals before it, which the producer
// kernels accumulated alongside the counts.  Resets the counts and the
// scatter's cursors.
__device__ __forceinline__ void scan_body(uint32_t* count, uint32_t* cursor, uint32_t* start,
                                          uint32_t cells, const uint32_t* tile_sum, Meta* meta, int bump,
                                          const uint32_t vb, const uint32_t vg) {
  __shared__ uint32_t s_warp[8], s_part[8];
  const uint32_t b = vb;
  // the block's counts and the totals of the tiles before it, loaded together
  const uint32_t c0 = b * kScanTile + threadIdx.x * 8;
  // 8 whole counts, read and written 16 bytes at a time where the arrays
  // allow it (the stage API's workspace may be only 4-byte aligned)
  const bool vec = (((uintptr_t)count | (uintptr_t)start | (uintptr_t)cursor) & 15u) == 0;
  const bool whole = vec && c0 + 8u <= cells;
  uint32_t v[8];
  if (whole) {
    const uint4 lo = *reinterpret_cast<const uint4*>(count + c0);
    const uint4 hi = *reinterpret_cast<const uint4*>(count + c0 + 4);
    v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
    v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = (c0 + i < cells) ? count[c0 + i] : 0u;
  }
  uint32_t part = 0;
  for (uint32_t t = threadIdx.x; t < b; t += blockDim.x) part += tile_sum[t];
  part = warp_sum(part);
  uint32_t tsum = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) tsum += v[i];
  uint32_t incl = tsum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, incl, o);
    if ((int)lane_id() >= o) incl += t;
  }
  if (lane_id() == 31) s_warp[threadIdx.x / 32] = incl;
  if (lane_id() == 0) s_part[threadIdx.x / 32] = part;
  __syncthreads();
  uint32_t run = incl - tsum;
#pragma unroll
  for (uint32_t w = 0; w < 8; w++) {
    run += s_part[w];
    if (w < threadIdx.x / 32) run += s_warp[w];
  }
  uint32_t st[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    st[i] = run;
    run += v[i];
  }
  if (whole) {
    *reinterpret_cast<uint4*>(start + c0) = make_uint4(st[0], st[1], st[2], st[3]);
    *reinterpret_cast<uint4*>(start + c0 + 4) = make_uint4(st[4], st[5], st[6], st[7]);
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(count + c0) = z;
    *reinterpret_cast<uint4*>(count + c0 + 4) = z;
    if (cursor) {
      *reinterpret_cast<uint4*>(cursor + c0) = z;
      *reinterpret_cast<uint4*>(cursor + c0 + 4) = z;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      if (c0 + i < cells) {
        start[c0 + i] = st[i];
        count[c0 + i] = 0u;
        if (cursor) cursor[c0 + i] = 0u;
      }
    }
  }
  if (b == vg - 1 && threadIdx.x == blockDim.x - 1) {
    start[cells] = run;
    meta->n_scatter = meta->n_alive + meta->n_pending;
    meta->n_pending = 0;
    meta->n_alive = run;
    meta->tile_next = 0;
    meta->tile_next2 = 0;
    meta->n_defer = 0;
    meta->n_light = 0;
    meta->n_heavy = 0;
    meta->n_heaviest = 0;
    if (bump) {
      meta->step += 1;
      meta->particle_steps += run;
    }
  }
}

__global__ void __launch_bounds__(256) k_scan(uint32_t* count, uint32_t* cursor, uint32_t* start,
                                              uint32_t cells, const uint32_t* tile_sum, Meta* meta,
                                              int bump) {
  chained_entry();
  scan_body(count, cursor, start, cells, tile_sum, meta, bump, blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(256) k_scan_b(const __grid_constant__ BatchOf<SortArgs> bv) {
  chained_entry();
  uint32_t vb, vg;
  const SortArgs& a = bv.locate(vb, vg);
  scan_body(a.count, a.cursor, a.start, a.cells, a.tile_sum, a.meta, 1, vb, vg);
}

// Scatter into sorted order: dst[start[key] + ticket] = src[i], orig = i.  The
// tickets come from per-cell cursors (one atomic per distinct key per group of
// 32).  Each warp takes kScatterU groups of 32 consecutive particles at once,
// so that their chains of key load -> ticket atomic -> stores overlap.  With
// STATE false only orig is written: one scattered 4-byte store per particle
// instead of seven (scattered stores, not the loads or the atomics, bound this
// kernel), and the split cell kernels gather the state through orig.
constexpr int kScatterU = 4;

template <bool STATE>
__device__ __forceinline__ void scatter_body(SoA src, SoA dst, const uint32_t* __restrict__ keys,
                                             const uint32_t* __restrict__ start, uint32_t* cursor,
                                             uint32_t* __restrict__ orig, uint32_t cells,
                                             uint32_t* tile_sum, uint32_t n_scan_tiles, Meta* meta,
                                             uint32_t capacity, const uint32_t vb, const uint32_t vg) {
  if (vb == 0)
    for (uint32_t t = threadIdx.x; t < n_scan_tiles; t += blockDim.x) tile_sum[t] = 0;
  const uint32_t n = meta->n_scatter;
  const uint32_t lane = lane_id();
  const uint32_t gw = (vb * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (vg * blockDim.x) >> 5;
  constexpr int U = kScatterU;
  const uint32_t stride = nw * 32u * U;
  // keys of the next iteration load while this one's tickets are in flight
  uint32_t nkey[U];
#pragma unroll
  for (int k = 0; k < U; k++) {
    const uint32_t i = gw * 32u * U + 32u * k + lane;
    nkey[k] = i < n ? __ldcs(&keys[i]) : kDeadKey;
  }
  for (uint32_t base = gw * 32u * U; base < n; base += stride) {
    uint32_t key[U];
    float x[U], y[U], z[U], u[U], v[U], w[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
      key[k] = nkey[k];
      const uint32_t i2 = base + stride + 32u * k + lane;
      nkey[k] = i2 < n ? __ldcs(&keys[i2]) : kDeadKey;
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      const uint32_t i = base + 32u * k + lane;
      x[k] = y[k] = z[k] = u[k] = v[k] = w[k] = 0.f;
      if (STATE && i < n) {
        x[k] = src.x[i]; y[k] = src.y[i]; z[k] = src.z[i];
        u[k] = src.u[i]; v[k] = src.v[i]; w[k] = src.w[i];
      }
    }
    // the ticket atomics of all groups first, then their broadcasts
    unsigned msk[U], peers[U];
    uint32_t st[U], got[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
      const uint32_t i = base + 32u * k + lane;
      const bool live = key[k] < cells;
      if (i < n && key[k] != kDeadKey && !live) atomicOr(&meta->error, kErrKeyRange);
      msk[k] = __ballot_sync(kFull, live);
      st[k] = 0;
      got[k] = 0;
      peers[k] = 0;
      if (live) {
        st[k] = __ldg(&start[key[k]]);
        peers[k] = __match_any_sync(msk[k], key[k]);
        if ((int)lane == __ffs(peers[k]) - 1) got[k] = atomicAdd(&cursor[key[k]], (uint32_t)__popc(peers[k]));
      }
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      if (!(key[k] < cells)) continue;
      const uint32_t i = base + 32u * k + lane;
      const uint32_t t = __shfl_sync(msk[k], got[k], __ffs(peers[k]) - 1) +
                         __popc(peers[k] & ((1u << lane) - 1u));
      const uint32_t d = st[k] + t;
      if (d >= capacity) {
        atomicOr(&meta->error, kErrKeyRange);
        continue;
      }
      if (STATE) {
        dst.x[d] = x[k]; dst.y[d] = y[k]; dst.z[d] = z[k];
        dst.u[d] = u[k]; dst.v[d] = v[k]; dst.w[d] = w[k];
      }
      orig[d] = i;
    }
  }
}

template <bool STATE>
__global__ void __launch_bounds__(256, 4) k_scatter(SoA src, SoA dst, const uint32_t* __restrict__ keys,
                                                    const uint32_t* __restrict__ start,
                                                    uint32_t* cursor, uint32_t* __restrict__ orig,
                                                    uint32_t cells, uint32_t* tile_sum,
                                                    uint32_t n_scan_tiles, Meta* meta,
                                                    uint32_t capacity) {
  chained_entry();
  scatter_body<STATE>(src, dst, keys, start, cursor, orig, cells, tile_sum, n_scan_tiles, meta, capacity,
                      blockIdx.x, gridDim.x);
}
// orig only (the split kernels)
__global__ void __launch_bounds__(256, 4) k_scatter_b(const __grid_constant__ BatchOf<SortArgs> bv) {
  chained_entry();
  uint32_t vb, vg;
  const SortArgs& a = bv.locate(vb, vg);
  const SoA none{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  scatter_body<false>(none, none, a.keys, a.start, a.cursor, a.orig, a.cells, a.tile_sum, a.n_scan_tiles,
                      a.meta, a.capacity, vb, vg);
}

// ------------------------------------------------------------ sort stage ----

// A counting sort: counts per key, their scan, each entry to its key's range
// in any order (a ticket from the key's count, which the scan left at zero),
// and the input order restored inside each key.  Counting without tickets
// (non-returning atomics) and taking them in the scatter, four groups of 32
// in flight per warp, costs less than storing them: 4.2M entries, 524,288
// keys: count and scatter 45 + 27 -> 19 + 35 us.
// Keys >= nkeys are left out of the sort (no ticket, no slot).
__global__ void __launch_bounds__(256) k_count_keys(const uint32_t* __restrict__ keys, uint32_t n, uint32_t nkeys,
                                                    uint32_t* count, uint32_t* tile_sum, uint32_t n_scan_tiles) {
  extern __shared__ uint32_t s_tile[];
  for (uint32_t t = threadIdx.x; t < n_scan_tiles; t += blockDim.x) s_tile[t] = 0;
  __syncthreads();
  constexpr int U = 4;
  for (uint32_t base = blockIdx.x * blockDim.x * U; base < n; base += gridDim.x * blockDim.x * U) {
    uint32_t key[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
      const uint32_t i = base + k * blockDim.x + threadIdx.x;
      key[k] = i < n ? keys[i] : kNone;
    }
#pragma unroll
    for (int k = 0; k < U; k++)
      if (key[k] < nkeys) warp_count_key(count, key[k], s_tile);
  }
  __syncthreads();
  flush_tile_hist(s_tile, tile_sum, n_scan_tiles);
}

// Where the scatter puts (value, input position) of an entry: pairs where the
// workspace is 8-byte aligned (one store, one sector), else two arrays.
template <bool PAIR>
struct ScatterOut {
  uint32_t* val;
  uint32_t* pos;
  __device__ __forceinline__ void put(uint32_t d, uint32_t v, uint32_t i) const {
    if (PAIR) {
      reinterpret_cast<uint2*>(val)[d] = make_uint2(v, i);
    } else {
      val[d] = v;
      pos[d] = i;
    }
  }
  __device__ __forceinline__ uint2 get(uint32_t d) const {
    return PAIR ? reinterpret_cast<const uint2*>(val)[d] : make_uint2(val[d], pos[d]);
  }
  __device__ __forceinline__ uint32_t position(uint32_t d) const { return PAIR ? val[2 * (size_t)d + 1] : pos[d]; }
};

template <bool PAIR>
__global__ void __launch_bounds__(256) k_scatter_kv(const uint32_t* __restrict__ keys,
                                                    const uint32_t* __restrict__ vals,
                                                    const uint32_t* __restrict__ start, uint32_t* cursor, uint32_t n,
                                                    uint32_t nkeys, ScatterOut<PAIR> out) {
  constexpr int U = 4;
  const uint32_t lane = lane_id();
  for (uint32_t base = blockIdx.x * blockDim.x * U; base < n; base += gridDim.x * blockDim.x * U) {
    uint32_t key[U], val[U], st[U], got[U];
    unsigned peers[U], msk[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
      const uint32_t i = base + k * blockDim.x + threadIdx.x;
      key[k] = i < n ? keys[i] : kNone;
      val[k] = i < n ? vals[i] : 0u;
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      const bool live = key[k] < nkeys;
      msk[k] = __ballot_sync(kFull, live);
      st[k] = got[k] = 0;
      peers[k] = 0;
      if (live) {
        st[k] = __ldg(&start[key[k]]);
        peers[k] = __match_any_sync(msk[k], key[k]);
        if ((int)lane == __ffs(peers[k]) - 1) got[k] = atomicAdd(&cursor[key[k]], (uint32_t)__popc(peers[k]));
      }
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      if (!(key[k] < nkeys)) continue;
      const uint32_t i = base + k * blockDim.x + threadIdx.x;
      const uint32_t t = __shfl_sync(msk[k], got[k], __ffs(peers[k]) - 1) + __popc(peers[k] & ((1u << lane) - 1u));
      out.put(st[k] + t, val[k], i);
    }
  }
}

// Restores input order within each key: entry of rank r (by input position)
// among its key's entries goes to start[key] + r.  A CTA takes kt keys at a
// time (at most kFixupThreads), in chunks of whole keys of at most kFixupCap
// entries in shared memory; tiles are small (launch_sort), so that a
// few thousand keys reach every SM (4,096 keys of 24: 35 us with tiles of 256
// keys on 16 CTAs, now 5 us; 524,288 keys of 8: 58, now 34 us).
constexpr int kFixupThreads = 128, kFixupCap = 768;

// A key with more than kFixupCap entries (m at s0, the whole CTA): its entries
// [i0, i1), at most 4 kFixupThreads, are ranked against the key's positions,
// kFixupCap at a time in shared memory.  Each thread ranks up to four entries
// and reads four positions per load: bound by the comparisons, m squared of
// them (1,000,000 entries in 400 keys 57 ms with chunks of 4,096 and 256
// threads, 3.3 ms with chunks of 1,024 and such keys ranked from global memory,
// now 0.53; 4.2M entries in 524,288 keys, 1 % of them in keys of 2,500, 4.1, 4.4
// and 2.5 ms).  Eight entries per thread take 1.9 ms for the latter, but
// registers that cost every sort 4 %; a kernel of its own costs its launch.
template <bool PAIR>
__device__ __forceinline__ void rank_large_key(uint32_t* spos, const ScatterOut<PAIR>& in, uint32_t s0, uint32_t m,
                                               uint32_t i0, uint32_t i1, uint32_t key, uint32_t* keys_out,
                                               uint32_t* vals_out) {
  constexpr int Q = 4;
  uint32_t my[Q], rank[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) {
    const uint32_t t = i0 + threadIdx.x + q * kFixupThreads;
    my[q] = t < i1 ? in.position(s0 + t) : 0u;
    rank[q] = 0;
  }
  for (uint32_t j0 = 0; j0 < m; j0 += kFixupCap) {
    const uint32_t nj = min((uint32_t)kFixupCap, m - j0);
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < kFixupCap; t += kFixupThreads)
      spos[t] = t < nj ? in.position(s0 + j0 + t) : kNone;  // (counts for nobody)
    __syncthreads();
#pragma unroll 2
    for (uint32_t j = 0; j < nj; j += 4) {
      const uint4 o = *reinterpret_cast<const uint4*>(spos + j);
#pragma unroll
      for (int q = 0; q < Q; q++)
        rank[q] += (uint32_t)(o.x < my[q]) + (uint32_t)(o.y < my[q]) + (uint32_t)(o.z < my[q]) + (uint32_t)(o.w < my[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < Q; q++) {
    const uint32_t t = i0 + threadIdx.x + q * kFixupThreads;
    if (t >= i1) break;
    keys_out[s0 + rank[q]] = key;
    vals_out[s0 + rank[q]] = in.get(s0 + t).x;
  }
}

template <bool PAIR>
__global__ void __launch_bounds__(kFixupThreads) k_segment_fixup(const uint32_t* __restrict__ start, uint32_t nkeys,
                                                                 uint32_t kt, ScatterOut<PAIR> in,
                                                                 uint32_t* __restrict__ keys_out,
                                                                 uint32_t* __restrict__ vals_out) {
  __shared__ uint32_t ls[kFixupThreads + 1];
  __shared__ __align__(16) uint32_t spos[kFixupCap];
  __shared__ uint8_t cellof[kFixupCap];  // the chunk's key of each entry
  const uint32_t ntiles = (nkeys + kt - 1) / kt;
  for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const uint32_t c0 = tile * kt, nct = min(kt, nkeys - c0);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i <= nct; i += blockDim.x) ls[i] = start[c0 + i];
    __syncthreads();
    uint32_t cur = 0;
    while (cur < nct) {
      const uint32_t base = ls[cur];
      const uint32_t c = cur + 1 + threadIdx.x;
      const int fits = (c <= nct) && (ls[c] - base <= (uint32_t)kFixupCap);
      const uint32_t k = __syncthreads_count(fits);
      if (k == 0) {  // a key above the chunk, in passes of nearly equal size
        const uint32_t m = ls[cur + 1] - base, passes = (m + 4 * kFixupThreads - 1) / (4 * kFixupThreads);
        const uint32_t per = (m + passes * kFixupThreads - 1) / (passes * kFixupThreads) * kFixupThreads;
        for (uint32_t i0 = 0; i0 < m; i0 += per)
          rank_large_key(spos, in, base, m, i0, min(m, i0 + per), c0 + cur, keys_out, vals_out);
        cur += 1;
        __syncthreads();
        continue;
      }
      const uint32_t n = ls[cur + k] - base;
      if (threadIdx.x < k)
        for (uint32_t j = ls[cur + threadIdx.x]; j < ls[cur + threadIdx.x + 1]; j++)
          cellof[j - base] = (uint8_t)threadIdx.x;
      uint32_t val[kFixupCap / kFixupThreads];
#pragma unroll
      for (int q = 0; q < kFixupCap / kFixupThreads; q++) {
        const uint32_t t = threadIdx.x + q * kFixupThreads;
        if (t < n) {
          const uint2 e = in.get(base + t);
          val[q] = e.x;
          spos[t] = e.y;
        }
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kFixupCap / kFixupThreads; q++) {
        const uint32_t t = threadIdx.x + q * kFixupThreads;
        if (t >= n) break;
        const uint32_t lo = cur + cellof[t];
        const uint32_t s0 = ls[lo] - base, e0 = ls[lo + 1] - base;
        const uint32_t my = spos[t];
        uint32_t rank = 0;
        for (uint32_t j = s0; j < e0; j++) rank += spos[j] < my;
        keys_out[base + s0 + rank] = c0 + lo;
        vals_out[base + s0 + rank] = val[q];
      }
      cur += k;
      __syncthreads();
    }
  }
}

// FindCellBoundariesDev (kernels/dsmc_kernel.cu:1734-1787): start/end per
// cell from sorted keys (cse zeroed by the caller) and the gather.
// A particle's six loads are in flight together, before its stores, and a
// thread takes one at a time: four gather slower (4.2M particles moved by less
// than 50 places: 74 us with a load and a store after the other, 53 with four
// particles' 24 loads, now 45).  The bounds alone are taken four at a time
// (20M keys: 33 us one at a time), in a kernel without the gather's registers.
template <bool GATHER>
__global__ void __launch_bounds__(256) k_bounds_reorder(const uint32_t* __restrict__ keys,
                                                        const uint32_t* __restrict__ idx, uint32_t n, uint32_t ncells,
                                                        uint2* cse, SoA src, SoA dst) {
  constexpr int U = GATHER ? 1 : 4;
  for (uint32_t base = blockIdx.x * blockDim.x * U; base < n; base += gridDim.x * blockDim.x * U) {
    uint32_t h[U], hp[U];
    float v[6];
    const uint32_t i0 = base + threadIdx.x;
    if (GATHER && i0 < n) {
      const uint32_t s = idx[i0];
      v[0] = src.x[s]; v[1] = src.y[s]; v[2] = src.z[s];
      v[3] = src.u[s]; v[4] = src.v[s]; v[5] = src.w[s];
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      const uint32_t i = i0 + k * blockDim.x;
      h[k] = i < n ? keys[i] : kNone;
      hp[k] = i > 0 && i < n ? keys[i - 1] : kNone;
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      const uint32_t i = i0 + k * blockDim.x;
      if (i >= n) continue;
      if (i == 0 || h[k] != hp[k]) {
        if (h[k] < ncells) cse[h[k]].x = i;
        if (i > 0 && hp[k] < ncells) cse[hp[k]].y = i;
      }
      if (i == n - 1 && h[k] < ncells) cse[h[k]].y = i + 1;
    }
    if (GATHER && i0 < n) {
      dst.x[i0] = v[0]; dst.y[i0] = v[1]; dst.z[i0] = v[2];
      dst.u[i0] = v[3]; dst.v[i0] = v[4]; dst.w[i0] = v[5];
    }
  }
}

// Stand-alone FP64 sampling, one thread per cell, a cell's loads four
// particles at a time and ahead of its sums, which are added in order (4,096
// cells of 100: 30 us with a load after the other, 23 with four at a time, 19
// with the next four and the sums so far under way; 524,288 cells of 8 27,
// 25 and 21 us; a single cell of 30,000 1.66, 2.39 and 1.78 ms).
__global__ void __launch_bounds__(256) k_sample_cells(const float* __restrict__ u, const float* __restrict__ v,
                                                      const float* __restrict__ w,
                                                      const uint32_t* __restrict__ start, uint32_t cells, double* acc,
                                                      size_t fs, size_t cs) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < cells; c += gridDim.x * blockDim.x) {
    const uint32_t s = start[c], e = start[c + 1];
    if (e <= s) continue;
    double sum[5];  // so far: loaded beside the first particles
#pragma unroll
    for (int f = 0; f < 5; f++) sum[f] = acc[f * fs + c * cs];
    double su = 0, sv = 0, sw = 0, se = 0;
    auto add = [&](float a, float b, float d) {
      const double x = a, y = b, z = d;
      su += x; sv += y; sw += z;
      se += x * x + y * y + z * z;
    };
    // the next four particles' loads run while these are added
    uint32_t i = s;
    float q[3][4];
    auto load = [&](uint32_t at) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        q[0][k] = u[at + k]; q[1][k] = v[at + k]; q[2][k] = w[at + k];
      }
    };
    if (e - s >= 4u) load(s);
    for (; i + 4u <= e; i += 4u) {
      float r[3][4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        r[0][k] = q[0][k]; r[1][k] = q[1][k]; r[2][k] = q[2][k];
      }
      if (e - i >= 8u) load(i + 4u);
#pragma unroll
      for (int k = 0; k < 4; k++) add(r[0][k], r[1][k], r[2][k]);
    }
    for (; i < e; i++) add(u[i], v[i], w[i]);
    acc[c * cs] = sum[0] + (double)(e - s);
    acc[fs + c * cs] = sum[1] + su;
    acc[2 * fs + c * cs] = sum[2] + sv;
    acc[3 * fs + c * cs] = sum[3] + sw;
    acc[4 * fs + c * cs] = sum[4] + se;
  }
}

// Collide stage: the NTC collisions of every cell of the caller's sorted
// velocities, in place.  A warp takes ct <= 32 consecutive cells, a lane each;
// cells with many pairs (Philox mode) follow, the whole warp on each.  The
// same draws and arithmetic per cell as the fused cell kernel in its
// 2048-particle form, which this replaces here: that one staged a chunk of
// cells per CTA between barriers, on 16 CTAs for 4,096 cells (4,096 cells of
// 24: 34 -> 12 us; 524,288 of 8: 183 -> 36 us).
constexpr int kCollideWarps = 8;
constexpr uint32_t kCollideClaim = 256;    // largest cell staged in shared memory
constexpr uint32_t kCollideGiant = 2048;   // above: one lane whatever its pairs
__global__ void __launch_bounds__(32 * kCollideWarps) k_collide_cells(const __grid_constant__ StepParams p,
                                                                      uint32_t ct) {
  __shared__ uint32_t s_claim[kCollideWarps][kCollideClaim];
  __shared__ float s_vel[kCollideWarps][3][kCollideClaim];
  const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
  for (uint32_t t = lane; t < kCollideClaim; t += 32) s_claim[warp][t] = 0xffffffffu;
  __syncwarp();
  const bool taus = p.rng_kind == 0;
  uint32_t sel = 0, col = 0;
  double sum_g = 0.0;
  const uint32_t tiles = (p.cells + ct - 1u) / ct;
  for (uint32_t t = blockIdx.x * kCollideWarps + warp; t < tiles; t += gridDim.x * kCollideWarps) {
    const uint32_t c = t * ct + lane;
    const bool mine = lane < ct && c < p.cells;
    uint32_t s = 0, n = 0;
    bool heavy = false;
    if (mine) {
      s = p.start[c];
      n = p.start[c + 1] - s;
      if (!taus && n >= 2 && n <= kCollideGiant) heavy = (uint32_t)ntc_fpc_fast(p, n, p.maxrem[c]) >= kHeavyMin;
    }
    if (mine && !heavy) {
      GlobalVel acc{p.in.u, p.in.v, p.in.w, s};
      CellState st{p.maxrem + c, taus ? p.seeds + c : nullptr, p.stat4 ? p.stat4 + c : nullptr};
      collide_cell(p, c, (int)n, acc, p.step_override, st, sel, col, sum_g);
    }
    __syncwarp();
    for (unsigned m = __ballot_sync(kFull, heavy); m; m &= m - 1u) {
      const int l = __ffs(m) - 1;
      const uint32_t hc = t * ct + (uint32_t)l, hs = __shfl_sync(kFull, s, l), hn = __shfl_sync(kFull, n, l);
      CellState st{p.maxrem + hc, nullptr, p.stat4 ? p.stat4 + hc : nullptr};
      GlobalVel acc{p.in.u, p.in.v, p.in.w, hs};
      if (hn > kCollideClaim) {
        ntc_heavy_warp<false>(p, hc, hn, acc, nullptr, p.step_override, st, sel, col, sum_g);
      } else {
        float* su = s_vel[warp][0];
        float* sv = s_vel[warp][1];
        float* sw = s_vel[warp][2];
        for (uint32_t k = lane; k < hn; k += 32) {
          su[k] = acc.u[hs + k];
          sv[k] = acc.v[hs + k];
          sw[k] = acc.w[hs + k];
        }
        __syncwarp();
        ntc_heavy_warp(p, hc, hn, GlobalVel{su, sv, sw, 0u}, s_claim[warp], p.step_override, st, sel, col, sum_g);
        __syncwarp();
        for (uint32_t k = lane; k < hn; k += 32) {
          acc.u[hs + k] = su[k];
          acc.v[hs + k] = sv[k];
          acc.w[hs + k] = sw[k];
        }
      }
      __syncwarp();
    }
  }
}

// Per-cell fields (n, ux, uy, uz, T), cell-major, from the FP64 sampling sums
// (5 x cells, SoA) of ns passes: ProcessAndOutputStatistics' arithmetic
// (kernels/dsmc_base.cu:104-163) in double with every rounding step explicit,
// the same steps as the host code; with fields == 0 the sums themselves,
// transposed to cell-major.
__global__ void k_cell_fields(const double* __restrict__ acc, uint32_t cells, double fnum,
                              double cell_volume, uint32_t ns, double mass, int fields,
                              double* __restrict__ out) {
  const double k3 = 3.0 * 1.3806e-23;
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < cells; c += gridDim.x * blockDim.x) {
    const double N = acc[c], a1 = acc[(size_t)cells + c], a2 = acc[2 * (size_t)cells + c],
                 a3 = acc[3 * (size_t)cells + c], a4 = acc[4 * (size_t)cells + c];
    double* o = out + 5 * (size_t)c;
    if (!fields) {
      o[0] = N; o[1] = a1; o[2] = a2; o[3] = a3; o[4] = a4;
      continue;
    }
    o[0] = ns ? __ddiv_rn(__dmul_rn(fnum, N), __dmul_rn(cell_volume, (double)ns)) : 0.0;
    if (N > 0) {
      const double ux = __ddiv_rn(a1, N), uy = __ddiv_rn(a2, N), uz = __ddiv_rn(a3, N);
      const double u2 = __dadd_rn(__dadd_rn(__dmul_rn(ux, ux), __dmul_rn(uy, uy)), __dmul_rn(uz, uz));
      o[1] = ux; o[2] = uy; o[3] = uz;
      o[4] = __ddiv_rn(__dmul_rn(mass, __dsub_rn(__ddiv_rn(a4, N), u2)), k3);
    } else {
      o[1] = o[2] = o[3] = o[4] = 0.0;
    }
  }
}

// ------------------------------------------------------------ init fill ----

// Initial population: part_per_cell particles per cell at uniform positions
// (GetRandomPosition, kernels/dsmc_kernel.cu:417-427) with either the
// reference's speed/angle sampler (GetRandomVelocity, :394-415) or an exact
// Maxwellian.  Random numbers come from Philox (the reference used its
// Mersenne-Twister table, which is not reproduced).

// Particle k of a cell is number cell * ppc + k (ppc: the most in any cell),
// which names its random stream.  A thread per number finds its cell by a
// division, but numbers stop at 32 bits, and one crowded cell on a large grid
// takes them further; WIDE: a thread per slot, its cell found among the slots
// (cell_count is then null, as in the fills from fields), and a number's upper
// word in the stream's next counter word.
constexpr uint64_t kFillNumbers = 0xF0000000ull;  // leaves room for a grid's stride
__device__ __forceinline__ uint32_t cell_of_slot(const uint32_t* slot, uint32_t cells, uint32_t d) {
  uint32_t lo = 0, hi = cells - 1u;  // the last cell that begins at or before d: empty ones come before it
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo + 1u) / 2u;
    if (slot[mid] <= d) lo = mid;
    else hi = mid - 1u;
  }
  return lo;
}

// A position in a cell from three uniforms.
__device__ __forceinline__ float3 fill_position(const InitParams& p, uint32_t cell, float a, float b, float c) {
  const uint32_t cx = cell % p.grid.dim.x;
  const uint32_t cy = (cell / p.grid.dim.x) % p.grid.dim.y;
  const uint32_t cz = cell / (p.grid.dim.x * p.grid.dim.y);
  const float3 lo = make_float3(p.grid.gmin.x + cx * p.grid.cell.x, p.grid.gmin.y + cy * p.grid.cell.y,
                                p.grid.gmin.z + cz * p.grid.cell.z);
  return make_float3(lo.x + a * p.grid.cell.x, lo.y + b * p.grid.cell.y, lo.z + c * p.grid.cell.z);
}

// Redraws of the listed particles' positions (at most 64, then the cell's
// known outside point): a warp per particle, its lanes testing 32 of the
// redraws at a time against the mesh; the first one outside counts, as if
// drawn one after the other.  A thread that drew them itself held its warp
// for up to 64 walks of the grid (fill of 65,536 cells around a sphere:
// 1231 us, now 168 us in two kernels).
constexpr uint32_t kRedraws = 64;
template <bool WIDE>
__global__ void __launch_bounds__(256) k_init_redraw(const __grid_constant__ InitParams p) {
  const uint32_t lane = lane_id(), n = *p.n_redo;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  // words the particle's stream has handed out before: velocity and position
  const uint32_t w0 = 4u + ((p.kind != 0 && p.cell_state && p.cell_mix) ? 1u : 0u) + 3u;
  for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += warps) {
    uint32_t i, ihi = 0, cell, d;
    if (WIDE) {
      d = p.redo[r];
      cell = cell_of_slot(p.cell_slot, p.cells, d);
      const uint64_t num = (uint64_t)cell * p.ppc + (d - p.cell_slot[cell]);
      i = (uint32_t)num;
      ihi = (uint32_t)(num >> 32);
    } else {
      i = p.redo[r];
      cell = i / p.ppc;
      d = p.cell_slot[cell] + (i - cell * p.ppc);
    }
    float3 q = make_float3(0.f, 0.f, 0.f);
    unsigned out = 0;
    for (uint32_t t0 = 0; t0 < kRedraws && !out; t0 += 32) {
      const uint32_t w = w0 + 3u * (t0 + lane), b = w >> 2, o = w & 3u;
      const uint4 x = philox_block(b, i, ihi, kPurposeInit, p.seed),
                  y = philox_block(b + 1u, i, ihi, kPurposeInit, p.seed);
      const uint32_t u[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
      auto uni = [&](uint32_t k) {
        uint32_t v = u[0];
#pragma unroll
        for (uint32_t m = 1; m < 8; m++)
          if (m == o + k) v = u[m];
        return ((float)(v >> 8) + 0.5f) * (1.0f / 16777216.0f);
      };
      q = fill_position(p, cell, uni(0), uni(1), uni(2));
      out = __ballot_sync(kFull, !inside_mesh(p.geom, q));
    }
    const int pick = out ? __ffs(out) - 1 : 31;  // none: the last redraw, unless a point is known
    if ((int)lane == pick) {
      if (!out && p.cell_point && p.cell_point[cell].w > 0.f) {
        const float4 c = p.cell_point[cell];
        q = make_float3(c.x, c.y, c.z);
      }
      p.out.x[d] = q.x; p.out.y[d] = q.y; p.out.z[d] = q.z;
    }
  }
}

template <bool WIDE>
__global__ void k_init_fill(const __grid_constant__ InitParams p) {
  const uint32_t total = WIDE ? p.n : p.cells * p.ppc;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    uint32_t i, ihi = 0, cell, d;
    if (WIDE) {
      d = t;
      cell = cell_of_slot(p.cell_slot, p.cells, d);
      const uint64_t num = (uint64_t)cell * p.ppc + (d - p.cell_slot[cell]);
      i = (uint32_t)num;
      ihi = (uint32_t)(num >> 32);
    } else {
      i = t;
      cell = i / p.ppc;
      const uint32_t k = i - cell * p.ppc, dst0 = p.cell_slot[cell];
      if (dst0 == kNone || k >= (p.cell_count ? p.cell_count[cell] : p.cell_slot[cell + 1] - dst0)) continue;
      d = dst0 + k;
    }
    PhiloxStream r;
    r.init(p.seed, i, ihi, kPurposeInit);
    float3 vel;
    if (p.kind == 0) {
      const float vv = p.vmp * sqrtf(-logf(r.uniform()));
      const float tetha = 2.0f * kPiF;
      vel.x = vv * sinf(r.uniform() * tetha) + p.stream.x;
      vel.y = vv * sinf(r.uniform() * tetha) + p.stream.y;
      vel.z = vv * sinf(r.uniform() * tetha) + p.stream.z;
    } else {
      float sd = (p.kind == 2 && (i & 1u)) ? p.vstd2 : p.vstd;
      float3 drift = p.stream;
      if (p.cell_state) {
        const float4 cs = p.cell_state[cell];
        drift = make_float3(cs.x, cs.y, cs.z);
        sd = cs.w;
        // a two-stream cell: a share of its particles from the free stream
        if (p.cell_mix && r.uniform() < p.cell_mix[cell]) {
          drift = p.stream;
          sd = p.vstd;
        }
      }
      const float r1 = r.uniform(), r2 = r.uniform(), r3 = r.uniform(), r4 = r.uniform();
      const float m1 = sd * sqrtf(-2.f * logf(r1)), m2 = sd * sqrtf(-2.f * logf(r3));
      float s1, c1, s2, c2;
      sincospif(2.0f * r2, &s1, &c1);
      sincospif(2.0f * r4, &s2, &c2);
      vel = make_float3(m1 * c1 + drift.x, m1 * s1 + drift.y, m2 * c2 + drift.z);
    }
    const float a = r.uniform(), b = r.uniform(), c = r.uniform();
    const float3 q = fill_position(p, cell, a, b, c);
    // a cell the mesh covers in part: a position inside the body is drawn
    // again (k_init_redraw)
    if (p.reject_inside && inside_mesh(p.geom, q)) p.redo[atomicAdd(p.n_redo, 1u)] = t;
    p.out.x[d] = q.x; p.out.y[d] = q.y; p.out.z[d] = q.z;
    p.out.u[d] = vel.x; p.out.v[d] = vel.y; p.out.w[d] = vel.z;
  }
}


// --------------------------------------------------------------- inflow ----

// Plan: number of particles the face injects this step (carrying the
// fractional remainder), reserved after the particles already in the array.
__device__ __forceinline__ void inject_plan_body(const InjectParams& p, uint32_t* plan, const uint32_t vb) {
  if (threadIdx.x != 0 || vb != 0) return;
  const float want = fmaf(__fmul_rn(p.inflow.number_flux, p.inflow.area), p.dt, *p.remainder);
  uint32_t k = want > 0.f ? (uint32_t)want : 0u;
  const uint32_t have = p.meta->n_alive + p.meta->n_pending;
  if (have + k > p.capacity) {
    atomicOr(&p.meta->error, kErrCapacity);
    k = have < p.capacity ? p.capacity - have : 0u;
  }
  *p.remainder = want - (float)k;
  plan[0] = have;  // first slot
  plan[1] = k;
  p.meta->n_pending += k;
  p.meta->injected += k;
}

__global__ void k_inject_plan(const __grid_constant__ InjectParams p, uint32_t* plan) {
  chained_entry();
  inject_plan_body(p, plan, blockIdx.x);
}
__global__ void k_inject_plan_b(const __grid_constant__ BatchOf<InjectParams> bv) {
  chained_entry();
  uint32_t vb, vg;
  const InjectParams& p = bv.locate(vb, vg);
  inject_plan_body(p, p.plan, vb);
}

// Inward normal speed of the drifting Maxwellian weighted by flux,
// f(z) ~ z exp(-(z - s)^2) for z = v_n / c_mp > 0, by rejection from the
// envelope (|y| + max(s,0)) exp(-y^2), y = z - s.  Rounding steps explicit
// (no contraction).
__device__ __forceinline__ float sample_flux_normal(float s, PhiloxStream& r) {
  const float sp = fmaxf(s, 0.f);
  const float w_abs = 1.f / fmaf(sp, 1.7724539f, 1.f);
  for (int it = 0; it < 64; it++) {
    float y;
    if (r.uniform() < w_abs) {
      y = sqrtf(-logf(r.uniform()));
      if (r.uniform() < 0.5f) y = -y;
    } else {
      const float a = r.uniform(), b = r.uniform();
      y = __fmul_rn(sqrtf(-logf(a)), cospif(2.0f * b));  // N(0, 1/2)
    }
    const float z = s + y;
    if (z <= 0.f) continue;
    if (r.uniform() * (fabsf(y) + sp) <= z) return z;
  }
  return fmaxf(s, 1e-3f);
}

__device__ __forceinline__ float& comp(float3& a, int k) { return k == 0 ? a.x : (k == 1 ? a.y : a.z); }
__device__ __forceinline__ float compc(const float3& a, int k) { return k == 0 ? a.x : (k == 1 ? a.y : a.z); }

__device__ __forceinline__ void inject_fill_body(const InjectParams& p, const uint32_t* plan,
                                                 const uint32_t vb, const uint32_t vg) {
  extern __shared__ uint32_t s_tile[];
  const uint32_t step = p.meta->step;
  for (uint32_t t = threadIdx.x; t < p.n_scan_tiles; t += blockDim.x) s_tile[t] = 0;
  __syncthreads();
  const uint32_t first = plan[0], k = plan[1];
  const int face = p.inflow.face;
  const int ax = face >> 1;
  const float sign = (face & 1) ? -1.f : 1.f;  // inward normal along +axis for the low face
  const GridGeom& g = p.grid;
  const float cmp = p.inflow.vstd * 1.41421356f;
  const float s = sign * compc(p.inflow.stream, ax) / cmp;
  for (uint32_t base = vb * blockDim.x; base < k; base += vg * blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    const bool active = i < k;
    bool live = false;
    uint32_t key = kDeadKey;
    if (active) {
      float3 pos = make_float3(0, 0, 0), vel = pos;
      PhiloxStream r;
      r.init(p.seed, i, step, kPurposeInject + (uint32_t)face);
      const float vn = __fmul_rn(__fmul_rn(sample_flux_normal(s, r), cmp), sign);
      const float a1 = r.uniform(), a2 = r.uniform();
      const float rad = __fmul_rn(p.inflow.vstd, sqrtf(__fmul_rn(-2.f, logf(a1))));
      float sn, cs;
      sincospif(2.0f * a2, &sn, &cs);
      const int a_t1 = (ax + 1) % 3, a_t2 = (ax + 2) % 3;
      comp(vel, ax) = vn;
      comp(vel, a_t1) = fmaf(rad, cs, compc(p.inflow.stream, a_t1));
      comp(vel, a_t2) = fmaf(rad, sn, compc(p.inflow.stream, a_t2));
      comp(pos, ax) = (face & 1) ? compc(g.gmax, ax) : compc(g.gmin, ax);
      comp(pos, a_t1) = fmaf(r.uniform(), compc(g.gmax, a_t1) - compc(g.gmin, a_t1), compc(g.gmin, a_t1));
      comp(pos, a_t2) = fmaf(r.uniform(), compc(g.gmax, a_t2) - compc(g.gmin, a_t2), compc(g.gmin, a_t2));
      const float frac = __fmul_rn(r.uniform(), p.dt);
      pos.x = fmaf(vel.x, frac, pos.x); pos.y = fmaf(vel.y, frac, pos.y); pos.z = fmaf(vel.z, frac, pos.z);
      live = !(pos.x < g.gmin.x || pos.x > g.gmax.x || pos.y < g.gmin.y || pos.y > g.gmax.y ||
               pos.z < g.gmin.z || pos.z > g.gmax.z);
      if (live) key = cell_id3d(g, pos.x, pos.y, pos.z);
      const uint32_t d = first + i;
      p.st.x[d] = pos.x; p.st.y[d] = pos.y; p.st.z[d] = pos.z;
      p.st.u[d] = vel.x; p.st.v[d] = vel.y; p.st.w[d] = vel.z;
      p.keys[d] = key;
    }
    if (active && live) warp_count_key(p.count, key, s_tile);
  }
  __syncthreads();
  flush_tile_hist(s_tile, p.tile_sum, p.n_scan_tiles);
}

__global__ void k_inject_fill(const __grid_constant__ InjectParams p, const uint32_t* plan) {
  chained_entry();
  inject_fill_body(p, plan, blockIdx.x, gridDim.x);
}
__global__ void k_inject_fill_b(const __grid_constant__ BatchOf<InjectParams> bv) {
  chained_entry();
  uint32_t vb, vg;
  const InjectParams& p = bv.locate(vb, vg);
  inject_fill_body(p, p.plan, vb, vg);
}

}  // namespace

int num_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
}

uint32_t grid_for(uint64_t work, int threads, int per_sm) {
  uint64_t need = (work + threads - 1) / threads;
  const uint64_t cap = (uint64_t)num_sms() * per_sm;
  if (need < 1) need = 1;
  return (uint32_t)(need < cap ? need : cap);
}

cudaError_t launch_index(const GridGeom& g, uint32_t cells, const float* x, const float* y,
                         const float* z, uint32_t n, uint32_t* keys, uint32_t* count,
                         uint32_t* tile_sum, uint32_t n_scan_tiles, int face_mode,
                         cudaStream_t stream) {
  (void)cells;
  const uint32_t grid = grid_for(n, 256, 8);
  k_index<<<grid, 256, n_scan_tiles * 4, stream>>>(g, x, y, z, n, keys, count, tile_sum,
                                                   n_scan_tiles, face_mode);
  return cudaGetLastError();
}

cudaError_t launch_scan(uint32_t* count, uint32_t* cursor, uint32_t* start, uint32_t cells,
                        const uint32_t* tile_sum, uint32_t n_scan_tiles, Meta* meta, int bump_step,
                        cudaStream_t stream, int carveout) {
  return launch_chained(k_scan, n_scan_tiles, 256, 0, stream, Chain(true, carveout), count, cursor, start, cells, tile_sum, meta,
                        bump_step);
}

cudaError_t launch_scatter(bool with_state, const SoA& src, SoA dst, const uint32_t* keys,
                           const uint32_t* start,
                           uint32_t* cursor, uint32_t* orig, uint32_t cells, uint32_t* tile_sum,
                           uint32_t n_scan_tiles, Meta* meta, uint32_t capacity,
                           cudaStream_t stream, int carveout) {
  const uint32_t grid = (uint32_t)num_sms() * 4;
  return launch_chained(with_state ? k_scatter<true> : k_scatter<false>, grid, 256, 0, stream, Chain(true, carveout), src, dst, keys,
                        start, cursor, orig, cells, tile_sum, n_scan_tiles, meta, capacity);
}

cudaError_t launch_move(const StepParams& p, uint32_t n, uint32_t step, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  if (p.has_geom) k_move<true, 1><<<grid_for(n, 256, 8), 256, 0, stream>>>(p, n, step);
  else if (n < kMoveByFour) k_move<false, 1><<<grid_for(n, 256, 8), 256, 0, stream>>>(p, n, step);
  else k_move<false, 4><<<grid_for(n, 1024, 8), 256, 0, stream>>>(p, n, step);
  return cudaGetLastError();
}

cudaError_t launch_cell_ids(const GridGeom& g, const float* x, const float* y, const float* z,
                            uint32_t n, uint32_t* keys, uint32_t* idx, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  k_cell_ids<<<grid_for(n, 1024, 8), 256, 0, stream>>>(g, x, y, z, n, keys, idx);
  return cudaGetLastError();
}

cudaError_t launch_sort(uint32_t* keys, uint32_t* vals, uint32_t n, uint32_t nkeys, uint32_t* count,
                        uint32_t* start, uint32_t* tile_sum, uint32_t* scratch, Meta* meta, cudaStream_t stream) {
  const uint32_t tiles = (nkeys + kScanTile - 1) / kScanTile;
  if (n) {
    k_count_keys<<<grid_for(n, 1024, 8), 256, tiles * 4, stream>>>(keys, n, nkeys, count, tile_sum, tiles);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  cudaError_t e = launch_scan(count, nullptr, start, nkeys, tile_sum, tiles, meta, 0, stream);
  if (e != cudaSuccess || !n) return e;
  // keys per CTA of the fixup: 64 where that makes eight tiles per SM, down to
  // 8 on small key ranges
  uint32_t kt = 64;
  while (kt > 8 && nkeys / kt < (uint32_t)num_sms() * 8u) kt >>= 1;
  // nor more than a chunk of entries on the average (10,000 entries in 8 keys: 846
  // us on one CTA, 77 on eight)
  while (kt > 1 && (uint64_t)n * kt > (uint64_t)nkeys * kFixupCap) kt >>= 1;
  const uint32_t ft = (nkeys + kt - 1) / kt, fgrid = std::min(ft, (uint32_t)num_sms() * 16u);
  const uint32_t sgrid = grid_for(n, 1024, 8);
  if (((uintptr_t)scratch & 7u) == 0) {
    const ScatterOut<true> o{scratch, nullptr};
    k_scatter_kv<true><<<sgrid, 256, 0, stream>>>(keys, vals, start, count, n, nkeys, o);
    k_segment_fixup<true><<<fgrid, kFixupThreads, 0, stream>>>(start, nkeys, kt, o, keys, vals);
  } else {
    const ScatterOut<false> o{scratch, scratch + n};
    k_scatter_kv<false><<<sgrid, 256, 0, stream>>>(keys, vals, start, count, n, nkeys, o);
    k_segment_fixup<false><<<fgrid, kFixupThreads, 0, stream>>>(start, nkeys, kt, o, keys, vals);
  }
  return cudaGetLastError();
}

cudaError_t launch_collide_cells(const StepParams& p, cudaStream_t stream) {
  if (p.cells == 0) return cudaSuccess;
  // 32 cells per warp where that makes a wave of warps, fewer on small grids
  uint32_t ct = 32;
  while (ct > 1 && p.cells / ct < (uint32_t)num_sms() * 16u) ct >>= 1;
  const uint32_t tiles = (p.cells + ct - 1) / ct;
  k_collide_cells<<<grid_for(tiles, kCollideWarps, 8), 32 * kCollideWarps, 0, stream>>>(p, ct);
  return cudaGetLastError();
}

cudaError_t launch_bounds_reorder(const uint32_t* keys, const uint32_t* idx, uint32_t n,
                                  uint32_t ncells, uint32_t* cse, const float* const src[6],
                                  float* const dst[6], cudaStream_t stream) {
  SoA s{const_cast<float*>(src ? src[0] : nullptr), const_cast<float*>(src ? src[1] : nullptr),
        const_cast<float*>(src ? src[2] : nullptr), const_cast<float*>(src ? src[3] : nullptr),
        const_cast<float*>(src ? src[4] : nullptr), const_cast<float*>(src ? src[5] : nullptr)};
  SoA d{dst ? dst[0] : nullptr, dst ? dst[1] : nullptr, dst ? dst[2] : nullptr,
        dst ? dst[3] : nullptr, dst ? dst[4] : nullptr, dst ? dst[5] : nullptr};
  if (src && dst)
    k_bounds_reorder<true><<<grid_for(n, 256, 8), 256, 0, stream>>>(keys, idx, n, ncells, (uint2*)cse, s, d);
  else
    k_bounds_reorder<false><<<grid_for(n, 1024, 8), 256, 0, stream>>>(keys, idx, n, ncells, (uint2*)cse, s, d);
  return cudaGetLastError();
}

cudaError_t launch_cell_fields(const double* acc, uint32_t cells, double fnum, double cell_volume,
                               uint32_t ns, double mass, int fields, double* out, cudaStream_t stream) {
  k_cell_fields<<<grid_for(cells, 256, 8), 256, 0, stream>>>(acc, cells, fnum, cell_volume, ns, mass,
                                                            fields, out);
  return cudaGetLastError();
}

cudaError_t launch_sample_cells(const float* u, const float* v, const float* w,
                                const uint32_t* start, uint32_t cells, double* acc,
                                size_t fstride, size_t cstride, cudaStream_t stream) {
  const uint32_t threads = cells < (uint32_t)num_sms() * 2048u ? 64u : 256u;  // small: a few thousand cells reach every SM
  const uint32_t grid = (cells + threads - 1u) / threads;
  if (grid) k_sample_cells<<<grid, threads, 0, stream>>>(u, v, w, start, cells, acc, fstride, cstride);
  return cudaGetLastError();
}

// One warp per cell, two of the 4x4x4 sub-cell centres per lane.
__global__ void k_outside_fraction(const GridGeom grid, const __grid_constant__ GeomView geom, uint32_t cells,
                                   float* frac, float4* point) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t cell = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); cell < cells;
       cell += warps) {
    const uint32_t cx = cell % grid.dim.x, cy = (cell / grid.dim.x) % grid.dim.y,
                   cz = cell / (grid.dim.x * grid.dim.y);
    const float3 lo = make_float3(grid.gmin.x + cx * grid.cell.x, grid.gmin.y + cy * grid.cell.y,
                                  grid.gmin.z + cz * grid.cell.z);
    const bool near = lo.x <= geom.grid.gmax.x && lo.x + grid.cell.x >= geom.grid.gmin.x &&
                      lo.y <= geom.grid.gmax.y && lo.y + grid.cell.y >= geom.grid.gmin.y &&
                      lo.z <= geom.grid.gmax.z && lo.z + grid.cell.z >= geom.grid.gmin.z;
    if (!near) {
      if (lane == 0) {
        frac[cell] = 1.f;
        point[cell] = make_float4(lo.x + 0.5f * grid.cell.x, lo.y + 0.5f * grid.cell.y,
                                  lo.z + 0.5f * grid.cell.z, 1.f);
      }
      continue;
    }
    bool out[2];
    float3 q[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t sidx = lane * 2u + (uint32_t)h;
      q[h] = make_float3(lo.x + ((sidx & 3u) + 0.5f) * 0.25f * grid.cell.x,
                         lo.y + (((sidx >> 2) & 3u) + 0.5f) * 0.25f * grid.cell.y,
                         lo.z + ((sidx >> 4) + 0.5f) * 0.25f * grid.cell.z);
      out[h] = !inside_mesh(geom, q[h]);
    }
    const unsigned m0 = __ballot_sync(0xffffffffu, out[0]);
    const unsigned m1 = __ballot_sync(0xffffffffu, out[1]);
    const uint32_t n_out = __popc(m0) + __popc(m1);
    const int src = m0 ? __ffs(m0) - 1 : (m1 ? __ffs(m1) - 1 : 0);
    const int which = m0 ? 0 : 1;
    const float px = __shfl_sync(0xffffffffu, which ? q[1].x : q[0].x, src);
    const float py = __shfl_sync(0xffffffffu, which ? q[1].y : q[0].y, src);
    const float pz = __shfl_sync(0xffffffffu, which ? q[1].z : q[0].z, src);
    if (lane == 0) {
      frac[cell] = (float)n_out / 64.f;
      point[cell] = make_float4(px, py, pz, n_out ? 1.f : 0.f);
    }
  }
}

// Distance from q to the triangle (a, b, c): inside the prism over the
// triangle the distance to its plane, otherwise the nearest of its edges
// (closest point of each edge segment).
__device__ float point_triangle_distance(float3 q, float3 a, float3 b, float3 c) {
  const float3 ab = make_float3(b.x - a.x, b.y - a.y, b.z - a.z);
  const float3 bc = make_float3(c.x - b.x, c.y - b.y, c.z - b.z);
  const float3 ca = make_float3(a.x - c.x, a.y - c.y, a.z - c.z);
  const float3 n = make_float3(ab.y * (-ca.z) - ab.z * (-ca.y), ab.z * (-ca.x) - ab.x * (-ca.z),
                               ab.x * (-ca.y) - ab.y * (-ca.x));
  const float nn = n.x * n.x + n.y * n.y + n.z * n.z;
  auto side = [&](float3 e, float3 p0) {
    const float3 r = make_float3(q.x - p0.x, q.y - p0.y, q.z - p0.z);
    const float3 x = make_float3(e.y * r.z - e.z * r.y, e.z * r.x - e.x * r.z, e.x * r.y - e.y * r.x);
    return x.x * n.x + x.y * n.y + x.z * n.z;
  };
  if (nn > 0.f && side(ab, a) >= 0.f && side(bc, b) >= 0.f && side(ca, c) >= 0.f) {
    const float h = (q.x - a.x) * n.x + (q.y - a.y) * n.y + (q.z - a.z) * n.z;
    return fabsf(h) * rsqrtf(nn);
  }
  auto seg = [&](float3 p0, float3 e) {
    const float ee = e.x * e.x + e.y * e.y + e.z * e.z;
    float t = ee > 0.f ? ((q.x - p0.x) * e.x + (q.y - p0.y) * e.y + (q.z - p0.z) * e.z) / ee : 0.f;
    t = fminf(fmaxf(t, 0.f), 1.f);
    const float3 d = make_float3(q.x - (p0.x + t * e.x), q.y - (p0.y + t * e.y), q.z - (p0.z + t * e.z));
    return sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
  };
  return fminf(seg(a, ab), fminf(seg(b, bc), seg(c, ca)));
}

// Clearance table on the refined grid `fine` (fac x fac x fac cells per cell
// of the triangle grid).  cdist holds each triangle-grid cell's Chebyshev
// distance in cells to the nearest cell holding triangles (-1: none at all).
// Cells at distance >= 2 keep the cell-count bound (cdist - 1) * cmin; the
// others take the exact distance from their centre to the triangles of the
// 27 triangle-grid cells around, less half their diagonal, capped by cmin
// (triangles farther out are at least one triangle-grid cell away).  All
// bounds are scaled by 0.999 to stay below the true distance.
__global__ void k_fine_clearance(const __grid_constant__ GeomView g, GridGeom fine, uint32_t fac,
                                 const int* __restrict__ cdist, float cmin, float* out) {
  const uint32_t n = fine.dim.x * fine.dim.y * fine.dim.z;
  const float hd = 0.5f * sqrtf(fine.cell.x * fine.cell.x + fine.cell.y * fine.cell.y +
                                fine.cell.z * fine.cell.z);
  for (uint32_t f = blockIdx.x * blockDim.x + threadIdx.x; f < n; f += gridDim.x * blockDim.x) {
    const uint32_t fx = f % fine.dim.x, fy = (f / fine.dim.x) % fine.dim.y,
                   fz = f / (fine.dim.x * fine.dim.y);
    const int cx = (int)(fx / fac), cy = (int)(fy / fac), cz = (int)(fz / fac);
    const int D = cdist[((uint32_t)cz * g.grid.dim.y + (uint32_t)cy) * g.grid.dim.x + (uint32_t)cx];
    float c;
    if (D < 0) {
      c = 3.0e38f;
    } else if (D >= 2) {
      c = 0.999f * (float)(D - 1) * cmin;
    } else {
      const float3 q = make_float3(fine.gmin.x + ((float)fx + 0.5f) * fine.cell.x,
                                   fine.gmin.y + ((float)fy + 0.5f) * fine.cell.y,
                                   fine.gmin.z + ((float)fz + 0.5f) * fine.cell.z);
      float best = 3.0e38f;
      for (int dz = -1; dz <= 1; dz++)
        for (int dy = -1; dy <= 1; dy++)
          for (int dx = -1; dx <= 1; dx++) {
            const int x = cx + dx, y = cy + dy, z = cz + dz;
            if (x < 0 || y < 0 || z < 0 || x >= (int)g.grid.dim.x || y >= (int)g.grid.dim.y ||
                z >= (int)g.grid.dim.z)
              continue;
            const uint2 se = g.start_end[((uint32_t)z * g.grid.dim.y + (uint32_t)y) * g.grid.dim.x + (uint32_t)x];
            for (uint32_t i = se.x; i < se.y; i++) {
              const float4 A = g.tri[kTriStride * (size_t)i], B = g.tri[kTriStride * (size_t)i + 1],
                           C = g.tri[kTriStride * (size_t)i + 2];
              best = fminf(best, point_triangle_distance(q, make_float3(A.x, A.y, A.z),
                                                         make_float3(B.x, B.y, B.z),
                                                         make_float3(C.x, C.y, C.z)));
            }
          }
      c = 0.999f * fmaxf(0.f, fminf(best - hd, cmin));
    }
    out[f] = c;
  }
}

__device__ __forceinline__ double axis_of(const double3& v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

// The slope bound of a triangle U that rises above T's plane, seen from T:
// the least k such that height(x) - tol <= k * sigma(x) at U's three
// vertices (so on all of U, both sides being linear) for one in-plane
// half-plane sigma <= 0 that holds T (an edge's outer side, or a direction
// of a vertex's normal cone: 3 edges and 7 directions per vertex).  As
// sigma(x) <= dist(x, T), every point of U then lies at most tol + k * dist
// above T's plane.  Infinity where no half-plane gives a bound.
__device__ double rise_slope(const double3 V[3], const double3 un[3], double3 n, const double3 W[3], double tol) {
  double best = 1e300;
  for (int c = 0; c < 24; c++) {
    // c < 3: edge c's outer normal (edge c runs from V[c] to V[c+1]); then 7
    // directions between the outer normals of the two edges at each vertex
    double3 u, P;
    if (c < 3) {
      u = un[c];
      P = V[c];
    } else {
      const int k = (c - 3) / 7, m = (c - 3) % 7;  // vertex k: edges k - 1 and k
      const double t = (m + 1) / 8.0;
      const double3 a = un[(k + 2) % 3], b = un[k];
      u = make_double3((1 - t) * a.x + t * b.x, (1 - t) * a.y + t * b.y, (1 - t) * a.z + t * b.z);
      const double l = sqrt(u.x * u.x + u.y * u.y + u.z * u.z);
      u = make_double3(u.x / l, u.y / l, u.z / l);
      P = V[k];
    }
    double lo = 0.0, hi = 1e300;
    bool ok = true;
    for (int q = 0; q < 3 && ok; q++) {
      const double3 d = make_double3(W[q].x - V[0].x, W[q].y - V[0].y, W[q].z - V[0].z);
      const double a = n.x * d.x + n.y * d.y + n.z * d.z - tol;
      const double b = u.x * (W[q].x - P.x) + u.y * (W[q].y - P.y) + u.z * (W[q].z - P.z);
      if (b > 1e-12) lo = fmax(lo, a / b);
      else if (b < -1e-12) hi = a > 0.0 ? -1.0 : fmin(hi, a / b);
      else ok = a <= 0.0;
    }
    if (ok && lo <= hi) best = fmin(best, lo);
  }
  return best;
}

// Reach of every bin entry's triangle T, for a particle that leaves T
// outward (re-emitted or reflected; it starts 1 um above T along T's normal):
// (r, k) such that a path shorter than r whose direction makes more than k
// with T's normal (the sine of its elevation) crosses no listed triangle.
// Every triangle U within rmax of T is listed in a cell that T's box, grown
// by rmax and one more cell, overlaps.  A U with no vertex more than tol
// above T's plane cannot be crossed from above it.  A U that rises above
// the plane either caps r by the distance between the two boxes (a lower
// bound of the distance between the triangles), or, when its slope bound
// (rise_slope) is below 1/2, raises k to that bound: a path of elevation
// above k climbs faster than U rises with the distance from T.  r is lowered
// by `slack` (the set-off and the rounding of the hit point) and by 0.1 %;
// (0, 2) where nothing is left.
__global__ void k_entry_reach(const __grid_constant__ GeomView g, uint32_t entries, float rmax, float tol,
                              float slack, float2* __restrict__ out) {
  const float grow = rmax + fmaxf(g.grid.cell.x, fmaxf(g.grid.cell.y, g.grid.cell.z));
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < entries; e += gridDim.x * blockDim.x) {
    const float4 A = g.tri[kTriStride * (size_t)e], B = g.tri[kTriStride * (size_t)e + 1],
                 C = g.tri[kTriStride * (size_t)e + 2];
    const float4 P = g.plane[e];
    const double3 V[3] = {make_double3(A.x, A.y, A.z), make_double3(B.x, B.y, B.z), make_double3(C.x, C.y, C.z)};
    // T's unit normal from its vertices in FP64 (the stored plane's orientation)
    const double3 e1 = make_double3(V[1].x - V[0].x, V[1].y - V[0].y, V[1].z - V[0].z);
    const double3 e2 = make_double3(V[2].x - V[0].x, V[2].y - V[0].y, V[2].z - V[0].z);
    double3 n = make_double3(e1.y * e2.z - e1.z * e2.y, e1.z * e2.x - e1.x * e2.z, e1.x * e2.y - e1.y * e2.x);
    const double nl = sqrt(n.x * n.x + n.y * n.y + n.z * n.z);
    float2 res = make_float2(0.f, 2.f);
    if (nl > 0.0) {
      n = make_double3(n.x / nl, n.y / nl, n.z / nl);
    }
    // the normal the wall response uses must agree with the vertices' one
    if (nl > 0.0 && n.x * P.x + n.y * P.y + n.z * P.z > 0.9999) {
      // in-plane outer normals of the edges V[c] -> V[c+1]
      double3 un[3];
      for (int c = 0; c < 3; c++) {
        const double3 a = V[c], b = V[(c + 1) % 3];
        const double3 d = make_double3(b.x - a.x, b.y - a.y, b.z - a.z);
        double3 u = make_double3(d.y * n.z - d.z * n.y, d.z * n.x - d.x * n.z, d.x * n.y - d.y * n.x);
        const double l = sqrt(u.x * u.x + u.y * u.y + u.z * u.z);
        u = make_double3(u.x / l, u.y / l, u.z / l);
        const double3 o = V[(c + 2) % 3];
        if (u.x * (o.x - a.x) + u.y * (o.y - a.y) + u.z * (o.z - a.z) > 0.0) u = make_double3(-u.x, -u.y, -u.z);
        un[c] = u;
      }
      const float lo[3] = {fminf(A.x, fminf(B.x, C.x)), fminf(A.y, fminf(B.y, C.y)), fminf(A.z, fminf(B.z, C.z))};
      const float hi[3] = {fmaxf(A.x, fmaxf(B.x, C.x)), fmaxf(A.y, fmaxf(B.y, C.y)), fmaxf(A.z, fmaxf(B.z, C.z))};
      const float gmn[3] = {g.grid.gmin.x, g.grid.gmin.y, g.grid.gmin.z};
      const float cs[3] = {g.grid.cell.x, g.grid.cell.y, g.grid.cell.z};
      const int dim[3] = {(int)g.grid.dim.x, (int)g.grid.dim.y, (int)g.grid.dim.z};
      int c0[3], c1[3];
      for (int k = 0; k < 3; k++) {
        c0[k] = max(0, (int)floorf((lo[k] - grow - gmn[k]) / cs[k]));
        c1[k] = min(dim[k] - 1, (int)floorf((hi[k] + grow - gmn[k]) / cs[k]));
      }
      double best = rmax, slope = 0.0;
      for (int z = c0[2]; z <= c1[2]; z++)
        for (int y = c0[1]; y <= c1[1]; y++)
          for (int x = c0[0]; x <= c1[0]; x++) {
            const uint2 se = g.start_end[((uint32_t)z * g.grid.dim.y + (uint32_t)y) * g.grid.dim.x + (uint32_t)x];
            if (se.x == kNone) continue;
            for (uint32_t j = se.x; j < se.y; j++) {
              double3 W[3];
              for (int k = 0; k < 3; k++) {
                const float4 q = g.tri[kTriStride * (size_t)j + k];
                W[k] = make_double3(q.x, q.y, q.z);
              }
              double up = -1.0;
              for (int k = 0; k < 3; k++)
                up = fmax(up, n.x * (W[k].x - V[0].x) + n.y * (W[k].y - V[0].y) + n.z * (W[k].z - V[0].z));
              if (up <= tol) continue;
              const double k_rise = rise_slope(V, un, n, W, tol);
              if (k_rise < 0.5) {
                slope = fmax(slope, k_rise);
                continue;
              }
              // no usable slope: the distance between the two boxes
              double d2 = 0.0;
              for (int k = 0; k < 3; k++) {
                const double w0 = axis_of(W[0], k), w1 = axis_of(W[1], k), w2 = axis_of(W[2], k);
                const double wl = fmin(w0, fmin(w1, w2)), wh = fmax(w0, fmax(w1, w2));
                const double gap = fmax(0.0, fmax(wl - hi[k], (double)lo[k] - wh));
                d2 += gap * gap;
              }
              best = fmin(best, sqrt(d2));
            }
          }
      const float r = fmaxf(0.f, 0.999f * (float)best - slack);
      if (r > 0.f) res = make_float2(r, __double2float_ru(slope));
    }
    out[e] = res;
  }
}

// The slab of every grid cell (GeomView::slab): n the normalised sum of the
// cell's triangle normals, [lo, hi] the range of n . v over every vertex of
// every listed triangle (FP64), widened by a margin; m = n / h, e = c / h
// with c the middle and h the half width.  Cells whose normals disagree
// (the sum shorter than half the count) pass every path.
__global__ void k_cell_slab(const __grid_constant__ GeomView g, uint32_t cells, float4* __restrict__ out) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < cells; c += gridDim.x * blockDim.x) {
    const uint2 se = g.start_end[c];
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    if (se.x != kNone && se.y > se.x) {
      double nx = 0.0, ny = 0.0, nz = 0.0;
      for (uint32_t i = se.x; i < se.y; i++) {
        const float4 P = g.plane[i];
        nx += P.x; ny += P.y; nz += P.z;
      }
      const double l = sqrt(nx * nx + ny * ny + nz * nz);
      if (l >= 0.5 * (double)(se.y - se.x)) {
        nx /= l; ny /= l; nz /= l;
        double lo = 1e300, hi = -1e300, mag = 0.0;
        for (uint32_t i = se.x; i < se.y; i++)
          for (int k = 0; k < 3; k++) {
            const float4 v = g.tri[kTriStride * (size_t)i + k];
            const double t = nx * v.x + ny * v.y + nz * v.z;
            lo = fmin(lo, t);
            hi = fmax(hi, t);
            mag = fmax(mag, fabs((double)v.x) + fabs((double)v.y) + fabs((double)v.z));
          }
        const double cmid = 0.5 * (lo + hi);
        const double h = 0.5 * (hi - lo) + 1e-6 + 1e-6 * mag;
        r = make_float4((float)(nx / h), (float)(ny / h), (float)(nz / h), (float)(cmid / h));
      }
    }
    out[c] = r;
  }
}

cudaError_t launch_cell_slab(const GeomView& g, uint32_t cells, float4* out, cudaStream_t stream) {
  if (cells == 0) return cudaSuccess;
  k_cell_slab<<<grid_for(cells, 128, 8), 128, 0, stream>>>(g, cells, out);
  return cudaGetLastError();
}

__global__ void k_clearance_at(const __grid_constant__ GeomView g, const float* __restrict__ xyz,
                               uint32_t n, float* __restrict__ out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float3 q = make_float3(xyz[3 * (size_t)i], xyz[3 * (size_t)i + 1], xyz[3 * (size_t)i + 2]);
    const uint32_t c = coll_cell_id(g.cgrid, q);
    out[i] = c == kNone ? -1.f : g.clear[c];
  }
}

cudaError_t launch_clearance_at(const GeomView& g, const float* xyz, uint32_t n, float* out,
                                cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  k_clearance_at<<<grid_for(n, 256, 8), 256, 0, stream>>>(g, xyz, n, out);
  return cudaGetLastError();
}

cudaError_t launch_entry_reach(const GeomView& g, uint32_t entries, float rmax, float tol, float slack,
                               float2* out, cudaStream_t stream) {
  if (entries == 0) return cudaSuccess;
  k_entry_reach<<<grid_for(entries, 128, 8), 128, 0, stream>>>(g, entries, rmax, tol, slack, out);
  return cudaGetLastError();
}

cudaError_t launch_fine_clearance(const GeomView& g, const GridGeom& fine, uint32_t fac,
                                  const int* cdist, float cmin, float* out, cudaStream_t stream) {
  const uint32_t n = fine.dim.x * fine.dim.y * fine.dim.z;
  k_fine_clearance<<<grid_for(n, 256, 8), 256, 0, stream>>>(g, fine, fac, cdist, cmin, out);
  return cudaGetLastError();
}

cudaError_t launch_outside_fraction(const GridGeom& grid, const GeomView& geom, uint32_t cells,
                                    float* frac, float4* point, cudaStream_t stream) {
  const uint32_t blocks = (uint32_t)std::min<uint64_t>(((uint64_t)cells + 7) / 8, 8u * num_sms());
  k_outside_fraction<<<blocks, 256, 0, stream>>>(grid, geom, cells, frac, point);
  return cudaGetLastError();
}

cudaError_t launch_init_fill(const InitParams& p, cudaStream_t stream) {
  const uint64_t total = (uint64_t)p.cells * p.ppc;
  const bool wide = total > kFillNumbers;
  if (wide && p.cell_count) return cudaErrorInvalidValue;
  const uint32_t grid = grid_for(wide ? p.n : total, 256, 8);
  if (p.reject_inside) {
    const cudaError_t e = cudaMemsetAsync(p.n_redo, 0, sizeof(uint32_t), stream);
    if (e != cudaSuccess) return e;
  }
  if (wide) k_init_fill<true><<<grid, 256, 0, stream>>>(p);
  else k_init_fill<false><<<grid, 256, 0, stream>>>(p);
  if (p.reject_inside && wide) k_init_redraw<true><<<(uint32_t)num_sms() * 4u, 256, 0, stream>>>(p);
  else if (p.reject_inside) k_init_redraw<false><<<(uint32_t)num_sms() * 4u, 256, 0, stream>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_scan_b(const BatchOf<SortArgs>& bv, uint32_t blocks, cudaStream_t stream) {
  return blocks ? launch_chained(k_scan_b, blocks, 256, 0, stream, false, bv) : cudaSuccess;
}

cudaError_t launch_scatter_b(const BatchOf<SortArgs>& bv, uint32_t blocks, cudaStream_t stream) {
  return blocks ? launch_chained(k_scatter_b, blocks, 256, 0, stream, false, bv) : cudaSuccess;
}

cudaError_t launch_inject_b(const BatchOf<InjectParams>& plan, uint32_t plan_blocks,
                            const BatchOf<InjectParams>& fill, uint32_t fill_blocks, size_t fill_smem,
                            cudaStream_t stream) {
  cudaError_t e = cudaSuccess;
  if (plan_blocks) e = launch_chained(k_inject_plan_b, plan_blocks, 32, 0, stream, false, plan);
  if (!e && fill_blocks) e = launch_chained(k_inject_fill_b, fill_blocks, 256, fill_smem, stream, false, fill);
  return e;
}

cudaError_t launch_inject(const InjectParams& p, cudaStream_t stream, int carveout) {
  cudaError_t e = launch_chained(k_inject_plan, 1, 32, 0, stream, Chain(true, carveout), p, p.plan);
  const uint32_t grid = (uint32_t)num_sms();
  if (!e) e = launch_chained(k_inject_fill, grid, 256, p.n_scan_tiles * 4, stream, Chain(true, carveout), p, p.plan);
  return e;
}

}  // namespace dsmcb
