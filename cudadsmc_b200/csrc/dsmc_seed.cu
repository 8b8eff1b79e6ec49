// Per-cell part of the fill from fields (dsmc_init_from_fields and its
// two-stream form): particle counts, Maxwellian states, free-stream shares and
// collision state of every cell, a thread per cell.
//
// Compiled without multiply-add contraction: every value is the one the plain
// sequence of IEEE operations gives.  On the host the bisection of 65,536
// cells (60 steps each, in doubles) took 13 ms of a fill's 15; here the whole
// kernel takes 12 us.
#include "dsmc_kernels.cuh"

namespace dsmcb {
namespace {

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Draw j (from 1) of the SplitMix64 sequence started at `seed`, in [0, 1).
__device__ __forceinline__ double unit_draw(uint64_t seed, uint64_t j) {
  return (double)(mix64(seed + j * 0x9E3779B97F4A7C15ull) >> 11) / 9007199254740992.0;
}

// Free-stream share alpha of a cell with mean velocity u and temperature T
// seen as a mixture of the free stream (U, T_inf) and a Maxwellian at the
// wall temperature T_w with drift u_b: the mixture's mean and energy match
// the cell's when
//   alpha e_inf + (1 - alpha) e_w + |u - alpha U|^2 / (1 - alpha) = 3kT/m + |u|^2
// (e = 3kT/m + |drift|^2 of a component), solved by bisection on
// [0, 0.98]; 0 where the cell is colder than the wall or no root lies there.
__device__ double two_stream_share(const double u[3], double T, const double U[3], double T_inf, double T_w,
                                   double kb_m) {
  const double e_inf = 3.0 * kb_m * T_inf + U[0] * U[0] + U[1] * U[1] + U[2] * U[2];
  const double e_w = 3.0 * kb_m * T_w;
  const double rhs = 3.0 * kb_m * T + u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
  auto f = [&](double a) {
    const double d0 = u[0] - a * U[0], d1 = u[1] - a * U[1], d2 = u[2] - a * U[2];
    return a * e_inf + (1.0 - a) * e_w + (d0 * d0 + d1 * d1 + d2 * d2) / (1.0 - a) - rhs;
  };
  double lo = 0.0, hi = 0.98;
  if (!(f(lo) < 0.0 && f(hi) > 0.0)) return 0.0;
  for (int it = 0; it < 60; it++) {
    const double mid = 0.5 * (lo + hi);
    if (f(mid) > 0.0) hi = mid;
    else lo = mid;
  }
  return 0.5 * (lo + hi);
}

constexpr int kThreads = 128;
static_assert(kScanTile % kThreads == 0, "a block lies in one scan tile");

__global__ void __launch_bounds__(kThreads) k_seed_cells(const SeedParams p) {
  __shared__ unsigned long long s_sum[kThreads / 32];
  __shared__ uint32_t s_max[kThreads / 32];
  const uint32_t cell = blockIdx.x * kThreads + threadIdx.x;
  uint32_t k = 0;
  if (cell < p.cells) {
    const float* f = p.fields + 5 * (size_t)cell;
    // n is averaged over the whole cell volume (as dsmc_read_fields gives
    // it), so a cell the body cuts receives its n V_c / F_N particles in the
    // part outside the body; a cell the body covers stays empty
    double expect = (isfinite(f[0]) && f[0] > 0.f && (!p.frac || p.frac[cell] > 0.f))
                        ? (double)f[0] * p.cell_volume / p.fnum : 0.0;
    // a cell that cannot be filled counts one more than there is room for, so
    // that the conversion holds and the total says so
    expect = fmin(expect, (double)p.capacity + 1.0);
    const double fl = floor(expect);
    k = (uint32_t)fl + (unit_draw(p.seed, 2 * (uint64_t)cell + 1) < expect - fl ? 1u : 0u);
    const float T = (isfinite(f[4]) && f[4] > 0.f) ? f[4] : p.temp;
    float4 st = make_float4(isfinite(f[1]) ? f[1] : 0.f, isfinite(f[2]) ? f[2] : 0.f, isfinite(f[3]) ? f[3] : 0.f,
                            sqrtf(p.kb_m * T));
    if (p.share) {
      // the share alpha from the free stream, the rest a Maxwellian whose
      // drift and temperature keep the cell's mean and energy (the wall
      // temperature itself at weight 1)
      const double u[3] = {st.x, st.y, st.z};
      const double U[3] = {p.stream[0], p.stream[1], p.stream[2]};
      const double a = p.weight * two_stream_share(u, T, U, p.temp, p.wall_temp, p.kb_m);
      p.share[cell] = (float)a;
      if (a > 0.0) {
        double ub[3], ub2 = 0.0, uu = 0.0, UU = 0.0;
        for (int q = 0; q < 3; q++) {
          ub[q] = (u[q] - a * U[q]) / (1.0 - a);
          ub2 += ub[q] * ub[q];
          uu += u[q] * u[q];
          UU += U[q] * U[q];
        }
        const double e = (3.0 * p.kb_m * T + uu - a * (3.0 * p.kb_m * p.temp + UU)) / (1.0 - a) - ub2;
        const double e3 = e / 3.0;
        st = make_float4((float)ub[0], (float)ub[1], (float)ub[2], (float)sqrt(e3 < 0.0 ? 0.0 : e3));
      }
    }
    p.state[cell] = st;
    // (sigma g)max scaled to the cell's temperature like the initial value
    // (InitSimulationProperties, kernels/dsmc_kernel.cu:329-331)
    const float Tm = T < p.temp ? p.temp : T;
    p.maxrem[cell] = make_float2(p.max_rel_vel * sqrtf(Tm / p.temp),
                                 (float)unit_draw(p.seed, 2 * (uint64_t)cell + 2));
    p.count[cell] = k;
  }
  // the total in 64 bits: no sum of counts may wrap round to one that fits
  unsigned long long sum = k;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const uint32_t mx = __reduce_max_sync(0xffffffffu, k);
  if ((threadIdx.x & 31u) == 0) {
    s_sum[threadIdx.x >> 5] = sum;
    s_max[threadIdx.x >> 5] = mx;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    uint32_t m = 0;
    for (int w = 0; w < kThreads / 32; w++) {
      t += s_sum[w];
      m = max(m, s_max[w]);
    }
    atomicAdd(&p.tile_sum[(blockIdx.x * kThreads) >> kScanShift], (uint32_t)t);
    atomicAdd(&p.totals->n, t);
    atomicMax(&p.totals->kmax, m);
  }
}

}  // namespace

cudaError_t launch_seed_cells(const SeedParams& p, cudaStream_t stream) {
  k_seed_cells<<<(p.cells + kThreads - 1) / kThreads, kThreads, 0, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace dsmcb
