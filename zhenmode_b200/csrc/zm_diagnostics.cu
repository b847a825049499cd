// Diagnostics of a state, outside the time step.
//
// k_diagnostics: the diagnostics closure of the reference factory
// (factory.py:752-760) on one column per thread: full density rho0 + rho'
// (physics/eos.py:13-18), hydrostatic pressure rho0 g eta (+ a surface load)
// plus the trapezoid integral of the wet-masked density anomaly
// (dynamics/pressure.py:32-42, 62-74), and the dual-face vertical velocity
// w = -Fz[k] wet (dynamics/transport.py:149-166), with Fz from k_fz.
//
// k_budget_partials / k_budget_final: the global heat, salt and volume
// snapshot of diagnostics/snapshot.py:67-128 (legacy node thickness), summed
// in float64 with compensation.  Each lane keeps a Neumaier sum over its
// elements; lanes, warps and blocks are combined as double-double values
// (TwoSum), and the per-block partials are folded by one block in block
// order, so the result is the same on every run.
#include "zm_dd.cuh"
#include "zm_kernels.cuh"

namespace zm {

__global__ void __launch_bounds__(128) k_diagnostics(Dev d, const float* __restrict__ T, const float* __restrict__ S,
                                                     const float* __restrict__ eta, const float* __restrict__ Fz,
                                                     const float* __restrict__ sp, float* __restrict__ rho,
                                                     float* __restrict__ pres, float* __restrict__ w) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= d.nx || j >= d.ny) return;
  const long long base = idx2(d, j, i);
  const uint64_t bits = __ldg(d.wbits + base);
  float p_bt = kRho0 * kG * ld(eta, base);
  if (sp) p_bt = p_bt + ld(sp, base);
  float p_bc = 0.f, r_prev = 0.f;
  for (int k = 0; k < d.nz; ++k) {
    const long long id = (long long)k * d.plane + base;
    const float r = rho_anom(ld(T, id), ld(S, id));
    const float wk = wetf(bits, k);
    const float rw = r * wk;
    if (k > 0) p_bc += kG * (0.5f * (r_prev + rw)) * d.vc.dz3d[k - 1];
    rho[id] = kRho0 + r;
    pres[id] = p_bt + p_bc;
    w[id] = -ld(Fz, id) * wk;
    r_prev = rw;
  }
}


// sums: 0 wet volume, 1 T volume, 2 S volume, 3 wet surface area,
// 4 T_top surface area, 5 S_top surface area, 6 total cell area.
__global__ void __launch_bounds__(256, 3) k_budget_partials(Dev d, const float* __restrict__ T,
                                                         const float* __restrict__ S,
                                                         const double* __restrict__ area,
                                                         const double* __restrict__ width,
                                                         double* __restrict__ partial) {
  __shared__ DD red[ZM_BUDGET_SUMS][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ncol = d.nx * d.ny, step = gridDim.x * 8;
  DD acc[ZM_BUDGET_SUMS];
#pragma unroll
  for (int q = 0; q < ZM_BUDGET_SUMS; ++q) acc[q] = DD{0.0, 0.0};
  const double wd0 = lane < d.nz ? width[lane] : 0.0, wd1 = lane + 32 < d.nz ? width[lane + 32] : 0.0;
  // One warp per column of the reference layout (nx, ny, nz), contiguous in z, BC of them in flight;
  // the float64 additions are the bound (fp64 pipe 46 %).  720 x 360 x 50: 175 us with one column
  // at a time and the surface sums on lane 0, 127 with four in flight (100 registers, two waves), 83 so.
  constexpr int BC = 2;
  for (int c0 = blockIdx.x * 8 + warp; c0 < ncol; c0 += BC * step) {
    double a[BC];
    float top[BC];
    uint64_t bits[BC];
    float t[BC][2], e[BC][2];
#pragma unroll
    for (int n = 0; n < BC; ++n) {
      const int col = c0 + n * step;
      a[n] = 0.0;
      top[n] = 0.f;
      bits[n] = 0ull;
      t[n][0] = t[n][1] = e[n][0] = e[n][1] = 0.f;
      if (col >= ncol) continue;
      const int i = col / d.ny, j = col - i * d.ny;
      a[n] = __ldg(area + col);
      bits[n] = wb(d, j, i);
      top[n] = __ldg(d.wet2 + idx2(d, j, i));
      const long long o = (long long)col * d.nz + lane;
      if (lane < d.nz) t[n][0] = __ldg(T + o), e[n][0] = __ldg(S + o);
      if (lane + 32 < d.nz) t[n][1] = __ldg(T + o + 32), e[n][1] = __ldg(S + o + 32);
    }
#pragma unroll
    for (int n = 0; n < BC; ++n) {  // past the last column: area and bits are zero
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double vol = (a[n] * (h ? wd1 : wd0)) * (double)((bits[n] >> (lane + 32 * h)) & 1ull);
        neumaier(acc[0], vol);
        neumaier(acc[1], (double)t[n][h] * vol);
        neumaier(acc[2], (double)e[n][h] * vol);
      }
    }
    // the surface sums: lane n takes column n
    double a1 = a[0];
    float w1 = top[0], t1 = __shfl_sync(0xffffffffu, t[0][0], 0), e1 = __shfl_sync(0xffffffffu, e[0][0], 0);
#pragma unroll
    for (int n = 1; n < BC; ++n) {
      const float tn = __shfl_sync(0xffffffffu, t[n][0], 0), en = __shfl_sync(0xffffffffu, e[n][0], 0);
      if (lane == n) a1 = a[n], w1 = top[n], t1 = tn, e1 = en;
    }
    if (lane < BC) {
      const double sa = a1 * (double)w1;
      neumaier(acc[3], sa);
      neumaier(acc[4], (double)t1 * sa);
      neumaier(acc[5], (double)e1 * sa);
      neumaier(acc[6], a1);
    }
  }
#pragma unroll
  for (int q = 0; q < ZM_BUDGET_SUMS; ++q) {
    DD x = two_sum(acc[q].hi, acc[q].lo);
    for (int o = 16; o > 0; o >>= 1) x = dd_add(x, shfl_dd(x, o));
    if (lane == 0) red[q][warp] = x;
  }
  __syncthreads();
  if (threadIdx.x < ZM_BUDGET_SUMS) {
    DD x = red[threadIdx.x][0];
    for (int w = 1; w < 8; ++w) x = dd_add(x, red[threadIdx.x][w]);
    partial[(blockIdx.x * ZM_BUDGET_SUMS + threadIdx.x) * 2] = x.hi;
    partial[(blockIdx.x * ZM_BUDGET_SUMS + threadIdx.x) * 2 + 1] = x.lo;
  }
}

// One warp per sum: lanes take every 32nd partial, then a tree; one thread per sum
// walked the 592 partials in 135 us.
__global__ void __launch_bounds__(32 * ZM_BUDGET_SUMS) k_budget_final(const double* __restrict__ partial, int nblocks,
                                                                      double* __restrict__ out) {
  const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  DD x{0.0, 0.0};
#pragma unroll 4
  for (int b = lane; b < nblocks; b += 32)
    x = dd_add(x, DD{__ldg(partial + (b * ZM_BUDGET_SUMS + q) * 2), __ldg(partial + (b * ZM_BUDGET_SUMS + q) * 2 + 1)});
  for (int o = 16; o > 0; o >>= 1) x = dd_add(x, shfl_dd(x, o));
  if (lane == 0) {
    out[2 * q] = x.hi;
    out[2 * q + 1] = x.lo;
  }
}

}  // namespace zm
