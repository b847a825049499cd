// Column-divergence projection of the stage-2 advective velocity
// (dynamics/projection.py:10-127, applied at timestepping/step.py:292-303).
//
// The reference solves A psi = b with jax.scipy.sparse.linalg.cg, where
//   A psi = -coldiv(grad3(psi)) area,   b = -(coldiv(u, v) / (dt g)) area,
// coldiv the level sum of the face-flux divergence times the node thickness
// on wet columns (transport.py:45-57) and grad3 the conservative gradient of
// the column-uniform psi (horizontal.py:126-151).  It corrects
// (u, v) -= dt g grad3(psi) and then, at most `refinements` times while the
// surface transport of the corrected velocity stays above rtol_t^2 times that
// of the input, solves again for the remaining divergence with an absolute
// floor tol ||b|| and corrects again.
//
// On the device:
//  * A is exactly a two-dimensional operator.  psi does not depend on the
//    level, so the level sum of the masked face fluxes needs only the
//    common-wet depths of two or three neighbouring columns.  With e_i(k) the
//    wet flag of the east face of column i at level k, H2_i = sum_k dz_k e_i
//    and H3_i = sum_k dz_k e_i e_{i+1}, the column flux through the east face is
//      Phi_i = 1/4 [ rdx_i (H3_{i-1} D_{i-1} + H2_i D_i)
//                  + rdx_{i+1} (H2_i D_i + H3_i D_{i+1}) ],   D_i = psi_{i+1} - psi_i,
//    and through the north face, with the face cosines cf_j = (c_j + c_{j+1})/2,
//      Psi_j = rdy cf_j / 4 [ (H2_j cf_j E_j + H3_{j-1} cf_{j-1} E_{j-1}) / c_j
//                           + (H3_j cf_{j+1} E_{j+1} + H2_j cf_j E_j) / c_{j+1} ].
//    k_proj_coef tabulates the three weights of each face once.
//  * The column divergence of the corrected velocity is that of the input plus
//    dt g (A psi) / area, so the right-hand side of a refinement is the
//    residual b - A psi_total of the first system and its transport norm is
//    (dt g)^2 sum res^2 / area.  The refinements therefore need no pass over
//    the 3-D fields: k_proj_rhs reads (u, v) once and k_proj_correct applies
//    the summed potential once.
//  * k_proj_res, for grids whose tiles fit in the SMs' shared memory, runs every
//    solve resident on the chip (below); k_proj_cg takes the larger grids.
//  * k_proj_cg runs every solve in one cooperative launch in float64, with the
//    loop of jax's cg: x = 0, r = b, z = M r, p = z, gamma = <r, z>; while the
//    squared residual (gamma without a preconditioner, <r, r> with one) is
//    above max(tol^2 <b, b>, atol^2) and k < maxiter: alpha = gamma / <p, Ap>,
//    x += alpha p, r -= alpha Ap, z = M r, beta = <r, z> / gamma, p = z + beta p.
//    The direction update is folded into the next product (each thread forms
//    z + beta p at its stencil points and stores its own), so an iteration
//    takes two grid barriers.  Dot products are summed per thread, per block in
//    a fixed tree and over blocks in block order by every block, so all blocks
//    take the same branches and the result does not depend on timing.  The
//    whole working set (a dozen 2-D float64 fields) stays in L2.
#include <algorithm>

#include "zm_kernels.cuh"
#include "zm_sync.cuh"

namespace zm {

namespace {

__device__ __forceinline__ double bitd(uint64_t bits, int k) { return (double)((bits >> k) & 1ull); }

__device__ double dz_sum(uint64_t bits, const double* __restrict__ dzn, int nz) {
  double s = 0.0;
  for (int k = 0; k < nz; ++k)
    if ((bits >> k) & 1ull) s += dzn[k];
  return s;
}

// Block partial sums of NQ values, tree order fixed, written to part[block].
template <int NQ>
__device__ __forceinline__ void block_partials(const double (&v)[NQ], double* part) {
  __shared__ double red[NQ][PJ_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    double x = v[q];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[q][warp] = x;
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double x = lane < nw ? red[q][lane] : 0.0;
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) part[blockIdx.x * ZM_PJ_SUMS + q] = x;
    }
  }
}

// Totals over all blocks, folded in block order; every block gets the same bits.
template <int NQ>
__device__ __forceinline__ void grid_totals(const double* part, double (&out)[NQ]) {
  __shared__ double tot[NQ];
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double x = 0.0;
      for (int b = lane; b < (int)gridDim.x; b += 32) x += __ldcg(part + b * ZM_PJ_SUMS + q);
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) tot[q] = x;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NQ; ++q) out[q] = tot[q];
  __syncthreads();
}

// Global sums through a grid barrier.  The partials alternate between two
// buffers: a block can only overwrite a buffer after every block has passed
// the next barrier, i.e. has finished reading it.
template <int NQ>
__device__ __forceinline__ bool reduce(const ProjArgs& a, int& red, const double (&v)[NQ], double (&out)[NQ]) {
  double* part = a.part + (size_t)(red & 1) * gridDim.x * ZM_PJ_SUMS;
  ++red;
  block_partials(v, part);
  if (!grid_barrier(a.bar, a.err, gridDim.x, a.max_polls)) return false;
  grid_totals(part, out);
  return true;
}

// (A q) at (j, i); val(g) gives q at the 2-D index g.  `center` receives q(j, i).
template <class V>
__device__ __forceinline__ double apply_a(const Dev& d, const ProjArgs& a, int j, int i, V val, double& center) {
  const long long n2 = d.plane;
  const int iw = west(d, i), ie = east(d, i);
  const int iww = west(d, iw), iee = east(d, ie);
  const int js = max(j - 1, 0), jss = max(j - 2, 0);
  const int jn = min(j + 1, d.ny - 1), jnn = min(j + 2, d.ny - 1);
  const int g = idx2(d, j, i), gw = idx2(d, j, iw), gs = idx2(d, js, i);
  const double pc = val(g);
  const double pw = val(gw), pww = val(idx2(d, j, iww));
  const double pe = val(idx2(d, j, ie)), pee = val(idx2(d, j, iee));
  const double ps = val(gs), pss = val(idx2(d, jss, i));
  const double pn = val(idx2(d, jn, i)), pnn = val(idx2(d, jnn, i));
  center = pc;
  const double fe = __ldg(a.cx + g) * (pc - pw) + __ldg(a.cx + n2 + g) * (pe - pc) +
                    __ldg(a.cx + 2 * n2 + g) * (pee - pe);
  const double fw = __ldg(a.cx + gw) * (pw - pww) + __ldg(a.cx + n2 + gw) * (pc - pw) +
                    __ldg(a.cx + 2 * n2 + gw) * (pe - pc);
  const double fn = __ldg(a.cy + g) * (pc - ps) + __ldg(a.cy + n2 + g) * (pn - pc) +
                    __ldg(a.cy + 2 * n2 + g) * (pnn - pn);
  const double fs = j > 0 ? __ldg(a.cy + gs) * (ps - pss) + __ldg(a.cy + n2 + gs) * (pc - ps) +
                                __ldg(a.cy + 2 * n2 + gs) * (pn - pc)
                          : 0.0;
  return -(__ldg(a.sxy + g) * (fe - fw) + __ldg(a.sxy + n2 + g) * (fn - fs));
}

// One CG solve (jax loop) into x, which the caller has zeroed together with
// a.p0, r = rhs and z = M rhs, followed by a barrier.  Returns the iteration
// count, or -1 if a grid barrier gave up.
__device__ int cg_solve(const Dev& d, const ProjArgs& a, double* x, double gamma, double rr, double atol2, int& red) {
  const bool ident = a.minv == nullptr;
  const int ncell = d.nx * d.ny;
  const int stride = gridDim.x * blockDim.x;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
  const double* pold = a.p0;
  double* pnew = a.p1;
  double beta = 0.0;
  int k = 0;
  while ((ident ? gamma : rr) > atol2 && k < a.niter) {
    double s[1] = {0.0};
    for (int c = t0; c < ncell; c += stride) {
      const int j = c / d.nx, i = c - j * d.nx;
      double pc;
      const double ap = apply_a(
          d, a, j, i, [&](int g) { return fma(beta, __ldcg(pold + g), __ldcg(a.z + g)); }, pc);
      const int g = idx2(d, j, i);
      pnew[g] = pc;
      a.Ap[g] = ap;
      s[0] += pc * ap;
    }
    double t[1];
    if (!reduce(a, red, s, t)) return -1;
    const double alpha = gamma / t[0];
    double s2[2] = {0.0, 0.0};
    for (int c = t0; c < ncell; c += stride) {
      const int j = c / d.nx, i = c - j * d.nx;
      const int g = idx2(d, j, i);
      x[g] = __ldcg(x + g) + alpha * __ldcg(pnew + g);
      const double rv = __ldcg(a.r + g) - alpha * __ldcg(a.Ap + g);
      const double zv = ident ? rv : rv * __ldg(a.minv + g);
      a.r[g] = rv;
      a.z[g] = zv;
      s2[0] += rv * zv;
      s2[1] += rv * rv;
    }
    double t2[2];
    if (!reduce(a, red, s2, t2)) return -1;
    beta = t2[0] / gamma;
    gamma = t2[0];
    rr = t2[1];
    double* tmp = const_cast<double*>(pold);
    pold = pnew;
    pnew = tmp;
    ++k;
  }
  return k;
}

}  // namespace

// Face weights of the column operator, the row factors, 1/area and the
// Jacobi inverse diagonal (projection.py:10-51: the per-level diagonal of the
// 3-D operator summed with the node thicknesses; 1 where it is not positive).
__global__ void __launch_bounds__(256) k_proj_coef(Dev d, const double* __restrict__ dzn,
                                                   const double* __restrict__ cosd, const double* __restrict__ area,
                                                   double* __restrict__ cx, double* __restrict__ cy,
                                                   double* __restrict__ sxy, double* __restrict__ minv,
                                                   double* __restrict__ rarea) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= d.nx || j >= d.ny) return;
  const long long n2 = d.plane;
  const int g = idx2(d, j, i);
  const int iw = west(d, i), ie = east(d, i), iee = east(d, ie);
  const uint64_t wc = wb(d, j, i), we = wb(d, j, ie), ww = wb(d, j, iw), wee = wb(d, j, iee);
  const uint64_t e_w = ww & wc, e_c = wc & we, e_e = we & wee;
  const double rdx = d.inv_dx_d[g], rdx_e = d.inv_dx_d[idx2(d, j, ie)];
  cx[g] = 0.25 * rdx * dz_sum(e_w & e_c, dzn, d.nz);
  cx[n2 + g] = 0.25 * (rdx + rdx_e) * dz_sum(e_c, dzn, d.nz);
  cx[2 * n2 + g] = 0.25 * rdx_e * dz_sum(e_c & e_e, dzn, d.nz);
  const double rdy = d.inv_dy_d;
  const double c = cosd[j];
  double y0 = 0.0, y1 = 0.0, y2 = 0.0;
  if (j + 1 < d.ny) {
    const double cn = cosd[j + 1];
    const double cf = 0.5 * (c + cn);
    const uint64_t n_c = wc & wb(d, j + 1, i);
    const uint64_t n_s = j > 0 ? (wb(d, j - 1, i) & wc) : 0ull;
    const uint64_t n_n = j + 2 < d.ny ? (wb(d, j + 1, i) & wb(d, j + 2, i)) : 0ull;
    const double q = 0.25 * rdy * cf;
    if (j > 0) y0 = q * dz_sum(n_s & n_c, dzn, d.nz) * (0.5 * (cosd[j - 1] + c)) / c;
    y1 = q * dz_sum(n_c, dzn, d.nz) * cf * (1.0 / c + 1.0 / cn);
    if (j + 2 < d.ny) y2 = q * dz_sum(n_c & n_n, dzn, d.nz) * (0.5 * (cn + cosd[j + 2])) / cn;
  }
  cy[g] = y0;
  cy[n2 + g] = y1;
  cy[2 * n2 + g] = y2;
  const double ar = area[g];
  sxy[g] = ar * rdx;
  sxy[n2 + g] = ar * rdy / c;
  rarea[g] = ar > 0.0 ? 1.0 / ar : 0.0;
  if (minv) {
    const double cnr = cosd[(j + 1) % d.ny], csr = cosd[(j - 1 + d.ny) % d.ny];
    const bool has_n = j + 1 < d.ny, has_s = j > 0;
    const uint64_t wn = has_n ? wb(d, j + 1, i) : 0ull, ws = has_s ? wb(d, j - 1, i) : 0ull;
    double sum = 0.0;
    for (int k = 0; k < d.nz; ++k) {
      double dxg = 0.0;
      if (d.nx > 2) {
        const double pos = bitd(e_c, k), neg = bitd(e_w, k);
        dxg = 0.25 * rdx * rdx * ((pos - neg) * (pos - neg) + pos * pos + neg * neg);
      }
      const double py = bitd(wc & wn, k) * (0.5 * (c + cnr));
      const double ny_ = bitd(wc & ws, k) * (0.5 * (c + csr));
      const double dyg = 0.25 * rdy * rdy *
                         ((py - ny_) * (py - ny_) / (c * c) + py * py / (c * cnr) + ny_ * ny_ / (c * csr));
      sum += (dxg + dyg) * dzn[k];
    }
    const double diag = ar * sum;
    minv[g] = diag > 0.0 ? 1.0 / diag : 1.0;
  }
}

// b = -(coldiv(u, v) / (dt g)) area (projection.py:64-80 with transport.py:45-57
// and horizontal.py:255-281), float64 from the float32 velocity.
__global__ void __launch_bounds__(256) k_proj_rhs(Dev d, const float* __restrict__ u, const float* __restrict__ v,
                                                  const double* __restrict__ dzn, const double* __restrict__ cosd,
                                                  const double* __restrict__ area, double dtg,
                                                  double* __restrict__ b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= d.nx || j >= d.ny) return;
  const int g = idx2(d, j, i);
  const int iw = west(d, i), ie = east(d, i);
  const uint64_t wc = wb(d, j, i);
  const uint64_t e_c = wc & wb(d, j, ie), e_w = wb(d, j, iw) & wc;
  const bool has_n = j + 1 < d.ny, has_s = j > 0;
  const uint64_t n_c = has_n ? (wc & wb(d, j + 1, i)) : 0ull;
  const uint64_t n_s = has_s ? (wb(d, j - 1, i) & wc) : 0ull;
  const int jn = has_n ? j + 1 : j, js = has_s ? j - 1 : j;
  const double rdx = d.inv_dx_d[g], rdy = d.inv_dy_d;
  const double c = cosd[j];
  const double cfn = has_n ? 0.5 * (c + cosd[j + 1]) : 0.0;
  const double cfs = has_s ? 0.5 * (cosd[j - 1] + c) : 0.0;
  double sum = 0.0;
  const int nk = levels_of(wc);  // a face of the column is open only where the column is wet
  for (int k = 0; k < nk; ++k) {
    const long long o = (long long)k * d.plane;
    const double uc = ld(u, o + g), ue = ld(u, o + idx2(d, j, ie)), uw = ld(u, o + idx2(d, j, iw));
    const double vc = ld(v, o + g), vn = ld(v, o + idx2(d, jn, i)), vs = ld(v, o + idx2(d, js, i));
    const double fxe = 0.5 * (uc + ue) * bitd(e_c, k);
    const double fxw = 0.5 * (uw + uc) * bitd(e_w, k);
    const double fyn = 0.5 * (vc + vn) * bitd(n_c, k) * cfn;
    const double fys = 0.5 * (vs + vc) * bitd(n_s, k) * cfs;
    sum += ((fxe - fxw) * rdx + (fyn - fys) * rdy / c) * dzn[k];
  }
  const double cdiv = sum * (double)__ldg(d.wet2 + g);
  b[g] = -(cdiv / dtg) * area[g];
}

__global__ void __launch_bounds__(PJ_THREADS, 1) k_proj_cg(Dev d, ProjArgs a) {
  grid_barrier_begin(a.bar);
  const bool ident = a.minv == nullptr;
  const int ncell = d.nx * d.ny;
  const int stride = gridDim.x * blockDim.x;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
  int red = 0;
  // r = b, z = M b, psi = 0, p = 0; <b, b>, <b, z>, sum b^2 / area
  double s[3] = {0.0, 0.0, 0.0};
  for (int c = t0; c < ncell; c += stride) {
    const int j = c / d.nx, i = c - j * d.nx;
    const int g = idx2(d, j, i);
    const double bv = __ldcg(a.b + g);
    const double zv = ident ? bv : bv * __ldg(a.minv + g);
    a.r[g] = bv;
    a.z[g] = zv;
    a.psi[g] = 0.0;
    a.p0[g] = 0.0;
    s[0] += bv * bv;
    s[1] += bv * zv;
    s[2] += bv * bv * __ldg(a.rarea + g);
  }
  double t[3];
  if (!reduce(a, red, s, t)) return;
  const double bb = t[0];
  const double floor2 = a.tol2 * bb;  // (tol ||b||)^2
  const double thresh = a.trtol2 * t[2];
  int it[3] = {0, 0, 0};
  int nref = 0;
  it[0] = cg_solve(d, a, a.psi, t[1], bb, a.tol2 * bb, red);
  if (it[0] < 0) return;
  for (int q = 0; q < a.refinements; ++q) {
    // residual of the corrected velocity: res = b - A psi
    double s3[3] = {0.0, 0.0, 0.0};
    for (int c = t0; c < ncell; c += stride) {
      const int j = c / d.nx, i = c - j * d.nx;
      const int g = idx2(d, j, i);
      double pc;
      const double ap = apply_a(d, a, j, i, [&](int h) { return __ldcg(a.psi + h); }, pc);
      const double res = __ldcg(a.b + g) - ap;
      const double zv = ident ? res : res * __ldg(a.minv + g);
      a.r[g] = res;
      a.z[g] = zv;
      a.x[g] = 0.0;
      a.p0[g] = 0.0;
      s3[0] += res * res;
      s3[1] += res * zv;
      s3[2] += res * res * __ldg(a.rarea + g);
    }
    double t3[3];
    if (!reduce(a, red, s3, t3)) return;
    if (!(t3[2] > thresh)) break;
    ++nref;
    it[1 + q] = cg_solve(d, a, a.x, t3[1], t3[0], fmax(a.tol2 * t3[0], floor2), red);
    if (it[1 + q] < 0) return;
    for (int c = t0; c < ncell; c += stride) {
      const int j = c / d.nx, i = c - j * d.nx;
      const int g = idx2(d, j, i);
      a.psi[g] = __ldcg(a.psi + g) + __ldcg(a.x + g);
    }
    // the next residual reads the neighbours' psi
    if (q + 1 < a.refinements || a.norms)
      if (!grid_barrier(a.bar, a.err, gridDim.x, a.max_polls)) return;
  }
  if (a.norms) {
    // ledger mode: squared surface-transport norms of the input and of the
    // corrected velocity, (dt g)^2 sum b^2 / area and (dt g)^2 sum res^2 / area
    // (diagnostics/budgets.py:175-183)
    double s4[1] = {0.0};
    for (int c = t0; c < ncell; c += stride) {
      const int j = c / d.nx, i = c - j * d.nx;
      const int g = idx2(d, j, i);
      double pc;
      const double res = __ldcg(a.b + g) - apply_a(d, a, j, i, [&](int h) { return __ldcg(a.psi + h); }, pc);
      s4[0] += res * res * __ldg(a.rarea + g);
    }
    double t4[1];
    if (!reduce(a, red, s4, t4)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.norms[0] = a.dtg * a.dtg * t[2];
      a.norms[1] = a.dtg * a.dtg * t4[0];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.stats[0] = it[0];
    a.stats[1] = it[1];
    a.stats[2] = it[2];
    a.stats[3] = nref;
  }
}

// (u, v) -= dt g grad3(psi) (projection.py:84-90 with horizontal.py:126-151).
__global__ void __launch_bounds__(256) k_proj_correct(Dev d, float* __restrict__ u, float* __restrict__ v,
                                                      const double* __restrict__ psi,
                                                      const double* __restrict__ cosd, double dtg) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= d.nx || j >= d.ny) return;
  const int g = idx2(d, j, i);
  const int iw = west(d, i), ie = east(d, i);
  const uint64_t wc = wb(d, j, i);
  const uint64_t e_c = wc & wb(d, j, ie), e_w = wb(d, j, iw) & wc;
  const bool has_n = j + 1 < d.ny, has_s = j > 0;
  const uint64_t pos = has_n ? (wc & wb(d, j + 1, i)) : 0ull;
  const uint64_t neg = has_s ? (wb(d, j - 1, i) & wc) : 0ull;
  const double pc = psi[g], pe = psi[idx2(d, j, ie)], pw = psi[idx2(d, j, iw)];
  const double pn = has_n ? psi[idx2(d, j + 1, i)] : pc, ps = has_s ? psi[idx2(d, j - 1, i)] : pc;
  const double c = cosd[j];
  const double cp = 0.5 * (c + cosd[(j + 1) % d.ny]), cm = 0.5 * (c + cosd[(j - 1 + d.ny) % d.ny]);
  const double hx = d.inv_dx_d[g] * 0.5, hy = (d.inv_dy_d / c) * 0.5;
  const double dxe = pe - pc, dxw = pc - pw, dyn = (pn - pc) * cp, dys = (pc - ps) * cm;
  const int nk = levels_of(wc);  // every face of a dry point is closed
  for (int k = 0; k < nk; ++k) {
    const long long o = (long long)k * d.plane + g;
    const double gx = hx * (dxe * bitd(e_c, k) + dxw * bitd(e_w, k));
    const double gy = hy * (dyn * bitd(pos, k) + dys * bitd(neg, k));
    u[o] = (float)((double)u[o] - dtg * gx);
    v[o] = (float)((double)v[o] - dtg * gy);
  }
}

// ---------------------------------------------------------------- resident form
//
// One block owns a tile of the grid.  The direction of steepest descent z
// and s = A p stay in shared memory with a two-cell halo, the face weights of
// the tile too, x, p and r in registers; the loop touches global memory only
// for what the blocks exchange.  What bounds an iteration is the latency of
// its grid-wide sums, so there is one exchange per iteration: with w = A z,
//   gamma = <r, z>, delta = <w, z>,  beta = gamma / gamma_old,
//   alpha = gamma / (delta - beta gamma / alpha_old),
//   p = z + beta p, s = w + beta s, x += alpha p, r -= alpha s, z = M r,
// the recurrences of Chronopoulos and Gear (1989), equal to the loop above in
// exact arithmetic for a symmetric A (zm_create checks the grid); both sums are formed
// before either scalar is needed.  The
// halo needs no second exchange: each block publishes its w along the tile's
// edges with the sums, and carries s and z of its halo cells with the same
// recurrences.
//
// Everything the blocks exchange is a 16-byte {value, sequence number} word,
// stored and loaded whole: a reader polls the word itself, so no fence, atomic
// or second load stands between a value and its use.  A block's partial sums
// go to every block's own list of words, one copy per reader: one list that
// all blocks poll is a few cache lines with up to 148 readers each, and cost
// 1.8 us more per exchange.  The lists are added in block order, so every
// block gets the same bits.
// Per iteration, against the streamed form's two barriers and two passes over
// L2 (10.0 us at 360x180 cells, 14.5 us at 720x360): 4.0 and 5.7 us; without
// the wait for the sums the loop takes 3.3 and 5.3 us, so what is left is the
// latency of the FP64 chains and of one store and load across the chip.

namespace {

template <int N>
struct PjInt {
  static constexpr int value = N;
};

struct ResShared {  // fixed part of the block's shared memory
  double red[ZM_PJ_SUMS][32];
  double tot[ZM_PJ_SUMS], part[ZM_PJ_SUMS][WORD_CHUNKS];
  double pad;  // an even number of doubles, for what follows
};

}  // namespace

// Shared memory of a tile of tx x ty cells.
size_t proj_res_smem(int tx, int ty) {
  const size_t halo = (size_t)(tx + 4) * (ty + 4), own = (size_t)tx * ty;
  return sizeof(ResShared) + sizeof(double) * (4 * (size_t)(tx + ty) + 2 * halo + 3 * (size_t)(tx + 1) * ty +
                                               3 * (size_t)tx * (ty + 1) + 2 * own);
}

// Thread (lx, chunk) owns CPT consecutive rows of column lx of the tile; with
// one row per thread the face weights of its cell stay in registers.  The
// index arithmetic is done before the loop.
template <int CPT>
__global__ void __launch_bounds__(PJ_RES_THREADS, 1) k_proj_res(Dev d, ProjArgs a) {
  extern __shared__ double pr_smem[];
  constexpr bool REGS = CPT == 1;
  constexpr int HS = 2;  // halo cells per thread held ready (the others are found again each time)
  const int tx = a.tile_x, ty = a.tile_y, PX = tx + 4, PY = ty + 4, nb = gridDim.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  ResShared& sh = *reinterpret_cast<ResShared*>(pr_smem);
  double* hv = pr_smem + sizeof(ResShared) / sizeof(double);  // gathered halo values
  double* z = hv + 4 * (tx + ty);          // [PY][PX]
  double* sv = z + PX * PY;                // [PY][PX]
  double* cx = sv + PX * PY;               // [3][ty][tx + 1]: east faces of columns -1 .. tx - 1
  double* cy = cx + 3 * (tx + 1) * ty;     // [3][ty + 1][tx]: north faces of rows -1 .. ty - 1
  double* sx = cy + 3 * tx * (ty + 1);     // [ty][tx] area / dx
  double* sy = sx + tx * ty;               // [ty][tx] area / (dy cos)
  Word* words = reinterpret_cast<Word*>(a.words);
  const bool ident = a.minv == nullptr;
  const long long n2 = d.plane;
  const int i0 = (int)(blockIdx.x % a.tiles_x) * tx, j0 = (int)(blockIdx.x / a.tiles_x) * ty;
  const int w_own = min(tx, d.nx - i0), h_own = min(ty, d.ny - j0);
  auto wrap = [&](int i) {
    i %= d.nx;
    return i < 0 ? i + d.nx : i;
  };
  for (int e = threadIdx.x; e < (tx + 1) * ty; e += blockDim.x) {
    const int r = e / (tx + 1), c = e - r * (tx + 1) - 1;
    const bool in = r < h_own && c < w_own;
    const int g = in ? idx2(d, j0 + r, wrap(i0 + c)) : 0;
    for (int q = 0; q < 3; ++q) cx[q * (tx + 1) * ty + e] = in ? __ldg(a.cx + q * n2 + g) : 0.0;
  }
  for (int e = threadIdx.x; e < tx * (ty + 1); e += blockDim.x) {
    const int r = e / tx - 1, c = e - (r + 1) * tx;
    const bool in = r < h_own && c < w_own && j0 + r >= 0;  // no face south of the first row
    const int g = in ? idx2(d, j0 + r, i0 + c) : 0;
    for (int q = 0; q < 3; ++q) cy[q * tx * (ty + 1) + e] = in ? __ldg(a.cy + q * n2 + g) : 0.0;
  }
  for (int e = threadIdx.x; e < tx * ty; e += blockDim.x) {
    const int r = e / tx, c = e - r * tx;
    const bool in = r < h_own && c < w_own;
    const int g = in ? idx2(d, j0 + r, i0 + c) : 0;
    sx[e] = in ? __ldg(a.sxy + g) : 0.0;
    sy[e] = in ? __ldg(a.sxy + n2 + g) : 0.0;
  }
  // ---- the thread's own cells
  const int lx = threadIdx.x % tx, ly0 = (int)(threadIdx.x / tx) * CPT;
  const int rows = lx < w_own ? min(CPT, h_own - ly0) : 0;  // owned rows, none where <= 0
  const int o0 = (ly0 + 2) * PX + lx + 2, g0 = idx2(d, j0 + ly0, i0 + lx);
  auto own = [&](int q) { return q < rows; };
  auto edge = [&](int q) { return lx < 2 || lx >= w_own - 2 || ly0 + q < 2 || ly0 + q >= h_own - 2; };
  Word* const pub0 = reinterpret_cast<Word*>(a.pub) + g0;
  // ---- halo: the cells two deep around the tile that the stencil reads, two
  // columns west and east, two rows south and north (none beyond the walls);
  // cell h as its place e in the padded tile and its 2-D index g
  const int n_halo = 4 * (h_own + w_own);
  auto halo_cell = [&](int h, int& e, int& g) {
    if (h >= n_halo) return false;
    int r, c;
    if (h < 4 * h_own) {
      const int s = h / h_own;
      r = h - s * h_own;
      c = s < 2 ? s - 2 : w_own + s - 2;
    } else {
      const int m = h - 4 * h_own, s = m / w_own;
      c = m - s * w_own;
      r = s < 2 ? s - 2 : h_own + s - 2;
    }
    if (j0 + r < 0 || j0 + r >= d.ny) return false;
    e = (r + 2) * PX + c + 2;
    g = idx2(d, j0 + r, wrap(i0 + c));
    return true;
  };
  // from the last thread down: the first warps gather the sums
  const int h0 = (int)(blockDim.x - 1 - threadIdx.x), hstep = (int)blockDim.x;
  int he[HS], hg[HS];  // place -1: no cell
#pragma unroll
  for (int s = 0; s < HS; ++s)
    if (h0 < 0 || !halo_cell(h0 + s * hstep, he[s], hg[s])) he[s] = -1;
  // f(e, g, h) over this thread's halo cells
  auto each_halo = [&](auto&& f) {
#pragma unroll
    for (int s = 0; s < HS; ++s)
      if (he[s] >= 0) f(he[s], hg[s], h0 + s * hstep);
    for (int h = h0 < 0 ? n_halo : h0 + HS * hstep; h < n_halo; h += hstep) {
      int e, g;
      if (halo_cell(h, e, g)) f(e, g, h);
    }
  };
  unsigned long long seq = *reinterpret_cast<volatile unsigned long long*>(a.seq) + 1;
  // Publishes own(q)'s value along the tile's edges; before exchange().
  auto publish = [&](int q, double v) {
    if (edge(q)) st_word(pub0 + (seq & 1) * n2 + q * d.P, v, seq);
  };
  // Sums of NQ values over the grid into `out`, the same bits in every block,
  // and the published values of the halo cells into hv.  Words alternate
  // between two sets: a block writes those of exchange n + 2 only after it has
  // seen every block's sums n + 1, which follow that block's reads of n.
  // False if a word did not come within the poll limit or a block gave up.
  const int nchunk = (nb + 31) / 32;
  auto exchange = [&](auto& v, auto& out) {
    constexpr int NQ = sizeof(v) / sizeof(double);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < NQ; ++q) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
    if (lane == 0) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) sh.red[q][warp] = v[q];
    }
    __syncthreads();
    bool ok = true;
    if (warp == 0) {
      double x[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) x[q] = lane < nw ? sh.red[q][lane] : 0.0;
#pragma unroll
      for (int o = PJ_RES_THREADS / 64; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < NQ; ++q) x[q] += __shfl_down_sync(0xffffffffu, x[q], o);
      if (lane == 0) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) sh.tot[q] = x[q];
      }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < NQ * nb; t += blockDim.x) {
      const int q = t / nb, dst = t - q * nb;
      st_word(words + ((size_t)((seq & 1) * nb + dst) * ZM_PJ_SUMS + q) * nb + blockIdx.x, sh.tot[q], seq);
    }
    const Word* mine = words + (size_t)((seq & 1) * nb + blockIdx.x) * ZM_PJ_SUMS * nb;
    for (int c = warp; c < NQ * nchunk; c += nw) {
      const int q = c / nchunk, blk = (c - q * nchunk) * 32 + lane;
      double y = 0.0;
      if (blk < nb) ok = wait_word(mine + q * nb + blk, seq, a.err, a.max_polls, y) && ok;
      __syncwarp();
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) y += __shfl_down_sync(0xffffffffu, y, o);
      if (lane == 0) sh.part[q][c - q * nchunk] = y;
    }
    const Word* pub = reinterpret_cast<const Word*>(a.pub) + (seq & 1) * n2;
    each_halo([&](int, int g, int h) { ok = ok && wait_word(pub + g, seq, a.err, a.max_polls, hv[h]); });
    ++seq;
    if (__syncthreads_or(!ok)) return false;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double y = sh.part[q][0];
      for (int c = 1; c < nchunk; ++c) y += sh.part[q][c];
      out[q] = y;
    }
    return true;
  };
  // ---- A f on the thread's cells, f a padded array
  const int fy = tx * (ty + 1), fx = (tx + 1) * ty;
  const int ey0 = ly0 * tx + lx, ex0 = ly0 * (tx + 1) + lx + 1;  // the face south of the first row, the one east of it
  __syncthreads();
  double k_[REGS ? 14 : 1];
  if (REGS && rows > 0) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      k_[q] = cx[q * fx + ex0];
      k_[3 + q] = cx[q * fx + ex0 - 1];
      k_[6 + q] = cy[q * fy + ey0 + tx];
      k_[9 + q] = cy[q * fy + ey0];
    }
    k_[12] = sx[ey0];
    k_[13] = sy[ey0];
  }
  auto apply = [&](const double* f, double (&out)[CPT]) {
#pragma unroll
    for (int q = 0; q < CPT; ++q) out[q] = 0.0;
    if (rows <= 0) return;
    const double* c = f + o0;
    if (REGS) {
      const double pc = c[0], pw = c[-1], pe = c[1], pn = c[PX], ps = c[-PX];
      const double dw = pc - pw, de = pe - pc, ds = pc - ps, dn = pn - pc;
      const double fe = k_[0] * dw + k_[1] * de + k_[2] * (c[2] - pe);
      const double fw = k_[3] * (pw - c[-2]) + k_[4] * dw + k_[5] * de;
      const double fn = k_[6] * ds + k_[7] * dn + k_[8] * (c[2 * PX] - pn);
      const double fs = k_[9] * (ps - c[-2 * PX]) + k_[10] * ds + k_[11] * dn;
      out[0] = -(k_[12] * (fe - fw) + k_[13] * (fn - fs));
      return;
    }
    const double* ky = cy + ey0;
    const double* kx = cx + ex0;
    // north flux of the row below the chunk
    double fs = ky[0] * (c[-PX] - c[-2 * PX]) + ky[fy] * (c[0] - c[-PX]) + ky[2 * fy] * (c[PX] - c[0]);
#pragma unroll
    for (int q = 0; q < CPT; ++q) {
      if (q >= rows) break;
      ky += tx;
      const double pc = c[0], pw = c[-1], pe = c[1], pn = c[PX];
      const double dw = pc - pw, de = pe - pc;
      const double fe = kx[0] * dw + kx[fx] * de + kx[2 * fx] * (c[2] - pe);
      const double fw = kx[-1] * (pw - c[-2]) + kx[fx - 1] * dw + kx[2 * fx - 1] * de;
      const double fn = ky[0] * (pc - c[-PX]) + ky[fy] * (pn - pc) + ky[2 * fy] * (c[2 * PX] - pn);
      out[q] = -(sx[ey0 + q * tx] * (fe - fw) + sy[ey0 + q * tx] * (fn - fs));
      fs = fn;
      c += PX;
      kx += tx + 1;
    }
  };
  for (int e = threadIdx.x; e < PX * PY; e += blockDim.x) z[e] = sv[e] = 0.0;
  __syncthreads();
  // z = M b, r = b; psi = 0
  double psi[CPT], x[CPT], r[CPT], p[CPT], w[CPT];
  double s2[2] = {0.0, 0.0}, t2[2];
#pragma unroll
  for (int q = 0; q < CPT; ++q) {
    psi[q] = r[q] = 0.0;
    if (own(q)) {
      const int g = g0 + q * d.P;
      r[q] = __ldcg(a.b + g);
      z[o0 + q * PX] = ident ? r[q] : r[q] * __ldg(a.minv + g);
      s2[0] += r[q] * r[q];
      s2[1] += r[q] * r[q] * __ldg(a.rarea + g);
      publish(q, r[q]);
    }
  }
  if (!exchange(s2, t2)) return;
  each_halo([&](int e, int g, int h) { z[e] = ident ? hv[h] : hv[h] * __ldg(a.minv + g); });
  __syncthreads();
  const double floor2 = a.tol2 * t2[0], thresh = a.trtol2 * t2[1], norm_in = t2[1];
  int it[3] = {0, 0, 0}, nref = 0;

  // one CG solve from r and z into x; NQ 2 without a preconditioner, where
  // <r, r> is gamma, else 3; returns the iterations, -1 after a timeout
  auto solve_n = [&](auto nq, double atol2) {
    constexpr int NQ = decltype(nq)::value;
    double gamma_old = 1.0, alpha_old = 1.0;
#pragma unroll
    for (int q = 0; q < CPT; ++q) x[q] = p[q] = 0.0;
    for (int k = 0;; ++k) {
      apply(z, w);
      double s[NQ], t[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) s[q] = 0.0;
#pragma unroll
      for (int q = 0; q < CPT; ++q) {
        if (!own(q)) continue;
        publish(q, w[q]);
        const double zq = NQ == 2 ? r[q] : z[o0 + q * PX];
        s[0] += r[q] * zq;
        s[1] += w[q] * zq;
        if (NQ > 2) s[NQ - 1] += r[q] * r[q];
      }
      if (!exchange(s, t)) return -1;
      if (!(t[NQ > 2 ? NQ - 1 : 0] > atol2) || k >= a.niter) return k;
      const double beta = k > 0 ? t[0] / gamma_old : 0.0;
      const double alpha = k > 0 ? t[0] / (t[1] - beta * t[0] / alpha_old) : t[0] / t[1];
      gamma_old = t[0];
      alpha_old = alpha;
      each_halo([&](int e, int g, int h) {
        const double sq = k > 0 ? fma(beta, sv[e], hv[h]) : hv[h];
        sv[e] = sq;
        z[e] -= alpha * (NQ == 2 ? sq : sq * __ldg(a.minv + g));
      });
#pragma unroll
      for (int q = 0; q < CPT; ++q) {
        if (!own(q)) continue;
        const int o = o0 + q * PX;
        p[q] = fma(beta, p[q], NQ == 2 ? r[q] : z[o]);
        const double sq = k > 0 ? fma(beta, sv[o], w[q]) : w[q];
        sv[o] = sq;
        x[q] += alpha * p[q];
        r[q] -= alpha * sq;
        z[o] = NQ == 2 ? r[q] : r[q] * __ldg(a.minv + g0 + q * d.P);
      }
      __syncthreads();
    }
  };
  auto solve = [&](double atol2) {
    return ident ? solve_n(PjInt<2>{}, atol2) : solve_n(PjInt<3>{}, atol2);
  };
  // w = A psi (through z, which the caller sets again)
  auto apply_psi = [&]() {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < CPT; ++q)
      if (own(q)) {
        z[o0 + q * PX] = psi[q];
        publish(q, psi[q]);
      }
    double s[1] = {0.0}, t[1];
    if (!exchange(s, t)) return false;
    each_halo([&](int e, int, int h) { z[e] = hv[h]; });
    __syncthreads();
    apply(z, w);
    __syncthreads();
    return true;
  };

  it[0] = solve(a.tol2 * t2[0]);
  if (it[0] < 0) return;
#pragma unroll
  for (int q = 0; q < CPT; ++q) psi[q] = x[q];
  for (int n = 0; n < a.refinements; ++n) {
    // residual of the corrected velocity: res = b - A psi
    if (!apply_psi()) return;
    double s[2] = {0.0, 0.0}, t[2];
#pragma unroll
    for (int q = 0; q < CPT; ++q) {
      if (!own(q)) continue;
      const int g = g0 + q * d.P;
      const double res = __ldcg(a.b + g) - w[q];
      r[q] = res;
      z[o0 + q * PX] = ident ? res : res * __ldg(a.minv + g);
      s[0] += res * res;
      s[1] += res * res * __ldg(a.rarea + g);
      publish(q, res);
    }
    if (!exchange(s, t)) return;
    if (!(t[1] > thresh)) break;
    each_halo([&](int e, int g, int h) { z[e] = ident ? hv[h] : hv[h] * __ldg(a.minv + g); });
    __syncthreads();
    ++nref;
    it[1 + n] = solve(fmax(a.tol2 * t[0], floor2));
    if (it[1 + n] < 0) return;
#pragma unroll
    for (int q = 0; q < CPT; ++q) psi[q] += x[q];
  }
#pragma unroll
  for (int q = 0; q < CPT; ++q)
    if (own(q)) a.psi[g0 + q * d.P] = psi[q];
  if (a.norms) {  // ledger mode, as in k_proj_cg
    if (!apply_psi()) return;
    double s[1] = {0.0}, t[1];
#pragma unroll
    for (int q = 0; q < CPT; ++q)
      if (own(q)) {
        const double res = __ldcg(a.b + g0 + q * d.P) - w[q];
        s[0] += res * res * __ldg(a.rarea + g0 + q * d.P);
        publish(q, 0.0);
      }
    if (!exchange(s, t)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.norms[0] = a.dtg * a.dtg * norm_in;
      a.norms[1] = a.dtg * a.dtg * t[0];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.stats[0] = it[0];
    a.stats[1] = it[1];
    a.stats[2] = it[2];
    a.stats[3] = nref;
    *a.seq = seq - 1;  // every block has read it: it took part in the last exchange
  }
}

void (*proj_res_kernel(int cpt))(Dev, ProjArgs) {
  return cpt <= 1 ? k_proj_res<1> : cpt == 2 ? k_proj_res<2> : cpt == 3 ? k_proj_res<3> : cpt == 4 ? k_proj_res<4> : k_proj_res<5>;
}

// The tile of the resident solver: at most one block per SM, a block's cells in
// PJ_RES_THREADS threads of at most five rows and its arrays in shared memory.  Fewest
// cells per block first (an iteration's work), but no fewer than `least`: below
// that the exchange grows with every block and the work is hidden (at 96x48
// cells 2.6 us per iteration with at least 256, 3.3 with 128, 2.9 with 512).
bool proj_res_tile(int nx, int ny, int sms, size_t smem_max, int least, ProjTile& best) {
  best = ProjTile{};
  for (int nty = 1; nty <= ny; ++nty)
    for (int ntx = 1; ntx <= nx && ntx * nty <= std::min(sms, 32 * WORD_CHUNKS); ++ntx) {
      ProjTile t{};
      t.x = (nx + ntx - 1) / ntx;
      t.y = (ny + nty - 1) / nty;
      // no empty tiles; a halo may reach past the next tile, every block waits for all sums
      t.tiles_x = (nx + t.x - 1) / t.x;
      t.tiles_y = (ny + t.y - 1) / t.y;
      if (t.x > PJ_RES_THREADS) continue;
      t.cpt = 1;
      while (t.cpt <= 5 && t.x * ((t.y + t.cpt - 1) / t.cpt) > PJ_RES_THREADS) ++t.cpt;
      if (t.cpt > 5) continue;
      t.blocks = t.tiles_x * t.tiles_y;
      t.threads = (t.x * ((t.y + t.cpt - 1) / t.cpt) + 31) / 32 * 32;
      t.smem = proj_res_smem(t.x, t.y);
      if (t.smem > smem_max) continue;
      const int cells = t.x * t.y;
      if (t.blocks > 1 && cells < least) continue;
      const int cost = cells * 8 + t.x + t.y;
      if (best.blocks == 0 || cost < best.x * best.y * 8 + best.x + best.y) best = t;
    }
  return best.blocks > 0;
}

}  // namespace zm
