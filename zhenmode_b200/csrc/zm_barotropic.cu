// Barotropic subcycle of the mode-split step (dynamics/barotropic.py:86-265,
// legacy branch; _subcycle of timestepping/subcycles.py:6-26).
//
// Resident path (k_bt_loop): one cooperative kernel runs all subcycles.  Each
// block owns one tile and keeps its float64 state (eta, ubt, vbt) with a
// two-cell halo, the static fields it stencils over and the forcing of its
// cells in shared memory for the whole loop.  Per subcycle:
//   1  the halo of eta, ubt, vbt from the neighbours' words of the previous
//      subcycle (and the polar cap of the velocities);
//   2  continuity eta* = (eta - dt H div(ubt wm, vbt wm)) wm on the tile and,
//      redundantly, on the four sides of its one-cell ring, so the gradient
//      needs no exchange;
//   3  sponge and relaxation of eta* with their volume refill; (cap active)
//      band-row partial sums, grid barrier, cap of eta*;
//   4  momentum: adjoint gradient of eta*, u* = ubt + dt (-g grad eta* + F),
//      backward-Euler Coriolis, implicit drag, wet mask; the cells within two
//      of the tile's edge publish eta*, u, v as exchange words.
// What bounds the loop is the latency of a subcycle (at 180x90 the work of one
// is 16200 cells).  A block waits only for its neighbours' words: no grid
// barrier, no fence, and a block may run ahead of far ones.  The counter barrier
// and the separate halo loads this replaces took 7.3 us per subcycle at every
// grid size up to 360x180 (9.5 at 720x360); a subcycle takes 2.0 us at 180x90,
// 3.2 at 360x180 and 4.7 at 720x360.  Grids between 300 and 405 thousand
// cells streamed before (three launches per subcycle, 0.49 ms at 800x400; now 0.165).
// An active polar cap keeps two counter barriers a subcycle: a whole step 0.50 ms at
// 90x45x15 (0.81 with the tiles and loads this replaces), 0.95 at 360x180x20 (1.18).
// The polar cap (numerics/horizontal.py:387-451) needs the wet-point zonal mean
// of each band row; blocks write per-tile partial row sums and every reader
// folds them in tile order, so the result does not depend on timing.  When no
// band row has a wet point the cap is the identity and its steps are skipped.
//
// Streaming path (k_bt_eta / k_bt_vel / k_cap2d): for grids whose tiles cannot
// all be resident, three plain kernels per subcycle in the same arithmetic.
//
// Every grid barrier polls with a bounded count; if it runs out the kernel
// records ZM_BT_ERR_BARRIER in *err and every block returns.
#include "zm_kernels.cuh"
#include "zm_sync.cuh"

namespace zm {

namespace {

// band-row index of row j (0..2nb-1), or -1 outside the cap bands
__device__ __forceinline__ int band_of(int ny, int nb, int j) {
  if (nb <= 0) return -1;
  if (j < nb) return j;
  if (j >= ny - nb) return j - (ny - 2 * nb);
  return -1;
}

// Backward-Euler Coriolis with the implicit linear drag
// (barotropic.py:86-265): u = (u* + fd v*) drag / (1 + fd^2), fd = f dt_bt.
// The factor drag / (1 + fd^2) is static per cell; both paths form it here.
__device__ __forceinline__ double bt_drag_factor(double fd, double drag) { return drag / (1.0 + fd * fd); }

constexpr int BT_H = 2;      // halo width
constexpr int BT_HS = 2;     // halo words per thread held ready
constexpr int BT_FIELDS = 3; // eta, ubt, vbt

// item flags: open faces, wet cell, owned cell, owned cell within two of the tile's edge
constexpr unsigned BT_E = 1u, BT_W = 2u, BT_N = 4u, BT_S = 8u, BT_WET = 16u, BT_OWN = 32u, BT_PUB = 64u, BT_LIVE = 128u;
constexpr int BT_ROW = 8;    // above the flags: the cell's padded row

struct BtFixed {  // the part of a block's shared memory whose size does not depend on the tile
  double mean[3][2 * ZM_BT_MAX_NB];  // band-row means: eta*, u, v
  double red[32];
  double part[WORD_CHUNKS];
  double tot;
};

}  // namespace

// Shared memory of a tile of tx x ty cells: eta, ubt, vbt, 1/dx on the padded
// tile, forcing and Coriolis factors of the owned cells, row factors, wet flags.
size_t bt_tile_smem(int tx, int ty) {
  const size_t pad = (size_t)(tx + 2 * BT_H) * (ty + 2 * BT_H), own = (size_t)tx * ty;
  return sizeof(BtFixed) + sizeof(double) * (4 * pad + 4 * own + 3 * (size_t)(ty + 2 * BT_H)) + (pad + 7) / 8 * 8;
}

// K: cells of continuity (tile and ring sides) per thread.
template <int K>
__global__ void __launch_bounds__(BT_THREADS, 1) k_bt_loop(Dev d, BtArgs a) {
  extern __shared__ double bt_smem[];
  const int tx = a.tile_x, ty = a.tile_y, PX = tx + 2 * BT_H, PY = ty + 2 * BT_H, PP = PX * PY;
  BtFixed& sh = *reinterpret_cast<BtFixed*>(bt_smem);
  double* E = bt_smem + sizeof(BtFixed) / sizeof(double);  // eta, then eta*
  double* U = E + PP;
  double* V = U + PP;
  double* ixs = V + PP;             // 1/dx
  double* fxs = ixs + PP;           // owned cells: forcing, f dt, drag / (1 + (f dt)^2)
  double* fys = fxs + tx * ty;
  double* fds = fys + tx * ty;
  double* rds = fds + tx * ty;
  double* iyc = rds + tx * ty;      // rows: 1 / (dy cos), cosine of the north and the south face
  double* cfp = iyc + PY;
  double* cfm = cfp + PY;
  unsigned char* wet = reinterpret_cast<unsigned char*>(cfm + PY);
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const unsigned nblocks = gridDim.x;
  const int bx = blockIdx.x % a.ntx, by = blockIdx.x / a.ntx;
  const int i0 = bx * tx, j0 = by * ty;
  const int w_own = min(tx, d.nx - i0), h_own = min(ty, d.ny - j0), n_own = w_own * h_own;
  const bool cap = a.cap_active != 0;
  if (cap) grid_barrier_begin(a.bar);
  auto wrap = [&](int i) {
    i %= d.nx;
    return i < 0 ? i + d.nx : i;
  };
  // ---- static fields and the initial state on the padded tile; beyond the walls only zero masks
  for (int r = tid; r < PY; r += nt) {
    const int j = min(max(j0 - BT_H + r, 0), d.ny - 1);
    iyc[r] = d.inv_dy_d / (double)__ldg(d.cosl + j);
    cfp[r] = (double)__ldg(d.cfp + j);
    cfm[r] = (double)__ldg(d.cfm + j);
  }
  for (int e = tid; e < PP; e += nt) {
    const int r = e / PX - BT_H, c = e - (r + BT_H) * PX - BT_H, j = j0 + r;
    const bool in = j >= 0 && j < d.ny && r < h_own + BT_H && c < w_own + BT_H;
    const int g = in ? idx2(d, j, wrap(i0 + c)) : 0;
    E[e] = in ? (double)__ldg(a.eta_in + g) : 0.0;
    U[e] = in ? a.ubt0[g] : 0.0;
    V[e] = in ? a.vbt0[g] : 0.0;
    ixs[e] = in ? __ldg(d.inv_dx_d + g) : 0.0;
    wet[e] = in && __ldg(d.wet2 + g) != 0.f;
  }
  const double fscale = 1.0 / (1025.0 * (double)d.H_sw);
  for (int e = tid; e < n_own; e += nt) {
    const int r = e / w_own, c = e - r * w_own, g = idx2(d, j0 + r, i0 + c);
    // total barotropic forcing F_rho + tau / (rho0 H)
    fxs[e] = (double)a.frx[g] + (double)__ldg(d.tau_x + g) * fscale;
    fys[e] = (double)a.fry[g] + (double)__ldg(d.tau_y + g) * fscale;
    const double fd = __ldg(d.fcor_d + g) * a.dtb;
    fds[e] = fd;
    rds[e] = bt_drag_factor(fd, a.drag);
  }
  __syncthreads();
  // ---- this thread's cells: the owned ones first, then the ring's sides
  const int n_eta = n_own + 2 * (w_own + h_own);
  int at[K], gi[K];
  unsigned fl[K];
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const int e = tid + q * nt;
    at[q] = 0;
    gi[q] = 0;
    fl[q] = 0u;
    if (e >= n_eta) continue;
    int r, c;
    if (e < n_own) {
      r = e / w_own;
      c = e - r * w_own;
    } else {
      const int m = e - n_own;
      if (m < 2 * h_own) {
        r = m % h_own;
        c = m < h_own ? -1 : w_own;
      } else {
        c = (m - 2 * h_own) % w_own;
        r = m - 2 * h_own < w_own ? -1 : h_own;
      }
    }
    const int j = j0 + r;
    if (j < 0 || j >= d.ny) continue;
    const int o = (r + BT_H) * PX + c + BT_H;
    at[q] = o;
    gi[q] = idx2(d, j, wrap(i0 + c));
    unsigned f = BT_LIVE | (unsigned)(r + BT_H) << BT_ROW;
    if (wet[o]) {
      f |= BT_WET;
      if (wet[o + 1]) f |= BT_E;
      if (wet[o - 1]) f |= BT_W;
      if (j < d.ny - 1 && wet[o + PX]) f |= BT_N;
      if (j > 0 && wet[o - PX]) f |= BT_S;
    }
    if (e < n_own) {
      f |= BT_OWN;
      if (r < BT_H || r >= h_own - BT_H || c < BT_H || c >= w_own - BT_H) f |= BT_PUB;
    }
    fl[q] = f;
  }
  // ---- the halo words the stencils read: eta on the ring's sides, u and v there
  // and on its corners, u two columns and v two rows out.  Word h as its place
  // (field * PP + cell) in shared memory and its index (field * plane + cell)
  const int n_halo = 8 * (w_own + h_own) + 8;
  auto halo_word = [&](int h, int& place, long long& index) {
    if (h >= n_halo) return false;
    int r, c, f;
    if (h < 8 * h_own) {  // west, east: eta, u, v at distance 1, u at distance 2
      const int s = h / h_own, k = s >> 1;
      r = h - s * h_own;
      const int dist = k == 3 ? 2 : 1;
      c = (s & 1) ? w_own - 1 + dist : -dist;
      f = k == 3 ? 1 : k;
    } else if (h < 8 * (h_own + w_own)) {  // south, north: eta, u, v at distance 1, v at distance 2
      const int m = h - 8 * h_own, s = m / w_own, k = s >> 1;
      c = m - s * w_own;
      const int dist = k == 3 ? 2 : 1;
      r = (s & 1) ? h_own - 1 + dist : -dist;
      f = k == 3 ? 2 : k;
    } else {  // corners: u and v
      const int m = h - 8 * (h_own + w_own);
      r = (m & 1) ? h_own : -1;
      c = (m & 2) ? w_own : -1;
      f = 1 + (m >> 2);
    }
    const int j = j0 + r;
    if (j < 0 || j >= d.ny) return false;
    place = f * PP + (r + BT_H) * PX + c + BT_H;
    index = f * d.plane + idx2(d, j, wrap(i0 + c));
    return true;
  };
  int hp[BT_HS];
  long long hx[BT_HS];
#pragma unroll
  for (int s = 0; s < BT_HS; ++s)
    if (!halo_word(tid + s * nt, hp[s], hx[s])) hp[s] = -1;
  Word* const words = reinterpret_cast<Word*>(a.pub);
  const long long set = BT_FIELDS * d.plane;
  const unsigned long long base = *a.seq;  // k_final advances it when every block is done
  unsigned long long sums = base;  // sequence number of the last grid-wide sum

  // Sum over the grid, the same bits in every block: each block stores its
  // partial sum into every block's own list (one copy per reader: a single
  // list would be a few cache lines that all blocks poll).
  auto grid_sum = [&](double v, double& out) {
    ++sums;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) sh.red[warp] = v;
    __syncthreads();
    if (warp == 0) {
      double x = lane < nw ? sh.red[lane] : 0.0;
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) sh.tot = x;
    }
    __syncthreads();
    Word* lists = reinterpret_cast<Word*>(a.sums) + (size_t)(sums & 1) * nblocks * nblocks;
    for (int t = tid; t < (int)nblocks; t += nt) st_word(lists + (size_t)t * nblocks + blockIdx.x, sh.tot, sums);
    bool ok = true;
    const int chunks = ((int)nblocks + 31) / 32;
    for (int c = warp; c < chunks; c += nw) {
      const int b = 32 * c + lane;
      double y = 0.0;
      if (b < (int)nblocks) ok = wait_word(lists + (size_t)blockIdx.x * nblocks + b, sums, a.err, a.max_polls, y) && ok;
      __syncwarp();
      for (int o = 16; o > 0; o >>= 1) y += __shfl_down_sync(0xffffffffu, y, o);
      if (lane == 0) sh.part[c] = y;
    }
    if (__syncthreads_or(!ok)) return false;
    out = sh.part[0];
    for (int c = 1; c < chunks; ++c) out += sh.part[c];
    return true;
  };
  // Decay of eta* by fac on the tile and its ring with the uniform refill of
  // the removed volume (barotropic.py:22-31).
  auto refill = [&](const double* fac) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (fl[q] & BT_OWN) {
        const double e0 = E[at[q]];
        s += a.area[gi[q]] * (e0 * fac[gi[q]] - e0);
      }
    double dv;
    if (!grid_sum(s, dv)) return false;
    const double shift = -dv / a.ocean;
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (fl[q] & BT_LIVE) E[at[q]] = E[at[q]] * fac[gi[q]] + ((fl[q] & BT_WET) ? shift : 0.0);
    __syncthreads();
    return true;
  };
  // wet-point partial sums of a padded field over the owned cells of each band row, one warp per row
  auto band_partials = [&](const double* f, double* part) {
    for (int r = warp; r < h_own; r += nw) {
      const int b = band_of(d.ny, a.nb, j0 + r);
      if (b < 0) continue;
      double s = 0.0;
      for (int c = lane; c < w_own; c += 32) {
        const int o = (r + BT_H) * PX + c + BT_H;
        if (wet[o]) s += f[o];
      }
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) part[b * a.ntx + bx] = s;
    }
  };
  auto band_means = [&](int q, const double* part) {
    for (int b = tid; b < 2 * a.nb; b += nt) {
      double s = 0.0;
      for (int t = 0; t < a.ntx; ++t) s += __ldcg(part + b * a.ntx + t);
      sh.mean[q][b] = s / a.count[b];
    }
  };
  // polar-cap blend of value f at row j
  auto cap_val = [&](int q, int j, bool w, double f) {
    const int b = band_of(d.ny, a.nb, j);
    if (b < 0) return f;
    const double wt = (double)a.wts[b < a.nb ? b : 2 * a.nb - 1 - b], m = w ? 1.0 : 0.0;
    return wt * (sh.mean[q][b] * m) + (1.0 - wt) * (f * m);
  };

  const double g9 = 9.81;
  for (int n = 0; n < a.nsub; ++n) {
    const int pout = n & 1;
    if (n > 0) {
      // 1: halo from the neighbours' words; caps on every cell
      const unsigned long long seq = base + n;
      const Word* in = words + (seq & 1) * set;
      bool ok = true;
#pragma unroll
      for (int s = 0; s < BT_HS; ++s)
        if (hp[s] >= 0) ok = wait_word(in + hx[s], seq, a.err, a.max_polls, E[hp[s]]) && ok;
      for (int h = tid + BT_HS * nt; h < n_halo && ok; h += nt) {
        int place;
        long long index;
        if (halo_word(h, place, index)) ok = wait_word(in + index, seq, a.err, a.max_polls, E[place]);
      }
      if (cap) {
        band_means(1, a.part_u[pout ^ 1]);
        band_means(2, a.part_v[pout ^ 1]);
      }
      if (__syncthreads_or(!ok)) return;
      if (cap) {
        for (int e = tid; e < PP; e += nt) {
          const int r = e / PX - BT_H, j = j0 + r;
          if (j < 0 || j >= d.ny || r >= h_own + BT_H) continue;
          U[e] = cap_val(1, j, wet[e], U[e]);
          V[e] = cap_val(2, j, wet[e], V[e]);
        }
        __syncthreads();
      }
    }
    // 2: continuity (numerics/horizontal.py:69-97 flux form); a cell reads its own eta only
#pragma unroll
    for (int q = 0; q < K; ++q) {
      const unsigned f = fl[q];
      if (!(f & BT_LIVE)) continue;
      const int o = at[q];
      double en = 0.0;
      if (f & BT_WET) {
        const int r = (int)(f >> BT_ROW);
        const double uc = U[o], vc = V[o];
        const double fe = (f & BT_E) ? 0.5 * (uc + U[o + 1]) : 0.0;
        const double fw = (f & BT_W) ? 0.5 * (U[o - 1] + uc) : 0.0;
        const double fn = (f & BT_N) ? 0.5 * (vc + V[o + PX]) * cfp[r] : 0.0;
        const double fs = (f & BT_S) ? 0.5 * (V[o - PX] + vc) * cfp[r - 1] : 0.0;
        en = E[o] - a.dtH * ((fe - fw) * ixs[o] + (fn - fs) * iyc[r]);
      }
      E[o] = en;
    }
    __syncthreads();
    // 2b: lateral sponge, then eta relaxation, each with its volume refill
    if (a.sponge && !refill(a.es)) return;
    if (a.relax && !refill(a.er)) return;
    // 3: polar cap of eta*
    if (cap) {
      band_partials(E, a.part_e[pout]);
      if (!grid_barrier(a.bar, a.err, nblocks, a.max_polls)) return;
      band_means(0, a.part_e[pout]);
      __syncthreads();
#pragma unroll
      for (int q = 0; q < K; ++q)
        if (fl[q] & BT_LIVE) E[at[q]] = cap_val(0, j0 + (int)(fl[q] >> BT_ROW) - BT_H, fl[q] & BT_WET, E[at[q]]);
      __syncthreads();
    }
    // 4: momentum on the owned cells; publish eta*, u, v along the edges
    const unsigned long long seq = base + n + 1;
    Word* out = words + (seq & 1) * set;
    const bool more = n + 1 < a.nsub;
#pragma unroll
    for (int q = 0; q < K; ++q) {
      const unsigned f = fl[q];
      if (!(f & BT_OWN)) continue;
      const int o = at[q], e = tid + q * nt;
      double un = 0.0, vn = 0.0;
      const double e0 = E[o];
      if (f & BT_WET) {
        const int r = (int)(f >> BT_ROW);
        const double de = (f & BT_E) ? E[o + 1] - e0 : 0.0, dw = (f & BT_W) ? e0 - E[o - 1] : 0.0;
        const double dn = (f & BT_N) ? (E[o + PX] - e0) * cfp[r] : 0.0, ds = (f & BT_S) ? (e0 - E[o - PX]) * cfm[r] : 0.0;
        const double gx = ixs[o] * 0.5 * (de + dw);
        const double gy = iyc[r] * 0.5 * (dn + ds);
        const double us = U[o] + a.dtb * (-g9 * gx + fxs[e]);
        const double vs = V[o] + a.dtb * (-g9 * gy + fys[e]);
        const double fd = fds[e], rd = rds[e];
        un = (us + fd * vs) * rd;
        vn = (vs - fd * us) * rd;
        if (a.sponge) {
          un *= a.es[gi[q]];
          vn *= a.es[gi[q]];
        }
      }
      U[o] = un;
      V[o] = vn;
      if ((f & BT_PUB) && more) {
        st_word(out + gi[q], e0, seq);
        st_word(out + d.plane + gi[q], un, seq);
        st_word(out + 2 * d.plane + gi[q], vn, seq);
      }
    }
    __syncthreads();  // the halo is overwritten next
    if (cap) {
      band_partials(U, a.part_u[pout]);
      band_partials(V, a.part_v[pout]);
      if (!grid_barrier(a.bar, a.err, nblocks, a.max_polls)) return;
    }
  }
  // ---- outputs: capped velocities and the float32 free surface
  if (cap) {
    const int plast = (a.nsub - 1) & 1;
    band_means(1, a.part_u[plast]);
    band_means(2, a.part_v[plast]);
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < K; ++q) {
    if (!(fl[q] & BT_OWN)) continue;
    const int o = at[q];
    double u = U[o], v = V[o];
    if (cap) {
      const int j = j0 + (int)(fl[q] >> BT_ROW) - BT_H;
      u = cap_val(1, j, fl[q] & BT_WET, u);
      v = cap_val(2, j, fl[q] & BT_WET, v);
    }
    a.ubt_out[gi[q]] = u;
    a.vbt_out[gi[q]] = v;
    a.eta_out[gi[q]] = (float)E[o];
  }
}

// After a launch that may have given up: the sequence numbers move past every
// word that it may have left (a launch has fewer than 2^33 exchanges, and
// 2^31 of these fit in a number), the barrier and error words are cleared.
// Thread 0 for the loop, thread 1 for the projection; null: none.
__global__ void k_sync_reset(unsigned long long* bt_seq, unsigned* bt_sync, unsigned long long* pj_seq,
                             unsigned* pj_sync) {
  unsigned long long* seq = threadIdx.x == 0 ? bt_seq : pj_seq;
  unsigned* sync = threadIdx.x == 0 ? bt_sync : pj_sync;
  if (seq) *seq += 1ull << 33;
  if (sync)
    for (int q = 0; q < 4; ++q) sync[q] = 0u;
}

void (*bt_loop_kernel(int k))(Dev, BtArgs) {
  return k <= 1 ? k_bt_loop<1> : k == 2 ? k_bt_loop<2> : k == 3 ? k_bt_loop<3> : k_bt_loop<4>;
}

// The tile of the resident kernel: at most one block per SM, its cells and ring
// sides on BT_THREADS threads of at most four, its arrays in shared memory.
// Fewest cells per block, but no fewer than `least`; blocks 0 if none fits.
BtTile bt_tile(int nx, int ny, int sms, size_t smem_max, int least) {
  BtTile best{};
  for (int nty = 1; nty <= ny; ++nty)
    for (int ntx = 1; ntx <= nx && ntx * nty <= min(sms, 32 * WORD_CHUNKS); ++ntx) {
      BtTile t{};
      t.x = (nx + ntx - 1) / ntx;
      t.y = (ny + nty - 1) / nty;
      t.tiles_x = (nx + t.x - 1) / t.x;
      t.blocks = t.tiles_x * ((ny + t.y - 1) / t.y);
      const int cells = t.x * t.y, n_eta = cells + 2 * (t.x + t.y);
      t.k = (n_eta + BT_THREADS - 1) / BT_THREADS;
      if (t.k > 4 || (t.blocks > 1 && cells < least)) continue;
      t.threads = ((n_eta + t.k - 1) / t.k + 31) / 32 * 32;
      t.smem = bt_tile_smem(t.x, t.y);
      if (t.smem > smem_max) continue;
      if (best.blocks == 0 || 8 * cells + t.x + t.y < 8 * best.x * best.y + best.x + best.y) best = t;
    }
  return best;
}

// ---- streaming path: one subcycle as three plain kernels

__global__ void __launch_bounds__(256) k_bt_eta(Dev d, const double* __restrict__ eta, const double* __restrict__ ubt,
                                                const double* __restrict__ vbt, double* __restrict__ eta_o,
                                                double dtH) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= d.nx || j >= d.ny) return;
  const int c = idx2(d, j, i), ce = idx2(d, j, east(d, i)), cw = idx2(d, j, west(d, i));
  const double w0 = __ldg(d.wet2 + c), we = __ldg(d.wet2 + ce), ww = __ldg(d.wet2 + cw);
  const double u0 = ubt[c] * w0, ue = ubt[ce] * we, uw = ubt[cw] * ww;
  const double fe = 0.5 * (u0 + ue) * (w0 * we);
  const double fw = 0.5 * (uw + u0) * (ww * w0);
  const double div_x = (fe - fw) * __ldg(d.inv_dx_d + c);
  double fn = 0.0, fs = 0.0;
  const double v0 = vbt[c] * w0;
  if (j < d.ny - 1) {
    const int cn = idx2(d, j + 1, i);
    const double wn = __ldg(d.wet2 + cn);
    fn = 0.5 * (v0 + vbt[cn] * wn) * (w0 * wn) * (double)__ldg(d.cfp + j);
  }
  if (j > 0) {
    const int cs = idx2(d, j - 1, i);
    const double ws = __ldg(d.wet2 + cs);
    fs = 0.5 * (vbt[cs] * ws + v0) * (ws * w0) * (double)__ldg(d.cfp + j - 1);
  }
  const double div = div_x + (fn - fs) * (d.inv_dy_d / (double)__ldg(d.cosl + j));
  eta_o[c] = (eta[c] - dtH * div) * w0;
}

__global__ void __launch_bounds__(256) k_bt_vel(Dev d, const double* __restrict__ eta, const double* __restrict__ ubt,
                                                const double* __restrict__ vbt, const double* __restrict__ Fx,
                                                const double* __restrict__ Fy, double* __restrict__ ubt_o,
                                                double* __restrict__ vbt_o, double dtb, double drag,
                                                const double* __restrict__ sv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= d.nx || j >= d.ny) return;
  const int c = idx2(d, j, i), ce = idx2(d, j, east(d, i)), cw = idx2(d, j, west(d, i));
  const double w0 = __ldg(d.wet2 + c), we = __ldg(d.wet2 + ce), ww = __ldg(d.wet2 + cw);
  const double e0 = eta[c];
  const double gx = __ldg(d.inv_dx_d + c) * 0.5 * ((eta[ce] - e0) * (w0 * we) + (e0 - eta[cw]) * (w0 * ww));
  double dyp = 0.0, dym = 0.0;
  if (j < d.ny - 1) {
    const int cn = idx2(d, j + 1, i);
    dyp = (eta[cn] - e0) * (w0 * __ldg(d.wet2 + cn)) * (double)__ldg(d.cfp + j);
  }
  if (j > 0) {
    const int cs = idx2(d, j - 1, i);
    dym = (e0 - eta[cs]) * (w0 * __ldg(d.wet2 + cs)) * (double)__ldg(d.cfm + j);
  }
  const double gy = (d.inv_dy_d / (double)__ldg(d.cosl + j)) * 0.5 * (dyp + dym);
  const double us = ubt[c] + dtb * (-9.81 * gx + Fx[c]);
  const double vs = vbt[c] + dtb * (-9.81 * gy + Fy[c]);
  const double fd = __ldg(d.fcor_d + c) * dtb, rd = bt_drag_factor(fd, drag);
  double un = (us + fd * vs) * rd * w0;
  double vn = (vs - fd * us) * rd * w0;
  if (sv) {
    un *= sv[c];
    vn *= sv[c];
  }
  ubt_o[c] = un;
  vbt_o[c] = vn;
}

// Uniform refill of the volume a decay removes (barotropic.py:22-31), streaming
// path: per-block partial sums of area (eta f - eta) ...
__global__ void __launch_bounds__(256) k_refill_part(Dev d, const double* __restrict__ eta,
                                                     const double* __restrict__ fac,
                                                     const double* __restrict__ area, double* __restrict__ part) {
  __shared__ double red[256];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int t = threadIdx.y * blockDim.x + threadIdx.x;
  double s = 0.0;
  if (i < d.nx && j < d.ny) {
    const int c = idx2(d, j, i);
    const double e0 = eta[c];
    s = area[c] * (e0 * fac[c] - e0);
  }
  red[t] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (t < o) red[t] += red[t + o];
    __syncthreads();
  }
  if (t == 0) part[blockIdx.y * gridDim.x + blockIdx.x] = red[0];
}

// ... then every block folds the partials in the same order and applies
// eta f + (-dV / ocean_area) wet.
__global__ void __launch_bounds__(256) k_refill_apply(Dev d, double* __restrict__ eta, const double* __restrict__ fac,
                                                      const double* __restrict__ part, int nparts, double ocean) {
  __shared__ double red[256];
  const int t = threadIdx.y * blockDim.x + threadIdx.x;
  double s = 0.0;
  for (int b = t; b < nparts; b += 256) s += part[b];
  red[t] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (t < o) red[t] += red[t + o];
    __syncthreads();
  }
  const double shift = -red[0] / ocean;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= d.nx || j >= d.ny) return;
  const int c = idx2(d, j, i);
  eta[c] = eta[c] * fac[c] + shift * (double)__ldg(d.wet2 + c);
}

// Polar cap of up to two 2-D float64 fields in place: one block per band row,
// blockIdx.y selects the field.
__global__ void __launch_bounds__(256) k_cap2d(Dev d, double* f0, double* f1, const float* __restrict__ wts,
                                               const double* __restrict__ count, int nb_rows) {
  __shared__ double red[256];
  const int r = blockIdx.x;  // 0..2*nb_rows-1
  double* f = blockIdx.y == 0 ? f0 : f1;
  if (!f) return;
  const int j = r < nb_rows ? r : d.ny - 2 * nb_rows + r;
  const double wt = (double)(r < nb_rows ? wts[r] : wts[2 * nb_rows - 1 - r]);
  double s = 0.0;
  for (int i = threadIdx.x; i < d.nx; i += blockDim.x) s += f[idx2(d, j, i)] * (double)__ldg(d.wet2 + idx2(d, j, i));
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  const double mean = red[0] / count[r];
  for (int i = threadIdx.x; i < d.nx; i += blockDim.x) {
    const double w = __ldg(d.wet2 + idx2(d, j, i));
    const double val = f[idx2(d, j, i)] * w;
    f[idx2(d, j, i)] = wt * (mean * w) + (1.0 - wt) * val;
  }
}

__global__ void __launch_bounds__(256) k_eta_to_float(Dev d, const double* __restrict__ e64, float* __restrict__ e32) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i < d.nx && j < d.ny) e32[idx2(d, j, i)] = (float)e64[idx2(d, j, i)];
}

// Barrier probe for the timeout path: `expected` arrivals are awaited but only
// gridDim.x blocks arrive, so with expected > gridDim.x every block gives up
// after max_polls polls and records ZM_BT_ERR_BARRIER.
__global__ void k_barrier_probe(unsigned* bar, unsigned* err, unsigned expected, unsigned max_polls) {
  grid_barrier_begin(bar);
  grid_barrier(bar, err, expected, max_polls);
}

}  // namespace zm
