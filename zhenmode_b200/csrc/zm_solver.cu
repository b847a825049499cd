// Host side of the B200 global ocean step: parameter derivation, device
// buffers, the kernel sequence of one step, CUDA-graph replay and the C ABI
// declared in include/zm_b200.h.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/zm_b200.h"
#include "zm_kernels.cuh"
#include "zm_staging.cuh"

using namespace zm;

namespace {

constexpr double kOmega = 7.2921e-5;
constexpr double kREarth = 6371.0e3;
constexpr double kPi = 3.14159265358979323846;

struct Err {
  int code;
  std::string msg;
};

#define ZM_CUDA(call)                                                             \
  do {                                                                            \
    cudaError_t e__ = (call);                                                     \
    if (e__ != cudaSuccess) throw Err{ZM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e__)}; \
  } while (0)

struct Fields4 {
  float *u = nullptr, *v = nullptr, *T = nullptr, *S = nullptr;
};

}  // namespace

struct zm_solver {
  Dev d{};
  int device = 0;
  int nx = 0, ny = 0, nz = 0, P = 0;
  size_t n2 = 0, n3 = 0;
  int n_subcyc = 1, n_nu = 1, adv_nsub = 1, conv_nsub = 1;
  double dt = 0, dt_bt = 0;
  int cap_rows = 0, cap_nb = 0;
  int vdiff = 0, freeze = 0;
  float bottom_decay = 1.f;
  double bt_drag = 1.0;
  FftPlan fft{};
  int fft_lines = 1;
  size_t fft_smem = 0;
  std::vector<void*> allocs;
  size_t bytes = 0;
  // resident states (ping-pong) and their free surfaces
  Fields4 st[2];
  float* eta[2] = {nullptr, nullptr};
  int cur = 0;
  // work fields
  // A dry point's T and S below its column's deepest wet level are not written in
  // s1, s2 and the tracer work fields of the N step, and their rates, Fz and the
  // filtered advection keep the 0 they were allocated with; no wet point reads them
  // with a weight.  So only the step's kernels write those fields: states from
  // outside it (diagnostics, closure rows) go to L.
  Fields4 s1, s2, W1, W2, L;
  float *Fz = nullptr, *Ayu = nullptr, *Ayv = nullptr, *Au = nullptr, *Av = nullptr;
  float *accT = nullptr, *accS = nullptr, *TsA = nullptr, *SsA = nullptr, *TsB = nullptr, *SsB = nullptr;
  float *dT1 = nullptr, *dS1 = nullptr, *Tp = nullptr, *Sp = nullptr, *Pu = nullptr, *Pv = nullptr;
  float *gsx = nullptr, *gsy = nullptr;  // pressure-gradient scratch
  float *pfx = nullptr, *pfy = nullptr;  // its depth mean per column
  // budget snapshot: cell areas (reference layout), node thicknesses, partials
  double *area64 = nullptr, *width64 = nullptr, *bpart = nullptr, *bout = nullptr;
  int bblocks = 0;
  // learned vertical-mixing closure (off until zm_set_closure)
  int nu_halo = NB_T;            // nu_h subcycles per pass (autotuned)
  int nu_warps = 8;              // warps (tile rows / NB_R) of the nu_h tiles (autotuned)
  bool want_tune = false;
  bool tuned = false;
  bool closure_on = false;
  MlpTc cw{};
  float* kappa3 = nullptr;       // [nz-1][ny][P] diffusivity per interface
  unsigned* cl_count = nullptr;  // [0] fallback columns of the last step, [1] tensor-core wait errors
  float cl_bound = 8.f;
  // FP64 stage/source ledger (zm_ledger_step): buffers allocated on first use
  bool ledger_on = false;
  double *led_acc = nullptr, *led_part = nullptr, *led_area = nullptr, *led_dzn = nullptr, *led_norms = nullptr;
  float *led_convT = nullptr, *led_convS = nullptr, *led_topT = nullptr, *led_topS = nullptr;
  // lateral sponge of the linear half step (null when off): decay per column, targets as anomalies
  float *sp_dec = nullptr, *sp_Tc = nullptr, *sp_Sc = nullptr;
  // column-divergence projection of the stage-2 advective velocity (off unless project_adv_vel)
  bool proj_on = false;
  ProjArgs pj{};
  int pj_blocks = 0;
  ProjTile pj_tile{};   // resident form of the solves (blocks 0: the grid does not fit)
  double pj_dtg = 0.0;
  double *pj_dzn = nullptr, *pj_cos = nullptr, *pj_area = nullptr;
  float *up = nullptr, *vp = nullptr;
  float *frx = nullptr, *fry = nullptr, *means = nullptr, *wts = nullptr;
  double *ubt0 = nullptr, *vbt0 = nullptr, *ubt[2] = {nullptr, nullptr}, *vbt[2] = {nullptr, nullptr};
  double *eta64[2] = {nullptr, nullptr}, *Fx = nullptr, *Fy = nullptr, *wts_d = nullptr;
  BtArgs bt{};          // persistent barotropic kernel arguments
  int bt_blocks = 0;
  BtTile btt{};
  unsigned long long* bt_seq = nullptr;  // sequence number of the loop's exchange words
  unsigned* bt_sync = nullptr;  // [0..1] barrier counter/generation, [2] error flags
  // reference-layout staging (zm_step_host)
  Fields4 ref;
  float* ref_eta = nullptr;
  // mutable forcing fields
  float *tau_x = nullptr, *tau_y = nullptr, *qheat = nullptr;
  unsigned int* flags = nullptr;  // [0] the classification zm_status reports, [1] that of the last step's result
  cudaStream_t cap_stream = nullptr;  // graphs are captured here, launched on the caller's stream
  cudaStream_t side = nullptr;        // the second branch of the N step (momentum advection)
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  // host-buffer steps: the copies run on their own stream, one event per field
  // each way, so that a field's layout change overlaps the next field's copy
  cudaStream_t copy_stream = nullptr;
  HostStage stage;  // pinned slots of zm_step_host for pageable arrays
  cudaEvent_t ev_copy[11] = {};
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  bool graphs_ready = false;
  unsigned graphs_built = 0;  // captures so far: who holds a copy of the step compares it
  // set while an ensemble captures this member: the cooperative barotropic
  // kernel waits for bt_wait and records bt_done, so that the members'
  // grid-barrier kernels never run at the same time
  cudaEvent_t bt_wait = nullptr, bt_done = nullptr;
  int kernels_per_step = 0;
  std::string last_error;
  // launch accounting: every kernel launch of the step is bracketed by
  // pb()/pe(); with profiling on, CUDA events time each launch class
  int launch_count = 0;
  bool profiling = false;
  struct ProfEv { int cls; cudaEvent_t a, b; };
  std::vector<ProfEv> prof;
  void pb(int cls, cudaStream_t s) {
    ++launch_count;
    if (!profiling) return;
    ProfEv e{cls, nullptr, nullptr};
    ZM_CUDA(cudaEventCreate(&e.a));
    ZM_CUDA(cudaEventCreate(&e.b));
    ZM_CUDA(cudaEventRecord(e.a, s));
    prof.push_back(e);
  }
  void pe(cudaStream_t s) {
    if (profiling) ZM_CUDA(cudaEventRecord(prof.back().b, s));
  }

  // Zeroed device memory.  Small arrays come from shared pieces of 16 MB: a
  // handle holds some eighty arrays, and one cudaMalloc and cudaMemset each
  // were most of the time to create one for a small grid.
  char* piece = nullptr;
  size_t piece_left = 0;
  template <class T>
  T* alloc(size_t count) {
    constexpr size_t PIECE = 16u << 20;
    const size_t need = (std::max<size_t>(count, 1) * sizeof(T) + 255) / 256 * 256;
    if (need > piece_left) {
      void* p = nullptr;
      const size_t take = std::max(need, PIECE);
      ZM_CUDA(cudaMalloc(&p, take));
      allocs.push_back(p);
      ZM_CUDA(cudaMemset(p, 0, take));
      // waited for: the caller's stream need not wait for the default one.  (On a stream of the handle's own the same
      // work took a hardware queue from the step's two graph branches: eight steps at 180x90x50 3.37 ms for 3.31.)
      ZM_CUDA(cudaStreamSynchronize(nullptr));
      bytes += take;
      if (take - need <= piece_left) return static_cast<T*>(p);  // the current piece has more left
      piece = static_cast<char*>(p);
      piece_left = take;
    }
    T* out = reinterpret_cast<T*>(piece);
    piece += need;
    piece_left -= need;
    return out;
  }
  float* f3() { return alloc<float>(n3); }
  float* f2() { return alloc<float>(n2); }
  Fields4 four() { return Fields4{f3(), f3(), f3(), f3()}; }

  template <class T>
  T* upload(const std::vector<T>& h) {
    T* p = alloc<T>(h.size());
    ZM_CUDA(cudaMemcpy(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
    return p;
  }

  ~zm_solver() {
    for (int g = 0; g < 2; ++g)
      if (graph[g]) cudaGraphExecDestroy(graph[g]);
    if (cap_stream) cudaStreamDestroy(cap_stream);
    if (side) cudaStreamDestroy(side);
    if (ev_fork) cudaEventDestroy(ev_fork);
    if (ev_join) cudaEventDestroy(ev_join);
    if (copy_stream) cudaStreamDestroy(copy_stream);
    for (cudaEvent_t e : ev_copy)
      if (e) cudaEventDestroy(e);
    for (void* p : allocs) cudaFree(p);
  }

  dim3 grid3(dim3 b) const { return dim3((nx + b.x - 1) / b.x, (ny + b.y - 1) / b.y, nz); }
  dim3 grid2(dim3 b) const { return dim3((nx + b.x - 1) / b.x, (ny + b.y - 1) / b.y, 1); }

  void check_launch() {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw Err{ZM_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e)};
  }

  // Set the nu_h launch shape.  Its strip classes are formed on the shape's first
  // use (at creation, between the autotuner's trials) and kept as they are: a
  // captured step holds its shape and the table of that shape, also after the
  // tuner has picked another one (an ensemble's graphs outlive its members' tuning).
  unsigned char* nu_tables[2][NB_T + 1] = {};  // [8 or 16 warps][halo]
  void set_nu_shape(int halo, int warps) {
    nu_halo = halo;
    nu_warps = warps;
    unsigned char*& table = nu_tables[warps == 16][halo];
    if (!table) {
      const dim3 g = nu_grid(d, warps, halo);
      const unsigned strips = g.x * g.y * warps;  // of every level
      table = alloc<unsigned char>((size_t)strips * g.z);
      k_nu_class<<<(strips + 7) / 8, dim3(32, 8)>>>(d, table, warps, halo, (int)g.x, (int)g.y);
      check_launch();
      ZM_CUDA(cudaStreamSynchronize(nullptr));  // any stream sees the table
    }
    d.nu_class = table;
  }

  // Clear the barrier and error words of the barotropic loop and the projection, where a state is loaded.
  // Their sequence numbers move past every word that a launch which gave up may have left behind.
  void reset_sync(cudaStream_t s) {
    k_sync_reset<<<1, 2, 0, s>>>(bt_seq, bt_sync, pj.seq, proj_on ? pj.bar : nullptr);
    check_launch();
  }
  // Poll limit of the waits between their blocks.  The captured steps hold it.
  void set_wait_limit(unsigned polls) { bt.max_polls = pj.max_polls = polls; }

  // ---------------------------------------------------------------- stages
  // Linear half step L(dt/2): src -> dst (dst must not alias src).
  void linear_half(cudaStream_t s, const Fields4& src, const Fields4& dst) {
    const float dth = (float)(dt / 2.0);
    const float* usub = src.u;
    const float* vsub = src.v;
    if (d.nu_h != 0.f) {
      const float dts = (float)(dt / 2.0 / n_nu);
      const float* a = src.u;
      const float* c = src.v;
      int done = 0, pass = 0;
      while (done < n_nu) {
        const int nsub = std::min(nu_halo, n_nu - done);
        const Fields4& o = (pass % 2 == 0) ? W1 : W2;
        pb(ZM_K_NU_SUB, s);
        ZM_CUDA(launch_nu_tb(s, d, nu_warps, a, c, o.u, o.v, dts, nsub, nu_halo, n_nu - done));
        pe(s);
        a = o.u;
        c = o.v;
        done += nsub;
        ++pass;
      }
      usub = a;
      vsub = c;
    }
    pb(ZM_K_LIN_FINISH, s);
    launch_lin_t(s, d, usub, vsub, src.u, src.v, src.T, src.S, dst.u, dst.v, dst.T, dst.S, dth,
                 vdiff || closure_on);
    pe(s);
    if (vdiff || closure_on) {
      pb(ZM_K_IMPLICIT, s);
      ZM_CUDA(launch_implicit_vdiff(s, d, dst.u, dst.v, dst.T, dst.S, src.u, src.v, dth, closure_on ? kappa3 : nullptr));
      pe(s);
    }
    if (ledger_on) led_stage(s, 0, src.T, src.S, nullptr, dst.T, dst.S, nullptr);  // step.py:138-140
    if (sp_dec && ledger_on) {  // step.py:158-161, from the diffused state
      k_led_sponge<<<led_grid(), dim3(32, 8), 0, s>>>(d, dst.T, dst.S, sp_dec, sp_Tc, sp_Sc, led_area, led_dzn,
                                                      led_part);
      const int b = ZM_LED_STAGE + 3;
      led_fold(s, 6, {{ZM_LED_SOURCE + 18, kHeat}, {ZM_LED_SOURCE + 19, kSalt}, {b, kHeat}, {b + 1, kSalt},
                      {ZM_LED_SCALE, kHeat}, {ZM_LED_SCALE + 1, kSalt}});
    }
    if (sp_dec) {  // lateral sponge after the diffusion (step.py:142-156)
      const dim3 c(32, 8);
      pb(ZM_K_LIN_FINISH, s);
      k_sponge<<<grid3(c), c, 0, s>>>(d, dst.u, dst.v, dst.T, dst.S, sp_dec, sp_Tc, sp_Sc);
      pe(s);
    }
    check_launch();
  }

  // Tracer residual at the evaluation state (u, v, T, S) with transport Fz.
  void tracer_residual(cudaStream_t s, int stage, const float* u, const float* v, const float* T, const float* S,
                       const float* Tbase, const float* Sbase, float* To, float* So) {
    const float dts = (float)(dt / adv_nsub);
    const float* cT = T;
    const float* cS = S;
    for (int n = 0; n < adv_nsub; ++n) {
      float* nT = (n % 2 == 0) ? TsA : TsB;
      float* nS = (n % 2 == 0) ? SsA : SsB;
      pb(ZM_K_TRACER_ADV, s);
      launch_tracer_adv(s, d, cT, cS, u, v, Fz, accT, accS, nT, nS, dts, n == 0, n == adv_nsub - 1,
                        ledger_on ? led_topT : nullptr, ledger_on ? led_topS : nullptr);
      pe(s);
      cT = nT;
      cS = nS;
    }
    RestArgs a{T, S, accT, accS, Tbase, Sbase, dT1, dS1, To, So, (float)dt, 1.f / (float)adv_nsub, conv_nsub, stage,
               closure_on ? 1 : 0, ledger_on ? led_convT : nullptr, ledger_on ? led_convS : nullptr};
    pb(ZM_K_TRACER_REST, s);
    launch_tracer_rest(s, d, a);
    pe(s);
    check_launch();
    if (ledger_on) led_rk(s, T, S);  // tendencies.py:211-214
  }

  void pgf(cudaStream_t s, PgfArgs a) {
    a.gsx = gsx;
    a.gsy = gsy;
    a.Fxs = pfx;
    a.Fys = pfy;
    pb(ZM_K_PGF, s);
    launch_pgf(s, d, a);
    pe(s);
    if (a.mode != 0) ++launch_count;  // launch_pgf adds the output pass (k_pgf_out)
    check_launch();
  }

  // T/S-independent part of the momentum residual, A = wm (dealiased
  // advection + surface wind - barotropic wind), into Au/Av.
  void momentum_advection_part(cudaStream_t s, const Fields4& src) {
    pb(ZM_K_FZ, s);
    launch_fz(s, d, src.u, src.v, Fz);
    pe(s);
    momentum_advection_rest(s, src);
  }
  // ... its part after the vertical transport Fz: advection and the dealias filter
  void momentum_advection_rest(cudaStream_t s, const Fields4& src) {
    const dim3 m(32, 8);
    pb(ZM_K_MADV, s);
    ZM_CUDA(launch_pdl(k_madv, dim3((nx + 31) / 32, (ny + MADV_TY - 1) / MADV_TY, nz), m, 0, s, d, src.u, src.v,
                       Fz, Ayu, Ayv));
    pe(s);
    pb(ZM_K_DEALIAS, s);
    ZM_CUDA(launch_dealias(s, d, fft, Ayu, Ayv, Au, Av, fft_lines, fft_smem, true));
    pe(s);
    check_launch();
  }

  // Pressure part P = wm (pgf_bc - F_rho) of the state's T/S, into Pu/Pv
  // (diagnostic stage; the step itself fuses it with the RK combination).
  void pressure_part(cudaStream_t s, const Fields4& src) {
    ZM_CUDA(cudaMemsetAsync(Au, 0, n3 * sizeof(float), s));
    ZM_CUDA(cudaMemsetAsync(Av, 0, n3 * sizeof(float), s));
    PgfArgs a{};
    a.T = src.T; a.S = src.S; a.u1 = src.u; a.v1 = src.v; a.Au = Au; a.Av = Av;
    a.Pu = Pu; a.Pv = Pv; a.uo = up; a.vo = vp; a.dt = (float)dt; a.mode = 1;
    pgf(s, a);
  }

  void copy_uv(cudaStream_t s, const float* a, const float* b, const Fields4& src, const Fields4& dst) {
    ZM_CUDA(cudaMemcpyAsync(dst.u, a, n3 * sizeof(float), cudaMemcpyDeviceToDevice, s));
    ZM_CUDA(cudaMemcpyAsync(dst.v, b, n3 * sizeof(float), cudaMemcpyDeviceToDevice, s));
    ZM_CUDA(cudaMemcpyAsync(dst.T, src.T, n3 * sizeof(float), cudaMemcpyDeviceToDevice, s));
    ZM_CUDA(cudaMemcpyAsync(dst.S, src.S, n3 * sizeof(float), cudaMemcpyDeviceToDevice, s));
  }

  // A cooperative launch.  Inside an ensemble capture it waits for the
  // previous member's cooperative kernels (bt_wait) and records bt_done, so
  // that no two grid-barrier kernels are resident at the same time.
  template <class... A>
  void coop_launch(cudaStream_t s, int cls, void (*kern)(A...), int blocks, int threads, size_t smem,
                   A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (bt_wait) ZM_CUDA(cudaStreamWaitEvent(s, bt_wait, 0));
    pb(cls, s);
    ZM_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
    pe(s);
    if (bt_done) ZM_CUDA(cudaEventRecord(bt_done, s));
  }

  // ---- ledger reductions (each: one partial-sum kernel, then the in-order fold)
  static constexpr double kHeat = 1025.0 * 3992.0, kSalt = 1025.0 / 1000.0;
  dim3 led_grid() const { return grid2(dim3(32, 8)); }
  void led_fold(cudaStream_t s, int nq, std::initializer_list<std::pair<int, double>> dst) {
    LedFold f{};
    int q = 0;
    for (auto& e : dst) {
      f.dst[q] = e.first;
      f.scale[q] = e.second;
      ++q;
    }
    for (; q < LED_Q; ++q) f.dst[q] = -1;
    const dim3 g = led_grid();
    k_led_fold<<<1, 32, 0, s>>>(led_part, (int)(g.x * g.y), nq, f, led_acc);
    check_launch();
  }
  // stage change between two states into stage `st_idx` (and the change scale)
  void led_stage(cudaStream_t s, int st_idx, const float* Tb, const float* Sb, const float* eb, const float* Ta,
                 const float* Sa, const float* ea) {
    k_led_diff<<<led_grid(), dim3(32, 8), 0, s>>>(d, Tb, Sb, eb, Ta, Sa, ea, led_area, led_dzn, led_part);
    const int b = ZM_LED_STAGE + 3 * st_idx;
    led_fold(s, 6, {{b, kHeat}, {b + 1, kSalt}, {b + 2, 1.0}, {ZM_LED_SCALE, kHeat}, {ZM_LED_SCALE + 1, kSalt},
                    {ZM_LED_SCALE + 2, 1.0}});
  }
  // one tracer residual's sources, processes and surface flux over dt/2
  void led_rk(cudaStream_t s, const float* Tev, const float* Sev) {
    k_led_rk<<<led_grid(), dim3(32, 8), 0, s>>>(d, Tev, Sev, accT, accS, led_topT, led_topS, led_convT, led_convS,
                                                Fz, 1.f / (float)adv_nsub, led_area, led_dzn, led_part);
    const double h = kHeat * dt / 2.0, sl = kSalt * dt / 2.0;
    const int P0 = ZM_LED_PROC, P1 = ZM_LED_PROC + 3, S0 = ZM_LED_SOURCE;
    led_fold(s, 16, {{P0, h}, {ZM_LED_PSCALE, h}, {P0 + 1, sl}, {ZM_LED_PSCALE + 1, sl},
                     {P1, h}, {ZM_LED_PSCALE, h}, {P1 + 1, sl}, {ZM_LED_PSCALE + 1, sl},
                     {S0, h}, {S0 + 3, h}, {S0 + 6, h}, {S0 + 9, h}, {S0 + 12 + 1, sl}, {S0 + 15 + 1, sl},
                     {ZM_LED_ADVB, h}, {ZM_LED_ADVB + 1, sl}});
  }
  void ensure_ledger() {
    if (led_acc) return;
    const dim3 g = led_grid();
    led_acc = alloc<double>(ZM_LED_COUNT);
    led_part = alloc<double>((size_t)g.x * g.y * LED_Q * 2);
    led_norms = alloc<double>(2);
    led_convT = f3();
    led_convS = f3();
    led_topT = f2();
    led_topS = f2();
  }

  // Column-divergence projection of (u, v) in place (projection.py:64-127).
  void project(cudaStream_t s, float* u, float* v) {
    const dim3 c(32, 8);
    pb(ZM_K_PROJECTION, s);
    k_proj_rhs<<<grid2(c), c, 0, s>>>(d, u, v, pj_dzn, pj_cos, pj_area, pj_dtg, const_cast<double*>(pj.b));
    pe(s);
    ProjArgs pa = pj;
    pa.norms = ledger_on ? led_norms : nullptr;
    if (pj_tile.blocks > 0)
      coop_launch(s, ZM_K_PROJECTION, proj_res_kernel(pj_tile.cpt), pj_tile.blocks, pj_tile.threads, pj_tile.smem, d,
                  pa);
    else
      coop_launch(s, ZM_K_PROJECTION, k_proj_cg, pj_blocks, PJ_THREADS, 0, d, pa);
    if (ledger_on) {
      k_led_proj<<<1, 32, 0, s>>>(led_norms, led_acc);
      check_launch();
    }
    pb(ZM_K_PROJECTION, s);
    k_proj_correct<<<grid2(c), c, 0, s>>>(d, u, v, pj.psi, pj_cos, pj_dtg);
    pe(s);
  }

  // Nonlinear RK2 step N(dt): src -> dst.
  void nonlinear(cudaStream_t s, const Fields4& src, const Fields4& dst) {
    pb(ZM_K_FZ, s);
    launch_fz(s, d, src.u, src.v, Fz);
    pe(s);
    // The momentum advection and its filter (latency-bound) and the stage-1
    // tracer residual (issue-bound) depend only on the state and Fz: they run
    // on two streams (two branches of the captured graph) and join before
    // the pressure part that needs both.
    ZM_CUDA(cudaEventRecord(ev_fork, s));
    ZM_CUDA(cudaStreamWaitEvent(side, ev_fork, 0));
    momentum_advection_rest(side, src);
    ZM_CUDA(cudaEventRecord(ev_join, side));
    // stage 1: tracers at the old velocity, momentum with the predicted tracers
    tracer_residual(s, 1, src.u, src.v, src.T, src.S, src.T, src.S, Tp, Sp);
    ZM_CUDA(cudaStreamWaitEvent(s, ev_join, 0));
    PgfArgs a{};
    a.T = Tp; a.S = Sp; a.u1 = src.u; a.v1 = src.v; a.Au = Au; a.Av = Av;
    a.Pu = Pu; a.Pv = Pv; a.uo = up; a.vo = vp; a.dt = (float)dt; a.mode = 1;
    pgf(s, a);
    // stage 2: tracers at the predicted velocity (or the old one if frozen)
    const float* u2 = src.u;
    const float* v2 = src.v;
    if (!freeze) {
      if (proj_on) project(s, up, vp);  // step.py:292-303
      pb(ZM_K_FZ, s);
      launch_fz(s, d, up, vp, Fz);
      pe(s);
      u2 = up;
      v2 = vp;
    }
    tracer_residual(s, 2, u2, v2, Tp, Sp, src.T, src.S, dst.T, dst.S);
    PgfArgs b{};
    b.T = dst.T; b.S = dst.S; b.u1 = src.u; b.v1 = src.v; b.Au = Au; b.Av = Av; b.Ppu = Pu; b.Ppv = Pv;
    b.uo = dst.u; b.vo = dst.v; b.dt = (float)dt; b.bottom_decay = bottom_decay; b.mode = 2;
    pgf(s, b);
  }

  // Barotropic subcycle and the final projection/cap/hold.
  void barotropic_and_final(cudaStream_t s, const Fields4& s3, const float* eta_in, const Fields4& held,
                            const Fields4& out, float* eta_out) {
    PgfArgs a{};
    a.T = s3.T; a.S = s3.S; a.u1 = s3.u; a.v1 = s3.v; a.frx = frx; a.fry = fry; a.ubt0 = ubt0; a.vbt0 = vbt0;
    a.mode = 0;
    a.flags = flags + 1;
    pgf(s, a);
    const dim3 c(32, 8);
    double *ubt_fin, *vbt_fin;
    if (bt_blocks > 0) {
      BtArgs a2 = bt;
      a2.eta_in = eta_in;
      a2.eta_out = eta_out;
      coop_launch(s, ZM_K_BAROTROPIC, bt_loop_kernel(btt.k), bt_blocks, btt.threads, btt.smem, d, a2);
      ubt_fin = bt.ubt_out;
      vbt_fin = bt.vbt_out;
    } else {
      pb(ZM_K_BAROTROPIC, s);
      ZM_CUDA(launch_pdl(k_bt_forcing, grid2(c), c, 0, s, d, frx, fry, Fx, Fy, eta_in, eta64[0]));
      pe(s);
      ZM_CUDA(cudaMemcpyAsync(ubt[0], ubt0, n2 * sizeof(double), cudaMemcpyDeviceToDevice, s));
      ZM_CUDA(cudaMemcpyAsync(vbt[0], vbt0, n2 * sizeof(double), cudaMemcpyDeviceToDevice, s));
      const bool cap = bt.cap_active != 0;
      for (int n = 0; n < n_subcyc; ++n) {
        const int a0 = n % 2, a1 = 1 - a0;
        pb(ZM_K_BAROTROPIC, s);
        k_bt_eta<<<grid2(c), c, 0, s>>>(d, eta64[a0], ubt[a0], vbt[a0], eta64[a1], bt.dtH);
        pe(s);
        for (int f = 0; f < 2; ++f) {  // sponge, then eta relaxation (barotropic.py:33-40)
          if (!(f == 0 ? bt.sponge : bt.relax)) continue;
          const double* fac = f == 0 ? bt.es : bt.er;
          const dim3 g2 = grid2(c);
          pb(ZM_K_BAROTROPIC, s);
          k_refill_part<<<g2, c, 0, s>>>(d, eta64[a1], fac, bt.area, bt.part_s);
          pe(s);
          pb(ZM_K_BAROTROPIC, s);
          k_refill_apply<<<g2, c, 0, s>>>(d, eta64[a1], fac, bt.part_s, (int)(g2.x * g2.y), bt.ocean);
          pe(s);
        }
        if (cap) {
          pb(ZM_K_BAROTROPIC, s);
          k_cap2d<<<dim3(2 * cap_nb, 1), 256, 0, s>>>(d, eta64[a1], nullptr, wts, bt.count, cap_nb);
          pe(s);
        }
        pb(ZM_K_BAROTROPIC, s);
        k_bt_vel<<<grid2(c), c, 0, s>>>(d, eta64[a1], ubt[a0], vbt[a0], Fx, Fy, ubt[a1], vbt[a1], dt_bt, bt_drag,
                                        bt.sponge ? bt.es : nullptr);
        pe(s);
        if (cap) {
          pb(ZM_K_BAROTROPIC, s);
          k_cap2d<<<dim3(2 * cap_nb, 2), 256, 0, s>>>(d, ubt[a1], vbt[a1], wts, bt.count, cap_nb);
          pe(s);
        }
      }
      const int fin = n_subcyc % 2;
      pb(ZM_K_BAROTROPIC, s);
      k_eta_to_float<<<grid2(c), c, 0, s>>>(d, eta64[fin], eta_out);
      pe(s);
      ubt_fin = ubt[fin];
      vbt_fin = vbt[fin];
    }
    if (cap_rows > 0) {
      pb(ZM_K_FINAL, s);
      ZM_CUDA(launch_pdl(k_cap3_means, dim3(2 * cap_nb, nz), dim3(256), 0, s, d, s3.u, s3.v, s3.T, s3.S, ubt_fin,
                         ubt0, vbt_fin, vbt0, means, cap_nb));
      pe(s);
    }
    pb(ZM_K_FINAL, s);
    ZM_CUDA(launch_pdl(k_final, grid3(c), c, 0, s, d, s3.u, s3.v, s3.T, s3.S, ubt_fin, ubt0, vbt_fin, vbt0, held.u,
                       held.v, held.T, held.S, means, wts, cap_rows > 0 ? cap_nb : 0, out.u, out.v, out.T, out.S,
                       bt_blocks > 0 ? bt_seq : nullptr, 2 * n_subcyc + 2, eta_out, flags + 1));
    pe(s);
    check_launch();
  }

  // learned closure: diffusivity per interface from the step's input state
  void closure(cudaStream_t s, const Fields4& in) {
    ZM_CUDA(cudaMemsetAsync(cl_count, 0, sizeof(unsigned), s));
    ClosureArgs a{};
    a.T = in.T; a.S = in.S; a.u = in.u; a.v = in.v; a.kappa3 = kappa3; a.fallback = cl_count; a.bound = cl_bound;
    const long long ncol = (long long)nx * ny;
    pb(ZM_K_CLOSURE, s);
    k_mlp_closure<<<mlp_tc_blocks(ncol), MLP_TC_THREADS, mlp_tc_smem(), s>>>(cw, d, a, cl_count + 1);
    pe(s);
    check_launch();
  }

  void full_step(cudaStream_t s, int from, int to) {
    const Fields4& in = st[from];
    if (closure_on) closure(s, in);
    linear_half(s, in, s1);
    nonlinear(s, s1, s2);
    if (ledger_on) led_stage(s, 2, s1.T, s1.S, nullptr, s2.T, s2.S, nullptr);  // step.py:366-368
    linear_half(s, s2, s1);
    barotropic_and_final(s, s1, eta[from], in, st[to], eta[to]);
    if (ledger_on) {
      // free surface (step.py:425-427): only eta changes; then the polar cap and
      // the land hold (step.py:452-453); dynamic ice is absent (no change)
      led_stage(s, 3, s1.T, s1.S, eta[from], s1.T, s1.S, eta[to]);
      led_stage(s, 4, s1.T, s1.S, nullptr, st[to].T, st[to].S, nullptr);
      // observed change (budgets.py:230-231) and eta times the surface tracers
      k_led_diff<<<led_grid(), dim3(32, 8), 0, s>>>(d, in.T, in.S, eta[from], st[to].T, st[to].S, eta[to], led_area,
                                                    led_dzn, led_part);
      led_fold(s, 6, {{ZM_LED_OBS, kHeat}, {ZM_LED_OBS + 1, kSalt}, {ZM_LED_OBS + 2, 1.0}});
      k_led_disp<<<led_grid(), dim3(32, 8), 0, s>>>(d, eta[from], in.T, in.S, eta[to], st[to].T, st[to].S, led_area,
                                                    led_part);
      led_fold(s, 2, {{ZM_LED_DISP, kHeat}, {ZM_LED_DISP + 1, kSalt}});
    }
  }

  // The classification of the state an advance ends with: its last step's own, or, where no
  // step ran, one pass over the state (72 us at 720 x 360 x 50, against 4 for the copy).
  void monitor(cudaStream_t s, int which, bool stepped) {
    if (stepped) {
      ZM_CUDA(cudaMemcpyAsync(flags, flags + 1, sizeof(unsigned int), cudaMemcpyDeviceToDevice, s));
      return;
    }
    ZM_CUDA(cudaMemsetAsync(flags, 0, sizeof(unsigned int), s));
    k_monitor<<<4 * 148, 256, 0, s>>>(d, st[which].u, st[which].v, st[which].T, st[which].S, eta[which],
                                      kMonitorVelocity, kMonitorEta, flags);
    check_launch();
  }

  // Time the launch shapes that change no result on the resident state,
  // through stages that only write work buffers, and keep the fastest:
  // nu_h halo width (3..NB_T), FFT lines per block (1..8), levels per block
  // of the tracer-advection and linear-finish column marches, tile rows of
  // the vertical-transport and pressure-gradient marches.
  void autotune(cudaStream_t s) {
    cudaEvent_t e0, e1;
    ZM_CUDA(cudaEventCreate(&e0));
    ZM_CUDA(cudaEventCreate(&e1));
    auto time_ms = [&](auto&& run) {
      run();
      ZM_CUDA(cudaEventRecord(e0, s));
      for (int r = 0; r < 3; ++r) run();
      ZM_CUDA(cudaEventRecord(e1, s));
      ZM_CUDA(cudaEventSynchronize(e1));
      float ms = 0.f;
      ZM_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      return ms;
    };
    try {
      const Fields4& in = st[cur];
      if (d.nu_h != 0.f) {
        float best = 1e30f;
        int pick = nu_halo, pick_w = nu_warps;
        for (int wq : {8, 16})
          for (int h = 3; h <= NB_T; ++h) {
            set_nu_shape(h, wq);
            const float ms = time_ms([&] { linear_half(s, in, s1); });
            if (ms < best) {
              best = ms;
              pick = h;
              pick_w = wq;
            }
          }
        set_nu_shape(pick, pick_w);
      }
      float best = 1e30f;
      int pick = fft_lines;
      for (int lines = 1; lines <= 8; lines *= 2) {
        const size_t smem = (size_t)2 * lines * nx * sizeof(float2);
        if (smem > 200 * 1024) break;
        fft_lines = lines;
        fft_smem = smem;
        const float ms = time_ms([&] { momentum_advection_part(s, in); });
        if (ms < best) {
          best = ms;
          pick = lines;
        }
      }
      fft_lines = pick;
      fft_smem = (size_t)2 * pick * nx * sizeof(float2);
      // column-march shapes: levels per block of the tracer advection and of
      // the linear finish, tile rows of the vertical transport and of the
      // pressure gradient (every point's arithmetic is the same in each)
      auto tune = [&](int& field, std::initializer_list<int> cands, auto&& run) {
        float b = 1e30f;
        int keep = field;
        for (int cand : cands) {
          field = cand;
          const float ms = time_ms(run);
          if (ms < b) {
            b = ms;
            keep = cand;
          }
        }
        field = keep;
      };
      const float dts = (float)(dt / adv_nsub);
      launch_fz(s, d, in.u, in.v, Fz);
      tune(d.ta_kc, {2, 3, 5, 8, 10, 13, 17, 25}, [&] {
        launch_tracer_adv(s, d, in.T, in.S, in.u, in.v, Fz, accT, accS, TsA, SsA, dts, 1, 0, nullptr, nullptr);
      });
      const float dth = (float)(dt / 2.0);
      tune(d.lt_kc, {2, 3, 5, 8, 10, 13, 17, 25}, [&] {
        launch_lin_t(s, d, in.u, in.v, in.u, in.v, in.T, in.S, s1.u, s1.v, s1.T, s1.S, dth, vdiff || closure_on);
      });
      tune(d.fz_rows, {4, 8}, [&] { launch_fz(s, d, in.u, in.v, Fz); });
      PgfArgs pa{};
      pa.T = in.T; pa.S = in.S; pa.u1 = in.u; pa.v1 = in.v; pa.frx = frx; pa.fry = fry; pa.ubt0 = ubt0;
      pa.vbt0 = vbt0; pa.gsx = gsx; pa.gsy = gsy; pa.Fxs = pfx; pa.Fys = pfy; pa.mode = 0;
      tune(d.pg_rows, {4, 8}, [&] { launch_pgf(s, d, pa); });
      check_launch();
    } catch (...) {
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      throw;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    tuned = true;
  }

  void drop_graphs() {
    for (cudaGraphExec_t& g : graph) {
      if (g) cudaGraphExecDestroy(g);
      g = nullptr;
    }
    graphs_ready = false;
  }
  void build_graphs() {
    cudaStream_t s = cap_stream;
    for (int g = 0; g < 2; ++g) {
      cudaGraph_t graph_def = nullptr;
      ZM_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
      const int before = launch_count;
      try {
        full_step(s, g, 1 - g);
        kernels_per_step = launch_count - before;
      } catch (...) {
        cudaStreamEndCapture(s, &graph_def);
        if (graph_def) cudaGraphDestroy(graph_def);
        throw;
      }
      ZM_CUDA(cudaStreamEndCapture(s, &graph_def));
      ZM_CUDA(cudaGraphInstantiate(&graph[g], graph_def, 0));
      cudaGraphDestroy(graph_def);
    }
    graphs_ready = true;
    ++graphs_built;
  }

  // layout conversion between reference arrays and internal fields
  void to_int3(cudaStream_t s, const float* src, float* dst, float offset) {
    launch_layout(s, d, LayoutArgs{{src}, {dst}, {offset}, 1, 0}, true);
  }
  void to_ref3(cudaStream_t s, const float* src, float* dst, float offset) {
    launch_layout(s, d, LayoutArgs{{src}, {dst}, {offset}, 1, 0}, false);
  }
  // tracers enter as anomalies from (T_ref, S_ref)
  void load(cudaStream_t s, const zm_state* in, const Fields4& f, float* e) {
    launch_layout(s, d, LayoutArgs{{in->u, in->v, in->T, in->S, in->eta}, {f.u, f.v, f.T, f.S, e},
                                   {0.f, 0.f, d.T_ref, d.S_ref, 0.f}, 4, 1}, true);
    check_launch();
  }
  void store(cudaStream_t s, const Fields4& f, const float* e, zm_state* out) {
    launch_layout(s, d, LayoutArgs{{f.u, f.v, f.T, f.S, e}, {out->u, out->v, out->T, out->S, out->eta},
                                   {0.f, 0.f, d.T_ref, d.S_ref, 0.f}, 4, 1}, false);
    check_launch();
  }
};

namespace {

void require(bool ok, int code, const std::string& msg) {
  if (!ok) throw Err{code, msg};
}

bool fft_factor(int n, FftPlan& plan) {
  plan.n = n;
  plan.nstages = 0;
  int m = n;
  const int radices[4] = {4, 2, 3, 5};
  for (int r : radices) {
    while (m % r == 0) {
      if (plan.nstages >= 24) return false;
      plan.radix[plan.nstages++] = r;
      m /= r;
    }
  }
  return m == 1;
}

std::vector<float> to_int2(const double* src, int nx, int ny, int P, double fill) {
  std::vector<float> out((size_t)ny * P, 0.f);
  for (int j = 0; j < ny; ++j)
    for (int i = 0; i < nx; ++i) out[(size_t)j * P + i] = (float)(src ? src[(size_t)i * ny + j] : fill);
  return out;
}

void build(zm_solver* s, const zm_grid* g, const zm_params* p) {
  require(g && p, ZM_ERR_INVALID, "null grid or params");
  const int nx = g->nx, ny = g->ny, nz = g->nz;
  require(nx >= 2 && ny >= 2 && nz >= 2, ZM_ERR_INVALID, "nx, ny and nz must be at least 2");
  require(nz <= ZM_MAXZ, ZM_ERR_UNSUPPORTED, "nz above 64 levels is not supported");
  require(g->dx_2d && g->cos_lat && g->f && g->z && g->dz && g->wet_mask, ZM_ERR_INVALID, "missing grid array");
  require(std::isfinite(g->dy) && g->dy > 0, ZM_ERR_INVALID, "dy must be positive and finite");
  require(std::isfinite(p->dt) && p->dt > 0, ZM_ERR_INVALID, "dt must be positive and finite");
  require(std::isfinite(p->dt_bt) && p->dt_bt > 0, ZM_ERR_INVALID, "dt_bt must be positive and finite");
  for (int k = 0; k + 1 < nz; ++k)
    require(g->z[k + 1] < g->z[k] && g->dz[k] > 0, ZM_ERR_INVALID, "z must be strictly descending");
  const int nb = p->polar_cap_rows + p->polar_cap_taper;
  require(p->polar_cap_rows >= 0 && p->polar_cap_taper >= 0, ZM_ERR_INVALID, "polar cap counts must be >= 0");
  require(!(p->polar_cap_rows > 0 && 2 * nb > ny), ZM_ERR_INVALID,
          "polar cap bands must not overlap; reduce rows/taper or disable the cap");
  require(p->limiter >= 0 && p->limiter <= 2, ZM_ERR_INVALID, "unknown limiter");
  FftPlan plan{};
  require(fft_factor(nx, plan), ZM_ERR_UNSUPPORTED, "nx must be a product of 2, 3 and 5 (longitude FFT filter)");

  cudaGetDevice(&s->device);
  s->nx = nx; s->ny = ny; s->nz = nz;
  s->P = (nx + 3) / 4 * 4;
  const int P = s->P;
  s->n2 = (size_t)ny * P;
  s->n3 = s->n2 * nz;
  s->dt = p->dt;
  s->n_subcyc = std::max(1, (int)std::nearbyint(p->dt / p->dt_bt));
  s->dt_bt = p->dt / s->n_subcyc;
  s->n_nu = std::max(1, p->nu_nsub > 0 ? (int)p->nu_nsub : s->n_subcyc);
  double dzmin = g->dz[0];
  for (int k = 0; k + 1 < nz; ++k) dzmin = std::min(dzmin, g->dz[k]);
  s->conv_nsub = std::max(1, (int)std::ceil(p->kappa_conv * p->dt / (0.4 * dzmin * dzmin)));
  s->adv_nsub = std::max(1, (int)std::ceil(p->dt * 4.0e-3 / (0.5 * dzmin)));
  s->cap_rows = p->polar_cap_rows;
  s->cap_nb = nb;
  s->vdiff = p->vertical_diffusion;
  s->want_tune = p->autotune != 0;
  s->freeze = p->freeze_adv_vel;
  s->bottom_decay = (float)std::exp(-p->r_bot * p->dt);
  s->bt_drag = 1.0 / (1.0 + p->r_bot * s->dt_bt);

  Dev& d = s->d;
  d.nx = nx; d.ny = ny; d.nz = nz; d.P = P;
  d.plane = (long long)s->n2;
  // ---- per-row metric
  std::vector<float> cosl(ny), inv_cos(ny), cfp(ny), cfm(ny), tanR(ny);
  for (int j = 0; j < ny; ++j) {
    const double c = g->cos_lat[j];
    cosl[j] = (float)c;
    inv_cos[j] = (float)(1.0 / c);
    cfp[j] = (float)(0.5 * (c + g->cos_lat[(j + 1) % ny]));
    cfm[j] = (float)(0.5 * (c + g->cos_lat[(j - 1 + ny) % ny]));
    const double sin_row = g->f[j] / (2.0 * kOmega);   // f[0, j]
    tanR[j] = (float)((sin_row / c) / kREarth);
  }
  d.cosl = s->upload(cosl); d.inv_cos = s->upload(inv_cos); d.cfp = s->upload(cfp); d.cfm = s->upload(cfm);
  d.tanR = s->upload(tanR);
  // ---- 2-D fields
  std::vector<float> inv_dx(s->n2, 1.f), inv_dx2(s->n2, 1.f), fc(s->n2, 0.f), rc(s->n2, 1.f), rs(s->n2, 0.f);
  std::vector<double> inv_dx_d(s->n2, 1.0), fc_d(s->n2, 0.0);
  std::vector<uint64_t> bits(s->n2, 0ull);
  for (int j = 0; j < ny; ++j)
    for (int i = 0; i < nx; ++i) {
      const size_t r = (size_t)i * ny + j, c = (size_t)j * P + i;
      const double dx = g->dx_2d[r];
      require(std::isfinite(dx) && dx > 0, ZM_ERR_INVALID, "dx_2d must be positive and finite");
      inv_dx[c] = (float)(1.0 / dx);
      inv_dx2[c] = (float)(1.0 / (dx * dx));
      inv_dx_d[c] = 1.0 / dx;
      fc[c] = (float)g->f[r];
      fc_d[c] = g->f[r];
      const double ang = g->f[r] * (p->dt / 2.0);
      rc[c] = (float)std::cos(ang);
      rs[c] = (float)std::sin(ang);
      uint64_t b = 0;
      for (int k = 0; k < nz; ++k) {
        const double w = g->wet_mask_3d ? g->wet_mask_3d[r * nz + k] : g->wet_mask[r];
        require(w == 0.0 || w == 1.0, ZM_ERR_UNSUPPORTED, "wet masks must be 0 or 1");
        if (w == 1.0) b |= 1ull << k;
      }
      bits[c] = b;
    }
  d.inv_dx = s->upload(inv_dx); d.inv_dx2 = s->upload(inv_dx2); d.fcor = s->upload(fc);
  d.rot_c = s->upload(rc); d.rot_s = s->upload(rs);
  d.inv_dx_d = s->upload(inv_dx_d); d.fcor_d = s->upload(fc_d);
  d.wbits = s->upload(bits);
  d.wet2 = s->upload(to_int2(g->wet_mask, nx, ny, P, 0.0));
  {  // face gates of the nu_h Laplacian, one byte per point
    unsigned char* gate = s->alloc<unsigned char>(s->n3);
    const dim3 b(32, 8), gr((P + 31) / 32, (ny + 7) / 8, nz);
    k_nu_gates<<<gr, b>>>(d, gate);
    ZM_CUDA(cudaGetLastError());
    ZM_CUDA(cudaDeviceSynchronize());
    d.nu_gate = gate;
    d.dx_rows = 1;
    for (int j = 0; j < ny && d.dx_rows; ++j)
      for (int i = 1; i < nx; ++i)
        if (inv_dx2[(size_t)j * P + i] != inv_dx2[(size_t)j * P]) d.dx_rows = 0;
    s->set_nu_shape(s->nu_halo, s->nu_warps);
    // wet levels of the column tiles
    const int ntx = (nx + 31) / 32;
    for (int ry : {8, 4}) {
      const int nty = (ny + ry - 1) / ry;
      uint64_t* t = s->alloc<uint64_t>((size_t)ntx * nty);
      k_tile_bits<<<(ntx * nty + 7) / 8, dim3(32, 8)>>>(d, t, ry, ntx, nty);
      ZM_CUDA(cudaGetLastError());
      (ry == 8 ? d.tile8 : d.tile4) = t;
    }
    // the lines of the longitude filter with a wet point
    std::vector<int> lines;
    std::vector<uint64_t> row(ny, 0ull);
    for (int j = 0; j < ny; ++j)
      for (int i = 0; i < nx; ++i) row[j] |= bits[(size_t)j * P + i];
    for (int k = 0; k < nz; ++k)
      for (int j = 0; j < ny; ++j)
        if (row[j] >> k & 1ull) lines.push_back(k * ny + j);
    plan.nlines = (int)lines.size();
    if (lines.empty()) lines.push_back(0);
    plan.lines = s->upload(lines);
  }
  int sms = 0;
  ZM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device));
  {
    // Levels per block of the tracer-advection and linear-finish marches (one tile shape): ten, which spread a block's
    // first loads best, unless that leaves fewer than eight blocks per SM (two waves); then as many as
    // give eight, down to two.  Per step at 90 x 45 x 15: 113 us with ten, 90 with two; 180 x 90 x 50:
    // 488 with ten, 443 with six (four blocks per SM), 412 with three (eight).
    const long long tiles = (long long)((nx + TA_X - 1) / TA_X) * ((ny + TA_Y - 1) / TA_Y);
    int kc = 10;
    while (kc > 2 && tiles * ((nz + kc - 1) / kc) < 8ll * sms) --kc;
    d.ta_kc = d.lt_kc = kc;
  }
  d.pg_rows = 4;
  d.fz_rows = 4;
  {
    std::vector<float> kh = to_int2(p->coastal_kappa_h, nx, ny, P, 0.0);
    std::vector<float> kv = to_int2(p->coastal_kappa_v, nx, ny, P, 0.0);
    for (int j = 0; j < ny; ++j)
      for (int i = 0; i < nx; ++i) {
        const size_t r = (size_t)i * ny + j, c = (size_t)j * P + i;
        kh[c] = (float)(p->kappa_h + (p->coastal_kappa_h ? p->coastal_kappa_h[r] : 0.0));
        kv[c] = (float)(p->kappa_v + (p->coastal_kappa_v ? p->coastal_kappa_v[r] : 0.0));
      }
    d.kh2 = s->upload(kh);
    d.kv2 = s->upload(kv);
  }
  s->tau_x = s->upload(to_int2(p->tau_x, nx, ny, P, 0.0));
  s->tau_y = s->upload(to_int2(p->tau_y, nx, ny, P, 0.0));
  s->qheat = s->upload(to_int2(p->q_heat, nx, ny, P, 0.0));
  d.tau_x = s->tau_x; d.tau_y = s->tau_y; d.qheat = s->qheat;
  // temperature / salinity targets, shifted like the tracers
  std::vector<float> tatm = to_int2(p->lambda_bulk > 0 ? p->t_atm : nullptr, nx, ny, P, 0.0);
  std::vector<float> rest_t = to_int2(p->coastal_restore_t, nx, ny, P, 0.0);
  std::vector<float> sref = to_int2(p->s_ref, nx, ny, P, 0.0);
  for (int j = 0; j < ny; ++j)
    for (int i = 0; i < nx; ++i) {
      const size_t r = (size_t)i * ny + j, c = (size_t)j * P + i;
      tatm[c] = (float)(((p->lambda_bulk > 0 && p->t_atm) ? p->t_atm[r] : 0.0) - p->T_ref);
      rest_t[c] = (float)((p->coastal_restore_t ? p->coastal_restore_t[r] : 0.0) - p->T_ref);
      sref[c] = (float)((p->s_ref ? p->s_ref[r] : 0.0) - p->S_ref);
    }
  d.tatm = s->upload(tatm);
  d.cbulk = s->upload(to_int2(p->coastal_bulk_lambda, nx, ny, P, 0.0));
  d.rest_c = s->upload(to_int2(p->coastal_restore_coef, nx, ny, P, 0.0));
  d.rest_T = s->upload(rest_t);
  d.sref = s->upload(sref);
  // ---- scalars
  d.inv_dy = (float)(1.0 / g->dy);
  d.inv_dy2 = (float)(1.0 / (g->dy * g->dy));
  d.inv_dy_d = 1.0 / g->dy;
  d.nu_h = (float)p->nu_h; d.nu_v = (float)p->nu_v; d.nu_bi = (float)p->nu_bi; d.kappa_bi = (float)p->kappa_bi;
  d.kappa_conv = (float)p->kappa_conv; d.r_bot = (float)p->r_bot; d.T_ref = (float)p->T_ref;
  d.S_ref = (float)p->S_ref;
  double H = 0.0;
  for (int k = 0; k + 1 < nz; ++k) H += g->dz[k];
  d.H_sw = (float)H;
  d.dz_surface = (float)std::fabs(g->z[0] - g->z[1]);
  d.lambda_bulk = (float)(p->t_atm ? p->lambda_bulk : 0.0);
  d.restore_S = (float)p->restore_coef_S;
  d.ice_salt = (float)p->ice_salt_flux;
  d.ice_freeze = (float)(p->ice_freeze_temp_c - p->T_ref);
  d.localize_conv = p->localize_conv;
  d.limiter = p->limiter;
  d.conservative_kv = p->conservative_kv;
  // ---- vertical coefficients (fd_metrics.py:55-98)
  Vert& vc = d.vc;
  const double* z = g->z;
  std::vector<double> gap(nz - 1);
  for (int k = 0; k + 1 < nz; ++k) gap[k] = std::fabs(z[k + 1] - z[k]);
  for (int k = 0; k < nz; ++k) {
    double node;
    if (k == 0) node = gap[0];
    else if (k == nz - 1) node = gap[nz - 2];
    else node = 0.5 * (gap[k - 1] + gap[k]);
    vc.dz_node[k] = (float)node;
    vc.inv_dz_node[k] = (float)(1.0 / node);
  }
  for (int k = 0; k + 1 < nz; ++k) {
    vc.inv_dz_iface[k] = (float)(1.0 / gap[k]);
    vc.dz3d[k] = (float)g->dz[k];
    vc.dznorm[k] = (float)(g->dz[k] / H);
  }
  for (int k = 1; k + 1 < nz; ++k) {
    const double hm = std::fabs(z[k - 1] - z[k]), hp = std::fabs(z[k + 1] - z[k]);
    const double den = hm * hp * (hm + hp) / 2.0;
    vc.d2_hi[k] = (float)(hm / den);
    vc.d2_lo[k] = (float)(hp / den);
    vc.ddz_inv[k] = (float)(1.0 / ((z[k] - z[k - 1]) + (z[k + 1] - z[k])));
  }
  vc.ddz_inv[0] = (float)(1.0 / (z[1] - z[0]));
  vc.ddz_inv[nz - 1] = (float)(1.0 / (z[nz - 1] - z[nz - 2]));
  vc.d2_top = (float)(2.0 / (gap[0] * gap[0]));
  vc.d2_bot = (float)(2.0 / (gap[nz - 2] * gap[nz - 2]));
  // the end rows in the interior form
  vc.d2_lo[0] = vc.d2_hi[nz - 1] = 0.f;
  vc.d2_hi[0] = vc.d2_top;
  vc.d2_lo[nz - 1] = vc.d2_bot;
  // ---- polar cap weights (numerics/horizontal.py:362-385), pole-inward
  std::vector<float> w(std::max(nb, 1), 0.f);
  for (int r = 0; r < p->polar_cap_rows; ++r) w[r] = 1.f;
  for (int t = 0; t < p->polar_cap_taper; ++t) {
    const double x = (kPi / 2.0) * (t + 1) / (p->polar_cap_taper + 1);
    w[p->polar_cap_rows + t] = (float)(std::cos(x) * std::cos(x));
  }
  s->wts = s->upload(w);
  // ---- FFT plan for the longitude dealias (factory.py:529-533)
  plan.keep = std::max(1, (int)((double)(nx / 2) * 2.0 / 3.0));
  {
    std::vector<int> bases;
    std::vector<float2> stw;
    int ns = 1;
    for (int st = 0; st < plan.nstages; ++st) {
      const int R = plan.radix[st], m = nx / R, stride = nx / (ns * R);
      plan.tab_off[st] = (int)bases.size();
      plan.tw_off[st] = (int)stw.size();
      for (int jj = 0; jj < m; ++jj) bases.push_back((jj / ns) * ns * R + jj % ns);
      for (int r = 1; r < R; ++r)
        for (int jj = 0; jj < m; ++jj) {
          const long long e = ((long long)(jj % ns) * r * stride) % nx;
          const double a = -2.0 * kPi * (double)e / nx;
          stw.push_back(make_float2((float)std::cos(a), (float)std::sin(a)));
        }
      ns *= R;
    }
    if (stw.empty()) stw.push_back(make_float2(1.f, 0.f));
    plan.base_tab = s->upload(bases);
    plan.stage_tw = s->upload(stw);
  }
  // 2/3-rule bin mask exactly as the reference forms it: numpy's
  // fftfreq(nx) * nx in float64, |.| <= keep
  std::vector<unsigned char> keepbin(nx);
  {
    const int half = (nx - 1) / 2 + 1;
    const double val = 1.0 / (double)nx;
    for (int m = 0; m < nx; ++m) {
      const int ms = m < half ? m : m - nx;
      const double kidx = ((double)ms * val) * (double)nx;
      keepbin[m] = std::fabs(kidx) <= (double)plan.keep ? 1 : 0;
    }
  }
  plan.keepbin = s->upload(keepbin);
  // twiddles of the register-resident form, exp(-2 pi i j / nx)
  if (fft_reg_split(nx, plan.r1, plan.r2, plan.r3)) {
    std::vector<float2> tw(nx);
    for (int j = 0; j < nx; ++j) {
      const double a = -2.0 * kPi * (double)j / nx;
      tw[j] = make_float2((float)std::cos(a), (float)std::sin(a));
    }
    plan.tw_full = s->upload(tw);
  }
  s->fft = plan;
  // Lines per block of the filter: four, fewer where shared memory or the number of lines (eight blocks
  // per SM) asks for it.  90 x 45 x 15: the filter takes 15 us with four lines, 12 with one;
  // 450 x 219 x 37: 1.131 ms a step with four, 1.139 with two, 1.158 with one.
  s->fft_lines = std::max(1, std::min(4, (int)((200 * 1024 / sizeof(float2)) / (2 * nx))));
  while (s->fft_lines > 1 && plan.nlines / s->fft_lines < 8 * sms) s->fft_lines /= 2;
  s->fft_smem = (size_t)2 * s->fft_lines * nx * sizeof(float2);
  require(s->fft_smem <= 227 * 1024, ZM_ERR_UNSUPPORTED, "nx too large for the shared-memory FFT filter");
  {
    // the attribute belongs to the kernel, not to this handle: allow the
    // device's opt-in maximum so that handles of every grid width can launch
    int optin = 0;
    ZM_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->device));
    require((int)s->fft_smem <= optin, ZM_ERR_UNSUPPORTED, "nx too large for the shared-memory FFT filter");
    ZM_CUDA(cudaFuncSetAttribute(k_dealias_lon, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
  }
  // ---- buffers
  for (int q = 0; q < 2; ++q) {
    s->st[q] = s->four();
    s->eta[q] = s->f2();
  }
  s->s1 = s->four(); s->s2 = s->four(); s->W1 = s->four(); s->W2 = s->four(); s->L = s->four();
  s->Fz = s->f3(); s->Ayu = s->f3(); s->Ayv = s->f3(); s->Au = s->f3(); s->Av = s->f3();
  s->accT = s->f3(); s->accS = s->f3(); s->TsA = s->f3(); s->SsA = s->f3(); s->TsB = s->f3(); s->SsB = s->f3();
  s->dT1 = s->f3(); s->dS1 = s->f3(); s->Tp = s->f3(); s->Sp = s->f3(); s->Pu = s->f3(); s->Pv = s->f3();
  s->gsx = s->f3(); s->gsy = s->f3();
  s->pfx = s->f2(); s->pfy = s->f2();
  s->up = s->f3(); s->vp = s->f3();
  s->frx = s->f2(); s->fry = s->f2();
  s->means = s->alloc<float>((size_t)4 * 2 * std::max(nb, 1) * nz);
  s->ubt0 = s->alloc<double>(s->n2); s->vbt0 = s->alloc<double>(s->n2);
  for (int q = 0; q < 2; ++q) {
    s->ubt[q] = s->alloc<double>(s->n2);
    s->vbt[q] = s->alloc<double>(s->n2);
    s->eta64[q] = s->alloc<double>(s->n2);
  }
  s->Fx = s->alloc<double>(s->n2); s->Fy = s->alloc<double>(s->n2);
  // ---- barotropic subcycle: resident tiles when they all fit on the GPU at
  // once, else the streaming kernels
  {
    require(nb <= ZM_BT_MAX_NB, ZM_ERR_UNSUPPORTED, "polar cap band wider than 64 rows");
    BtArgs& a = s->bt;
    a.nb = p->polar_cap_rows > 0 ? nb : 0;
    a.nsub = s->n_subcyc;
    a.dtH = s->dt_bt * (double)d.H_sw;
    a.dtb = s->dt_bt;
    a.drag = s->bt_drag;
    // wet counts of the band rows, max(count, 1); the cap is the identity when
    // every band row is land
    std::vector<double> cnt(std::max(1, 2 * a.nb), 1.0);
    a.cap_active = 0;
    for (int b = 0; b < 2 * a.nb; ++b) {
      const int j = b < a.nb ? b : ny - 2 * a.nb + b;
      double c = 0.0;
      for (int i = 0; i < nx; ++i) c += g->wet_mask[(size_t)i * ny + j];
      if (c > 0.0) a.cap_active = 1;
      cnt[b] = std::max(c, 1.0);
    }
    a.count = s->upload(cnt);
    a.wts = s->wts;
    a.ubt0 = s->ubt0;
    a.vbt0 = s->vbt0;
    a.frx = s->frx;
    a.fry = s->fry;
    int sms = 0, coop = 0, optin = 0;
    ZM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device));
    ZM_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, s->device));
    ZM_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->device));
    require(p->bt_kernel >= ZM_BT_AUTO && p->bt_kernel <= ZM_BT_STREAMING, ZM_ERR_INVALID, "unknown bt_kernel");
    optin -= 64;  // the barrier's own static words
    s->btt = bt_tile(nx, ny, sms, (size_t)optin, 128);
    bool fits = coop && s->btt.blocks > 0;
    if (fits) {
      auto kern = bt_loop_kernel(s->btt.k);
      int per_sm = 0;
      ZM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
      ZM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, s->btt.threads, s->btt.smem));
      fits = s->btt.blocks <= per_sm * sms;
    }
    // the documented limit of an explicit request: four 32 x 16 tiles per SM
    const bool named = (long long)((nx + 31) / 32) * ((ny + 15) / 16) <= 4ll * sms;
    require((fits && named) || p->bt_kernel != ZM_BT_RESIDENT, ZM_ERR_UNSUPPORTED,
            "barotropic tiles do not fit on the GPU at once (bt_kernel = ZM_BT_RESIDENT)");
    // the loop knows wet and dry cells; a mask with weights between takes the streaming kernels, which multiply by it
    const bool binary = std::all_of(g->wet_mask, g->wet_mask + (size_t)nx * ny, [](double w) { return w == 0.0 || w == 1.0; });
    s->bt_blocks = (fits && binary && p->bt_kernel != ZM_BT_STREAMING) ? s->btt.blocks : 0;
    if (s->bt_blocks > 0) {
      a.tile_x = s->btt.x;
      a.tile_y = s->btt.y;
      a.ntx = s->btt.tiles_x;
      a.pub = s->alloc<double>((size_t)2 * 2 * 3 * s->n2);  // 16-byte words
      a.sums = s->alloc<double>((size_t)2 * 2 * s->bt_blocks * s->bt_blocks);
      s->bt_seq = s->alloc<unsigned long long>(1);
      a.seq = s->bt_seq;
      a.ubt_out = s->alloc<double>(s->n2);
      a.vbt_out = s->alloc<double>(s->n2);
      const size_t np = (size_t)std::max(1, 2 * a.nb) * a.ntx;
      for (int q = 0; q < 2; ++q) {
        a.part_e[q] = s->alloc<double>(np);
        a.part_u[q] = s->alloc<double>(np);
        a.part_v[q] = s->alloc<double>(np);
      }
    }
    s->bt_sync = s->alloc<unsigned>(4);
    a.bar = s->bt_sync;
    a.err = s->bt_sync + 2;
  }
  {
    // lateral sponge and eta relaxation (factory.py:456-521)
    BtArgs& a = s->bt;
    bool sponge = false, relax = false;
    if (p->sponge_rate) {
      for (size_t q = 0; q < (size_t)nx * ny; ++q) {
        require(std::isfinite(p->sponge_rate[q]) && p->sponge_rate[q] >= 0.0, ZM_ERR_INVALID,
                "sponge_rate must be finite and nonnegative");
        if (p->sponge_rate[q] > 0.0) sponge = true;
      }
    }
    require(std::isfinite(p->eta_relax_rate) && p->eta_relax_rate >= 0.0, ZM_ERR_INVALID,
            "eta_relax_rate must be finite and nonnegative");
    if (p->eta_relax_mask && p->eta_relax_rate > 0.0) {
      for (size_t q = 0; q < (size_t)nx * ny; ++q) {
        require(std::isfinite(p->eta_relax_mask[q]), ZM_ERR_INVALID, "eta_relax_mask must be finite");
        if (p->eta_relax_mask[q] != 0.0) relax = true;
      }
    }
    if (sponge || relax) {
      std::vector<double> area(s->n2, 0.0), es(s->n2, 1.0), er(s->n2, 1.0);
      double ocean = 0.0;
      for (int i = 0; i < nx; ++i)
        for (int j = 0; j < ny; ++j) {
          const size_t r = (size_t)i * ny + j, c = (size_t)j * P + i;
          area[c] = g->dx_2d[r] * g->dy;
          ocean += area[c] * g->wet_mask[r];
          if (sponge) es[c] = std::exp(-p->sponge_rate[r] * s->dt_bt);
          if (relax) er[c] = std::exp(-p->eta_relax_rate * s->dt_bt * p->eta_relax_mask[r]);
        }
      a.area = s->upload(area);
      a.ocean = std::max(ocean, 1.0);
      a.sponge = sponge ? 1 : 0;
      a.relax = relax ? 1 : 0;
      a.es = s->upload(es);
      a.er = s->upload(er);
      a.part_s = s->alloc<double>((size_t)((nx + 31) / 32) * ((ny + 7) / 8));
    }
    if (sponge) {
      require(p->T_clim && p->S_clim, ZM_ERR_INVALID, "the sponge needs T_clim and S_clim");
      std::vector<float> dec(s->n2, 1.f), tc(s->n3, 0.f), sc(s->n3, 0.f);
      for (int i = 0; i < nx; ++i)
        for (int j = 0; j < ny; ++j) {
          const size_t r = (size_t)i * ny + j;
          dec[(size_t)j * P + i] = (float)std::exp(-p->sponge_rate[r] * (p->dt / 2.0));
          for (int k = 0; k < nz; ++k) {
            const double tv = p->T_clim[r * nz + k], sv = p->S_clim[r * nz + k];
            require(std::isfinite(tv) && std::isfinite(sv), ZM_ERR_INVALID, "T_clim and S_clim must be finite");
            const size_t id = (size_t)k * s->n2 + (size_t)j * P + i;
            tc[id] = (float)(tv - p->T_ref);
            sc[id] = (float)(sv - p->S_ref);
          }
        }
      s->sp_dec = s->upload(dec);
      s->sp_Tc = s->upload(tc);
      s->sp_Sc = s->upload(sc);
    }
  }
  // projection options are validated whether or not the projection is on (factory.py:368-386)
  require(p->projection_niter > 0, ZM_ERR_INVALID, "projection_niter must be a positive integer");
  require(std::isfinite(p->projection_rtol) && p->projection_rtol >= 0.0, ZM_ERR_INVALID,
          "projection_rtol must be finite and positive");
  require(p->projection_preconditioner == ZM_PROJ_NONE || p->projection_preconditioner == ZM_PROJ_JACOBI,
          ZM_ERR_INVALID, "projection_preconditioner must be none or jacobi");
  require(p->projection_max_refinements >= 0 && p->projection_max_refinements <= 2, ZM_ERR_INVALID,
          "projection_max_refinements must be an integer from 0 to 2");
  if (p->project_adv_vel && !p->freeze_adv_vel) {
    // column projection (projection.py:10-127): tolerances with the float32 floors
    const double eps32 = 1.1920928955078125e-07;
    const double tol = std::max(p->projection_rtol > 0.0 ? p->projection_rtol : 1e-12, 32.0 * eps32);
    const double trtol = std::max(1e-10, 32.0 * eps32);
    int per_sm = 0, sms = 0, coop = 0;
    ZM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_proj_cg, PJ_THREADS, 0));
    ZM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device));
    ZM_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, s->device));
    require(coop && per_sm >= 1, ZM_ERR_UNSUPPORTED, "the column projection needs a cooperative launch");
    s->pj_blocks = std::max(1, std::min(sms, (int)(((long long)nx * ny + PJ_THREADS - 1) / PJ_THREADS)));
    std::vector<double> dzn(nz), cosd(ny), area(s->n2, 0.0);
    for (int k = 0; k < nz; ++k) {
      if (k == 0) dzn[k] = std::fabs(g->z[1] - g->z[0]);
      else if (k == nz - 1) dzn[k] = std::fabs(g->z[nz - 1] - g->z[nz - 2]);
      else dzn[k] = 0.5 * (std::fabs(g->z[k] - g->z[k - 1]) + std::fabs(g->z[k + 1] - g->z[k]));
    }
    for (int j = 0; j < ny; ++j) cosd[j] = g->cos_lat[j];
    for (int j = 0; j < ny; ++j)
      for (int i = 0; i < nx; ++i) {
        const size_t r = (size_t)i * ny + j;
        area[(size_t)j * P + i] = g->dx_2d[r] * g->dy * g->wet_mask[r];
      }
    s->pj_dzn = s->upload(dzn);
    s->pj_cos = s->upload(cosd);
    s->pj_area = s->upload(area);
    ProjArgs& a = s->pj;
    double* cx = s->alloc<double>(3 * s->n2);
    double* cy = s->alloc<double>(3 * s->n2);
    double* sxy = s->alloc<double>(2 * s->n2);
    double* minv = p->projection_preconditioner == ZM_PROJ_JACOBI ? s->alloc<double>(s->n2) : nullptr;
    double* rarea = s->alloc<double>(s->n2);
    const dim3 c(32, 8);
    k_proj_coef<<<s->grid2(c), c>>>(s->d, s->pj_dzn, s->pj_cos, s->pj_area, cx, cy, sxy, minv, rarea);
    s->check_launch();
    a.cx = cx; a.cy = cy; a.sxy = sxy; a.minv = minv; a.rarea = rarea;
    a.b = s->alloc<double>(s->n2);
    a.psi = s->alloc<double>(s->n2);
    a.x = s->alloc<double>(s->n2);
    a.r = s->alloc<double>(s->n2);
    a.z = s->alloc<double>(s->n2);
    a.p0 = s->alloc<double>(s->n2);
    a.p1 = s->alloc<double>(s->n2);
    a.Ap = s->alloc<double>(s->n2);
    a.part = s->alloc<double>((size_t)2 * s->pj_blocks * ZM_PJ_SUMS);
    unsigned* sync = s->alloc<unsigned>(4);
    a.bar = sync;
    a.err = sync + 2;
    a.stats = s->alloc<int>(4);
    a.tol2 = tol * tol;
    a.trtol2 = trtol * trtol;
    a.niter = p->projection_niter;
    a.refinements = p->projection_max_refinements;
    int optin = 0;
    ZM_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->device));
    // The resident form's recurrences take <p, A p> from <z, A z>, which holds for a symmetric A: dx / cos the
    // same in every row (an area over dy cos is then a constant of the meridian), a mask of 0 and 1, no wet
    // level where it is 0.  Other grids take k_proj_cg, which forms <p, A p> itself.
    bool symmetric = true;
    for (int i = 0; i < nx && symmetric; ++i)
      for (int j = 0; j < ny; ++j) {
        const size_t r = (size_t)i * ny + j;
        const double w = g->wet_mask[r], q = g->dx_2d[r] / g->cos_lat[j], q0 = g->dx_2d[(size_t)i * ny] / g->cos_lat[0];
        bool wet = false;
        for (int k = 0; k < nz; ++k) wet = wet || (g->wet_mask_3d ? g->wet_mask_3d[r * nz + k] : w) == 1.0;
        symmetric = symmetric && (w == 1.0 || (w == 0.0 && !wet)) && std::fabs(q - q0) <= 1e-10 * std::fabs(q0);
      }
    if (symmetric && proj_res_tile(nx, ny, sms, (size_t)optin, 256, s->pj_tile)) {
      auto kern = proj_res_kernel(s->pj_tile.cpt);
      ZM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
      ZM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, s->pj_tile.threads, s->pj_tile.smem));
      if (per_sm < 1) s->pj_tile.blocks = 0;
    }
    if (s->pj_tile.blocks > 0) {
      a.tile_x = s->pj_tile.x;
      a.tile_y = s->pj_tile.y;
      a.tiles_x = s->pj_tile.tiles_x;
      a.pub = s->alloc<double>(4 * s->n2);
      a.words = s->alloc<double>((size_t)2 * ZM_PJ_SUMS * s->pj_tile.blocks * s->pj_tile.blocks * 2);
      a.seq = s->alloc<unsigned long long>(1);
    }
    s->pj_dtg = p->dt * 9.81;
    a.dtg = s->pj_dtg;
    s->proj_on = true;
  }
  s->set_wait_limit(ZM_BT_BARRIER_POLLS);
  const size_t nref3 = (size_t)nx * ny * nz;
  s->ref = Fields4{s->alloc<float>(nref3), s->alloc<float>(nref3), s->alloc<float>(nref3), s->alloc<float>(nref3)};
  s->ref_eta = s->alloc<float>((size_t)nx * ny);
  s->flags = s->alloc<unsigned int>(2);
  {
    // budget snapshot (diagnostics/snapshot.py:42-64, 67-128)
    std::vector<double> area((size_t)nx * ny), width(nz);
    for (size_t q = 0; q < area.size(); ++q) area[q] = g->dx_2d[q] * g->dy;
    for (int k = 0; k < nz; ++k) {
      if (k == 0) width[k] = std::fabs(g->z[1] - g->z[0]);
      else if (k == nz - 1) width[k] = std::fabs(g->z[nz - 1] - g->z[nz - 2]);
      else width[k] = 0.5 * (std::fabs(g->z[k] - g->z[k - 1]) + std::fabs(g->z[k + 1] - g->z[k]));
    }
    s->area64 = s->upload(area);
    s->width64 = s->upload(width);
    // the ledger's cell areas in the internal layout and node thicknesses
    std::vector<double> area_int(s->n2, 0.0);
    for (int i = 0; i < nx; ++i)
      for (int j = 0; j < ny; ++j) area_int[(size_t)j * P + i] = g->dx_2d[(size_t)i * ny + j] * g->dy;
    s->led_area = s->upload(area_int);
    s->led_dzn = s->upload(width);
    int sms = 0;
    ZM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device));
    s->bblocks = std::max(1, std::min(3 * sms, (int)(((long long)nx * ny + 7) / 8)));
    s->bpart = s->alloc<double>((size_t)s->bblocks * ZM_BUDGET_SUMS * 2);
    s->bout = s->alloc<double>(ZM_BUDGET_SUMS * 2);
  }
  ZM_CUDA(cudaStreamCreateWithFlags(&s->cap_stream, cudaStreamNonBlocking));
  ZM_CUDA(cudaStreamCreateWithFlags(&s->side, cudaStreamNonBlocking));
  ZM_CUDA(cudaEventCreateWithFlags(&s->ev_fork, cudaEventDisableTiming));
  ZM_CUDA(cudaEventCreateWithFlags(&s->ev_join, cudaEventDisableTiming));
  ZM_CUDA(cudaDeviceSynchronize());
}

int fail(zm_solver* s, const Err& e) {
  if (s) s->last_error = e.msg;
  return e.code;
}

}  // namespace

extern "C" {

int zm_create(const zm_grid* grid, const zm_params* params, zm_solver** out) {
  if (!out) return ZM_ERR_INVALID;
  *out = nullptr;
  zm_solver* s = new zm_solver();
  try {
    build(s, grid, params);
  } catch (const Err& e) {
    std::fprintf(stderr, "zm_create: %s\n", e.msg.c_str());
    const int code = e.code;
    delete s;
    return code;
  }
  *out = s;
  return ZM_OK;
}

int zm_info(const zm_solver* s, int32_t* out, int32_t n) {
  if (!s || !out) return ZM_ERR_INVALID;
  const int32_t v[17] = {s->n_subcyc, s->n_nu, s->adv_nsub, s->conv_nsub, s->P, (int32_t)(s->bytes >> 20),
                         s->kernels_per_step, s->bt_blocks, s->bt.cap_active, s->nu_halo, s->fft_lines,
                         s->d.ta_kc, s->d.lt_kc, s->d.fz_rows, s->d.pg_rows, s->nu_warps,
                         s->pj_tile.blocks > 0 ? s->pj_tile.cpt : 0};
  for (int q = 0; q < n && q < 17; ++q) out[q] = v[q];
  return ZM_OK;
}

int zm_load_state(zm_solver* s, void* stream, const zm_state* in) {
  if (!s || !in || !in->u || !in->v || !in->T || !in->S || !in->eta) return ZM_ERR_INVALID;
  try {
    s->reset_sync((cudaStream_t)stream);
    s->load((cudaStream_t)stream, in, s->st[s->cur], s->eta[s->cur]);
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_store_state(zm_solver* s, void* stream, zm_state* out) {
  if (!s || !out || !out->u || !out->v || !out->T || !out->S || !out->eta) return ZM_ERR_INVALID;
  try {
    s->store((cudaStream_t)stream, s->st[s->cur], s->eta[s->cur], out);
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_advance(zm_solver* s, void* stream, int32_t nsteps) {
  if (!s || nsteps < 0) return ZM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    if (s->want_tune && !s->tuned) s->autotune(st);
    if (!s->graphs_ready) s->build_graphs();
    for (int n = 0; n < nsteps; ++n) {
      ZM_CUDA(cudaGraphLaunch(s->graph[s->cur], st));
      s->cur = 1 - s->cur;
    }
    s->monitor(st, s->cur, nsteps > 0);
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

// ---------------------------------------------------------------- ensembles

struct zm_ensemble {
  std::vector<zm_solver*> m;
  std::vector<int> parity;      // members' state index when graph[0] was captured
  std::vector<unsigned> built;  // their own captures then
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  bool ready = false;
  cudaStream_t cap = nullptr;
  std::vector<cudaStream_t> side;
  std::vector<cudaEvent_t> fork, join, bt;
  int launches = 0;
  ~zm_ensemble() {
    for (int g = 0; g < 2; ++g)
      if (graph[g]) cudaGraphExecDestroy(graph[g]);
    for (auto e : fork) cudaEventDestroy(e);
    for (auto e : join) cudaEventDestroy(e);
    for (auto e : bt) cudaEventDestroy(e);
    for (auto st : side) cudaStreamDestroy(st);
    if (cap) cudaStreamDestroy(cap);
  }
  // one graph stepping every member once, members on forked streams
  void capture() {
    for (int g = 0; g < 2; ++g) {
      if (graph[g]) {
        cudaGraphExecDestroy(graph[g]);
        graph[g] = nullptr;
      }
    }
    parity.resize(m.size());
    built.resize(m.size());
    for (size_t q = 0; q < m.size(); ++q) {
      parity[q] = m[q]->cur;
      built[q] = m[q]->graphs_built;
    }
    for (int g = 0; g < 2; ++g) {
      cudaGraph_t def = nullptr;
      ZM_CUDA(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
      int count = 0;
      try {
        ZM_CUDA(cudaEventRecord(fork[0], cap));
        for (size_t q = 0; q < m.size(); ++q) {
          zm_solver* s = m[q];
          ZM_CUDA(cudaStreamWaitEvent(side[q], fork[0], 0));
          s->bt_wait = q > 0 ? bt[q - 1] : nullptr;
          s->bt_done = bt[q];
          const int from = g == 0 ? parity[q] : 1 - parity[q];
          const int before = s->launch_count;
          s->full_step(side[q], from, 1 - from);
          count += s->launch_count - before;
          s->bt_wait = s->bt_done = nullptr;
          ZM_CUDA(cudaEventRecord(join[q], side[q]));
          ZM_CUDA(cudaStreamWaitEvent(cap, join[q], 0));
        }
      } catch (...) {
        for (auto* s : m) s->bt_wait = s->bt_done = nullptr;
        cudaStreamEndCapture(cap, &def);
        if (def) cudaGraphDestroy(def);
        throw;
      }
      ZM_CUDA(cudaStreamEndCapture(cap, &def));
      ZM_CUDA(cudaGraphInstantiate(&graph[g], def, 0));
      cudaGraphDestroy(def);
      launches = count;
    }
    ready = true;
  }
};

int zm_ensemble_create(zm_solver* const* members, int32_t n, zm_ensemble** out) {
  if (!members || n < 1 || !out) return ZM_ERR_INVALID;
  for (int q = 0; q < n; ++q)
    if (!members[q]) return ZM_ERR_INVALID;
  for (int q = 0; q < n; ++q)
    for (int r = q + 1; r < n; ++r)
      if (members[q] == members[r]) return ZM_ERR_INVALID;
  auto* e = new zm_ensemble();
  e->m.assign(members, members + n);
  bool ok = cudaStreamCreateWithFlags(&e->cap, cudaStreamNonBlocking) == cudaSuccess;
  e->side.resize(n, nullptr);
  e->fork.resize(1, nullptr);
  e->join.resize(n, nullptr);
  e->bt.resize(n, nullptr);
  ok = ok && cudaEventCreateWithFlags(&e->fork[0], cudaEventDisableTiming) == cudaSuccess;
  for (int q = 0; q < n && ok; ++q) {
    ok = cudaStreamCreateWithFlags(&e->side[q], cudaStreamNonBlocking) == cudaSuccess &&
         cudaEventCreateWithFlags(&e->join[q], cudaEventDisableTiming) == cudaSuccess &&
         cudaEventCreateWithFlags(&e->bt[q], cudaEventDisableTiming) == cudaSuccess;
  }
  if (!ok) {
    delete e;
    return ZM_ERR_CUDA;
  }
  *out = e;
  return ZM_OK;
}

int zm_ensemble_advance(zm_ensemble* e, void* stream, int32_t nsteps, int32_t* kernels_per_step) {
  if (!e || nsteps < 0) return ZM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    // a capture exists, every member still has the graphs it had then (no
    // closure change, no tuning), and all members stepped alike since
    bool stale = !e->ready || e->parity.size() != e->m.size();
    int rel = 0;
    if (!stale) {
      rel = -1;
      for (size_t q = 0; q < e->m.size(); ++q) {
        if (!e->m[q]->graphs_ready || e->m[q]->graphs_built != e->built[q]) stale = true;
        const int r = e->m[q]->cur == e->parity[q] ? 0 : 1;
        if (rel < 0) rel = r;
        else if (r != rel) stale = true;
      }
    }
    if (stale) {
      for (auto* s : e->m) {
        if (s->want_tune && !s->tuned) s->autotune(st);
        if (!s->graphs_ready) s->build_graphs();
      }
      ZM_CUDA(cudaDeviceSynchronize());
      e->capture();
      rel = 0;
    }
    for (int n = 0; n < nsteps; ++n) {
      ZM_CUDA(cudaGraphLaunch(e->graph[rel], st));
      for (auto* s : e->m) s->cur = 1 - s->cur;
      rel = 1 - rel;
    }
    for (auto* s : e->m) s->monitor(st, s->cur, nsteps > 0);
    if (kernels_per_step) *kernels_per_step = e->launches;
  } catch (const Err& err) {
    std::fprintf(stderr, "zm_ensemble_advance: %s\n", err.msg.c_str());
    return err.code;
  }
  return ZM_OK;
}

void zm_ensemble_destroy(zm_ensemble* e) { delete e; }

int zm_step(zm_solver* s, void* stream, const zm_state* in, zm_state* out, int32_t nsteps) {
  int rc = zm_load_state(s, stream, in);
  if (rc) return rc;
  rc = zm_advance(s, stream, nsteps);
  if (rc) return rc;
  return zm_store_state(s, stream, out);
}

int zm_step_host(zm_solver* s, void* stream, const zm_state* in, zm_state* out, int32_t nsteps) {
  if (!s || !in || !out) return ZM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    if (!s->copy_stream) {
      ZM_CUDA(cudaStreamCreateWithFlags(&s->copy_stream, cudaStreamNonBlocking));
      for (cudaEvent_t& e : s->ev_copy) ZM_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    cudaStream_t cs = s->copy_stream;
    cudaEvent_t* ev = s->ev_copy;  // [0] start, [1..5] inputs copied, [6..10] outputs laid out
    const size_t b3 = (size_t)s->nx * s->ny * s->nz * sizeof(float), b2 = (size_t)s->nx * s->ny * sizeof(float);
    float* ref[5] = {s->ref.u, s->ref.v, s->ref.T, s->ref.S, s->ref_eta};
    const float* hin[5] = {in->u, in->v, in->T, in->S, in->eta};
    float* hout[5] = {out->u, out->v, out->T, out->S, out->eta};
    Fields4& a = s->st[s->cur];
    float* fin[4] = {a.u, a.v, a.T, a.S};
    const float offs[4] = {0.f, 0.f, s->d.T_ref, s->d.S_ref};
    // the copies start after the work already queued on the caller's stream
    ZM_CUDA(cudaEventRecord(ev[0], st));
    ZM_CUDA(cudaStreamWaitEvent(cs, ev[0], 0));
    s->reset_sync(st);
    const void* all[10];
    for (int f = 0; f < 5; ++f) all[f] = hin[f], all[5 + f] = hout[f];
    // Pageable arrays are staged by several threads, pinned ones copied directly.
    if (HostStage::pageable(all, 10) && s->stage.wanted(4 * b3 + b2) && s->stage.ready()) {
      HostStage::Piece up[5], down[5];
      for (int f = 0; f < 5; ++f) {
        const size_t n = f < 4 ? b3 : b2;
        up[f] = {const_cast<char*>(reinterpret_cast<const char*>(hin[f])), reinterpret_cast<char*>(ref[f]), n};
        down[f] = {reinterpret_cast<char*>(hout[f]), reinterpret_cast<char*>(ref[f]), n};
      }
      int rc = ZM_OK;
      ZM_CUDA(s->stage.run(s->device, cs, up, down, 5, [&] {
        ZM_CUDA(cudaEventRecord(ev[1], cs));
        ZM_CUDA(cudaStreamWaitEvent(st, ev[1], 0));
        const zm_state r{ref[0], ref[1], ref[2], ref[3], ref[4]};
        s->load(st, &r, a, s->eta[s->cur]);
        rc = zm_advance(s, stream, nsteps);
        if (rc) return false;
        zm_state o = r;
        s->store(st, s->st[s->cur], s->eta[s->cur], &o);
        ZM_CUDA(cudaEventRecord(ev[6], st));
        ZM_CUDA(cudaStreamWaitEvent(cs, ev[6], 0));
        return true;
      }));
      ZM_CUDA(cudaStreamSynchronize(st));
      return rc;
    }
    for (int f = 0; f < 5; ++f) {
      ZM_CUDA(cudaMemcpyAsync(ref[f], hin[f], f < 4 ? b3 : b2, cudaMemcpyHostToDevice, cs));
      ZM_CUDA(cudaEventRecord(ev[1 + f], cs));
    }
    for (int f = 0; f < 5; ++f) {
      ZM_CUDA(cudaStreamWaitEvent(st, ev[1 + f], 0));
      if (f < 4) s->to_int3(st, ref[f], fin[f], offs[f]);
      else launch_layout(st, s->d, LayoutArgs{{ref[4]}, {s->eta[s->cur]}, {0.f}, 0, 1}, true);
    }
    s->check_launch();
    int rc = zm_advance(s, stream, nsteps);
    if (rc) return rc;
    Fields4& b = s->st[s->cur];
    float* fout[4] = {b.u, b.v, b.T, b.S};
    for (int f = 0; f < 5; ++f) {
      if (f < 4) s->to_ref3(st, fout[f], ref[f], offs[f]);
      else launch_layout(st, s->d, LayoutArgs{{s->eta[s->cur]}, {ref[4]}, {0.f}, 0, 1}, false);
      ZM_CUDA(cudaEventRecord(ev[6 + f], st));
      ZM_CUDA(cudaStreamWaitEvent(cs, ev[6 + f], 0));
      ZM_CUDA(cudaMemcpyAsync(hout[f], ref[f], f < 4 ? b3 : b2, cudaMemcpyDeviceToHost, cs));
    }
    s->check_launch();
    ZM_CUDA(cudaStreamSynchronize(cs));
    ZM_CUDA(cudaStreamSynchronize(st));
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_set_forcing(zm_solver* s, void* stream, const float* tau_x, const float* tau_y, const float* q_heat) {
  if (!s) return ZM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    const dim3 c(32, 8);
    if (tau_x) k_ref_to_int2<<<s->grid2(c), c, 0, st>>>(s->d, tau_x, s->tau_x);
    if (tau_y) k_ref_to_int2<<<s->grid2(c), c, 0, st>>>(s->d, tau_y, s->tau_y);
    if (q_heat) k_ref_to_int2<<<s->grid2(c), c, 0, st>>>(s->d, q_heat, s->qheat);
    s->check_launch();
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_set_forcing_seasonal(zm_solver* s, void* stream, const float* tau_x, const float* tau_y, const float* q_heat,
                            double day, double blend_days) {
  if (!s || !std::isfinite(day) || !std::isfinite(blend_days)) return ZM_ERR_INVALID;
  // weights as inputs/forcing/seasonal.py:86-103 forms them (30-day months)
  const double month_len = 30.0;
  const double mpos = std::fmod(day, month_len) + (std::fmod(day, month_len) < 0 ? month_len : 0.0);
  int mi = (int)std::floor(day / month_len) % 12;
  if (mi < 0) mi += 12;
  const int prev = (mi + 11) % 12, next = (mi + 1) % 12;
  double w_after = 0.0, w_before = 0.0;
  if (blend_days > 0.0) {
    const double half = blend_days / 2.0;
    w_after = std::min(1.0, std::max(0.0, (mpos - (month_len - half)) / blend_days));
    w_before = std::min(1.0, std::max(0.0, (half - mpos) / blend_days));
  }
  const float wc = (float)(1.0 - w_after - w_before), wn = (float)w_after, wp = (float)w_before;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    const dim3 c(32, 8);
    const float* stacks[3] = {tau_x, tau_y, q_heat};
    float* outs[3] = {s->tau_x, s->tau_y, s->qheat};
    for (int q = 0; q < 3; ++q)
      if (stacks[q]) k_forcing_blend<<<s->grid2(c), c, 0, st>>>(s->d, stacks[q], prev, mi, next, wp, wc, wn, outs[q]);
    s->check_launch();
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_run_stage(zm_solver* s, void* stream, int32_t stage, const zm_state* in, zm_state* out) {
  if (!s || !in || !out || stage < 1 || stage > 8) return ZM_ERR_INVALID;
  if (stage == 8 && !s->proj_on) return fail(s, Err{ZM_ERR_INVALID, "stage 8 needs project_adv_vel"});
  cudaStream_t st = (cudaStream_t)stream;
  try {
    s->reset_sync(st);
    s->load(st, in, s->st[s->cur], s->eta[s->cur]);
    const int a = s->cur, b = 1 - s->cur;
    if (stage <= 2) {  // the stages leave dry tracers alone; here they are part of the result
      ZM_CUDA(cudaMemcpyAsync(s->st[b].T, s->st[a].T, s->n3 * sizeof(float), cudaMemcpyDeviceToDevice, st));
      ZM_CUDA(cudaMemcpyAsync(s->st[b].S, s->st[a].S, s->n3 * sizeof(float), cudaMemcpyDeviceToDevice, st));
    }
    if (stage == 1) {
      s->linear_half(st, s->st[a], s->st[b]);
    } else if (stage == 2) {
      s->nonlinear(st, s->st[a], s->st[b]);
    } else if (stage == 3) {
      s->full_step(st, a, b);
    } else if (stage == 4) {
      s->momentum_advection_part(st, s->st[a]);
      s->copy_uv(st, s->Au, s->Av, s->st[a], s->st[b]);
    } else if (stage == 5) {
      s->pressure_part(st, s->st[a]);
      s->copy_uv(st, s->Pu, s->Pv, s->st[a], s->st[b]);
    } else if (stage == 6) {
      s->momentum_advection_part(st, s->st[a]);
      s->copy_uv(st, s->Ayu, s->Ayv, s->st[a], s->st[b]);
    } else if (stage == 8) {
      s->project(st, s->st[a].u, s->st[a].v);
      s->copy_uv(st, s->st[a].u, s->st[a].v, s->st[a], s->st[b]);
    } else {
      ZM_CUDA(launch_dealias(st, s->d, s->fft, s->st[a].u, s->st[a].v, s->Au, s->Av, s->fft_lines, s->fft_smem,
                             false));
      s->check_launch();
      s->copy_uv(st, s->Au, s->Av, s->st[a], s->st[b]);
    }
    if (stage != 3)
      ZM_CUDA(cudaMemcpyAsync(s->eta[b], s->eta[a], s->n2 * sizeof(float), cudaMemcpyDeviceToDevice, st));
    s->store(st, s->st[b], s->eta[b], out);
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_profile(zm_solver* s, void* stream, float* ms, int32_t* launches, int32_t n) {
  if (!s || !ms || !launches || n < ZM_K_COUNT) return ZM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    for (int c = 0; c < ZM_K_COUNT; ++c) { ms[c] = 0.f; launches[c] = 0; }
    s->profiling = true;
    s->prof.clear();
    try {
      s->full_step(st, s->cur, 1 - s->cur);
    } catch (...) {
      s->profiling = false;
      throw;
    }
    s->profiling = false;
    s->cur = 1 - s->cur;
    ZM_CUDA(cudaStreamSynchronize(st));
    for (auto& e : s->prof) {
      float t = 0.f;
      ZM_CUDA(cudaEventElapsedTime(&t, e.a, e.b));
      ms[e.cls] += t;
      launches[e.cls] += 1;
      cudaEventDestroy(e.a);
      cudaEventDestroy(e.b);
    }
    s->prof.clear();
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_barrier_probe(zm_solver* s, void* stream, int32_t blocks, int32_t expected, int32_t max_polls) {
  if (!s || blocks < 1 || expected < blocks || max_polls < 1) return ZM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    int sms = 0;
    ZM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device));
    if (blocks > sms) return fail(s, Err{ZM_ERR_INVALID, "barrier probe: more blocks than SMs"});
    ZM_CUDA(cudaMemsetAsync(s->bt_sync, 0, 4 * sizeof(unsigned), st));
    k_barrier_probe<<<blocks, 32, 0, st>>>(s->bt.bar, s->bt.err, (unsigned)expected, (unsigned)max_polls);
    s->check_launch();
    ZM_CUDA(cudaStreamSynchronize(st));
    unsigned berr = 0;
    ZM_CUDA(cudaMemcpy(&berr, s->bt.err, sizeof(berr), cudaMemcpyDeviceToHost));
    ZM_CUDA(cudaMemsetAsync(s->bt_sync, 0, 4 * sizeof(unsigned), st));
    ZM_CUDA(cudaStreamSynchronize(st));
    if (berr) return fail(s, Err{ZM_ERR_TIMEOUT, "barrier probe timed out"});
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_set_wait_limit(zm_solver* s, int32_t max_polls) {
  if (!s) return ZM_ERR_INVALID;
  try {
    s->set_wait_limit(max_polls < 0 ? ZM_BT_BARRIER_POLLS : (unsigned)max_polls);
    ZM_CUDA(cudaDeviceSynchronize());
    s->drop_graphs();
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_diagnostics(zm_solver* s, void* stream, const zm_state* in, const float* surface_pressure_pa, float* rho,
                   float* pressure, float* w) {
  if (!s || !in || !in->u || !in->v || !in->T || !in->S || !in->eta || !rho || !pressure || !w)
    return ZM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    // the caller's state goes to work buffers that are idle between steps
    s->load(st, in, s->L, s->frx);
    const float* sp = nullptr;
    const dim3 c(32, 4);
    if (surface_pressure_pa) {
      k_ref_to_int2<<<s->grid2(dim3(32, 8)), dim3(32, 8), 0, st>>>(s->d, surface_pressure_pa, s->fry);
      sp = s->fry;
    }
    launch_fz(st, s->d, s->L.u, s->L.v, s->Fz);
    k_diagnostics<<<s->grid2(c), c, 0, st>>>(s->d, s->L.T, s->L.S, s->frx, s->Fz, sp, s->W1.u, s->W1.v, s->W2.u);
    s->check_launch();
    launch_layout(st, s->d, LayoutArgs{{s->W1.u, s->W1.v, s->W2.u}, {rho, pressure, w}, {}, 3, 0}, false);
    s->check_launch();
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_tracer_terms(zm_solver* s, void* stream, const zm_state* in, float* terms) {
  if (!s || !in || !in->u || !in->v || !in->T || !in->S || !in->eta || !terms) return ZM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t nref = (size_t)s->nx * s->ny * s->nz;
  try {
    // the caller's state goes to work buffers that are idle between steps
    s->load(st, in, s->L, s->frx);
    launch_fz(st, s->d, s->L.u, s->L.v, s->Fz);
    launch_tracer_terms(st, s->d, s->L.T, s->L.S, s->L.u, s->L.v, s->Fz, s->W1.u, s->W1.v, s->W1.T, s->W1.S);
    s->check_launch();
    launch_layout(st, s->d, LayoutArgs{{s->W1.u, s->W1.v, s->W1.T, s->W1.S},
                                       {terms, terms + nref, terms + 2 * nref, terms + 3 * nref}, {}, 4, 0}, false);
    s->check_launch();
    ZM_CUDA(cudaMemsetAsync(terms + 4 * nref, 0, 2 * nref * sizeof(float), st));  // GM, Redi: off
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_budgets(zm_solver* s, void* stream, const float* T, const float* S, double rho0, double cp, double* out) {
  if (!s || !T || !S || !out || !std::isfinite(rho0) || !std::isfinite(cp)) return ZM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  double sums[2 * ZM_BUDGET_SUMS];
  try {
    k_budget_partials<<<s->bblocks, 256, 0, st>>>(s->d, T, S, s->area64, s->width64, s->bpart);
    k_budget_final<<<1, 32 * ZM_BUDGET_SUMS, 0, st>>>(s->bpart, s->bblocks, s->bout);
    s->check_launch();
    ZM_CUDA(cudaMemcpyAsync(sums, s->bout, sizeof(sums), cudaMemcpyDeviceToHost, st));
    ZM_CUDA(cudaStreamSynchronize(st));
  } catch (const Err& e) {
    return fail(s, e);
  }
  double v[ZM_BUDGET_SUMS];
  for (int q = 0; q < ZM_BUDGET_SUMS; ++q) v[q] = sums[2 * q] + sums[2 * q + 1];
  if (!(v[0] > 0.0)) return fail(s, Err{ZM_ERR_INVALID, "total wet volume is zero; check the grid/mask"});
  out[0] = v[1] / v[0];          // mean_T
  out[1] = v[2] / v[0];          // mean_S
  out[2] = v[4] / v[3];          // mean_T_top
  out[3] = v[5] / v[3];          // mean_S_top
  out[4] = rho0 * cp * v[1];     // heat_content_J
  out[5] = rho0 / 1000.0 * v[2]; // salt_content_kg
  out[6] = v[0];                 // total_volume_m3
  out[7] = v[0] / v[6];          // mean_depth_m
  return ZM_OK;
}

int zm_set_closure(zm_solver* s, void* stream, const float* params, float bound) {
  if (!s || (params && !(bound > 0.f))) return ZM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    if (params) {
      if (s->nz > 51) return fail(s, Err{ZM_ERR_UNSUPPORTED, "the learned closure covers at most 50 levels"});
      if (!s->kappa3) {
        s->kappa3 = s->alloc<float>((size_t)std::max(1, s->nz - 1) * s->d.plane);
        s->cl_count = s->alloc<unsigned>(2);
        __nv_bfloat16* W = s->alloc<__nv_bfloat16>((size_t)(2 * ZM_MLP_IN + ZM_MLP_OUT) * ZM_MLP_IN);
        float* b = s->alloc<float>(2 * ZM_MLP_IN + ZM_MLP_OUT);
        s->cw = MlpTc{W, b, b + ZM_MLP_IN, b + 2 * ZM_MLP_IN};
        ZM_CUDA(cudaFuncSetAttribute(k_mlp_closure, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp_tc_smem()));
      }
      const int rc = zm_mlp_pack_tc(stream, params, (void*)s->cw.packed);
      if (rc != ZM_OK) return fail(s, Err{rc, "packing the closure weights failed"});
      const long long off_b1 = (long long)ZM_MLP_IN * ZM_MLP_IN, off_b2 = 2 * off_b1 + ZM_MLP_IN,
                      off_b3 = off_b2 + ZM_MLP_IN + (long long)ZM_MLP_OUT * ZM_MLP_IN;
      float* b = const_cast<float*>(s->cw.b1);
      ZM_CUDA(cudaMemcpyAsync(b, params + off_b1, ZM_MLP_IN * sizeof(float), cudaMemcpyDeviceToDevice, st));
      ZM_CUDA(cudaMemcpyAsync(b + ZM_MLP_IN, params + off_b2, ZM_MLP_IN * sizeof(float), cudaMemcpyDeviceToDevice, st));
      ZM_CUDA(cudaMemcpyAsync(b + 2 * ZM_MLP_IN, params + off_b3, ZM_MLP_OUT * sizeof(float),
                              cudaMemcpyDeviceToDevice, st));
      ZM_CUDA(cudaMemsetAsync(s->cl_count, 0, 2 * sizeof(unsigned), st));
    }
    const bool on = params != nullptr;
    if (on != s->closure_on || (on && bound != s->cl_bound)) {  // the captured steps change shape or hold the old bound
      if (on) s->cl_bound = bound;
      s->closure_on = on;
      ZM_CUDA(cudaStreamSynchronize(st));
      s->drop_graphs();
    }
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_autotune(zm_solver* s, void* stream, int32_t* nu_halo, int32_t* fft_lines) {
  if (!s) return ZM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    s->autotune(st);
    s->drop_graphs();
  } catch (const Err& e) {
    return fail(s, e);
  }
  if (nu_halo) *nu_halo = s->nu_halo;
  if (fft_lines) *fft_lines = s->fft_lines;
  return ZM_OK;
}

int zm_closure_stats(zm_solver* s, uint32_t* fallback_columns, uint32_t* wait_errors) {
  if (!s || !fallback_columns || !wait_errors) return ZM_ERR_INVALID;
  if (!s->cl_count) {
    *fallback_columns = 0;
    *wait_errors = 0;
    return ZM_OK;
  }
  unsigned c[2];
  const cudaError_t e = cudaMemcpy(c, s->cl_count, sizeof(c), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return fail(s, Err{ZM_ERR_CUDA, std::string("zm_closure_stats: ") + cudaGetErrorString(e)});
  *fallback_columns = c[0];
  *wait_errors = c[1];
  return c[1] ? ZM_ERR_TIMEOUT : ZM_OK;
}

int zm_closure_kappa(zm_solver* s, void* stream, const zm_state* in, float* kappa) {
  if (!s || !in || !in->u || !in->v || !in->T || !in->S || !in->eta || !kappa) return ZM_ERR_INVALID;
  if (!s->closure_on) return fail(s, Err{ZM_ERR_INVALID, "zm_closure_kappa: no closure set"});
  cudaStream_t st = (cudaStream_t)stream;
  try {
    s->load(st, in, s->L, s->frx);
    s->closure(st, s->L);
    const long long ncol = (long long)s->nx * s->ny;
    k_kappa_rows<<<(unsigned)((ncol + 127) / 128), 128, 0, st>>>(s->d, s->kappa3, kappa);
    s->check_launch();
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_closure_features(zm_solver* s, void* stream, const zm_state* in, float* X, float* T, float* M) {
  if (!s || !in || !in->u || !in->v || !in->T || !in->S || !in->eta || !X || !T || !M) return ZM_ERR_INVALID;
  if (s->nz > 51) return fail(s, Err{ZM_ERR_UNSUPPORTED, "the learned closure covers at most 50 levels"});
  cudaStream_t st = (cudaStream_t)stream;
  try {
    s->load(st, in, s->L, s->frx);
    ClosureArgs a{};
    a.T = s->L.T; a.S = s->L.S; a.u = s->L.u; a.v = s->L.v; a.X = X; a.Tt = T; a.Mt = M;
    const long long ncol = (long long)s->nx * s->ny;
    k_closure_features<<<(unsigned)((ncol + 127) / 128), 128, 0, st>>>(s->d, a);
    s->check_launch();
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_status(zm_solver* s, int32_t* monitor_code) {
  if (!s || !monitor_code) return ZM_ERR_INVALID;
  unsigned int f = 0;
  cudaError_t e = cudaMemcpy(&f, s->flags, sizeof(f), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return fail(s, Err{ZM_ERR_CUDA, std::string("zm_status: ") + cudaGetErrorString(e)});
  *monitor_code = (f & 1u) ? 1 : (f & 2u) ? 3 : (f & 4u) ? 4 : 0;
  unsigned berr = 0;
  e = cudaMemcpy(&berr, s->bt.err, sizeof(berr), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return fail(s, Err{ZM_ERR_CUDA, std::string("zm_status: ") + cudaGetErrorString(e)});
  if (berr) return fail(s, Err{ZM_ERR_TIMEOUT, "barotropic grid barrier timed out"});
  if (s->proj_on) {
    e = cudaMemcpy(&berr, s->pj.err, sizeof(berr), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return fail(s, Err{ZM_ERR_CUDA, std::string("zm_status: ") + cudaGetErrorString(e)});
    if (berr) return fail(s, Err{ZM_ERR_TIMEOUT, "column projection grid barrier timed out"});
  }
  return ZM_OK;
}

int zm_ledger_step(zm_solver* s, void* stream, const zm_state* in, zm_state* out, double* raw, int32_t n) {
  if (!s || !in || !out || !raw || n < ZM_LED_COUNT) return ZM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  try {
    s->ensure_ledger();
    ZM_CUDA(cudaMemsetAsync(s->led_acc, 0, ZM_LED_COUNT * sizeof(double), st));
    s->reset_sync(st);
    s->load(st, in, s->st[s->cur], s->eta[s->cur]);
    const int a = s->cur, b = 1 - s->cur;
    s->ledger_on = true;
    try {
      s->full_step(st, a, b);
    } catch (...) {
      s->ledger_on = false;
      throw;
    }
    s->ledger_on = false;
    s->cur = b;
    s->store(st, s->st[b], s->eta[b], out);
    ZM_CUDA(cudaMemcpyAsync(raw, s->led_acc, ZM_LED_COUNT * sizeof(double), cudaMemcpyDeviceToHost, st));
    ZM_CUDA(cudaStreamSynchronize(st));
  } catch (const Err& e) {
    return fail(s, e);
  }
  return ZM_OK;
}

int zm_projection_stats(zm_solver* s, int32_t* out, int32_t n) {
  if (!s || !out || n < 0) return ZM_ERR_INVALID;
  if (!s->proj_on) return fail(s, Err{ZM_ERR_INVALID, "the column projection is off"});
  int v[4] = {0, 0, 0, 0};
  const cudaError_t e = cudaMemcpy(v, s->pj.stats, sizeof(v), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return fail(s, Err{ZM_ERR_CUDA, std::string("zm_projection_stats: ") + cudaGetErrorString(e)});
  for (int q = 0; q < n && q < 4; ++q) out[q] = v[q];
  return ZM_OK;
}

const char* zm_last_error(const zm_solver* s) { return s ? s->last_error.c_str() : "null solver"; }

void zm_destroy(zm_solver* s) { delete s; }

}  // extern "C"
