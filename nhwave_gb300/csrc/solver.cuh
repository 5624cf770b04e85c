// solver.cuh -- host orchestration of one scenario on one CUDA stream:
// device arena, the reference's subroutine sequence as kernel launches, the
// Poisson solve with FP64 iterative refinement, and field transfer.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "psolve.cuh"
#include "setup_host.h"

namespace nhw {

void set_last_error(const std::string& s);

#define NHW_CU(x)                                                                   \
  do {                                                                              \
    cudaError_t e_ = (x);                                                           \
    if (e_ != cudaSuccess) {                                                        \
      set_last_error(std::string(#x) + ": " + cudaGetErrorString(e_));              \
      return NHW_ERR_CUDA;                                                          \
    }                                                                               \
  } while (0)

inline unsigned cdiv(long long n, int b) { return (unsigned)((n + b - 1) / b); }

class SolverBase {
 public:
  virtual ~SolverBase() {}
  virtual int setup(const double* depth, const double* eta0, const double* uvw0) = 0;
  virtual int get_field(int f, void* host) = 0;
  virtual int set_field(int f, const void* host) = 0;
  virtual int field_shape(int f, int dims[3], int* eb) const = 0;
  virtual int get_scalars(nhw_scalars* out) = 0;
  virtual int set_time(double t, double dt, int rs) = 0;
  virtual int estimate_dt() = 0;
  virtual int update_bathymetry() = 0;
  virtual int update_wave_bc() = 0;
  virtual int set_wave_phases(int n, const double* phases) = 0;
  virtual int set_wave_spectrum(int nf, int nd, const double* freq, const double* dire, const double* spc,
                                const double* phases) = 0;
  virtual int update_mask() = 0;
  virtual int update_vars() = 0;
  virtual int source_terms() = 0;
  virtual int fluxes() = 0;
  virtual int eval_duvw(int istep) = 0;
  virtual int sponge_damping() = 0;
  virtual int eval_turb(int istep) = 0;
  virtual int step() = 0;
  virtual int mass(double* m) = 0;
  virtual int statistics(double* out7) = 0;
  virtual int sync() = 0;
  virtual bool is_setup() const = 0;
  virtual double total_time() const = 0;
  virtual int sim_steps() const = 0;
  virtual int bind() = 0;
  virtual int run_timed(int nsteps, double* ms) = 0;
  virtual int run(int nsteps, int* done) = 0;
  virtual int profile(int on) = 0;
  virtual int profile_report(char* buf, int len) = 0;
  virtual int time_smoother(int reps, long long flush, double* us) = 0;
  virtual int checkpoint_bytes(size_t* bytes) = 0;
  virtual int save_state(void* host, size_t bytes) = 0;
  virtual int load_state(const void* host, size_t bytes) = 0;
};

// a field of the device layout as the caller's dense array (32-bit decode, as
// k_box)
template <class T>
__global__ void __launch_bounds__(256) k_pack(const void* src, int kind, double* dd, int* di, int nx, int ny, int nz,
                                              int sy, long long sz) {
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (unsigned)nx * (unsigned)ny * (unsigned)nz) return;
  const unsigned r = t / (unsigned)nx, k = r / (unsigned)ny;
  const long long s = (int)(t - r * (unsigned)nx) + (long long)sy * (int)(r - k * (unsigned)ny) + sz * (int)k;
  if (kind == 0) dd[t] = (double)((const T*)src)[s];
  else if (kind == 1) dd[t] = ((const double*)src)[s];
  else di[t] = ((const int*)src)[s];
}
template <class T>
__global__ void k_unpack(void* dst, int kind, const double* sd, const int* si, int nx, int ny, int nz, int sy,
                         long long sz) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)nx * ny * nz) return;
  const int i = (int)(t % nx);
  const long long r = t / nx;
  const int j = (int)(r % ny), k = (int)(r / ny);
  const long long s = i + (long long)sy * j + sz * k;
  if (kind == 0) ((T*)dst)[s] = (T)sd[t];
  else if (kind == 1) ((double*)dst)[s] = sd[t];
  else ((int*)dst)[s] = si[t];
}
template <class T>
__global__ void k_single(Dev<T> S, int what) {
  if (gated_off(S)) return;
  if (what == 0) OpSourceArea{}(S, 0, 0);
}
// update_vars: D0 = D, Eta0 = Eta (2-D, FP64), DU0/DV0/DW0 = DU/DV/DW (3-D)
template <class T>
__global__ void __launch_bounds__(256) k_update_vars(Dev<T> S, long long n2, long long n3) {
  if (gated_off(S)) return;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n3; t += (long long)gridDim.x * blockDim.x) {
    S.DU0[t] = S.DU[t];
    S.DV0[t] = S.DV[t];
    S.DW0[t] = S.DW[t];
    if (S.DTke0) {   // k-epsilon (src/nhwave.F:5483-5484)
      S.DTke0[t] = S.DTke[t];
      S.DEps0[t] = S.DEps[t];
    }
    if (S.U0) {   // Orlanski boundary: the previous step's velocities move back one level
      S.U00[t] = S.U0[t]; S.V00[t] = S.V0[t]; S.W00[t] = S.W0[t];
      S.U0[t] = S.U[t]; S.V0[t] = S.V[t]; S.W0[t] = S.W[t];
    }
    if (t < n2) {
      if (S.Eta00) S.Eta00[t] = S.Eta0[t];
      S.D0[t] = S.D[t];
      S.Eta0[t] = S.Eta[t];
    }
  }
}

template <class T>
class Solver final : public SolverBase {
 public:
  nhw_params p{};
  Dev<T> S{};
  cudaStream_t st = nullptr;
  char* arena = nullptr;
  size_t arena_bytes = 0;
  bool estimate_only = false;
  size_t state_bytes = 0;   // arena prefix that holds the prognostic state (grids .. P)
  DevScal* h_sc = nullptr;     // pinned mirror of S.sc
  double* d_out = nullptr;     // small device output
  double* h_out = nullptr;
  double* d_stage = nullptr;   // field staging (double / int32)
  size_t stage_elems = 0;
  size_t n2 = 0, n3 = 0;
  bool ready = false;
  int it_order = 3;
  static constexpr bool kFP32 = sizeof(T) == 4;
  // launch accounting and optional per-kernel CUDA-event timing
  long long launches = 0;
  bool prof_on = false;
  struct Rec { const char* name; cudaEvent_t a, b; };
  std::vector<Rec> recs;
  std::vector<cudaEvent_t> evpool;
  size_t evused = 0;
  cudaEvent_t ev_run0 = nullptr, ev_run1 = nullptr;
  // multigrid hierarchy (level 0 is the fine operator)
  std::vector<MGL<T>> mg;
  bool use_mg = true;
  T mg_w = (T)1;
  int mg_coarse_sweeps = 2;   // red-black sweeps on the coarsest level (fastest of 2, 4, 6 on C2)
  // persistent solve (psolve.cuh): one cooperative launch per pressure solve
  bool use_persistent = false;
  bool use_gmres = false;   // krylov_kernel 2 with multigrid: GMRES (krylov.cuh); else BiCGSTAB
  int ps_nb = 0;             // blocks of the launch
  size_t ps_smem = 0;        // dynamic shared memory per block
  double* ps_part = nullptr; // [2][ps_nb][4] partial sums
  PsGroup<T>* d_group = nullptr;
  cudaError_t launch_err = cudaSuccess;

  cudaEvent_t take_event() {
    if (evused == evpool.size()) {
      cudaEvent_t e;
      cudaEventCreate(&e);
      evpool.push_back(e);
    }
    return evpool[evused++];
  }
  template <class F>
  void L(const char* name, F f) {
    ++launches;
    if (capturing) ++cap_counts[cap_level];
    if (!prof_on) { f(); return; }
    cudaEvent_t a = take_event(), b = take_event();
    cudaEventRecord(a, st);
    f();
    cudaEventRecord(b, st);
    recs.push_back({name, a, b});
  }

  ~Solver() override {
    if (st) cudaStreamSynchronize(st);
    for (auto e : evpool) cudaEventDestroy(e);
    for (auto& g : graphs) cudaGraphExecDestroy(g.exec);
    drop_step_graphs();
    for (auto c : cap_st)
      if (c) cudaStreamDestroy(c);
    if (ev_run0) cudaEventDestroy(ev_run0);
    if (ev_run1) cudaEventDestroy(ev_run1);
    if (arena) cudaFree(arena);
    if (spc_table) cudaFree(spc_table);
    if (h_sc) cudaFreeHost(h_sc);
    if (h_out) cudaFreeHost(h_out);
    if (ev_fork) cudaEventDestroy(ev_fork);
    if (ev_join) cudaEventDestroy(ev_join);
    if (mg_st) cudaStreamDestroy(mg_st);
    if (st) cudaStreamDestroy(st);
  }

  int bind() override {
    NHW_CU(cudaSetDevice(p.device));
    return NHW_OK;
  }
  int create(const nhw_params& q) {
    p = q;
    int rc = check_params(p);
    if (rc) return rc;
    rc = bind();
    if (rc) return rc;
    const int M = p.Mglob, N = p.Nglob, K = p.Kglob;
    S.M = M; S.N = N; S.K = K;
    S.Mloc = M + 2 * NG; S.Nloc = N + 2 * NG; S.Kloc = K + 2 * NG;
    S.sy = S.Mloc + 1;
    S.sz = (long long)S.sy * (S.Nloc + 1);
    S.IB = NG; S.IE = M + NG - 1; S.JB = NG; S.JE = N + NG - 1; S.KB = NG; S.KE = K + NG - 1;
    S.neq = M * N * K;
    // column-walk matvecs: two chunks of levels per column on tall grids
    // (twice the threads; each chunk reloads one level above and below)
    S.col_chunks = K >= 16 ? 2 : 1;
    S.col_kc = (K + S.col_chunks - 1) / S.col_chunks;
    S.dx = p.dx; S.dy = p.dy; S.min_dep = p.min_dep; S.cfl = p.cfl;
    S.cxx = -1. / (p.dx * p.dx); S.cyy = -1. / (p.dy * p.dy);
    S.i2dx = 0.5 / p.dx; S.i2dy = 0.5 / p.dy;
    S.dxT = (T)p.dx; S.hdxT = (T)(0.5 * p.dx); S.idxT = (T)(1.0 / p.dx);
    S.dyT = (T)p.dy; S.hdyT = (T)(0.5 * p.dy); S.idyT = (T)(1.0 / p.dy);
    S.dt_min = p.dt_min; S.dt_max = p.dt_max;
    S.fcor = 2.0 * (double)7.29e-5f * std::sin(p.slat);
    S.froude_on = p.froude_cap_on; S.froude_cap = p.froude_cap;
    S.tol = p.tol; S.itmax = p.itmax;
    S.max_ir = kFP32 ? 12 : 30;
    // Each refinement sweep's BiCGSTAB stops at this fraction of its own
    // starting residual (or at the outer tolerance, if that needs less), and
    // the next sweep restarts from a fresh FP64 residual: a Krylov solve
    // driven deeper converges more slowly per iteration.  FP32 form, against
    // a floor of 2e-5: C2 7.25 -> 6.87 iterations per solve and 10.96 ->
    // 10.58 ms/step, C3 14.97 -> 13.96 (1e-4 to 5e-4 alike; 1e-3 slower
    // again).  FP64 form, against one sweep to the tolerance: C2 46.95 ->
    // 45.88, C3 61.70 -> 59.34 ms/step (1e-2 and above slower on C3).
    S.tol_floor = kFP32 ? 2e-4 : 3e-3;
    S.total_time = p.total_time; S.sim_steps = p.sim_steps;
    S.graph_mode = 0; S.h_go = S.h_ir = S.h_inner = 0;
    S.non_hydro = p.non_hydro; S.sponge_on = p.sponge_on;
    S.hllc = p.hllc ? 1 : 0;
    S.bc_x0 = p.bc_x0; S.bc_xn = p.bc_xn; S.bc_y0 = p.bc_y0; S.bc_yn = p.bc_yn;
    S.visc_top = kSmall + 0.5 * (p.visc + 0.0 + 0.0 + p.visc + 0.0 + 0.0);
    S.v_cmu = p.visc;
    S.bc_z0 = p.bc_z0; S.ibot = p.ibot; S.cd0 = p.cd0; S.zob = p.zob;
    S.viscous = p.viscous_flow ? 1 : 0;
    if (S.viscous) {   // seeding viscosity of initial (src/initialize.F:3172-3195)
      const double tke = (double)1.e-9f, eps = (double)1.e-9f;
      S.v_cmut0 = (p.rng ? (double)8.5e-2f : (double)9.0e-2f) * (tke * tke) / eps;
      S.v_cmu = p.visc; S.v_cvs = p.cvs; S.v_chs = p.chs;
      S.v_schmidt = p.schmidt; S.v_number = p.viscous_number;
      S.ivturb = p.ivturb; S.ihturb = p.ihturb;
      S.ke_rng = p.rng ? 1 : 0; S.ke_prod = p.prod_type; S.ke_dmin = 2.0 * p.min_dep;
      const int w = p.wavemaker;   // WaveMaker(1:3) is INT, LEF or FOC
      S.ke_quiet = (w == NHW_WM_INT_LIN || w == NHW_WM_INT_SOL || w == NHW_WM_INT_CON || w == NHW_WM_INT_JON ||
                    w == NHW_WM_INT_TMA || w == NHW_WM_INT_SPC || w == NHW_WM_INT_IRR || w == NHW_WM_LEF_LIN ||
                    w == NHW_WM_LEF_SOL || w == NHW_WM_LEF_STK || w == NHW_WM_LEF_CON || w == NHW_WM_LEF_TID ||
                    w == NHW_WM_LEF_JON || w == NHW_WM_LEF_TMA || w == NHW_WM_LEF_SPC || w == NHW_WM_FOCUSED) ? 1 : 0;
      S.les_lef = ((w >= NHW_WM_LEF_LIN && w <= NHW_WM_LEF_CON) || w == NHW_WM_LEF_TID || w == NHW_WM_LEF_JON ||
                   w == NHW_WM_LEF_TMA || w == NHW_WM_LEF_SPC) ? 1 : 0;
      S.les_int = (w == NHW_WM_INT_LIN || w == NHW_WM_INT_SOL || w == NHW_WM_INT_CON || w == NHW_WM_INT_JON ||
                   w == NHW_WM_INT_TMA || w == NHW_WM_INT_SPC || w == NHW_WM_INT_IRR) ? 1 : 0;
    }
    S.wavemaker = p.wavemaker;
    S.wm_amp = p.amp_wave; S.wm_xw = p.xsource_west; S.wm_xe = p.xsource_east;
    S.wm_ys = p.ysource_suth; S.wm_yn = p.ysource_nrth;
    S.cur_wave = p.cur_wave; S.tramp = p.tramp;
    S.slide = p.slide_type == NHW_SLIDE_RIGID_3D;
    if (S.slide) {
      S.sl_e = (double)0.717f;
      const double alpha0 = p.slide_angle * kPi / 180.;
      const double slope0 = p.slope_angle * kPi / 180.;
      S.sl_kb = 2.0 * std::acosh(1.0 / S.sl_e) / p.slide_l;
      S.sl_kw = 2.0 * std::acosh(1.0 / S.sl_e) / p.slide_w;
      S.sl_cosa = std::cos(alpha0); S.sl_sina = std::sin(alpha0);
      S.sl_cosslope = std::cos(slope0);
      S.sl_t0 = p.slide_ut / p.slide_a0;
      S.sl_s0 = p.slide_ut * p.slide_ut / p.slide_a0;
      S.sl_T = p.slide_t; S.sl_x0 = p.slide_x0; S.sl_y0 = p.slide_y0;
    }
    n2 = (size_t)S.sy * (S.Nloc + 1);
    n3 = (size_t)S.sz * (S.Kloc + 1);
    const size_t neq = (size_t)S.neq;
    // ---- arena layout
    std::vector<std::pair<void**, size_t>> plan;
    auto add = [&](auto** ptr, size_t bytes) { plan.push_back({(void**)ptr, bytes}); };
    add(&S.sig, sizeof(double) * (S.Kloc + 1));
    add(&S.dsig, sizeof(double) * S.Kloc);
    add(&S.sigc, sizeof(double) * S.Kloc);
    add(&S.xc, sizeof(double) * S.Mloc);
    add(&S.yc, sizeof(double) * S.Nloc);
    S.nwave = p.wavemaker == NHW_WM_FOCUSED ? p.nwave : 0;
    S.foc_xb = p.x_breaking; S.foc_tb = p.t_breaking; S.foc_dc = p.depth_comp; S.foc_sd = p.sd_return;
    if (S.nwave) add((double**)&S.foc, sizeof(double) * 3 * S.nwave);
    S.njon = (p.wavemaker == NHW_WM_LEF_JON || p.wavemaker == NHW_WM_LEF_TMA || p.wavemaker == NHW_WM_INT_JON ||
              p.wavemaker == NHW_WM_INT_TMA) ? p.numfreq : 0;
    if (S.njon) add((double**)&S.jon, sizeof(double) * kJonSlots * S.njon);
    for (const double** lv : {&S.lv_x, &S.lv_y, &S.lv_up, &S.lv_dn, &S.lv_h, &S.lv_ds, &S.lv_fint})
      add((double**)lv, sizeof(double) * S.Kloc);
    add((T**)&S.lvT, sizeof(T) * 3 * S.Kloc);
    double** d2[] = {&S.D, &S.D0, &S.Eta, &S.Eta0, &S.Hc, &S.Hc0, &S.Ho, &S.Hfx, &S.Hfy, &S.Hfx0, &S.Hfy0,
                     &S.DelxH, &S.DelyH, &S.DeltH, &S.DeltHo, &S.Delt2H, &S.DelxEta, &S.DelyEta, &S.SourceX,
                     &S.SourceY, &S.SourceC, &S.Sponge, &S.R1, &S.Wsx, &S.Wsy, &S.EtaxL, &S.EtaxR, &S.EtayL,
                     &S.EtayR, &S.zUL, &S.zVL, &S.zWL, &S.zUR, &S.zVR, &S.zWR,
                     &S.cf_hx, &S.cf_ex, &S.cf_hy, &S.cf_ey, &S.cf_invD};
    for (auto pp : d2) add(pp, sizeof(double) * n2);
    int** i2p[] = {&S.Mask, &S.MaskT, &S.Mask_Struct, &S.Mask9};
    for (auto pp : i2p) add(pp, sizeof(int) * n2);
    T** t3[] = {&S.U, &S.V, &S.W, &S.DU, &S.DV, &S.DW, &S.DU0, &S.DV0, &S.DW0, &S.Omega,
                &S.Ex, &S.Fx, &S.Gx, &S.Hx, &S.Ey, &S.Fy, &S.Gy, &S.Hy, &S.Fz, &S.Gz, &S.Hz};
    for (auto pp : t3) add(pp, sizeof(T) * n3);
    if (p.bc_xn == 6 || p.bc_xn == 3) {   // east boundary: two earlier time levels (checkpointed state)
      add(&S.Eta00, sizeof(double) * n2);
      for (T** pp : {&S.U0, &S.V0, &S.W0, &S.U00, &S.V00, &S.W00}) add(pp, sizeof(T) * n3);
    }
    if (p.bc_xn == 3)   // FLUX_LR's outflow velocities of this and the previous step (checkpointed state)
      for (double** pp : {&S.Uxni, &S.Uxni0}) add(pp, sizeof(double) * S.Nloc * S.Kloc);
    if (p.viscous_flow) {   // sigma_transform's inputs, read by the next stage, and the
      // eddy viscosities of the last eval_turb (checkpointed state)
      for (double** pp : {&S.scD, &S.scEx, &S.scEy, &S.scHx, &S.scHy}) add(pp, sizeof(double) * n2);
      for (T** pp : {&S.CmuVt, &S.CmuHt}) add(pp, sizeof(T) * n3);
    }
    const bool ke = p.viscous_flow && (p.ivturb == 10 || p.ivturb == 3);
    if (ke)   // k-epsilon state (checkpointed)
      for (T** pp : {&S.Tke, &S.Eps, &S.DTke, &S.DEps, &S.DTke0, &S.DEps0}) add(pp, sizeof(T) * n3);
    add(&S.P, sizeof(double) * n3);
    if (p.viscous_flow) {   // explicit viscous terms of the stage, sigma slopes, level constants
      for (T** pp : {&S.Dxx, &S.Dxy, &S.Dyx, &S.Dyy, &S.Dzx, &S.Dzy, &S.vsx, &S.vsy, &S.vlx, &S.vly})
        add(pp, sizeof(T) * n3);
      add((double**)&S.lvv, sizeof(double) * kLvN * S.Kloc);
    }
    if (p.viscous_flow && p.ivturb == 30) {   // dynamic LES scratch
      S.ld_n = (long long)n3;
      add(&S.ld, sizeof(T) * n3 * 31);
    }
    if (ke && p.ivturb == 10) {   // slopes the 3-D production reads, surface values of the stage
      for (T** pp : {&S.keDxU, &S.keDyU, &S.keDxV, &S.keDyV, &S.keDxW, &S.keDyW}) add(pp, sizeof(T) * n3);
      for (double** pp : {&S.keTopK, &S.keTopE}) add(pp, sizeof(double) * n2);
    }
    // west-boundary wave values, recomputed every step (after the checkpointed state)
    add(&S.Ein, sizeof(double) * S.Nloc);
    add(&S.Din, sizeof(double) * S.Nloc);
    for (double** pp : {&S.Uin, &S.Vin, &S.Win}) add(pp, sizeof(double) * S.Nloc * S.Kloc);
    if (p.bc_xn == 3) {   // east-boundary values, recomputed every step
      for (double** pp : {&S.Ein_xn, &S.Din_xn}) add(pp, sizeof(double) * S.Nloc);
      for (double** pp : {&S.Uin_xn, &S.Vin_xn, &S.Win_xn}) add(pp, sizeof(double) * S.Nloc * S.Kloc);
    }
    add(&S.coef64, sizeof(double) * NCOMPACT * neq);
    add(&S.rhs64, sizeof(double) * neq);
    add(&S.xsol64, sizeof(double) * neq);
    add(&S.res64, sizeof(double) * neq);
    if (kFP32) add(&S.coefT, sizeof(T) * NCOMPACT * neq);
    T** tk[] = {&S.lcp, &S.linv, &S.kx, &S.kr, &S.kr0, &S.kp, &S.kph, &S.kv, &S.ks, &S.ksh, &S.kt};
    for (auto pp : tk) add(pp, sizeof(T) * neq);
    add(&S.partials, sizeof(double) * 8 * (cdiv((long long)neq, 256) + 8));
    // multigrid levels: horizontal 2x2 aggregation while a direction has >= 4 cells
    use_mg = p.precond == 0;
    use_gmres = use_mg && p.krylov_kernel == 2;
    mg_w = (T)(p.mg_weight > 0.f ? p.mg_weight : 1.0f);
    if (p.mg_coarse_sweeps > 0) mg_coarse_sweeps = p.mg_coarse_sweeps;
    if (p.mg_cta_columns > 0) cta_columns = p.mg_cta_columns;
    mg.clear();
    {
      MGL<T> L0{};
      L0.M = M; L0.N = N; L0.K = K; L0.n = M * N * K;
      mg.push_back(L0);
      double ratio = p.dy / p.dx;   // spacing ratio of the level, as far as the first levels even it out
      int semi = 0;
      while (use_mg && mg.size() < kPsMaxLevels) {
        MGL<T>& f = mg.back();
        // Aggregates of agg x agg columns while a direction keeps at least two
        // aggregates; by default 2 x 2, and 4 x 4 on the last levels -- one
        // launched level fewer.  4 x 4 starts at 1024 columns on narrow
        // levels and at 512 where both sides are above 16: there the first
        // 4 x 4 level costs iterations (basin 200 x 300 x 12 FP32+IR: 5.2 ->
        // 4.2 a solve, 5.77 -> 5.10 ms/step; 64 x 64 x 10 3.51 -> 2.91; from
        // 256 columns 320 x 320 x 15 is slower again, 8.97 -> 9.37).
        const bool fixed = p.mg_aggregate > 1;
        const int last = std::min(f.M, f.N) > 16 ? 512 : 1024;
        const int agg = fixed ? p.mg_aggregate : ((long long)f.M * f.N <= last ? 4 : 2);
        int rx = f.M >= 2 * agg ? agg : (f.M >= 4 ? 2 : 1), ry = f.N >= 2 * agg ? agg : (f.N >= 4 ? 2 : 1);
        if ((rx == 1 && ry == 1) || f.M * f.N <= 32) break;
        // Grids whose spacings differ by 1.5 times or more: the in-level
        // coupling along the finer spacing is (dy/dx)^2 times the other, and
        // a red-black sweep hardly smooths across the weak one, so the first
        // levels aggregate pairs along the finer spacing alone until the
        // level's spacings are near each other (at most six such levels).
        // Submerged bar 1024 x 64 x 20, dy/dx = 2: 7.3 -> 4.7 iterations a
        // solve, 10.5 -> 8.8 ms/step; 128 x 40 x 12, dy/dx = 1/4: 12.8 ->
        // 4.3, 6.70 -> 3.48.  Drawn at 1.5 because the further level costs
        // as much as it saves there (dy/dx = 1.37: 4.75 -> 5.53 ms/step
        // with it; 1.5: 7.96 -> 7.72).
        // A row of cells has no weak coupling, but pairs save a long one
        // iterations too (1000 x 1: 8.2 -> 7.2).  From 64 cells on they would
        // make a coarsest level of up to 32, which the block's sweeps solve
        // poorly (60 x 1 x 8, dy/dx = 2: 18.6 iterations, 7.2 ms/step FP64; in
        // fours 9.6 and 4.4; 100 x 1, dy/dx = 4: 10.3 -> 7.2).
        const bool last_of_row = (f.M == 1 || f.N == 1) && f.M * f.N <= 64;
        if (!fixed && semi < 6 && !last_of_row) {
          if (rx > 1 && ratio >= 1.5) {
            rx = 2; ry = 1; ratio *= 0.5; ++semi;
          } else if (ry > 1 && ratio * 1.5 <= 1.0) {
            rx = 1; ry = 2; ratio *= 2.0; ++semi;
          }
        }
        f.rx = rx; f.ry = ry;
        f.Mc = (f.M + rx - 1) / rx; f.Nc = (f.N + ry - 1) / ry;
        MGL<T> c{};
        c.M = f.Mc; c.N = f.Nc; c.K = K; c.n = c.M * c.N * K;
        mg.push_back(c);
      }
    }
    std::vector<T**> mgptr;
    if (use_mg) {
      add(&S.sp0, sizeof(T) * 7 * 2 * (size_t)K * N * ((M + 1) / 2));
      if (tiles_at(0)) {
        add(&S.kq, sizeof(T) * neq);
        add(&mg[0].xp, sizeof(T) * neq);
      }
    }
    if (kFP32 && !p.hllc)   // 2-D face states (scratch of one stage)
      for (T** ft : {&S.fxT, &S.fyT}) add(ft, sizeof(T) * 6 * n2);
    for (size_t l = 1; l < mg.size(); ++l) {
      const size_t nl = (size_t)mg[l].n;
      add((T**)&mg[l].coef, sizeof(T) * NCOMPACT * nl);
      // Levels above the tiles' size take the half-sweeps of level 0; so do
      // smaller ones that mg_aggregate keeps off the tiles, in FP32 (160 x 96 x
      // 12 in aggregates of 8: 10.2 -> 9.5 ms/step; FP64 33.4 -> 34.1).
      const bool split = kFP32 || (long long)mg[l].M * mg[l].N > 4096 || tiles_of(mg[l]) > kTiles;
      if (!tiled(mg[l]) && split && (int)l < first_block_level() && (long long)mg[l].M * mg[l].N > cta_columns)
        add((T**)&mg[l].sp, sizeof(T) * 7 * 2 * (size_t)K * mg[l].N * ((mg[l].M + 1) / 2));
      add((T**)&mg[l].lcp, sizeof(T) * nl);
      add((T**)&mg[l].linv, sizeof(T) * nl);
      add(&mg[l].x, sizeof(T) * nl);
      if (tiles_at((int)l)) add(&mg[l].xp, sizeof(T) * nl);
      add(&mg[l].b, sizeof(T) * nl);
    }
    // persistent solve: every block resident (cooperative launch), at most
    // one block per 2048 unknowns
    use_persistent = use_mg && p.krylov_kernel == 1 && (int)mg.size() <= kPsMaxLevels;
    if (use_gmres) {
      add(&S.gmV, sizeof(T) * (kGmMax + 1) * (size_t)neq);
      add(&S.gmZ, sizeof(T) * kGmMax * (size_t)neq);
      add(&S.gmT, sizeof(T) * kGmTSize);
      add(&S.gm, sizeof(double) * kGmSize);
      add(&S.gm_part, sizeof(double) * kGmMax * (size_t)cdiv((long long)neq, 256 * kCPT));
    }
    if (use_mg && (int)mg.size() <= kPsMaxLevels)   // partial sums of the scenario's group, up to kPsMaxBlocks
      add(&ps_part, sizeof(double) * 2 * 4 * kPsMaxBlocks);
    if (use_persistent) {
      ps_smem = sizeof(T) * 4 * 32 * K;
      NHW_CU(cudaFuncSetAttribute(k_psolve<T, kPsBY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ps_smem));
      int dev = 0, nsm = 0, per_sm = 0;
      NHW_CU(cudaGetDevice(&dev));
      NHW_CU(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
      NHW_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_psolve<T, kPsBY>, 32 * kPsBY, ps_smem));
      if (per_sm < 1) {
        set_last_error("persistent solve: no block fits on a multiprocessor");
        return NHW_ERR_CUDA;
      }
      ps_nb = std::max(1, std::min(std::min(per_sm * nsm, kPsMaxBlocks), (int)cdiv((long long)neq, 2048)));
      add(&d_group, sizeof(PsGroup<T>));
    }
    add(&S.sc, sizeof(DevScal));
    add(&d_out, sizeof(double) * 8);
    stage_elems = std::max(n3, (size_t)(S.Mloc + 1) * (S.Nloc + 1) * (S.Kloc + 1));
    add(&d_stage, sizeof(double) * stage_elems);
    size_t total = 0;
    for (auto& e : plan) total += (e.second + 255) & ~size_t(255);
    if (estimate_only) {   // device bytes a scenario would hold, nothing allocated
      arena_bytes = total;
      return NHW_OK;
    }
    NHW_CU(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    NHW_CU(cudaStreamCreateWithFlags(&mg_st, cudaStreamNonBlocking));
    NHW_CU(cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming));
    NHW_CU(cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming));
    cudaError_t e = cudaMalloc((void**)&arena, total);
    if (e != cudaSuccess) {
      set_last_error(std::string("cudaMalloc arena: ") + cudaGetErrorString(e));
      arena = nullptr;
      return NHW_ERR_NOMEM;
    }
    arena_bytes = total;
    NHW_CU(cudaMemsetAsync(arena, 0, total, st));
    size_t off = 0;
    for (auto& e2 : plan) { *e2.first = arena + off; off += (e2.second + 255) & ~size_t(255); }
    // everything a step carries to the next lies in front of the Poisson scratch
    state_bytes = (size_t)((char*)(S.P + n3) - arena);
    if (!kFP32) S.coefT = (T*)S.coef64;
    mg[0].coef = S.coefT;
    mg[0].lcp = S.lcp; mg[0].linv = S.linv; mg[0].sp = S.sp0;
    mg[0].cxx = mg[0].cxl = (T)S.cxx; mg[0].cyy = mg[0].cyl = (T)S.cyy;
    for (size_t l = 1; l < mg.size(); ++l) coarse_couplings(mg[l - 1], mg[l]);
    {
      const int shm = (int)(sizeof(T) * 4 * 32 * 64);
      NHW_CU(cudaFuncSetAttribute(k_mg_smooth_blk<T, true, MgB<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_smooth_blk<T, false, MgB<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_smooth_blk<T, false, MgInP<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_smooth_blk<T, false, MgInS<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
      if constexpr (kFP32) {
        NHW_CU(cudaFuncSetAttribute(k_mg_smooth_split<T, true, MgB<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
        NHW_CU(cudaFuncSetAttribute(k_mg_smooth_split<T, false, MgB<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
        NHW_CU(cudaFuncSetAttribute(k_mg_smooth_split<T, false, MgInP<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
        NHW_CU(cudaFuncSetAttribute(k_mg_smooth_split<T, false, MgInS<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
        NHW_CU(cudaFuncSetAttribute(k_mg_smooth_split<T, false, MgInV<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
      } else {
        NHW_CU(cudaFuncSetAttribute(k_mg_smooth_split_strided<T, true, MgB<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
        NHW_CU(cudaFuncSetAttribute(k_mg_smooth_split_strided<T, false, MgB<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
        NHW_CU(cudaFuncSetAttribute(k_mg_smooth_split_strided<T, false, MgInP<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
        NHW_CU(cudaFuncSetAttribute(k_mg_smooth_split_strided<T, false, MgInS<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
        NHW_CU(cudaFuncSetAttribute(k_mg_smooth_split_strided<T, false, MgInV<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
      }
      NHW_CU(cudaFuncSetAttribute(k_mg_smooth_blk<T, false, MgInV<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm));
    }
    {
      const int shm = (int)tile_smem<TileS, T>(KMAX);
      const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
      NHW_CU(cudaFuncSetAttribute(k_mg_down<T, true, TileS, 1, TileInP<T>>, at, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_down<T, true, TileS, 1, TileInS<T>>, at, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_down<T, false, TileS, 1, TileB<T>>, at, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_up<T, true, TileS, 1>, at, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_up<T, false, TileS, 1>, at, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_down<T, true, TileS, 2, TileInP<T>>, at, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_down<T, true, TileS, 2, TileInS<T>>, at, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_down<T, false, TileS, 2, TileB<T>>, at, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_up<T, true, TileS, 2>, at, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_up<T, false, TileS, 2>, at, shm));
      NHW_CU(cudaFuncSetAttribute(k_mg_cycle<T, 1>, at, (int)cycle_smem<T>(KMAX)));
      NHW_CU(cudaFuncSetAttribute(k_mg_cycle<T, 2>, at, (int)cycle_smem<T>(KMAX)));
    }
    NHW_CU(cudaFuncSetAttribute(k_ke_column<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ke_smem(32, KMAX)));
    NHW_CU(cudaFuncSetAttribute(k_vert_visc<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)vv_smem(KMAX)));
    NHW_CU(cudaFuncSetAttribute(k_mg_cta_cycle<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(sizeof(T) * 4 * 32 * 64)));
    NHW_CU(cudaMallocHost((void**)&h_sc, sizeof(DevScal)));
    NHW_CU(cudaMallocHost((void**)&h_out, sizeof(double) * 8));
    std::memset(h_sc, 0, sizeof(DevScal));
    h_sc->dt = p.dt_ini;
    h_sc->rho_dt = kRho0 / p.dt_ini; h_sc->dt_rho = p.dt_ini / kRho0;
    h_sc->dtmin_bits = (unsigned long long)dbits(kLarge);
    NHW_CU(cudaMemcpyAsync(S.sc, h_sc, sizeof(DevScal), cudaMemcpyHostToDevice, st));
    NHW_CU(cudaStreamSynchronize(st));
    return NHW_OK;
  }
  static long long dbits(double x) { long long b; std::memcpy(&b, &x, 8); return b; }

  // ---------------------------------------------------------------- launchers
  // Threads of a block of independent items: 256, and fewer on small grids so
  // that their blocks reach all 152 SMs -- 2048 columns in blocks of 256 run
  // on 8 of them, each with one SM's FP64 pipe for all its columns (GB300,
  // 256 x 8 x 10 FP64, by block: vel_bc_b 52 -> 34 us with 32)
  static int block_of(long long n) {
    int b = 256;
    while (b > 32 && n < 152LL * 2 * b) b /= 2;
    return b;
  }
  template <class Op> void allcols(Op op) {
    const long long n = (long long)S.Mloc * S.Nloc;
    const int b = block_of(n);
    L(Op::kName, [&] { k_allcols<T, Op><<<cdiv(n, b), b, 0, st>>>(S, op); });
  }
  template <class Op> void incols(Op op) {
    const long long n = (long long)S.M * S.N;
    const int b = block_of(n);
    L(Op::kName, [&] { k_incols<T, Op><<<cdiv(n, b), b, 0, st>>>(S, op); });
  }
  template <class Op> void box(Op op, int nx, int ny, int nz, int ox, int oy, int oz) {
    const long long n = (long long)nx * ny * nz;
    const int b = block_of(n);
    L(Op::kName, [&] { k_box<T, Op><<<cdiv(n, b), b, 0, st>>>(S, op, nx, ny, nz, ox, oy, oz); });
  }
  void dt_min() {
    const long long n = (long long)S.M * S.N;
    const int b = block_of(n);
    L("dt_min", [&] { k_dt_min<T><<<cdiv(n, b), b, 0, st>>>(S); });
  }
  template <class Op> void cells(Op op) { box(op, S.M, S.N, S.K, S.IB, S.JB, S.KB); }
  unsigned red_blocks() const { return cdiv(S.neq, 256 * kCPT); }
  // the column-walk matvec kernels: one thread per column and chunk of levels
  unsigned col_blocks() const { return cdiv((long long)S.M * S.N * S.col_chunks, 256); }
  unsigned matvec_blocks() const { return kColumnWalk<T> ? col_blocks() : red_blocks(); }

  int check() {
    cudaError_t e = launch_err != cudaSuccess ? launch_err : cudaGetLastError();
    launch_err = cudaSuccess;
    if (e != cudaSuccess) {
      set_last_error(std::string("kernel launch: ") + cudaGetErrorString(e));
      if (capturing) cap_ok(e, "kernel launch");
      return NHW_ERR_CUDA;
    }
    return NHW_OK;
  }
  int pull_scalars() {
    NHW_CU(cudaMemcpyAsync(h_sc, S.sc, sizeof(DevScal), cudaMemcpyDeviceToHost, st));
    NHW_CU(cudaStreamSynchronize(st));
    return NHW_OK;
  }
  int sync() override {
    NHW_CU(cudaStreamSynchronize(st));
    return check();
  }
  bool is_setup() const override { return ready; }
  double total_time() const override { return p.total_time; }
  int sim_steps() const override { return p.sim_steps; }

  // -------------------------------------------------------------- fields
  struct FieldDesc { void* ptr; int kind; int nx, ny, nz; };  // kind 0 = T, 1 = double, 2 = int
  FieldDesc desc(int f) const {
    const int Ml = S.Mloc, Nl = S.Nloc, Kl = S.Kloc;
    switch (f) {
      case NHW_F_D: return {S.D, 1, Ml, Nl, 1};
      case NHW_F_D0: return {S.D0, 1, Ml, Nl, 1};
      case NHW_F_ETA: return {S.Eta, 1, Ml, Nl, 1};
      case NHW_F_ETA0: return {S.Eta0, 1, Ml, Nl, 1};
      case NHW_F_HC: return {S.Hc, 1, Ml, Nl, 1};
      case NHW_F_HC0: return {S.Hc0, 1, Ml, Nl, 1};
      case NHW_F_DELXH: return {S.DelxH, 1, Ml, Nl, 1};
      case NHW_F_DELYH: return {S.DelyH, 1, Ml, Nl, 1};
      case NHW_F_DELXETA: return {S.DelxEta, 1, Ml, Nl, 1};
      case NHW_F_DELYETA: return {S.DelyEta, 1, Ml, Nl, 1};
      case NHW_F_DELTH: return {S.DeltH, 1, Ml, Nl, 1};
      case NHW_F_DELT2H: return {S.Delt2H, 1, Ml, Nl, 1};
      case NHW_F_SOURCEX: return {S.SourceX, 1, Ml, Nl, 1};
      case NHW_F_SOURCEY: return {S.SourceY, 1, Ml, Nl, 1};
      case NHW_F_SOURCEC: return {S.SourceC, 1, Ml, Nl, 1};
      case NHW_F_SPONGE: return {S.Sponge, 1, Ml, Nl, 1};
      case NHW_F_R1: return {S.R1, 1, Ml, Nl, 1};
      case NHW_F_HFX: return {S.Hfx, 1, Ml + 1, Nl, 1};
      case NHW_F_HFX0: return {S.Hfx0, 1, Ml + 1, Nl, 1};
      case NHW_F_ETAXL: return {S.EtaxL, 1, Ml + 1, Nl, 1};
      case NHW_F_ETAXR: return {S.EtaxR, 1, Ml + 1, Nl, 1};
      case NHW_F_HFY: return {S.Hfy, 1, Ml, Nl + 1, 1};
      case NHW_F_HFY0: return {S.Hfy0, 1, Ml, Nl + 1, 1};
      case NHW_F_ETAYL: return {S.EtayL, 1, Ml, Nl + 1, 1};
      case NHW_F_ETAYR: return {S.EtayR, 1, Ml, Nl + 1, 1};
      case NHW_F_MASK: return {S.Mask, 2, Ml, Nl, 1};
      case NHW_F_MASK_STRUCT: return {S.Mask_Struct, 2, Ml, Nl, 1};
      case NHW_F_MASK9: return {S.Mask9, 2, Ml, Nl, 1};
      case NHW_F_U: return {S.U, 0, Ml, Nl, Kl};
      case NHW_F_V: return {S.V, 0, Ml, Nl, Kl};
      case NHW_F_W: return {S.W, 0, Ml, Nl, Kl};
      case NHW_F_DU: return {S.DU, 0, Ml, Nl, Kl};
      case NHW_F_DV: return {S.DV, 0, Ml, Nl, Kl};
      case NHW_F_DW: return {S.DW, 0, Ml, Nl, Kl};
      case NHW_F_DU0: return {S.DU0, 0, Ml, Nl, Kl};
      case NHW_F_DV0: return {S.DV0, 0, Ml, Nl, Kl};
      case NHW_F_DW0: return {S.DW0, 0, Ml, Nl, Kl};
      case NHW_F_P: return {S.P, 1, Ml, Nl, Kl};
      case NHW_F_OMEGA: return {S.Omega, 0, Ml, Nl, Kl + 1};
      case NHW_F_EX: return {S.Ex, 0, Ml + 1, Nl, Kl};
      case NHW_F_FX: return {S.Fx, 0, Ml + 1, Nl, Kl};
      case NHW_F_GX: return {S.Gx, 0, Ml + 1, Nl, Kl};
      case NHW_F_HX: return {S.Hx, 0, Ml + 1, Nl, Kl};
      case NHW_F_EY: return {S.Ey, 0, Ml, Nl + 1, Kl};
      case NHW_F_FY: return {S.Fy, 0, Ml, Nl + 1, Kl};
      case NHW_F_GY: return {S.Gy, 0, Ml, Nl + 1, Kl};
      case NHW_F_HY: return {S.Hy, 0, Ml, Nl + 1, Kl};
      case NHW_F_FZ: return {S.Fz, 0, Ml, Nl, Kl + 1};
      case NHW_F_GZ: return {S.Gz, 0, Ml, Nl, Kl + 1};
      case NHW_F_HZ: return {S.Hz, 0, Ml, Nl, Kl + 1};
      case NHW_F_CMUVT: return {S.CmuVt, 0, Ml, Nl, Kl};   // null (no field) on the inviscid path
      case NHW_F_CMUHT: return {S.CmuHt, 0, Ml, Nl, Kl};
      case NHW_F_TKE: return {S.Tke, 0, Ml, Nl, Kl};   // null (no field) unless IVTURB = 10
      case NHW_F_EPS: return {S.Eps, 0, Ml, Nl, Kl};
      case NHW_F_DTKE: return {S.DTke, 0, Ml, Nl, Kl};
      case NHW_F_DEPS: return {S.DEps, 0, Ml, Nl, Kl};
      default: return {nullptr, -1, 0, 0, 0};
    }
  }
  int field_shape(int f, int dims[3], int* eb) const override {
    FieldDesc d = desc(f);
    if (!d.ptr) return NHW_ERR_ARG;
    dims[0] = d.nx; dims[1] = d.ny; dims[2] = d.nz;
    *eb = d.kind == 2 ? 4 : 8;
    return NHW_OK;
  }
  // The device address of `bytes` of page-locked host memory that a kernel can
  // store `elem`-byte values to, nullptr for any other: the address must be a
  // multiple of elem (a copy takes any, a store does not), all of the bytes must
  // lie in one allocation or registration (between two there may be a gap), and
  // the device must be allowed to write them.
  static void* mapped(void* host, size_t bytes, size_t elem) {
    static const auto get = [] {
      void* f = nullptr;
      cudaDriverEntryPointQueryResult r;
      if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &r) != cudaSuccess ||
          r != cudaDriverEntryPointSuccess) {
        cudaGetLastError();
        f = nullptr;
      }
      return reinterpret_cast<decltype(&cuPointerGetAttributes)>(f);
    }();
    if (!get) return nullptr;
    CUmemorytype type = (CUmemorytype)0;   // stays so for pageable memory
    CUdeviceptr dev = 0, start = 0;
    size_t size = 0;
    unsigned managed = 0;
    unsigned long long access = 0;
    CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE,      CU_POINTER_ATTRIBUTE_DEVICE_POINTER,
                                  CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE,
                                  CU_POINTER_ATTRIBUTE_IS_MANAGED,       CU_POINTER_ATTRIBUTE_ACCESS_FLAGS};
    void* out[] = {&type, &dev, &start, &size, &managed, &access};
    if (get(6, what, out, (CUdeviceptr)host) != CUDA_SUCCESS) return nullptr;
    if (type != CU_MEMORYTYPE_HOST || managed || !dev || dev % elem ||
        access != CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE || dev < start || dev - start > size ||
        size - (dev - start) < bytes)
      return nullptr;
    return (void*)dev;
  }
  // Into page-locked memory the packing kernel writes directly, which spares
  // the staging pass and the copy's start (GB300, one field read with its
  // call: 0.6 MB 25 -> 21 us, 3 MB 37 -> 32 us, 13 MB 104 -> 87 us); other host
  // memory (mapped) goes through the staging buffer and the copy engine.
  int get_field(int f, void* host) override {
    FieldDesc d = desc(f);
    if (!d.ptr || !host) return NHW_ERR_ARG;
    const long long n = (long long)d.nx * d.ny * d.nz;
    const size_t elem = d.kind == 2 ? 4 : 8, bytes = (size_t)n * elem;
    void* direct = mapped(host, bytes, elem);
    double* out = direct ? (double*)direct : d_stage;
    k_pack<T><<<cdiv(n, 256), 256, 0, st>>>(d.ptr, d.kind, out, (int*)out, d.nx, d.ny, d.nz, S.sy, S.sz);
    NHW_CU(cudaGetLastError());
    if (!direct) NHW_CU(cudaMemcpyAsync(host, d_stage, bytes, cudaMemcpyDeviceToHost, st));
    NHW_CU(cudaStreamSynchronize(st));
    return NHW_OK;
  }
  int set_field(int f, const void* host) override {
    FieldDesc d = desc(f);
    if (!d.ptr || !host) return NHW_ERR_ARG;
    const long long n = (long long)d.nx * d.ny * d.nz;
    NHW_CU(cudaMemcpyAsync(d_stage, host, n * (d.kind == 2 ? 4 : 8), cudaMemcpyHostToDevice, st));
    k_unpack<T><<<cdiv(n, 256), 256, 0, st>>>(d.ptr, d.kind, d_stage, (const int*)d_stage, d.nx, d.ny, d.nz, S.sy, S.sz);
    NHW_CU(cudaGetLastError());
    NHW_CU(cudaStreamSynchronize(st));
    return NHW_OK;
  }

  // this scenario as one group of the persistent solve: nb blocks from b0
  PsGroup<T> make_group(int nb, int b0, int coarse_sweeps) const {
    PsGroup<T> g{};
    g.S = S;
    g.S.graph_mode = 0;
    const int nl = (int)mg.size();
    for (int l = 0; l < nl; ++l) g.L[l] = mg[l];
    g.nl = first_block_level();   // the first block always solves at least the coarsest level
    g.ntot = nl;
    g.w = mg_w;
    g.coarse_sweeps = coarse_sweeps;
    g.b0 = b0;
    g.nb = nb;
    g.bar_nb = nb + (p.test_barrier_extra > 0 ? p.test_barrier_extra : 0);
    g.part = ps_part;
    return g;
  }
  int upload_group() {
    if (!use_persistent) return NHW_OK;
    const PsGroup<T> g = make_group(ps_nb, 0, mg_coarse_sweeps);
    NHW_CU(cudaMemcpyAsync(d_group, &g, sizeof(g), cudaMemcpyHostToDevice, st));
    NHW_CU(cudaStreamSynchronize(st));
    return NHW_OK;
  }
  bool persistent_capable() const { return use_mg && (int)mg.size() <= kPsMaxLevels; }

  // ---------------------------------------------- capture into an ensemble
  // The ensemble captures this scenario's kernels on a branch stream of its
  // own; every kernel is gated by sc->step_go, which k_dt_finalize sets.
  cudaStream_t ens_saved_st = nullptr;
  int ens_saved_sweeps = 0;
  // root: the ensemble's capture graph (conditional handles belong to it)
  int ens_begin(cudaStream_t s, cudaGraph_t root, int coarse_sweeps) {
    if (!cap_st[0])
      for (auto& c : cap_st) NHW_CU(cudaStreamCreateWithFlags(&c, cudaStreamNonBlocking));
    ens_saved_st = st;
    ens_saved_sweeps = mg_coarse_sweeps;
    mg_coarse_sweeps = coarse_sweeps;
    st = s;
    capturing = true;
    cap_root = root;
    cap_depth = 0;
    cap_level = 3;
    cap_err.clear();
    S.graph_mode = 1;
    S.h_go = 0;
    return NHW_OK;
  }
  int ens_end() {
    st = ens_saved_st;
    mg_coarse_sweeps = ens_saved_sweeps;
    capturing = false;
    S.graph_mode = 0;
    if (!cap_err.empty()) {
      set_last_error(cap_err);
      return NHW_ERR_CUDA;
    }
    return NHW_OK;
  }
  void ens_prefix() {   // estimate_dt (gated), bathymetry, mask, update_vars
    dt_min();
    L("dt_finalize", [&] { k_dt_finalize<T><<<1, 1, 0, st>>>(S, 1); });
    if (S.slide) update_bathymetry();
    update_wave_bc();
    update_mask();
    update_vars();
  }
  void ens_stage_head(int s) {   // source_terms, fluxes, eval_duvw up to the solve
    source_terms();
    fluxes();
    stage_pre(s);
  }
  int ens_solve() { return poisson_solve(); }   // phase-by-phase, loops in conditional nodes
  void ens_join_mg() { join_mg(); }   // before the ensemble's own solve (persistent groups)
  void ens_reset_counts() {
    for (auto& c : cap_counts) c = 0;
    cap_solves = 0;
  }
  void ens_stage_tail(int s) {   // eval_duvw after the solve, sponge, eval_turb
    stage_post(s);
    if (S.sponge_on) sponge_damping();
    launch_turb(s);
  }
  int pull() { return pull_scalars(); }
  const DevScal& scal() const { return *h_sc; }
  int order() const { return it_order; }
  const Dev<T>& dev() const { return S; }
  const nhw_params& params() const { return p; }

  // ----------------------------------------------------------------- setup
  int setup(const double* depth, const double* eta0, const double* uvw0) override {
    drop_step_graphs();   // a new set-up changes captured kernel arguments
    HostInit h;
    int rc = host_setup(p, depth, eta0, uvw0, h);
    if (rc) return rc;
    it_order = h.it_order;
    for (int q = 0; q < 3; ++q) { S.alpha[q] = h.alpha[q]; S.beta[q] = h.beta[q]; }
    S.wm_segma = h.wm_segma; S.wm_celerity = h.wm_celerity; S.wm_wnumy = h.wm_wnumy;
    S.wm_atmp = h.wm_atmp; S.wm_xstart = h.wm_xstart;
    S.lef = ((p.wavemaker >= NHW_WM_LEF_LIN && p.wavemaker <= NHW_WM_LEF_TID) || p.wavemaker == NHW_WM_LEF_JON ||
             p.wavemaker == NHW_WM_LEF_TMA || p.wavemaker == NHW_WM_LEF_SPC) ? p.wavemaker : 0;
    // LEF_JON / LEF_TMA / INT_JON / INT_TMA (the 2-D spectra's tables come
    // from nhw_set_wave_spectrum)
    if (S.njon && !h.jon.empty())
      NHW_CU(cudaMemcpyAsync((void*)S.jon, h.jon.data(), sizeof(double) * h.jon.size(), cudaMemcpyHostToDevice, st));
    S.east = p.bc_xn == 3 ? p.wavemaker : 0;   // RIG_LIN or FLUX_LR (check_params)
    if (S.lef == NHW_WM_FOCUSED)
      NHW_CU(cudaMemcpyAsync((void*)S.foc, h.foc.data(), sizeof(double) * h.foc.size(), cudaMemcpyHostToDevice, st));
    S.lef_amp = p.amp_wave; S.lef_dep = p.dep_wave; S.lef_per = p.per_wave;
    S.lef_e2 = h.lef_e2; S.lef_u2 = h.lef_u2;
    S.con_mod = h.con_mod; S.con_len = h.con_len; S.con_ytr = h.con_ytr; S.con_ck = h.con_ck; S.con_x0 = h.con_x0;
    S.lef_segma = h.lef_segma; S.lef_wn = h.lef_wn; S.lef_shd = h.lef_shd; S.lef_stokes = h.lef_stokes;
    S.lef_sinth = h.lef_sinth; S.lef_costh = h.lef_costh;
    S.lef_cel = h.lef_cel; S.lef_atmp = h.lef_atmp; S.lef_xstart = h.lef_xstart; S.lef_c2 = h.lef_c2;
    S.wm_i0 = S.IB; S.wm_i1 = S.IB - 1;   // empty unless a source column exists
    for (int i = S.IB; i <= S.IE; ++i)
      if (h.xc[i] >= p.xsource_west && h.xc[i] <= p.xsource_east) {
        if (S.wm_i1 < S.wm_i0) S.wm_i0 = i;
        S.wm_i1 = i;
      }
    NHW_CU(cudaMemcpyAsync((void*)S.sig, h.sig.data(), sizeof(double) * h.sig.size(), cudaMemcpyHostToDevice, st));
    NHW_CU(cudaMemcpyAsync((void*)S.dsig, h.dsig.data(), sizeof(double) * h.dsig.size(), cudaMemcpyHostToDevice, st));
    NHW_CU(cudaMemcpyAsync((void*)S.sigc, h.sigc.data(), sizeof(double) * h.sigc.size(), cudaMemcpyHostToDevice, st));
    NHW_CU(cudaMemcpyAsync((void*)S.xc, h.xc.data(), sizeof(double) * h.xc.size(), cudaMemcpyHostToDevice, st));
    NHW_CU(cudaMemcpyAsync((void*)S.yc, h.yc.data(), sizeof(double) * h.yc.size(), cudaMemcpyHostToDevice, st));
    {  // per-level reciprocals of the Poisson assembly and the projection
      std::vector<double> lx(S.Kloc, 0.0), ly(S.Kloc, 0.0), lu(S.Kloc, 0.0), ld(S.Kloc, 0.0), lh(S.Kloc, 0.0),
          lds(S.Kloc, 0.0), lf(S.Kloc, 0.0);
      for (int k = 1; k < S.Kloc; ++k) {
        const double dk = h.dsig[k], dm = h.dsig[k - 1], s = dk + dm, hk = 0.5 * (dk + dm);
        lx[k] = 1.0 / (2. * p.dx * s);
        ly[k] = 1.0 / (2. * p.dy * s);
        lu[k] = 1.0 / (hk * dk);
        ld[k] = 1.0 / (hk * dm);
        lh[k] = 1.0 / hk;
        lds[k] = 1.0 / dk;
        lf[k] = dk / (dk + dm);
      }
      const std::vector<double>* src[] = {&lx, &ly, &lu, &ld, &lh, &lds, &lf};
      const double* dst[] = {S.lv_x, S.lv_y, S.lv_up, S.lv_dn, S.lv_h, S.lv_ds, S.lv_fint};
      for (int q = 0; q < 7; ++q)
        NHW_CU(cudaMemcpyAsync((void*)dst[q], src[q]->data(), sizeof(double) * S.Kloc, cudaMemcpyHostToDevice, st));
      std::vector<T> lt(3 * (size_t)S.Kloc, (T)0);
      for (int k = 0; k < S.Kloc; ++k) {
        lt[k] = (T)(1.0 / h.dsig[k]);
        if (k > 0) lt[S.Kloc + k] = (T)(h.sigc[k] - h.sigc[k - 1]);
        lt[2 * S.Kloc + k] = (T)(0.5 * h.dsig[k]);
      }
      NHW_CU(cudaMemcpyAsync((void*)S.lvT, lt.data(), sizeof(T) * lt.size(), cudaMemcpyHostToDevice, st));
      std::vector<double> lv(kLvN * (size_t)S.Kloc, 0.0);
      for (int k = 1; k < S.Kloc - 1; ++k) {
        const double d0 = h.dsig[k], du = h.dsig[k + 1], dd = h.dsig[k - 1];
        const double ck = (d0 + du) / 2.0, ck1 = (dd + d0) / 2.0;
        const double v[kLvN] = {du / (d0 + du), d0 / (d0 + du), d0 / (d0 + dd), dd / (d0 + dd), ck, ck1,
                                -ck / (ck + ck1) / ck1, (ck - ck1) / (ck * ck1), ck1 / (ck + ck1) / ck,
                                1.0 / (ck1 * (ck1 + ck)), 1.0 / (ck * (ck1 + ck)), 1.0 / (ck * ck1),
                                1.0 / (h.sigc[k + 1] - h.sigc[k - 1]), 1.0 / (0.5 * d0 * (d0 + dd)),
                                1.0 / (0.5 * d0 * (d0 + du))};
        for (int n = 0; n < kLvN; ++n) lv[n * (size_t)S.Kloc + k] = v[n];
      }
      if (S.lvv)
        NHW_CU(cudaMemcpyAsync((void*)S.lvv, lv.data(), sizeof(double) * lv.size(), cudaMemcpyHostToDevice, st));
      NHW_CU(cudaStreamSynchronize(st));
    }
    struct Up { int f; const void* src; } ups[] = {
        {NHW_F_HC, h.Hc.data()}, {NHW_F_HC0, h.Hc0.data()}, {NHW_F_DELXH, h.DelxH.data()},
        {NHW_F_DELYH, h.DelyH.data()}, {NHW_F_ETA, h.Eta.data()}, {NHW_F_ETA0, h.Eta.data()},
        {NHW_F_D, h.D.data()}, {NHW_F_SPONGE, h.Sponge.data()}, {NHW_F_HFX, h.Hfx.data()},
        {NHW_F_HFX0, h.Hfx.data()}, {NHW_F_HFY, h.Hfy.data()}, {NHW_F_HFY0, h.Hfy.data()},
        {NHW_F_MASK, h.Mask.data()}, {NHW_F_MASK_STRUCT, h.Mask_Struct.data()},
        {NHW_F_MASK9, h.Mask9.data()}, {NHW_F_U, h.U.data()}, {NHW_F_V, h.V.data()}, {NHW_F_W, h.W.data()}};
    for (auto& u : ups) {
      rc = set_field(u.f, u.src);
      if (rc) return rc;
    }
    {  // Wsx / Wsy are not public fields
      FieldDesc dx_{S.Wsx, 1, S.Mloc, S.Nloc, 1}, dy_{S.Wsy, 1, S.Mloc, S.Nloc, 1};
      for (auto pr : {std::make_pair(dx_, h.Wsx.data()), std::make_pair(dy_, h.Wsy.data())}) {
        const long long n = (long long)S.Mloc * S.Nloc;
        NHW_CU(cudaMemcpyAsync(d_stage, pr.second, n * 8, cudaMemcpyHostToDevice, st));
        k_unpack<T><<<cdiv(n, 256), 256, 0, st>>>(pr.first.ptr, 1, d_stage, nullptr, S.Mloc, S.Nloc, 1, S.sy, S.sz);
        NHW_CU(cudaStreamSynchronize(st));
      }
    }
    std::memset(h_sc, 0, sizeof(DevScal));
    h_sc->time = 0.0; h_sc->dt = p.dt_ini; h_sc->run_step = 0;
    h_sc->rho_dt = kRho0 / p.dt_ini; h_sc->dt_rho = p.dt_ini / kRho0;
    h_sc->dtmin_bits = (unsigned long long)dbits(kLarge);
    NHW_CU(cudaMemcpyAsync(S.sc, h_sc, sizeof(DevScal), cudaMemcpyHostToDevice, st));
    // initial: vel_bc on the initial velocities, with CmuVt = CmuHt = 0
    // (src/initialize.F:2667-2668), then DU = D*U*Mask and the seeding
    // eddy viscosities
    if (S.CmuVt) {
      NHW_CU(cudaMemsetAsync(S.CmuVt, 0, sizeof(T) * n3, st));
      NHW_CU(cudaMemsetAsync(S.CmuHt, 0, sizeof(T) * n3, st));
    }
    if (S.keDxU) {   // k-epsilon scratch of a previous set-up (the state is seeded below)
      T* ks[] = {S.keDxU, S.keDyU, S.keDxV, S.keDyV, S.keDxW, S.keDyW};
      for (T* a : ks) {
        NHW_CU(cudaMemsetAsync(a, 0, sizeof(T) * n3, st));
      }
    }
    incols(OpVelBcA{});
    box(OpVelBcLat{}, S.Mloc, S.Nloc, S.K, 0, 0, S.KB);
    incols(OpVelBcB{});
    L(OpInitDU::kName, [&] {
      k_allcells<T, OpInitDU><<<cdiv((long long)S.Mloc * S.Nloc * S.Kloc, 256), 256, 0, st>>>(S, OpInitDU{});
    });
    rc = sync();
    if (rc) return rc;
    {
      const int rg = upload_group();
      if (rg) return rg;
    }
    ready = true;
    return NHW_OK;
  }

  int get_scalars(nhw_scalars* o) override {
    int rc = pull_scalars();
    if (rc) return rc;
    std::memset(o, 0, sizeof(*o));
    o->time = h_sc->time; o->dt = h_sc->dt; o->dt_old = h_sc->dt_old; o->run_step = h_sc->run_step;
    o->last_krylov_iters = h_sc->inner_total; o->total_krylov_iters = h_sc->total_it;
    o->poisson_solves = h_sc->solves; o->last_rel_residual = h_sc->relres64;
    o->last_refinements = h_sc->ir_count; o->status = h_sc->status;
    return NHW_OK;
  }
  int set_time(double t, double dt, int rs) override {
    int rc = pull_scalars();
    if (rc) return rc;
    h_sc->time = t; h_sc->dt = dt; h_sc->run_step = rs;
    h_sc->rho_dt = kRho0 / dt; h_sc->dt_rho = dt / kRho0;
    NHW_CU(cudaMemcpyAsync(S.sc, h_sc, sizeof(DevScal), cudaMemcpyHostToDevice, st));
    return sync();
  }

  // -------------------------------------------------- reference subroutines
  int estimate_dt() override {
    dt_min();
    L("dt_finalize", [&] { k_dt_finalize<T><<<1, 1, 0, st>>>(S, 0); });
    int rc = pull_scalars();
    if (rc) return rc;
    if (h_sc->status == NHW_ERR_DT_MIN) return NHW_ERR_DT_MIN;
    return check();
  }
  int update_bathymetry() override {
    if (!S.slide) return NHW_OK;
    allcols(OpSlideA{});
    allcols(OpSlideB{});
    box(OpSlideC{}, S.Mloc + 1, S.Nloc + 1, 1, 0, 0, 0);
    return check();
  }
  // LEF_SPC: the spectrum's components in a device table of their own
  // (spc2d.txt's data is an input of the run, like the depth, not state)
  double* spc_table = nullptr;
  int set_wave_spectrum(int nf, int nd, const double* freq, const double* dire, const double* spc,
                        const double* phases) override {
    const bool internal = p.wavemaker == NHW_WM_INT_SPC || p.wavemaker == NHW_WM_INT_IRR;
    if (p.wavemaker != NHW_WM_LEF_SPC && !internal) {
      set_last_error("nhw_set_wave_spectrum: the handle runs none of LEF_SPC, INT_SPC, INT_IRR");
      return NHW_ERR_ARG;
    }
    std::vector<double> tab;
    const bool ok = internal ? internal_spectrum_components(p, nf, nd, freq, dire, spc, phases, tab)
                             : spectrum_components(p, nf, nd, freq, dire, spc, phases, tab);
    if (!ok) {
      set_last_error("nhw_set_wave_spectrum: needs 2 <= numfreq, 2 <= numdir, numfreq * numdir <= 12000, a "
                     "finite, non-negative spectrum, for INT_SPC / INT_IRR directions within 90 degrees of the "
                     "x axis, and for INT_IRR the phases");
      return NHW_ERR_ARG;
    }
    NHW_CU(cudaStreamSynchronize(st));
    if (spc_table) cudaFree(spc_table);
    spc_table = nullptr;
    NHW_CU(cudaMalloc((void**)&spc_table, sizeof(double) * tab.size()));
    NHW_CU(cudaMemcpy(spc_table, tab.data(), sizeof(double) * tab.size(), cudaMemcpyHostToDevice));
    S.jon = spc_table;
    S.njon = nf * nd;
    drop_step_graphs();   // captured kernels hold the table's address and size
    return NHW_OK;
  }
  // the reference's RanPhs given by the driver (LEF_JON / LEF_TMA / INT_JON / INT_TMA)
  int set_wave_phases(int n, const double* phases) override {
    const bool jon = p.wavemaker == NHW_WM_LEF_JON || p.wavemaker == NHW_WM_LEF_TMA ||
                     p.wavemaker == NHW_WM_INT_JON || p.wavemaker == NHW_WM_INT_TMA;
    if (!jon || !S.njon || n != S.njon || !phases) {
      set_last_error("nhw_set_wave_phases: the handle runs no JONSWAP / TMA wave of this many components");
      return NHW_ERR_ARG;
    }
    NHW_CU(cudaMemcpyAsync((void*)(S.jon + kJonPhase * S.njon), phases, sizeof(double) * n,
                           cudaMemcpyHostToDevice, st));
    NHW_CU(cudaStreamSynchronize(st));
    return NHW_OK;
  }
  int update_wave_bc() override {
    if (!S.lef && !S.east) return NHW_OK;
    if (S.lef == NHW_WM_LEF_SPC && !S.njon) {
      set_last_error("LEF_SPC: no spectrum yet (nhw_set_wave_spectrum)");
      return NHW_ERR_STATE;
    }
    if (S.lef) box(OpWaveBC{}, 1, S.Nloc, 1, 0, 0, 0);
    if (S.east == NHW_WM_RIG_LIN) box(OpWaveBCEast{}, 1, S.Nloc, 1, 0, 0, 0);
    if (S.east == NHW_WM_FLUX_LR) L("flux_lr", [&] { k_flux_lr<T><<<1, 256, 0, st>>>(S); });
    return check();
  }
  int update_mask() override {
    allcols(OpMaskA{});
    allcols(OpMaskB{});
    return check();
  }
  int update_vars() override {
    L("update_vars", [&] {
      k_update_vars<T><<<std::min<unsigned>(cdiv((long long)n3, 256), 4096), 256, 0, st>>>(S, (long long)n2,
                                                                                            (long long)n3);
    });
    return check();
  }
  int source_terms() override {
    if ((p.wavemaker == NHW_WM_INT_SPC || p.wavemaker == NHW_WM_INT_IRR) && !S.njon) {
      set_last_error("INT_SPC / INT_IRR: no spectrum yet (nhw_set_wave_spectrum)");
      return NHW_ERR_STATE;
    }
    if (S.wavemaker) L("source_area", [&] { k_single<T><<<1, 1, 0, st>>>(S, 0); });
    incols(OpSource{});
    return check();
  }
  // The FP64 form's face kernels share quotients and slopes between faces in
  // blocks; below about 2^16 cells the FP64 pipes are not full and a face a
  // thread has the shorter chain (256 x 8 x 10, all five: 156 against 169 us).
  // FP32+IR, which multiplies by reciprocals, keeps a face a thread across x
  // (1024 x 64 x 20: flux_x 49.5 us against 61.2, 768 x 768 x 20: 467 against
  // 509); across y, where a face a thread reads each row four times, blocks
  // pay from about 2^20 cells (flux_y + omega_y 515 x 30 x 15: 28.7 against
  // 33.3 us in blocks, 1024 x 64 x 20: 86.0 against 76.5, 768 x 768 x 20: 758
  // against 545).
  // Narrow grids leave most of a block without faces (flux + omega in us, a
  // face a thread against blocks; FP64, 82,000 cells: x, M = 12 235 against 501,
  // 24 235 / 265, 33 235 / 236, 36 234 / 221, 48 230 / 177; y, M = 16 188 / 207, 20 192 / 146,
  // 36 186 / 200, 40 186 / 179, N = 1 366 / 373, 2 290 / 267; FP32+IR across y,
  // 1,060,000 cells, by the share of threads with a face: 0.6 77 / 91, 0.75 76 /
  // 79, 0.93 78 / 74).
  bool face_blocks_x() const { return !kFP32 && S.neq >= 65536 && S.M >= 33; }
  bool face_blocks_y() const {
    constexpr int rows = kFaceYy - 2;   // of faces
    const double lanes = (double)S.M / ((double)kFaceYx * cdiv(S.M, kFaceYx));
    if (!kFP32) return S.neq >= 65536 && S.N >= 2 && lanes >= 0.6;
    return S.neq >= 1 << 20 && lanes * (S.N + 1) / ((double)rows * cdiv(S.N + 1, rows)) >= 0.8;
  }
  bool flux_z_walks() const { return !kFP32 && S.neq >= 65536; }
  // as few chunks of levels as leave about 8 blocks an SM
  template <class Face>
  void faces() {
    constexpr bool x = Face::kDir == 0;
    const int ntile = x ? (int)cdiv(S.M + 1, kFaceX - 2) : (int)cdiv(S.N + 1, kFaceYy - 2);
    const int nrow = x ? S.N : (int)cdiv(S.M, kFaceYx);
    const int chunks = (int)std::min<long long>(S.K, std::max<long long>(1, 152LL * 8 / ((long long)ntile * nrow)));
    const int kc = (S.K + chunks - 1) / chunks;
    const unsigned nb = (unsigned)ntile * nrow * cdiv(S.K, kc);
    L(Face::kName, [&] {
      k_faces<T, Face><<<nb, x ? dim3(kFaceX) : dim3(kFaceYx, kFaceYy), 0, st>>>(S, kc, ntile, nrow);
    });
  }
  void flux_z_walk() {
    const long long cols = (long long)S.M * S.N;
    const int chunks = (int)std::min<long long>(S.K + 1, std::max<long long>(1, 152LL * 512 / cols));
    const int kc = (S.K + 1 + chunks - 1) / chunks;
    L("flux_z", [&] { k_flux_z_walk<T><<<cdiv(cols * cdiv(S.K + 1, kc), 128), 128, 0, st>>>(S, kc); });
  }
  int fluxes() override {
    allcols(OpSlopeEta{});
    if (S.fxT) box(OpFacePrep{0}, S.M + 1, S.N + 1, 1, S.IB, S.JB, 0);
    if constexpr (kFP32) {
      box(OpFluxX{}, S.M + 1, S.N, S.K, S.IB, S.JB, S.KB);
    } else {
      if (face_blocks_x()) faces<FluxXFace<T>>();
      else box(OpFluxX{}, S.M + 1, S.N, S.K, S.IB, S.JB, S.KB);
    }
    if (face_blocks_y()) faces<FluxYFace<T>>();
    else box(OpFluxY{}, S.M, S.N + 1, S.K, S.IB, S.JB, S.KB);
    if (!flux_z_walks()) box(OpFluxZ{}, S.M, S.N, S.K + 1, S.IB, S.JB, S.KB);
    else if constexpr (!kFP32) flux_z_walk();
    if (S.keDxW) cells(OpKeSlopes{0});   // delxyzFun's DelxW / DelyW, read by the 3-D k-epsilon
    return check();
  }
  void get_uvw() {
    cells(OpGetUVW{});
    incols(OpVelBcA{});
    box(OpVelBcLat{}, S.Mloc, S.Nloc, S.K, 0, 0, S.KB);
    incols(OpVelBcB{});
  }
  // generate_coef_rhs (src/pressure.F:475-840), line factors, initial guess
  // and the multigrid coarse operators
  // The coarse multigrid operators (Galerkin products and line factors)
  // depend on level 0's operator alone: they are formed on a second stream,
  // forked after the assembly, while level 0's line factors, the initial
  // guess and the first FP64 residual run on the main one; join_mg() merges
  // the streams before the first V-cycle.  In a captured graph the fork and
  // join are edges of the graph.
  cudaStream_t mg_st = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  bool mg_forked = false;
  void join_mg() {
    if (!mg_forked) return;
    cudaStreamWaitEvent(st, ev_join, 0);
    mg_forked = false;
  }
  // as few chunks of levels as leave about 8 blocks an SM
  template <int PX, int PY>
  void poisson_coef() {
    const int nx = (int)cdiv(S.M, PX - 2), ny = (int)cdiv(S.N, PY - 2);
    const int chunks = (int)std::min<long long>(S.K, std::max<long long>(1, 152LL * 8 / ((long long)nx * ny)));
    const int kc = (S.K + chunks - 1) / chunks;
    const unsigned nb = (unsigned)nx * ny * cdiv(S.K, kc);
    L("poisson_coef", [&] { k_poisson_coef<T, PX, PY><<<nb, dim3(PX, PY), 0, st>>>(S, kc, nx, ny); });
  }
  // The block shape with the fewest threads for the grid's columns, and 30 x 8
  // columns, whose rows are the longest reads, unless another saves a quarter of
  // them; below 2048 columns, where the launch's latency decides, a third (us,
  // 30 x 8 against the shape taken, 20 levels: 1 x 4100 402 / 55, 4 x 1025 107 /
  // 33, 16 x 256 35 / 27, 40 x 1500 307 / 223, 4100 x 1 60 / 33; FP32+IR 32 x 1875
  // 395 / 223; 10 levels: 12 x 125 18.4 / 14.3, but 16 x 93 12.3 / 14.3 in 8 x 30)
  void poisson_blocks() {
    auto threads = [&](int px, int py) { return (long long)px * py * cdiv(S.M, px - 2) * cdiv(S.N, py - 2); };
    const double most = (long long)S.M * S.N < 2048 ? 0.65 : 0.75;
    const long long n = (long long)(threads(32, 10) * most), ny = threads(10, 32), nyy = threads(4, 80),
                    nxx = threads(80, 4);
    const long long best = std::min({n, ny, nyy, nxx});
    if (best == n) poisson_coef<32, 10>();
    else if (best == ny) poisson_coef<10, 32>();
    else if (best == nyy) poisson_coef<4, 80>();
    else poisson_coef<80, 4>();
  }
  void poisson_setup() {
    incols(OpColFactors{});
    poisson_blocks();
    if (use_mg && mg.size() > 1) {
      cudaEventRecord(ev_fork, st);
      cudaStreamWaitEvent(mg_st, ev_fork, 0);
      cudaStream_t main_st = st;
      st = mg_st;
      for (size_t l = 1; l < mg.size(); ++l) {
        MGL<T> f = mg[l - 1];
        MGL<T>& c = mg[l];
        const int bg = block_of(c.n), bf = block_of((long long)c.M * c.N);
        L("mg_galerkin", [&] {
          k_mg_galerkin<T><<<cdiv(c.n, bg), bg, 0, st>>>(f, (T*)c.coef, (T*)c.sp, c.M, c.N);
        });
        L("mg_factor", [&] {
          k_mg_factor<T><<<cdiv((long long)c.M * c.N, bf), bf, 0, st>>>(c, (T*)c.lcp, (T*)c.linv, (T*)c.sp);
        });
      }
      cudaEventRecord(ev_join, st);
      st = main_st;
      mg_forked = true;
    }
    incols(OpLineFactor{});
  }
  // P from the solution, ghosts mirrored (src/pressure.F:185-239)
  void poisson_finish() {
    cells(OpPFromX{});
    allcols(OpPGhost{});
  }
  int poisson_solve() {
    if (use_persistent) {
      join_mg();
      // count, generation and error word of the solve's grid barrier start at zero
      NHW_CU(cudaMemsetAsync(&S.sc->bar_count, 0, 3 * sizeof(unsigned int), st));
      const int gated = capturing ? 1 : 0;
      L("psolve", [&] {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)ps_nb);
        cfg.blockDim = dim3(32, kPsBY);
        cfg.dynamicSmemBytes = ps_smem;
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, k_psolve<T, kPsBY>, (const PsGroup<T>*)d_group, 1, gated);
        if (e != cudaSuccess && launch_err == cudaSuccess) launch_err = e;
      });
      if (launch_err != cudaSuccess) {
        set_last_error(std::string("persistent solve launch: ") + cudaGetErrorString(launch_err));
        launch_err = cudaSuccess;
        return NHW_ERR_CUDA;
      }
      if (capturing) return NHW_OK;
      int rc = pull_scalars();
      if (rc) return rc;
      rc = check();
      return rc ? rc : h_sc->pstat;
    }
    if (capturing) {
      ++cap_solves;
      // device-side loops: refinement sweeps around BiCGSTAB iterations
      S.h_ir = new_handle();      // before the kernels that set them are captured
      S.h_inner = new_handle();
      residual<true>();
      join_mg();
      cond_node(S.h_ir, cudaGraphCondTypeWhile, [&] {
        inner_init();
        cond_node(S.h_inner, cudaGraphCondTypeWhile, [&] { one_iteration(); }, 2);
        inner_finish();
        residual<false>();
      }, 1);
      return NHW_OK;
    }
    // host-driven loops over the same device-side decisions
    residual<true>();
    join_mg();
    int rc = pull_scalars();
    if (rc) return rc;
    while (h_sc->ir_go) {
      inner_init();
      int chunk = 4;
      while (true) {
        rc = run_iterations(chunk);
        if (rc) return rc;
        rc = pull_scalars();
        if (rc) return rc;
        if (h_sc->conv != 0) break;
        if (chunk < 16) chunk *= 2;
      }
      inner_finish();
      residual<false>();
      rc = pull_scalars();
      if (rc) return rc;
    }
    rc = check();
    return rc ? rc : h_sc->pstat;
  }
  // the reducing Krylov kernels in slices (krylov.cuh) while their blocks are
  // fewer than the SMs
  bool sliced() const { return red_blocks() <= (unsigned)kSlicedBlocks; }
  bool paired() const { return red_blocks() <= (unsigned)kPairedBlocks; }
  template <bool kFirst>
  void residual() {
    L("res64", [&] {
      if (sliced()) k_res64_sl<T, kFirst><<<red_blocks() * kSlices, 256, 0, st>>>(S);
      else if (paired()) k_res64_pr<T, kFirst><<<red_blocks() * 2, 256, 0, st>>>(S);
      else k_res64<T, kFirst><<<red_blocks(), 256, 0, st>>>(S);
    });
  }
  // start and end of one inner solve (one refinement sweep)
  void inner_init() {
    if (use_gmres) L("gm_init", [&] { k_gm_init<T><<<red_blocks(), 256, 0, st>>>(S); });
    else L("bicg_init", [&] {
      if (sliced()) k_bicg_init_sl<T><<<red_blocks() * kSlices, 256, 0, st>>>(S);
      else k_bicg_init<T><<<red_blocks(), 256, 0, st>>>(S);
    });
  }
  void inner_finish() {
    if (use_gmres) L("x_update", [&] { k_gm_xupd<T><<<cdiv(S.neq, 256), 256, 0, st>>>(S); });
    else L("x_update", [&] { k_xupd<T><<<cdiv(S.neq, 256), 256, 0, st>>>(S); });
  }
  // `chunk` Krylov iterations; replayed from a captured CUDA graph unless the
  // per-kernel profiler is on (its events would become graph nodes)
  struct ChunkGraph { int chunk; cudaGraphExec_t exec; long long kernels; };
  std::vector<ChunkGraph> graphs;
  bool use_graphs = true;
  int run_iterations(int chunk) {
    if (!use_graphs || prof_on) {
      for (int c = 0; c < chunk; ++c) one_iteration();
      return check();
    }
    for (auto& g : graphs)
      if (g.chunk == chunk) {
        NHW_CU(cudaGraphLaunch(g.exec, st));
        launches += g.kernels;
        return NHW_OK;
      }
    cudaGraph_t graph;
    const long long l0 = launches;
    NHW_CU(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    for (int c = 0; c < chunk; ++c) one_iteration();
    NHW_CU(cudaStreamEndCapture(st, &graph));
    cudaGraphExec_t exec;
    NHW_CU(cudaGraphInstantiate(&exec, graph, 0));
    cudaGraphDestroy(graph);
    graphs.push_back({chunk, exec, launches - l0});
    launches = l0;
    NHW_CU(cudaGraphLaunch(exec, st));
    launches += graphs.back().kernels;
    return NHW_OK;
  }
  void one_iteration() {
    if (use_gmres) {   // z_j = M^-1 v_j (v_j formed by the first sweeps), then Arnoldi
      vcycle(S.kp, S.kph, kFineV);
      L("gm_arnoldi", [&] { k_gm_arnoldi<T><<<red_blocks(), 256, 0, st>>>(S); });
      L("gm_orth", [&] { k_gm_orth<T><<<red_blocks(), 256, 0, st>>>(S); });
      return;
    }
    const unsigned cb = cdiv((long long)S.M * S.N, 128);
    if (use_mg) {
      vcycle(S.kp, S.kph, kFineP);   // p is formed by the fine level's first sweeps
    } else {
      L("bicg_p", [&] { k_bicg_p<T><<<cb, 128, 0, st>>>(S); });
    }
    L("bicg_v", [&] {
      if (sliced()) {
        k_bicg_v_sl<T><<<matvec_blocks() * kSlices, 256, 0, st>>>(S);
        return;
      }
      if constexpr (!kColumnWalk<T>)
        if (paired()) {
          k_bicg_v_pr<T><<<red_blocks() * 2, 256, 0, st>>>(S);
          return;
        }
      k_bicg_v<T><<<matvec_blocks(), 256, 0, st>>>(S);
    });
    if (use_mg) {
      vcycle(S.ks, S.ksh, kFineS);   // s likewise
    } else {
      L("bicg_s", [&] { k_bicg_s<T><<<cb, 128, 0, st>>>(S); });
    }
    L("bicg_t", [&] {
      if (sliced()) {
        k_bicg_t_sl<T><<<matvec_blocks() * kSlices, 256, 0, st>>>(S);
        return;
      }
      if constexpr (!kColumnWalk<T>)
        if (paired()) {
          k_bicg_t_pr<T><<<red_blocks() * 2, 256, 0, st>>>(S);
          return;
        }
      k_bicg_t<T><<<matvec_blocks(), 256, 0, st>>>(S);
    });
    L("bicg_xr", [&] {
      if (sliced()) k_bicg_xr_sl<T><<<red_blocks() * kSlices, 256, 0, st>>>(S);
      else if (red_blocks() <= 2u * kSlicedBlocks) k_bicg_xr_pr<T><<<red_blocks() * 2, 256, 0, st>>>(S);
      else k_bicg_xr<T><<<red_blocks(), 256, 0, st>>>(S);
    });
  }
  // multigrid V-cycle: x ~= A^-1 b on level 0
  int cta_columns = 64;    // levels up to this many columns run in one block (mg_cta_columns)
  // the first level of the block cycle: at most its kCtaLevels last levels, and
  // always the coarsest, which has no level below it to restrict to, even where
  // it has more than cta_columns columns
  int first_block_level() const {
    const int nl = (int)mg.size();
    int lc = 0;
    while (lc < nl && (long long)mg[lc].M * mg[lc].N > cta_columns) ++lc;
    return std::min(std::max(lc, nl - kCtaLevels), nl - 1);
  }
  template <class In>
  void smooth(const MGL<T>& Lv, int color, int zero_x, int level, const Prolong<T>& P, In in) {
    static const char* names[] = {"mg_smooth_l0", "mg_smooth_l1", "mg_smooth_l2", "mg_smooth_l3",
                                  "mg_smooth_l4", "mg_smooth_l5", "mg_smooth_l6", "mg_smooth_l7+"};
    const int pair = (Lv.M + 1 - color) / 2 + (Lv.M + color) / 2;
    const long long nthr = (long long)pair * ((Lv.N + 1) / 2);
    const int by = std::min(Lv.K, 32);
    const size_t shm = sizeof(T) * 4 * 32 * Lv.K;
    L(names[level < 7 ? level : 7], [&] {
      if (Lv.sp) {   // colour-split operator
        const long long nq = (long long)((Lv.M + 1) / 2) * Lv.N;
        if constexpr (kFP32) {
          // one thread per column and chunk of kSplitLevels levels: short
          // blocks, 7 resident per SM, so that a half-sweep of C2 runs in
          // one wave (with 20 threads per column it took 2.25 waves)
          const int by = std::min((Lv.K + kSplitLevels - 1) / kSplitLevels, kSplitMaxThreads / 32);
          if (P.xc)
            k_mg_smooth_split<T, true, In><<<cdiv(nq, 32), dim3(32, by), shm, st>>>(Lv, S.sc, color, zero_x, P, in);
          else
            k_mg_smooth_split<T, false, In><<<cdiv(nq, 32), dim3(32, by), shm, st>>>(Lv, S.sc, color, zero_x, P, in);
        } else {
          // at most 8 threads per column, each loading ceil(K/8) levels
          const int lpt = (Lv.K + 7) / 8, by = std::min((Lv.K + lpt - 1) / lpt, 32);
          if (P.xc)
            k_mg_smooth_split_strided<T, true, In><<<cdiv(nq, 32), dim3(32, by), shm, st>>>(Lv, S.sc, color, zero_x,
                                                                                         P, in);
          else
            k_mg_smooth_split_strided<T, false, In><<<cdiv(nq, 32), dim3(32, by), shm, st>>>(Lv, S.sc, color, zero_x,
                                                                                          P, in);
        }
      } else if (P.xc)
        k_mg_smooth_blk<T, true, In><<<cdiv(nthr, 32), dim3(32, by), shm, st>>>(Lv, S.sc, color, zero_x, P, in);
      else
        k_mg_smooth_blk<T, false, In><<<cdiv(nthr, 32), dim3(32, by), shm, st>>>(Lv, S.sc, color, zero_x, P, in);
    });
  }
  // Levels whose half of the V-cycle runs as one launch of small tiles
  // (mg_tile.cuh).  Up to 4096 columns a tile launch takes less time than the
  // passes one by one, although it solves the tiles' borders more than once
  // (GB300, one level of 20 sigma levels, down / up in us): FP32 64 x 8
  // 9.3 / 8.3 -> 5.1 / 4.8, 128 x 32 10.5 / 8.8 -> 7.1 / 7.3, but 256 x 32
  // 10.3 / 8.8 -> 12.4 / 13.2; FP64 64 x 8 15.6 / 34 -> 12.6 / 15.0, 128 x 32
  // 16.3 / 34 -> 19.6 / 24.3.  Narrow levels leave most of a tile's rows
  // empty, so the tiles are limited too: to those of 4096 columns and a
  // quarter more in FP64, and to twice as many in FP32, whose idle lanes cost
  // less (ms/step without tiles / with up to 256 / 512 / 1024 of them, 20
  // sigma levels: FP64 4096 x 1 17.3 / 17.8 / 22.3 / 28.5, 2048 x 1 14.4 / 14.9
  // / 19.6, 819 x 5, 410 tiles, 31.9 / 24.6 / 25.7, 63 x 65, 272 tiles, 16.0 /
  // 12.7 / 12.4; FP32 4096 x 1 5.2 / 4.5 / 4.6 / 4.9, 819 x 5 8.0 / 5.3 / 4.6).
  // Aggregates must fill whole tiles.
  static constexpr int kTiles = kFP32 ? 512 : 320;
  static bool tiled(const MGL<T>& Lv) {
    auto pow2 = [](int r) { return r == 1 || r == 2 || r == 4; };
    return (long long)Lv.M * Lv.N <= 4096 && tiles_of(Lv) <= kTiles && pow2(Lv.rx) && pow2(Lv.ry);
  }
  // whether level l's half of the V-cycle runs so: GMRES forms its basis vector
  // in the separate passes of level 0
  bool tiles_at(int l) const { return l < first_block_level() && tiled(mg[l]) && (l > 0 || !use_gmres); }
  static unsigned tiles_of(const MGL<T>& Lv) { return cdiv(Lv.M, TileS::TX) * cdiv(Lv.N, TileS::TY); }
  // Levels a thread: two where one each would not fit a block, or where the
  // blocks (2 threads a cell) are more than the 152 SMs hold at 64 registers
  // a thread (FP32 128 x 32 x 20: 9.5 / 9.1 -> 7.1 / 7.3 us; 64 x 64 x 10
  // 4.8 / 4.6 with one, 5.0 / 5.4 with two)
  static int tile_lpt(const MGL<T>& Lv) { return Lv.K > 32 || 2LL * Lv.n > 152 * 1024 ? 2 : 1; }
  template <bool kFine, class In>
  void down(int l, In in) {
    static const char* names[] = {"mg_down_l0", "mg_down_l1", "mg_down_l2", "mg_down_l3",
                                  "mg_down_l4", "mg_down_l5", "mg_down_l6", "mg_down_l7+"};
    const MGL<T> f = mg[l], c = mg[l + 1];
    const int nx = (int)cdiv(f.M, TileS::TX);
    const unsigned nb = tiles_of(f);
    L(names[l < 7 ? l : 7], [&] {
      if (tile_lpt(f) == 1)
        k_mg_down<T, kFine, TileS, 1, In><<<nb, dim3(32, f.K), tile_smem<TileS, T>(f.K), st>>>(f, c, nx, S.sc, in);
      else
        k_mg_down<T, kFine, TileS, 2, In>
            <<<nb, dim3(32, (f.K + 1) / 2), tile_smem<TileS, T>(f.K), st>>>(f, c, nx, S.sc, in);
    });
  }
  template <bool kFine>
  void up(int l, const Prolong<T>& pr) {
    static const char* names[] = {"mg_up_l0", "mg_up_l1", "mg_up_l2", "mg_up_l3",
                                  "mg_up_l4", "mg_up_l5", "mg_up_l6", "mg_up_l7+"};
    const MGL<T> f = mg[l];
    const int nx = (int)cdiv(f.M, TileS::TX);
    const unsigned nb = tiles_of(f);
    L(names[l < 7 ? l : 7], [&] {
      if (tile_lpt(f) == 1)
        k_mg_up<T, kFine, TileS, 1><<<nb, dim3(32, f.K), tile_smem<TileS, T>(f.K), st>>>(f, pr, nx, S.sc);
      else
        k_mg_up<T, kFine, TileS, 2>
            <<<nb, dim3(32, (f.K + 1) / 2), tile_smem<TileS, T>(f.K), st>>>(f, pr, nx, S.sc);
    });
  }
  // the levels from `lc` on in one block
  template <int LPT>
  void cycle(const MGSet<T>& set, int cnt) {
    L("mg_coarse_cycle", [&] {
      k_mg_cycle<T, LPT><<<1, kCycleSlots * ((S.K + LPT - 1) / LPT), cycle_smem<T>(S.K), st>>>(set, cnt, S.sc, mg_w,
                                                                                           mg_coarse_sweeps);
    });
  }
  // b is formed on the fly by level 0's first passes: BiCGSTAB's p or s, or
  // GMRES' basis vector
  enum FineIn { kFineP, kFineS, kFineV };
  void vcycle(T* b, T* x, FineIn fine_in) {
    mg[0].b = b;
    mg[0].x = x;
    const int nl = (int)mg.size(), lc = first_block_level();
    const Prolong<T> none{nullptr, (T)0, 1, 1, 1, 1, 1, 1};
    auto in_v = [&] { return MgInV<T>{S.kt, S.kp, S.gmV, S.gmT + kGmTInv, (size_t)S.neq}; };
    if (lc == 0) {   // the whole hierarchy in one block: form b first
      const unsigned nb = cdiv(S.neq, 256);
      if (fine_in == kFineP) L("bicg_p", [&] { k_bicg_p_cell<T><<<nb, 256, 0, st>>>(S); });
      else if (fine_in == kFineS) L("bicg_s", [&] { k_bicg_s_cell<T><<<nb, 256, 0, st>>>(S); });
      else L("gm_v", [&] { k_gm_v_cell<T><<<nb, 256, 0, st>>>(S, in_v()); });
    }
    static const char* rnames[] = {"mg_restrict_l0", "mg_restrict_l1", "mg_restrict_l2", "mg_restrict_l3",
                                   "mg_restrict_l4", "mg_restrict_l5", "mg_restrict_l6", "mg_restrict_l7+"};
    for (int l = 0; l < lc; ++l) {
      if (tiles_at(l)) {
        if (l > 0) down<false>(l, TileB<T>{mg[l].b});
        else if (fine_in == kFineP) down<true>(0, TileInP<T>{S.kp, S.kr, S.kq});
        else down<true>(0, TileInS<T>{S.ks, S.kr, S.kv});
        continue;
      }
      for (int color = 0; color < 2; ++color) {
        const int zx = color == 0 ? 1 : 0;
        if (l > 0) smooth(mg[l], color, zx, l, none, MgB<T>{mg[l].b});
        else if (fine_in == kFineP) smooth(mg[0], color, zx, 0, none, MgInP<T>{S.kp, S.kr, S.kv});
        else if (fine_in == kFineS) smooth(mg[0], color, zx, 0, none, MgInS<T>{S.ks, S.kr, S.kv});
        else smooth(mg[0], color, zx, 0, none, in_v());
      }
      MGL<T> f = mg[l], c = mg[l + 1];
      L(rnames[l < 7 ? l : 7], [&] { k_mg_restrict_c0<T><<<cdiv(c.n, 256), 256, 0, st>>>(f, c, S.sc); });
    }
    {
      MGSet<T> set{};
      int slots = 0;
      for (int l = lc; l < nl; ++l) {
        set.L[l - lc] = mg[l];
        slots = std::max(slots, cycle_slots(mg[l]));
      }
      const int cnt = nl - lc;
      // Levels of up to 32 slots a colour and 40 sigma levels take the form
      // that keeps x and the operator on chip (32 x 2 and 8 x 2 columns, 20
      // levels: FP32 21.9 -> 15.2 us, FP64 74.7 -> 50.2; 40 levels FP32 36.6
      // -> 25.6, FP64 140 -> 103); with more slots the FP64 form spills and
      // is slower (5 x 12 columns: 76.8 against 82.7 us)
      if (slots <= kCycleSlots && S.K <= 20) cycle<1>(set, cnt);
      else if (slots <= kCycleSlots && S.K <= 40) cycle<2>(set, cnt);
      else
        L("mg_coarse_cycle", [&] {
          k_mg_cta_cycle<T><<<1, 1024, sizeof(T) * 4 * 32 * S.K, st>>>(set, cnt, S.sc, mg_w, mg_coarse_sweeps);
        });
    }
    static const char* pnames[] = {"mg_prolong_l0", "mg_prolong_l1", "mg_prolong_l2", "mg_prolong_l3",
                                   "mg_prolong_l4", "mg_prolong_l5", "mg_prolong_l6", "mg_prolong_l7+"};
    for (int l = lc - 1; l >= 0; --l) {
      const MGL<T>& f = mg[l];
      const MGL<T>& c = mg[l + 1];
      const Prolong<T> pr = prolong_from(f, c, mg_w);
      if (tiles_at(l)) {
        if (l > 0) up<false>(l, pr);
        else up<true>(0, pr);
        continue;
      }
      // levels of 8192 columns or more: the correction in its own pass (C2:
      // 15.3 -> 14.7 ms/step FP32+IR, 63.9 -> 56.9 FP64); on smaller levels
      // one launch more costs more than the interpolations it saves
      if ((long long)f.M * f.N >= 8192) {
        const long long nt = (long long)((f.M + 1) / 2) * f.N * f.K;
        L(pnames[l < 7 ? l : 7], [&] { k_mg_prolong0<T><<<cdiv(nt, 256), 256, 0, st>>>(f, pr, S.sc); });
        smooth(f, 1, 0, l, none, MgB<T>{f.b});
      } else {
        smooth(f, 1, 0, l, pr, MgB<T>{f.b});
      }
      smooth(f, 0, 0, l, none, MgB<T>{f.b});
    }
  }

  // eval_duvw up to the pressure solve: explicit stage update, surface BC,
  // slopes, velocities and the Poisson system
  void stage_pre(int s) {
    if (S.viscous) {
      box(OpViscSlopes{}, S.M + 2, S.N + 2, S.K + 2, S.IB - 1, S.JB - 1, S.KB - 1);
      cells(OpDiffusion{});
    }
    incols(OpExplicit{s});
    allcols(OpWlBcEta{});
    allcols(OpSlopeEta{true});
    if (S.viscous)
      L("vertical_viscous", [&] {
        k_vert_visc<T><<<cdiv((long long)S.M * S.N, 32), dim3(32, kVvThreadsY), vv_smem(S.K), st>>>(S);
      });
    if (S.non_hydro) {
      get_uvw();
      poisson_setup();
    }
  }
  // eval_duvw after the pressure solve: projection, SSP-RK combination,
  // velocities and Omega
  void stage_post(int s) {
    if (S.non_hydro) {
      poisson_finish();
      if (kFP32) {
        const long long cols = (long long)S.M * S.N;
        const int chunks = (int)std::min<long long>(S.K, std::max<long long>(1, 152LL * 1024 / cols));
        const int kc = (S.K + chunks - 1) / chunks;
        L("projection", [&] { k_projection32<T><<<cdiv(cols * cdiv(S.K, kc), 128), 128, 0, st>>>(S, kc); });
      }
      else cells(OpProjection{});
    }
    cells(OpSSP{s});
    get_uvw();
    if (S.fxT) box(OpFacePrep{1}, S.M + 1, S.N + 1, 1, S.IB, S.JB, 0);
    if constexpr (kFP32) {
      box(OpOmegaX{}, S.M + 1, S.N, S.K, S.IB, S.JB, S.KB);
    } else {
      if (face_blocks_x()) faces<OmegaXFace<T>>();
      else box(OpOmegaX{}, S.M + 1, S.N, S.K, S.IB, S.JB, S.KB);
    }
    if (face_blocks_y()) faces<OmegaYFace<T>>();
    else box(OpOmegaY{}, S.M, S.N + 1, S.K, S.IB, S.JB, S.KB);
    incols(OpOmegaScan{});
    if (S.keDxU) cells(OpKeSlopes{1});   // get_Omega's DelxU .. DelyV, before sponge_damping
  }
  int eval_duvw(int istep) override {
    if (istep < 1 || istep > it_order) return NHW_ERR_ARG;
    const int s = istep - 1;
    stage_pre(s);
    int status = NHW_OK;
    if (S.non_hydro) {
      status = poisson_solve();
      if (status == NHW_ERR_CUDA) return status;
    }
    stage_post(s);
    int rc = check();
    return rc ? rc : status;
  }
  int sponge_damping() override {
    allcols(OpSponge{});
    return check();
  }
  // eval_turb (src/nhwave.F:6544-6782) of stage s (0-based): the eddy
  // viscosities CmuVt / CmuHt the next stage's viscous terms read, from the
  // velocities after sponge_damping; with IVTURB = 10 the k-epsilon step
  // first.  Inviscid flow has none.
  void launch_turb(int s) {
    if (!S.viscous) return;
    if (S.ivturb == 10) {
      allcols(OpKeTop{});
      L("kepsilon_column", [&] {
        // blocks of 32 columns, of 16 or 8 while those are fewer than two an
        // SM (FP32+IR, 32 / 16 / 8 columns: 96 x 6 x 20 210 / 151 / 99 us,
        // 200 x 12 x 10 140 / 91 / 90, 515 x 30 x 15 480 / 493 / 518)
        const long long cols = (long long)S.M * S.N;
        int cb = 32;
        while (cb > 8 && cols < 152LL * 2 * cb) cb /= 2;
        const int by = std::min(S.K, kKeThreads / cb);
        k_ke_column<T><<<cdiv((long long)S.M * S.N, cb), dim3(cb, by), ke_smem(cb, S.K), st>>>(S, s);
      });
      box(OpKeSidesX{}, S.N * S.Kloc, 1, 1, 0, 0, 0);
      box(OpKeSidesY{}, S.Mloc * S.Kloc, 1, 1, 0, 0, 0);
      allcols(OpKeFinal{});
    }
    if (S.ivturb == 3) {
      incols(OpKe2Column{s});
      box(OpKe2Sides{0}, S.N * S.K, 1, 1, 0, 0, 0);
      box(OpKe2Sides{1}, S.M * S.K, 1, 1, 0, 0, 0);
      allcols(OpKe2Final{});
    }
    if (S.ivturb == 30) {   // les_dyn (src/nhwave.F:7989-8410)
      auto every = [&](auto op) {
        L(decltype(op)::kName, [&] {
          k_allcells<T, decltype(op)><<<cdiv((long long)S.Mloc * S.Nloc * S.Kloc, 256), 256, 0, st>>>(S, op);
        });
      };
      auto mirror = [&](int f0, int f1, int north_all) {
        box(OpLdMirror{0, f0, f1, north_all}, S.M * S.N, 1, 1, 0, 0, 0);
        box(OpLdMirror{1, f0, f1, north_all}, S.N * S.K, 1, 1, 0, 0, 0);
        box(OpLdMirror{2, f0, f1, north_all}, S.M * S.K, 1, 1, 0, 0, 0);
      };
      every(OpLdStrain{});
      mirror(0, 6, 0);   // Sij: the reference's north loop writes the sixth component only
      every(OpLdSab{});
      every(OpLdFilter{});
      mirror(7, 29, 1);
      every(OpLdCoef{});
      every(OpLdSmooth{});
      mirror(30, 31, 1);
      every(OpLdVisc{});
      box(OpLdMirror{0, -1, 0, 1}, S.M * S.N, 1, 1, 0, 0, 0);   // CmuVt: bed and surface, then the sides
      box(OpLesSides{0}, S.N * S.K, 1, 1, 0, 0, 0);
      box(OpLesSides{1}, S.M * S.K, 1, 1, 0, 0, 0);
    }
    if (S.ivturb == 20) {
      cells(OpLesCell{});
      incols(OpLesColumn{});
      box(OpLesSides{0}, S.N * S.K, 1, 1, 0, 0, 0);
      box(OpLesSides{1}, S.M * S.K, 1, 1, 0, 0, 0);
    }
    allcols(OpTurbV{});
    if (S.ihturb == 2) {
      cells(OpTurbH{});
      box(OpTurbHGhost{}, S.N * S.K + S.M * S.K + S.M * S.N, 1, 1, 0, 0, 0);
    }
  }
  int eval_turb(int istep) override {
    if (istep < 1 || istep > it_order) return NHW_ERR_ARG;
    launch_turb(istep - 1);
    return check();
  }
  // everything of one time step after estimate_dt (src/nhwave.F:119-200)
  int step_body() {
    if (S.slide) update_bathymetry();
    update_wave_bc();
    update_mask();
    int rc = update_vars();
    if (rc) return rc;
    int worst = NHW_OK;
    for (int s = 1; s <= it_order; ++s) {
      source_terms();
      fluxes();
      rc = eval_duvw(s);
      if (rc == NHW_ERR_CUDA) return rc;
      if (rc != NHW_OK && worst == NHW_OK) worst = rc;
      if (S.sponge_on) sponge_damping();
      launch_turb(s - 1);
    }
    rc = check();
    return rc ? rc : worst;
  }
  int step_eager() {
    int rc = estimate_dt();
    if (rc) return rc;
    return step_body();
  }

  // ------------------------------------------------ whole-step CUDA graphs
  // A time step is captured once into a graph whose loops run on the device:
  // an IF node holds the step behind k_dt_finalize's decision, and in each
  // pressure solve a WHILE node holds the refinement sweeps and a nested
  // WHILE node the BiCGSTAB iterations; the kernels that end a reduction set
  // the node conditions.  Stepping then needs no host round trip.
  // sgraph[0] is the plain step, sgraph[1] the gated step used by run().
  struct StepGraph {
    cudaGraphExec_t exec = nullptr;
    long long per_launch = 0, per_step = 0, per_sweep = 0, per_iter = 0;  // kernel launches
  };
  StepGraph sgraph[2];
  bool capturing = false;
  std::string cap_err;
  cudaGraph_t cap_root = nullptr;
  cudaStream_t cap_st[4] = {nullptr, nullptr, nullptr, nullptr};
  int cap_depth = 0, cap_level = 3, cap_solves = 0;
  long long cap_counts[4] = {0, 0, 0, 0};   // step body, sweep body, iteration body, outside
  int64_t acc_step = 0, acc_ir = 0, acc_it = 0;   // counters at the last launch accounting

  bool cap_ok(cudaError_t e, const char* what) {
    if (e != cudaSuccess && cap_err.empty()) cap_err = std::string(what) + ": " + cudaGetErrorString(e);
    return e == cudaSuccess;
  }
  unsigned long long new_handle() {
    cudaGraphConditionalHandle h = 0;
    cap_ok(cudaGraphConditionalHandleCreate(&h, cap_root, 0, cudaGraphCondAssignDefault), "conditional handle");
    return h;
  }
  // Appends a conditional node to the capture on `st` and captures `body`
  // into its body graph on a stream of its own; `level` says which launch
  // counter the body's kernels go to.
  template <class F>
  void cond_node(unsigned long long h, cudaGraphConditionalNodeType type, F body, int level) {
    if (!cap_err.empty() || cap_depth >= 4) { cap_ok(cudaErrorNotSupported, "conditional nesting"); return; }
    cudaStreamCaptureStatus cs;
    unsigned long long id = 0;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    const cudaGraphEdgeData* ed = nullptr;
    size_t nd = 0;
    if (!cap_ok(cudaStreamGetCaptureInfo(st, &cs, &id, &g, &deps, &ed, &nd), "capture info")) return;
    cudaGraphNodeParams cp{};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = type;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    if (!cap_ok(cudaGraphAddNode(&node, g, deps, ed, nd, &cp), "conditional node")) return;
    if (!cap_ok(cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1, cudaStreamSetCaptureDependencies),
                "capture dependencies"))
      return;
    cudaStream_t outer = st;
    const int outer_level = cap_level;
    st = cap_st[cap_depth++];
    cap_level = level;
    if (cap_ok(cudaStreamBeginCaptureToGraph(st, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                             cudaStreamCaptureModeRelaxed), "body capture")) {
      body();
      cudaGraph_t gb = nullptr;
      cap_ok(cudaStreamEndCapture(st, &gb), "body capture end");
    }
    st = outer;
    --cap_depth;
    cap_level = outer_level;
  }
  int capture_step(int gated) {
    StepGraph& G = sgraph[gated];
    if (G.exec) return NHW_OK;
    if (!cap_st[0])
      for (auto& c : cap_st) NHW_CU(cudaStreamCreateWithFlags(&c, cudaStreamNonBlocking));
    cudaGraph_t g = nullptr;
    NHW_CU(cudaGraphCreate(&g, 0));
    cap_err.clear();
    cap_root = g;
    for (auto& c : cap_counts) c = 0;
    cap_level = 3;
    cap_solves = 0;
    const Dev<T> saved = S;
    const long long l0 = launches;
    capturing = true;
    S.graph_mode = 1;
    S.h_go = use_persistent ? 0 : new_handle();
    if (cap_ok(cudaStreamBeginCaptureToGraph(st, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal),
               "step capture")) {
      dt_min();
      L("dt_finalize", [&] { k_dt_finalize<T><<<1, 1, 0, st>>>(S, gated); });
      if (use_persistent)
        step_body();   // every kernel checks sc->step_go; no loops left on the host side
      else
        cond_node(S.h_go, cudaGraphCondTypeIf, [&] { step_body(); }, 0);
      cudaGraph_t gg = nullptr;
      cap_ok(cudaStreamEndCapture(st, &gg), "step capture end");
    }
    capturing = false;
    S = saved;
    launches = l0;
    cudaGetLastError();
    if (cap_err.empty()) {
      cudaGraphExec_t ex = nullptr;
      if (cap_ok(cudaGraphInstantiate(&ex, g, 0), "step graph instantiate")) G.exec = ex;
    }
    cudaGraphDestroy(g);
    if (!cap_err.empty()) {
      set_last_error(cap_err);
      return NHW_ERR_CUDA;
    }
    const long long ns = std::max(cap_solves, 1);
    G.per_launch = cap_counts[3];
    G.per_step = cap_counts[0];
    G.per_sweep = cap_counts[1] / ns;
    G.per_iter = cap_counts[2] / ns;
    return NHW_OK;
  }
  void drop_step_graphs() {
    for (auto& G : sgraph) {
      if (G.exec) cudaGraphExecDestroy(G.exec);
      G = StepGraph{};
    }
  }
  // kernel launches of `n` graph launches, from the device counters
  void account(const StepGraph& G, int n) {
    launches += G.per_launch * n + G.per_step * (h_sc->run_step - acc_step) +
                G.per_sweep * (h_sc->total_ir - acc_ir) + G.per_iter * (h_sc->total_it - acc_it);
    snapshot();
  }
  void snapshot() {
    acc_step = h_sc->run_step;
    acc_ir = h_sc->total_ir;
    acc_it = h_sc->total_it;
  }
  bool graph_path() const { return use_graphs && !prof_on; }

  int step() override {
    if (!ready) return NHW_ERR_STATE;
    if (!graph_path()) return step_eager();
    int rc = capture_step(0);
    if (rc) return rc;
    rc = pull_scalars();
    if (rc) return rc;
    snapshot();
    NHW_CU(cudaGraphLaunch(sgraph[0].exec, st));
    rc = pull_scalars();
    if (rc) return rc;
    account(sgraph[0], 1);
    rc = check();
    if (rc) return rc;
    if (h_sc->status == NHW_ERR_DT_MIN) return NHW_ERR_DT_MIN;
    return h_sc->step_status;
  }
  // nhw_run: steps while TIME < TOTAL_TIME and RUN_STEP < SIM_STEPS, at most
  // nsteps; stops at DT_MIN or a non-finite pressure solve.  Graph launches
  // go out in batches with one host round trip per batch.
  int run(int nsteps, int* done_out) override {
    if (!ready) return NHW_ERR_STATE;
    int done = 0, rc = NHW_OK;
    if (!graph_path()) {
      for (; done < nsteps; ++done) {
        rc = pull_scalars();
        if (rc) break;
        if (!(h_sc->time < p.total_time && h_sc->run_step < p.sim_steps)) break;
        rc = step_eager();
        if (rc != NHW_OK && rc != NHW_ERR_KRYLOV_NOCONV) { ++done; break; }
        rc = NHW_OK;
      }
      if (done_out) *done_out = done;
      return rc;
    }
    rc = capture_step(1);
    if (rc) return rc;
    NHW_CU(cudaMemsetAsync(&S.sc->step_status, 0, sizeof(int32_t), st));
    rc = pull_scalars();
    if (rc) return rc;
    snapshot();
    constexpr int kBatch = 16;
    while (done < nsteps) {
      const int64_t rs0 = h_sc->run_step;
      const int b = std::min(kBatch, nsteps - done);
      for (int q = 0; q < b; ++q) NHW_CU(cudaGraphLaunch(sgraph[1].exec, st));
      rc = pull_scalars();
      if (rc) break;
      account(sgraph[1], b);
      rc = check();
      if (rc) break;
      const int adv = (int)(h_sc->run_step - rs0);
      done += adv;
      if (h_sc->status == NHW_ERR_DT_MIN) { ++done; rc = NHW_ERR_DT_MIN; break; }
      if (h_sc->step_status == NHW_ERR_NAN) { rc = NHW_ERR_NAN; break; }
      if (adv < b) break;
    }
    if (done_out) *done_out = std::min(done, nsteps);
    return rc;
  }
  int run_timed(int nsteps, double* ms) override {
    if (!ready) return NHW_ERR_STATE;
    if (!ev_run0) { NHW_CU(cudaEventCreate(&ev_run0)); NHW_CU(cudaEventCreate(&ev_run1)); }
    const bool graphs_on = graph_path();
    if (graphs_on) {
      int rc = capture_step(0);
      if (rc) return rc;
      NHW_CU(cudaMemsetAsync(&S.sc->worst, 0, sizeof(int32_t), st));
      rc = pull_scalars();
      if (rc) return rc;
      snapshot();
    }
    NHW_CU(cudaStreamSynchronize(st));
    NHW_CU(cudaEventRecord(ev_run0, st));
    int worst = NHW_OK;
    for (int n = 0; n < nsteps; ++n) {
      if (graphs_on) {
        NHW_CU(cudaGraphLaunch(sgraph[0].exec, st));
        continue;
      }
      int rc = step_eager();
      if (rc != NHW_OK && rc != NHW_ERR_KRYLOV_NOCONV) return rc;
      if (rc != NHW_OK) worst = rc;
    }
    NHW_CU(cudaEventRecord(ev_run1, st));
    NHW_CU(cudaEventSynchronize(ev_run1));
    float f = 0.f;
    NHW_CU(cudaEventElapsedTime(&f, ev_run0, ev_run1));
    *ms = (double)f;
    if (graphs_on) {
      int rc = pull_scalars();
      if (rc) return rc;
      account(sgraph[0], nsteps);
      rc = check();
      if (rc) return rc;
      if (h_sc->status == NHW_ERR_DT_MIN) return NHW_ERR_DT_MIN;
      worst = h_sc->worst;
    }
    return worst;
  }
  int profile(int on) override {
    NHW_CU(cudaStreamSynchronize(st));
    if (on) { recs.clear(); evused = 0; }
    prof_on = on != 0;
    return NHW_OK;
  }
  // Device time of one level-0 half-sweep, the largest kernel of a step on
  // grids whose level 0 does not take the tiles; on those that it does
  // (tiled()), the half-sweeps timed here are GMRES' and not BiCGSTAB's.
  // Events around single launches add several microseconds to each, so the
  // launches are timed in bulk: a CUDA graph of `reps` rounds, each a write
  // of `flush` bytes (evicting the L2) and then the four level-0 half-sweeps
  // of a V-cycle in their order (colour 0 from x = 0, colour 1, colour 1,
  // colour 0), against a graph of the writes alone.  b is the Krylov residual
  // and x a preconditioner scratch vector: no state is written.
  int time_smoother(int reps, long long flush, double* us) override {
    if (!ready || !S.non_hydro || !use_mg || mg.empty() || !mg[0].sp) return NHW_ERR_STATE;
    if (reps < 1 || flush < 0) return NHW_ERR_ARG;
    NHW_CU(cudaStreamSynchronize(st));
    if (!ev_run0) { NHW_CU(cudaEventCreate(&ev_run0)); NHW_CU(cudaEventCreate(&ev_run1)); }
    int32_t conv = 0;
    NHW_CU(cudaMemcpy(&conv, &S.sc->conv, sizeof(conv), cudaMemcpyDeviceToHost));
    void* fb = nullptr;
    if (flush > 0) NHW_CU(cudaMalloc(&fb, (size_t)flush));
    // from here on every path restores conv and frees the buffer
    int rc = cu(cudaMemset(&S.sc->conv, 0, sizeof(conv)));
    MGL<T> L0 = mg[0];
    L0.b = S.kr;
    L0.x = S.kph;
    const Prolong<T> none{nullptr, (T)0, 1, 1, 1, 1, 1, 1};
    const bool was = prof_on;
    prof_on = false;
    const long long launches0 = launches;
    float ms[2] = {0.f, 0.f};
    for (int pass = 0; pass < 2 && rc == NHW_OK; ++pass) {
      cudaGraph_t g = nullptr;
      cudaGraphExec_t ge = nullptr;
      rc = cu(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
      if (rc) break;
      for (int r = 0; r < reps; ++r) {
        if (fb) cudaMemsetAsync(fb, r & 0xff, (size_t)flush, st);
        if (pass == 0) {
          smooth(L0, 0, 1, 0, none, MgB<T>{L0.b});
          smooth(L0, 1, 0, 0, none, MgB<T>{L0.b});
          smooth(L0, 1, 0, 0, none, MgB<T>{L0.b});
          smooth(L0, 0, 0, 0, none, MgB<T>{L0.b});
        }
      }
      rc = cu(cudaStreamEndCapture(st, &g));
      if (!rc) rc = cu(cudaGraphInstantiate(&ge, g, 0));
      if (!rc) rc = cu(cudaGraphLaunch(ge, st));   // warm-up
      if (!rc) rc = cu(cudaEventRecord(ev_run0, st));
      if (!rc) rc = cu(cudaGraphLaunch(ge, st));
      if (!rc) rc = cu(cudaEventRecord(ev_run1, st));
      if (!rc) rc = cu(cudaStreamSynchronize(st));
      if (!rc) rc = cu(cudaEventElapsedTime(&ms[pass], ev_run0, ev_run1));
      if (ge) cudaGraphExecDestroy(ge);
      if (g) cudaGraphDestroy(g);
    }
    launches = launches0;
    prof_on = was;
    cudaStreamSynchronize(st);
    if (fb) cudaFree(fb);
    const int rc2 = cu(cudaMemcpy(&S.sc->conv, &conv, sizeof(conv), cudaMemcpyHostToDevice));
    if (rc) return rc;
    if (rc2) return rc2;
    *us = 1000.0 * ((double)ms[0] - (double)ms[1]) / (4.0 * reps);
    return check();
  }
  int cu(cudaError_t e) {
    if (e == cudaSuccess) return NHW_OK;
    set_last_error(std::string("smoother timing: ") + cudaGetErrorString(e));
    return NHW_ERR_CUDA;
  }
  int profile_report(char* buf, int len) override {
    NHW_CU(cudaStreamSynchronize(st));
    std::vector<std::string> names;
    std::vector<long long> cnt;
    std::vector<double> tot;
    for (auto& r : recs) {
      float f = 0.f;
      cudaEventElapsedTime(&f, r.a, r.b);
      size_t q = 0;
      while (q < names.size() && names[q] != r.name) ++q;
      if (q == names.size()) { names.push_back(r.name); cnt.push_back(0); tot.push_back(0.0); }
      ++cnt[q];
      tot[q] += f;
    }
    std::string out = "launches " + std::to_string(launches) + "\n";
    char line[160];
    for (size_t q = 0; q < names.size(); ++q) {
      std::snprintf(line, sizeof(line), "%s %lld %.6f\n", names[q].c_str(), cnt[q], tot[q]);
      out += line;
    }
    if (buf && len > 0) {
      const int n = std::min<int>((int)out.size(), len - 1);
      std::memcpy(buf, out.data(), n);
      buf[n] = 0;
    }
    return (int)out.size();
  }
  // ------------------------------------------------------ checkpoint/resume
  // A snapshot is a header, the device scalars (TIME, dt, RUN_STEP, solver
  // counters) and the arena prefix from the grids through P: every array a
  // step reads before writing it.  The Poisson and Krylov arrays after it are
  // rebuilt by every solve and are not saved.
  // 2: per-cell eddy viscosities of viscous flow and the k-epsilon state
  // in the state prefix
  static constexpr int32_t kCkptVersion = 2;
  struct CkptHeader {
    char magic[8];
    int32_t version, precision, M, N, K, reserved;
    uint64_t state_bytes, scal_bytes;
  };
  size_t ckpt_size() const { return sizeof(CkptHeader) + sizeof(DevScal) + state_bytes; }
  int checkpoint_bytes(size_t* bytes) override {
    *bytes = ckpt_size();
    return NHW_OK;
  }
  int save_state(void* host, size_t bytes) override {
    if (!ready) return NHW_ERR_STATE;
    if (!host || bytes < ckpt_size()) return NHW_ERR_ARG;
    CkptHeader h{};
    std::memcpy(h.magic, "NHWCKPT1", 8);
    h.version = kCkptVersion;
    h.precision = kFP32 ? NHW_FP32_IR : NHW_FP64;
    h.M = S.M; h.N = S.N; h.K = S.K;
    h.state_bytes = state_bytes;
    h.scal_bytes = sizeof(DevScal);
    char* out = static_cast<char*>(host);
    std::memcpy(out, &h, sizeof(h));
    NHW_CU(cudaStreamSynchronize(st));
    NHW_CU(cudaMemcpy(out + sizeof(h), S.sc, sizeof(DevScal), cudaMemcpyDeviceToHost));
    NHW_CU(cudaMemcpy(out + sizeof(h) + sizeof(DevScal), arena, state_bytes, cudaMemcpyDeviceToHost));
    return NHW_OK;
  }
  int load_state(const void* host, size_t bytes) override {
    if (!ready) return NHW_ERR_STATE;
    if (!host || bytes < sizeof(CkptHeader)) return NHW_ERR_ARG;
    CkptHeader h{};
    std::memcpy(&h, host, sizeof(h));
    if (std::memcmp(h.magic, "NHWCKPT1", 8) != 0 || h.version != kCkptVersion) {
      set_last_error("nhw_load_state: not a checkpoint of this library");
      return NHW_ERR_ARG;
    }
    if (h.precision != (kFP32 ? NHW_FP32_IR : NHW_FP64) || h.M != S.M || h.N != S.N || h.K != S.K ||
        h.state_bytes != state_bytes || h.scal_bytes != sizeof(DevScal) || bytes < ckpt_size()) {
      set_last_error("nhw_load_state: checkpoint of a different grid, precision or build");
      return NHW_ERR_ARG;
    }
    const char* in = static_cast<const char*>(host);
    NHW_CU(cudaStreamSynchronize(st));
    NHW_CU(cudaMemcpy(S.sc, in + sizeof(h), sizeof(DevScal), cudaMemcpyHostToDevice));
    NHW_CU(cudaMemcpy(arena, in + sizeof(h) + sizeof(DevScal), state_bytes, cudaMemcpyHostToDevice));
    return pull_scalars();
  }

  int mass(double* m) override {
    L("mass", [&] { k_mass<T><<<1, 1, 0, st>>>(S, d_out); });
    NHW_CU(cudaMemcpyAsync(h_out, d_out, sizeof(double), cudaMemcpyDeviceToHost, st));
    NHW_CU(cudaStreamSynchronize(st));
    *m = h_out[0];
    return check();
  }
  // MassVolume, Energy, MaxEta, MinEta, MaxU, MaxV, MaxW
  int statistics(double* out7) override {
    const int nb = (int)cdiv((long long)S.M * S.N, 256);
    L("statistics", [&] {
      k_stats<T><<<nb, 256, 0, st>>>(S);
      k_stats_final<T><<<1, 256, 0, st>>>(S, nb, d_out);
    });
    NHW_CU(cudaMemcpyAsync(h_out, d_out, sizeof(double) * kStatN, cudaMemcpyDeviceToHost, st));
    NHW_CU(cudaStreamSynchronize(st));
    for (int m = 0; m < kStatN; ++m) out7[m] = h_out[m];
    return check();
  }
};

SolverBase* make_solver_fp64(const nhw_params& p, int* status);
SolverBase* make_solver_fp32(const nhw_params& p, int* status);
int device_bytes_fp64(const nhw_params& p, size_t* bytes);
int device_bytes_fp32(const nhw_params& p, size_t* bytes);

// device memory a scenario's handle holds (its arena), computed without allocating
template <class T>
int device_bytes_t(const nhw_params& p, size_t* bytes) {
  Solver<T> s;
  s.estimate_only = true;
  const int rc = s.create(p);
  *bytes = s.arena_bytes;
  return rc;
}

template <class T>
SolverBase* make_solver_t(const nhw_params& p, int* status) {
  auto* s = new Solver<T>();
  int rc = s->create(p);
  if (status) *status = rc;
  if (rc) { delete s; return nullptr; }
  return s;
}

}  // namespace nhw
