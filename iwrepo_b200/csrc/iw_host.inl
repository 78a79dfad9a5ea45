// Host side of the library: setup tables, handle, step orchestration, C ABI.
// Included at the end of iw_lib.cu (it launches the kernels defined there).
//
// Host setup code is compiled without floating-point contraction
// (-Xcompiler -ffp-contract=off) so the tables equal the ones the reference
// builds (setup.f, penalty.f param_set) bit for bit.

struct Tables {
  std::vector<double> zpts, wg, alpol, D, D2, sigma, Lfil;
};

// One system kind: 0 pressure, 1 u/v, 2 w, 3 rho.
enum { SYS_P = 0, SYS_U, SYS_W, SYS_T, SYS_KINDS };

#ifndef IW_INST
namespace {

// --------------------------------------------------------------------------
// setup.f restated for the host (GLL points, weights, Legendre table,
// Costa-Don derivative matrix).
// --------------------------------------------------------------------------
void h_legen(std::vector<double>& al, int n, double xc) {
  al.assign(n + 2, 0.0);
  al[0] = 1.;
  al[1] = xc;
  for (int k = 1; k <= n; ++k) {
    int kp = k + 1, km = k - 1;
    al[kp] = (2. * k + 1.) * xc * al[k] / kp - k * al[km] / kp;
  }
}

void h_jacobf(int n, double& poly, double& pder, double& polym1, double& pderm1, double& polym2, double& pderm2,
              double x) {
  poly = 1.0;
  pder = 0.0;
  if (n == 0) return;
  double polylst = poly, pderlst = pder;
  poly = x;
  pder = 1.0;
  if (n == 1) return;
  double psave = 0, pdsave = 0;
  for (int k = 2; k <= n; ++k) {
    double a1 = 2. * k * (k + 0.0) * (2. * k + 0.0 - 2.);
    double a2 = (2. * k + 0.0 - 1.) * (0.0);
    double b3 = (2. * k + 0.0 - 2.);
    double a3 = b3 * (b3 + 1.) * (b3 + 2.);
    double a4 = 2. * (k + 0.0 - 1.) * (k + 0.0 - 1.) * (2. * k + 0.0);
    double polyn = ((a2 + a3 * x) * poly - a4 * polylst) / a1;
    double pdern = ((a2 + a3 * x) * pder - a4 * pderlst + a3 * poly) / a1;
    psave = polylst;
    pdsave = pderlst;
    polylst = poly;
    poly = polyn;
    pderlst = pder;
    pder = pdern;
  }
  polym1 = polylst;
  pderm1 = pderlst;
  polym2 = psave;
  pderm2 = pdsave;
}

void h_jacobl(int n, std::vector<double>& xcol) {
  std::vector<double> xjac(n + 3, 0.0);
  int np = n + 1;
  double pnp1p, pdnp1p, pnp, pdnp, pnm1p, pdnm1, pnp1m, pdnp1m, pnm, pdnm, pnm1m;
  h_jacobf(np, pnp1p, pdnp1p, pnp, pdnp, pnm1p, pdnm1, 1.0);
  h_jacobf(np, pnp1m, pdnp1m, pnm, pdnm, pnm1m, pdnm1, -1.0);
  double det = pnp * pnm1m - pnm * pnm1p;
  double rp = -pnp1p, rm = -pnp1m;
  double a = (rp * pnm1m - rm * pnm1p) / det;
  double b = (rm * pnp - rp * pnm) / det;
  xjac[1] = 1.0;
  int nh = (n + 1) / 2;
  double dth = 3.14159265 / (2 * n + 1);
  double cd_ = std::cos(2. * dth), sd = std::sin(2. * dth), cs = std::cos(dth), ss = std::sin(dth);
  for (int j = 2; j <= nh; ++j) {
    double x = cs;
    for (int k = 1; k <= 10; ++k) {
      double pnp1, pdnp1, pn, pdn, pnm1;
      h_jacobf(np, pnp1, pdnp1, pn, pdn, pnm1, pdnm1, x);
      double poly = pnp1 + a * pn + b * pnm1;
      double pder = pdnp1 + a * pdn + b * pdnm1;
      double recsum = 0.0;
      for (int i = 1; i <= j - 1; ++i) recsum = recsum + 1.0 / (x - xjac[i]);
      double delx = -poly / (pder - recsum * poly);
      x = x + delx;
      if (std::fabs(delx) < 1.0e-12) break;
    }
    xjac[j] = x;
    double cssave = cs * cd_ - ss * sd;
    ss = cs * sd + ss * cd_;
    cs = cssave;
  }
  xjac[np] = -1.0;
  for (int i = 2; i <= nh; ++i) xjac[n + 2 - i] = -xjac[i];
  if (n % 2 == 0) xjac[nh + 1] = 0.0;
  xcol.assign(n + 1, 0.0);
  for (int k = 0; k <= n; ++k) xcol[k] = xjac[n - k + 1];
}

Tables h_tables(int N, double p, double amp, double fackc) {
  Tables t;
  int n = N - 1;
  h_jacobl(n, t.zpts);
  t.wg.assign(N, 0.0);
  t.alpol.assign((size_t)N * N, 0.0);
  std::vector<double> al;
  for (int k = 0; k <= n; ++k) {
    h_legen(al, n, t.zpts[k]);
    t.wg[k] = 2. / ((double)(n * (n + 1)) * al[n] * al[n] + 1.0e-30);
    for (int j = 0; j <= n; ++j) t.alpol[(size_t)j * N + k] = al[j];
  }
  std::vector<double> c(N);
  const auto& x = t.zpts;
  for (int k = 0; k <= n; ++k) {
    double prod = 1.;
    for (int l = 0; l <= n; ++l)
      if (l != k) prod = prod * (x[k] - x[l]);
    c[k] = prod;
  }
  t.D.assign((size_t)N * N, 0.0);
  t.D2 = t.D;
  for (int k = 0; k <= n; ++k)
    for (int j = 0; j <= n; ++j) t.D[k * N + j] = (k != j) ? c[k] / (c[j] * (x[k] - x[j])) : 0.;
  for (int k = 0; k <= n; ++k) {
    double s = 0.;
    for (int j = 0; j <= n; ++j)
      if (k != j) s = s + t.D[k * N + j];
    t.D[k * N + k] = -s;
  }
  for (int k = 0; k <= n; ++k)
    for (int j = 0; j <= n; ++j)
      t.D2[k * N + j] = (k != j) ? 2.0 * (t.D[k * N + k] * t.D[k * N + j] - t.D[k * N + j] / (x[k] - x[j])) : 0.;
  for (int k = 0; k <= n; ++k) {
    double s = 0.;
    for (int j = 0; j <= n; ++j)
      if (k != j) s = s + t.D2[k * N + j];
    t.D2[k * N + k] = -s;
  }
  // specfilter (filtering.f:1225-1243)
  int kc = (int)(fackc * n);
  t.sigma.assign(N, 1.0);
  for (int k = 0; k <= n; ++k)
    if (k >= kc) {
      double theta = (double)(k - kc) / (double)(n - kc);
      t.sigma[k] = std::exp(-amp * std::pow(theta, 2. * p));
    }
  // precombined filter: out(k1) = sum_j L(k1,j) f(j)
  t.Lfil.assign((size_t)N * N, 0.0);
  for (int k1 = 0; k1 < N; ++k1)
    for (int jj = 0; jj < N; ++jj) {
      long double s = 0;
      for (int k = 0; k <= n; ++k) {
        long double ck = (k == n) ? 0.5L * n : (k + 0.5L);
        s += (long double)t.alpol[(size_t)k * N + k1] * t.sigma[k] * ck * t.wg[jj] * t.alpol[(size_t)k * N + jj];
      }
      t.Lfil[k1 * N + jj] = (double)s;
    }
  return t;
}

// penalty.f:57-157 param_set
void h_param_set(double omega, const iw_params& pp, int ifbc, double& a0, double& b0, double& t0, double eps,
                 double ybar) {
  if (ifbc == 0) {
    a0 = 1.;
    b0 = 0.;
    double fac = pp.facdir * ((2. / ybar) * (2. / ybar));
    t0 = fac * eps / (a0 * (omega * omega));
  } else if (ifbc == 1) {
    a0 = 0.;
    b0 = 1.;
    double fac = pp.facneumn * 2. / ybar;
    t0 = fac / (b0 * omega);
  } else {
    a0 = 1.;
    b0 = 1.;
    double ck = a0 * omega / b0;
    double dn = 1. / (omega * eps * b0);
    double t1 = std::sqrt(ck * ck + eps * ck);
    double t2 = 2. * ck - 2. * t1;
    double facm = ((1. / eps) >= 1.e5) ? pp.facrobin : 1.;
    t0 = facm * dn * (eps + t2) * 2. / ybar;
  }
}

// all penalty parameters of one system (penalty_setup + penalty_main ends)
void h_penalty(int ns, int N, const iw_params& pp, double eps, int bot, int top, double* out /*6*ns*/) {
  double omega = 2. / (double)((N + 1) * (N + 2));
  double *pa = out, *pb = out + ns, *pg = out + 2 * ns, *pd = out + 3 * ns, *pt1 = out + 4 * ns, *pt2 = out + 5 * ns;
  for (int i = 0; i < 6 * ns; ++i) out[i] = 0.0;
  double a0, b0, t0;
  for (int ks = 1; ks < ns - 1; ++ks) {
    h_param_set(omega, pp, 2, a0, b0, t0, eps, pp.zh[ks]);
    pa[ks] = a0;
    pb[ks] = b0;
    pt1[ks] = t0;
    pg[ks] = a0;
    pd[ks] = b0;
    pt2[ks] = t0;
  }
  h_param_set(omega, pp, bot, a0, b0, t0, eps, pp.zh[0]);
  pa[0] = a0;
  pb[0] = b0;
  pt1[0] = t0;
  if (ns > 1) {
    h_param_set(omega, pp, 2, a0, b0, t0, eps, pp.zh[0]);
    pg[0] = a0;
    pd[0] = b0;
    pt2[0] = t0;
  }
  h_param_set(omega, pp, top, a0, b0, t0, eps, pp.zh[ns - 1]);
  pg[ns - 1] = a0;
  pd[ns - 1] = b0;
  pt2[ns - 1] = t0;
  if (ns > 1) {
    h_param_set(omega, pp, 2, a0, b0, t0, eps, pp.zh[ns - 1]);
    pa[ns - 1] = a0;
    pb[ns - 1] = b0;
    pt1[ns - 1] = t0;
  }
}

FftPlan make_plan(int M) {
  FftPlan p;
  memset(&p, 0, sizeof p);
  p.M = M;
  int m = M, ns = 1;
  auto lg2 = [](int v) {
    if (v <= 0 || (v & (v - 1))) return -1;
    int l = 0;
    while ((1 << l) < v) ++l;
    return l;
  };
  auto push = [&](int r) {
    p.rad[p.npass] = r;
    p.ns[p.npass] = ns;
    p.nbsh[p.npass] = lg2(M / r);
    p.nssh[p.npass] = lg2(ns);
    p.inb[p.npass] = 1.0f / (float)(M / r);
    p.ins[p.npass] = 1.0f / (float)ns;
    ns *= r;
    p.npass++;
  };
  // powers of two: ceil(a/3) passes of radix <= 8, bits spread evenly
  // (512 -> 8*8*8, 256 -> 8*8*4); larger radices cost more registers than
  // they save in passes.  Mixed lengths: the fewest passes over 8, 6, 5, 4, 3, 2,
  // and of those the smallest sum of radices (96 -> 6*4*4, 120 -> 6*5*4).
  int a2 = 0, a3 = 0, a5 = 0;
  while (m % 2 == 0) m /= 2, ++a2;
  while (m % 3 == 0) m /= 3, ++a3;
  while (m % 5 == 0) m /= 5, ++a5;
  int best6 = 0, bestn = 1 << 30, bests = 0;
  for (int n6 = 0; n6 <= std::min(a2, a3); ++n6) {
    const int b2 = a2 - n6, n = n6 + (b2 + 2) / 3 + (a3 - n6);
    int sum = 6 * n6 + 3 * (a3 - n6);
    for (int q = 0, np = (b2 + 2) / 3; q < np; ++q) sum += 1 << (b2 / np + (q < b2 % np ? 1 : 0));
    if (n < bestn || (n == bestn && sum < bests)) {
      best6 = n6;
      bestn = n;
      bests = sum;
    }
  }
  for (int q = 0; q < best6; ++q) push(6);
  a2 -= best6;
  a3 -= best6;
  for (int q = 0, np = (a2 + 2) / 3; q < np; ++q) push(1 << (a2 / np + (q < a2 % np ? 1 : 0)));
  for (int q = 0; q < a3; ++q) push(3);
  for (int q = 0; q < a5; ++q) push(5);
  if (m != 1) p.npass = -1;
  return p;
}

}  // namespace
#endif  // IW_INST

template <typename C>
std::vector<C> twiddles(int n, int count) {  // exp(-2 pi i e / n), e < count
  std::vector<C> w(count);
  for (int e = 0; e < count; ++e) {
    long double a = -2.0L * 3.14159265358979323846264338327950288L * e / n;
    w[e].x = (decltype(w[e].x))std::cos(a);
    w[e].y = (decltype(w[e].x))std::sin(a);
  }
  return w;
}

// per-precision device buffers
template <typename T>
struct FieldSet {
  T* F[4] = {0, 0, 0, 0};
  T* Fn[4] = {0, 0, 0, 0};
  T* Fnm[4] = {0, 0, 0, 0};
  T* Sn[4] = {0, 0, 0, 0};
  T* Snm[4] = {0, 0, 0, 0};
  T* F1[4] = {0, 0, 0, 0};
  T* Z4[4] = {0, 0, 0, 0};
  T* Y12[12] = {0};
  T* X11[11] = {0};
  T* B8[8] = {0};
  T* G = 0;  // interface planes
  typename cplx_t<T>::type *Wm = 0, *Wn = 0, *Wy = 0;
};

struct iw_handle {
  iw_dims d;
  iw_params p;
  int dev = 0;
  cudaStream_t st = 0;
  int nx, ny, nz, N, ns, nxpp, nxh, nxhp, nyh, ndims, ncol;
  size_t ntot, plane;
  bool mixed = false;
  // adaptive time step (imaxcalc = 1): the wave frequency that bounds the step
  // (Tlim) and the change in progress (COMMON /vardtflags/ ivardt, idtstep
  // and cdt of comtime.h)
  double xomega = 0, cdt = 1.0;
  int ivardt = 0, idtstep = 0;
  // 1 after iw_read_restart in the reference's mode (main.f istart = 1): the
  // first step's schedule uses variable-step coefficients with ratio cdt
  int istart = 0;
  // asynchronous field dumps (iw_write_fields): pinned staging buffer, the
  // event after the last copy into it, and the writer thread of the last dump
  void* out_host = nullptr;
  size_t out_bytes = 0;
  cudaEvent_t out_ev = nullptr;
  std::thread* out_thread = nullptr;
  int out_status = 0;
  std::string out_msg;
  // animation dumps (solver.f:136-222): interval (0 = off), the time of the
  // last dump (COMMON /Dump/ Tdump), the file counter, directory and staging
  double dtanim = 0, tdump = 0;
  int ianimc = 0;
  bool anim_pending = false;  // this step's convec dumps (after stage A)
  std::string anim_dir;
  void* anim_host = nullptr;
  size_t anim_bytes = 0;
  // Legendre spectra (main.f:905-910, speclegencalc): every nlegspec steps
  // (0 = off), |a_k| per (subdomain, x, k) on the device, staged to the host
  int nlegspec = 0;
  std::string leg_dir;
  double* dlegspec = nullptr;
  void* leg_host = nullptr;
  size_t leg_bytes = 0;
  // TKE budget (postp, main.f:935-936): every npostp steps (0 = off)
  int npostp = 0;
  double tstart = 0;
  std::string postp_dir;
  bool postp_started = false;  // headers written
  double* dpostp = nullptr;    // per-(y, z) row sums
  Tables tab;
  // device tables
  double *ddzinv = 0, *dpart = 0;  // diagnostics: dt-free CFL spacing per level, per-block partials
  double *dDt = 0, *dD2t = 0, *dLt = 0;  // transposed D, D2, Legendre filter (t[k*N + k1] = D[k1][k])
  double *dD = 0, *dD2 = 0, *dL = 0, *dh = 0, *dxw = 0, *dyw = 0, *dcf = 0, *dzg = 0, *dzh = 0;
  double *dwg = 0, *dal = 0, *dsig = 0, *dmeang = 0;
  double *dwnl = 0, *dwvr = 0, *dred = 0;
  int* dcnt = 0;
  int* dflag = 0;
  int* derr = 0;  // device error words: [0] non-finite state, [1] a bounded device wait gave up
  int* herr = 0;  // pinned host copy of derr, written after each eager step or graph run
  double* hstat = 0;  // pinned: k_xrow_stats' partials and four ints behind them
  cudaEvent_t err_ev = 0;
  bool err_ev_live = false;
  FftPlan plx, ply;
  FieldSet<double> f64;
  FieldSet<double> tw64;  // twiddles only: FP64 transforms of host fields in a mixed run
  FieldSet<float> f32;
  // systems
  std::vector<double> akv;     // distinct kx^2+ky^2 values
  std::vector<int> col_u;      // column -> distinct index
  std::vector<int> order;      // columns sorted by distinct index
  double* dakv = 0;            // akv on the device
  int* dcolorder = 0;          // columns sorted by distinct index
  int nsys_kind[SYS_KINDS] = {0, 0, 0, 0};
  double* dab[SYS_KINDS] = {0, 0, 0, 0};
  int* dipiv[SYS_KINDS] = {0, 0, 0, 0};
  int* dinfo[SYS_KINDS] = {0, 0, 0, 0};
  SysDesc* dsys[SYS_KINDS] = {0, 0, 0, 0};
  double* dpen[SYS_KINDS] = {0, 0, 0, 0};
  int* dcolsys[SYS_KINDS] = {0, 0, 0, 0};
  // block inverses of the viscous / diffusive systems
  struct BI {
    void* ainv = 0;
    double *minv = 0, *pen = 0, *lvec = 0;
    double* ainv_raw = 0;  // unfiltered inverses of systems [0, nsys_raw) when ainv has the filter folded in
    int nsys_raw = 0;
    SysDesc* sys = 0;
    int* colsys = 0;
    void release() {
      for (void* p : {ainv, (void*)minv, (void*)pen, (void*)lvec, (void*)ainv_raw, (void*)sys, (void*)colsys}) cudaFree(p);
      *this = BI();
    }
  } bi[SYS_KINDS];
  // device scratch and FP64 twiddles of the routines on host fields (iw_abi.inl)
  double* scr = nullptr;
  size_t scr_n = 0;
  std::mutex scr_mu, tw_mu;
  int fail_alloc = 0;  // iw_fail_allocation: device allocations until one is refused
  bool use_bi = true;
  // grouped solve tasks per kind (columns sharing a system, <= G per task)
  Task* dtasks[SYS_KINDS] = {0, 0, 0, 0};
  int ntask[SYS_KINDS] = {0, 0, 0, 0};
  std::vector<Task> htasks[SYS_KINDS];
  // tasks [0, nrefine) get one FP64 residual sweep: their systems have an
  // estimated condition number above kRefineCond (small kx^2+ky^2 pressure)
  int nrefine[SYS_KINDS] = {0, 0, 0, 0};
  // system-grouped tasks of k_solve_sys (up to 4 u/v or 8 other columns of
  // one system each) for the sorted columns after tasks [0, nold) of k_solve_cta
  Task* dtasks2[SYS_KINDS] = {0, 0, 0, 0};
  int ntask2[SYS_KINDS] = {0, 0, 0, 0};
  int nold[SYS_KINDS] = {0, 0, 0, 0};
  // 0: k_solve_cta for every task, 1: k_solve_sys, 2: k_solve_tc (k_solve_sys where it does not apply), 3: k_solve_sys2
  int use_sys = 2;
  int sys_role[4] = {-1, -1, -1, -1};  // per solve role (u/v, w, rho, pressure), set by iw_autotune; -1: use_sys
  int nsm = 148;  // SMs of the device (persistent kernels)
  double bi_bdfv[SYS_KINDS] = {-1, -1, -1, -1};
  bool bi_fold[SYS_KINDS] = {false, false, false, false};  // Legendre filter folded into ainv
  // distinct subdomain blocks: subdomain ks uses block bmap[ks]; brep[b] is a
  // subdomain of block b
  int nb = 0;
  int bmap[IW_MAX_SUBD] = {};
  // launch choices set by iw_autotune (0 / -1: built-in heuristic)
  cudaStream_t st2 = nullptr;  // side branch of a step (side_fork)
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  int tune_ytx = 0;  // y-tile width
  int tune_xthr = 0;  // threads per x-row CTA: 256 or 128, 0: by length
  int tune_a = -1;   // stage A: -1 tensor cores, 1 register-column, 0 tiled
  int tune_e = -1;   // stage E: -1, 2, 3 tensor cores, 1 register-column, 0 tiled
  int brep[IW_MAX_SUBD] = {};
  double bi_dt[SYS_KINDS] = {-1, -1, -1, -1};
  double fac_bdfv[SYS_KINDS] = {-1, -1, -1, -1};  // bdfv the factors were built for
  double fac_dt[SYS_KINDS] = {-1, -1, -1, -1};
  // time stepping
  double t = 0;
  int istep = 0;
  Coefs c{1, 0, 0, 1, 0, 0, 1, 0};
  int avg_count[4] = {0, 0, 0, 0};
  size_t bytes = 0;
  // helm batched
  std::map<std::string, int> helm_keys;
  // per-phase timing with CUDA events on the handle's stream
  int prof = 0;
  cudaEvent_t ev[32];
  int nev = 0;
  int ev_phase[32];
  double phase_ms[16] = {0};
  long phase_n[16] = {0};
};

// phases: 0 stageA, 1 yinv, 2 xrow, 3 yfwd, 4 wviscrot, 5 stageE, 6 press,
// 7 visc_uv, 8 visc_w, 9 visc_t, 10 iface, 11 factor
// Work beside the handle's stream: what is launched on the stream that side_fork returns is ordered
// after all work before it and, from side_join on, before all work after it (in a capture, a
// branch of the graph).  One stream while the phases are timed.
static cudaStream_t side_fork(iw_handle* h) {
  if (h->prof) return h->st;
  cudaEventRecord(h->ev_fork, h->st);
  cudaStreamWaitEvent(h->st2, h->ev_fork, 0);
  return h->st2;
}
static void side_join(iw_handle* h) {
  if (h->prof) return;
  cudaEventRecord(h->ev_join, h->st2);
  cudaStreamWaitEvent(h->st, h->ev_join, 0);
}
static void side_free(iw_handle* h) {  // the streams and their events
  if (h->ev_fork) cudaEventDestroy(h->ev_fork);
  if (h->ev_join) cudaEventDestroy(h->ev_join);
  if (h->st2) cudaStreamDestroy(h->st2);
  if (h->st) cudaStreamDestroy(h->st);
}
static void mark(iw_handle* h, int phase) {
  if (!h->prof || h->nev >= 32) return;
  cudaEventRecord(h->ev[h->nev], h->st);
  h->ev_phase[h->nev] = phase;
  h->nev++;
}
static void prof_flush(iw_handle* h) {
  if (!h->prof || h->nev < 2) {
    h->nev = 0;
    return;
  }
  cudaEventSynchronize(h->ev[h->nev - 1]);
  for (int i = 1; i < h->nev; ++i) {
    float ms = 0;
    cudaEventElapsedTime(&ms, h->ev[i - 1], h->ev[i]);
    int ph = h->ev_phase[i];
    h->phase_ms[ph] += ms;
    h->phase_n[ph] += 1;
  }
  h->nev = 0;
}

static iw_handle* g_bound = nullptr;
constexpr size_t kPartDoubles = 6400;  // per-block partials of k_xrow_stats

// Every host<->device copy goes through the handle's (non-blocking) stream
// and waits for it: a plain cudaMemcpy from pageable memory may return before
// its DMA reaches device memory, and work queued on a non-blocking stream is
// not ordered after it.
static cudaError_t scopy(iw_handle* h, void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
  cudaError_t e = cudaMemcpyAsync(dst, src, bytes, kind, h->st);
  if (e != cudaSuccess) return e;
  return cudaStreamSynchronize(h->st);
}

template <typename T>
static int dalloc(iw_handle* h, T** p, size_t n) {
  *p = nullptr;
  if (h->fail_alloc > 0 && --h->fail_alloc == 0) return set_err(IW_ERR_NOMEM, "allocation refused (iw_fail_allocation)");
  cudaError_t e = cudaMalloc((void**)p, n * sizeof(T) + 16);
  if (e != cudaSuccess) {
    cudaGetLastError();  // reported here: no later check finds it again
    return set_err(IW_ERR_NOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  }
  h->bytes += n * sizeof(T);
  return 0;
}
template <typename T>
static int up(iw_handle* h, T** p, const std::vector<T>& v) {
  int r = dalloc(h, p, v.size());
  if (r) return r;
  const cudaError_t e = scopy(h, *p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(*p);
    *p = nullptr;
    return set_err(IW_ERR_CUDA, std::string("upload: ") + cudaGetErrorString(e));
  }
  return 0;
}

static double pi2_of(const iw_handle*) { return 8.0 * std::atan(1.0); }

static Geo geo(const iw_handle* h) {
  Geo g;
  g.nx = h->nx;
  g.ny = h->ny;
  g.nz = h->nz;
  g.N = h->N;
  g.ns = h->ns;
  g.nxpp = h->nxpp;
  g.nxh = h->nxh;
  g.nxhp = h->nxhp;
  g.nyh = h->nyh;
  g.plane = h->plane;
  g.ntot = h->ntot;
  g.scaley = 1. / (double)h->ny;
  g.dt = h->p.dt;
  g.D = h->dD;
  g.Lfil = h->dL;
  g.hfac = h->dh;
  g.xw = h->dxw;
  g.yw = h->dyw;
  g.cfour = h->dcf;
  g.zg = h->dzg;
  return g;
}

template <typename T>
static int alloc_fields(iw_handle* h, FieldSet<T>& fs) {
  size_t n = h->ntot;
  for (int q = 0; q < 4; ++q) {
    for (T** p : {&fs.F[q], &fs.Fn[q], &fs.Fnm[q], &fs.Sn[q], &fs.Snm[q], &fs.F1[q], &fs.Z4[q]}) {
      if (dalloc(h, p, n)) return IW_ERR_NOMEM;
      CK(cudaMemset(*p, 0, n * sizeof(T)));
    }
  }
  for (int q = 0; q < 12; ++q)
    if (dalloc(h, &fs.Y12[q], n)) return IW_ERR_NOMEM;
  for (int q = 0; q < 11; ++q)
    if (dalloc(h, &fs.X11[q], n)) return IW_ERR_NOMEM;
  for (int q = 0; q < 8; ++q)
    if (dalloc(h, &fs.B8[q], n)) return IW_ERR_NOMEM;
  if (h->ns > 1 && dalloc(h, &fs.G, h->plane * 16 * (size_t)(h->ns - 1))) return IW_ERR_NOMEM;
  typedef typename cplx_t<T>::type C;
  int M = h->nx / 2;
  auto wm = twiddles<C>(M, M);
  auto wn = twiddles<C>(h->nx, M + 1);
  auto wy = twiddles<C>(h->ny, h->ny);
  if (up(h, &fs.Wm, wm) || up(h, &fs.Wn, wn) || up(h, &fs.Wy, wy)) return IW_ERR_NOMEM;
  return 0;
}

template <typename T>
static void free_fields(FieldSet<T>& fs) {
  for (int q = 0; q < 4; ++q)
    for (T* p : {fs.F[q], fs.Fn[q], fs.Fnm[q], fs.Sn[q], fs.Snm[q], fs.F1[q], fs.Z4[q]}) cudaFree(p);
  for (int q = 0; q < 12; ++q) cudaFree(fs.Y12[q]);
  for (int q = 0; q < 11; ++q) cudaFree(fs.X11[q]);
  for (int q = 0; q < 8; ++q) cudaFree(fs.B8[q]);
  cudaFree(fs.G);
  cudaFree(fs.Wm);
  cudaFree(fs.Wn);
  cudaFree(fs.Wy);
}

#ifndef IW_INST
// ---------------------------------------------------------------------------
// systems: distinct kx^2+ky^2 (the matrix of a column depends on it only)
// ---------------------------------------------------------------------------
static int build_distinct(iw_handle* h) {
  std::vector<double> ak(h->ncol);
  for (int j = 0; j < h->ny; ++j)
    for (int ii = 0; ii < h->nxhp; ++ii) {
      double xw = ii * (8.0 * std::atan(1.0) / h->p.xlen);
      double ywv = 0.0;
      if (h->ny > 1) {
        double beta = 8.0 * std::atan(1.0) / h->p.ylen;
        int jj = j + 1;  // 1-based
        ywv = (jj <= h->nyh) ? (jj - 1) * beta : -(h->ny + 1 - jj) * beta;
      }
      ak[(size_t)j * h->nxhp + ii] = xw * xw + ywv * ywv;
    }
  std::vector<double> s = ak;
  std::sort(s.begin(), s.end());
  s.erase(std::unique(s.begin(), s.end()), s.end());
  h->akv = s;
  h->col_u.resize(h->ncol);
  for (int c = 0; c < h->ncol; ++c) h->col_u[c] = (int)(std::lower_bound(s.begin(), s.end(), ak[c]) - s.begin());
  std::vector<int> order(h->ncol);
  for (int c = 0; c < h->ncol; ++c) order[c] = c;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return h->col_u[a] < h->col_u[b]; });
  h->order = order;
  return up(h, &h->dcolorder, order) || up(h, &h->dakv, h->akv);
}

static int kind_bcs(const iw_handle* h, int kind, int& bot, int& top) {
  if (kind == SYS_P || kind == SYS_T) {
    bot = 1;
    top = 1;
  } else if (kind == SYS_U) {
    bot = h->p.bc_variant == IW_BC_NOSLIP ? 0 : 1;
    top = 1;
  } else {
    bot = 0;
    top = 0;
  }
  return 0;
}

// tasks: runs of the sorted column order that share one system, split into
// pieces of at most G columns
// systems above this estimated condition number get a residual sweep
constexpr double kRefineCond = 1e5;

static int build_tasks(iw_handle* h, int kind, const std::vector<int>& colsys, int G) {
  const std::vector<int>& order = h->order;
  std::vector<Task> tasks;
  int i = 0;
  while (i < h->ncol) {
    const int s = colsys[order[i]];
    int jn = i;
    while (jn < h->ncol && colsys[order[jn]] == s && jn - i < (s < 0 ? 1 : G)) ++jn;
    tasks.push_back(Task{s, i, jn - i});
    i = jn;
  }
  Task* d = nullptr;
  if (up(h, &d, tasks)) return IW_ERR_NOMEM;
  cudaFree(h->dtasks[kind]);
  h->dtasks[kind] = d;
  h->ntask[kind] = (int)tasks.size();
  h->htasks[kind] = tasks;
  return 0;
}

// tasks of k_solve_sys: after the k_solve_cta prefix (the refined tasks and
// the columns without a system, which sort first), runs of the sorted column
// order that share one system, in pieces of at most 4 (u/v) or 8 columns.  nrefine: the
// refined tasks; the handle takes it and the tasks over together, or neither.
static int build_sys_tasks(iw_handle* h, int kind, int nrefine) {
  const auto& tk = h->htasks[kind];
  const int skip = (kind == SYS_P || kind == SYS_W) && h->akv[0] == 0.0 ? 1 : 0;
  int nold = nrefine;
  while (nold < (int)tk.size() && tk[nold].sys < 0) ++nold;
  const int G = kind == SYS_U ? kSysR / 4 : kSysR / 2;
  const std::vector<int>& order = h->order;
  std::vector<Task> tasks;
  int i = nold < (int)tk.size() ? tk[nold].first : h->ncol;
  while (i < h->ncol) {
    const int s = h->col_u[order[i]] - skip;
    int jn = i;
    while (jn < h->ncol && h->col_u[order[jn]] - skip == s && jn - i < G) ++jn;
    tasks.push_back(Task{s, i, jn - i});
    i = jn;
  }
  Task* d = nullptr;
  if (!tasks.empty() && up(h, &d, tasks)) return IW_ERR_NOMEM;
  cudaFree(h->dtasks2[kind]);
  h->dtasks2[kind] = d;
  h->ntask2[kind] = (int)tasks.size();
  h->nold[kind] = nold;
  h->nrefine[kind] = nrefine;
  return 0;
}

// SGBTF2 of nsys assembled bands (k_band_lu)
static void launch_band_lu(cudaStream_t st, int nsys, int n, int N, double* ab, int* ipiv, int* info) {
  const size_t sm = lu_smem(N);
  set_smem(k_band_lu, sm);
  // A step's barrier costs more with eight warps than four, its update more with three warps than seven (us, 128 / 256
  // threads; one system of 12 x 3 points 64 / 74, 17 x 4 107 / 125, penalty_main_ with 25 x 12 748 / 661;
  // a first isolated solve of 2112 columns of 17 x 4 1089 / 1200).
  k_band_lu<<<nsys, N <= 17 ? kLuThreads / 2 : kLuThreads, sm, st>>>(n, N, ab, ipiv, info);
}

// (re)build the factors of one kind for the current bdfv/dt
static int build_factors(iw_handle* h, int kind) {
  const int ns = h->ns, N = h->N, n = h->nz, ldab = 3 * N + 1;
  const int nd = (int)h->akv.size();
  int bot, top;
  kind_bcs(h, kind, bot, top);
  // distinct systems of this kind; pressure and w skip ak == 0
  std::vector<int> dmap(nd, -1);
  std::vector<SysDesc> sys;
  std::vector<double> pen;
  const double facvel = 1. / (h->p.xnu * h->p.dt), fact = 1. / (h->p.xkappa * h->p.dt);
  for (int u = 0; u < nd; ++u) {
    double ak = h->akv[u];
    if ((kind == SYS_P || kind == SYS_W) && ak == 0.0) continue;
    double eps;
    if (kind == SYS_P)
      eps = 1. / ak;
    else if (kind == SYS_T)
      eps = 1. / (ak + h->c.bdfv * fact);
    else
      eps = 1. / (ak + h->c.bdfv * facvel);
    SysDesc sd;
    memset(&sd, 0, sizeof sd);
    sd.eps = eps;
    sd.ifbcbot = bot;
    sd.ifbctop = top;
    std::vector<double> pp(6 * ns);
    h_penalty(ns, N, h->p, eps, bot, top, pp.data());
    sd.tau1_bot = pp[4 * ns + 0];
    sd.tau2_top = pp[5 * ns + ns - 1];
    dmap[u] = (int)sys.size();
    sys.push_back(sd);
    pen.insert(pen.end(), pp.begin(), pp.end());
  }
  std::vector<int> colsys(h->ncol);
  for (int c = 0; c < h->ncol; ++c) colsys[c] = dmap[h->col_u[c]];
  const int nsys = (int)sys.size();
  if (build_tasks(h, kind, colsys, 2)) return IW_ERR_NOMEM;
  if (h->nsys_kind[kind] != nsys) {
    cudaFree(h->dab[kind]);
    cudaFree(h->dipiv[kind]);
    cudaFree(h->dinfo[kind]);
    cudaFree(h->dsys[kind]);
    cudaFree(h->dpen[kind]);
    cudaFree(h->dcolsys[kind]);
    h->dab[kind] = 0;
    if (nsys > 0) {
      if (dalloc(h, &h->dab[kind], (size_t)nsys * ldab * n) || dalloc(h, &h->dipiv[kind], (size_t)nsys * n) ||
          dalloc(h, &h->dinfo[kind], (size_t)nsys) || dalloc(h, &h->dsys[kind], (size_t)nsys) ||
          dalloc(h, &h->dpen[kind], (size_t)nsys * 6 * ns))
        return IW_ERR_NOMEM;
    }
    if (dalloc(h, &h->dcolsys[kind], (size_t)h->ncol)) return IW_ERR_NOMEM;
    h->nsys_kind[kind] = nsys;
  }
  if (nsys > 0) {
    CK(cudaMemcpyAsync(h->dsys[kind], sys.data(), nsys * sizeof(SysDesc), cudaMemcpyHostToDevice, h->st));
    CK(cudaMemcpyAsync(h->dpen[kind], pen.data(), pen.size() * sizeof(double), cudaMemcpyHostToDevice, h->st));
  }
  CK(cudaMemcpyAsync(h->dcolsys[kind], colsys.data(), colsys.size() * sizeof(int), cudaMemcpyHostToDevice, h->st));
  if (nsys > 0) {
    FactorArgs fa;
    fa.sys = h->dsys[kind];
    fa.pen = h->dpen[kind];
    fa.ab = h->dab[kind];
    fa.nsys = nsys;
    fa.D = h->dD;
    fa.D2 = h->dD2;
    fa.zh = h->dzh;
    k_assemble_band<<<nsys, 128, 0, h->st>>>(geo(h), fa);
    launch_band_lu(h->st, nsys, n, N, fa.ab, h->dipiv[kind], h->dinfo[kind]);
    CK(launch_error());
    // host copies must stay alive until the copies finish
    CK(cudaStreamSynchronize(h->st));
    std::vector<int> info(nsys);
    CK(scopy(h, info.data(), h->dinfo[kind], nsys * sizeof(int), cudaMemcpyDeviceToHost));
    for (int s = 0; s < nsys; ++s)
      if (info[s] != 0) return set_err(IW_ERR_PIVOT, "zero pivot in band factorisation");
  } else {
    CK(cudaStreamSynchronize(h->st));
  }
  h->fac_bdfv[kind] = h->c.bdfv;
  h->fac_dt[kind] = h->p.dt;
  return 0;
}

// Tables of nsys systems (k_build_systems) for epsilon = 1 / (ak + c0)
static int build_systems(iw_handle* h, const double* dak, int nsys, double c0, int bot, int top, bool fold, int nraw,
                         double* ainv, double* ainv_raw, double* lvec, double* minv, double* pen, SysDesc* sys) {
  if (nsys <= 0) return 0;
  BuildArgs b;
  memset(&b, 0, sizeof b);
  b.N = h->N;
  b.ns = h->ns;
  b.nb = h->nb;
  b.nsys = nsys;
  b.nraw = nraw;
  b.bot = bot;
  b.top = top;
  b.c0 = c0;
  b.facdir = h->p.facdir;
  b.facneumn = h->p.facneumn;
  b.facrobin = h->p.facrobin;
  memcpy(b.bmap, h->bmap, sizeof b.bmap);
  memcpy(b.brep, h->brep, sizeof b.brep);
  b.ak = dak;
  b.D = h->dD;
  b.D2 = h->dD2;
  b.zh = h->dzh;
  b.L = fold ? h->dL : nullptr;
  b.sys = sys;
  b.pen = pen;
  b.ainv = ainv;
  b.ainv_raw = ainv_raw;
  b.lvec = lvec;
  b.minv = minv;
  const size_t sm = build_smem(h->N, h->ns);
  set_smem(k_build_systems, sm);
  k_build_systems<<<nsys, 64 * kBuildGroups, sm, h->st>>>(b);
  CK(launch_error());
  return 0;
}

// cond(I - eps (2/h)^2 D2 + penalty) <~ 1 + eps max_ks (2/h_ks)^2 |D2|_inf
static double cond_slope(const iw_handle* h) {
  const int N = h->N;
  double d2n = 0;
  for (int k1 = 0; k1 < N; ++k1) {
    double rs = 0;
    for (int k = 0; k < N; ++k) rs += std::fabs(h->tab.D2[(size_t)k1 * N + k]);
    d2n = std::max(d2n, rs);
  }
  double hmin = 1e300;
  for (int ks = 0; ks < h->ns; ++ks) hmin = std::min(hmin, h->p.zh[ks]);
  return d2n * (2.0 / hmin) * (2.0 / hmin);
}

// block inverses of one kind.  The systems of a kind are the distinct kx^2+ky^2 whatever
// dt and bdfv are, so their number, the tables' memory, the column map and the tasks
// are made once; a change of dt or bdfv is one kernel in stream order.  Where an allocation
// fails, the handle's sizes, lists and pointers stay those of what it has, and no table counts
// as built, so that the next step builds them.
static int build_blockinv(iw_handle* h, int kind, bool fold) {
  const int ns = h->ns, N = h->N, m = 2 * (ns - 1);
  const int skip = (kind == SYS_P || kind == SYS_W) && h->akv[0] == 0.0 ? 1 : 0;  // no system at k = 0
  const int nsys = (int)h->akv.size() - skip;
  int bot, top;
  kind_bcs(h, kind, bot, top);
  const double facvel = 1. / (h->p.xnu * h->p.dt), fact = 1. / (h->p.xkappa * h->p.dt);
  const double c0 = kind == SYS_P ? 0.0 : kind == SYS_T ? h->c.bdfv * fact : h->c.bdfv * facvel;
  iw_handle::BI& B = h->bi[kind];
  h->bi_dt[kind] = -1;
  if (!B.colsys) {
    const size_t n1 = std::max(nsys, 1), had = h->bytes;
    iw_handle::BI nb;
    char* ai = nullptr;
    std::vector<int> colsys(h->ncol);
    for (int c = 0; c < h->ncol; ++c) colsys[c] = h->col_u[c] - skip;
    // (+16 bytes: k_solve_sys copies whole 16-byte units)
    const int r = dalloc(h, &ai, n1 * h->nb * N * N * sizeof(double) + 16) || dalloc(h, &nb.minv, n1 * std::max(m * m, 1)) ||
                  dalloc(h, &nb.pen, n1 * 6 * ns) || dalloc(h, &nb.sys, n1) || dalloc(h, &nb.lvec, n1 * std::max(m, 1) * N) ||
                  up(h, &nb.colsys, colsys) || build_tasks(h, kind, colsys, kind == SYS_U ? 1 : 2);
    nb.ainv = ai;
    if (r) {
      nb.release();
      h->bytes = had;
      return IW_ERR_NOMEM;
    }
    B = nb;
    h->nrefine[kind] = -1;  // no list of tasks yet
  }
  // tasks [0, last] get a residual sweep: the systems above the condition bound
  const double rho = cond_slope(h);
  int last = -1, nraw = 0;
  const auto& tk = h->htasks[kind];
  for (int t = 0; t < (int)tk.size(); ++t)
    if (tk[t].sys >= 0 && 1.0 + 1. / (h->akv[tk[t].sys + skip] + c0) * rho > kRefineCond) last = t;
  if (fold)
    for (int t = 0; t <= last; ++t) nraw = std::max(nraw, tk[t].sys + 1);
  if (h->nrefine[kind] != last + 1 && build_sys_tasks(h, kind, last + 1)) return IW_ERR_NOMEM;
  if (B.nsys_raw != nraw) {
    cudaFree(B.ainv_raw);
    B.ainv_raw = nullptr;
    B.nsys_raw = 0;
    if (nraw > 0 && dalloc(h, &B.ainv_raw, (size_t)nraw * h->nb * N * N)) return IW_ERR_NOMEM;
    B.nsys_raw = nraw;
  }
  if (int r = build_systems(h, h->dakv + skip, nsys, c0, bot, top, fold, nraw, (double*)B.ainv, B.ainv_raw, B.lvec, B.minv,
                            B.pen, B.sys))
    return r;
  h->bi_bdfv[kind] = h->c.bdfv;
  h->bi_dt[kind] = h->p.dt;
  h->bi_fold[kind] = fold;
  return 0;
}

// cpen: whether the coming solves filter their solutions.  The filter is
// folded into the block inverses only when it runs every step.
static int ensure_factors(iw_handle* h, int cpen) {
  if (h->use_bi) {
    const bool fold = cpen && h->p.ispecfilterexp == 1 && h->p.nspecfilterexp == 1;
    for (int k = SYS_P; k <= SYS_T; ++k)
      if (h->bi_dt[k] != h->p.dt || (k != SYS_P && h->bi_bdfv[k] != h->c.bdfv) || h->bi_dt[k] < 0 ||
          h->bi_fold[k] != fold) {
        int r = build_blockinv(h, k, fold);
        if (r) return r;
      }
  }
  for (int k = 0; k < SYS_KINDS; ++k) {
    if (h->use_bi) continue;
    bool need = h->fac_dt[k] != h->p.dt || (k != SYS_P && h->fac_bdfv[k] != h->c.bdfv);
    if (h->fac_dt[k] < 0) need = true;
    if (need) {
      int r = build_factors(h, k);
      if (r) return r;
    }
  }
  return 0;
}

#endif  // IW_INST

static SolveTabs solve_tabs(iw_handle* h, int kind) {
  SolveTabs tb;
  tb.ab = h->dab[kind];
  tb.ipiv = h->dipiv[kind];
  tb.sys = h->dsys[kind];
  tb.col_sys = h->dcolsys[kind];
  tb.wg = h->dwg;
  tb.alpol = h->dal;
  tb.sigma = h->dsig;
  tb.meang = h->dmeang;
  tb.col_order = h->dcolorder;
  return tb;
}

// ---------------------------------------------------------------------------
// the step
// ---------------------------------------------------------------------------
// operator bucket of the register-column kernels (0: use the tiled kernels)
static int zop_bucket(int N) {
  for (int nm : {9, 17, 21, 25, 29, 33})
    if (N <= nm) return nm;
  return 0;
}

template <typename T, int NM>
static ZOp<T, NM> make_zop(const iw_handle* h) {
  ZOp<T, NM> op;
  memset(&op, 0, sizeof op);
  for (int k1 = 0; k1 < h->N; ++k1)
    for (int k2 = 0; k2 < h->N; ++k2) {
      op.D[k1 * NM + k2] = (T)h->tab.D[(size_t)k1 * h->N + k2];
      op.L[k1 * NM + k2] = h->tab.Lfil[(size_t)k1 * h->N + k2] - (k1 == k2 ? 1.0 : 0.0);
    }
  return op;
}

// CTAs of the persistent tensor-core z kernels: `occ` per SM, W warps each, no more
// than there are tiles of 8 points
static int z_grid(const iw_handle* h, int W, int occ) {
  const int tiles = (int)((h->plane + 7) / 8) * 4 * h->ns;
  return std::min((tiles + W - 1) / W, occ * h->nsm);
}

template <typename T, int NM>
static void launch_stageA_r(iw_handle* h, FieldSet<T>& fs, int proj, T* z3) {
  dim3 grid((unsigned)((h->plane + 127) / 128), (unsigned)h->ns, 4);
  k_stageA_r<T, NM><<<grid, 128, 0, h->st>>>(geo(h), make_zop<T, NM>(h), fs.F[0], fs.F[1], fs.F[2], fs.F[3], fs.F1[0],
                                             fs.F1[1], fs.F1[2], fs.F1[3], fs.Z4[0], fs.Z4[1], fs.Z4[2], z3, proj,
                                             h->derr);
}

template <typename T>
void launch_stageA(iw_handle* h, FieldSet<T>& fs, int proj, int* err) {
  T* z3 = proj < 0 ? fs.Z4[3] : nullptr;  // no step uses d rho / dz (rho is advected in flux form)
  // tensor-core kernel (proj < 0, the derivative alone, exists only there)
  if ((h->tune_a < 0 || proj < 0) && h->N <= kTcMaxN) {
    const size_t sm = (size_t)tc_op_doubles(h->N) * sizeof(double);
    const int blocks = z_grid(h, 16, 2);
#define IW_ATCASE(NT)                                                                                                   \
  case NT:                                                                                                              \
    k_stageA_t<T, NT><<<blocks, 512, sm, h->st>>>(geo(h), fs.F[0], fs.F[1], fs.F[2], fs.F[3], fs.F1[0], fs.F1[1],       \
                                                  fs.F1[2], fs.F1[3], fs.Z4[0], fs.Z4[1], fs.Z4[2], z3, proj,     \
                                                  err);                                                             \
    return;
    switch (tc_nt(h->N)) { IW_ATCASE(2) IW_ATCASE(3) IW_ATCASE(4) IW_ATCASE(5) }
#undef IW_ATCASE
  }
  switch (h->tune_a == 0 ? 0 : zop_bucket(h->N)) {
    case 9: launch_stageA_r<T, 9>(h, fs, proj, z3); return;
    case 17: launch_stageA_r<T, 17>(h, fs, proj, z3); return;
    case 21: launch_stageA_r<T, 21>(h, fs, proj, z3); return;
    case 25: launch_stageA_r<T, 25>(h, fs, proj, z3); return;
    case 29: launch_stageA_r<T, 29>(h, fs, proj, z3); return;
    case 33: launch_stageA_r<T, 33>(h, fs, proj, z3); return;
    default: break;
  }
  dim3 grid((unsigned)((h->nxpp + kTX - 1) / kTX), (unsigned)(h->ny * h->ns), 4);
  size_t smem = (size_t)(h->N * h->N + h->N * kTX) * sizeof(T);
  k_stageA<T><<<grid, kTX * kTW, smem, h->st>>>(geo(h), fs.F[0], fs.F[1], fs.F[2], fs.F[3], fs.F1[0], fs.F1[1],
                                                fs.F1[2], fs.F1[3], fs.Z4[0], fs.Z4[1], fs.Z4[2], z3, proj,
                                                h->derr);
}

// Stage E on the tensor cores: the default where it applies
static bool stageE_is_t(const iw_handle* h) { return (h->tune_e < 0 || h->tune_e >= 2) && h->N <= kTcMaxN; }

// cols: u* to whole-column scratch fields (Y12[0..3]) instead of F; only with stageE_is_t
template <typename T>
void launch_stageE(iw_handle* h, FieldSet<T>& fs, int cols) {
  EArgs<T> a;
  for (int q = 0; q < 4; ++q) {
    a.B[q] = fs.B8[q];
    a.Z[q] = fs.B8[4 + q];
    a.F1[q] = fs.F1[q];
    a.Fn[q] = fs.Fn[q];
    a.Snold[q] = fs.Sn[q];
    a.Snm_w[q] = fs.Snm[q];
    a.Fnm_w[q] = fs.Fnm[q];
    a.F[q] = fs.F[q];
  }
  a.wnl = h->dwnl;
  a.filter = h->p.ispecfilternl == 1;
  if (stageE_is_t(h)) {
    if (cols)
      for (int q = 0; q < 4; ++q) a.F[q] = fs.Y12[q];
    const size_t ops = ((size_t)2 * tc_nc(h->N) * tc_ap(h->N) + 8) * sizeof(double);  // (the warps' tiles follow)
    const int W = (int)std::min<size_t>(sizeof(T) == 4 ? 20 : 16, (226 * 1024 - ops) / ze_buf<T>(h->N));
    const size_t sm = ops + (size_t)W * ze_buf<T>(h->N);
    const int blocks = z_grid(h, W, 1), v16 = (h->plane * sizeof(T)) % 16 == 0;
#define IW_ETCASE(NT)                                                                                        \
  case NT:                                                                                                   \
    set_smem(k_stageE_t<T, NT>, sm);           \
    k_stageE_t<T, NT><<<blocks, 32 * W, sm, h->st>>>(geo(h), a, h->c, cols, v16);                            \
    return;
    switch (tc_nt(h->N)) { IW_ETCASE(2) IW_ETCASE(3) IW_ETCASE(4) IW_ETCASE(5) }
#undef IW_ETCASE
  }
  const dim3 rgrid((unsigned)((h->plane + 127) / 128), (unsigned)h->ns, 4);
  switch (h->tune_e == 1 ? zop_bucket(h->N) : 0) {  // (a launch choice; else, N > 40, tiled)
#define IW_ECASE(NM)                                                                          \
  case NM:                                                                                    \
    k_stageE_r<T, NM><<<rgrid, 128, 0, h->st>>>(geo(h), a, h->c, make_zop<T, NM>(h));         \
    return;
    IW_ECASE(9)
    IW_ECASE(17)
    IW_ECASE(21)
    IW_ECASE(25)
    IW_ECASE(29)
    IW_ECASE(33)
#undef IW_ECASE
    default: break;
  }
  dim3 grid((unsigned)((h->nxpp + kTX - 1) / kTX), (unsigned)(h->ny * h->ns), 4);
  size_t smem = (size_t)h->N * h->N * sizeof(double) + (size_t)(h->N * h->N + 2 * h->N * kTX) * sizeof(T);
  if constexpr (sizeof(T) == 4) {
    k_stageE_f32<<<grid, kTX * kTW, smem, h->st>>>(geo(h), a, h->c);  // at most 39 KB
  } else {
    set_smem(k_stageE<T>, smem);  // > 48 KB from N = 42 on
    k_stageE<T><<<grid, kTX * kTW, smem, h->st>>>(geo(h), a, h->c);
  }
}

// values per lane of a warp transform of length M
static int fft_dpt(int M) {
  const int d = (M + 31) / 32;
  return d <= 4 ? 4 : d <= 8 ? 8 : d <= 16 ? 16 : 32;
}

template <typename T>
static int ystride_of(int ny, int tx) {
  return tx == 16 ? YLay<T, 16>::stride(ny) : tx == 8 ? YLay<T, 8>::stride(ny) : ystride(ny);
}
template <typename T>
static int ytx(const iw_handle* h, bool two) {  // y-FFT tile width
  const size_t cs = 2 * sizeof(T);
  int tx = h->tune_ytx > 0 ? h->tune_ytx : 8;
  if (tx == 8 && h->ny <= 128) tx = 16;  // short columns share warps (y kernels of 64^2 x 68 FP64: 76 -> 63 us)
  while (tx > 2 && (two ? 2 : 1) * (size_t)tx * ystride_of<T>(h->ny, tx) * cs > 110 * 1024) tx /= 2;
  return tx;
}

template <typename T, int TX, bool TWO>
static void launch_y_tx(iw_handle* h, YJobs<T>& jobs, dim3 grid, size_t smem,
                        const typename cplx_t<T>::type* Wy) {
  Geo g = geo(h);
  const bool p2 = (h->ny & (h->ny - 1)) == 0;
  if constexpr (TX == 16) {  // compile-time plans for the common power-of-two lengths
    switch (p2 ? h->ny : 0) {
#define IW_YCT(MC, D)                                                                                        \
  case MC:                                                                                                   \
    set_smem(k_yfft<T, TX, D, true, TWO, MC>, smem); \
    k_yfft<T, TX, D, true, TWO, MC><<<grid, 256, smem, h->st>>>(g, jobs, h->ply, Wy);                    \
    return;
      IW_YCT(64, 8)
      IW_YCT(128, 8)
#undef IW_YCT
      default: break;
    }
  }
  if constexpr (TX == 8) {
    switch (p2 ? h->ny : 0) {
#define IW_YCT(MC, D)                                                                                        \
  case MC:                                                                                                   \
    set_smem(k_yfft<T, TX, D, true, TWO, MC>, smem); \
    k_yfft<T, TX, D, true, TWO, MC><<<grid, 256, smem, h->st>>>(g, jobs, h->ply, Wy);                    \
    return;
      IW_YCT(256, 8)
      IW_YCT(512, 16)
#undef IW_YCT
      default: break;
    }
  }
  switch (fft_dpt(h->ny) * (p2 ? 1 : -1)) {
#define IW_YCASE(D, P)                                                                                       \
  case (P ? D : -D):                                                                                         \
    if constexpr (TX < 16 || D == 4) { /* 16 columns only for ny <= 128 */                                   \
      set_smem(k_yfft<T, TX, D, P, TWO>, smem);                                                              \
      k_yfft<T, TX, D, P, TWO><<<grid, 256, smem, h->st>>>(g, jobs, h->ply, Wy);                    \
    }                                                                                                        \
    break;
    IW_YCASE(4, true)
    IW_YCASE(8, true)
    IW_YCASE(16, true)
    IW_YCASE(32, true)
    IW_YCASE(4, false)
    IW_YCASE(8, false)
    IW_YCASE(16, false)
    IW_YCASE(32, false)
#undef IW_YCASE
  }
}

template <typename T>
void launch_y(iw_handle* h, FieldSet<T>& fs, YJobs<T>& jobs, int njobs, int nplanes, bool four) {
  typedef typename cplx_t<T>::type C;
  if (h->ny == 1) {
    const size_t nc = h->plane * (size_t)nplanes / 2;
    k_y1<T><<<dim3((unsigned)((nc + 255) / 256), (unsigned)njobs), 256, 0, h->st>>>(jobs, nc);
    return;
  }
  int tx = ytx<T>(h, four);
  // FP32 columns of 16 or 32 rows in fewer tiles of 16 columns than SMs (one field of few planes, as in iw_postp): tiles of
  // 4, a warp per column (iw_postp, 16 / 4 columns: 16 x 16 x 9 397 / 383 us, 32 x 32 x 18 484 / 448, 64 x 32 x 36 566 / 557;
  // 180 tiles gain nothing, FP64 and 64 rows lose: 16 x 16 x 9 384 / 405, 16 x 64 x 18 601 / 649).  Same bits.
  if (sizeof(T) == 4 && tx == 16 && (h->ny == 16 || h->ny == 32) && (h->nxhp + 15) / 16 * nplanes * njobs < h->nsm) tx = 4;
  const int ntile = (h->nxhp + tx - 1) / tx;
  dim3 grid(ntile, nplanes, njobs);
  const size_t smem = (four ? 2 : 1) * (size_t)tx * ystride_of<T>(h->ny, tx) * sizeof(C);
  switch (four ? -tx : tx) {
#define IW_YTX(TX)                                                                        \
  case TX: launch_y_tx<T, TX, false>(h, jobs, grid, smem, fs.Wy); break;         \
  case -TX: launch_y_tx<T, TX, true>(h, jobs, grid, smem, fs.Wy); break;
    IW_YTX(16)
    IW_YTX(8)
    IW_YTX(4)
    IW_YTX(2)  // (two columns of ny <= 1024 always fit)
#undef IW_YTX
  }
}

#define DISPATCH_N(h, FN, ...)                    \
  do {                                            \
    if ((h)->N <= 16)                             \
      FN<T, 16>(__VA_ARGS__);                     \
    else if ((h)->N <= 24)                        \
      FN<T, 24>(__VA_ARGS__);                     \
    else if ((h)->N <= 32)                        \
      FN<T, 32>(__VA_ARGS__);                     \
    else                                          \
      FN<T, 48>(__VA_ARGS__);                     \
  } while (0)

// History rotation by pointer swap (solver.f:447-478): the buffer written
// with S (level n) becomes Sn, the one written with F2 becomes Fn.  The
// arrangement repeats every 2 steps.
template <typename T>
static void rotate_levels(FieldSet<T>& fs) {
  for (int q = 0; q < 4; ++q) {
    std::swap(fs.Sn[q], fs.Snm[q]);
    std::swap(fs.Fn[q], fs.Fnm[q]);
  }
}

// convec (solver.f:6-514).  proj=1 also applies the maxcalc round trip that
// precedes it in the main loop (main.f:657).
template <typename T>
static int anim_dump(iw_handle* h, FieldSet<T>& fs);
template <typename T>
static int legspec_dump(iw_handle* h, FieldSet<T>& fs);
template <typename T>
static int postp_step(iw_handle* h, FieldSet<T>& fs);

// lengths nx / 2 with a kernel of their own (k_xrow_reg)
static bool xrow_reg_length(int M) {
  for (int nb : {8, 16, 32})
    for (int r0 : {2, 4, 6, 8, 10})
      if (M == r0 * nb && (nb == 8 || r0 >= 6)) return true;
  return false;
}
// K_C for the lengths of k_xrow_reg; false for any other
template <typename T>
static bool launch_xrow_reg(iw_handle* h, FieldSet<T>& fs, const NLArgs<T>& a) {
  switch (h->nx / 2) {
#define IW_XREG(R0, NB)                                                                                          \
  case R0 * NB: {                                                                                                \
    typedef XReg<T, R0, NB> X;                                                                                   \
    set_smem(k_xrow_reg<T, R0, NB>, X::smem);     \
    k_xrow_reg<T, R0, NB><<<dim3((h->ny + X::YR - 1) / X::YR, h->nz), X::threads, X::smem, h->st>>>(geo(h), a, fs.Wm, \
                                                                                                    fs.Wn);      \
    return true;                                                                                                 \
  }
    IW_XREG(2, 8)
    IW_XREG(4, 8)
    IW_XREG(6, 8)
    IW_XREG(8, 8)
    IW_XREG(10, 8)
    IW_XREG(6, 16)
    IW_XREG(8, 16)
    IW_XREG(10, 16)
    IW_XREG(6, 32)
    IW_XREG(8, 32)
    IW_XREG(10, 32)
#undef IW_XREG
    default: return false;
  }
}

// K_C: x rows; of the other lengths one CTA per (y, z) row (k_xrow_nl) with 256 threads, or
// 128 (short rows, or when the autotuner measured that faster, tune_xthr)
template <typename T>
void launch_xrow(iw_handle* h, FieldSet<T>& fs) {
  typedef typename cplx_t<T>::type C;
  Geo g = geo(h);
  const int M = h->nx / 2;
  // short rows: fewer warps, each with several rows (rows of 32..128 values fill a warp only together)
  const int xthr = h->tune_xthr > 0 ? h->tune_xthr : M <= 128 ? 128 : 256;
  {
    NLArgs<T> a;
    memset(&a, 0, sizeof a);
    for (int q = 0; q < 10; ++q) a.in[q] = fs.Y12[q];  // u v w t | dy u v w | dz u v w
    for (int q = 0; q < 11; ++q) a.out[q] = fs.X11[q];
    const double bz = h->p.brunt;
    const double rg = -(h->p.rho0 * (bz * bz) / h->p.grav);
    a.coef_buoy = (bz * bz) / rg;
    a.rg = rg;
    const double omega = 2. / (double)((h->N + 1) * (h->N + 2));
    for (int ks = 0; ks < h->ns; ++ks) a.tau_pen[ks] = 0.5 / omega * (2. / h->p.zh[ks]);
    a.forcing = h->p.forcing;
    if (h->p.forcing) {
      double pi2 = 8. * std::atan(1.0);
      double xk = pi2 / h->p.xlen, xm = pi2 / (2. * h->p.zlen);
      double om = (h->p.brunt * xk) / std::sqrt(xk * xk + xm * xm);
      double zdim = h->p.xlen, um = h->p.umax, xa = h->p.xacrit;
      double ph = (h->t <= h->p.fwave * (pi2 / om)) ? 1.0 : 0.0;
      a.f_xk = xk;
      a.f_xm = xm;
      a.f_om = om;
      a.f_t = h->t;
      a.f_amp_u = -(1 / xk) * (xa * um) * xm * um / zdim * ph;
      a.f_amp_w = (xa * um) * (um / zdim) * ph;
      a.f_amp_r = (xa * um) * (-(1 / om)) * bz * bz * (h->p.rho0 / h->p.grav) * (um / zdim) * ph;
    }
    a.dx = (pi2_of(h) / (pi2_of(h) / h->p.xlen)) / h->nx;
    if (launch_xrow_reg<T>(h, fs, a)) return;
    const size_t smem = 17 * (size_t)xstride(M) * sizeof(C);
    dim3 grid(h->ny, h->nz);
    const bool p2 = (M & (M - 1)) == 0;
    switch (M) {  // compile-time plan
#define IW_XCT(MC, D)                                                                                       \
  case MC:                                                                                                  \
    set_smem(k_xrow_nl<T, D, true, MC>, smem); \
    k_xrow_nl<T, D, true, MC><<<grid, xthr, smem, h->st>>>(g, a, h->plx, fs.Wm, fs.Wn);                     \
    goto xrow_done;
      IW_XCT(512, 16)
#undef IW_XCT
      default: break;
    }
    switch (fft_dpt(M) * (p2 ? 1 : -1)) {
#define IW_XCASE(D, P)                                                                                   \
  case (P ? D : -D):                                                                                     \
    set_smem(k_xrow_nl<T, D, P>, smem);   \
    k_xrow_nl<T, D, P><<<grid, xthr, smem, h->st>>>(g, a, h->plx, fs.Wm, fs.Wn);                        \
    break;
        IW_XCASE(4, true)
        IW_XCASE(8, true)
      IW_XCASE(16, true)
      IW_XCASE(32, true)
        IW_XCASE(4, false)
        IW_XCASE(8, false)
      IW_XCASE(16, false)
      IW_XCASE(32, false)
#undef IW_XCASE
    }
  xrow_done:;
  }
}

// k_xrow_stats over n entries, nblk CTAs each
template <typename T>
void launch_xstats(iw_handle* h, FieldSet<T>& fs, const StatRows<T>& a, int n, int nblk) {
  typedef typename cplx_t<T>::type C;
  const int M = h->nx / 2;
  const size_t smem = (size_t)(kStatThreads / 32) * 2 * xstride(M) * sizeof(C);
  const dim3 grid((unsigned)nblk, (unsigned)n);
  const Geo g = geo(h);
  const bool p2 = (M & (M - 1)) == 0;
  switch (p2 && M >= 32 && M <= 512 ? M : 0) {  // compile-time plans for power-of-two lengths
#define IW_SCT(MC, D)                                                                                            \
  case MC:                                                                                                       \
    set_smem(k_xrow_stats<T, D, true, MC>, smem);  \
    k_xrow_stats<T, D, true, MC><<<grid, kStatThreads, smem, h->st>>>(g, a, h->plx, fs.Wm, fs.Wn, h->dpart);     \
    return;
    IW_SCT(32, 8)
    IW_SCT(64, 8)
    IW_SCT(128, 8)
    IW_SCT(256, 8)
    IW_SCT(512, 16)
#undef IW_SCT
    default: break;
  }
  switch (fft_dpt(M) * (p2 ? 1 : -1)) {
#define IW_SCASE(D, P)                                                                                       \
  case (P ? D : -D):                                                                                         \
    set_smem(k_xrow_stats<T, D, P>, smem);     \
    k_xrow_stats<T, D, P><<<grid, kStatThreads, smem, h->st>>>(g, a, h->plx, fs.Wm, fs.Wn, h->dpart);        \
    break;
    IW_SCASE(4, true)
    IW_SCASE(8, true)
    IW_SCASE(16, true)
    IW_SCASE(32, true)
    IW_SCASE(4, false)
    IW_SCASE(8, false)
    IW_SCASE(16, false)
    IW_SCASE(32, false)
#undef IW_SCASE
  }
}

#ifndef IW_INST
template <typename T>
static int convec_impl(iw_handle* h, FieldSet<T>& fs, int proj, int cols = 0) {
  typedef typename cplx_t<T>::type C;
  Geo g = geo(h);
  const int M = h->nx / 2;
  mark(h, -1);
  // K_A
  launch_stageA<T>(h, fs, proj, h->derr);
  mark(h, 0);
  if (h->anim_pending) {  // the dump sees the fields convec sees: projected, mean w removed
    h->anim_pending = false;
    int r = anim_dump<T>(h, fs);
    if (r) return r;
  }
  // wall pressure BC term (before the histories rotate): a few columns' latency, beside the
  // transforms, which it shares no output with; stage E overwrites its inputs and waits
  auto wall_term = [&](cudaStream_t st) {
    const dim3 wgrid((unsigned)((h->nxhp + 31) / 32), (unsigned)h->ny, 2);
    k_wviscrot<T><<<wgrid, 192, 0, st>>>(g, fs.F1[0], fs.F1[1], fs.F1[2], fs.Fn[0], fs.Fn[1], fs.Fn[2], fs.Fnm[0],
                                         fs.Fnm[1], fs.Fnm[2], h->c, h->p.xnu, h->dwvr);
  };
  if (!h->prof) wall_term(side_fork(h));
  // K_B: y-inverse of 10 arrays (rho is advected in flux form: none of its derivatives are needed)
  {
    YJobs<T> jb;
    memset(&jb, 0, sizeof jb);
    for (int q = 0; q < 4; ++q) jb.j[q] = YJob<T>{fs.F1[q], nullptr, fs.Y12[q], 0};
    for (int q = 0; q < 3; ++q) {
      jb.j[4 + q] = YJob<T>{fs.F1[q], nullptr, fs.Y12[4 + q], 1};
      jb.j[7 + q] = YJob<T>{fs.Z4[q], nullptr, fs.Y12[7 + q], 0};
    }
    launch_y<T>(h, fs, jb, 10, h->nz, false);
  }
  mark(h, 1);
  // K_C
  launch_xrow<T>(h, fs);
  mark(h, 2);
  // K_D: y-forward; B_q = Y(A_q) + i ky Y(P_q), Z_q = Y(P_zq)
  {
    YJobs<T> jb;
    memset(&jb, 0, sizeof jb);
    // X11: Au Av Aw At | uv vv vw vt | uw ww wt ;  B8: Bu Bv Bw Bt | Zu Zv Zw Zt
    for (int q = 0; q < 4; ++q) jb.j[q] = YJob<T>{fs.X11[q], fs.X11[4 + q], fs.B8[q], 3};
    launch_y<T>(h, fs, jb, 4, h->nz, true);
    YJobs<T> jz;
    memset(&jz, 0, sizeof jz);
    jz.j[0] = YJob<T>{fs.X11[8], nullptr, fs.B8[4], 2};   // uw
    jz.j[1] = YJob<T>{fs.X11[6], nullptr, fs.B8[5], 2};   // vw
    jz.j[2] = YJob<T>{fs.X11[9], nullptr, fs.B8[6], 2};   // ww
    jz.j[3] = YJob<T>{fs.X11[10], nullptr, fs.B8[7], 2};  // wt
    launch_y<T>(h, fs, jz, 4, h->nz, false);
  }
  mark(h, 3);
  if (h->prof)  // a phase of its own
    wall_term(h->st);
  else
    side_join(h);
  mark(h, 4);
  // K_E
  launch_stageE<T>(h, fs, cols);
  mark(h, 5);
  rotate_levels(fs);
  return 0;
}

// main.f:741,832: the step after a change of dt (idtstep = 1) still has the
// old step in its history
static bool dt_adapting(const iw_handle* h) { return h->ivardt == 1 && h->idtstep < 2; }

static void set_var_fac_bdf(iw_handle* h) {  // two steps of dt, then one of cdt*dt
  const double d1 = h->p.dt, d2 = h->p.dt, d3 = h->cdt * h->p.dt;
  h->c.fac1 = abvar1_(&d1, &d2, &d3);
  h->c.fac2 = abvar2_(&d1, &d2, &d3);
  h->c.fac3 = abvar3_(&d1, &d2, &d3);
  h->c.bdf1 = bdfvar1_(&d1, &d2, &d3);
  h->c.bdf2 = bdfvar2_(&d1, &d2, &d3);
  h->c.bdf3 = bdfvar3_(&d1, &d2, &d3);
}

static void set_var_bdfv(iw_handle* h) {
  const double d1 = h->p.dt, d2 = h->p.dt, d3 = h->cdt * h->p.dt;
  h->c.bdfv = bdfvarv_(&d1, &d2, &d3);
}

// coefficient schedule for the next step (main.f:700-777): SS2/BDF2 after the
// first step of a new run, the variable-step form after the first step of a
// restarted one (istart = 1) and after a change of dt, SS3/BDF3 otherwise
static void schedule_after_convec(iw_handle* h) {
  if (h->istep < 2) {
    if (h->istart == 0) {
      h->c.fac1 = 2.;
      h->c.fac2 = -1.;
      h->c.fac3 = 0.;
      h->c.bdf1 = 2.;
      h->c.bdf2 = -0.5;
      h->c.bdf3 = 0.;
    } else {
      set_var_fac_bdf(h);
    }
  } else if (!dt_adapting(h)) {
    h->c.fac1 = 3.;
    h->c.fac2 = -3.;
    h->c.fac3 = 1.;
    h->c.bdf1 = 3.;
    h->c.bdf2 = -1.5;
    h->c.bdf3 = 1. / 3.;
  } else {
    set_var_fac_bdf(h);
  }
}

// bdfv for the next step's Helmholtz operators (main.f:815-855).  A change of
// dt ends in the step that made it (idtstep = 1 there): cdt = 1, ivardt = 0.
// The first step of a restarted run leaves both as they are.
static void schedule_after_calcuvwt(iw_handle* h) {
  if (h->istep < 2) {
    if (h->istart == 0)
      h->c.bdfv = 1.5;
    else
      set_var_bdfv(h);
  } else if (!dt_adapting(h)) {
    h->c.bdfv = 11. / 6.;
  } else {
    set_var_bdfv(h);
    h->cdt = 1.;
    h->ivardt = 0;
  }
}

template <typename T>
static int step_cfl(iw_handle* h, FieldSet<T>& fs, double* cflx, double* cflz);

// The adaptive rule of maxcalc (various.f:892-982) at the start of a step.
// The CFL numbers (two inverse transforms, a reduction and a read-back) are
// only needed once more than 20 steps of the current dt lie behind t; before
// that the rule cannot change dt.  A change sets the step's variable-step
// coefficients (the history holds one step of the new dt and two of the old)
// and, through dt and bdfv, new Helmholtz operators.
template <typename T>
static int adapt_dt(iw_handle* h, FieldSet<T>& fs) {
  if (!(std::trunc(h->t / h->p.dt) > 20.0)) return IW_OK;
  double cflx = 0, cflz = 0;
  int r = step_cfl<T>(h, fs, &cflx, &cflz);
  if (r) return r;
  double dtn = 0, cdt = 0;
  if (!iw_dt_rule(cflx, cflz, h->t, h->p.dt, h->xomega, &dtn, &cdt)) return IW_OK;
  h->p.dt = dtn;
  h->cdt = cdt;
  const double d1 = dtn, d2 = cdt * dtn, d3 = cdt * dtn;
  h->c = Coefs{abvar1_(&d1, &d2, &d3),  abvar2_(&d1, &d2, &d3),  abvar3_(&d1, &d2, &d3),  bdfvar1_(&d1, &d2, &d3),
               bdfvar2_(&d1, &d2, &d3), bdfvar3_(&d1, &d2, &d3), bdfvarv_(&d1, &d2, &d3), dtn};
  h->ivardt = 1;
  h->idtstep = 0;
  return IW_OK;
}

#endif  // IW_INST

// The solve variant a role resolves to (IW_LAUNCH_SOLVE values): its own
// choice or the handle's, where the variant applies; 0 where no grouped kernel
// does (more rows than threads, tables too large for shared memory, a filter
// that is not folded into the inverses).
static int role_kind(int role) { return role == 0 ? SYS_U : role == 1 ? SYS_W : role == 2 ? SYS_T : SYS_P; }
template <typename T>
static int solve_variant(const iw_handle* h, int role, int cpen) {
  int us = h->sys_role[role] >= 0 ? h->sys_role[role] : h->use_sys;
  const bool fold = h->bi_fold[role_kind(role)] && cpen;
  if (!us || h->nz > kSysMaxRows || (cpen && !fold)) return 0;
  // variant 3 (two rows per thread) exists for u/v, w and rho when a subdomain's
  // row pairs fit one CTA; otherwise the one-row grouped kernel takes its place
  if (us == 3 && (role == 3 || (h->ns * ((h->N + 1) / 2) + 31) / 32 * 32 > kSys2MaxThreads)) us = 1;
  const size_t lim = 200 * 1024;
  if (us == 2 && (h->N > kTcMaxN || tc_smem<T>(h->nz, h->N, h->ns, h->nb, role == 3).total > lim)) us = 1;
  if (us != 2 && sys_smem(h->nz, h->N, h->ns, h->nb, role == 3).total * sizeof(double) > lim) us = 0;
  return us;
}

static double role_rdiv(const iw_handle* h, int role) {
  return role == 2 ? h->p.dt * h->p.xkappa : h->p.xnu * h->p.dt;
}
// w whose only task without k_solve_tc is the (0,0) column (no system, w = 0):
// the kernel writes that column itself
static bool tc_zero00(const iw_handle* h, int role) {
  const int kind = role_kind(role);
  return role == 1 && h->nrefine[kind] == 0 && h->nold[kind] == 1 && h->htasks[kind][0].sys < 0 &&
         h->htasks[kind][0].first == 0 && h->htasks[kind][0].count == 1;
}

// k_solve_tc over nblk tasks of the jobs
template <typename T>
static void launch_jobs_tc(iw_handle* h, const TcJobs<T>& jobs, int nblk, const int* order) {
  const Geo g = geo(h);
  const size_t smem = tc_smem<T>(h->nz, h->N, h->ns, h->nb, false).total;
#define IW_TC_CASE(NT)                                                                               \
  case NT:                                                                                           \
    set_smem(k_solve_tc<T, NT>, smem); \
    k_solve_tc<T, NT><<<nblk, 32 * h->ns, smem, h->st>>>(g, jobs, order, h->dmeang);                 \
    break;
  switch (tc_nt(h->N)) { IW_TC_CASE(2) IW_TC_CASE(3) IW_TC_CASE(4) IW_TC_CASE(5) }
#undef IW_TC_CASE
}

// k_helm_tc over ntask tasks
template <typename T>
void launch_helm_tc(iw_handle* h, const HelmTc& H, int ntask) {
  const size_t smem = helm_smem(h->nz, h->N, h->ns, h->nb).total;
  const Geo g = geo(h);
  const dim3 grid((unsigned)ntask, 2);
#define IW_HT_CASE(NT)                                                                              \
  case NT:                                                                                          \
    set_smem(k_helm_tc<NT>, smem);    \
    k_helm_tc<NT><<<grid, 32 * h->ns, smem, h->st>>>(g, H);                                         \
    break;
  switch (tc_nt(h->N)) { IW_HT_CASE(2) IW_HT_CASE(3) IW_HT_CASE(4) IW_HT_CASE(5) }
#undef IW_HT_CASE
}

// The system-grouped tensor-core solves of the listed roles (0..2: one launch
// for all of them; 3: the pressure).  The row tiles of 8 are fixed at compile
// time; one warp per subdomain.
template <typename T>
void launch_solve_tc(iw_handle* h, FieldSet<T>& fs, const int* roles, int nroles, int kstart, int cols) {
  const Geo g = geo(h);
  const int nt = tc_nt(h->N);
  const size_t smem = tc_smem<T>(h->nz, h->N, h->ns, h->nb, roles[0] == 3).total;
  T* const* S = cols ? fs.Y12 : fs.F;  // where stage E left u*, v*, w*, rho*
  if (roles[0] == 3) {
    if (h->ntask2[SYS_P] <= 0) return;
    const auto& B = h->bi[SYS_P];
    BlockInv bi;
    memset(&bi, 0, sizeof bi);
    bi.ainv = B.ainv;
    bi.lvec = B.lvec;
    bi.minv = B.minv;
    bi.sys = B.sys;
    bi.nb = h->nb;
    memcpy(bi.bmap, h->bmap, sizeof bi.bmap);
    const dim3 grid((unsigned)h->ntask2[SYS_P], 2);
#define IW_TC_CASE(NT)                                                                                             \
  case NT:                                                                                                         \
    set_smem(k_press_tc<T, NT>, smem);               \
    k_press_tc<T, NT><<<grid, 32 * h->ns, smem, h->st>>>(g, bi, h->dtasks2[SYS_P], h->dcolorder, S[0], S[1], S[2], \
                                                         h->dDt, h->dwnl, h->dwvr, kstart, cols);                  \
    break;
    switch (nt) { IW_TC_CASE(2) IW_TC_CASE(3) IW_TC_CASE(4) IW_TC_CASE(5) }
#undef IW_TC_CASE
    return;
  }
  TcJobs<T> jobs;
  memset(&jobs, 0, sizeof jobs);
  jobs.nb = h->nb;
  jobs.cols = cols;
  memcpy(jobs.bmap, h->bmap, sizeof jobs.bmap);
  int nblk = 0;
  for (int i = 0; i < nroles; ++i) {
    const int role = roles[i], kind = role_kind(role);
    if (h->ntask2[kind] <= 0) continue;
    const auto& B = h->bi[kind];
    TcJob<T>& j = jobs.j[jobs.n++];
    j.ainv = (const double*)B.ainv;
    j.lvec = B.lvec;
    j.minv = B.minv;
    j.sys = B.sys;
    j.tasks = h->dtasks2[kind];
    j.first = nblk;
    j.per = role == 0 ? 4 : 2;
    j.zero00 = tc_zero00(h, role);
    j.meanu = role == 0 ? h->p.meanu_damping : 0;
    j.rdiv = role_rdiv(h, role);
    j.irdiv = 1.0 / j.rdiv;
    j.F0 = fs.F[role == 0 ? 0 : role + 1];
    j.F1 = fs.F[1];
    j.S0 = S[role == 0 ? 0 : role + 1];
    j.S1 = S[1];
    nblk += h->ntask2[kind];
  }
  if (nblk > 0) launch_jobs_tc<T>(h, jobs, nblk, h->dcolorder);
}

template <typename T>
void launch_solve_bi(iw_handle* h, FieldSet<T>& fs, int role, int cpen, int kstart, int cols, bool tc_done) {
  constexpr int R = 4;
  const int kind = role_kind(role);
  BlockInv bi;
  bi.ainv = h->bi[kind].ainv;
  bi.minv = h->bi[kind].minv;
  bi.pen = h->bi[kind].pen;
  bi.sys = h->bi[kind].sys;
  bi.col_sys = h->bi[kind].colsys;
  bi.col_order = h->dcolorder;
  bi.lvec = h->bi[kind].lvec;
  bi.nb = h->nb;
  memcpy(bi.bmap, h->bmap, sizeof bi.bmap);
  const int mm = std::max(2 * (h->ns - 1), 1);
  // the pressure keeps its u*, v*, w* columns in shared memory as well
  const size_t sm = ((size_t)2 * R * h->nz + 2 * R * mm) * sizeof(double) +
                    (role == 3 ? (size_t)3 * R * h->nz * sizeof(T) : 0);
  T *F0, *F1 = nullptr, *F2 = nullptr;
  T* const* S = cols ? fs.Y12 : fs.F;  // where stage E left u*, v*, w*, rho*
  if (role == 3) {
    F0 = S[0];
    F1 = S[1];
    F2 = S[2];
  } else if (role == 0) {
    F0 = fs.F[0];
    F1 = fs.F[1];
  } else {
    F0 = role == 1 ? fs.F[2] : fs.F[3];
  }
  const double rd = role_rdiv(h, role);
  const int meanu = role == 0 ? h->p.meanu_damping : 0;
  if (sm > 48 * 1024) set_smem(k_solve_cta<T, R>, sm);
  // refined prefix, then the rest
  // With the filter folded into ainv, the refined prefix uses the unfiltered
  // copy and the filter pass; the rest needs no filter pass.
  const int nref = h->nrefine[kind], nt = h->ntask[kind];
  const bool fold = h->bi_fold[kind] && cpen;
  // a grouped kernel for the tasks after the prefix, when one applies
  const int us = solve_variant<T>(h, role, cpen);
  const bool tc = us == 2;
  int nend = us ? std::max(h->nold[kind], nref) : nt;
  if (tc && tc_zero00(h, role) && h->ntask2[kind] > 0) nend = 0;
  // the refined columns (a few long chains) beside the others, which they share nothing with
  const bool beside = tc && !tc_done && nend > 0;
  const cudaStream_t st = beside ? side_fork(h) : h->st;
  auto main_part = [&]() {
    if (tc && !tc_done) launch_solve_tc<T>(h, fs, &role, 1, kstart, cols);
  };
  if (!beside || h->prof) main_part();
  if (us && !tc && h->ntask2[kind] > 0) {
    const size_t smsys = sys_smem(h->nz, h->N, h->ns, h->nb, role == 3).total * sizeof(double);
    const int nthr = (h->nz + 31) / 32 * 32, nthr2 = (h->ns * ((h->N + 1) / 2) + 31) / 32 * 32;
    Geo g = geo(h);
    const double* mg = h->dmeang;
    if (us == 3) {
#define IW_SYS2_LAUNCH(RL)                                                                                   \
  do {                                                                                                       \
    set_smem(k_solve_sys2<T, RL>, smsys);      \
    k_solve_sys2<T, RL><<<h->ntask2[kind], nthr2, smsys, h->st>>>(g, bi, h->dtasks2[kind], h->dcolorder, F0, \
                                                                  F1, rd, meanu, mg, h->derr);              \
  } while (0)
      if (role == 0)
        IW_SYS2_LAUNCH(0);
      else if (role == 1)
        IW_SYS2_LAUNCH(1);
      else
        IW_SYS2_LAUNCH(2);
#undef IW_SYS2_LAUNCH
    } else {
#define IW_SYS_LAUNCH(RL)                                                                                           \
  do {                                                                                                              \
    set_smem(k_solve_sys<T, RL>, smsys);              \
    k_solve_sys<T, RL><<<h->ntask2[kind], nthr, smsys, h->st>>>(g, bi, h->dtasks2[kind], h->dcolorder, F0, F1, F2, \
                                                                rd, meanu, mg, h->dDt, h->dwnl, h->dwvr, kstart,   \
                                                                h->derr);                                          \
  } while (0)
      if (role == 0)
        IW_SYS_LAUNCH(0);
      else if (role == 1)
        IW_SYS_LAUNCH(1);
      else if (role == 2)
        IW_SYS_LAUNCH(2);
      else
        IW_SYS_LAUNCH(3);
#undef IW_SYS_LAUNCH
    }
  }
  for (int part = 0; part < 2; ++part) {
    const int t0 = part == 0 ? 0 : nref, cnt = part == 0 ? nref : nend - nref;
    if (cnt <= 0) continue;
    BlockInv b2 = bi;
    int cp = cpen;
    if (fold) {
      if (part == 0)
        b2.ainv = h->bi[kind].ainv_raw;
      else
        cp = 0;
    }
    k_solve_cta<T, R><<<cnt, kSolveThreads, sm, st>>>(geo(h), b2, solve_tabs(h, kind), h->dtasks[kind] + t0, F0, F1,
                                                          F2, S[role == 0 || role == 3 ? 0 : role + 1], S[1], cols, rd, role, cp, meanu, part == 0 ? 1 : 0, h->dDt, h->dD2t,
                                                          h->dLt, h->dzh, h->dwnl, h->dwvr, kstart);
  }
  if (beside && !h->prof) {
    main_part();
    side_join(h);
  }
}

// The kernels that these launch are compiled in translation units of their own
// (iw_inst.cu, once per storage type and group), all at the same time.
#define IW_INST_FFT(X, T)                                                       \
  X template void launch_y<T>(iw_handle*, FieldSet<T>&, YJobs<T>&, int, int, bool); \
  X template void launch_xrow<T>(iw_handle*, FieldSet<T>&);                    \
  X template void launch_xstats<T>(iw_handle*, FieldSet<T>&, const StatRows<T>&, int, int);
#define IW_INST_Z(X, T)                                                             \
  X template void launch_stageA<T>(iw_handle*, FieldSet<T>&, int, int*);            \
  X template void launch_stageE<T>(iw_handle*, FieldSet<T>&, int);                  \
  X template void launch_solve_tc<T>(iw_handle*, FieldSet<T>&, const int*, int, int, int); \
  X template void launch_solve_bi<T>(iw_handle*, FieldSet<T>&, int, int, int, int, bool);
#if defined(IW_INST)
#if IW_INST == 1
IW_INST_FFT(, float)
#elif IW_INST == 2
IW_INST_FFT(, double)
#elif IW_INST == 3
IW_INST_Z(, float)
#else
IW_INST_Z(, double)
template void launch_helm_tc<double>(iw_handle*, const HelmTc&, int);
#endif
#else
extern template void launch_helm_tc<double>(iw_handle*, const HelmTc&, int);
IW_INST_FFT(extern, float)
IW_INST_FFT(extern, double)
IW_INST_Z(extern, float)
IW_INST_Z(extern, double)

// calcuvwt (calcuvwt_noslip.f / calcuvwt.f) on u*,v*,w*,rho* held in F.
template <typename T>
static int calcuvwt_impl(iw_handle* h, FieldSet<T>& fs, int cpen, int cols = 0) {
  Geo g = geo(h);
  // a warp's right-hand sides (k_visc 4 columns of nz, k_press_g as many): four warps share a CTA while they fit in
  // shared memory, two above nz = 1816 (nz <= 64 x 48)
  const int warps = (size_t)4 * 4 * h->nz * sizeof(double) <= 227 * 1024 ? 4 : 2;
  const unsigned nblk = (unsigned)((h->ncol + warps - 1) / warps);
  const size_t smem = (size_t)warps * 4 * h->nz * sizeof(double);
  const int kstart = h->p.bc_variant == IW_BC_NOSLIP ? 1 : 0;
  set_smem(k_visc<T>, smem);
  if (h->use_bi) {
    launch_solve_bi<T>(h, fs, 3, cpen, kstart, cols, false);
  } else {
  {
    constexpr int G = 2;
    const int wpb = warps;
    const size_t smp = (size_t)wpb * 2 * G * h->nz * sizeof(double);
    set_smem(k_press_g<T, G>, smp);
    k_press_g<T, G><<<(h->ntask[SYS_P] + wpb - 1) / wpb, 32 * wpb, smp, h->st>>>(
        g, solve_tabs(h, SYS_P), h->dtasks[SYS_P], h->ntask[SYS_P], fs.F[0], fs.F[1], fs.F[2], h->dwnl, h->dwvr, cpen,
        kstart);
  }
  }
  mark(h, 6);
  const double xnudt = h->p.xnu * h->p.dt, dtk = h->p.dt * h->p.xkappa;
  if (h->use_bi) {
    // one launch for all roles on the tensor-core kernel (separate ones while
    // the phases are timed)
    int tcr[3], ntc = 0;
    for (int role = 0; role < 3 && !h->prof; ++role)
      if (solve_variant<T>(h, role, cpen) == 2) tcr[ntc++] = role;
    if (ntc > 0) launch_solve_tc<T>(h, fs, tcr, ntc, kstart, cols);
    for (int role = 0; role < 3; ++role) {
      launch_solve_bi<T>(h, fs, role, cpen, kstart, cols, !h->prof);
      mark(h, 7 + role);
    }
  } else {
    k_visc<T><<<nblk, 32 * warps, smem, h->st>>>(g, solve_tabs(h, SYS_U), fs.F[0], fs.F[1], xnudt, 0, cpen,
                                                  h->p.meanu_damping);
    mark(h, 7);
    k_visc<T><<<nblk, 32 * warps, smem, h->st>>>(g, solve_tabs(h, SYS_W), fs.F[2], fs.F[2], xnudt, 1, cpen, 0);
    mark(h, 8);
    k_visc<T><<<nblk, 32 * warps, smem, h->st>>>(g, solve_tabs(h, SYS_T), fs.F[3], fs.F[3], dtk, 2, cpen, 0);
    mark(h, 9);
  }
  return 0;
}

template <typename T>
static int iface_avg(iw_handle* h, FieldSet<T>& fs, bool count, int nf = 4) {
  typedef typename cplx_t<T>::type C;
  Geo g = geo(h);
  const dim3 pgrid((unsigned)((h->ny + 127) / 128), (unsigned)h->nz, (unsigned)nf);
  if (h->ns < 2) {
    k_project_planes<T><<<pgrid, 128, 0, h->st>>>(g, fs.F[0], fs.F[1], fs.F[2], fs.F[3], 0);
    return 0;
  }
  const int ng = nf * (h->ns - 1);  // plane groups (field, interface)
  const dim3 ggrid((unsigned)((h->plane + 255) / 256), (unsigned)(ng * 4));  // 4 planes per group
  k_iface_gather<T><<<ggrid, 256, 0, h->st>>>(g, fs.F[0], fs.F[1], fs.F[2], fs.F[3], fs.G, 0);
  {
    YJobs<T> jb;
    memset(&jb, 0, sizeof jb);
    jb.j[0] = YJob<T>{fs.G, nullptr, fs.G, 0};
    launch_y<T>(h, fs, jb, 1, ng * 4, false);
  }
  if (count) CK(cudaMemsetAsync(h->dcnt, 0, 4 * sizeof(int), h->st));
  {
    const int M = h->nx / 2;
    size_t smem = 2 * 4 * (size_t)M * sizeof(C);
    set_smem(k_iface_rows<T>, smem);
    dim3 grid(h->ny, ng);
    k_iface_rows<T><<<grid, 128, smem, h->st>>>(g, fs.G, h->plx, fs.Wm, fs.Wn, h->dcnt);
  }
  {
    YJobs<T> jb;
    memset(&jb, 0, sizeof jb);
    jb.j[0] = YJob<T>{fs.G, nullptr, fs.G, 2};
    launch_y<T>(h, fs, jb, 1, ng * 4, false);
  }
  k_project_planes<T><<<pgrid, 128, 0, h->st>>>(g, fs.F[0], fs.F[1], fs.F[2], fs.F[3], 0);
  k_iface_gather<T><<<ggrid, 256, 0, h->st>>>(g, fs.F[0], fs.F[1], fs.F[2], fs.F[3], fs.G, 1);
  return 0;
}

// Whether stage E leaves u*, v*, w*, rho* as whole columns in scratch for the
// solves: all four solve roles on the tensor-core kernel, which then read (and the
// pressure writes) consecutive rows instead of one value per z-plane.
template <typename T>
static int step_cols(const iw_handle* h, int cpen) {
  bool ok = h->use_bi && stageE_is_t(h);
  for (int role = 0; role < 4 && ok; ++role) ok = solve_variant<T>(h, role, cpen) == 2;
  return ok;
}

template <typename T>
static int full_step(iw_handle* h, FieldSet<T>& fs) {
  h->istep += 1;
  int r;
  if (h->p.imaxcalc == 1 && (r = adapt_dt<T>(h, fs))) return r;
  if (h->ivardt == 1) h->idtstep += 1;  // main.f:660-662
  if (h->dtanim > 0 && (h->t - h->tdump) >= h->dtanim) {  // solver.f:141-142, inside convec
    h->tdump = h->t;
    h->ianimc += 1;
    h->anim_pending = true;
  }
  const int cpen = (h->p.ispecfilterexp == 1) && (h->istep % h->p.nspecfilterexp == 0);
  r = ensure_factors(h, cpen);
  if (r) {  // nothing of the step ran
    h->istep -= 1;
    if (h->ivardt == 1) h->idtstep -= 1;
    return r;
  }
  const int cols = step_cols<T>(h, cpen);
  convec_impl<T>(h, fs, 1, cols);
  schedule_after_convec(h);
  calcuvwt_impl<T>(h, fs, cpen, cols);
  schedule_after_calcuvwt(h);
  h->t = h->t + h->p.dt;
  if (h->nlegspec > 0 && h->istep % h->nlegspec == 0 && (r = legspec_dump<T>(h, fs))) return r;  // main.f:905-910
  if (h->p.navgintrfc > 0 && h->istep % h->p.navgintrfc == 0) {
    iface_avg<T>(h, fs, true);
    mark(h, 10);
  }
  if (h->npostp > 0 && h->istep % h->npostp == 0 && (r = postp_step<T>(h, fs))) return r;  // main.f:935-936
  prof_flush(h);
  CK(launch_error());
  return 0;
}

// ---------------------------------------------------------------------------
// Autotuning of launch choices: candidates are timed with CUDA events on the
// handle's stream, on zero-filled scratch fields standing in for the state
// (the state itself is not touched; the scratch is rewritten by the next step).
// Choices: y-tile width (2, 4, 8 columns), stage A and stage E variant
// (register-column or tiled).  All candidates compute the same step; the stage
// variants differ only in the order of floating-point sums.
// ---------------------------------------------------------------------------
template <typename T>
static int tune_impl(iw_handle* h, FieldSet<T>& fs, int* choice) {
  const size_t n = h->ntot;
  for (auto* a : fs.Y12) CK(cudaMemsetAsync(a, 0, n * sizeof(T), h->st));
  for (auto* a : fs.X11) CK(cudaMemsetAsync(a, 0, n * sizeof(T), h->st));
  for (auto* a : fs.B8) CK(cudaMemsetAsync(a, 0, n * sizeof(T), h->st));
  FieldSet<T> ts = fs;  // state arrays pointed at scratch
  for (int q = 0; q < 4; ++q) {
    ts.F[q] = fs.Y12[q];
    ts.F1[q] = fs.Y12[4 + q];
    ts.Z4[q] = fs.Y12[8 + q];
    ts.Fn[q] = fs.X11[q];
    ts.Fnm[q] = fs.X11[4 + q];
    ts.Sn[q] = fs.X11[7 + q];
    ts.Snm[q] = fs.B8[q];
  }
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  auto timeit = [&](auto&& launch) {
    launch();
    cudaEventRecord(e0, h->st);
    for (int r = 0; r < 3; ++r) launch();
    cudaEventRecord(e1, h->st);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    return ms;
  };
  const int save[4] = {h->tune_ytx, h->tune_a, h->tune_e, h->use_sys};
  // y tiles: the 10-job inverse and the 4-job forward-with-fold launches.  8 stands for the tiles taken by size (16
  // columns where ny <= 128; narrower ones of two transforms that do not fit in shared memory); a narrower
  // choice replaces it if its tiles differ and it is 2 % faster.
  float best = 0.f;
  int besttx = 8, seen1 = 0, seen2 = 0;
  for (int tx : {8, 4, 2}) {
    h->tune_ytx = tx;
    const int w1 = ytx<T>(h, false), w2 = ytx<T>(h, true);
    if (w1 == seen1 && w2 == seen2) continue;
    seen1 = w1;
    seen2 = w2;
    const float ms = timeit([&] {
      YJobs<T> ji, jf;
      memset(&ji, 0, sizeof ji);
      memset(&jf, 0, sizeof jf);
      for (int q = 0; q < 10; ++q) ji.j[q] = YJob<T>{fs.Y12[q], nullptr, fs.X11[q], q < 7 ? 0 : 1};
      for (int q = 0; q < 4; ++q) jf.j[q] = YJob<T>{fs.X11[q], fs.X11[4 + q], fs.B8[4 + q], 3};
      launch_y<T>(h, ts, ji, 10, h->nz, false);
      launch_y<T>(h, ts, jf, 4, h->nz, true);
    });
    if (tx == 8 || ms < 0.98f * best) {
      best = ms;
      besttx = tx;
    }
  }
  h->tune_ytx = besttx;
  // threads per x-row CTA (scratch rows in, scratch rows out), where the length's kernel has the choice
  if (!xrow_reg_length(h->nx / 2)) {
    float bx = 0.f;
    int bestx = 256;
    for (int xt : {256, 128}) {
      h->tune_xthr = xt;
      const float t = timeit([&] { launch_xrow<T>(h, ts); });
      if (xt == 256 || t < bx) {
        bx = t;
        bestx = xt;
      }
    }
    h->tune_xthr = bestx;
  }
  // stage A and stage E variants
  // Where the tensor-core kernels apply (N <= 40) they were the fastest at every size measured (64^2 x (4 x 17) to
  // 512^2 x (12 x 33), both precisions) and are kept; the older variants round differently in mixed precision, so a
  // tuned run keeps the bits of an untuned one.  Larger N: tiled or, within the register buckets, register-column.
  int besta = -1, beste = h->N <= kTcMaxN ? 2 : -1;
  if (h->N > kTcMaxN) {
    float bt = 0;
    for (int v = 0; v < 2; ++v) {
      if (v == 1 && !zop_bucket(h->N)) continue;
      h->tune_e = v;
      const float t = timeit([&] { launch_stageE<T>(h, ts, 0); });
      if (beste < 0 || t < bt) {
        bt = t;
        beste = v;
      }
    }
  }
  h->tune_a = besta;
  h->tune_e = beste;
  // solves: system-grouped kernel or one task of <= 4 right-hand sides per
  // CTA (the u/v solve; the tables are built first if no step has run yet)
  if (ensure_factors(h, (h->p.ispecfilterexp == 1) && ((h->istep + 1) % h->p.nspecfilterexp == 0)) == IW_OK &&
      h->use_bi) {
    const int cpen = (h->p.ispecfilterexp == 1) && ((h->istep + 1) % h->p.nspecfilterexp == 0);
    const int kstart = h->p.bc_variant == IW_BC_NOSLIP ? 1 : 0;
    // each solve role (pressure, u/v, w, rho) keeps its own fastest variant; with all four on the
    // tensor cores stage E hands them whole columns, which no mixture matched
    bool all_tc = stageE_is_t(h);
    for (int role = 0; role < 4; ++role) {
      h->sys_role[role] = 2;
      all_tc = all_tc && solve_variant<T>(h, role, cpen) == 2;
    }
    for (int role : {3, 0, 1, 2}) {
      if (all_tc) continue;
      float best = 0;
      int bestv = 1;
      for (int v = 0; v < 4; ++v) {
        if (v == 2 && h->N > kTcMaxN) continue;
        if (v == 3 && (role == 3 || (h->ns * ((h->N + 1) / 2) + 31) / 32 * 32 > kSys2MaxThreads)) continue;
        h->sys_role[role] = v;
        const float t = timeit([&] { launch_solve_bi<T>(h, ts, role, cpen, kstart, 0, false); });
        if (v == 0 || t < best) {
          best = t;
          bestv = v;
        }
      }
      h->sys_role[role] = bestv;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  const cudaError_t err = launch_error();
  if (err != cudaSuccess) {
    h->tune_ytx = save[0];
    h->tune_xthr = 0;
    h->tune_a = save[1];
    h->tune_e = save[2];
    h->use_sys = save[3];
    for (int& r : h->sys_role) r = -1;
    return set_err(IW_ERR_CUDA, std::string("autotune: ") + cudaGetErrorString(err));
  }
  if (choice) {
    choice[0] = h->tune_ytx;
    choice[1] = h->tune_a;
    choice[2] = h->tune_e;
    choice[3] = h->sys_role[3] >= 0 ? h->sys_role[3] : h->use_sys;
  }
  return IW_OK;
}

// ---------------------------------------------------------------------------
// CUDA-graph replay of whole steps.
//
// From step 4 on, with a fixed dt, the SS3/BDF3 coefficients and the solver
// tables no longer change.  The launches of a step and their arguments are
// then the same from step to step, up to the history buffers, whose pointer
// arrangement repeats every 2 steps.  Two captured graphs (one per
// arrangement), launched alternately, therefore replay the step exactly.
// Conditions that would make a step depend on its number keep the eager path:
// paddle forcing (time in the arguments), a filter not applied every step,
// interface averaging less often than every step, per-phase profiling, an
// adaptive step (its rule reads the CFL numbers back at every step), animation
// dumps (their schedule depends on t), Legendre spectra, the TKE budget.
// ---------------------------------------------------------------------------
static bool graph_ready(const iw_handle* h) {
  return h->istep >= 3 && !h->prof && !h->p.forcing && (h->p.ispecfilterexp != 1 || h->p.nspecfilterexp == 1) &&
         h->p.navgintrfc <= 1 && h->p.imaxcalc != 1 && !(h->dtanim > 0) && h->nlegspec <= 0 && h->npostp <= 0;
}

static int step_dispatch(iw_handle* h) { return h->mixed ? full_step<float>(h, h->f32) : full_step<double>(h, h->f64); }

static void rotate_host(iw_handle* h) {
  if (h->mixed)
    rotate_levels(h->f32);
  else
    rotate_levels(h->f64);
}

// One step of every handle captured into one graph whose launch on s0 runs
// the members as independent branches.  The host-side step counters are put
// back after capture (they advance when the graph runs).
static int capture_step(iw_handle* const* hs, int n, cudaStream_t s0, cudaGraphExec_t* out) {
  *out = nullptr;
  cudaEvent_t fork = nullptr;
  std::vector<cudaEvent_t> join(n, nullptr);
  CK(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
  for (auto& e : join) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  int rc = IW_OK, stepped = 0;
  CK(cudaStreamBeginCapture(s0, cudaStreamCaptureModeThreadLocal));
  cudaEventRecord(fork, s0);
  for (int i = 0; i < n; ++i) {
    iw_handle* h = hs[i];
    cudaStreamWaitEvent(h->st, fork, 0);
    const int is = h->istep;
    const double t = h->t;
    rc = step_dispatch(h);
    h->istep = is;
    h->t = t;
    ++stepped;
    cudaEventRecord(join[i], h->st);
    cudaStreamWaitEvent(s0, join[i], 0);
    if (rc != IW_OK) break;
  }
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(s0, &g);
  if (rc == IW_OK && e != cudaSuccess)
    rc = set_err(IW_ERR_CUDA, std::string("graph capture of the step failed: ") + cudaGetErrorString(e));
  if (rc == IW_OK) {
    const cudaError_t ei = cudaGraphInstantiate(out, g, 0);
    if (ei != cudaSuccess) rc = set_err(IW_ERR_CUDA, std::string("graph instantiation failed: ") + cudaGetErrorString(ei));
  }
  if (g) cudaGraphDestroy(g);
  if (rc != IW_OK) {
    launch_error();  // reported here; the next call starts without it
    for (int i = 0; i < stepped; ++i) rotate_host(hs[i]);  // nothing ran: undo the host-side rotation
  }
  cudaEventDestroy(fork);
  for (auto& ev : join) cudaEventDestroy(ev);
  return rc;
}

// nsteps steps of every handle (all graph_ready, same device) as alternating
// graph launches on a private stream, ordered after and before the handles'
// own streams.
// Device error words -> IW_ERR_*.  Stage A flags a NaN or Inf in the state
// it reads at the start of every step; a bounded wait of a solve kernel that
// gave up flags a timeout.  The words stay set until the state is replaced.
static int err_code(const int* w) {
  if (w[0]) return set_err(IW_ERR_NONFINITE, "non-finite value in the state (found by a step's stage A)");
  if (w[1]) return set_err(IW_ERR_TIMEOUT, "a bounded device wait gave up (the solver tables did not arrive)");
  return IW_OK;
}
// the host copy left by the last step whose copy has completed (no wait)
static int poll_errors(iw_handle* h) {
  if (!h->err_ev_live || cudaEventQuery(h->err_ev) != cudaSuccess) return IW_OK;
  return err_code(h->herr);
}
// queue the copy of the words behind the work just launched (not while capturing)
static void post_errors(iw_handle* h) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(h->st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return;
  if (cudaMemcpyAsync(h->herr, h->derr, 2 * sizeof(int), cudaMemcpyDeviceToHost, h->st) == cudaSuccess &&
      cudaEventRecord(h->err_ev, h->st) == cudaSuccess)
    h->err_ev_live = true;
}
// wait for the handle's stream and check the words
static int sync_errors(iw_handle* h) {
  int w[2] = {0, 0};
  CK(scopy(h, w, h->derr, sizeof w, cudaMemcpyDeviceToHost));
  return err_code(w);
}
// a new state: forget earlier findings
static int clear_errors(iw_handle* h) {
  CK(cudaMemsetAsync(h->derr, 0, 2 * sizeof(int), h->st));
  CK(cudaStreamSynchronize(h->st));
  h->herr[0] = h->herr[1] = 0;
  h->err_ev_live = false;
  return IW_OK;
}

static int run_graphs(iw_handle* const* hs, int n, int nsteps) {
  if (nsteps <= 0) return IW_OK;
  cudaStream_t s0 = nullptr;
  CK(cudaStreamCreateWithFlags(&s0, cudaStreamNonBlocking));
  cudaEvent_t ev = nullptr;
  CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  for (int i = 0; i < n; ++i) {
    CK(cudaEventRecord(ev, hs[i]->st));
    CK(cudaStreamWaitEvent(s0, ev, 0));
  }
  cudaGraphExec_t gx[2] = {nullptr, nullptr};
  int rc = capture_step(hs, n, s0, &gx[0]);  // arrangement p; host moves to p+1
  if (rc == IW_OK) {
    rc = capture_step(hs, n, s0, &gx[1]);  // arrangement p+1; host back to p
    if (rc != IW_OK)
      for (int i = 0; i < n; ++i) rotate_host(hs[i]);
  }
  if (rc == IW_OK) {
    for (int k = 0; k < nsteps && rc == IW_OK; ++k) {
      const cudaError_t e = cudaGraphLaunch(gx[k & 1], s0);
      if (e != cudaSuccess) rc = set_err(IW_ERR_CUDA, std::string("graph launch failed: ") + cudaGetErrorString(e));
      else
        for (int i = 0; i < n; ++i) {  // host-side state follows each replayed step
          hs[i]->istep += 1;
          hs[i]->t += hs[i]->p.dt;
          rotate_host(hs[i]);
        }
    }
    cudaEventRecord(ev, s0);
    for (int i = 0; i < n; ++i) {
      cudaStreamWaitEvent(hs[i]->st, ev, 0);
      post_errors(hs[i]);
    }
  }
  for (auto& g : gx)
    if (g) cudaGraphExecDestroy(g);
  cudaEventDestroy(ev);
  cudaStreamDestroy(s0);
  return rc;
}

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" {

const char* iw_last_error(void) { return g_err.c_str(); }
int iw_last_status(void) { return g_status; }

int iw_init(const iw_dims* dims, const iw_params* prm, int device, iw_handle** out) {
  if (!dims || !prm || !out) return set_err(IW_ERR_CONFIG, "null argument");
  *out = nullptr;
  const iw_dims& d = *dims;
  if (d.nx < 4 || d.nx % 2 || make_plan(d.nx / 2).npass < 0) return set_err(IW_ERR_CONFIG, "nx: need even, radices 2,3,5");
  if (d.ny < 1 || (d.ny > 1 && (d.ny % 2 || make_plan(d.ny).npass < 0)))
    return set_err(IW_ERR_CONFIG, "ny: need 1 or even with radices 2,3,5");
  if (d.nzloc < 3 || d.nzloc > 48) return set_err(IW_ERR_CONFIG, "nzloc outside [3,48]");
  if (d.nsubd < 1 || d.nsubd > IW_MAX_SUBD) return set_err(IW_ERR_CONFIG, "nsubd outside [1,64]");
  {
    const size_t cs = prm->precision == IW_PREC_FP64 ? 16 : 8;
    // (the row kernel holds 17 rows; lengths are accepted while 20 would fit)
    if (20 * (size_t)xstride(d.nx / 2) * cs > 227 * 1024 || d.nx / 2 > 1024)
      return set_err(IW_ERR_CONFIG, "nx too large: nx <= 2048, and 20 rows of nx/2+1 values within the 227 KB of shared memory");
    if ((size_t)ystride(d.ny) * cs > 110 * 1024 || d.ny > 1024)
      return set_err(IW_ERR_CONFIG, "ny too large for the y-transform kernel");
  }
  double zsum = 0;
  for (int k = 0; k < d.nsubd; ++k) {
    if (!(prm->zh[k] > 0)) return set_err(IW_ERR_CONFIG, "subdomain height must be positive");
    zsum += prm->zh[k];
  }
  if (std::fabs(zsum - prm->zlen) > 1e-9 * std::max(1.0, prm->zlen))
    return set_err(IW_ERR_CONFIG, "subdomain heights do not add up to zlen");
  if (!(prm->dt > 0) || !(prm->xnu > 0) || !(prm->xkappa > 0)) return set_err(IW_ERR_CONFIG, "dt, xnu, xkappa > 0");
  if (prm->forcing < IW_PADDLE_OFF || prm->forcing > IW_PADDLE_ABOVE_BOTTOM)
    return set_err(IW_ERR_CONFIG, "forcing: IW_PADDLE_OFF, IW_PADDLE_ALL_LEVELS or IW_PADDLE_ABOVE_BOTTOM");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return set_err(IW_ERR_CUDA, "no CUDA device");
  iw_handle* h = new iw_handle();
  h->d = d;
  h->p = *prm;
  if (device >= 0) {
    h->dev = device;
    if (cudaSetDevice(device) != cudaSuccess) {
      delete h;
      return set_err(IW_ERR_CUDA, "cudaSetDevice failed");
    }
  } else {
    cudaGetDevice(&h->dev);
  }
  cudaDeviceGetAttribute(&h->nsm, cudaDevAttrMultiProcessorCount, h->dev);
  h->nx = d.nx;
  h->ny = d.ny;
  h->N = d.nzloc;
  h->ns = d.nsubd;
  h->nz = d.nzloc * d.nsubd;
  h->nxpp = d.nx + 2;
  h->nxh = d.nx / 2;
  h->nxhp = h->nxh + 1;
  h->nyh = d.ny / 2;
  h->ndims = d.ny > 1 ? 3 : 2;
  h->plane = (size_t)h->nxpp * h->ny;
  h->ntot = h->plane * h->nz;
  h->ncol = h->nxhp * h->ny;
  h->mixed = prm->precision == IW_PREC_MIXED;
  h->use_bi = prm->solver == 0 && d.nsubd <= 16;
  if (h->N > kTcMaxN) h->use_sys = 1;
  h->plx = make_plan(h->nx / 2);
  h->ply = make_plan(h->ny);
  if (cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking) != cudaSuccess ||
      cudaStreamCreateWithFlags(&h->st2, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&h->ev_fork, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&h->ev_join, cudaEventDisableTiming) != cudaSuccess) {
    side_free(h);
    delete h;
    return set_err(IW_ERR_CUDA, "stream");
  }
  h->tab = h_tables(h->N, prm->p, prm->amp, prm->fackc);
  // wavenumbers and grids (setup.f:77-166)
  const double pi2 = 8.0 * std::atan(1.0);
  const double alpha = pi2 / prm->xlen, beta = pi2 / prm->ylen;
  std::vector<double> xw(h->nxhp), yw(h->ny, 0.0), zg(h->nz), hf(h->ns), zh(h->ns), mg(h->nz);
  for (int i = 0; i < h->nxhp; ++i) xw[i] = i * alpha;
  for (int j = 1; j <= h->nyh; ++j) {
    yw[j - 1] = (j - 1) * beta;
    yw[h->ny - j] = -j * beta;
  }
  for (int ks = 0; ks < h->ns; ++ks) {
    hf[ks] = 2. / prm->zh[ks];
    zh[ks] = prm->zh[ks];
    for (int kl = 0; kl < h->N; ++kl) zg[ks * h->N + kl] = prm->z0[ks] + 0.5 * prm->zh[ks] * (h->tab.zpts[kl] + 1.0);
  }
  for (int k = 0; k < h->nz; ++k) {
    double r = (zg[k] - prm->zcen) / prm->xlen;
    mg[k] = 1.0 - std::exp(-prm->xbcrit * (r * r));
  }
  // Fourier filter factor per column (filtering.f:849-900 with kc = 0)
  std::vector<double> cf(h->ncol);
  {
    double akmax = std::sqrt(xw[h->nxhp - 1] * xw[h->nxhp - 1] + yw[h->nyh] * yw[h->nyh]);
    for (int j = 0; j < h->ny; ++j)
      for (int ii = 0; ii < h->nxhp; ++ii) {
        double ak = std::sqrt(xw[ii] * xw[ii] + yw[j] * yw[j]);
        double theta = ak / akmax;
        cf[(size_t)j * h->nxhp + ii] = std::exp(-prm->amp * std::pow(theta, 2. * prm->pf));
      }
  }
  std::vector<double> Dt(h->N * h->N), D2t(h->N * h->N), Lt(h->N * h->N);
  for (int k1 = 0; k1 < h->N; ++k1)
    for (int k = 0; k < h->N; ++k) {
      Dt[(size_t)k * h->N + k1] = h->tab.D[(size_t)k1 * h->N + k];
      D2t[(size_t)k * h->N + k1] = h->tab.D2[(size_t)k1 * h->N + k];
      Lt[(size_t)k * h->N + k1] = h->tab.Lfil[(size_t)k1 * h->N + k];
    }
  int r = 0;
  r |= up(h, &h->dDt, Dt) || up(h, &h->dD2t, D2t) || up(h, &h->dLt, Lt);
  {
    // 1/dz of the CFL in z (various.f:665-987): zf merges the duplicated
    // interface points; the point below zf(1) is the word before it, z(nz);
    // the top level has no CFL
    const int N = h->N, ns = h->ns, nz = h->nz;
    std::vector<double> zf((size_t)ns * (N - 1) + 2, 0.0), zgl(nz), dzi(nz, 0.0);
    for (int ks = 0; ks < ns; ++ks)
      for (int kl = 0; kl < N; ++kl) {
        const double z = prm->z0[ks] + 0.5 * prm->zh[ks] * (h->tab.zpts[kl] + 1.0);
        zgl[ks * N + kl] = z;
        zf[(size_t)ks * (N - 1) + kl + 1] = z;
      }
    for (int ks = 0; ks < ns; ++ks)
      for (int kl = 0; kl < N; ++kl) {
        const int k = ks * N + kl, kg = ks * (N - 1) + kl + 1;
        if (k == nz - 1) continue;
        const double zm = kg - 1 >= 1 ? zf[kg - 1] : zgl[nz - 1];
        dzi[k] = 1.0 / (zf[kg] - zm);
      }
    r |= up(h, &h->ddzinv, dzi) || dalloc(h, &h->dpart, kPartDoubles);
  }
  r |= up(h, &h->dD, h->tab.D) || up(h, &h->dD2, h->tab.D2) || up(h, &h->dL, h->tab.Lfil) || up(h, &h->dh, hf) ||
       up(h, &h->dxw, xw) || up(h, &h->dyw, yw) || up(h, &h->dcf, cf) || up(h, &h->dzg, zg) || up(h, &h->dzh, zh) ||
       up(h, &h->dwg, h->tab.wg) || up(h, &h->dal, h->tab.alpol) || up(h, &h->dsig, h->tab.sigma) ||
       up(h, &h->dmeang, mg);
  r |= dalloc(h, &h->dwnl, h->plane * 2) || dalloc(h, &h->dwvr, h->plane * 2) || dalloc(h, &h->dred, std::max<size_t>(64, 4 * (size_t)h->nz)) ||
       dalloc(h, &h->dcnt, 8) || dalloc(h, &h->dflag, 4) || dalloc(h, &h->derr, 2) ||
       cudaHostAlloc((void**)&h->herr, 2 * sizeof(int), cudaHostAllocDefault) != cudaSuccess ||
       cudaEventCreateWithFlags(&h->err_ev, cudaEventDisableTiming) != cudaSuccess;
  if (!r) {
    cudaMemset(h->dcnt, 0, 8 * sizeof(int));
    cudaMemset(h->derr, 0, 2 * sizeof(int));
    h->herr[0] = h->herr[1] = 0;
    cudaMemset(h->dwnl, 0, h->plane * 2 * sizeof(double));
    cudaMemset(h->dwvr, 0, h->plane * 2 * sizeof(double));
    r = h->mixed ? alloc_fields(h, h->f32) : alloc_fields(h, h->f64);
  }
  if (!r) r = build_distinct(h);
  if (r) {
    iw_destroy(h);
    return IW_ERR_NOMEM;
  }
  // distinct subdomain blocks of the penalty systems: a block is fixed by
  // epsilon, its height and whether it has neighbours below and above
  h->nb = 0;
  for (int ks = 0; ks < h->ns; ++ks) {
    int found = -1;
    for (int b = 0; b < h->nb && found < 0; ++b) {
      const int r = h->brep[b];
      if ((r > 0) == (ks > 0) && (r < h->ns - 1) == (ks < h->ns - 1) && prm->zh[r] == prm->zh[ks]) found = b;
    }
    if (found < 0) {
      found = h->nb;
      h->brep[h->nb++] = ks;
    }
    h->bmap[ks] = found;
  }
  h->c = Coefs{1., 0., 0., 1., 0., 0., 1., prm->dt};
  {  // main.f:341-346 (bruntz = brunt)
    const double pi2 = 8. * std::atan(1.0), kx = pi2 / prm->xlen, m = pi2 / (2. * prm->zlen);
    h->xomega = (prm->brunt * kx) / std::sqrt(kx * kx + m * m);
  }
  *out = h;
  return IW_OK;
}

static int out_join(iw_handle* h);
static void helm_free(iw_handle* h);

int iw_destroy(iw_handle* h) {
  if (!h) return IW_OK;
  cudaSetDevice(h->dev);
  out_join(h);
  helm_free(h);
  if (h->out_host) cudaFreeHost(h->out_host);
  if (h->anim_host) cudaFreeHost(h->anim_host);
  if (h->leg_host) cudaFreeHost(h->leg_host);
  cudaFree(h->dlegspec);
  cudaFree(h->dpostp);
  if (h->out_ev) cudaEventDestroy(h->out_ev);
  free_fields(h->f64);
  free_fields(h->f32);
  free_fields(h->tw64);
  cudaFree(h->scr);
  for (double* p : {h->ddzinv, h->dpart, h->dDt, h->dD2t, h->dLt, h->dD, h->dD2, h->dL, h->dh, h->dxw, h->dyw, h->dcf, h->dzg, h->dzh, h->dwg, h->dal, h->dsig,
                    h->dmeang, h->dwnl, h->dwvr, h->dred})
    cudaFree(p);
  cudaFree(h->dcnt);
  cudaFree(h->dflag);
  cudaFree(h->derr);
  if (h->herr) cudaFreeHost(h->herr);
  if (h->hstat) cudaFreeHost(h->hstat);
  if (h->err_ev) cudaEventDestroy(h->err_ev);
  cudaFree(h->dcolorder);
  cudaFree(h->dakv);
  for (int k = 0; k < SYS_KINDS; ++k) {
    cudaFree(h->dtasks[k]);
    cudaFree(h->dtasks2[k]);
    h->bi[k].release();
    cudaFree(h->dab[k]);
    cudaFree(h->dipiv[k]);
    cudaFree(h->dinfo[k]);
    cudaFree(h->dsys[k]);
    cudaFree(h->dpen[k]);
    cudaFree(h->dcolsys[k]);
  }
  side_free(h);
  if (g_bound == h) g_bound = nullptr;
  delete h;
  return IW_OK;
}

static int copy_level(iw_handle* h, int level, double* host, bool up_dir) {
  // level 0 F, 1 Fn, 2 Fnm, 3 Sn, 4 Snm.  The host side is always FP64.  For
  // FP32 fields each half field goes through a scratch field that holds
  // ntot/2 doubles (the scratch is free between steps): a stream-ordered copy
  // and a conversion kernel per half, no allocation, one wait at the end.
  // With pinned host memory the copies run at full link speed.
  const size_t n = h->ntot;
  for (int q = 0; q < 4; ++q) {
    if (h->mixed) {
      float* const* L = level == 0 ? h->f32.F : level == 1 ? h->f32.Fn : level == 2 ? h->f32.Fnm : level == 3 ? h->f32.Sn : h->f32.Snm;
      float* dp = L[q];
      for (int half = 0; half < 2; ++half) {
        const size_t o = half ? n / 2 : 0, c = half ? n - n / 2 : n / 2;
        // c doubles fit in a scratch field of n floats when c <= n/2 + 1 (n is even: nxpp is)
        double* tmp = (double*)h->f32.Y12[half];
        if (up_dir) {
          CK(cudaMemcpyAsync(tmp, host + q * n + o, c * sizeof(double), cudaMemcpyHostToDevice, h->st));
          k_convert<double, float><<<1184, 256, 0, h->st>>>(tmp, dp + o, c);
        } else {
          k_convert<float, double><<<1184, 256, 0, h->st>>>(dp + o, tmp, c);
          CK(cudaMemcpyAsync(host + q * n + o, tmp, c * sizeof(double), cudaMemcpyDeviceToHost, h->st));
        }
        CK(launch_error());
      }
    } else {
      double* const* L = level == 0 ? h->f64.F : level == 1 ? h->f64.Fn : level == 2 ? h->f64.Fnm : level == 3 ? h->f64.Sn : h->f64.Snm;
      double* dp = L[q];
      if (up_dir)
        CK(cudaMemcpyAsync(dp, host + q * n, n * sizeof(double), cudaMemcpyHostToDevice, h->st));
      else
        CK(cudaMemcpyAsync(host + q * n, dp, n * sizeof(double), cudaMemcpyDeviceToHost, h->st));
    }
  }
  CK(cudaStreamSynchronize(h->st));
  return 0;
}

int iw_upload_state(iw_handle* h, const double* uvwt, const double* uvwt_n, const double* uvwt_nm, const double* s_n,
                    const double* s_nm, double t, int istep_done) {
  if (!h) return set_err(IW_ERR_STATE, "null handle");
  cudaSetDevice(h->dev);
  const double* src[5] = {uvwt, uvwt_n, uvwt_nm, s_n, s_nm};
  for (int l = 0; l < 5; ++l)
    if (src[l]) {
      int r = copy_level(h, l, const_cast<double*>(src[l]), true);
      if (r) return r;
    }
  if (int r = clear_errors(h)) return r;
  h->t = t;
  h->istep = istep_done;
  h->cdt = 1.;
  h->ivardt = 0;
  h->idtstep = 0;
  h->istart = 0;
  if (istep_done == 0) {
    h->c = Coefs{1., 0., 0., 1., 0., 0., 1., h->p.dt};
  } else if (istep_done == 1) {
    h->c = Coefs{2., -1., 0., 2., -0.5, 0., 1.5, h->p.dt};
  } else {
    h->c = Coefs{3., -3., 1., 3., -1.5, 1. / 3., 11. / 6., h->p.dt};
  }
  return IW_OK;
}

int iw_download_state(iw_handle* h, double* uvwt, double* uvwt_n, double* uvwt_nm, double* s_n, double* s_nm) {
  if (!h) return set_err(IW_ERR_STATE, "null handle");
  cudaSetDevice(h->dev);
  double* dst[5] = {uvwt, uvwt_n, uvwt_nm, s_n, s_nm};
  for (int l = 0; l < 5; ++l)
    if (dst[l]) {
      int r = copy_level(h, l, dst[l], false);
      if (r) return r;
    }
  return IW_OK;
}

int iw_step(iw_handle* h) {
  if (!h) return set_err(IW_ERR_STATE, "null handle");
  cudaSetDevice(h->dev);
  int r = poll_errors(h);
  if (r) return r;
  r = h->mixed ? full_step<float>(h, h->f32) : full_step<double>(h, h->f64);
  post_errors(h);
  return r;
}

int iw_run(iw_handle* h, int nsteps, int use_graph) {
  if (!h) return set_err(IW_ERR_STATE, "null handle");
  cudaSetDevice(h->dev);
  int r = poll_errors(h);
  if (r) return r;
  int s = 0;
  for (; s < nsteps && !(use_graph && graph_ready(h)); ++s) {
    r = step_dispatch(h);
    if (r) return r;
    post_errors(h);
    if ((r = poll_errors(h))) return r;
  }
  return run_graphs(&h, 1, nsteps - s);
}

int iw_autotune(iw_handle* h, int* choices) {
  if (!h) return set_err(IW_ERR_STATE, "null handle");
  cudaSetDevice(h->dev);
  return h->mixed ? tune_impl<float>(h, h->f32, choices) : tune_impl<double>(h, h->f64, choices);
}

int iw_set_launch(iw_handle* h, int which, int value) {
  if (!h) return set_err(IW_ERR_STATE, "null handle");
  switch (which) {
    case IW_LAUNCH_YTILE:
      if (value != 0 && value != 2 && value != 4 && value != 8) return set_err(IW_ERR_CONFIG, "y tile: 0, 2, 4 or 8");
      h->tune_ytx = value;
      return IW_OK;
    case IW_LAUNCH_STAGE_A:
    case IW_LAUNCH_STAGE_E:
      if (value < -1 || value > (which == IW_LAUNCH_STAGE_E ? 3 : 1))
        return set_err(IW_ERR_CONFIG, "stage variant: -1, 0, 1 (or 2, 3 for stage E)");
      if (value == 1 && !zop_bucket(h->N)) return set_err(IW_ERR_CONFIG, "register-column stages need N <= 33");
      if (value >= 2 && h->N > kTcMaxN) return set_err(IW_ERR_CONFIG, "tensor-core stage E needs N <= 40");
      (which == IW_LAUNCH_STAGE_A ? h->tune_a : h->tune_e) = value;
      return IW_OK;
    case IW_LAUNCH_SOLVE:
      if (value < 0 || value > 3) return set_err(IW_ERR_CONFIG, "solve variant: 0, 1, 2 or 3");
      if (value == 2 && h->N > kTcMaxN) return set_err(IW_ERR_CONFIG, "tensor-core solve needs N <= 40");
      h->use_sys = value;
      for (int& r : h->sys_role) r = -1;
      return IW_OK;
    case IW_LAUNCH_XROW_THREADS:
      if (value != 0 && value != 128 && value != 256) return set_err(IW_ERR_CONFIG, "x-row threads: 0, 128 or 256");
      h->tune_xthr = value;
      return IW_OK;
    case IW_LAUNCH_SOLVE_UV:
    case IW_LAUNCH_SOLVE_W:
    case IW_LAUNCH_SOLVE_RHO:
    case IW_LAUNCH_SOLVE_PRESSURE: {
      if (value < -1 || value > 3) return set_err(IW_ERR_CONFIG, "solve variant: -1, 0, 1, 2 or 3");
      if (value == 2 && h->N > kTcMaxN) return set_err(IW_ERR_CONFIG, "tensor-core solve needs N <= 40");
      const int role = which == IW_LAUNCH_SOLVE_UV ? 0 : which == IW_LAUNCH_SOLVE_W ? 1
                       : which == IW_LAUNCH_SOLVE_RHO ? 2 : 3;
      h->sys_role[role] = value;
      return IW_OK;
    }
    default:
      return set_err(IW_ERR_CONFIG, "unknown launch choice");
  }
}

int iw_get_launch(iw_handle* h, int which, int* value) {
  if (!h || !value) return set_err(IW_ERR_STATE, "iw_get_launch: null argument");
  switch (which) {
    case IW_LAUNCH_YTILE: *value = h->tune_ytx; return IW_OK;
    case IW_LAUNCH_STAGE_A: *value = h->tune_a; return IW_OK;
    case IW_LAUNCH_STAGE_E: *value = h->tune_e; return IW_OK;
    case IW_LAUNCH_SOLVE: *value = h->use_sys; return IW_OK;
    case IW_LAUNCH_SOLVE_UV: *value = h->sys_role[0]; return IW_OK;
    case IW_LAUNCH_SOLVE_W: *value = h->sys_role[1]; return IW_OK;
    case IW_LAUNCH_SOLVE_RHO: *value = h->sys_role[2]; return IW_OK;
    case IW_LAUNCH_SOLVE_PRESSURE: *value = h->sys_role[3]; return IW_OK;
    case IW_LAUNCH_XROW_THREADS: *value = h->tune_xthr > 0 ? h->tune_xthr : h->nx <= 256 ? 128 : 256; return IW_OK;
    default: return set_err(IW_ERR_CONFIG, "unknown launch choice");
  }
}

int iw_ensemble_run(iw_handle* const* members, int n, int nsteps) {
  if (!members || n <= 0 || nsteps < 0) return set_err(IW_ERR_STATE, "iw_ensemble_run: bad argument");
  for (int i = 0; i < n; ++i) {
    if (!members[i]) return set_err(IW_ERR_STATE, "iw_ensemble_run: null member");
    if (members[i]->dev != members[0]->dev) return set_err(IW_ERR_CONFIG, "iw_ensemble_run: members on different devices");
    for (int j = 0; j < i; ++j)
      if (members[j] == members[i]) return set_err(IW_ERR_CONFIG, "iw_ensemble_run: a member is listed twice");
  }
  cudaSetDevice(members[0]->dev);
  // eager steps (members overlap on their own streams) until every member can
  // be replayed from a graph
  int s = 0;
  for (;; ++s) {
    bool all = true;
    for (int i = 0; i < n; ++i) all = all && graph_ready(members[i]);
    if (all || s >= nsteps) break;
    for (int i = 0; i < n; ++i) {
      int r = step_dispatch(members[i]);
      if (r) return r;
    }
  }
  if (s >= nsteps) return IW_OK;
  bool all = true;
  for (int i = 0; i < n; ++i) all = all && graph_ready(members[i]);
  if (!all) {  // a member that never qualifies (forcing, profiling, ...): eager
    for (; s < nsteps; ++s)
      for (int i = 0; i < n; ++i) {
        int r = step_dispatch(members[i]);
        if (r) return r;
      }
    return IW_OK;
  }
  return run_graphs(members, n, nsteps - s);
}

int iw_step_coefs(iw_handle* h, const iw_coefs* c) {
  if (!h || !c) return set_err(IW_ERR_STATE, "null argument");
  h->c = Coefs{c->fac1, c->fac2, c->fac3, c->bdf1, c->bdf2, c->bdf3, c->bdfv, c->dt};
  if (c->dt > 0 && c->dt != h->p.dt) h->p.dt = c->dt;
  return iw_step(h);
}

int iw_set_coefs(iw_handle* h, const iw_coefs* c, double t) {
  if (!h || !c) return set_err(IW_ERR_STATE, "null argument");
  if (!(c->dt > 0)) return set_err(IW_ERR_CONFIG, "iw_set_coefs: dt must be positive");
  h->c = Coefs{c->fac1, c->fac2, c->fac3, c->bdf1, c->bdf2, c->bdf3, c->bdfv, c->dt};
  h->p.dt = c->dt;
  h->t = t;
  return IW_OK;
}

int iw_sync(iw_handle* h) {
  if (!h) return set_err(IW_ERR_STATE, "null handle");
  CK(cudaStreamSynchronize(h->st));
  return sync_errors(h);
}

int iw_field_ptr(iw_handle* h, int f, void** dptr) {
  if (!h || f < 0 || f > 3 || !dptr) return set_err(IW_ERR_STATE, "bad argument");
  *dptr = h->mixed ? (void*)h->f32.F[f] : (void*)h->f64.F[f];
  return IW_OK;
}

int iw_stream(iw_handle* h, void** stream) {
  if (!h || !stream) return set_err(IW_ERR_STATE, "bad argument");
  *stream = (void*)h->st;
  return IW_OK;
}

int iw_fail_allocation(iw_handle* h, int nth) {
  if (!h || nth < 0) return set_err(IW_ERR_STATE, "bad argument");
  h->fail_alloc = nth;
  return IW_OK;
}

int iw_device_bytes(iw_handle* h, size_t* bytes) {
  if (!h || !bytes) return set_err(IW_ERR_STATE, "bad argument");
  *bytes = h->bytes;
  return IW_OK;
}

int iw_bind(iw_handle* h) {
  g_bound = h;
  return IW_OK;
}

// Per-phase device time (CUDA events on the handle's stream).  enable=1
// starts recording (and zeroes the totals), 0 stops.  Phases: 0 stageA,
// 1 y-inverse, 2 x-row NL, 3 y-forward, 4 wviscrot, 5 stageE, 6 pressure,
// 7 u/v solve, 8 w solve, 9 rho solve, 10 interface averaging.
int iw_profile(iw_handle* h, int enable) {
  if (!h) return set_err(IW_ERR_STATE, "null handle");
  if (enable && !h->prof) {
    for (int i = 0; i < 32; ++i) cudaEventCreate(&h->ev[i]);
  }
  if (!enable && h->prof) {
    for (int i = 0; i < 32; ++i) cudaEventDestroy(h->ev[i]);
  }
  h->prof = enable;
  h->nev = 0;
  for (int i = 0; i < 16; ++i) {
    h->phase_ms[i] = 0;
    h->phase_n[i] = 0;
  }
  return IW_OK;
}

int iw_profile_read(iw_handle* h, double* ms16, long* n16) {
  if (!h) return set_err(IW_ERR_STATE, "null handle");
  for (int i = 0; i < 16; ++i) {
    if (ms16) ms16[i] = h->phase_ms[i];
    if (n16) n16[i] = h->phase_n[i];
  }
  return IW_OK;
}

}  // extern "C"


// ---------------------------------------------------------------------------
// isolated batched Helmholtz solves (one system per column, lambda given)
// ---------------------------------------------------------------------------
// What the kernels of the band LU read
struct HelmCache {
  double* ab = nullptr;
  float* ab32 = nullptr;
  int* ipiv = nullptr;
  int* info = nullptr;
  SysDesc* sys = nullptr;
  double* pen = nullptr;
  int* colsys = nullptr;
};
// The tables of one set of lambdas.  Each part is made by the first call that needs it: the factors of the
// systems [0, nlu) and their FP32 copy (lu, c.ab32), the columns by system (order), the block inverses of the
// systems [first, nsys) with their tasks and the columns left to the band LU (tcm).  Freed with the handle.
struct HelmEntry {
  HelmCache c;
  std::vector<double> lam;  // distinct lambdas, ascending
  std::vector<int> cs;      // column -> system
  int nsys = 0, first = 0;  // mode 0 takes the systems from first on to k_helm_tc
  char* lu = nullptr;
  int nlu = 0;
  size_t lu_bytes = 0;
  int* order = nullptr;
  char* tcm = nullptr;
  int ntask = 0, nlist = 0;
  double *ainv = nullptr, *lvec = nullptr, *minv = nullptr, *pen = nullptr;
  SysDesc* sys = nullptr;
  Task* tasks = nullptr;
  int* list = nullptr;
};
static std::map<std::pair<iw_handle*, std::string>, HelmEntry> g_helm;
static std::mutex g_helm_mu;  // of the map: handles of other threads add entries and go away; an entry is its handle's alone

// y = A x for the penalty matrix of system s (matrix-free, FP64)
// row r; x(i): element i
template <typename X>
__device__ __forceinline__ double apply_A_row(const Geo& g, const double* __restrict__ D2, const double* __restrict__ zh,
                                              double eps, const double* __restrict__ pen, X&& x, int r) {
  const int N = g.N, ns = g.ns;
  const int ks = r / N, k1 = r % N, km = ks * N;
  const double *pa = pen, *pb = pen + ns, *pg = pen + 2 * ns, *pd = pen + 3 * ns, *pt1 = pen + 4 * ns,
               *pt2 = pen + 5 * ns;
  const double h2 = (2.0 / zh[ks]);
  double s2 = 0;
  for (int k = 0; k < N; ++k) s2 += D2[k1 * N + k] * x(km + k);
  double y = x(r) - eps * h2 * h2 * s2;
  if (k1 == 0) {
    double s0 = 0;
    for (int k = 0; k < N; ++k) s0 += g.D[0 * N + k] * x(km + k);
    y += pt1[ks] * pa[ks] * x(km) - pt1[ks] * pb[ks] * eps * h2 * s0;
    if (ks > 0) {
      double hl = 2.0 / zh[ks - 1];
      double sl = 0;
      for (int k = 0; k < N; ++k) sl += g.D[(N - 1) * N + k] * x(km - N + k);
      y += -0.5 * pt1[ks] * pa[ks] * x(km) + 0.5 * pt1[ks] * pb[ks] * eps * h2 * s0 - 0.5 * pt1[ks] * pa[ks] * x(km - 1) +
           0.5 * pt1[ks] * pb[ks] * eps * hl * sl;
    }
  }
  if (k1 == N - 1) {
    double s1 = 0;
    for (int k = 0; k < N; ++k) s1 += g.D[(N - 1) * N + k] * x(km + k);
    y += pt2[ks] * pg[ks] * x(km + N - 1) + pt2[ks] * pd[ks] * eps * h2 * s1;
    if (ks < ns - 1) {
      double hr = 2.0 / zh[ks + 1];
      double sr = 0;
      for (int k = 0; k < N; ++k) sr += g.D[0 * N + k] * x(km + N + k);
      y += -0.5 * pt2[ks] * pg[ks] * x(km + N - 1) - 0.5 * pt2[ks] * pd[ks] * eps * h2 * s1 -
           0.5 * pt2[ks] * pg[ks] * x(km + N) - 0.5 * pt2[ks] * pd[ks] * eps * hr * sr;
    }
  }
  return y;
}

__device__ void band_solve_warp_f(const float* __restrict__ ab, const int* __restrict__ ipiv, float* b, int nr, int n,
                                  int kl, int ku, int lane) {
  const int ldab = 2 * kl + ku + 1, kd = ku + kl + 1;
  for (int j = 1; j <= n - 1; ++j) {
    const int lm = min(kl, n - j);
    const int l = __ldg(ipiv + j - 1);
    const float* col = ab + (size_t)ldab * (j - 1);
    for (int r = 0; r < nr; ++r) {
      float* br = b + (size_t)r * n;
      const float bj = br[j - 1], bl = br[l - 1];
      const float y = (l != j) ? bl : bj;
      float nv0 = 0, nv1 = 0;
      const int i0 = lane + 1, i1 = lane + 33;
      if (i0 <= lm) {
        int row = j + i0;
        float old = (row == l) ? bj : br[row - 1];
        nv0 = old - __ldg(col + kd + i0 - 1) * y;
      }
      if (i1 <= lm) {
        int row = j + i1;
        float old = (row == l) ? bj : br[row - 1];
        nv1 = old - __ldg(col + kd + i1 - 1) * y;
      }
      __syncwarp();
      if (i0 <= lm) br[j + i0 - 1] = nv0;
      if (i1 <= lm) br[j + i1 - 1] = nv1;
      if (lane == 0) br[j - 1] = y;
      __syncwarp();
    }
  }
  const int k = kl + ku, kplus1 = k + 1;
  for (int j = n; j >= 1; --j) {
    const float* col = ab + (size_t)ldab * (j - 1);
    const float dg = __ldg(col + kplus1 - 1);
    const int lo = max(1, j - k), l = kplus1 - j;
    for (int r = 0; r < nr; ++r) {
      float* br = b + (size_t)r * n;
      float xj = br[j - 1] / dg;
      float nv[3];
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        int i = j - 1 - lane - 32 * m;
        nv[m] = (i >= lo) ? br[i - 1] - xj * __ldg(col + l + i - 1) : 0.f;
      }
      __syncwarp();
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        int i = j - 1 - lane - 32 * m;
        if (i >= lo) br[i - 1] = nv[m];
      }
      if (lane == 0) br[j - 1] = xj;
      __syncwarp();
    }
  }
}

// mode 0: FP64 factors and solve; mode 1: FP32 solve + one FP64 residual
// refinement sweep.  rhs/sol: [ncol][nz] complex (re,im); list: the columns, or all.
static __global__ void k_helm(Geo g, HelmCache hc, const double* __restrict__ rhs, double* __restrict__ sol, int ncol,
                              int mode, const double* __restrict__ D2, const double* __restrict__ zh,
                              const int* __restrict__ list) {
  extern __shared__ __align__(16) double smh[];
  const int warps = blockDim.x / 32, wid = threadIdx.x / 32, lane = threadIdx.x & 31;
  if (blockIdx.x * warps + wid >= ncol) return;
  const int c = list ? list[blockIdx.x * warps + wid] : blockIdx.x * warps + wid;
  const int n = g.nz, N = g.N, ldab = 3 * N + 1;
  const int s = hc.colsys[c];
  double* b = smh + (size_t)wid * 6 * n;  // b (2n), x (2n), r (2n)
  for (int k = lane; k < n; k += 32) {
    b[k] = rhs[((size_t)c * n + k) * 2];
    b[n + k] = rhs[((size_t)c * n + k) * 2 + 1];
  }
  __syncwarp();
  if (mode == 0) {
    band_solve_warp(hc.ab + (size_t)s * ldab * n, hc.ipiv + (size_t)s * n, b, 2, n, N, N, lane);
    for (int k = lane; k < n; k += 32) {
      sol[((size_t)c * n + k) * 2] = b[k];
      sol[((size_t)c * n + k) * 2 + 1] = b[n + k];
    }
    return;
  }
  double* x = b + 2 * n;
  float* xf = (float*)(b + 4 * n);  // 2n floats
  for (int k = lane; k < 2 * n; k += 32) xf[k] = (float)b[k];
  __syncwarp();
  const float* ab32 = hc.ab32 + (size_t)s * ldab * n;
  const int* ip = hc.ipiv + (size_t)s * n;
  band_solve_warp_f(ab32, ip, xf, 2, n, N, N, lane);
  for (int k = lane; k < 2 * n; k += 32) x[k] = (double)xf[k];
  __syncwarp();
  const double eps = hc.sys[s].eps;
  const double* pen = hc.pen + (size_t)s * 6 * g.ns;
  for (int k = lane; k < n; k += 32) {
    double r0 = b[k] - apply_A_row(g, D2, zh, eps, pen, [&](int i) { return x[i]; }, k);
    double r1 = b[n + k] - apply_A_row(g, D2, zh, eps, pen, [&](int i) { return x[n + i]; }, k);
    xf[k] = (float)r0;
    xf[n + k] = (float)r1;
  }
  __syncwarp();
  band_solve_warp_f(ab32, ip, xf, 2, n, N, N, lane);
  for (int k = lane; k < n; k += 32) {
    sol[((size_t)c * n + k) * 2] = x[k] + (double)xf[k];
    sol[((size_t)c * n + k) * 2 + 1] = x[n + k] + (double)xf[n + k];
  }
}

// Mode 1 with a right-hand side per lane: a warp takes 16 columns in the order of their
// systems (real and imaginary part in neighbouring lanes) and keeps their vectors in shared
// memory, [row][lane] FP32.  A lane runs its own band sweep: no shuffles and no
// barriers, the factor entries of a step are independent loads that lanes of one
// system share, and the updates of a step are independent.  The arithmetic of every element and
// its order are band_solve_warp_f's, so the FP32 sweeps give the same bits.  The FP64
// residual walks block by block; a block's residual replaces its x one block later (the
// next block's coupling row still reads it) and x waits in sol.
// NB >= N: the entries of the next step's factor column are loaded while the current
// one is applied (registers; NB = 0: no prefetch, any N).
template <int NB>
__device__ __forceinline__ void band_sweep_lane(const float* __restrict__ ab, const int* __restrict__ ipiv, float* b,
                                                int n, int N) {
  const int ldab = 3 * N + 1, k = 2 * N;  // b: element i at b[32 i]
  if constexpr (NB == 0) {
    for (int j = 0; j < n - 1; ++j) {
      const int lm = min(N, n - 1 - j), l = __ldg(ipiv + j) - 1;
      const float* col = ab + (size_t)ldab * j + k;
      float* bj = b + 32 * j;
      const float v = bj[0], y = b[32 * l];
      if (l != j) {
        b[32 * l] = v;
        bj[0] = y;
      }
#pragma unroll 8
      for (int i = 1; i <= lm; ++i) bj[32 * i] = __fmaf_rn(-__ldg(col + i), y, bj[32 * i]);
    }
    for (int j = n - 1; j >= 0; --j) {
      const float* col = ab + (size_t)ldab * j + k;
      float* bj = b + 32 * j;
      const float xj = __fdiv_rn(bj[0], __ldg(col));
      bj[0] = xj;
      const int m = min(k, j);
#pragma unroll 8
      for (int i = 1; i <= m; ++i) bj[-32 * i] = __fmaf_rn(-xj, __ldg(col - i), bj[-32 * i]);
    }
  } else {
    float m[NB], mn[NB];
    int l = __ldg(ipiv) - 1, ln = 0;
#pragma unroll
    for (int i = 0; i < NB; ++i) m[i] = i < min(N, n - 1) ? __ldg(ab + k + 1 + i) : 0.f;
    for (int j = 0; j < n - 1; ++j) {
      const int lm = min(N, n - 1 - j);
      if (j + 1 < n - 1) {
        const float* cn = ab + (size_t)ldab * (j + 1) + k + 1;
        const int lmn = min(N, n - 2 - j);
        ln = __ldg(ipiv + j + 1) - 1;
#pragma unroll
        for (int i = 0; i < NB; ++i) mn[i] = i < lmn ? __ldg(cn + i) : 0.f;
      }
      float* bj = b + 32 * j;
      const float v = bj[0], y = b[32 * l];
      if (l != j) {
        b[32 * l] = v;
        bj[0] = y;
      }
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (i < lm) bj[32 * (i + 1)] = __fmaf_rn(-m[i], y, bj[32 * (i + 1)]);
      l = ln;
#pragma unroll
      for (int i = 0; i < NB; ++i) m[i] = mn[i];
    }
    float v[2 * NB], vn[2 * NB], dg, dgn = 0.f;
    {
      const float* col = ab + (size_t)ldab * (n - 1) + k;
      dg = __ldg(col);
#pragma unroll
      for (int i = 0; i < 2 * NB; ++i) v[i] = i < min(k, n - 1) ? __ldg(col - 1 - i) : 0.f;
    }
    for (int j = n - 1; j >= 0; --j) {
      if (j > 0) {
        const float* col = ab + (size_t)ldab * (j - 1) + k;
        const int mm = min(k, j - 1);
        dgn = __ldg(col);
#pragma unroll
        for (int i = 0; i < 2 * NB; ++i) vn[i] = i < mm ? __ldg(col - 1 - i) : 0.f;
      }
      float* bj = b + 32 * j;
      const float xj = __fdiv_rn(bj[0], dg);
      bj[0] = xj;
      const int mj = min(k, j);
#pragma unroll
      for (int i = 0; i < 2 * NB; ++i)
        if (i < mj) bj[-32 * (i + 1)] = __fmaf_rn(-xj, v[i], bj[-32 * (i + 1)]);
      dg = dgn;
#pragma unroll
      for (int i = 0; i < 2 * NB; ++i) v[i] = vn[i];
    }
  }
}
static size_t helm32_smem(int n, int N) { return (size_t)(n + 2 * N) * 32 * sizeof(float); }
template <int NB>
static __global__ void __launch_bounds__(32) k_helm32(Geo g, HelmCache hc, const double* __restrict__ rhs,
                                                      double* __restrict__ sol, int ncol, const double* __restrict__ D2,
                                                      const double* __restrict__ zh, const int* __restrict__ order) {
  extern __shared__ __align__(16) float smf[];
  const int n = g.nz, N = g.N, ldab = 3 * N + 1, lane = threadIdx.x;
  const int at = blockIdx.x * 16 + (lane >> 1);
  if (at >= ncol) return;
  const int c = order[at], s = hc.colsys[c];
  const double* rc = rhs + (size_t)c * n * 2 + (lane & 1);
  double* xc = sol + (size_t)c * n * 2 + (lane & 1);
  float* b = smf + lane;
  float* tmp = smf + (size_t)n * 32 + lane;  // two blocks of residuals
  const float* ab = hc.ab32 + (size_t)s * ldab * n;
  const int* ip = hc.ipiv + (size_t)s * n;
#pragma unroll 8
  for (int k = 0; k < n; ++k) b[32 * k] = (float)rc[2 * k];
  band_sweep_lane<NB>(ab, ip, b, n, N);
  const double eps = hc.sys[s].eps;
  const double* pen = hc.pen + (size_t)s * 6 * g.ns;
  auto x = [&](int i) { return (double)b[32 * i]; };
  for (int ks = 0; ks < g.ns; ++ks) {
    float* t = tmp + (ks & 1) * N * 32;
    for (int k1 = 0; k1 < N; ++k1) {
      const int r = ks * N + k1;
      t[32 * k1] = (float)(rc[2 * r] - apply_A_row(g, D2, zh, eps, pen, x, r));
    }
    if (ks > 0) {  // block ks - 1 is read no more
      const float* p = tmp + ((ks - 1) & 1) * N * 32;
      for (int k1 = 0; k1 < N; ++k1) {
        const int r = (ks - 1) * N + k1;
        const double x1 = x(r);
        b[32 * r] = p[32 * k1];
        xc[2 * r] = x1;
      }
    }
  }
  const float* p = tmp + ((g.ns - 1) & 1) * N * 32;
  for (int k1 = 0; k1 < N; ++k1) {
    const int r = (g.ns - 1) * N + k1;
    const double x1 = x(r);
    b[32 * r] = p[32 * k1];
    xc[2 * r] = x1;
  }
  band_sweep_lane<NB>(ab, ip, b, n, N);
  for (int k = 0; k < n; ++k) xc[2 * k] += (double)b[32 * k];
}

// Pieces of one device allocation: each piece's offset, the total in `at`
static size_t carve(size_t& at, size_t bytes) {
  const size_t o = at;
  at += (bytes + 255) & ~(size_t)255;
  return o;
}

// the columns by system
static std::vector<int> helm_order(const HelmEntry& E) {
  std::vector<int> at(E.nsys + 1, 0), order(E.cs.size());
  for (int u : E.cs) ++at[u + 1];
  for (int u = 0; u < E.nsys; ++u) at[u + 1] += at[u];
  for (size_t c = 0; c < order.size(); ++c) order[at[E.cs[c]]++] = (int)c;
  return order;
}

// Band LU of the systems [0, need), and their FP32 copy for mode 1
static int helm_lu(iw_handle* h, HelmEntry& E, int need, bool fp32, int bot, int top) {
  const int n = h->nz, N = h->N, ldab = 3 * N + 1, ns = h->ns;
  const size_t band = (size_t)ldab * n;
  if (E.nlu < need) {
    size_t at = 0;
    const size_t osys = carve(at, need * sizeof(SysDesc)), open = carve(at, (size_t)need * 6 * ns * sizeof(double)), up_to = at;
    const size_t oab = carve(at, need * band * sizeof(double)), opiv = carve(at, (size_t)need * n * sizeof(int)),
                 oinfo = carve(at, need * sizeof(int));
    std::vector<char> host(up_to, 0);
    for (int u = 0; u < need; ++u) {
      SysDesc& sd = ((SysDesc*)(host.data() + osys))[u];
      double* pen = (double*)(host.data() + open) + (size_t)u * 6 * ns;
      sd.eps = 1. / E.lam[u];
      sd.ifbcbot = bot;
      sd.ifbctop = top;
      h_penalty(ns, N, h->p, sd.eps, bot, top, pen);
      sd.tau1_bot = pen[4 * ns];
      sd.tau2_top = pen[5 * ns + ns - 1];
    }
    char* m = nullptr;
    if (dalloc(h, &m, at)) return IW_ERR_NOMEM;
    const cudaError_t e = scopy(h, m, host.data(), up_to, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
      cudaFree(m);
      return set_err(IW_ERR_CUDA, std::string("upload: ") + cudaGetErrorString(e));
    }
    h->bytes -= E.lu_bytes + (E.c.ab32 ? E.nlu * band * sizeof(float) : 0);
    cudaFree(E.lu);
    cudaFree(E.c.ab32);
    E.lu = m;
    E.lu_bytes = at;
    E.nlu = need;
    E.c.sys = (SysDesc*)(m + osys);
    E.c.pen = (double*)(m + open);
    E.c.ab = (double*)(m + oab);
    E.c.ipiv = (int*)(m + opiv);
    E.c.info = (int*)(m + oinfo);
    E.c.ab32 = nullptr;
    FactorArgs fa;
    fa.sys = E.c.sys;
    fa.pen = E.c.pen;
    fa.ab = E.c.ab;
    fa.nsys = need;
    fa.D = h->dD;
    fa.D2 = h->dD2;
    fa.zh = h->dzh;
    k_assemble_band<<<need, 128, 0, h->st>>>(geo(h), fa);
    launch_band_lu(h->st, need, n, N, E.c.ab, E.c.ipiv, E.c.info);
  }
  if (fp32 && !E.c.ab32) {
    if (dalloc(h, &E.c.ab32, E.nlu * band)) return IW_ERR_NOMEM;
    k_convert<double, float><<<2048, 256, 0, h->st>>>(E.c.ab, E.c.ab32, E.nlu * band);
  }
  CK(launch_error());
  return 0;
}

// Block inverses of the systems [first, nsys), their tasks and the columns of the other systems
static int helm_blocks(iw_handle* h, HelmEntry& E, int bot, int top) {
  if (E.tcm) return 0;
  const int N = h->N, ns = h->ns, m = 2 * (ns - 1), nt = E.nsys - E.first, ncol = (int)E.cs.size();
  const std::vector<int> order = helm_order(E);
  std::vector<Task> tasks;
  std::vector<int> list;
  for (int i = 0; i < ncol;) {
    const int u = E.cs[order[i]];
    int j = i;
    while (j < ncol && E.cs[order[j]] == u && j - i < kSysR / 2) ++j;
    if (u < E.first)
      list.insert(list.end(), order.begin() + i, order.begin() + j);
    else
      tasks.push_back(Task{u - E.first, i, j - i});
    i = j;
  }
  size_t at = 0;
  const size_t olam = carve(at, nt * sizeof(double)), otask = carve(at, tasks.size() * sizeof(Task)),
               olist = carve(at, list.size() * sizeof(int)), up_to = at;
  const size_t oainv = carve(at, (size_t)nt * h->nb * N * N * sizeof(double)),
               olvec = carve(at, (size_t)nt * m * N * sizeof(double)), ominv = carve(at, (size_t)nt * m * m * sizeof(double)),
               open = carve(at, (size_t)nt * 6 * ns * sizeof(double)), osys = carve(at, nt * sizeof(SysDesc));
  std::vector<char> host(up_to, 0);
  memcpy(host.data() + olam, E.lam.data() + E.first, nt * sizeof(double));
  memcpy(host.data() + otask, tasks.data(), tasks.size() * sizeof(Task));
  if (!list.empty()) memcpy(host.data() + olist, list.data(), list.size() * sizeof(int));
  if (!E.order && up(h, &E.order, order)) return IW_ERR_NOMEM;
  char* d = nullptr;
  if (dalloc(h, &d, at)) return IW_ERR_NOMEM;
  const cudaError_t e = scopy(h, d, host.data(), up_to, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(d);
    return set_err(IW_ERR_CUDA, std::string("upload: ") + cudaGetErrorString(e));
  }
  double* pen = (double*)(d + open);
  SysDesc* sys = (SysDesc*)(d + osys);
  if (int r = build_systems(h, (double*)(d + olam), nt, 0.0, bot, top, false, 0, (double*)(d + oainv), nullptr,
                            (double*)(d + olvec), (double*)(d + ominv), pen, sys)) {
    cudaFree(d);
    return r;
  }
  E.tcm = d;
  E.tasks = (Task*)(d + otask);
  E.ntask = (int)tasks.size();
  E.list = (int*)(d + olist);
  E.nlist = (int)list.size();
  E.ainv = (double*)(d + oainv);
  E.lvec = (double*)(d + olvec);
  E.minv = (double*)(d + ominv);
  E.pen = pen;
  E.sys = sys;
  return 0;
}

static int helm_batched(iw_handle* h, const double* lam_dev, int ncol, int bot, int top, const double* rhs,
                        double* sol, int mode) {
  std::vector<double> lam(ncol);
  CK(scopy(h, lam.data(), lam_dev, ncol * sizeof(double), cudaMemcpyDeviceToHost));
  // key: the lambda set and BCs
  uint64_t hs = 1469598103934665603ULL;
  for (double v : lam) {
    uint64_t b;
    memcpy(&b, &v, 8);
    hs = (hs ^ b) * 1099511628211ULL;
  }
  char kb[96];
  snprintf(kb, sizeof kb, "%d|%d|%d|%llx", ncol, bot, top, (unsigned long long)hs);
  auto key = std::make_pair(h, std::string(kb));
  const int n = h->nz, N = h->N, ns = h->ns;
  HelmEntry* found = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_helm_mu);
    auto it = g_helm.find(key);
    if (it != g_helm.end()) found = &it->second;
  }
  if (!found) {
    HelmEntry E;
    E.lam = lam;
    std::sort(E.lam.begin(), E.lam.end());
    E.lam.erase(std::unique(E.lam.begin(), E.lam.end()), E.lam.end());
    E.nsys = (int)E.lam.size();
    E.cs.resize(ncol);
    for (int c = 0; c < ncol; ++c) E.cs[c] = (int)(std::lower_bound(E.lam.begin(), E.lam.end(), lam[c]) - E.lam.begin());
    // Block inverses (system-grouped, on the tensor cores) for the systems whose estimated condition
    // needs no residual sweep, as in the time step; the others keep the pivoted band LU.
    const bool tc = h->ns <= 16 && N <= kTcMaxN && n <= kSysMaxRows &&
                    helm_smem(n, N, ns, h->nb).total <= 200 * 1024;
    const double rho = cond_slope(h);
    E.first = E.nsys;
    if (tc)
      while (E.first > 0 && E.lam[E.first - 1] > 0 && 1.0 + rho / E.lam[E.first - 1] <= kRefineCond) --E.first;
    if (up(h, &E.c.colsys, E.cs)) return IW_ERR_NOMEM;
    std::lock_guard<std::mutex> lk(g_helm_mu);
    found = &g_helm.emplace(key, std::move(E)).first->second;
  }
  HelmEntry& E = *found;
  // k_helm_tc copies whole complex values: 16-byte aligned columns
  const bool tc = mode == 0 && E.first < E.nsys && (((uintptr_t)rhs | (uintptr_t)sol) & 15) == 0;
  cudaStream_t st = h->st;  // of k_helm: beside k_helm_tc where the columns are split between them
  if (tc) {
    if (int r = helm_blocks(h, E, bot, top)) return r;
    HelmTc H;
    memset(&H, 0, sizeof H);
    H.ainv = E.ainv;
    H.lvec = E.lvec;
    H.minv = E.minv;
    H.pen = E.pen;
    H.sys = E.sys;
    H.D = h->dD;
    H.D2t = h->dD2t;
    H.zh = h->dzh;
    H.tasks = E.tasks;
    H.order = E.order;
    H.rhs = rhs;
    H.sol = sol;
    H.nb = h->nb;
    memcpy(H.bmap, h->bmap, sizeof H.bmap);
    // the factors of the other systems first: after a failure nothing of the solution is written
    if (E.nlist > 0)
      if (int r = helm_lu(h, E, E.first, false, bot, top)) return r;
    if (E.nlist > 0) st = side_fork(h);
    launch_helm_tc<double>(h, H, E.ntask);
    CK(launch_error());
  } else if (int r = helm_lu(h, E, E.nsys, mode != 0, bot, top)) {
    return r;
  }
  const int nc = tc ? E.nlist : ncol;
  const int warps = 4;
  const size_t sm32 = helm32_smem(n, N), smem = (size_t)warps * 6 * n * sizeof(double);
  // Mode 1 by the number of columns.  k_helm (a warp per column) is a short chain, k_helm32 (a lane per right-hand
  // side) a two to five times longer one that the whole chip's columns share.  k_helm's columns come in waves of what is
  // resident (two CTAs of four warps per SM, one where shared memory holds no more); from the second wave on the
  // longer chain is the cheaper one, without its prefetch (N > 33) from the fourth.  Both give the same bits.
  // us, k_helm / k_helm32, at 64, 1024 and 2048 columns (148 SMs: 1184 a wave): N = 9, ns = 12 165/243, 182/249, 326/257;
  // N = 25, ns = 8 371/655, 403/672, 745/675; N = 33, ns = 12 749/1347, 808/1366, 1582/1401; at 1024, 3072 and 4096:
  // N = 36, ns = 4 330/1034, 889/1052, 1165/1078; N = 40, ns = 8 773/2575, 2345/2689, 3560/3513.
  const int wave = warps * h->nsm * (2 * smem <= 224 * 1024 ? 2 : 1);
  if (mode != 0 && sm32 <= 200 * 1024 && rhs != sol && ncol > (N <= 33 ? 1 : 3) * wave) {
    // (the prefetch of the next factor column costs 6 NB registers; beyond 33 it spills)
    auto* kern = N <= 9 ? k_helm32<9> : N <= 17 ? k_helm32<17> : N <= 25 ? k_helm32<25> : N <= 33 ? k_helm32<33> : k_helm32<0>;
    if (!E.order && up(h, &E.order, helm_order(E))) return IW_ERR_NOMEM;
    set_smem(kern, sm32);
    kern<<<(ncol + 15) / 16, 32, sm32, h->st>>>(geo(h), E.c, rhs, sol, ncol, h->dD2, h->dzh, E.order);
    CK(launch_error());
  } else if (nc > 0) {
    set_smem(k_helm, smem);
    k_helm<<<(nc + warps - 1) / warps, 32 * warps, smem, st>>>(geo(h), E.c, rhs, sol, nc, mode, h->dD2, h->dzh,
                                                               tc ? E.list : nullptr);
    if (st != h->st) side_join(h);
    CK(launch_error());
  }
  return 0;
}

// the isolated-solve tables of a handle that goes away
static void helm_free(iw_handle* h) {
  std::lock_guard<std::mutex> lk(g_helm_mu);
  for (auto it = g_helm.begin(); it != g_helm.end();) {
    if (it->first.first != h) {
      ++it;
      continue;
    }
    HelmEntry& E = it->second;
    for (void* p : {(void*)E.c.colsys, (void*)E.lu, (void*)E.c.ab32, (void*)E.order, (void*)E.tcm}) cudaFree(p);
    it = g_helm.erase(it);
  }
}

#include "iw_abi.inl"
#include "iw_restart.inl"
#include "iw_output.inl"
#include "iw_postp.inl"
#endif  // IW_INST
