// ddc_api.cu -- host side of the B200 ddCOSMO library: the C ABI of
// include/ddcosmo_gpu.h, the module state (context), the ddinit pipeline and
// the Jacobi/DIIS driver.  All device work runs on the context's stream.
#include <algorithm>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "ddc_internal.h"
#include "lebedev_orbits.inc"

using namespace ddc;

namespace {

struct HBuf {  // pinned host memory
  void* p = nullptr;
  size_t bytes = 0;
  ~HBuf() {
    if (p) cudaFreeHost(p);
  }
  cudaError_t ensure(size_t b) {
    if (b <= bytes) return cudaSuccess;
    if (p) cudaFreeHost(p);
    p = nullptr;
    bytes = 0;
    const cudaError_t e = cudaMallocHost(&p, b);
    if (e == cudaSuccess) bytes = b;
    return e;
  }
};
double now_s() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch())
      .count();
}

// ---------------------------------------------------------------------------
// Lebedev grid (llgrid, llgnew.f:5-91).  Each orbit record {code, a, b, v}
// expands to its Oh-symmetric points (gen_oh, llgnew.f:93-681): for every
// coordinate pattern ("shape") of the orbit, the signs of the non-zero
// coordinates are enumerated with the first non-zero coordinate varying
// fastest.  This reproduces the reference's point order, which fixes the
// order of the cavity points.
// ---------------------------------------------------------------------------
int snap_ngrid(int ngrid) {
  int best = 0, inear = 100000;
  for (int i = 0; i < LEB_NSIZES; i++) {
    int d = std::abs(leb_sizes[i] - ngrid);
    if (d < inear) {
      inear = d;
      best = i;
    }
  }
  return leb_sizes[best];
}

void expand_orbit(int code, double a, double b, double v, std::vector<double>& out) {
  // shapes: indices into {0, a, b, c}; 0 = zero coordinate
  static const int shapes1[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
  static const int shapes2[3][3] = {{0, 1, 1}, {1, 0, 1}, {1, 1, 0}};
  static const int shapes3[1][3] = {{1, 1, 1}};
  static const int shapes4[3][3] = {{1, 1, 2}, {1, 2, 1}, {2, 1, 1}};
  static const int shapes5[6][3] = {{1, 2, 0}, {2, 1, 0}, {1, 0, 2},
                                    {2, 0, 1}, {0, 1, 2}, {0, 2, 1}};
  static const int shapes6[6][3] = {{1, 2, 3}, {1, 3, 2}, {2, 1, 3},
                                    {2, 3, 1}, {3, 1, 2}, {3, 2, 1}};
  const int(*shp)[3] = nullptr;
  int nshape = 0;
  double c = 0.0;
  switch (code) {
    case 1: a = 1.0; shp = shapes1; nshape = 3; break;
    case 2: a = std::sqrt(0.5); shp = shapes2; nshape = 3; break;
    case 3: a = std::sqrt(1.0 / 3.0); shp = shapes3; nshape = 1; break;
    case 4: b = std::sqrt(1.0 - 2.0 * a * a); shp = shapes4; nshape = 3; break;
    case 5: b = std::sqrt(1.0 - a * a); shp = shapes5; nshape = 6; break;
    case 6: c = std::sqrt(1.0 - a * a - b * b); shp = shapes6; nshape = 6; break;
    default: return;
  }
  const double val[4] = {0.0, a, b, c};
  for (int s = 0; s < nshape; s++) {
    int nz[3], nnz = 0;
    for (int k = 0; k < 3; k++)
      if (shp[s][k]) nz[nnz++] = k;
    for (int sg = 0; sg < (1 << nnz); sg++) {
      double p[3];
      for (int k = 0; k < 3; k++) p[k] = val[shp[s][k]];
      for (int q = 0; q < nnz; q++)
        if (sg & (1 << q)) p[nz[q]] = -p[nz[q]];
      out.push_back(p[0]);
      out.push_back(p[1]);
      out.push_back(p[2]);
      out.push_back(v);
    }
  }
}

bool lebedev(int ngrid, std::vector<double>& g4) {
  int gi = -1;
  for (int i = 0; i < LEB_NSIZES; i++)
    if (leb_sizes[i] == ngrid) gi = i;
  if (gi < 0) return false;
  g4.clear();
  for (int o = 0; o < leb_orbit_cnt[gi]; o++) {
    const leb_orbit_rec& r = leb_orbits[leb_orbit_off[gi] + o];
    expand_orbit(r.code, r.a, r.b, r.v, g4);
  }
  const double pi = 4.0 * std::atan(1.0);
  for (size_t i = 3; i < g4.size(); i += 4) g4[i] = g4[i] * 4.0 * pi;
  return (int)(g4.size() / 4) == ngrid;
}

}  // namespace

// ---------------------------------------------------------------------------
// context (the module state of ddcosmo.f90:87-127)
// ---------------------------------------------------------------------------
struct ddc_ctx {
  ddc_params prm{};
  YlmTables tb{};
  cudaStream_t st = nullptr;
  bool own_stream = true;
  long long launches = 0;
  // stage timers: event pairs recorded around stages, resolved at sync points
  std::vector<cudaEvent_t> ev_pool;
  std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> ev_pending;
  double st_ms[ST_N] = {0};
  long long st_calls[ST_N] = {0};
  std::string err;
  bool ready = false;
  bool tables_ready = false;  // static_tables done
  bool far_tables = false;    // farBT, farDT built
  int nsph = 0, ncav = 0, nylm = 0, ngrid = 0, npair = 0;
  long long ntri = 0;
  std::vector<double> h_grid;  // x,y,z,w per point
  DBuf gpos;                   // position of each Lebedev point in the patch-ordered grid
  // geometry
  bool order_on = false;
  DBuf ls_order;
  DBuf sph, grid, basis, bw, fi, ui, zi, inl, nl, rev, pn_ptr, pn, ls_ptr, ls, ntri_pt, pt_ptr,
      pt_idx;
  DBuf lsstart, fxa, fda, fvec;
  DBuf pcnt;     // triples per pair (ddinit scratch)
  DBuf pn_bits;  // per pair, which grid points lie inside the neighbour (ddinit scratch)
  // batched molecules: partition, per-target N-body ranges, per-molecule DIIS state
  int nmol = 1;
  bool batch_init = false;  // set while ddc_batch_energy_forces initialises
  bool batch = false;       // the solve belongs to ddc_batch_energy_forces
  std::vector<int> h_off;
  DBuf b_sphmol;        // molecule of each sphere (batched solves)
  DBuf b_cmol, b_cfirst;  // molecule of each solver chunk, first chunk of each molecule
  // state of the Jacobi/DIIS solves (SolverSys), both systems side by side
  DBuf s_int, s_dbl, s_slot, s_gram, s_coef, s_part, s_log;
  HBuf hstate;           // the solver's state on the host
  int* hstop = nullptr;  // mapped host memory: [2] stop reports, [2] active counts
  int* dstop = nullptr;
  cudaEvent_t ev_sweep[4] = {};
  SweepMask sweep{};    // set while a solver sweep is launched
  DBuf d_off, mrange, tr_cav, tr_nuc, b_out;
  const int2* mrange_ptr() const { return nmol > 1 ? mrange.as<int2>() : nullptr; }
  DBuf cavoff, cavidx, cavpt, ccav, cnt, scan_tmp;
  DBuf csph, cx, cy, cz;  // csph(3,n) and SoA centres
  // work
  DBuf pot, xig, gbuf, rhs, y, partials, red, hist_x, hist_e;
  DBuf phi, psi, sigma, s, q, fx, zeta, ef1, ef2, ef_scratch, uchi;
  DBuf in1, in2, in3, in4, out1;  // staging for host-pointer calls
  // mixed precision: FP32 basis copy, FP32 grid fields, refinement vectors
  DBuf bw_f, pot_f, xi_f, rres, eres;
  // static geometry of the gather-list triples: FP32 (mixed path)
  DBuf tgeo4;
  bool tgeo_on = false;
  // and FP64 (FP64 path)
  DBuf tgeo4d;
  bool tgeo64_on = false;
  // second solve set (direct and adjoint solved together) and the fused
  // operator's per-triple lx values
  DBuf y2, hist_x2, hist_e2, rres2, eres2, tval;
  // the two dense contractions of every operator application (projection
  // onto the harmonics, expansion to the grid): the folded kernels' tables;
  // tc plans the tensor-core kernels of the mixed path, whose FP32 grid field
  // pot_f has rows ldp_f floats apart
  FoldTab fold{};
  DBuf fold_img, fold_first, fold_lm, fold_p, fold_xw, fold_xb;
  TcPlan tc;
  bool fold_f32 = false;  // mixed: the folded kernels too
  int ldp_f = 0;
  // learned initial guess: the attached model, its feature rows, and flags
  // for the flows (rhs/psi/sigma/s of the last flow are valid; the initial
  // guesses are already in place)
  ddc_guess* gmodel = nullptr;
  DBuf gfeat;
  bool have_flow = false, guess_preset = false;
  // near / far split of the solute potential and field at the cavity:
  // tables of degree kFarDegree on the grid, the per-sphere expansions
  YlmTables tbP{};
  DBuf farBT, farDT, farA;
  bool far_on = false;
  // grouped multipole field of zeta at the nuclei (mixed energy+force flow)
  DBuf zg_cell, zg_sph, zg_start, zg_cen, zg_npt, zg_ptr, zg_cnt, zg_tmp, zg_M, zg_pk, zg_scr;
  ZGroups zg;
  bool zg_on = false;  // cell groups built for this molecule (single molecule, >= 4,096 spheres)
  bool zfar_on = false;
  // pinned landing buffer of the small device-to-host reads (reduced sums)
  double* hred = nullptr;
  // second stream of the force tail: the field of zeta at the nuclei runs
  // beside the force kernels (events: fork after zeta, join before its use)
  cudaStream_t st2 = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  cudaStream_t st_out = nullptr;  // results to the host beside the force kernels
  cudaEvent_t ev_out = nullptr;
  cudaEvent_t ev_mark[3] = {};    // ends of the phases of a run
  unsigned int stage_mask = ~0u;  // stages timed when prm.timing is set

  Launch L() { return Launch{st, &launches}; }
  DevGeo geo() const {
    DevGeo g;
    g.nsph = nsph;
    g.ngrid = ngrid;
    g.nylm = nylm;
    g.ncav = ncav;
    g.npair = npair;
    g.ntri = ntri;
    g.sph = sph.as<double4>();
    g.grid = grid.as<double4>();
    g.basis = basis.as<double>();
    g.bw = bw.as<double>();
    g.fi = fi.as<double>();
    g.ui = ui.as<double>();
    g.zi = zi.as<double>();
    g.inl = inl.as<int>();
    g.nl = nl.as<int>();
    g.rev = rev.as<int>();
    g.pn_ptr = pn_ptr.as<int>();
    g.pn = pn.as<uint16_t>();
    g.pt_ptr = pt_ptr.as<int>();
    g.pt_idx = pt_idx.as<int>();
    g.tgeo4 = tgeo_on ? tgeo4.as<float4>() : nullptr;
    g.tgeo4d = tgeo64_on ? tgeo4d.as<double4>() : nullptr;
    g.ls_ptr = ls_ptr.as<int>();
    g.ls_order = order_on ? ls_order.as<int>() : nullptr;
    g.ls = ls.as<int>();
    g.lsstart = lsstart.as<int>();
    g.ntri_pt = ntri_pt.as<uint8_t>();
    g.cavoff = cavoff.as<int>();
    g.cavidx = cavidx.as<int>();
    g.cavpt = cavpt.as<int>();
    g.ccav = ccav.as<double>();
    g.act = sweep;
    return g;
  }
};

namespace {

int fail(ddc_ctx* c, int code, const std::string& msg) {
  if (c) c->err = msg;
  return code;
}

// On failure the runtime's last-error state is cleared as well, so that a
// rejected launch configuration does not resurface in a later call.
#define CK(expr)                                                                          \
  do {                                                                                    \
    cudaError_t _e = (expr);                                                              \
    if (_e != cudaSuccess) {                                                              \
      cudaGetLastError();                                                                 \
      return fail(ctx, _e == cudaErrorMemoryAllocation ? DDC_ERR_NOMEM : DDC_ERR_CUDA,    \
                  std::string(#expr) + ": " + cudaGetErrorString(_e));                    \
    }                                                                                     \
  } while (0)

#define CKI(expr)                  \
  do {                             \
    int _r = (expr);               \
    if (_r != DDC_OK) return _r;   \
  } while (0)

// input array: device pointer as is, host array copied into staging
int stage_in(ddc_ctx* ctx, const double* p, size_t count, DBuf& buf, const double** out) {
  if (count == 0) {
    *out = p;
    return DDC_OK;
  }
  if (!p) return fail(ctx, DDC_ERR_PARAM, "null input array");
  if (ctx->prm.device_pointers) {
    *out = p;
    return DDC_OK;
  }
  CK(buf.ensure(count * sizeof(double)));
  CK(cudaMemcpyAsync(buf.p, p, count * sizeof(double), cudaMemcpyHostToDevice, ctx->st));
  *out = buf.as<double>();
  return DDC_OK;
}
// output: device pointer written directly; host array via a device buffer
int out_ptr(ddc_ctx* ctx, double* p, size_t count, DBuf& buf, double** dev) {
  if (ctx->prm.device_pointers && p) {
    *dev = p;
    return DDC_OK;
  }
  CK(buf.ensure((count ? count : 1) * sizeof(double)));
  *dev = buf.as<double>();
  return DDC_OK;
}
int finish_out(ddc_ctx* ctx, double* p, const double* dev, size_t count) {
  if (p && dev != p && count)
    CK(cudaMemcpyAsync(p, dev, count * sizeof(double),
                       ctx->prm.device_pointers ? cudaMemcpyDeviceToDevice
                                                : cudaMemcpyDeviceToHost,
                       ctx->st));
  return DDC_OK;
}
// Stage-timer events are turned into times in batches: resolving them at
// every synchronisation would put that host work between a solver step's
// reduction and its next launch.
void resolve_timers(ddc_ctx* ctx) {
  for (auto& pe : ctx->ev_pending) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, pe.second.first, pe.second.second) == cudaSuccess) {
      ctx->st_ms[pe.first] += ms;
      ctx->st_calls[pe.first] += 1;
    }
    ctx->ev_pool.push_back(pe.second.first);
    ctx->ev_pool.push_back(pe.second.second);
  }
  ctx->ev_pending.clear();
}

int sync(ddc_ctx* ctx) {
  CK(cudaStreamSynchronize(ctx->st));
  if (ctx->tc.err_h && *ctx->tc.err_h) {
    const int code = *ctx->tc.err_h;
    *ctx->tc.err_h = 0;
    return fail(ctx, DDC_ERR_CUDA,
                "tensor-core contraction gave up waiting (code " + std::to_string(code) + ")");
  }
  if (ctx->ev_pending.size() >= 1024) resolve_timers(ctx);
  return DDC_OK;
}

// Times the enclosed launches on the context stream (when timing is on).
struct StageScope {
  ddc_ctx* c;
  int stage;
  cudaEvent_t a = nullptr, b = nullptr;
  cudaEvent_t take() {
    cudaEvent_t e = nullptr;
    if (!c->ev_pool.empty()) {
      e = c->ev_pool.back();
      c->ev_pool.pop_back();
    } else if (cudaEventCreate(&e) != cudaSuccess) {
      e = nullptr;
    }
    return e;
  }
  cudaStream_t on;
  StageScope(ddc_ctx* ctx, int s, cudaStream_t stream = nullptr)
      : c(ctx), stage(s), on(stream ? stream : ctx->st) {
    if (!c->prm.timing || !((c->stage_mask >> s) & 1u)) return;
    a = take();
    b = take();
    if (a && b) cudaEventRecord(a, on);
  }
  ~StageScope() {
    if (!a || !b) return;
    cudaEventRecord(b, on);
    c->ev_pending.push_back({stage, {a, b}});
  }
};

void build_tables_for(YlmTables& tb, int lmax, double eta, int ngrid) {
  memset(&tb, 0, sizeof(tb));
  const double pi = 4.0 * std::atan(1.0), sq2 = std::sqrt(2.0);
  std::vector<double> fact(std::max(2 * lmax + 1, 2));
  fact[0] = 1.0;
  fact[1] = 1.0;
  for (int i = 3; i <= 2 * lmax + 1; i++) fact[i - 1] = (double)(i - 1) * fact[i - 2];
  for (int l = 0; l <= lmax; l++) {
    double fl = (2.0 * (double)l + 1.0) / (4.0 * pi);
    double ffl = std::sqrt(fl);
    tb.facl[l] = fl;
    tb.facs[l * (l + 1) / 2] = ffl;
    for (int m = 1; m <= l; m++) {
      double fnorm = sq2 * ffl * std::sqrt(fact[l - m] / fact[l + m]);
      if (m % 2 == 1) fnorm = -fnorm;
      tb.facs[l * (l + 1) / 2 + m] = fnorm;
    }
    for (int m = 0; m <= l; m++) {
      int e = l * (l + 1) / 2 + m;
      tb.K[e] = tb.facs[e] / fl;
      if (l >= m + 2) {
        tb.A[e] = (2.0 * l - 1.0) / (double)(l - m);
        tb.B[e] = ((double)(l + m) - 1.0) / (double)(l - m);
      }
    }
  }
  for (int m = 0; m <= lmax; m++) {
    double gm2 = 1.0, gm1 = 1.0;  // gam_{l-2}, gam_{l-1}
    for (int l = m; l <= lmax; l++) {
      const int e = l * (l + 1) / 2 + m;
      double gam;
      if (l == m) {
        gam = 1.0;
      } else if (l == m + 1) {
        gam = 2.0 * m + 1.0;
      } else {
        gam = tb.A[e] * gm1;
        tb.Bn[e] = tb.B[e] * gm2 / gam;
      }
      tb.Kg[e] = tb.K[e] * gam;
      gm2 = gm1;
      gm1 = gam;
    }
  }
  double pre = 1.0;  // (-1)^m (2m-1)!!
  for (int m = 0; m <= lmax; m++) {
    if (m > 0) pre *= -(2.0 * m - 1.0);
    for (int l = m; l <= lmax; l++) tb.Kp[l * (l + 1) / 2 + m] = pre * tb.Kg[l * (l + 1) / 2 + m];
  }
  tb.eta = eta;
  tb.lmax = lmax;
  tb.nylm = (lmax + 1) * (lmax + 1);
  tb.ngrid = ngrid;
}
void build_tables(ddc_ctx* c) {
  build_tables_for(c->tb, c->prm.lmax, c->prm.eta, c->ngrid);
  // the degree of the far-field expansions of the solute potential
  build_tables_for(c->tbP, kFarDegree, c->prm.eta, c->ngrid);
}

// the sum of the blocks' partial sums, in a fixed order, to hred[0]
int reduce_to_pinned(ddc_ctx* ctx) {
  {
    StageScope sc(ctx, ST_REDUCE);
    CK(launch_reduce_partials(ctx->L(), ctx->partials.as<double>(), reduce_blocks(),
                              ctx->red.as<double>()));
  }
  CK(cudaMemcpyAsync(ctx->hred, ctx->red.p, sizeof(double), cudaMemcpyDeviceToHost, ctx->st));
  return DDC_OK;
}
int reduce_to_host(ddc_ctx* ctx, double* host) {
  CKI(reduce_to_pinned(ctx));
  CKI(sync(ctx));
  *host = ctx->hred[0];
  return DDC_OK;
}

// The per-item counts scanned into 32-bit offsets must total less than 2^31.
int check_count_total(ddc_ctx* ctx, unsigned long long total, const char* what) {
  if (total >= (unsigned long long)INT_MAX)
    return fail(ctx, DDC_ERR_UNSUPPORTED,
                std::string("more than 2^31 - 1 ") + what + " (" + std::to_string(total) + ")");
  return DDC_OK;
}

// most products (harmonics x spheres x grid points) of a contraction that the
// mixed operators fold
constexpr long long kFoldProducts = 200000000;

// What depends on the parameters alone (degree, grid, eta), once per context:
// the constants, the grid, the basis with its transposes and weights.
int static_tables(ddc_ctx* ctx) {
  if (ctx->tables_ready) return DDC_OK;
  const int G = ctx->ngrid, NY = ctx->nylm;
  auto L = ctx->L();
  build_tables(ctx);
  CK(prepare_lxs(ctx->prm.lmax));
  if (!lebedev(G, ctx->h_grid)) return fail(ctx, DDC_ERR_PARAM, "bad Lebedev size");
  CK(ctx->grid.ensure(sizeof(double4) * G));
  CK(ctx->gpos.ensure(sizeof(int) * G));
  {
    // the grid octant by octant, in each by the Morton order of the points'
    // absolute coordinates: 32 consecutive points form a compact patch of the
    // sphere, so that a warp's points lie inside nearly the same neighbours
    // (k_fiui skips together those that miss the patch; the triple values, the
    // fields and the point lists that consecutive threads read are adjacent),
    // and the mirror images of consecutive points are consecutive
    std::vector<std::pair<uint64_t, int>> key(G);
    for (int k = 0; k < G; k++) {
      uint64_t m = 0;
      uint32_t c[3];
      for (int d = 0; d < 3; d++) {
        const double x = ctx->h_grid[4 * k + d];
        if (x < 0.0) m |= 1u << d;
        c[d] = (uint32_t)std::min(1023.0, std::floor(std::fabs(x) * 1023.5));
      }
      for (int b = 9; b >= 0; b--)
        for (int d = 0; d < 3; d++) m = (m << 1) | ((c[d] >> b) & 1u);
      key[k] = {m, k};
    }
    std::sort(key.begin(), key.end());
    std::vector<double> g4(4 * (size_t)G);
    std::vector<int> gpos(G);
    for (int k = 0; k < G; k++) {
      gpos[key[k].second] = k;
      for (int d = 0; d < 4; d++) g4[4 * k + d] = ctx->h_grid[4 * key[k].second + d];
    }
    CK(cudaMemcpyAsync(ctx->grid.p, g4.data(), sizeof(double4) * G, cudaMemcpyHostToDevice,
                       ctx->st));
    CK(cudaMemcpyAsync(ctx->gpos.p, gpos.data(), sizeof(int) * G, cudaMemcpyHostToDevice,
                       ctx->st));
    std::vector<short> img, lm;
    std::vector<uint8_t> first;
    if (!fold_tables(g4, ctx->prm.lmax, ctx->fold, img, first, lm))
      return fail(ctx, DDC_ERR_STATE, "the grid is not symmetric under reflections");
    auto upload = [&](DBuf& b, const auto& v) -> int {
      CK(b.ensure(v.size() * sizeof(v[0])));
      CK(cudaMemcpyAsync(b.p, v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice, ctx->st));
      return DDC_OK;
    };
    CKI(upload(ctx->fold_img, img));
    CKI(upload(ctx->fold_first, first));
    CKI(upload(ctx->fold_lm, lm));
    ctx->fold.img = ctx->fold_img.as<short>();
    ctx->fold.first = ctx->fold_first.as<uint8_t>();
    ctx->fold.lm = ctx->fold_lm.as<short>();
  }
  CK(ctx->basis.ensure(sizeof(double) * G * NY));
  CK(ctx->bw.ensure(sizeof(double) * G * NY));
  CK(launch_basis(L, ctx->tb, ctx->grid.as<double4>(), ctx->basis.as<double>(),
                  ctx->bw.as<double>()));
  CK(ctx->fold_p.ensure(sizeof(double) * ctx->fold.psize));
  CK(ctx->fold_xw.ensure(sizeof(double) * ctx->fold.xsize));
  CK(ctx->fold_xb.ensure(sizeof(double) * ctx->fold.xsize));
  CK(launch_fold_pack(L, ctx->fold, ctx->basis.as<double>(), ctx->bw.as<double>(),
                      ctx->fold_p.as<double>(), ctx->fold_xw.as<double>(),
                      ctx->fold_xb.as<double>()));
  ctx->fold.pf = ctx->fold_p.as<double>();
  ctx->fold.xfw = ctx->fold_xw.as<double>();
  ctx->fold.xfb = ctx->fold_xb.as<double>();
  ctx->tables_ready = true;
  return DDC_OK;
}

// ---------------------------------------------------------------------------
// ddinit (ddcosmo.f90:159-483) on device buffers
// ---------------------------------------------------------------------------
int do_init(ddc_ctx* ctx, int n, const std::vector<double4>& hsph) {
  ctx->ready = false;
  ctx->tgeo_on = false;
  ctx->tgeo64_on = false;
  ctx->nsph = n;
  ctx->nylm = (ctx->prm.lmax + 1) * (ctx->prm.lmax + 1);
  ctx->ngrid = snap_ngrid(ctx->prm.ngrid);
  const int N = n, G = ctx->ngrid, NY = ctx->nylm;
  const long long NP = (long long)N * G;
  // grid fields, cavity and triple lists are indexed with 32-bit integers
  if (NP >= (long long)INT_MAX)
    return fail(ctx, DDC_ERR_UNSUPPORTED, "nsph * ngrid exceeds 2^31 - 1 grid points");
  if (!ctx->hred) CK(cudaMallocHost(&ctx->hred, sizeof(double) * 2 * (kMaxHist + 1)));
  CK(ctx->red.ensure(sizeof(double) * 2 * (kMaxHist + 1)));
  // red holds the counts' totals during ddinit: [0] pairs, [1] cavity points,
  // [2] triples
  CountStats* stats = ctx->red.as<CountStats>();
  CountStats* hstats = reinterpret_cast<CountStats*>(ctx->hred);
  auto L = ctx->L();
  CK(ctx->sph.ensure(sizeof(double4) * std::max(N, 1)));
  CK(cudaMemcpyAsync(ctx->sph.p, hsph.data(), sizeof(double4) * N, cudaMemcpyHostToDevice,
                     ctx->st));
  CKI(static_tables(ctx));
  // cell groups of one large molecule: candidates for the neighbour list,
  // the near lists of the cavity far field and the groups of the field of
  // zeta (DDC_CELLS_OFF=1 keeps the all-pairs scans: a diagnostic switch)
  {
    const char* coff = std::getenv("DDC_CELLS_OFF");
    ctx->zg_on = ctx->nmol <= 1 && N >= kZetaMinSpheres && !(coff && coff[0] == '1');
    if (ctx->zg_on) {
      CK(ctx->zg_cell.ensure(sizeof(int) * N));
      CK(ctx->zg_sph.ensure(sizeof(int) * N));
      CK(ctx->zg_start.ensure(sizeof(int) * (N + 1)));
      CK(ctx->zg_cen.ensure(sizeof(double4) * N));
      CK(ctx->zg_cnt.ensure(sizeof(int)));
      ZGroups& z = ctx->zg;
      z.cellid = ctx->zg_cell.as<int>();
      z.gsph = ctx->zg_sph.as<int>();
      z.gstart = ctx->zg_start.as<int>();
      z.gcen = ctx->zg_cen.as<double4>();
      z.gnpt = nullptr;
      z.gptr = nullptr;
      CK(launch_zgroups_cells(L, N, ctx->sph.as<double4>(), z, ctx->zg_cnt.as<int>(),
                              reinterpret_cast<int*>(ctx->hred)));
    }
  }
  // neighbour list
  CK(ctx->cnt.ensure(sizeof(int) * (N + 1)));
  CK(ctx->inl.ensure(sizeof(int) * (N + 1)));
  if (N > 0) {
    if (ctx->zg_on)
      CK(launch_csr_count_cells(L, N, ctx->sph.as<double4>(), ctx->zg, ctx->cnt.as<int>()));
    else
      CK(launch_csr_count(L, N, ctx->sph.as<double4>(), ctx->cnt.as<int>(), ctx->mrange_ptr()));
  }
  size_t tb_bytes = scan_temp_bytes(N);
  CK(ctx->scan_tmp.ensure(tb_bytes));
  CK(scan_counts(L, ctx->cnt.as<int>(), ctx->inl.as<int>(), N, ctx->scan_tmp.p, tb_bytes, stats));
  CK(cudaMemcpyAsync(hstats, stats, sizeof(CountStats), cudaMemcpyDeviceToHost, ctx->st));
  CKI(sync(ctx));
  CKI(check_count_total(ctx, hstats[0].total, "neighbour pairs"));
  const int npair = (int)hstats[0].total;
  ctx->npair = npair;
  CK(ctx->nl.ensure(sizeof(int) * std::max(npair, 1)));
  CK(ctx->rev.ensure(sizeof(int) * std::max(npair, 1)));
  {
    // a point's triples are counted with 8 bits (the reference
    // caps the list at nngmax = 100 per sphere on average, ddcosmo.f90:87)
    const int mx = hstats[0].largest;
    const size_t smem = 32 * (size_t)mx + 4 * (size_t)mx + 32 * (size_t)G;
    if (mx > 255 || smem > 200 * 1024)
      return fail(ctx, DDC_ERR_UNSUPPORTED, "a sphere has too many neighbours (" +
                                                std::to_string(mx) + ")");
  }
  if (N > 0) {
    if (ctx->zg_on)
      CK(launch_csr_fill_cells(L, N, ctx->sph.as<double4>(), ctx->zg, ctx->inl.as<int>(),
                               ctx->nl.as<int>()));
    else
      CK(launch_csr_fill(L, N, ctx->sph.as<double4>(), ctx->inl.as<int>(), ctx->nl.as<int>(),
                         ctx->mrange_ptr()));
    CK(launch_csr_rev(L, N, ctx->inl.as<int>(), ctx->nl.as<int>(), ctx->rev.as<int>()));
  }
  // fi, ui, zi
  CK(ctx->fi.ensure(sizeof(double) * std::max(NP, 1LL)));
  CK(ctx->ui.ensure(sizeof(double) * std::max(NP, 1LL)));
  CK(ctx->ntri_pt.ensure(std::max(NP, 1LL)));
  if (ctx->prm.igrad) CK(ctx->zi.ensure(sizeof(double) * 3 * std::max(NP, 1LL)));
  else ctx->zi.release();
  CK(launch_fiui(L, ctx->tb, N, ctx->sph.as<double4>(), ctx->grid.as<double4>(),
                 ctx->inl.as<int>(), ctx->nl.as<int>(), ctx->fi.as<double>(),
                 ctx->ui.as<double>(),
                 ctx->prm.igrad ? ctx->zi.as<double>() : nullptr, ctx->ntri_pt.as<uint8_t>()));
  // cavity counts, and the pair-major triple lists' counts
  CK(ctx->cavoff.ensure(sizeof(int) * (N + 1)));
  CK(launch_cav_count(L, N, G, ctx->ui.as<double>(), ctx->cnt.as<int>()));
  CK(scan_counts(L, ctx->cnt.as<int>(), ctx->cavoff.as<int>(), N, ctx->scan_tmp.p, tb_bytes,
                 stats + 1));
  CK(ctx->pcnt.ensure(sizeof(int) * ((size_t)npair + 1)));
  CK(ctx->pn_ptr.ensure(sizeof(int) * ((size_t)npair + 1)));
  CK(ctx->pn_bits.ensure(sizeof(unsigned) * std::max(npair, 1) * (size_t)((G + 31) / 32)));
  CK(launch_pair_count(L, N, npair, G, ctx->sph.as<double4>(), ctx->grid.as<double4>(),
                       ctx->inl.as<int>(), ctx->nl.as<int>(), ctx->pcnt.as<int>(),
                       ctx->pn_bits.as<unsigned>()));
  CK(ctx->scan_tmp.ensure(std::max(tb_bytes, scan_temp_bytes(npair))));
  CK(scan_counts(L, ctx->pcnt.as<int>(), ctx->pn_ptr.as<int>(), npair, ctx->scan_tmp.p,
                 ctx->scan_tmp.bytes, stats + 2));
  CK(cudaMemcpyAsync(hstats + 1, stats + 1, 2 * sizeof(CountStats), cudaMemcpyDeviceToHost,
                     ctx->st));
  CKI(sync(ctx));
  CKI(check_count_total(ctx, hstats[2].total, "(sphere, point, neighbour) triples"));
  const int ncav = (int)hstats[1].total, ntri = (int)hstats[2].total;
  ctx->ncav = ncav;
  ctx->ntri = ntri;
  CK(ctx->cavidx.ensure(sizeof(int) * std::max(NP, 1LL)));
  CK(ctx->cavpt.ensure(sizeof(int) * std::max(ncav, 1)));
  CK(ctx->ccav.ensure(sizeof(double) * 3 * std::max(ncav, 1)));
  CK(launch_cav_fill(L, N, G, ctx->gpos.as<int>(), ctx->ui.as<double>(), ctx->sph.as<double4>(),
                     ctx->grid.as<double4>(), ctx->cavoff.as<int>(), ctx->cavidx.as<int>(),
                     ctx->cavpt.as<int>(), ctx->ccav.as<double>()));
  CK(ctx->pn.ensure(sizeof(uint16_t) * std::max(ntri, 1)));
  CK(launch_pair_fill(L, N, npair, G, ctx->sph.as<double4>(), ctx->grid.as<double4>(),
                      ctx->inl.as<int>(), ctx->nl.as<int>(), ctx->pn_bits.as<unsigned>(),
                      ctx->pn_ptr.as<int>(), ctx->pn.as<uint16_t>()));
  CK(ctx->ls_ptr.ensure(sizeof(int) * (N + 1)));
  CK(launch_ls_count(L, N, ctx->inl.as<int>(), ctx->rev.as<int>(), ctx->pn_ptr.as<int>(),
                     ctx->cnt.as<int>()));
  CK(scan_counts(L, ctx->cnt.as<int>(), ctx->ls_ptr.as<int>(), N, ctx->scan_tmp.p,
                 ctx->scan_tmp.bytes, stats));
  // The triple passes take the longest lists first: the blocks of a last wave
  // are then the shortest.  The pass gains at every size (lx alone 4 to 15 %, lmax
  // 8 and 10), whole solves only with enough spheres; why few lose was not
  // traced.  ms to 1e-9 by rising index / longest first:
  //   energy and forces (both systems), 302 points:
  //     lmax 6, FP64     2,000 spheres 8.87 / 8.03, 5,000 16.8 / 15.8
  //     lmax 6, mixed    900 4.42 / 4.65, 1,184 5.06 / 5.33, 1,300 4.41 / 4.33, 2,000 7.16 / 6.66
  //     lmax 8, FP64     320 3.89 / 4.22, 643 4.93 / 5.05, 900 5.55 / 5.25, 2,000 11.0 / 10.2
  //     lmax 10, mixed   320 4.04 / 4.20, 643 5.03 / 4.92, 2,000 10.4 / 9.9
  //   one system (cosmo):
  //     lmax 6, FP64, 110 points  643 2.17 / 2.69, 1,300 2.60 / 2.83, 1,600 3.53 / 3.77, 2,000 4.06 / 3.94
  //     lmax 8, FP64     643 3.43 / 3.64, 900 3.56 / 3.70, 1,184 4.74 / 4.55, 2,000 7.55 / 6.78
  //     lmax 10, mixed   643 3.26 / 3.41, 900 3.58 / 3.45
  // So the line lies between 600 and 1,800 spheres, by degree, precision and
  // number of systems, and not at a number of waves (lmax 6 in FP32 has eight
  // blocks per SM, lmax 8 four); one line stands for all.  Nor where one block
  // would sort for long.
  ctx->order_on = N > 2 * 4 * 148 && N <= 65536;
  if (ctx->order_on) {
    CK(ctx->ls_order.ensure(sizeof(int) * N));
    CK(launch_ls_order(L, N, ctx->ls_ptr.as<int>(), stats, ctx->ls_order.as<int>()));
  }
  CK(ctx->ls.ensure(sizeof(int) * std::max(ntri, 1)));
  CK(ctx->lsstart.ensure(sizeof(int) * std::max(npair, 1)));
  CK(launch_ls_fill(L, N, ctx->inl.as<int>(), ctx->nl.as<int>(), ctx->rev.as<int>(),
                    ctx->pn_ptr.as<int>(), ctx->pn.as<uint16_t>(), ctx->ls_ptr.as<int>(), G,
                    ctx->ls.as<int>(), ctx->lsstart.as<int>()));
  CK(ctx->pt_ptr.ensure(sizeof(int) * (size_t)(NP + 1)));
  CK(ctx->pt_idx.ensure(sizeof(int) * std::max(ntri, 1)));
  CK(launch_pt_fill(L, N, G, ctx->inl.as<int>(), ctx->pn_ptr.as<int>(), ctx->pn.as<uint16_t>(),
                    ctx->lsstart.as<int>(), ctx->ntri_pt.as<uint8_t>(), ctx->pt_ptr.as<int>(),
                    ctx->pt_idx.as<int>()));
  // centres for the electrostatics
  CK(ctx->csph.ensure(sizeof(double) * 3 * std::max(N, 1)));
  CK(ctx->cx.ensure(sizeof(double) * std::max(N, 1)));
  CK(ctx->cy.ensure(sizeof(double) * std::max(N, 1)));
  CK(ctx->cz.ensure(sizeof(double) * std::max(N, 1)));
  CK(launch_csph_pack(L, N, ctx->sph.as<double4>(), ctx->csph.as<double>(), ctx->cx.as<double>(),
                      ctx->cy.as<double>(), ctx->cz.as<double>()));
  // solver work buffers
  const size_t nv = (size_t)N * NY;
  const int nd = std::max(ctx->prm.ndiis, 1);
  CK(ctx->pot.ensure(sizeof(double) * std::max(NP, 1LL)));
  CK(ctx->xig.ensure(sizeof(double) * std::max(NP, 1LL)));
  CK(ctx->uchi.ensure(sizeof(double) * std::max(NP, 1LL)));
  for (DBuf* b : {&ctx->rhs, &ctx->y, &ctx->psi, &ctx->sigma, &ctx->s})
    CK(b->ensure(sizeof(double) * std::max(nv, (size_t)1)));
  CK(ctx->hist_x.ensure(sizeof(double) * std::max(nv, (size_t)1) * nd));
  CK(ctx->hist_e.ensure(sizeof(double) * std::max(nv, (size_t)1) * nd));
  CK(ctx->partials.ensure(sizeof(double) * reduce_blocks()));
  CK(ctx->red.ensure(sizeof(double) * 2 * (kMaxHist + 1)));
  if (ctx->prm.igrad && !ctx->st2) {
    CK(cudaStreamCreateWithFlags(&ctx->st2, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&ctx->ev_fork, cudaEventDisableTiming));
    CK(cudaEventCreateWithFlags(&ctx->ev_join, cudaEventDisableTiming));
  }
  if (ctx->prm.precision == DDC_PREC_MIXED) {
    // The two contractions of the FP32 operators: folded (FP64 arithmetic,
    // ddc_fold.cu) up to kFoldProducts products; above that on tcgen05 (split
    // TF32, ddc_tc.cu) up to 128 harmonics (lmax 10) and as FP32 SIMT GEMMs on an
    // FP32 copy of bw beyond.  The folded kernels' blocks are short, the tcgen05
    // ones' wide; projection + expansion us, folded against tcgen05, with 4 us of
    // events: lmax 6, 302 points, 8,000 spheres (1.2e8 products) 15 + 20 against
    // 21 + 20, 13,000 (1.9e8) 19 + 27 against 23 + 23, 18,000 (2.7e8) 24 + 35
    // against 24 + 25; lmax 8, 302 points, 18,000 (4.4e8) 27 + 36 against 25 + 31.
    // (lmax 10, 590 points is for the folded ones longer, 5,000 spheres, 3.6e8,
    // 24 + 25 against 29 + 35; 20,000, 1.4e9, 49 + 63 against 37 + 49.)  With few
    // harmonics only molecules of a size that no program solves pass the line
    // (lmax 0, 110 points: 1.8 million spheres).
    // Diagnostic switches of the environment, with which the tests compare the
    // paths: DDC_TC_OFF=1 takes the SIMT contractions at any size, DDC_FOLD=0
    // never folds, DDC_FOLD=1 always.
    const char* tc_off = std::getenv("DDC_TC_OFF");
    const char* fold = std::getenv("DDC_FOLD");
    const bool tc_env = !(tc_off && tc_off[0] == '1');
    ctx->fold_f32 = tc_env && (fold && fold[0] ? fold[0] == '1' : (long long)NY * NP <= kFoldProducts);
    const bool tc = tc_supported(NY) && tc_env && !ctx->fold_f32;
    ctx->ldp_f = tc ? (G + 3) / 4 * 4 : G;
    CK(ctx->pot_f.ensure(sizeof(float) * std::max<long long>((long long)N * ctx->ldp_f, 1LL)));
    CK(ctx->xi_f.ensure(sizeof(float) * std::max(NP, 1LL)));
    if (tc) {
      CK(tc_plan(L, ctx->tc, ctx->bw.as<double>(), N, NY, G,
                 ctx->pot_f.as<float>(), ctx->ldp_f));
      // tile widths by measurement (rhs and y are free work vectors here)
      CK(tc_autotune(L, ctx->tc, ctx->rhs.as<double>(), ctx->y.as<double>(),
                     ctx->xi_f.as<float>()));
    } else if (ctx->fold_f32) {
      ctx->tc.on = false;
    } else {
      ctx->tc.on = false;
      CK(ctx->bw_f.ensure(sizeof(float) * G * NY));
      CK(launch_to_float(L, (long long)G * NY, ctx->bw.as<double>(), ctx->bw_f.as<float>()));
    }
    for (DBuf* b : {&ctx->rres, &ctx->eres})
      CK(b->ensure(sizeof(double) * std::max(nv, (size_t)1)));
    // the FP32 fused pass reads each triple's static geometry instead of
    // recomputing it every iteration (16 bytes per triple)
    ctx->tgeo_on = false;
    CK(ctx->tgeo4.ensure(sizeof(float4) * std::max<long long>(ctx->ntri, 1)));
    CK(launch_lxs_geo(L, ctx->tb, ctx->geo(), ctx->tgeo4.as<float4>()));
    ctx->tgeo_on = true;
  }
  if (ctx->prm.precision != DDC_PREC_MIXED && ctx->prm.pair_solves) {
    // the FP64 fused pass of the paired solves reads each triple's static
    // geometry (32 bytes per triple) instead of recomputing it
    CK(ctx->tgeo4d.ensure(sizeof(double4) * std::max<long long>(ctx->ntri, 1)));
    CK(launch_lxs_geo_f64(L, ctx->tb, ctx->geo(), ctx->tgeo4d.as<double4>()));
    ctx->tgeo64_on = true;
  }
  if (ctx->prm.igrad && ctx->prm.pair_solves) {
    CK(ctx->y2.ensure(sizeof(double) * std::max(nv, (size_t)1)));
    CK(ctx->hist_x2.ensure(sizeof(double) * std::max(nv, (size_t)1) * nd));
    CK(ctx->hist_e2.ensure(sizeof(double) * std::max(nv, (size_t)1) * nd));
    if (ctx->prm.precision == DDC_PREC_MIXED)
      for (DBuf* b : {&ctx->rres2, &ctx->eres2})
        CK(b->ensure(sizeof(double) * std::max(nv, (size_t)1)));
  }
  // per-triple lx values of the fused passes (FP64 size: the mixed path also
  // takes FP64 steps in its refinement)
  CK(ctx->tval.ensure(sizeof(double) * std::max<long long>(ctx->ntri, 1)));
  // near / far split of the solute potential at the cavity for large systems
  // (DDC_FAR_OFF=1 in the environment keeps the direct sums: a diagnostic
  // switch for the tests)
  {
    const char* off = std::getenv("DDC_FAR_OFF");
    // a batch sums each molecule's own charges: the split pays only when one
    // of its molecules is large (the direct per-molecule sums of the
    // 256-globule batch, 1,952 spheres at most, take half the time of the
    // split, whose near lists hold most of each molecule)
    int largest = N;
    if (ctx->batch_init) {
      largest = 0;
      for (int k = 0; k < ctx->nmol; k++)
        largest = std::max(largest, ctx->h_off[k + 1] - ctx->h_off[k]);
    }
    ctx->far_on = largest >= kFarMinSpheres && G <= 640 && !(off && off[0] == '1');
    if (ctx->far_on) {
      const int YP = ctx->tbP.nylm;
      CK(ctx->farBT.ensure(sizeof(double) * YP * G));
      CK(ctx->farDT.ensure(sizeof(double) * 3 * YP * G));
      CK(ctx->farA.ensure(sizeof(double) * (size_t)YP * N));
      if (!ctx->far_tables)
        CK(launch_far_tables(L, ctx->tbP, ctx->grid.as<double4>(), G, ctx->farBT.as<double>(),
                             ctx->farDT.as<double>()));
      ctx->far_tables = true;
    }
    // the field of zeta at the nuclei of one large molecule in the mixed
    // flow: spheres grouped for the multipole far field (DDC_ZFAR_OFF=1, or
    // DDC_FAR_OFF=1, keeps the direct FP32 pair sums)
    const char* zoff = std::getenv("DDC_ZFAR_OFF");
    ctx->zfar_on = ctx->zg_on && ctx->prm.precision == DDC_PREC_MIXED && ctx->prm.igrad &&
                   !(off && off[0] == '1') && !(zoff && zoff[0] == '1');
    if (ctx->zfar_on) {
      CK(ctx->zg_npt.ensure(sizeof(int) * (N + 1)));
      CK(ctx->zg_ptr.ensure(sizeof(int) * (N + 1)));
      const size_t tb = zgroups_scan_bytes(N);
      CK(ctx->zg_tmp.ensure(tb));
      ZGroups& z = ctx->zg;
      z.gnpt = ctx->zg_npt.as<int>();
      z.gptr = ctx->zg_ptr.as<int>();
      CK(launch_zgroups_points(L, ctx->cavoff.as<int>(), z, ctx->zg_tmp.p, tb));
      CK(ctx->zg_M.ensure(sizeof(float2) * zgroups_moment_count(z)));
      CK(ctx->zg_pk.ensure(sizeof(float4) * std::max(ctx->ncav, 1)));
      CK(ctx->zg_scr.ensure(sizeof(double) * 3 * (size_t)zgroups_nchunk(z) * N));
    }
  }
  ctx->ready = true;
  return DDC_OK;
}

// ---------------------------------------------------------------------------
// the operators' two dense contractions, on the context's stream
// ---------------------------------------------------------------------------
// y(lm,i) = alpha sum_n bw(lm,n) pot(n,i): intrhs over every sphere
// (matvec.f90:131-135, bw = w_n Y_lm(s_n))
int gemm_proj(ddc_ctx* ctx, double alpha, const double* pot, double* y) {
  CK(launch_fold_proj(ctx->L(), ctx->fold, ctx->nsph, alpha, pot, ctx->ngrid, y, ctx->sweep));
  return DDC_OK;
}
// projection of the FP32 field (rows ldp_f apart) into the FP64 vector y
int gemm_proj_f32(ddc_ctx* ctx, float alpha, const float* pot, double* y) {
  if (ctx->fold_f32)
    CK(launch_fold_proj(ctx->L(), ctx->fold, ctx->nsph, (double)alpha, pot, ctx->ldp_f, y,
                        ctx->sweep));
  else if (ctx->tc.on)
    CK(launch_proj_tc(ctx->L(), ctx->tc, alpha, y, ctx->sweep));
  else
    CK(launch_proj_f32_simt(ctx->L(), ctx->nylm, ctx->nsph, ctx->ngrid, alpha,
                            ctx->bw_f.as<float>(), pot, ctx->ldp_f, y));
  return DDC_OK;
}
// xi(n,i) = sum_lm basis(lm,n) s(lm,i)   (matvec.f90:189-204); weighted: w_n xi
int gemm_xi(ddc_ctx* ctx, const double* s, double* xig, bool weighted) {
  CK(launch_fold_xi(ctx->L(), ctx->fold, weighted, ctx->nsph, s, xig, ctx->ngrid, ctx->sweep));
  return DDC_OK;
}
// FP32 w_n xi of the FP64 vector s
int gemm_xi_f32(ddc_ctx* ctx, const double* s, float* xig) {
  if (ctx->fold_f32)
    CK(launch_fold_xi(ctx->L(), ctx->fold, true, ctx->nsph, s, xig, ctx->ngrid, ctx->sweep));
  else if (ctx->tc.on)
    CK(launch_xi_tc(ctx->L(), ctx->tc, s, xig, ctx->sweep));
  else
    CK(launch_xi_f32_simt(ctx->L(), ctx->nylm, ctx->nsph, ctx->ngrid, ctx->bw_f.as<float>(),
                          s, xig));
  return DDC_OK;
}

// ---------------------------------------------------------------------------
// operators on device vectors
// ---------------------------------------------------------------------------
int op_lx(ddc_ctx* ctx, const double* x, double* y) {
  DevGeo g = ctx->geo();
  {
    // the lx part of the fused pass (one value per triple), then the sums
    // per grid point
    StageScope sc(ctx, ST_LX_POT);
    CK(launch_lx_vals(ctx->L(), ctx->tb, g, x, ctx->tval.as<double>()));
    CK(launch_lx_gather(ctx->L(), g, ctx->tval.as<double>(), ctx->pot.as<double>()));
  }
  StageScope sc(ctx, ST_PROJ);
  // y = -Bw pot   (intrhs then negate, matvec.f90:131-135)
  return gemm_proj(ctx, -1.0, ctx->pot.as<double>(), y);
}
int op_xi(ddc_ctx* ctx, const double* x, double* xig, bool weighted = false) {
  StageScope sc(ctx, ST_XI);
  return gemm_xi(ctx, x, xig, weighted);
}
int op_lstarx(ddc_ctx* ctx, const double* x, double* y) {
  CKI(op_xi(ctx, x, ctx->xig.as<double>(), true));
  StageScope sc(ctx, ST_LSTARX);
  CK(launch_lstarx_acc(ctx->L(), ctx->tb, ctx->geo(), ctx->xig.as<double>(), y));
  return DDC_OK;
}

// FP32 operators of the mixed-precision path (vectors stay FP64)
int op_lx_f32(ddc_ctx* ctx, const double* x, double* y) {
  {
    StageScope sc(ctx, ST_LX_POT);
    DevGeo g = ctx->geo();
    CK(launch_lx_vals_f32(ctx->L(), ctx->tb, g, x, ctx->tval.as<float>()));
    CK(launch_lx_gather_f32(ctx->L(), g, ctx->tval.as<float>(), ctx->pot_f.as<float>(),
                            ctx->ldp_f));
  }
  StageScope sc(ctx, ST_PROJ);
  return gemm_proj_f32(ctx, -1.f, ctx->pot_f.as<float>(), y);
}
int op_lstarx_f32(ddc_ctx* ctx, const double* x, double* y) {
  {
    StageScope sc(ctx, ST_XI);
    CKI(gemm_xi_f32(ctx, x, ctx->xi_f.as<float>()));
  }
  StageScope sc(ctx, ST_LSTARX);
  CK(launch_lstarx_acc_f32(ctx->L(), ctx->tb, ctx->geo(), ctx->xi_f.as<float>(), y));
  return DDC_OK;
}

// y = L x and z = L* s (off-diagonal parts) from one pass over the triples
int op_pair(ddc_ctx* ctx, const double* x, double* y, const double* s, double* z) {
  DevGeo g = ctx->geo();
  CKI(op_xi(ctx, s, ctx->xig.as<double>(), true));
  {
    StageScope sc(ctx, ST_LXS);
    CK(launch_lxs(ctx->L(), ctx->tb, g, x, ctx->xig.as<double>(), ctx->tval.as<double>(), z));
  }
  {
    StageScope sc(ctx, ST_GATHER);
    CK(launch_lx_gather(ctx->L(), g, ctx->tval.as<double>(), ctx->pot.as<double>()));
  }
  StageScope sc(ctx, ST_PROJ);
  return gemm_proj(ctx, -1.0, ctx->pot.as<double>(), y);
}
int op_pair_f32(ddc_ctx* ctx, const double* x, double* y, const double* s, double* z) {
  DevGeo g = ctx->geo();
  {
    StageScope sc(ctx, ST_XI);
    CKI(gemm_xi_f32(ctx, s, ctx->xi_f.as<float>()));
  }
  {
    StageScope sc(ctx, ST_LXS);
    CK(launch_lxs_f32(ctx->L(), ctx->tb, g, x, ctx->xi_f.as<float>(), ctx->tval.as<float>(), z));
  }
  {
    StageScope sc(ctx, ST_GATHER);
    CK(launch_lx_gather_f32(ctx->L(), g, ctx->tval.as<float>(), ctx->pot_f.as<float>(),
                            ctx->ldp_f));
  }
  StageScope sc(ctx, ST_PROJ);
  return gemm_proj_f32(ctx, -1.f, ctx->pot_f.as<float>(), y);
}

// ---------------------------------------------------------------------------
// Jacobi/DIIS (jacobi_diis.f90) over one system, or the direct and the adjoint
// one together with one fused L / L* pass per sweep; one molecule or a batch.
// The iteration itself lives on the device (ddc_solver.cu); the host launches
// sweeps a little ahead of the device and stops when no molecule runs.
//
// Mixed precision: iterative refinement.  Each outer step forms in FP64 the
// residual r = rhs - L x and the Jacobi increment d = D^-1 r at x; its H-norm
// is the reference's convergence test (jacobi_diis.f90:143-150), so a molecule
// stops exactly when its FP64 Jacobi increment is below 10^-iconv.  Otherwise
// the correction equation L e = r is solved with Jacobi/DIIS on the FP32
// operator (from e = d, to 1e-4 relative, FP32 history) and x += e.  From the
// reference or the zero start the first residual (at a start that is never
// converged) comes from the FP32 operator, and the test runs from the second
// refinement on.
// ---------------------------------------------------------------------------
// DIIS history length: the reference's ndiis (jacobi_diis.f90) for the FP64
// solves; at most kInnerDiis for the FP32 inner solves of the mixed
// refinement, whose kernels read the whole history from HBM every iteration
// (20k workload: 15 instead of 25 entries keeps the 88 / 85 iterations and
// took 6 ms off a 190 ms step)
constexpr int kInnerDiis = 15;

struct System {
  bool adjoint = false;
  const double* rhs = nullptr;
  double* x = nullptr;               // start in, solution out (device)
  int* iters = nullptr;              // per molecule (host), or null
  ddc_solve_info* inf = nullptr;
};

// norms of a report
constexpr int kNorms = sizeof(ddc_solve_info::norms) / sizeof(double);
// integer and double state arrays of a system, nmol entries each
enum { SI_NMAT, SI_STATUS, SI_ITERS, SI_RESTARTS, SI_EXT, SI_MAXK, SI_RUN, SI_ITS, SI_OUTER, SI_RST,
       SI_UPD, SI_CNT, SI_N };
enum { SD_NORM, SD_LAST, SD_TOLK, SD_N };

// Molecules that a solve treats one by one.  A call on single systems (cosmo)
// solves whatever the context holds as one, also after a batch.
int solver_molecules(const ddc_ctx* ctx) { return ctx->batch ? ctx->nmol : 1; }

int solver_setup(ddc_ctx* ctx, SolverArgs& a, const System* sys, int ns, bool mixed) {
  const int nmol = solver_molecules(ctx), nylm = ctx->nylm;
  memset(&a, 0, sizeof(a));
  a.nmol = nmol;
  a.nsph = ctx->nsph;
  a.nylm = nylm;
  a.ndiis = mixed ? std::min(ctx->prm.ndiis, kInnerDiis) : ctx->prm.ndiis;
  a.max_iter = ctx->prm.max_iter;
  a.tol = std::pow(10.0, -(double)ctx->prm.iconv);
  a.n_total = (long long)ctx->nsph * nylm;
  a.chunk = solver_chunk(a.n_total, nmol == 1);
  for (int l = 0; l <= ctx->prm.lmax; l++) {
    a.facl[l] = ctx->tb.facl[l];
    a.hw[l] = 1.0 / (1.0 + l);
  }
  if (nmol == 1) {
    a.nchunk = (int)((a.n_total + a.chunk - 1) / a.chunk);
    a.nonempty = ctx->nsph > 0;
  } else {
    std::vector<int> cfirst(nmol + 1, 0), cmol, sphmol(ctx->nsph);
    for (int k = 0; k < nmol; k++) {
      const int n = ctx->h_off[k + 1] - ctx->h_off[k];
      const int nc = (int)(((long long)n * nylm + a.chunk - 1) / a.chunk);
      cmol.insert(cmol.end(), nc, k);
      cfirst[k + 1] = cfirst[k] + nc;
      a.nonempty += n > 0;
      std::fill(sphmol.begin() + ctx->h_off[k], sphmol.begin() + ctx->h_off[k + 1], k);
    }
    a.nchunk = cfirst[nmol];
    CK(ctx->b_cmol.ensure(sizeof(int) * std::max(a.nchunk, 1)));
    CK(ctx->b_cfirst.ensure(sizeof(int) * (nmol + 1)));
    CK(ctx->b_sphmol.ensure(sizeof(int) * std::max(ctx->nsph, 1)));
    if (a.nchunk)
      CK(cudaMemcpyAsync(ctx->b_cmol.p, cmol.data(), sizeof(int) * a.nchunk,
                         cudaMemcpyHostToDevice, ctx->st));
    CK(cudaMemcpyAsync(ctx->b_cfirst.p, cfirst.data(), sizeof(int) * (nmol + 1),
                       cudaMemcpyHostToDevice, ctx->st));
    if (ctx->nsph)
      CK(cudaMemcpyAsync(ctx->b_sphmol.p, sphmol.data(), sizeof(int) * ctx->nsph,
                         cudaMemcpyHostToDevice, ctx->st));
    CKI(sync(ctx));  // the host vectors go out of scope
    a.off = ctx->d_off.as<int>();
    a.cmol = ctx->b_cmol.as<int>();
    a.cfirst = ctx->b_cfirst.as<int>();
  }
  const int nd = std::max(a.ndiis, 1);
  CK(ctx->s_int.ensure(sizeof(int) * 2 * (SI_N * (size_t)nmol + 1)));
  CK(ctx->s_dbl.ensure(sizeof(double) * 2 * SD_N * nmol));
  CK(ctx->s_slot.ensure(sizeof(int) * 2 * (size_t)nmol * nd));
  CK(ctx->s_gram.ensure(sizeof(double) * 2 * (size_t)nmol * nd * nd));
  CK(ctx->s_coef.ensure(sizeof(double) * 2 * (size_t)nmol * kMaxHist));
  const size_t parts = (size_t)std::max(solver_parts(a.nchunk, a.chunk), 1) * (kMaxHist + 1);
  CK(ctx->s_part.ensure(sizeof(double) * 2 * parts));
  // the norms of a single solve: what its report holds, and with iprint what is
  // printed (the first million), not one per iteration that max_iter allows
  a.nlog = ctx->batch ? 0 : std::min(ctx->prm.max_iter, ctx->prm.iprint > 0 ? 1 << 20 : kNorms);
  CK(ctx->s_log.ensure(sizeof(double) * 2 * (size_t)a.nlog));
  if (!ctx->hstop) {
    CK(cudaHostAlloc(&ctx->hstop, sizeof(int) * 4, cudaHostAllocMapped));
    CK(cudaHostGetDevicePointer(&ctx->dstop, ctx->hstop, 0));
  }
  if (!ctx->ev_sweep[0])
    for (cudaEvent_t& e : ctx->ev_sweep)
      CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  a.active = ctx->s_int.as<int>() + 2 * SI_N * (size_t)nmol;
  a.hstop = ctx->dstop;
  for (int q = 0; q < ns; q++) {
    SolverSys& s = a.sys[q];
    int* si = ctx->s_int.as<int>() + (size_t)q * SI_N * nmol;
    double* sd = ctx->s_dbl.as<double>() + (size_t)q * SD_N * nmol;
    s.nmat = si + (size_t)SI_NMAT * nmol;
    s.status = si + (size_t)SI_STATUS * nmol;
    s.iters = si + (size_t)SI_ITERS * nmol;
    s.restarts = si + (size_t)SI_RESTARTS * nmol;
    s.ext = si + (size_t)SI_EXT * nmol;
    s.maxk = si + (size_t)SI_MAXK * nmol;
    s.run = si + (size_t)SI_RUN * nmol;
    s.its = si + (size_t)SI_ITS * nmol;
    s.outer = si + (size_t)SI_OUTER * nmol;
    s.rst = si + (size_t)SI_RST * nmol;
    s.upd = si + (size_t)SI_UPD * nmol;
    s.cnt = reinterpret_cast<unsigned*>(si + (size_t)SI_CNT * nmol);
    s.norm = sd + (size_t)SD_NORM * nmol;
    s.last = sd + (size_t)SD_LAST * nmol;
    s.tolk = sd + (size_t)SD_TOLK * nmol;
    s.slot = ctx->s_slot.as<int>() + (size_t)q * nmol * nd;
    s.gram = ctx->s_gram.as<double>() + (size_t)q * nmol * nd * nd;
    s.coef = ctx->s_coef.as<double>() + (size_t)q * nmol * kMaxHist;
    s.part = ctx->s_part.as<double>() + (size_t)q * parts;
    s.log = ctx->s_log.as<double>() + (size_t)q * a.nlog;
    s.hx = (q ? ctx->hist_x2 : ctx->hist_x).p;
    s.he = (q ? ctx->hist_e2 : ctx->hist_e).p;
    s.y = (q ? ctx->y2 : ctx->y).as<double>();
    s.orhs = sys[q].rhs;
    s.ox = sys[q].x;
    s.r = mixed ? (q ? ctx->rres2 : ctx->rres).as<double>() : nullptr;
    s.rhs = mixed ? s.r : s.orhs;
    s.x = mixed ? (q ? ctx->eres2 : ctx->eres).as<double>() : s.ox;
  }
  return DDC_OK;
}

int op_single(ddc_ctx* ctx, bool f32, bool adjoint, const double* in, double* out) {
  if (!f32) return adjoint ? op_lstarx(ctx, in, out) : op_lx(ctx, in, out);
  return adjoint ? op_lstarx_f32(ctx, in, out) : op_lx_f32(ctx, in, out);
}
// y = O x for the systems [q0, q1), skipping the molecules whose state (mask)
// is not zero in every one of them; outer: at the outer iterate
int solver_op(ddc_ctx* ctx, const SolverArgs& a, const System* sys, int q0, int q1, bool f32,
              bool outer) {
  auto mask = [&](int q) { return outer ? a.sys[q].run : a.sys[q].status; };
  auto in = [&](int q) { return outer ? a.sys[q].ox : a.sys[q].x; };
  auto out = [&](int q) { return const_cast<double*>(a.sys[q].y); };
  ctx->sweep = SweepMask{a.cmol ? ctx->b_sphmol.as<int>() : nullptr, mask(q0),
                         q1 - q0 == 2 ? mask(q0 + 1) : nullptr};
  int rc;
  if (q1 - q0 == 2) {
    const int d = sys[0].adjoint ? 1 : 0, j = 1 - d;
    rc = f32 ? op_pair_f32(ctx, in(d), out(d), in(j), out(j))
             : op_pair(ctx, in(d), out(d), in(j), out(j));
  } else {
    rc = op_single(ctx, f32, sys[q0].adjoint, in(q0), out(q0));
  }
  ctx->sweep = SweepMask{};
  return rc;
}

// Sweeps until every molecule of every system has stopped.  The device
// reports the sweep in which a system's last molecule stopped through mapped
// memory; the host reads it `ahead` sweeps later, so that it stays ahead of
// the device, and then leaves the system out (or ends).  A stopped molecule's
// blocks return at once, so the sweeps launched too many are cheap; the
// decision depends on finished sweeps alone, so the launches of a solve are
// always the same.
int solver_sweeps(ddc_ctx* ctx, SolverArgs& a, const System* sys, int q0, int q1, bool f32) {
  // one sweep ahead where a sweep takes a few hundred microseconds, else two
  const int ahead = ctx->ntri * ctx->nylm > 200000000LL ? 1 : 2;
  constexpr int NE = sizeof(ctx->ev_sweep) / sizeof(ctx->ev_sweep[0]);
  volatile int* stop = ctx->hstop;
  stop[0] = stop[1] = 0;
  for (int it = 1; q0 < q1; it++) {
    CKI(solver_op(ctx, a, sys, q0, q1, f32, false));
    a.first = q0;
    a.sweep = it;
    {
      StageScope sc(ctx, ST_JACOBI);
      CK(launch_solver_step(ctx->L(), a, q1 - q0, f32, 0));
    }
    {
      StageScope sc(ctx, ST_COMBINE);
      CK(launch_solver_step(ctx->L(), a, q1 - q0, f32, 1));
    }
    CK(cudaEventRecord(ctx->ev_sweep[it % NE], ctx->st));
    const int done = it - ahead;
    if (done < 1) continue;
    CK(cudaEventSynchronize(ctx->ev_sweep[done % NE]));
    auto stopped = [&](int q) { return stop[q] != 0 && stop[q] <= done; };
    while (q0 < q1 && stopped(q0)) q0++;
    while (q1 > q0 && stopped(q1 - 1)) q1--;
    if (done > ctx->prm.max_iter)  // every molecule's budget is spent by now
      return fail(ctx, DDC_ERR_STATE, "the solver did not stop within its budget");
  }
  a.first = 0;
  return DDC_OK;
}

// increment norms of iterations [from[q], to[q]) (iprint), interleaved as the
// systems iterate
int print_log(ddc_ctx* ctx, const SolverArgs& a, int ns, const int* from, const int* to) {
  std::vector<double> log[2];
  int most = 0;
  for (int q = 0; q < ns; q++) {
    log[q].resize(std::max(std::min(to[q], a.nlog) - from[q], 0));
    most = std::max(most, (int)log[q].size());
    if (!log[q].empty())
      CK(cudaMemcpyAsync(log[q].data(), a.sys[q].log + from[q], sizeof(double) * log[q].size(),
                         cudaMemcpyDeviceToHost, ctx->st));
  }
  CKI(sync(ctx));
  for (int i = 0; i < most; i++)
    for (int q = 0; q < ns; q++)
      if (i < (int)log[q].size())
        printf("  iter=%4d residual norm: %14.4E\n", from[q] + i + 1, log[q][i]);
  return DDC_OK;
}

// Solves the systems; reports go to sys[q].inf and .iters.  One molecule that
// does not converge: DDC_ERR_NOCONV with the last iterate in x; a non-finite
// increment: DDC_ERR_NUMERIC.
int solve_systems(ddc_ctx* ctx, const System* sys, int ns) {
  const double t0 = now_s();
  const bool mixed = ctx->prm.precision == DDC_PREC_MIXED;
  const bool one = !ctx->batch;
  const bool log = ctx->prm.iprint > 0 && one;
  const int nmol = solver_molecules(ctx);
  if (ctx->batch && ctx->prm.ndiis == 0)
    return fail(ctx, DDC_ERR_UNSUPPORTED, "batched solves need DIIS");
  for (int q = 0; q < ns; q++) memset(sys[q].inf, 0, sizeof(*sys[q].inf));
  SolverArgs a;
  CKI(solver_setup(ctx, a, sys, ns, mixed));
  CK(launch_solver_begin(ctx->L(), a, ns, mixed));
  // the state comes back in one go, through pinned memory: the integers, the
  // doubles, and one molecule's norms
  const size_t nsi = 2 * (SI_N * (size_t)nmol + 1), nsd = 2 * SD_N * (size_t)nmol;
  const int nlog = std::min(kNorms, a.nlog);
  CK(ctx->hstate.ensure(sizeof(double) * (nsd + 2 * (size_t)nlog) + sizeof(int) * nsi));
  double* sd = static_cast<double*>(ctx->hstate.p);
  double* slog = sd + nsd;
  int* si = reinterpret_cast<int*>(slog + 2 * nlog);
  auto read_state = [&](bool norms) -> int {
    CK(cudaMemcpyAsync(si, ctx->s_int.p, sizeof(int) * nsi, cudaMemcpyDeviceToHost, ctx->st));
    CK(cudaMemcpyAsync(sd, ctx->s_dbl.p, sizeof(double) * nsd, cudaMemcpyDeviceToHost, ctx->st));
    for (int q = 0; norms && nlog && q < ns; q++)
      CK(cudaMemcpyAsync(slog + (size_t)q * nlog, a.sys[q].log, sizeof(double) * nlog,
                         cudaMemcpyDeviceToHost, ctx->st));
    return sync(ctx);
  };
  auto I = [&](int q, int w, int k) { return si[((size_t)q * SI_N + w) * nmol + k]; };
  auto D = [&](int q, int w, int k) { return sd[((size_t)q * SD_N + w) * nmol + k]; };
  if (!mixed) {
    if (a.nonempty) CKI(solver_sweeps(ctx, a, sys, 0, ns, false));
    if (log) {
      CKI(read_state(false));
      const int from[2] = {0, 0}, to[2] = {I(0, SI_ITERS, 0), ns > 1 ? I(1, SI_ITERS, 0) : 0};
      CKI(print_log(ctx, a, ns, from, to));
    }
  } else {
    const bool f32_first = !ctx->guess_preset && (ctx->prm.guess == DDC_GUESS_REFERENCE ||
                                                   ctx->prm.guess == DDC_GUESS_ZERO);
    int printed[2] = {0, 0};
    for (int round = 0; round < 64 && a.nonempty; round++) {
      const bool f32_res = f32_first && round == 0;
      CKI(solver_op(ctx, a, sys, 0, ns, f32_res, true));
      {
        StageScope sc(ctx, ST_JACOBI);
        CK(launch_solver_residual(ctx->L(), a, ns, f32_res));
      }
      CK(cudaMemcpyAsync(ctx->hstop + 2, a.active, sizeof(int) * 2, cudaMemcpyDeviceToHost,
                         ctx->st));
      CKI(sync(ctx));
      if (log) {
        CKI(read_state(false));
        for (int q = 0; q < ns; q++)
          if (I(q, SI_OUTER, 0) == round + 1)
            printf("  refinement %d: %s increment norm %14.4E\n", round + 1,
                   f32_res ? "FP32" : "FP64", D(q, SD_LAST, 0));
      }
      const bool run0 = ctx->hstop[2] != 0, run1 = ns > 1 && ctx->hstop[3] != 0;
      if (!run0 && !run1) break;
      // the systems that have molecules left
      CKI(solver_sweeps(ctx, a, sys, run0 ? 0 : 1, run1 ? 2 : 1, true));
      CK(launch_solver_update(ctx->L(), a, ns));
      if (log) {
        CKI(read_state(false));
        const int to[2] = {I(0, SI_ITS, 0), ns > 1 ? I(1, SI_ITS, 0) : 0};
        CKI(print_log(ctx, a, ns, printed, to));
        printed[0] = to[0];
        printed[1] = to[1];
      }
    }
  }
  CKI(read_state(true));
  int rc = DDC_OK;
  for (int q = 0; q < ns; q++) {
    ddc_solve_info& f = *sys[q].inf;
    int maxit = 0, maxout = 0, nfail = 0, restarts = 0;
    double worst = 0.0;
    bool finite = true;
    for (int k = 0; k < nmol; k++) {
      const bool empty = one ? ctx->nsph == 0 : ctx->h_off[k + 1] == ctx->h_off[k];
      const int state = I(q, mixed ? SI_RUN : SI_STATUS, k);
      const int it = mixed ? I(q, SI_ITS, k) : I(q, SI_ITERS, k);
      if (sys[q].iters) sys[q].iters[k] = it;
      maxit = std::max(maxit, it);
      maxout = std::max(maxout, mixed ? I(q, SI_OUTER, k) : 0);
      restarts += mixed ? I(q, SI_RST, k) : I(q, SI_RESTARTS, k);
      if (state != 1 && !empty) nfail++;
      if (state == 3) finite = false;
      if (!empty) worst = std::max(worst, D(q, mixed ? SD_LAST : SD_NORM, k));
    }
    f.iterations = maxit;
    f.refinements = maxout;
    f.converged = nfail == 0;
    f.diis_restarts = restarts;
    f.final_norm = worst;
    if (one) {
      const int n = std::min(maxit, nlog);
      if (n > 0) memcpy(f.norms, slog + (size_t)q * nlog, sizeof(double) * n);
    }
    if (rc != DDC_OK || !nfail) continue;
    if (!one)
      rc = fail(ctx, DDC_ERR_NOCONV, std::to_string(nfail) + " molecule(s) did not converge" +
                                         (sys[q].adjoint ? " (adjoint)" : ""));
    else if (!finite)
      rc = fail(ctx, DDC_ERR_NUMERIC, "non-finite increment norm");
    else
      rc = fail(ctx, DDC_ERR_NOCONV, sys[q].adjoint ? "adjoint ddCOSMO did not converge"
                                                    : "ddCOSMO did not converge");
  }
  for (int q = 0; q < ns; q++) sys[q].inf->seconds = now_s() - t0;
  return rc;
}

int solve(ddc_ctx* ctx, bool adjoint, const double* rhs, double* x, ddc_solve_info* info) {
  ddc_solve_info loc{};
  System s;
  s.adjoint = adjoint;
  s.rhs = rhs;
  s.x = x;
  s.inf = info ? info : &loc;
  return solve_systems(ctx, &s, 1);
}

int need_ready(ddc_ctx* ctx) {
  if (!ctx) return DDC_ERR_PARAM;
  if (!ctx->ready) return fail(ctx, DDC_ERR_STATE, "context not initialised (call ddc_init)");
  return DDC_OK;
}

// dot product on device, deterministic
int dot_dev(ddc_ctx* ctx, long long n, const double* a, const double* b, double* out) {
  CK(launch_dot_partial(ctx->L(), n, a, b, ctx->partials.as<double>(), reduce_blocks()));
  return reduce_to_host(ctx, out);
}

// Solute potential (and, with ef, field) at the context's cavity points from
// charges q at its sphere centres (mkrhs.f90:102-114, main.f90:241): near /
// far split for large systems, direct sums otherwise.  trange: per-target
// source ranges of a batch (direct path); the split uses the molecule ranges.
int solute_pot_field(ddc_ctx* ctx, const double* q, double* phi, double* ef, const int2* trange) {
  const int N = ctx->nsph, NC = ctx->ncav;
  StageScope sc(ctx, ST_COULOMB);
  if (ctx->far_on) {
    CK(launch_far_pot_field(ctx->L(), ctx->tbP, N, ctx->ngrid, ctx->sph.as<double4>(), q,
                            ctx->mrange_ptr(), kFarRho, ctx->cavoff.as<int>(),
                            ctx->cavpt.as<int>(), ctx->ccav.as<double>(), ctx->farBT.as<double>(),
                            ctx->farDT.as<double>(), ctx->farA.as<double>(), phi, ef,
                            ctx->zg_on ? &ctx->zg : nullptr));
  } else if (ef) {
    CK(launch_coulomb_pot_field(ctx->L(), N, q, ctx->cx.as<double>(), ctx->cy.as<double>(),
                                ctx->cz.as<double>(), NC, ctx->ccav.as<double>(), phi, ef,
                                trange));
  } else {
    const int nchunk = trange ? 1 : efield_chunks(N, NC);
    if (nchunk > 1) CK(ctx->ef_scratch.ensure(sizeof(double) * (size_t)std::max(NC, 1) * nchunk));
    CK(launch_coulomb_pot(ctx->L(), N, q, ctx->cx.as<double>(), ctx->cy.as<double>(),
                          ctx->cz.as<double>(), NC, ctx->ccav.as<double>(), phi,
                          ctx->ef_scratch.as<double>(), nchunk, trange));
  }
  return DDC_OK;
}

// right-hand side of the direct solve from the cavity potential: wghpot and
// intrhs (cosmo.f90:104-117)
int direct_rhs(ddc_ctx* ctx, const double* phi, double* rhs) {
  CK(ctx->gbuf.ensure(sizeof(double) * std::max<long long>((long long)ctx->nsph * ctx->ngrid, 1)));
  StageScope sc(ctx, ST_RHS);
  CK(launch_wghpot(ctx->L(), ctx->geo(), phi, ctx->gbuf.as<double>()));
  CK(launch_fold_proj(ctx->L(), ctx->fold, ctx->nsph, 1.0, ctx->gbuf.as<double>(), ctx->ngrid,
                      rhs, SweepMask{}));
  return DDC_OK;
}

// cosmo on device vectors: phi (ncav) or glm -> sigma
int cosmo_dev(ddc_ctx* ctx, int star, int cart, const double* phi, const double* glm,
              const double* psi, double* sigma, double* esolv, ddc_solve_info* info) {
  const long long n = (long long)ctx->nsph * ctx->nylm;
  const int gmode = ctx->prm.guess == DDC_GUESS_ZERO ? 1 : 0;
  // the start is the caller's (USER) or was set by the energy+force flow
  const bool keep = ctx->prm.guess == DDC_GUESS_USER || ctx->guess_preset;
  if (ctx->prm.guess == DDC_GUESS_LEARNED && !ctx->guess_preset)
    return fail(ctx, DDC_ERR_PARAM,
                "the learned guess is formed by ddc_energy_forces / ddc_batch_energy_forces");
  if (!star) {
    double* rhs = ctx->rhs.as<double>();
    if (cart) {
      CKI(direct_rhs(ctx, phi, rhs));
    } else {
      CK(cudaMemcpyAsync(rhs, glm, sizeof(double) * n, cudaMemcpyDeviceToDevice, ctx->st));
    }
    if (!keep) CK(launch_guess(ctx->L(), ctx->tb, n, rhs, sigma, gmode));
    CKI(solve(ctx, false, rhs, sigma, info));
    if (esolv) {
      double d = 0.0;
      CKI(dot_dev(ctx, n, sigma, psi, &d));
      *esolv = 0.5 * ((ctx->prm.eps - 1.0) / ctx->prm.eps) * d;
    }
  } else {
    if (!keep) CK(launch_guess(ctx->L(), ctx->tb, n, psi, sigma, gmode));
    CKI(solve(ctx, true, psi, sigma, info));
  }
  return DDC_OK;
}

// learned initial guesses x (direct) and s (adjoint, may be NULL) from the
// context's rhs g and psi: facl * rhs plus the model's correction
int learned_guess(ddc_ctx* ctx, const double* g, const double* psi, double* x, double* s) {
  ddc_guess* m = ctx->gmodel;
  if (!m) return fail(ctx, DDC_ERR_STATE, "DDC_GUESS_LEARNED needs a model (ddc_set_guess_model)");
  const int nin = guess_nfeat(m);
  CK(ctx->gfeat.ensure(sizeof(float) * std::max<long long>((long long)ctx->nsph * nin, 1)));
  CK(launch_guess_features(ctx->L(), ctx->nsph, ctx->nylm, nin, g, psi, ctx->sph.as<double4>(),
                           ctx->mrange_ptr(), ctx->gfeat.as<float>()));
  CK(guess_infer(ctx->L(), m, ctx->tb, ctx->nsph, ctx->gfeat.as<float>(), g, psi, x, s));
  return DDC_OK;
}

// forces_dd on device vectors (forces_dd.f90:91-164)
// xi_ready: xig already holds xi of s (the energy+force flow forms it first
// for zeta)
int forces_dev(ddc_ctx* ctx, const double* phi, const double* sigma, const double* s, double* fx,
               bool xi_ready = false) {
  if (!ctx->prm.igrad || !ctx->zi.p)
    return fail(ctx, DDC_ERR_STATE, "forces need igrad=1 at init (zi)");
  if (!xi_ready) CKI(op_xi(ctx, s, ctx->xig.as<double>()));
  {
    // u_chi(a, n) = sum over the neighbours b of chi(t) * intmlp(X_b): the
    // lx sum (weight chi / f) per triple, then per grid point times f
    StageScope sc(ctx, ST_UCHI);
    DevGeo g = ctx->geo();
    CK(launch_lx_vals(ctx->L(), ctx->tb, g, sigma, ctx->tval.as<double>()));
    CK(launch_lx_gather(ctx->L(), g, ctx->tval.as<double>(), ctx->uchi.as<double>(), true));
  }
  const double fep = 0.5 * (ctx->prm.eps - 1.0) / ctx->prm.eps;
  CK(ctx->fxa.ensure(sizeof(double) * 3 * std::max(ctx->nsph, 1)));
  CK(ctx->fda.ensure(sizeof(double) * 3 * std::max<long long>(ctx->ntri, 1)));
  const int nlm = (ctx->prm.lmax + 1) * (ctx->prm.lmax + 2) / 2;
  CK(ctx->fvec.ensure(sizeof(double2) * 4 * nlm * std::max(ctx->nsph, 1)));
  StageScope sc(ctx, ST_FORCES);
  CK(launch_forces(ctx->L(), ctx->tb, ctx->geo(), sigma, ctx->xig.as<double>(),
                   ctx->uchi.as<double>(), phi, fep, fx, ctx->fxa.as<double>(),
                   ctx->fda.as<double>(), ctx->fvec.as<double2>()));
  return DDC_OK;
}

}  // namespace

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

int ddc_default_params(ddc_params* p) {
  if (!p) return DDC_ERR_PARAM;
  memset(p, 0, sizeof(*p));
  p->lmax = 6;
  p->ngrid = 110;
  p->iconv = 7;
  p->igrad = 1;
  p->eps = 78.3553;
  p->eta = 0.2;
  p->iprint = 0;
  p->max_iter = 200;
  p->ndiis = 25;
  p->precision = DDC_PREC_FP64;
  p->guess = DDC_GUESS_REFERENCE;
  p->device = 0;
  p->device_pointers = 0;
  p->pair_solves = 1;
  return DDC_OK;
}

const char* ddc_status_string(int s) {
  switch (s) {
    case DDC_OK: return "ok";
    case DDC_ERR_PARAM: return "invalid parameter";
    case DDC_ERR_STATE: return "invalid call order";
    case DDC_ERR_CUDA: return "CUDA error";
    case DDC_ERR_NOMEM: return "device allocation failed";
    case DDC_ERR_NOCONV: return "solver did not converge";
    case DDC_ERR_UNSUPPORTED: return "unsupported parameter";
    case DDC_ERR_NUMERIC: return "non-finite result";
    case DDC_ERR_CAPACITY:
      return "problem exceeds the fixed scratch of the allocation-free entry point";
    default: return "unknown status";
  }
}

int ddc_create(const ddc_params* p, ddc_ctx** out) {
  if (!p || !out) return DDC_ERR_PARAM;
  *out = nullptr;
  if (p->lmax < 0 || p->lmax > DDC_MAX_LMAX) return DDC_ERR_UNSUPPORTED;
  if (p->ngrid <= 0 || p->iconv < 0 || p->eps <= 0.0 || !(p->eta > 0.0 && p->eta <= 1.0) ||
      p->max_iter <= 0 || p->ndiis < 0 || p->ndiis > kMaxHist || (p->ndiis > 0 && p->ndiis <= 10))
    return DDC_ERR_PARAM;
  if (p->precision != DDC_PREC_FP64 && p->precision != DDC_PREC_MIXED) return DDC_ERR_PARAM;
  if (p->guess < DDC_GUESS_REFERENCE || p->guess > DDC_GUESS_LEARNED) return DDC_ERR_PARAM;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return DDC_ERR_CUDA;
  if (p->device < 0 || p->device >= ndev) return DDC_ERR_PARAM;
  if (cudaSetDevice(p->device) != cudaSuccess) return DDC_ERR_CUDA;
  ddc_ctx* c = new ddc_ctx();
  c->prm = *p;
  if (p->stream) {
    c->st = (cudaStream_t)p->stream;
    c->own_stream = false;
  } else if (cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking) != cudaSuccess) {
    delete c;
    return DDC_ERR_CUDA;
  }
  *out = c;
  return DDC_OK;
}

int ddc_destroy(ddc_ctx* c) {
  if (!c) return DDC_OK;
  cudaSetDevice(c->prm.device);
  if (c->st) cudaStreamSynchronize(c->st);
  cudaStream_t st = c->own_stream ? c->st : nullptr;
  for (auto& pe : c->ev_pending) {
    cudaEventDestroy(pe.second.first);
    cudaEventDestroy(pe.second.second);
  }
  for (cudaEvent_t e : c->ev_pool) cudaEventDestroy(e);
  tc_release(c->tc);
  if (c->hred) cudaFreeHost(c->hred);
  if (c->hstop) cudaFreeHost(c->hstop);
  for (cudaEvent_t e : c->ev_sweep)
    if (e) cudaEventDestroy(e);
  if (c->st2) cudaStreamSynchronize(c->st2);
  if (c->st_out) cudaStreamDestroy(c->st_out);
  if (c->ev_out) cudaEventDestroy(c->ev_out);
  for (cudaEvent_t e : c->ev_mark)
    if (e) cudaEventDestroy(e);
  if (c->ev_fork) cudaEventDestroy(c->ev_fork);
  if (c->ev_join) cudaEventDestroy(c->ev_join);
  if (c->st2) cudaStreamDestroy(c->st2);
  delete c;
  if (st) cudaStreamDestroy(st);
  return DDC_OK;
}

const char* ddc_last_error(ddc_ctx* c) { return c ? c->err.c_str() : "null context"; }

long long ddc_launch_count(ddc_ctx* c) { return c ? c->launches : 0; }

int ddc_stage_count(void) { return ST_N; }
const char* ddc_stage_name(int k) {
  static const char* names[ST_N] = {"init",    "coulomb_pot", "rhs",       "lx_pot",
                                    "proj_gemm", "xi_gemm",   "lstarx",    "jacobi_step",
                                    "diis_combine", "reduce", "uchi_pot",  "forces",
                                    "zeta",    "efield",      "contract",  "lx_lstarx",
                                    "lx_gather"};
  return (k >= 0 && k < ST_N) ? names[k] : "";
}
int ddc_stage_times(ddc_ctx* c, double* ms, long long* calls) {
  if (!c) return DDC_ERR_PARAM;
  cudaSetDevice(c->prm.device);
  if (!c->ev_pending.empty()) {
    if (cudaStreamSynchronize(c->st) != cudaSuccess) return DDC_ERR_CUDA;
    resolve_timers(c);
  }
  for (int k = 0; k < ST_N; k++) {
    if (ms) ms[k] = c->st_ms[k];
    if (calls) calls[k] = c->st_calls[k];
  }
  return DDC_OK;
}
int ddc_set_timed_stages(ddc_ctx* c, unsigned int mask) {
  if (!c) return DDC_ERR_PARAM;
  c->stage_mask = mask;
  return DDC_OK;
}
int ddc_reset_stage_times(ddc_ctx* c) {
  if (!c) return DDC_ERR_PARAM;
  cudaSetDevice(c->prm.device);
  if (!c->ev_pending.empty()) {
    if (cudaStreamSynchronize(c->st) != cudaSuccess) return DDC_ERR_CUDA;
    resolve_timers(c);
  }
  for (int k = 0; k < ST_N; k++) {
    c->st_ms[k] = 0.0;
    c->st_calls[k] = 0;
  }
  return DDC_OK;
}

}  // extern "C"

// FMA throughput probe: 8 dependent chains per thread, 8 blocks of 256 per SM
static int fma_peak(int device, bool fp32, double* gflops) {
  if (!gflops) return DDC_ERR_PARAM;
  if (cudaSetDevice(device) != cudaSuccess) return DDC_ERR_CUDA;
  cudaDeviceProp pr;
  if (cudaGetDeviceProperties(&pr, device) != cudaSuccess) return DDC_ERR_CUDA;
  long long launches = 0;
  cudaStream_t st;
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return DDC_ERR_CUDA;
  Launch L{st, &launches};
  double* out = nullptr;
  cudaEvent_t a, b;
  cudaMalloc(&out, sizeof(double));
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  const int blocks = pr.multiProcessorCount * 8, iters = fp32 ? 8192 : 4096;
  auto run = [&](int it) {
    if (fp32) launch_fp32_probe(L, blocks, it, reinterpret_cast<float*>(out));
    else launch_fp64_probe(L, blocks, it, out);
  };
  run(64);  // warm up
  cudaEventRecord(a, st);
  run(iters);
  cudaEventRecord(b, st);
  cudaError_t e = cudaStreamSynchronize(st);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(out);
  cudaStreamDestroy(st);
  if (e != cudaSuccess || ms <= 0.f) return DDC_ERR_CUDA;
  double flops = 2.0 * 8.0 * (double)iters * blocks * 256.0;
  *gflops = flops / (ms * 1e-3) / 1e9;
  return DDC_OK;
}

extern "C" {
int ddc_fp64_peak(int device, double* gflops) { return fma_peak(device, false, gflops); }
int ddc_fp32_peak(int device, double* gflops) { return fma_peak(device, true, gflops); }

// ddc_init without the wait at its end
static int init_spheres(ddc_ctx* ctx, int n, const double* x, const double* y, const double* z,
                        const double* r) {
  if (!ctx) return DDC_ERR_PARAM;
  if (n < 0 || (n > 0 && (!x || !y || !z || !r))) return fail(ctx, DDC_ERR_PARAM, "bad input");
  cudaSetDevice(ctx->prm.device);
  std::vector<double4> hs(n);
  if (ctx->prm.device_pointers) {
    std::vector<double> hx(n), hy(n), hz(n), hr(n);
    if (n) {
      CK(cudaMemcpy(hx.data(), x, sizeof(double) * n, cudaMemcpyDeviceToHost));
      CK(cudaMemcpy(hy.data(), y, sizeof(double) * n, cudaMemcpyDeviceToHost));
      CK(cudaMemcpy(hz.data(), z, sizeof(double) * n, cudaMemcpyDeviceToHost));
      CK(cudaMemcpy(hr.data(), r, sizeof(double) * n, cudaMemcpyDeviceToHost));
    }
    for (int i = 0; i < n; i++) hs[i] = make_double4(hx[i], hy[i], hz[i], hr[i]);
  } else {
    for (int i = 0; i < n; i++) hs[i] = make_double4(x[i], y[i], z[i], r[i]);
  }
  for (int i = 0; i < n; i++)
    if (!(hs[i].w > 0.0)) return fail(ctx, DDC_ERR_PARAM, "radii must be positive");
  if (!ctx->batch_init) ctx->nmol = 1;
  ctx->have_flow = false;
  StageScope sc(ctx, ST_INIT);
  return do_init(ctx, n, hs);
}
int ddc_init(ddc_ctx* ctx, int n, const double* x, const double* y, const double* z,
             const double* r) {
  CKI(init_spheres(ctx, n, x, y, z, r));
  const int rc = sync(ctx);
  if (rc != DDC_OK) ctx->ready = false;
  return rc;
}

int ddc_sizes(ddc_ctx* ctx, int* nsph, int* ncav, int* nylm, int* ngrid) {
  CKI(need_ready(ctx));
  if (nsph) *nsph = ctx->nsph;
  if (ncav) *ncav = ctx->ncav;
  if (nylm) *nylm = ctx->nylm;
  if (ngrid) *ngrid = ctx->ngrid;
  return DDC_OK;
}

static int get_dev_array(ddc_ctx* ctx, double* out, const void* src, size_t count) {
  CKI(need_ready(ctx));
  if (!out) return fail(ctx, DDC_ERR_PARAM, "null output");
  if (count == 0) return DDC_OK;
  CK(cudaMemcpyAsync(out, src, sizeof(double) * count,
                     ctx->prm.device_pointers ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                     ctx->st));
  return sync(ctx);
}

int ddc_get_ccav(ddc_ctx* ctx, double* ccav) {
  CKI(need_ready(ctx));
  return get_dev_array(ctx, ccav, ctx->ccav.p, 3 * (size_t)ctx->ncav);
}
int ddc_get_ui(ddc_ctx* ctx, double* ui) {
  CKI(need_ready(ctx));
  if (!ui) return fail(ctx, DDC_ERR_PARAM, "null output");
  cudaSetDevice(ctx->prm.device);
  const size_t np = (size_t)ctx->nsph * ctx->ngrid;
  double* d;
  CKI(out_ptr(ctx, ui, np, ctx->out1, &d));
  CK(launch_grid_order(ctx->L(), ctx->nsph, ctx->ngrid, ctx->gpos.as<int>(), ctx->ui.as<double>(),
                       d));
  CKI(finish_out(ctx, ui, d, np));
  return sync(ctx);
}
int ddc_get_csph(ddc_ctx* ctx, double* csph) {
  CKI(need_ready(ctx));
  return get_dev_array(ctx, csph, ctx->csph.p, 3 * (size_t)ctx->nsph);
}
int ddc_get_grid(ddc_ctx* ctx, double* grid, double* w) {
  CKI(need_ready(ctx));
  for (int i = 0; i < ctx->ngrid; i++) {
    if (grid)
      for (int k = 0; k < 3; k++) grid[3 * i + k] = ctx->h_grid[4 * i + k];
    if (w) w[i] = ctx->h_grid[4 * i + 3];
  }
  return DDC_OK;
}

// the stream of results that go to the host beside kernels
static int out_stream(ddc_ctx* ctx) {
  if (!ctx->st_out) CK(cudaStreamCreateWithFlags(&ctx->st_out, cudaStreamNonBlocking));
  if (!ctx->ev_out) CK(cudaEventCreateWithFlags(&ctx->ev_out, cudaEventDisableTiming));
  return DDC_OK;
}
int ddc_mkrhs(ddc_ctx* ctx, int n, const double* charge, const double* x, const double* y,
              const double* z, int ncav, const double* ccav, double* phi, int nylm, double* psi) {
  if (!ctx) return DDC_ERR_PARAM;
  cudaSetDevice(ctx->prm.device);
  if (n < 0 || ncav < 0 || nylm <= 0) return fail(ctx, DDC_ERR_PARAM, "bad sizes");
  if (!ccav) {
    CKI(need_ready(ctx));
    if (ncav != ctx->ncav) return fail(ctx, DDC_ERR_PARAM, "ncav does not match the context");
  }
  const double *dq, *dx, *dy, *dz, *dc;
  CKI(stage_in(ctx, charge, n, ctx->in1, &dq));
  CKI(stage_in(ctx, x, n, ctx->in2, &dx));
  CKI(stage_in(ctx, y, n, ctx->in3, &dy));
  CKI(stage_in(ctx, z, n, ctx->in4, &dz));
  if (ccav) CKI(stage_in(ctx, ccav, 3 * (size_t)ncav, ctx->ef2, &dc));
  else dc = ctx->ccav.as<double>();
  double *dphi, *dpsi;
  CKI(out_ptr(ctx, phi, ncav, ctx->phi, &dphi));
  CKI(out_ptr(ctx, psi, (size_t)n * nylm, ctx->out1, &dpsi));
  const int nchunk = efield_chunks(n, ncav);
  // (one piece goes straight to phi)
  if (nchunk > 1) CK(ctx->ef_scratch.ensure(sizeof(double) * (size_t)std::max(ncav, 1) * nchunk));
  const bool host = !ctx->prm.device_pointers && psi && n > 0;
  if (host) {
    CK(launch_psi(ctx->L(), n, nylm, dq, dpsi));
    // psi goes to the host while the potential is summed (30,001 charges, 49
    // harmonics: 12 MB, 0.85 ms with the caller's page faults)
    CKI(out_stream(ctx));
    CK(cudaEventRecord(ctx->ev_out, ctx->st));
    CK(cudaStreamWaitEvent(ctx->st_out, ctx->ev_out, 0));
  }
  cudaError_t e = launch_coulomb_pot(ctx->L(), n, dq, dx, dy, dz, ncav, dc, dphi,
                                     ctx->ef_scratch.as<double>(), nchunk, nullptr);
  if (host && e == cudaSuccess) {
    e = cudaMemcpyAsync(psi, dpsi, sizeof(double) * (size_t)n * nylm, cudaMemcpyDeviceToHost,
                        ctx->st_out);
    const cudaError_t w = cudaStreamSynchronize(ctx->st_out);
    if (e == cudaSuccess) e = w;
  }
  CK(e);
  // on device arrays psi comes last: it may lie over the charges
  if (!host) CK(launch_psi(ctx->L(), n, nylm, dq, dpsi));
  CKI(finish_out(ctx, phi, dphi, ncav));
  if (!host) CKI(finish_out(ctx, psi, dpsi, (size_t)n * nylm));
  return sync(ctx);
}

int ddc_rhs(ddc_ctx* ctx, const double* phi, double* g) {
  CKI(need_ready(ctx));
  cudaSetDevice(ctx->prm.device);
  const double* dphi;
  CKI(stage_in(ctx, phi, ctx->ncav, ctx->in1, &dphi));
  double* dg;
  CKI(out_ptr(ctx, g, (size_t)ctx->nsph * ctx->nylm, ctx->out1, &dg));
  CK(ctx->gbuf.ensure(sizeof(double) * std::max<long long>((long long)ctx->nsph * ctx->ngrid, 1)));
  CK(launch_wghpot(ctx->L(), ctx->geo(), dphi, ctx->gbuf.as<double>()));
  CK(launch_fold_proj(ctx->L(), ctx->fold, ctx->nsph, 1.0, ctx->gbuf.as<double>(), ctx->ngrid, dg,
                      SweepMask{}));
  CKI(finish_out(ctx, g, dg, (size_t)ctx->nsph * ctx->nylm));
  return sync(ctx);
}

int ddc_cosmo(ddc_ctx* ctx, int star, int cart, const double* phi, const double* glm,
              const double* psi, double* sigma, double* esolv, ddc_solve_info* info) {
  CKI(need_ready(ctx));
  cudaSetDevice(ctx->prm.device);
  if (!sigma) return fail(ctx, DDC_ERR_PARAM, "null sigma");
  const size_t nv = (size_t)ctx->nsph * ctx->nylm;
  const double *dphi = nullptr, *dglm = nullptr, *dpsi = nullptr;
  if (!star) {
    if (cart) CKI(stage_in(ctx, phi, ctx->ncav, ctx->in1, &dphi));
    else CKI(stage_in(ctx, glm, nv, ctx->in1, &dglm));
    if (esolv) CKI(stage_in(ctx, psi, nv, ctx->in2, &dpsi));
  } else {
    CKI(stage_in(ctx, psi, nv, ctx->in2, &dpsi));
  }
  double* dsig;
  if (ctx->prm.device_pointers) {
    dsig = sigma;
  } else {
    dsig = ctx->sigma.as<double>();
    if (ctx->prm.guess == DDC_GUESS_USER)
      CK(cudaMemcpyAsync(dsig, sigma, sizeof(double) * nv, cudaMemcpyHostToDevice, ctx->st));
  }
  int rc = cosmo_dev(ctx, star, cart, dphi, dglm, dpsi, dsig, star ? nullptr : esolv, info);
  if (rc != DDC_OK && rc != DDC_ERR_NOCONV) return rc;
  if (!ctx->prm.device_pointers)
    CK(cudaMemcpyAsync(sigma, dsig, sizeof(double) * nv, cudaMemcpyDeviceToHost, ctx->st));
  CKI(sync(ctx));
  return rc;
}

int ddc_forces_dd(ddc_ctx* ctx, const double* phi, const double* sigma, const double* s,
                  double* fx) {
  CKI(need_ready(ctx));
  cudaSetDevice(ctx->prm.device);
  const size_t nv = (size_t)ctx->nsph * ctx->nylm;
  const double *dphi, *dsig, *ds;
  CKI(stage_in(ctx, phi, ctx->ncav, ctx->in1, &dphi));
  CKI(stage_in(ctx, sigma, nv, ctx->in2, &dsig));
  CKI(stage_in(ctx, s, nv, ctx->in3, &ds));
  double* dfx;
  CKI(out_ptr(ctx, fx, 3 * (size_t)ctx->nsph, ctx->fx, &dfx));
  CKI(forces_dev(ctx, dphi, dsig, ds, dfx));
  CKI(finish_out(ctx, fx, dfx, 3 * (size_t)ctx->nsph));
  return sync(ctx);
}

static int mkxi_common(ddc_ctx* ctx, const double* s, double* out, double scale) {
  CKI(need_ready(ctx));
  cudaSetDevice(ctx->prm.device);
  const double* ds;
  CKI(stage_in(ctx, s, (size_t)ctx->nsph * ctx->nylm, ctx->in1, &ds));
  double* dout;
  CKI(out_ptr(ctx, out, ctx->ncav, ctx->zeta, &dout));
  CKI(op_xi(ctx, ds, ctx->xig.as<double>()));
  CK(launch_mkxi(ctx->L(), ctx->tb, ctx->geo(), ctx->xig.as<double>(), scale, dout));
  CKI(finish_out(ctx, out, dout, ctx->ncav));
  return sync(ctx);
}
int ddc_mkzeta(ddc_ctx* ctx, const double* s, double* zeta) {
  if (!ctx) return DDC_ERR_PARAM;
  return mkxi_common(ctx, s, zeta, 0.5 * ((ctx->prm.eps - 1.0) / ctx->prm.eps));
}
int ddc_mkxi(ddc_ctx* ctx, const double* s, double* xi) { return mkxi_common(ctx, s, xi, 1.0); }

int ddc_efld(ddc_ctx* ctx, int nsrc, const double* src, const double* csrc, int ntrg,
             const double* ctrg, double* ef) {
  if (!ctx) return DDC_ERR_PARAM;
  cudaSetDevice(ctx->prm.device);
  if (nsrc < 0 || ntrg < 0) return fail(ctx, DDC_ERR_PARAM, "bad sizes");
  auto ctx_coords = [&](int cnt, const double** out) -> int {
    CKI(need_ready(ctx));
    if (cnt == ctx->ncav) *out = ctx->ccav.as<double>();
    else if (cnt == ctx->nsph) *out = ctx->csph.as<double>();
    else return fail(ctx, DDC_ERR_PARAM, "NULL coordinates need ncav or nsph points");
    return DDC_OK;
  };
  const double *dsrc, *dcs, *dct;
  CKI(stage_in(ctx, src, nsrc, ctx->in1, &dsrc));
  if (csrc) CKI(stage_in(ctx, csrc, 3 * (size_t)nsrc, ctx->in2, &dcs));
  else CKI(ctx_coords(nsrc, &dcs));
  if (ctrg) CKI(stage_in(ctx, ctrg, 3 * (size_t)ntrg, ctx->in3, &dct));
  else CKI(ctx_coords(ntrg, &dct));
  double* def;
  CKI(out_ptr(ctx, ef, 3 * (size_t)ntrg, ctx->out1, &def));
  int nchunk = efield_chunks(nsrc, ntrg);
  CK(ctx->ef_scratch.ensure(sizeof(double) * 3 * (size_t)std::max(ntrg, 1) * nchunk));
  CK(launch_efield(ctx->L(), nsrc, dsrc, dcs, ntrg, dct, def, ctx->ef_scratch.as<double>(),
                   nchunk, nullptr));
  CKI(finish_out(ctx, ef, def, 3 * (size_t)ntrg));
  return sync(ctx);
}

int ddc_lx(ddc_ctx* ctx, const double* x, double* y) {
  CKI(need_ready(ctx));
  cudaSetDevice(ctx->prm.device);
  const size_t nv = (size_t)ctx->nsph * ctx->nylm;
  const double* dx;
  CKI(stage_in(ctx, x, nv, ctx->in1, &dx));
  double* dy;
  CKI(out_ptr(ctx, y, nv, ctx->out1, &dy));
  if (ctx->prm.precision == DDC_PREC_MIXED)
    CKI(op_lx_f32(ctx, dx, dy));
  else
    CKI(op_lx(ctx, dx, dy));
  CKI(finish_out(ctx, y, dy, nv));
  return sync(ctx);
}
int ddc_lstarx(ddc_ctx* ctx, const double* x, double* y) {
  CKI(need_ready(ctx));
  cudaSetDevice(ctx->prm.device);
  const size_t nv = (size_t)ctx->nsph * ctx->nylm;
  const double* dx;
  CKI(stage_in(ctx, x, nv, ctx->in1, &dx));
  double* dy;
  CKI(out_ptr(ctx, y, nv, ctx->out1, &dy));
  if (ctx->prm.precision == DDC_PREC_MIXED)
    CKI(op_lstarx_f32(ctx, dx, dy));
  else
    CKI(op_lstarx(ctx, dx, dy));
  CKI(finish_out(ctx, y, dy, nv));
  return sync(ctx);
}
int ddc_lx_lstarx(ddc_ctx* ctx, const double* x, double* y, const double* s, double* z) {
  CKI(need_ready(ctx));
  cudaSetDevice(ctx->prm.device);
  const size_t nv = (size_t)ctx->nsph * ctx->nylm;
  CK(ctx->tval.ensure(sizeof(double) * std::max<long long>(ctx->ntri, 1)));
  const double *dx, *ds;
  CKI(stage_in(ctx, x, nv, ctx->in1, &dx));
  CKI(stage_in(ctx, s, nv, ctx->in2, &ds));
  double *dy, *dz;
  CKI(out_ptr(ctx, y, nv, ctx->out1, &dy));
  if (ctx->prm.device_pointers) {
    dz = z;
  } else {
    CK(ctx->in3.ensure(sizeof(double) * std::max(nv, (size_t)1)));
    dz = ctx->in3.as<double>();
  }
  if (!dz) return fail(ctx, DDC_ERR_PARAM, "null output array");
  // z may lie over x: the pass writes rows of z while other blocks still read
  // theirs of x, so it then reads a copy (y and s need none: s is read before
  // the pass, y written after it)
  const uintptr_t xa = reinterpret_cast<uintptr_t>(dx), za = reinterpret_cast<uintptr_t>(dz);
  if (xa < za + sizeof(double) * nv && za < xa + sizeof(double) * nv) {
    CK(ctx->in1.ensure(sizeof(double) * nv));
    CK(cudaMemcpyAsync(ctx->in1.p, dx, sizeof(double) * nv, cudaMemcpyDeviceToDevice, ctx->st));
    dx = ctx->in1.as<double>();
  }
  if (ctx->prm.precision == DDC_PREC_MIXED)
    CKI(op_pair_f32(ctx, dx, dy, ds, dz));
  else
    CKI(op_pair(ctx, dx, dy, ds, dz));
  CKI(finish_out(ctx, y, dy, nv));
  CKI(finish_out(ctx, z, dz, nv));
  return sync(ctx);
}
int ddc_ldm1x(ddc_ctx* ctx, const double* x, double* y) {
  CKI(need_ready(ctx));
  cudaSetDevice(ctx->prm.device);
  const size_t nv = (size_t)ctx->nsph * ctx->nylm;
  const double* dx;
  CKI(stage_in(ctx, x, nv, ctx->in1, &dx));
  double* dy;
  CKI(out_ptr(ctx, y, nv, ctx->out1, &dy));
  CK(launch_ldm1x(ctx->L(), ctx->tb, (long long)nv, dx, dy));
  CKI(finish_out(ctx, y, dy, nv));
  return sync(ctx);
}
int ddc_hnorm(ddc_ctx* ctx, const double* x, double* norm) {
  CKI(need_ready(ctx));
  cudaSetDevice(ctx->prm.device);
  if (!norm) return fail(ctx, DDC_ERR_PARAM, "null norm");
  const size_t nv = (size_t)ctx->nsph * ctx->nylm;
  const double* dx;
  CKI(stage_in(ctx, x, nv, ctx->in1, &dx));
  CK(launch_hnorm_partial(ctx->L(), ctx->tb, (long long)nv, dx, ctx->partials.as<double>(),
                          reduce_blocks()));
  double ss = 0.0;
  CKI(reduce_to_host(ctx, &ss));
  *norm = std::sqrt(ss / (double)std::max(ctx->nsph, 1));
  return DDC_OK;
}

// What a run hands back without waiting for it: the times of its phases, from
// events at their ends, and the energy's sum in pinned memory.  Both are taken
// when the call returns, whatever it returns.
struct RunEnd {
  ddc_ctx* ctx;
  ddc_run_info* inf;
  double t0, t3 = 0.0;  // start; end of the solve, where mark 2 lies
  int marks = 0;
  double* esolv = nullptr;
  double fac = 0.0;
  int mark() {
    cudaEvent_t& e = ctx->ev_mark[marks];
    if (!e) CK(cudaEventCreate(&e));
    CK(cudaEventRecord(e, ctx->st));
    ++marks;
    return DDC_OK;
  }
  ~RunEnd() {
    if (marks == 0) return;
    if (marks < 3) {  // ended early: the end is now
      if (cudaStreamSynchronize(ctx->st) != cudaSuccess) return;
      t3 = now_s();
      while (marks < 3)
        if (mark() != DDC_OK) return;
    }
    if (cudaStreamSynchronize(ctx->st) != cudaSuccess) return;
    if (esolv) *esolv = fac * ctx->hred[0];
    float a = 0.0f, b = 0.0f;
    if (cudaEventElapsedTime(&a, ctx->ev_mark[0], ctx->ev_mark[2]) != cudaSuccess ||
        cudaEventElapsedTime(&b, ctx->ev_mark[1], ctx->ev_mark[2]) != cudaSuccess)
      return;
    inf->t_init = t3 - 1e-3 * a - t0;
    inf->t_mkrhs = 1e-3 * (a - b);
    inf->t_direct = 1e-3 * b;
  }
};

int ddc_energy_forces(ddc_ctx* ctx, int n, const double* charge, const double* x,
                      const double* y, const double* z, const double* rvdw, double* esolv,
                      double* sigma, double* s, double* fx, ddc_run_info* info) {
  if (!ctx || !esolv) return DDC_ERR_PARAM;
  cudaSetDevice(ctx->prm.device);
  ddc_run_info loc{};
  ddc_run_info* inf = info ? info : &loc;
  memset(inf, 0, sizeof(*inf));
  RunEnd run{ctx, inf, now_s()};
  CKI(init_spheres(ctx, n, x, y, z, rvdw));
  CKI(run.mark());
  const int N = ctx->nsph, NC = ctx->ncav;
  const size_t nv = (size_t)N * ctx->nylm;
  const double* dq;
  CKI(stage_in(ctx, charge, N, ctx->q, &dq));
  CK(ctx->phi.ensure(sizeof(double) * std::max(NC, 1)));
  double* dphi = ctx->phi.as<double>();
  double* dpsi = ctx->psi.as<double>();
  // mkrhs (mkrhs.f90:102-120) with the context's own centres and cavity; with
  // forces, the solute field at the cavity (main.f90:241-253) comes from the
  // same pass over the pairs
  if (ctx->prm.igrad) CK(ctx->ef1.ensure(sizeof(double) * 3 * std::max(NC, 1)));
  CKI(solute_pot_field(ctx, dq, dphi, ctx->prm.igrad ? ctx->ef1.as<double>() : nullptr,
                       nullptr));
  CK(launch_psi(ctx->L(), N, ctx->nylm, dq, dpsi));
  CKI(run.mark());
  double* dsig = ctx->sigma.as<double>();
  double* ds = ctx->s.as<double>();
  if (ctx->prm.guess == DDC_GUESS_USER) {
    // sigma (and s) carry the initial guesses in, e.g. the previous frame's
    // solutions (the sigma slot of cosmo.f90:136-138, 174-176)
    if (!sigma || (ctx->prm.igrad && !s))
      return fail(ctx, DDC_ERR_PARAM, "user guess needs sigma and s on entry");
    const cudaMemcpyKind k =
        ctx->prm.device_pointers ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    CK(cudaMemcpyAsync(dsig, sigma, sizeof(double) * nv, k, ctx->st));
    if (ctx->prm.igrad) CK(cudaMemcpyAsync(ds, s, sizeof(double) * nv, k, ctx->st));
  }
  const bool paired = ctx->prm.igrad && ctx->prm.pair_solves;
  if (paired) {
    // both systems at once: the adjoint right-hand side psi is known before
    // the direct solve, and each round applies L and L* in one fused pass
    double* rhs = ctx->rhs.as<double>();
    CKI(direct_rhs(ctx, dphi, rhs));
    if (ctx->prm.guess == DDC_GUESS_LEARNED) {
      CKI(learned_guess(ctx, rhs, dpsi, dsig, ds));
    } else if (ctx->prm.guess != DDC_GUESS_USER) {
      const int gmode = ctx->prm.guess == DDC_GUESS_ZERO ? 1 : 0;
      CK(launch_guess(ctx->L(), ctx->tb, (long long)nv, rhs, dsig, gmode));
      CK(launch_guess(ctx->L(), ctx->tb, (long long)nv, dpsi, ds, gmode));
    }
    const System sys[2] = {{false, rhs, dsig, nullptr, &inf->direct},
                           {true, dpsi, ds, nullptr, &inf->adjoint}};
    CKI(solve_systems(ctx, sys, 2));
    run.t3 = now_s();
    CKI(run.mark());
    CK(launch_dot_partial(ctx->L(), (long long)nv, dsig, dpsi, ctx->partials.as<double>(),
                          reduce_blocks()));
    CKI(reduce_to_pinned(ctx));
    run.esolv = esolv;
    run.fac = 0.5 * ((ctx->prm.eps - 1.0) / ctx->prm.eps);
  } else {
    if (ctx->prm.guess == DDC_GUESS_LEARNED) {
      // both starts from the model before the solves (cosmo_dev recomputes
      // the same rhs and keeps them)
      CKI(direct_rhs(ctx, dphi, ctx->rhs.as<double>()));
      CKI(learned_guess(ctx, ctx->rhs.as<double>(), dpsi, dsig, ctx->prm.igrad ? ds : nullptr));
      ctx->guess_preset = true;
    }
    const int rc = cosmo_dev(ctx, 0, 1, dphi, nullptr, dpsi, dsig, esolv, &inf->direct);
    if (rc != DDC_OK || !ctx->prm.igrad) ctx->guess_preset = false;
    if (rc != DDC_OK) return rc;
  }
  if (!paired) {
    run.t3 = now_s();
    CKI(run.mark());
  }
  double* dfx = nullptr;
  if (ctx->prm.igrad) {
    if (!paired) {
      const int rc = cosmo_dev(ctx, 1, 0, nullptr, nullptr, dpsi, ds, nullptr, &inf->adjoint);
      ctx->guess_preset = false;
      if (rc != DDC_OK) return rc;
    }
    const double t4 = now_s();
    inf->t_adjoint = t4 - run.t3;
    CK(ctx->fx.ensure(sizeof(double) * 3 * std::max(N, 1)));
    dfx = ctx->fx.as<double>();
    // zeta first (ddmkzeta, ddcosmo.f90:1758-1806): the field of zeta at the
    // nuclei (main.f90:259-265) then runs on the second stream beside the
    // force kernels, which keep the FP64 pipe busy while it loads the FP32
    // (or FP64) pipe
    CKI(op_xi(ctx, ds, ctx->xig.as<double>()));
    CK(ctx->zeta.ensure(sizeof(double) * std::max(NC, 1)));
    double fep = 0.5 * ((ctx->prm.eps - 1.0) / ctx->prm.eps);
    {
      StageScope sc(ctx, ST_ZETA);
      CK(launch_mkxi(ctx->L(), ctx->tb, ctx->geo(), ctx->xig.as<double>(), fep,
                     ctx->zeta.as<double>()));
    }
    CK(ctx->ef2.ensure(sizeof(double) * 3 * std::max(N, 1)));
    const bool mixed = ctx->prm.precision == DDC_PREC_MIXED;
    const int ch2 = mixed ? efield_chunks_f32(NC, N) : efield_chunks(NC, N);
    if (!ctx->zfar_on) CK(ctx->ef_scratch.ensure(sizeof(double) * 3 * ((size_t)ch2 * N + 1)));
    // in mixed precision the force-only field of zeta uses FP32 pair
    // arithmetic, with the grouped multipole far field for large molecules
    auto efield = mixed ? launch_efield_f32 : launch_efield;
    CK(cudaEventRecord(ctx->ev_fork, ctx->st));
    CK(cudaStreamWaitEvent(ctx->st2, ctx->ev_fork, 0));
    {
      StageScope sc(ctx, ST_EFIELD, ctx->st2);
      if (ctx->zfar_on)
        CK(launch_zeta_field_far(Launch{ctx->st2, &ctx->launches}, N, ctx->sph.as<double4>(),
                                 ctx->cavoff.as<int>(), ctx->ccav.as<double>(),
                                 ctx->zeta.as<double>(), ctx->zg, ctx->zg_pk.as<float4>(),
                                 ctx->zg_M.as<float2>(), ctx->zg_scr.as<double>(),
                                 ctx->ef2.as<double>()));
      else
        CK(efield(Launch{ctx->st2, &ctx->launches}, NC, ctx->zeta.as<double>(),
                  ctx->ccav.as<double>(), N, ctx->csph.as<double>(), ctx->ef2.as<double>(),
                  ctx->ef_scratch.as<double>(), ch2, nullptr));
    }
    CK(cudaEventRecord(ctx->ev_join, ctx->st2));
    // forces and the zeta contraction on the main stream; whatever happens
    // there, the second stream is joined before this call returns, so no
    // later call can reuse ef2 / ef_scratch while the field is still running
    int frc = forces_dev(ctx, dphi, dsig, ds, dfx, true);
    if (frc == DDC_OK) {
      // solute field at the cavity (from the mkrhs pass) times zeta
      // (main.f90:241-253)
      StageScope sc(ctx, ST_CONTRACT);
      cudaError_t e = launch_zeta_efld_contract(ctx->L(), ctx->geo(), ctx->zeta.as<double>(),
                                                ctx->ef1.as<double>(), dfx);
      if (e != cudaSuccess) {
        cudaGetLastError();
        frc = fail(ctx, DDC_ERR_CUDA,
                   std::string("launch_zeta_efld_contract: ") + cudaGetErrorString(e));
      }
    }
    if (frc != DDC_OK) {
      cudaStreamSynchronize(ctx->st2);
      return frc;
    }
    // the field of zeta at the nuclei times the charges, after the join
    CK(cudaStreamWaitEvent(ctx->st, ctx->ev_join, 0));
    {
      StageScope sc(ctx, ST_CONTRACT);
      CK(launch_charge_efld_contract(ctx->L(), N, dq, ctx->ef2.as<double>(), dfx));
    }
    if (!ctx->prm.device_pointers) {
      // the solutions go to the host while the force kernels run (5,000
      // spheres: 2 x 4.8 MB into memory that is touched for the first time,
      // 3.7 ms beside 4.1 ms of kernels); the solves have ended, so no event
      // is needed
      CKI(out_stream(ctx));
      cudaError_t e = cudaSuccess;
      for (auto o : {std::make_pair(sigma, dsig), std::make_pair(s, ds)})
        if (e == cudaSuccess && o.first && nv)
          e = cudaMemcpyAsync(o.first, o.second, sizeof(double) * nv, cudaMemcpyDeviceToHost,
                              ctx->st_out);
      const cudaError_t w = cudaStreamSynchronize(ctx->st_out);
      CK(e);
      CK(w);
    }
    CKI(sync(ctx));
    const double t5 = now_s();
    inf->t_forces = t5 - t4;  // forces and both field contractions, overlapped
    inf->t_efld = 0.0;
  }
  if (!ctx->prm.igrad || ctx->prm.device_pointers) CKI(finish_out(ctx, sigma, dsig, nv));
  if (ctx->prm.igrad) {
    if (ctx->prm.device_pointers) CKI(finish_out(ctx, s, ds, nv));
    CKI(finish_out(ctx, fx, dfx, 3 * (size_t)N));
  }
  CKI(sync(ctx));
  inf->nsph = N;
  inf->ncav = NC;
  inf->nylm = ctx->nylm;
  inf->ngrid = ctx->ngrid;
  inf->ntriples = ctx->ntri;
  inf->npairs = ctx->npair;
  ctx->have_flow = true;
  return DDC_OK;
}


int ddc_batch_energy_forces(ddc_ctx* ctx, int nmol, const int* off, const double* charge,
                            const double* x, const double* y, const double* z,
                            const double* rvdw, double* esolv, double* fx, int* iters,
                            ddc_run_info* info) {
  if (!ctx || nmol <= 0 || !off || !esolv) return DDC_ERR_PARAM;
  cudaSetDevice(ctx->prm.device);
  if (off[0] != 0) return fail(ctx, DDC_ERR_PARAM, "off[0] must be 0");
  for (int k = 0; k < nmol; k++)
    if (off[k + 1] < off[k]) return fail(ctx, DDC_ERR_PARAM, "offsets must not decrease");
  const int N = off[nmol];
  ddc_run_info loc{};
  ddc_run_info* inf = info ? info : &loc;
  memset(inf, 0, sizeof(*inf));
  double t0 = now_s();
  // molecule partition: per-sphere index range of its molecule
  ctx->nmol = nmol;
  ctx->h_off.assign(off, off + nmol + 1);
  {
    std::vector<int2> mr(std::max(N, 1));
    for (int k = 0; k < nmol; k++)
      for (int i = off[k]; i < off[k + 1]; i++) mr[i] = make_int2(off[k], off[k + 1]);
    CK(ctx->mrange.ensure(sizeof(int2) * std::max(N, 1)));
    CK(cudaMemcpyAsync(ctx->mrange.p, mr.data(), sizeof(int2) * std::max(N, 1),
                       cudaMemcpyHostToDevice, ctx->st));
    CK(ctx->d_off.ensure(sizeof(int) * (nmol + 1)));
    CK(cudaMemcpyAsync(ctx->d_off.p, off, sizeof(int) * (nmol + 1), cudaMemcpyHostToDevice,
                       ctx->st));
  }
  ctx->batch_init = true;
  int rc = ddc_init(ctx, N, x, y, z, rvdw);
  ctx->batch_init = false;
  if (rc != DDC_OK) {
    ctx->nmol = 1;
    return rc;
  }
  ctx->nmol = nmol;
  double t1 = now_s();
  inf->t_init = t1 - t0;
  const int NC = ctx->ncav;
  const size_t nv = (size_t)N * ctx->nylm;
  CK(ctx->tr_cav.ensure(sizeof(int2) * std::max(NC, 1)));
  CK(ctx->tr_nuc.ensure(sizeof(int2) * std::max(N, 1)));
  CK(launch_batch_ranges(ctx->L(), N, ctx->ngrid, NC, ctx->mrange.as<int2>(), ctx->cavpt.as<int>(),
                         ctx->cavoff.as<int>(), ctx->tr_cav.as<int2>(), ctx->tr_nuc.as<int2>()));
  const double* dq;
  CKI(stage_in(ctx, charge, N, ctx->q, &dq));
  CK(ctx->phi.ensure(sizeof(double) * std::max(NC, 1)));
  double* dphi = ctx->phi.as<double>();
  double* dpsi = ctx->psi.as<double>();
  // the potential and (with forces) the solute field at the cavity, each
  // molecule's points from its own nuclei
  if (ctx->prm.igrad) CK(ctx->ef1.ensure(sizeof(double) * 3 * std::max(NC, 1)));
  CKI(solute_pot_field(ctx, dq, dphi, ctx->prm.igrad ? ctx->ef1.as<double>() : nullptr,
                       ctx->tr_cav.as<int2>()));
  CK(launch_psi(ctx->L(), N, ctx->nylm, dq, dpsi));
  CKI(sync(ctx));
  double t2 = now_s();
  inf->t_mkrhs = t2 - t1;
  double* dsig = ctx->sigma.as<double>();
  double* ds = ctx->s.as<double>();
  const long long n = (long long)nv;
  const bool paired = ctx->prm.igrad && ctx->prm.pair_solves;
  auto batch_solve = [&](const System* sys, int ns) {
    ctx->batch = true;
    const int r = solve_systems(ctx, sys, ns);
    ctx->batch = false;
    return r;
  };
  // direct solve (and the adjoint with it when paired)
  {
    double* rhs = ctx->rhs.as<double>();
    CKI(direct_rhs(ctx, dphi, rhs));
    const bool learned = ctx->prm.guess == DDC_GUESS_LEARNED;
    if (learned)
      CKI(learned_guess(ctx, rhs, dpsi, dsig, ctx->prm.igrad ? ds : nullptr));
    else
      CK(launch_guess(ctx->L(), ctx->tb, n, rhs, dsig, ctx->prm.guess == DDC_GUESS_ZERO ? 1 : 0));
    std::vector<int> it(nmol), ita(nmol);
    // the adjoint right-hand side psi is known already: paired systems share
    // each sweep's fused L / L* pass
    if (paired && !learned)
      CK(launch_guess(ctx->L(), ctx->tb, n, dpsi, ds, ctx->prm.guess == DDC_GUESS_ZERO ? 1 : 0));
    const System sys[2] = {{false, rhs, dsig, it.data(), &inf->direct},
                           {true, dpsi, ds, ita.data(), &inf->adjoint}};
    CKI(batch_solve(sys, paired ? 2 : 1));
    if (iters)
      for (int k = 0; k < nmol; k++) {
        iters[2 * k] = it[k];
        if (paired) iters[2 * k + 1] = ita[k];
      }
  }
  CK(ctx->b_out.ensure(sizeof(double) * nmol));
  const double fep = 0.5 * ((ctx->prm.eps - 1.0) / ctx->prm.eps);
  CK(launch_batch_dot(ctx->L(), nmol, ctx->d_off.as<int>(), ctx->nylm, dsig, dpsi, fep,
                      ctx->b_out.as<double>()));
  CK(cudaMemcpyAsync(esolv, ctx->b_out.p, sizeof(double) * nmol, cudaMemcpyDeviceToHost, ctx->st));
  CKI(sync(ctx));
  double t3 = now_s();
  inf->t_direct = t3 - t2;
  if (ctx->prm.igrad) {
    if (!paired) {
      if (ctx->prm.guess != DDC_GUESS_LEARNED)
        CK(launch_guess(ctx->L(), ctx->tb, n, dpsi, ds, ctx->prm.guess == DDC_GUESS_ZERO ? 1 : 0));
      std::vector<int> it(nmol);
      const System sys{true, dpsi, ds, it.data(), &inf->adjoint};
      CKI(batch_solve(&sys, 1));
      if (iters)
        for (int k = 0; k < nmol; k++) iters[2 * k + 1] = it[k];
    }
    double t4 = now_s();
    inf->t_adjoint = t4 - t3;
    CK(ctx->fx.ensure(sizeof(double) * 3 * std::max(N, 1)));
    double* dfx = ctx->fx.as<double>();
    CKI(forces_dev(ctx, dphi, dsig, ds, dfx));
    CK(ctx->zeta.ensure(sizeof(double) * std::max(NC, 1)));
    {
      StageScope sc(ctx, ST_ZETA);
      CK(launch_mkxi(ctx->L(), ctx->tb, ctx->geo(), ctx->xig.as<double>(), fep,
                     ctx->zeta.as<double>()));
    }
    CKI(sync(ctx));
    double t5 = now_s();
    inf->t_forces = t5 - t4;
    CK(ctx->ef2.ensure(sizeof(double) * 3 * std::max(N, 1)));
    const int parts = efield_parts(N);
    CK(ctx->ef_scratch.ensure(sizeof(double) * 3 * (size_t)std::max(N, 1) * parts));
    {
      StageScope sc(ctx, ST_EFIELD);
      // each nucleus from the cavity points of its own molecule; in mixed
      // precision with FP32 pair arithmetic (FP64 sums), as the
      // single-molecule flow does for this force-only field
      auto efield = ctx->prm.precision == DDC_PREC_MIXED ? launch_efield_f32 : launch_efield;
      CK(efield(ctx->L(), NC, ctx->zeta.as<double>(), ctx->ccav.as<double>(), N,
                ctx->csph.as<double>(), ctx->ef2.as<double>(), ctx->ef_scratch.as<double>(), parts,
                ctx->tr_nuc.as<int2>()));
    }
    {
      StageScope sc(ctx, ST_CONTRACT);
      CK(launch_zeta_efld_contract(ctx->L(), ctx->geo(), ctx->zeta.as<double>(),
                                   ctx->ef1.as<double>(), dfx));
      CK(launch_charge_efld_contract(ctx->L(), N, dq, ctx->ef2.as<double>(), dfx));
    }
    CKI(finish_out(ctx, fx, dfx, 3 * (size_t)N));
    CKI(sync(ctx));
    inf->t_efld = now_s() - t5;
  }
  inf->nsph = N;
  inf->ncav = NC;
  inf->nylm = ctx->nylm;
  inf->ngrid = ctx->ngrid;
  inf->ntriples = ctx->ntri;
  inf->npairs = ctx->npair;
  ctx->have_flow = true;
  return DDC_OK;
}

// training rows of the learned guess from the last flow (ddc_guess.cu)
int ddc_guess_features(ddc_ctx* ctx, float* feat) {
  if (!ctx || !feat) return DDC_ERR_PARAM;
  if (!ctx->have_flow)
    return fail(ctx, DDC_ERR_STATE, "guess features need a ddc_energy_forces or batch call first");
  if (!ctx->gmodel) return fail(ctx, DDC_ERR_STATE, "no guess model (ddc_set_guess_model)");
  cudaSetDevice(ctx->prm.device);
  CK(launch_guess_features(ctx->L(), ctx->nsph, ctx->nylm, guess_nfeat(ctx->gmodel),
                           ctx->rhs.as<double>(), ctx->psi.as<double>(), ctx->sph.as<double4>(),
                           ctx->mrange_ptr(), feat));
  return sync(ctx);
}
int ddc_guess_targets(ddc_ctx* ctx, float* target) {
  if (!ctx || !target) return DDC_ERR_PARAM;
  if (!ctx->have_flow || !ctx->prm.igrad)
    return fail(ctx, DDC_ERR_STATE, "guess targets need an energy+force call (igrad=1) first");
  if (!ctx->gmodel) return fail(ctx, DDC_ERR_STATE, "no guess model (ddc_set_guess_model)");
  cudaSetDevice(ctx->prm.device);
  CK(launch_guess_targets(ctx->L(), ctx->tb, ctx->nsph, guess_nout(ctx->gmodel),
                          ctx->rhs.as<double>(), ctx->psi.as<double>(), ctx->sigma.as<double>(),
                          ctx->s.as<double>(), target));
  return sync(ctx);
}
int ddc_set_guess_model(ddc_ctx* ctx, ddc_guess* m) {
  if (!ctx) return DDC_ERR_PARAM;
  if (m && guess_lmax(m) != ctx->prm.lmax)
    return fail(ctx, DDC_ERR_PARAM, "guess model was built for another lmax");
  ctx->gmodel = m;
  return DDC_OK;
}

}  // extern "C"
