// ddc_internal.h -- shared declarations of the B200 ddCOSMO library.
//
// Layout in HBM (one molecule per context, sizes for N spheres, G grid
// points, Y = (lmax+1)^2 harmonics, P neighbour pairs, T triples):
//   sph[N]         double4 {x, y, z, r} (bohr)
//   grid[G]        double4 {sx, sy, sz, w} (unit vectors, 4pi-scaled weights), in
//                  patch (Morton) order: every grid index n below is in this
//                  order; the cavity and the arrays that cross the interface
//                  follow the Lebedev order (gpos)
//   basis[G][Y]    Y_lm(s_n); bw[G][Y] = basis * w  (the intrhs operator)
//   inl[N+1], nl[P]      CSR neighbour list, 0-based, ascending j (ddinit)
//   rev[P]               index of (j,i) for the entry (i,j)
//   fi, ui[N][G]         overlap count f_i(n) and cavity weight U_i(n)
//   zi[N][G][3]          grad f (forces only)
//   pn_ptr[P+1], pn[T]   per pair (i,j): grid points n of sphere i with
//                        t_n^ij < 1 (point inside sphere j), ascending n
//   ls_ptr[N+1], ls[T]   per sphere i: j * G + n for j in N_i (CSR order) and the
//                        points n of sphere j inside sphere i (adjoint gather)
//   ntri[N][G]           number of neighbours containing point (i,n)
//   pt_ptr[N*G+1], pt_idx[T]  per point: where its triples sit in the gather lists
//   cavoff[N+1], cavidx[N][G], cavpt[ncav], ccav[ncav][3]
// Vectors X(nylm,nsph) live as X[i*nylm + lm], like the reference.
#pragma once
#include <cuda.h>  // CUtensorMap (type only; the driver is reached through cudart)
#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "../../include/ddcosmo_gpu.h"

#define DDC_NLM_CAP ((DDC_MAX_LMAX + 1) * (DDC_MAX_LMAX + 2) / 2)

namespace ddc {

// Device buffer owned by a context (freed with it).
struct DBuf {
  void* p = nullptr;
  size_t bytes = 0;
  ~DBuf() { release(); }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
  }
  cudaError_t ensure(size_t b) {
    if (b <= bytes && p) return cudaSuccess;
    release();
    if (b == 0) b = 16;
    cudaError_t e = cudaMalloc(&p, b);
    if (e == cudaSuccess) bytes = b;
    return e;
  }
  template <class T>
  T* as() const {
    return reinterpret_cast<T*>(p);
  }
};

// Plan of the tensor-core contractions of the mixed-precision operators
// (ddc_tc.cu): tile widths, pipeline depths, the split images of the static
// operands, the TMA descriptor of the FP32 grid field and an error flag in
// mapped host memory that a kernel sets when one of its bounded waits runs out.
struct TcPlan {
  bool on = false;
  bool packed = false;       // the static images are built (they depend on bw alone)
  bool tuned = false;        // tile widths measured for tune_key's shape
  long long tune_key = 0;
  int tuned_bn_proj = 0, tuned_bn_xi = 0;
  bool xi_split = false, tuned_xi_split = false;  // expansion: one grid tile per CTA
  float ms_proj = 0.f, ms_xi = 0.f;  // measured launch times of the chosen widths
  int nsph = 0, nylm = 0, ngrid = 0, ldp = 0;
  int kc_proj = 0, bn_proj = 0, ns_proj = 0, smem_proj = 0;
  int mt_xi = 0, kc_xi = 0, bn_xi = 0, ns_xi = 0, smem_xi = 0;
  DBuf img_proj, img_xi;
  alignas(64) CUtensorMap tm_pot;
  float* pot_f = nullptr;
  int* err_h = nullptr;
  int* err_d = nullptr;
};

// Constants of the spherical-harmonic recurrences, indexed by (l, m >= 0)
// packed as l*(l+1)/2 + m.  Passed by value to the kernels (parameter space
// is a broadcast constant bank, so per-(l,m) reads are free).
struct YlmTables {
  double facl[DDC_MAX_LMAX + 1];  // (2l+1)/(4pi): D^-1 block (ddcosmo.f90:233)
  double facs[DDC_NLM_CAP];       // Y_lm normalisation incl. odd-m sign (:236-242)
  double K[DDC_NLM_CAP];          // facs / facl
  double A[DDC_NLM_CAP];          // (2l-1)/(l-m): Legendre recurrence
  double B[DDC_NLM_CAP];          // (l+m-1)/(l-m)
  // normalised recurrence of the far-field and force kernels: Pt_l^m = gam_lm Q_l^m with
  // Q_m = Pt_m^m, Q_{m+1} = c t Q_m, Q_l = c t Q_{l-1} - beta_lm t^2 Q_{l-2};
  // Kg = K * gam folds the scale into the contractions
  double Bn[DDC_NLM_CAP], Kg[DDC_NLM_CAP];
  // Kg times the signed (2m-1)!! of the prefix P_m^m: the scale of the monic
  // recurrence in Cartesian powers (ddc_lxs.cu)
  double Kp[DDC_NLM_CAP];
  double eta;
  int lmax, nylm, ngrid;
};

// What the operator kernels (ddc_lxs.cu) need of the tables.
struct LxsTab {
  double kp[DDC_NLM_CAP];
  double eta, ie5;  // eta and eta^-5
};

// Device geometry handed to every kernel.
// Spheres a solver sweep may skip: those of molecules whose systems have
// all stopped (their operator outputs are not read again).  st0 == null:
// every sphere is computed.
struct SweepMask {
  const int* mol;  // [nsph] molecule of each sphere, or null: one molecule
  const int* st0;  // [nmol] status of the first system (0: running)
  const int* st1;  // [nmol] status of the second system, or null
};

// Tables of the folded contractions (ddc_fold.cu): orbits of the grid under the
// three reflections and the eight parity classes of the harmonics.
struct FoldTab {
  int norb, otiles;  // orbits, tiles of eight orbits
  int oc;            // orbits per pass of a block
  int nylm;
  int psize, xsize;  // entries of pf; of xfw and xfb
  int cnt[8], poff[8], xoff[8];  // harmonics per class, first entries in pf and xf*
  const short* img;              // [norb][8] grid point of image k (bits: x, y, z)
  const uint8_t* first;          // [norb] images that are other points than earlier ones
  const short* lm;               // [8][32] the classes' harmonics
  const double *pf, *xfw, *xfb;  // operands in fragment order
};

// Indices into lists and fields of up to 2^31 - 2 entries, formed so that no
// sum passes 2^31 where threads of a last block lie beyond the end.
// Entry k of the list [q0, q1), its last where the list is shorter:
__host__ __device__ inline int list_entry(int q0, int q1, int k) {
  const int last = q1 - q0 - 1;
  return q0 + (k < last ? k : last);
}
// Point of thread tid in step i of a block of n threads that takes `steps` steps:
__host__ __device__ inline unsigned step_point(unsigned block, unsigned steps, unsigned i,
                                               unsigned n, unsigned tid) {
  return (block * steps + i) * n + tid;
}

#ifdef __CUDACC__
// The kernels of a solver sweep follow one another with a dependency on all
// of the previous kernel.  Launched with launch_chained they are scheduled
// while that kernel still runs (programmatic dependent launch) and begin with
// chain_wait, which every thread of them executes before anything else: it
// returns when the previous kernel has finished and its writes are visible.
// What that kernel writes is then read with ordinary loads: it changes while
// this kernel is resident, so the read-only path (ld.global.nc, which the
// compiler also chooses for const __restrict__ pointers, and may move above the
// wait) is for tables that no kernel of a sweep writes.
// Saves about 1 us between two kernels.
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
cudaError_t launch_chained(void (*kfn)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                           A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kfn, static_cast<P>(args)...);
}
// True for a sphere of a molecule whose systems have all stopped.
__device__ __forceinline__ bool sweep_skip(const SweepMask& m, int sph) {
  if (!m.st0) return false;
  const int k = m.mol ? m.mol[sph] : 0;
  return m.st0[k] != 0 && (!m.st1 || m.st1[k] != 0);
}
// True for every thread of the block when the spheres [i0, i0 + w) are all
// skipped (a block barrier: call it from every thread, w <= blockDim.x)
__device__ __forceinline__ bool sweep_skip_tile(const SweepMask& m, int i0, int w, int nsph) {
  if (!m.st0) return false;
  const int i = i0 + (int)threadIdx.x;
  return __syncthreads_and((int)threadIdx.x >= w || i >= nsph || sweep_skip(m, i)) != 0;
}
#endif

struct DevGeo {
  int nsph, ngrid, nylm, ncav, npair;
  // geometry (u, v, z, W) of each gather-list triple (ddc_lxs.cu): FP32 in
  // the mixed path, FP64 in the FP64 path; null if absent
  const float4* tgeo4;
  const double4* tgeo4d;
  long long ntri;
  const double4* sph;
  const double4* grid;
  const double* basis;
  const double* bw;
  const double* fi;
  const double* ui;
  const double* zi;
  const int* inl;
  const int* nl;
  const int* rev;
  const int* pn_ptr;
  const uint16_t* pn;
  const int* ls_ptr;
  const int* ls_order;  // spheres by falling length of their lists, or null: as they are
  const int* ls;  // gather list: a * ngrid + n of each triple
  const int* pt_ptr;   // per point (a, n): its entries of pt_idx
  const int* pt_idx;   // positions of its triples in the gather lists, CSR order
  const int* lsstart;  // per CSR entry (j,i): start of that pair's block in i's gather list
  const uint8_t* ntri_pt;
  const int* cavoff;
  const int* cavidx;
  const int* cavpt;
  const double* ccav;
  SweepMask act;
};

// Stages timed with CUDA events when ddc_params.timing = 1.
enum Stage {
  ST_INIT = 0, ST_COULOMB, ST_RHS, ST_LX_POT, ST_PROJ, ST_XI, ST_LSTARX, ST_JACOBI,
  ST_COMBINE, ST_REDUCE, ST_UCHI, ST_FORCES, ST_ZETA, ST_EFIELD, ST_CONTRACT, ST_LXS,
  ST_GATHER, ST_N
};

// Longest DIIS history.
constexpr int kMaxHist = 32;
// State of one system (direct or adjoint) of a Jacobi/DIIS solve: device
// arrays, one entry per molecule unless noted.
struct SolverSys {
  const double* rhs;   // what the iteration solves for: the system's
  const double* y;     //   right-hand side, its operator output (O x) and its
  double* x;           //   iterate; mixed: the inner system r, O e, e
  const double* orhs;  // mixed: the outer right-hand side and iterate, and r
  double* ox;
  double* r;
  void* hx;  // [ndiis][n_total] history of iterates and increments, FP64 or
  void* he;  //   FP32 (inner solves of the mixed refinement)
  int* nmat;      // next history position, 1-based
  int* slot;      // [nmol][ndiis] logical -> physical history slot
  int* status;    // 0 running, 1 converged, 2 budget spent, 3 non-finite
  int* iters;     // iterations of this (inner) solve
  int* restarts;  // singular DIIS systems of this (inner) solve
  int* ext;       // terms of the extrapolation; negative: take the Jacobi iterate
  int* maxk;      // iteration budget
  int* run;       // mixed, outer: 0 refining, 1 converged, 2 budget spent, 3 non-finite
  int* its;       // mixed, outer: iterations, refinements and restarts so far
  int* outer;
  int* rst;
  int* upd;       // the inner solve ran
  unsigned* cnt;  // arrival counters, zero between kernels
  double* norm;   // last increment norm
  double* last;   // last outer increment norm
  double* tolk;   // tolerance
  double* coef;   // [nmol][kMaxHist] extrapolation coefficients
  double* gram;   // [nmol][ndiis][ndiis] inner products by physical slot
  double* part;   // [nchunk][kMaxHist+1] per-chunk partial sums
  double* log;    // [nlog] increment norms of the first iterations (one molecule)
};
struct SolverArgs {
  int nmol, nonempty, nsph, nylm, ndiis, max_iter;
  int nchunk, chunk;  // chunks of `chunk` elements
  int first;          // system of grid row 0
  int sweep;          // number of the sweep, from 1
  int nlog;           // length of the systems' logs
  double tol;
  long long n_total;
  const int* off;     // [nmol+1] sphere offsets of the molecules; with cmol
  const int* cmol;    // [nchunk] molecule of each chunk, or null: one molecule
  const int* cfirst;  // [nmol+1] first chunk of each molecule
  int* active;        // [2] molecules still running
  int* hstop;         // [2] mapped host memory: the sweep that stopped the system
  double facl[DDC_MAX_LMAX + 1];  // D^-1 of degree l
  double hw[DDC_MAX_LMAX + 1];    // 1 / (1 + l): weights of the increment norm
  SolverSys sys[2];
};

// ---------------------------------------------------------------------------
// Kernel launchers (ddc_kernels.cu).  All run on `st` and return the CUDA
// error of the launch.  `launches` is incremented per kernel launched.
// ---------------------------------------------------------------------------
struct Launch {
  cudaStream_t st;
  long long* launches;
};

// init
cudaError_t launch_basis(Launch L, const YlmTables& tb, const double4* grid, double* basis,
                         double* bw);
// mrange: per sphere, the index range of its molecule (nullptr: one molecule)
cudaError_t launch_csr_count(Launch L, int nsph, const double4* sph, int* cnt,
                             const int2* mrange);
cudaError_t launch_csr_fill(Launch L, int nsph, const double4* sph, const int* inl, int* nl,
                            const int2* mrange);
cudaError_t launch_csr_rev(Launch L, int nsph, const int* inl, const int* nl, int* rev);
cudaError_t launch_fiui(Launch L, const YlmTables& tb, int nsph, const double4* sph,
                        const double4* grid, const int* inl, const int* nl,
                        double* fi, double* ui, double* zi, uint8_t* ntri);
cudaError_t launch_cav_count(Launch L, int nsph, int ngrid, const double* ui, int* cnt);
// gpos: position of each Lebedev point in the grid (which is in patch order)
cudaError_t launch_cav_fill(Launch L, int nsph, int ngrid, const int* gpos, const double* ui,
                            const double4* sph, const double4* grid, const int* cavoff,
                            int* cavidx, int* cavpt, double* ccav);
cudaError_t launch_grid_order(Launch L, int nsph, int ngrid, const int* gpos, const double* f,
                              double* out);
cudaError_t launch_pair_count(Launch L, int nsph, int npair, int ngrid, const double4* sph,
                              const double4* grid, const int* inl, const int* nl, int* cnt,
                              unsigned* bits);  // bits: [npair][ceil(ngrid / 32)] words
cudaError_t launch_pair_fill(Launch L, int nsph, int npair, int ngrid, const double4* sph,
                             const double4* grid, const int* inl, const int* nl,
                             const unsigned* bits, const int* pn_ptr, uint16_t* pn);
cudaError_t launch_ls_count(Launch L, int nsph, const int* inl, const int* rev, const int* pn_ptr,
                            int* cnt);
cudaError_t launch_ls_fill(Launch L, int nsph, const int* inl, const int* nl, const int* rev,
                           const int* pn_ptr, const uint16_t* pn, const int* ls_ptr, int ngrid,
                           int* ls, int* lsstart);
cudaError_t launch_pt_fill(Launch L, int nsph, int ngrid, const int* inl, const int* pn_ptr,
                           const uint16_t* pn, const int* lsstart, const uint8_t* ntri,
                           int* pt_ptr, int* pt_idx);
// exclusive scan of n ints (out[n] = total; in[n] is overwritten); temp is
// device scratch of temp_bytes
cudaError_t scan_exclusive(Launch L, int* in, int* out, int n, void* temp, size_t temp_bytes);
size_t scan_temp_bytes(int n);
// the same with the total in 64 bits and the largest count
struct CountStats {
  unsigned long long total;
  int largest;
};
cudaError_t scan_counts(Launch L, int* cnt, int* out, int n, void* temp, size_t temp_bytes,
                        CountStats* st);
// order[n]: the lists of ptr[n+1] by falling length (to a 1,024th of the longest)
cudaError_t launch_ls_order(Launch L, int n, const int* ptr, const CountStats* st, int* order);

// operators over the triples (ddc_lxs.cu): lx values, one per triple in
// gather-list order, for k_lx_gather, and / or the L* rows.  xi holds the
// weighted field w_n xi_a(n).  The FP32 variants are the mixed path's: xi and
// val in FP32, X and y in FP64, geometry from g.tgeo4; the FP64 ones take
// g.tgeo4d if there, else evaluate the geometry in the pass.
cudaError_t launch_lxs(Launch L, const YlmTables& tb, const DevGeo& g, const double* X,
                       const double* xi, double* val, double* y);
cudaError_t launch_lx_vals(Launch L, const YlmTables& tb, const DevGeo& g, const double* X,
                           double* val);
cudaError_t launch_lstarx_acc(Launch L, const YlmTables& tb, const DevGeo& g, const double* xi,
                              double* y);
cudaError_t launch_lxs_f32(Launch L, const YlmTables& tb, const DevGeo& g, const double* X,
                           const float* xi, float* val, double* y);
cudaError_t launch_lx_vals_f32(Launch L, const YlmTables& tb, const DevGeo& g, const double* X,
                               float* val);
cudaError_t launch_lstarx_acc_f32(Launch L, const YlmTables& tb, const DevGeo& g,
                                  const float* xi, double* y);
// attributes of those kernels for one degree, once per context and device
cudaError_t prepare_lxs(int lmax);
// the triples' geometry (g.tgeo4, g.tgeo4d), once per molecule
cudaError_t launch_lxs_geo(Launch L, const YlmTables& tb, const DevGeo& g, float4* tg);
cudaError_t launch_lxs_geo_f64(Launch L, const YlmTables& tb, const DevGeo& g, double4* tg);
// pot_a(n) = sum of the lx values of the triples of (a, n); chi: times
// max(f_a(n), 1), the u_chi sum of the forces
cudaError_t launch_lx_gather(Launch L, const DevGeo& g, const double* val, double* pot,
                             bool chi = false);
// FP32 field rows are ldp >= ngrid floats apart (the tensor-core projection
// reads them with TMA, which wants 16-byte row strides)
cudaError_t launch_lx_gather_f32(Launch L, const DevGeo& g, const float* val, float* pot,
                                 int ldp);
cudaError_t launch_to_float(Launch L, long long n, const double* x, float* y);
// projection C(lm,i) = alpha sum_n w_n Y_lm(s_n) B(n,i) and expansion
// xi(n,i) = [w_n] sum_lm Y_lm(s_n) s(lm,i) over the reflection classes of grid
// and harmonics (ddc_fold.cu); FP64 arithmetic, FP64 or FP32 grid fields with
// rows ldb / ldc apart.  With act, blocks of skipped spheres are left alone.
bool fold_tables(const std::vector<double>& g4, int lmax, FoldTab& t, std::vector<short>& img,
                 std::vector<uint8_t>& first, std::vector<short>& lm);
cudaError_t launch_fold_pack(Launch L, const FoldTab& t, const double* basis, const double* bw,
                             double* pf, double* xw, double* xb);
template <class TB>
cudaError_t launch_fold_proj(Launch L, const FoldTab& t, int N, double alpha, const TB* B, int ldb,
                             double* C, const SweepMask& act);
template <class TC>
cudaError_t launch_fold_xi(Launch L, const FoldTab& t, bool weighted, int N, const double* s,
                           TC* xi, int ldc, const SweepMask& act);
// FP32 SIMT projection / expansion (mixed path, more than 128 harmonics)
cudaError_t launch_proj_f32_simt(Launch L, int nylm, int nsph, int ngrid, float alpha,
                                 const float* bw_f, const float* pot, int ldp, double* y);
cudaError_t launch_xi_f32_simt(Launch L, int nylm, int nsph, int ngrid, const float* bw_f,
                               const double* s, float* xi);
cudaError_t launch_wghpot(Launch L, const DevGeo& g, const double* phi, double* gbuf);
cudaError_t launch_ldm1x(Launch L, const YlmTables& tb, long long n, const double* x, double* y);
cudaError_t launch_guess(Launch L, const YlmTables& tb, long long n, const double* rhs,
                         double* x, int mode);

// tensor-core contractions of the mixed-precision operators (ddc_tc.cu):
// projection y = alpha * bw pot (FP64 out) and expansion w xi = bw^T s (FP32
// out), split-TF32 on tcgen05 for nylm <= 128
bool tc_supported(int nylm);
cudaError_t tc_plan(Launch L, TcPlan& p, const double* bw, int nsph, int nylm,
                    int ngrid, float* pot_f, int ldp);
// pick the tile widths of both kernels by timing the candidates (y, xi are
// scratch; s is zeroed)
cudaError_t tc_autotune(Launch L, TcPlan& p, const double* s, double* y, float* xi);
cudaError_t launch_proj_tc(Launch L, const TcPlan& p, double alpha, double* y,
                           const SweepMask& act = SweepMask{});
cudaError_t launch_xi_tc(Launch L, const TcPlan& p, const double* s, float* xi,
                         const SweepMask& act = SweepMask{});
void tc_release(TcPlan& p);

// learned initial guess (ddc_guess.cu)
int guess_nfeat(const ddc_guess* m);
int guess_nout(const ddc_guess* m);
int guess_lmax(const ddc_guess* m);
// raw per-sphere features [nsph][nin]: g (nylm), psi(00), radius, 16-bin
// histogram of the distances to the other centres of the sphere's molecule
cudaError_t launch_guess_features(Launch L, int nsph, int nylm, int nin, const double* g,
                                  const double* psi, const double4* sph, const int2* mrange,
                                  float* feat);
// training targets [nsph][nout]: X - facl g and S - facl psi
cudaError_t launch_guess_targets(Launch L, const YlmTables& tb, int nsph, int nout,
                                 const double* g, const double* psi, const double* X,
                                 const double* S, float* t);
// x = facl g + model correction, s = facl psi + model correction
cudaError_t guess_infer(Launch L, ddc_guess* m, const YlmTables& tb, int nsph, const float* feat,
                        const double* g, const double* psi, double* x, double* s);

// Jacobi/DIIS on the device (ddc_solver.cu), over the first ns systems of a
// (from a.first on): starting state; one half of an iteration after
// y = O x (which 0: Jacobi step and Gram solve, 1: extrapolation and stop
// test); the mixed refinement's residual at ox with y = O ox, and x += e
int solver_chunk(long long n_total, bool one);
// rows of the partial sums
int solver_parts(int nchunk, int chunk);
cudaError_t launch_solver_begin(Launch L, const SolverArgs& a, int ns, bool mixed);
cudaError_t launch_solver_step(Launch L, const SolverArgs& a, int ns, bool f32, int which);
cudaError_t launch_solver_residual(Launch L, const SolverArgs& a, int ns, bool f32_res);
cudaError_t launch_solver_update(Launch L, const SolverArgs& a, int ns);

cudaError_t launch_hnorm_partial(Launch L, const YlmTables& tb, long long n, const double* x,
                                 double* partials, int nblk);
cudaError_t launch_dot_partial(Launch L, long long n, const double* a, const double* b,
                               double* partials, int nblk);
// out[0] = sum_b partials[b], fixed order
cudaError_t launch_reduce_partials(Launch L, const double* partials, int nblk, double* out);
int reduce_blocks();

// electrostatics
// near / far split of the solute potential (and field) at the cavity points:
// charges farther than kFarRho * r_i from a sphere enter through a local
// expansion of degree kFarDegree about its centre, the others directly; used
// from kFarMinSpheres spheres on (below, the direct sums are cheaper)
constexpr int kFarDegree = 10;
constexpr double kFarRho = 8.0;
constexpr int kFarMinSpheres = 4096;
// BT[lm][n] = Y_lm(s_n), DT[k][lm][n] = grad_k R_lm(s_n) for the degree of tbP
cudaError_t launch_far_tables(Launch L, const YlmTables& tbP, const double4* grid, int ngrid,
                              double* BT, double* DT);
struct ZGroups;  // cell groups of one molecule (below)
// phi (and ef, if not null) at the cavity points; A: scratch [nsph][nylm(tbP)];
// zg (null for a batch): the near charges are searched in the candidate groups
cudaError_t launch_far_pot_field(Launch L, const YlmTables& tbP, int nsph, int ngrid,
                                 const double4* sph, const double* q, const int2* mrange,
                                 double rho, const int* cavoff, const int* cavpt,
                                 const double* ccav, const double* BT, const double* DT,
                                 double* A, double* phi, double* ef, const ZGroups* zg);
// Field of the cavity charges zeta at the nuclei in the mixed-precision
// energy+force flow (force-only, FP32 pair arithmetic): from
// kZetaMinSpheres spheres on, the spheres are grouped by the cells of a
// uniform grid (side >= kZetaCell bohr, Morton order), and a group farther
// than kZetaRho group radii from a nucleus acts through its multipole
// expansion of degree kZetaDegree; nearer groups are summed directly
constexpr int kZetaDegree = 16;
constexpr double kZetaRho = 3.0;
constexpr double kZetaCell = 12.0;
constexpr int kZetaMinSpheres = 4096;
// Cell groups of one molecule of kZetaMinSpheres spheres or more: the
// candidates of the neighbour list, of the near lists of the cavity far
// field and the source groups of the field of zeta
struct ZGroups {
  int ngroup = 0;
  int* cellid = nullptr;   // [nsph] scratch
  int* gsph = nullptr;     // [nsph] spheres in group order
  int* gstart = nullptr;   // [nsph+1] group g owns gsph[gstart[g] .. gstart[g+1])
  double4* gcen = nullptr; // [nsph] centroid and radius of each group
  int* gnpt = nullptr;     // [nsph+1] cavity points per group
  int* gptr = nullptr;     // [nsph+1] their exclusive scan
};
size_t zgroups_scan_bytes(int nsph);
// the cell groups of one molecule: members, centroids and radii (one host
// read of the group count); used by the neighbour list, the near lists of
// the cavity far field and the field of zeta
cudaError_t launch_zgroups_cells(Launch L, int nsph, const double4* sph, ZGroups& zg,
                                 int* dcount, int* hcount);
// per-group cavity-point counts and offsets (gnpt, gptr) for the field of zeta
cudaError_t launch_zgroups_points(Launch L, const int* cavoff, ZGroups& zg, void* scan_tmp,
                                  size_t scan_bytes);
// neighbour list of one molecule from its cell groups (same lists as
// launch_csr_count / launch_csr_fill)
cudaError_t launch_csr_count_cells(Launch L, int nsph, const double4* sph, const ZGroups& zg,
                                   int* cnt);
cudaError_t launch_csr_fill_cells(Launch L, int nsph, const double4* sph, const ZGroups& zg,
                                  const int* inl, int* nl);
int zgroups_nchunk(const ZGroups& zg);
size_t zgroups_moment_count(const ZGroups& zg);
// ef(3, nsph) from zeta(ncav); zpk[ncav], M[moment count], scratch
// [nchunk][nsph][3]
cudaError_t launch_zeta_field_far(Launch L, int nsph, const double4* sph, const int* cavoff,
                                  const double* ccav, const double* zeta, const ZGroups& zg,
                                  float4* zpk, float2* M, double* scratch, double* ef);
// trange: per target, the source index range it sums over (nullptr: all)
// launch_coulomb_pot plus the field of the same sources at the targets, ef (3, ntrg)
cudaError_t launch_coulomb_pot_field(Launch L, int nsrc, const double* q, const double* sx,
                                     const double* sy, const double* sz, int ntrg,
                                     const double* ctrg, double* phi, double* ef,
                                     const int2* trange);
// phi of charges at any points, partial sums as in launch_efield below
cudaError_t launch_coulomb_pot(Launch L, int nsrc, const double* q, const double* sx,
                               const double* sy, const double* sz, int ntrg, const double* ctrg,
                               double* phi, double* scratch, int nchunk, const int2* trange);
cudaError_t launch_psi(Launch L, int n, int nylm, const double* q, double* psi);
// field of sources (q at csrc(3,nsrc)) at targets ctrg(3,ntrg); partial sums
// over `nchunk` source chunks go to scratch[nchunk][ntrg][3]
cudaError_t launch_efield(Launch L, int nsrc, const double* q, const double* csrc, int ntrg,
                          const double* ctrg, double* ef, double* scratch, int nchunk,
                          const int2* trange);
int efield_chunks(int nsrc, int ntrg);
int efield_parts(int ntrg);  // nchunk where every target has its own range
// load k_efield / k_efield_reduce on the current device (one-time set-up)
cudaError_t preload_efield();
int efield_chunks_f32(int nsrc, int ntrg);
// FP32 pair arithmetic, FP64 accumulation (mixed-precision force terms)
cudaError_t launch_efield_f32(Launch L, int nsrc, const double* q, const double* csrc, int ntrg,
                              const double* ctrg, double* ef, double* scratch, int nchunk,
                              const int2* trange);

// forces
// fxa (3,N), fda (3,T) and fv (4 (lmax+1)(lmax+2)/2 pairs per sphere) are
// scratch of the force kernels
cudaError_t launch_forces(Launch L, const YlmTables& tb, const DevGeo& g, const double* sigma,
                          const double* s_xi, const double* u_chi, const double* phi,
                          double fep, double* fx, double* fxa, double* fda, double2* fv);
cudaError_t launch_mkxi(Launch L, const YlmTables& tb, const DevGeo& g, const double* xi_grid,
                        double scale, double* out);
cudaError_t launch_zeta_efld_contract(Launch L, const DevGeo& g, const double* zeta,
                                      const double* ef, double* fx);
cudaError_t launch_charge_efld_contract(Launch L, int n, const double* q, const double* ef,
                                        double* fx);
// batched solves
cudaError_t launch_batch_dot(Launch L, int nmol, const int* off, int nylm, const double* a,
                             const double* b, double scale, double* out);
cudaError_t launch_batch_ranges(Launch L, int nsph, int ngrid, int ncav, const int2* mrange,
                                const int* cavpt, const int* cavoff, int2* tr_cav, int2* tr_nuc);

// FP64 FMA throughput probe: each thread runs `iters` x 8 independent FMA chains
cudaError_t launch_fp64_probe(Launch L, int blocks, int iters, double* out);
cudaError_t launch_fp32_probe(Launch L, int blocks, int iters, float* out);

cudaError_t launch_csph_pack(Launch L, int n, const double4* sph, double* csph, double* sx,
                             double* sy, double* sz);

}  // namespace ddc
