// ddc_kernels.cu -- sm_100a kernels of the ddCOSMO path.
//
// Conventions.  Set-defining geometry (the neighbour test, t < 1, f_i, U_i,
// the switch band) is evaluated with round-to-nearest intrinsics in the
// reference's operation order (ddcosmo.f90:310-411, 1707-1716), so the GPU
// takes the same discrete decisions as an IEEE evaluation of the reference
// loops.  Inside the hot loops the arithmetic is free to contract and to
// reorder (values only), and every reduction has a fixed order, so results
// are deterministic from run to run.
#include <climits>

#include <cub/cub.cuh>
#include <type_traits>

#include "ddc_internal.h"

namespace ddc {

#define DADD __dadd_rn
#define DSUB __dsub_rn
#define DMUL __dmul_rn
#define DDIV __ddiv_rn

__host__ __device__ constexpr int lmi(int l, int m) { return l * (l + 1) / 2 + m; }


// ---------------------------------------------------------------------------
// exact geometry helpers
// ---------------------------------------------------------------------------
// v = (c_a + r_a * s) - c_b, |v|, t = |v| / r_b   (ddcosmo.f90:378-380)
struct Rel {
  double vx, vy, vz, vv, t;
};
__device__ __forceinline__ Rel rel_exact(double4 ca, double4 g, double4 cb) {
  Rel r;
  r.vx = DSUB(DADD(ca.x, DMUL(ca.w, g.x)), cb.x);
  r.vy = DSUB(DADD(ca.y, DMUL(ca.w, g.y)), cb.y);
  r.vz = DSUB(DADD(ca.z, DMUL(ca.w, g.z)), cb.z);
  r.vv = __dsqrt_rn(DADD(DADD(DMUL(r.vx, r.vx), DMUL(r.vy, r.vy)), DMUL(r.vz, r.vz)));
  r.t = DDIV(r.vv, cb.w);
  return r;
}
// |ca + ra g - cb|^2 with the rounding steps of rel_exact; above
// rb^2 (1 + 1e-10) the point is outside sphere b by far more than the
// rounding of rel_exact's t, so t >= 1 there: chi(t) = 0 and the pair
// contributes nothing (a cheap test ahead of the square root and division)
__device__ __forceinline__ bool rel_outside(double4 ca, double4 g, double4 cb) {
  const double vx = DSUB(DADD(ca.x, DMUL(ca.w, g.x)), cb.x);
  const double vy = DSUB(DADD(ca.y, DMUL(ca.w, g.y)), cb.y);
  const double vz = DSUB(DADD(ca.z, DMUL(ca.w, g.z)), cb.z);
  const double s2 = DADD(DADD(DMUL(vx, vx), DMUL(vy, vy)), DMUL(vz, vz));
  return s2 > cb.w * cb.w * (1.0 + 1e-10);
}

// switch function chi(t) and chi'(t) for se = -1 (ddcosmo.f90:566-655)
__device__ __forceinline__ double eta5(double eta) {
  double e2 = DMUL(eta, eta);
  return DMUL(DMUL(e2, e2), eta);
}
__device__ __forceinline__ double fsw_exact(double x, double eta) {
  if (x >= 1.0) return 0.0;
  if (x <= DSUB(1.0, eta)) return 1.0;
  double a = DSUB(DMUL(15.0, eta), 12.0);
  double b = DADD(DSUB(DMUL(DMUL(10.0, eta), eta), DMUL(15.0, eta)), 6.0);
  double xm = DSUB(x, 1.0);
  double p = DMUL(DMUL(xm, xm), DSUB(1.0, x));
  double q = DADD(DADD(DMUL(DMUL(6.0, x), x), DMUL(a, x)), b);
  return DDIV(DMUL(p, q), eta5(eta));
}
__device__ __forceinline__ double dfsw_exact(double x, double eta) {
  if (x >= 1.0) return 0.0;
  if (x <= DSUB(1.0, eta)) return 0.0;
  double xm = DSUB(x, 1.0);
  double xe = DADD(xm, eta);
  return DDIV(DMUL(DMUL(DMUL(DMUL(30.0, DSUB(1.0, x)), xm), xe), xe), eta5(eta));
}
// ---------------------------------------------------------------------------
// reference spherical harmonics (init only): ylmbas ddcosmo.f90:830-895
// ---------------------------------------------------------------------------
__device__ void ylmbas_ref(const YlmTables& tb, double sx, double sy, double sz, double* basloc) {
  const int lmax = tb.lmax;
  double vplm[(DDC_MAX_LMAX + 1) * (DDC_MAX_LMAX + 1)];
  double vc[DDC_MAX_LMAX + 2], vs[DDC_MAX_LMAX + 2];
  double cthe = sz;
  double sthe = __dsqrt_rn(DSUB(1.0, DMUL(cthe, cthe)));
  if (sthe != 0.0) {
    double cphi = DDIV(sx, sthe), sphi = DDIV(sy, sthe);
    vc[0] = 1.0; vs[0] = 0.0; vc[1] = cphi; vs[1] = sphi;
    for (int m = 2; m <= lmax; m++) {
      vc[m] = DSUB(DMUL(DMUL(2.0, cphi), vc[m - 1]), vc[m - 2]);
      vs[m] = DSUB(DMUL(DMUL(2.0, cphi), vs[m - 1]), vs[m - 2]);
    }
  } else {
    for (int m = 0; m <= lmax; m++) { vc[m] = 1.0; vs[m] = 0.0; }
  }
  // polleg (ddcosmo.f90:1056-1094)
  double fact = 1.0, pmm = 1.0;
  for (int m = 0; m <= lmax; m++) {
    int ind = (m + 1) * (m + 1) - 1;
    vplm[ind] = pmm;
    if (m == lmax) break;
    double fm = (double)m;
    double pmm1 = DMUL(DMUL(cthe, DADD(DMUL(2.0, fm), 1.0)), pmm);
    vplm[ind + 2 * m + 2] = pmm1;
    double pmmo = pmm;
    for (int l = m + 2; l <= lmax; l++) {
      double fl = (double)l;
      double pll = DDIV(DSUB(DMUL(DMUL(cthe, DSUB(DMUL(2.0, fl), 1.0)), pmm1),
                             DMUL(DSUB(DADD(fl, fm), 1.0), pmm)),
                        DSUB(fl, fm));
      vplm[l * l + l + m] = pll;
      pmm = pmm1;
      pmm1 = pll;
    }
    pmm = DMUL(DMUL(-pmmo, fact), sthe);
    fact = DADD(fact, 2.0);
  }
  for (int l = 0; l <= lmax; l++) {
    int ind = l * l + l;
    basloc[ind] = DMUL(tb.facs[lmi(l, 0)], vplm[ind]);
    for (int m = 1; m <= l; m++) {
      double plm = vplm[ind + m];
      basloc[ind + m] = DMUL(DMUL(tb.facs[lmi(l, m)], plm), vc[m]);
      basloc[ind - m] = DMUL(DMUL(tb.facs[lmi(l, m)], plm), vs[m]);
    }
  }
}

__global__ void k_basis(const YlmTables tb, const double4* __restrict__ grid, double* basis,
                        double* bw) {
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= tb.ngrid) return;
  double4 g = grid[n];
  double* b = basis + (size_t)n * tb.nylm;
  ylmbas_ref(tb, g.x, g.y, g.z, b);
  for (int k = 0; k < tb.nylm; k++) bw[(size_t)n * tb.nylm + k] = b[k] * g.w;
}

cudaError_t launch_basis(Launch L, const YlmTables& tb, const double4* grid, double* basis,
                         double* bw) {
  k_basis<<<(tb.ngrid + 63) / 64, 64, 0, L.st>>>(tb, grid, basis, bw);
  ++*L.launches;
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// CSR neighbour list: warp per sphere, ballot over candidates in index order
// (ddcosmo.f90:308-324); d^2 <= (r_i + r_j)^2
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool is_nb(double4 a, double4 b) {
  double dx = DSUB(a.x, b.x), dy = DSUB(a.y, b.y), dz = DSUB(a.z, b.z);
  double d2 = DADD(DADD(DMUL(dx, dx), DMUL(dy, dy)), DMUL(dz, dz));
  double rs = DADD(a.w, b.w);
  return d2 <= DMUL(rs, rs);
}

template <bool FILL>
__global__ void k_csr(int nsph, const double4* __restrict__ sph, int* cnt, const int* inl,
                      int* nl, const int2* __restrict__ mrange) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= nsph) return;
  const int i = warp;
  const double4 ci = sph[i];
  int base = FILL ? inl[i] : 0;
  // candidates: the sphere's own molecule (all spheres for a single molecule)
  const int jlo = mrange ? mrange[i].x : 0, jhi = mrange ? mrange[i].y : nsph;
  for (int j0 = jlo; j0 < jhi; j0 += 32) {
    int j = j0 + lane;
    bool nb = false;
    if (j < jhi && j != i) nb = is_nb(ci, sph[j]);
    unsigned mask = __ballot_sync(0xffffffffu, nb);
    if (FILL && nb) nl[base + __popc(mask & ((1u << lane) - 1u))] = j;
    base += __popc(mask);
  }
  if (!FILL && lane == 0) cnt[i] = base;
}

cudaError_t launch_csr_count(Launch L, int nsph, const double4* sph, int* cnt,
                             const int2* mrange) {
  k_csr<false><<<(nsph + 7) / 8, 256, 0, L.st>>>(nsph, sph, cnt, nullptr, nullptr, mrange);
  ++*L.launches;
  return cudaGetLastError();
}
cudaError_t launch_csr_fill(Launch L, int nsph, const double4* sph, const int* inl, int* nl,
                            const int2* mrange) {
  k_csr<true><<<(nsph + 7) / 8, 256, 0, L.st>>>(nsph, sph, nullptr, inl, nl, mrange);
  ++*L.launches;
  return cudaGetLastError();
}

// The same lists for one molecule from its cell groups (ddc_zfar.cu): a warp
// per sphere tests the groups' bounding spheres (a neighbour j of i lies in
// a group g with |c_i - c_g| <= r_i + R_g, since R_g >= |c_j - c_g| + r_j;
// a 1e-6 bohr margin covers rounding), then the candidate groups' members
// with the same overlap test as k_csr.  The fill pass ranks the sphere's
// neighbours (all distinct) into ascending order, so the list is the one
// k_csr writes.  Neighbour counts are at most 255 (checked before the fill).
template <bool FILL>
__global__ void __launch_bounds__(256) k_csr_cells(int nsph, const double4* __restrict__ sph,
                                                   const ZGroups zg, int* cnt, const int* inl,
                                                   int* nl) {
  __shared__ int buf[8][256];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + w;
  if (i >= nsph) return;  // warp-uniform; no block barriers
  const double4 ci = sph[i];
  int found = 0;
  for (int g0 = 0; g0 < zg.ngroup; g0 += 32) {
    const int g = g0 + lane;
    bool cand = false;
    if (g < zg.ngroup) {
      const double4 cg = zg.gcen[g];
      const double dx = ci.x - cg.x, dy = ci.y - cg.y, dz = ci.z - cg.z;
      const double lim = ci.w + cg.w + 1e-6;
      cand = dx * dx + dy * dy + dz * dz <= lim * lim;
    }
    unsigned m = __ballot_sync(0xffffffffu, cand);
    while (m) {
      const int gg = g0 + __ffs(m) - 1;
      m &= m - 1;
      const int s0 = zg.gstart[gg], s1 = zg.gstart[gg + 1];
      for (int k0 = s0; k0 < s1; k0 += 32) {
        const int k = k0 + lane;
        int j = -1;
        bool nb = false;
        if (k < s1) {
          j = zg.gsph[k];
          nb = j != i && is_nb(ci, sph[j]);
        }
        const unsigned bm = __ballot_sync(0xffffffffu, nb);
        if (FILL && nb) {
          const int pos = found + __popc(bm & ((1u << lane) - 1u));
          if (pos < 256) buf[w][pos] = j;
        }
        found += __popc(bm);
      }
    }
  }
  if constexpr (!FILL) {
    if (lane == 0) cnt[i] = found;
  } else {
    __syncwarp();
    const int base = inl[i], nf = min(found, 256);
    for (int e = lane; e < nf; e += 32) {
      const int v = buf[w][e];
      int r = 0;
      for (int f = 0; f < nf; ++f) r += buf[w][f] < v;
      nl[base + r] = v;
    }
  }
}
cudaError_t launch_csr_count_cells(Launch L, int nsph, const double4* sph, const ZGroups& zg,
                                   int* cnt) {
  k_csr_cells<false><<<(nsph + 7) / 8, 256, 0, L.st>>>(nsph, sph, zg, cnt, nullptr, nullptr);
  ++*L.launches;
  return cudaGetLastError();
}
cudaError_t launch_csr_fill_cells(Launch L, int nsph, const double4* sph, const ZGroups& zg,
                                  const int* inl, int* nl) {
  k_csr_cells<true><<<(nsph + 7) / 8, 256, 0, L.st>>>(nsph, sph, zg, nullptr, inl, nl);
  ++*L.launches;
  return cudaGetLastError();
}

// rev[k] for k = (i, j): position of i in the neighbour list of j
__global__ void k_csr_rev(int nsph, const int* __restrict__ inl, const int* __restrict__ nl,
                          int* rev) {
  int i = blockIdx.x;
  for (int k = inl[i] + threadIdx.x; k < inl[i + 1]; k += blockDim.x) {
    int j = nl[k];
    int lo = inl[j], hi = inl[j + 1] - 1, pos = -1;
    while (lo <= hi) {
      int mid = (lo + hi) >> 1;
      int v = nl[mid];
      if (v == i) { pos = mid; break; }
      if (v < i) lo = mid + 1; else hi = mid - 1;
    }
    rev[k] = pos;
  }
}
cudaError_t launch_csr_rev(Launch L, int nsph, const int* inl, const int* nl, int* rev) {
  if (nsph == 0) return cudaSuccess;
  k_csr_rev<<<nsph, 32, 0, L.st>>>(nsph, inl, nl, rev);
  ++*L.launches;
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// fi, ui, zi (ddcosmo.f90:363-411) and the per-point count of containing
// neighbours.  Thread per (sphere, grid point); a sphere's points (in patch
// order, as the whole grid is kept) are padded to whole warps, so that a warp's 32 points lie
// close together on the sphere and skip together the neighbours whose cap
// they all miss (rel_outside: those add exactly nothing).  Each point sums
// its neighbours in CSR order, as the reference does.
// ---------------------------------------------------------------------------
__global__ void k_fiui(const YlmTables tb, int nsph, const double4* __restrict__ sph,
                       const double4* __restrict__ grid,
                       const int* __restrict__ inl, const int* __restrict__ nl, double* fi,
                       double* ui, double* zi, uint8_t* ntri) {
  const int G = tb.ngrid, GP = (G + 31) & ~31;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)nsph * GP) return;
  const int i = (int)(t / GP), n = (int)(t - (long long)i * GP);
  if (n >= G) return;
  const long long p = (long long)i * G + n;
  double4 ci = sph[i], g = grid[n];
  double f = 0.0, zx = 0.0, zy = 0.0, zz = 0.0;
  int cnt = 0;
  const double eta = tb.eta;
  for (int k = inl[i]; k < inl[i + 1]; k++) {
    double4 cj = sph[nl[k]];
    if (rel_outside(ci, g, cj)) continue;  // t >= 1: no contribution
    Rel r = rel_exact(ci, g, cj);
    double xt = fsw_exact(r.t, eta);
    if (zi && r.t < 1.0 && r.t > DSUB(1.0, eta)) {
      double fac = DDIV(dfsw_exact(r.t, eta), cj.w);
      zx = DADD(zx, DDIV(DMUL(fac, r.vx), r.vv));
      zy = DADD(zy, DDIV(DMUL(fac, r.vy), r.vv));
      zz = DADD(zz, DDIV(DMUL(fac, r.vz), r.vv));
    }
    f = DADD(f, xt);
    if (r.t < 1.0) cnt++;
  }
  fi[p] = f;
  ui[p] = f <= 1.0 ? DSUB(1.0, f) : 0.0;
  ntri[p] = (uint8_t)(cnt > 255 ? 255 : cnt);
  if (zi) {
    zi[3 * p + 0] = zx;
    zi[3 * p + 1] = zy;
    zi[3 * p + 2] = zz;
  }
}
cudaError_t launch_fiui(Launch L, const YlmTables& tb, int nsph, const double4* sph,
                        const double4* grid, const int* inl, const int* nl,
                        double* fi, double* ui, double* zi, uint8_t* ntri) {
  const long long nt = (long long)nsph * ((tb.ngrid + 31) & ~31);
  if (nt == 0) return cudaSuccess;
  k_fiui<<<(unsigned)((nt + 255) / 256), 256, 0, L.st>>>(tb, nsph, sph, grid, inl, nl, fi,
                                                         ui, zi, ntri);
  ++*L.launches;
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// cavity compaction (ddcosmo.f90:422-468): points with ui > 0, sphere-major
// ---------------------------------------------------------------------------
__global__ void k_cav_count(int ngrid, const double* __restrict__ ui, int* cnt) {
  int i = blockIdx.x;
  int c = 0;
  for (int n = threadIdx.x; n < ngrid; n += blockDim.x) c += ui[(size_t)i * ngrid + n] > 0.0;
  typedef cub::BlockReduce<int, 256> BR;
  __shared__ typename BR::TempStorage tmp;
  int tot = BR(tmp).Sum(c);
  if (threadIdx.x == 0) cnt[i] = tot;
}
cudaError_t launch_cav_count(Launch L, int nsph, int ngrid, const double* ui, int* cnt) {
  if (nsph == 0) return cudaSuccess;
  k_cav_count<<<nsph, 256, 0, L.st>>>(ngrid, ui, cnt);
  ++*L.launches;
  return cudaGetLastError();
}

__global__ void k_cav_fill(int ngrid, const int* __restrict__ gpos, const double* __restrict__ ui,
                           const double4* __restrict__ sph, const double4* __restrict__ grid,
                           const int* __restrict__ cavoff, int* cavidx, int* cavpt, double* ccav) {
  int i = blockIdx.x;
  typedef cub::BlockScan<int, 256> BS;
  __shared__ typename BS::TempStorage tmp;
  __shared__ int carry;
  if (threadIdx.x == 0) carry = cavoff[i];
  __syncthreads();
  double4 ci = sph[i];
  // the cavity is numbered in the Lebedev order: point o sits at gpos[o]
  for (int n0 = 0; n0 < ngrid; n0 += 256) {
    const int o = n0 + threadIdx.x, n = o < ngrid ? gpos[o] : ngrid;
    size_t p = (size_t)i * ngrid + n;
    int flag = (n < ngrid && ui[p] > 0.0) ? 1 : 0;
    int pos, tot;
    BS(tmp).ExclusiveSum(flag, pos, tot);
    int base = carry;
    if (n < ngrid) {
      if (flag) {
        int c = base + pos;
        double4 g = grid[n];
        cavidx[p] = c;
        cavpt[c] = (int)p;
        ccav[3 * (size_t)c + 0] = DADD(ci.x, DMUL(ci.w, g.x));
        ccav[3 * (size_t)c + 1] = DADD(ci.y, DMUL(ci.w, g.y));
        ccav[3 * (size_t)c + 2] = DADD(ci.z, DMUL(ci.w, g.z));
      } else {
        cavidx[p] = -1;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) carry = base + tot;
    __syncthreads();
  }
}
cudaError_t launch_cav_fill(Launch L, int nsph, int ngrid, const int* gpos, const double* ui,
                            const double4* sph, const double4* grid, const int* cavoff,
                            int* cavidx, int* cavpt, double* ccav) {
  if (nsph == 0) return cudaSuccess;
  k_cav_fill<<<nsph, 256, 0, L.st>>>(ngrid, gpos, ui, sph, grid, cavoff, cavidx, cavpt, ccav);
  ++*L.launches;
  return cudaGetLastError();
}

// out(o, i) = ui(gpos[o], i): a grid field in the Lebedev order
__global__ void k_grid_order(long long np, int ngrid, const int* __restrict__ gpos,
                             const double* __restrict__ f, double* out) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const int o = (int)(p % ngrid);
  out[p] = f[p - o + gpos[o]];
}
cudaError_t launch_grid_order(Launch L, int nsph, int ngrid, const int* gpos, const double* f,
                              double* out) {
  const long long np = (long long)nsph * ngrid;
  if (np == 0) return cudaSuccess;
  k_grid_order<<<(unsigned)((np + 255) / 256), 256, 0, L.st>>>(np, ngrid, gpos, f, out);
  ++*L.launches;
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// pair-major triple lists: for CSR entry k = (i, j), the grid points n of
// sphere i with t_n^ij < 1 (calcv's test, ddcosmo.f90:1707-1716).  Warp per
// pair, ballot over points in ascending order.
// ---------------------------------------------------------------------------
// The count pass stores each pair's membership bits (one 32-bit word per 32
// grid points), and the fill pass expands them: the exact geometry of every
// (pair, point) is evaluated once
template <bool FILL>
__global__ void k_pairs(int nsph, int npair, int ngrid, const double4* __restrict__ sph,
                        const double4* __restrict__ grid, const int* __restrict__ inl,
                        const int* __restrict__ nl, int* cnt, unsigned* __restrict__ bits,
                        const int* pn_ptr, uint16_t* pn) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= npair) return;
  const int k = warp;
  const int nw = (ngrid + 31) >> 5;
  unsigned* kb = bits + (size_t)k * nw;
  if constexpr (!FILL) {
    // sphere owning entry k: binary search in inl
    int lo = 0, hi = nsph - 1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (inl[mid] <= k) lo = mid; else hi = mid - 1;
    }
    const int i = lo, j = nl[k];
    const double4 ci = sph[i], cj = sph[j];
    int total = 0;
    for (int w = 0; w < nw; ++w) {
      const int n = 32 * w + lane;
      bool in = false;
      if (n < ngrid) in = rel_exact(ci, grid[n], cj).t < 1.0;
      const unsigned mask = __ballot_sync(0xffffffffu, in);
      if (lane == 0) kb[w] = mask;
      total += __popc(mask);
    }
    if (lane == 0) cnt[k] = total;
  } else {
    int base = pn_ptr[k];
    for (int w = 0; w < nw; ++w) {
      const unsigned mask = kb[w];
      if ((mask >> lane) & 1u) {
        const int pos = base + __popc(mask & ((1u << lane) - 1u));
        pn[pos] = (uint16_t)(32 * w + lane);
      }
      base += __popc(mask);
    }
  }
}
cudaError_t launch_pair_count(Launch L, int nsph, int npair, int ngrid, const double4* sph,
                              const double4* grid, const int* inl, const int* nl, int* cnt,
                              unsigned* bits) {
  if (npair == 0) return cudaSuccess;
  k_pairs<false><<<(npair + 7) / 8, 256, 0, L.st>>>(nsph, npair, ngrid, sph, grid, inl, nl, cnt,
                                                    bits, nullptr, nullptr);
  ++*L.launches;
  return cudaGetLastError();
}
cudaError_t launch_pair_fill(Launch L, int nsph, int npair, int ngrid, const double4* sph,
                             const double4* grid, const int* inl, const int* nl,
                             const unsigned* bits, const int* pn_ptr, uint16_t* pn) {
  if (npair == 0) return cudaSuccess;
  k_pairs<true><<<(npair + 7) / 8, 256, 0, L.st>>>(nsph, npair, ngrid, sph, grid, inl, nl,
                                                   nullptr, const_cast<unsigned*>(bits), pn_ptr,
                                                   pn);
  ++*L.launches;
  return cudaGetLastError();
}

// adjoint gather list: for sphere i, for j in N_i (CSR order), points of j
// inside i = pair list of entry rev(k) (adjrhs ddcosmo.f90:1316-1381)
__global__ void k_ls_count(int nsph, const int* __restrict__ inl, const int* __restrict__ rev,
                           const int* __restrict__ pn_ptr, int* cnt) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nsph) return;
  int c = 0;
  for (int k = inl[i]; k < inl[i + 1]; k++) {
    int kk = rev[k];
    c += pn_ptr[kk + 1] - pn_ptr[kk];
  }
  cnt[i] = c;
}
cudaError_t launch_ls_count(Launch L, int nsph, const int* inl, const int* rev, const int* pn_ptr,
                            int* cnt) {
  if (nsph == 0) return cudaSuccess;
  k_ls_count<<<(nsph + 127) / 128, 128, 0, L.st>>>(nsph, inl, rev, pn_ptr, cnt);
  ++*L.launches;
  return cudaGetLastError();
}
__global__ void k_ls_fill(int nsph, const int* __restrict__ inl, const int* __restrict__ nl,
                          const int* __restrict__ rev, const int* __restrict__ pn_ptr,
                          const uint16_t* __restrict__ pn, const int* __restrict__ ls_ptr,
                          int ngrid, int* ls, int* lsstart) {
  int i = blockIdx.x;
  int off = ls_ptr[i];
  for (int k = inl[i]; k < inl[i + 1]; k++) {
    int kk = rev[k], j = nl[k];
    int a = pn_ptr[kk], b = pn_ptr[kk + 1];
    if (threadIdx.x == 0) lsstart[kk] = off;  // where pair (j, i) sits in i's gather list
    for (int t = threadIdx.x; t < b - a; t += blockDim.x) ls[off + t] = j * ngrid + pn[a + t];
    off += b - a;
  }
}
cudaError_t launch_ls_fill(Launch L, int nsph, const int* inl, const int* nl, const int* rev,
                           const int* pn_ptr, const uint16_t* pn, const int* ls_ptr, int ngrid,
                           int* ls, int* lsstart) {
  if (nsph == 0) return cudaSuccess;
  k_ls_fill<<<nsph, 128, 0, L.st>>>(nsph, inl, nl, rev, pn_ptr, pn, ls_ptr, ngrid, ls, lsstart);
  ++*L.launches;
  return cudaGetLastError();
}

__global__ void k_sum_counts(const int* __restrict__ cnt, int n, CountStats* out) {
  unsigned long long v = 0;
  int m = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    v += (unsigned long long)(unsigned)cnt[i];
    m = max(m, cnt[i]);
  }
  for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0 && v) {  // integer sum and maximum: order-free
    atomicAdd(&out->total, v);
    atomicMax(&out->largest, m);
  }
}
// Counting sort of the lists by falling length, one block.  Lists of one bucket
// come in any order: it only sets which block of a pass takes which list.
constexpr int kOrderB = 1024;
__global__ void __launch_bounds__(kOrderB) k_ls_order(int n, const int* __restrict__ ptr,
                                                      const CountStats* __restrict__ st,
                                                      int* __restrict__ order) {
  typedef cub::BlockScan<int, kOrderB> BS;
  __shared__ typename BS::TempStorage tmp;
  __shared__ int at[kOrderB];
  const float scale = (float)kOrderB / (float)(st->largest + 1);
  auto bucket = [&](int i) {
    return kOrderB - 1 - min(kOrderB - 1, (int)((float)(ptr[i + 1] - ptr[i]) * scale));
  };
  at[threadIdx.x] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kOrderB) atomicAdd(&at[bucket(i)], 1);
  __syncthreads();
  int v = at[threadIdx.x];
  BS(tmp).ExclusiveSum(v, v);
  at[threadIdx.x] = v;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kOrderB) order[atomicAdd(&at[bucket(i)], 1)] = i;
}
cudaError_t launch_ls_order(Launch L, int n, const int* ptr, const CountStats* st, int* order) {
  if (n == 0) return cudaSuccess;
  k_ls_order<<<1, kOrderB, 0, L.st>>>(n, ptr, st, order);
  ++*L.launches;
  return cudaGetLastError();
}

// The scan, the total and the maximum of a short list: one block, eight
// counts per thread and step.
constexpr int kScanT = 1024, kScanU = 8;
__global__ void __launch_bounds__(kScanT) k_scan_short(const int* __restrict__ cnt, int n,
                                                      int* __restrict__ out, CountStats* st) {
  typedef cub::BlockScan<int, kScanT> BS;
  __shared__ typename BS::TempStorage tmp;
  __shared__ unsigned long long s_tot;
  __shared__ int s_max;
  if (threadIdx.x == 0) {
    s_tot = 0;
    s_max = 0;
  }
  unsigned long long tot = 0;
  int mx = 0, run = 0;
  for (int b0 = 0; b0 < n; b0 += kScanT * kScanU) {
    const int i0 = b0 + threadIdx.x * kScanU;
    int v[kScanU], sum;
#pragma unroll
    for (int k = 0; k < kScanU; ++k) {
      v[k] = i0 + k < n ? cnt[i0 + k] : 0;
      tot += (unsigned long long)(unsigned)v[k];
      mx = max(mx, v[k]);
    }
    __syncthreads();  // tmp is free
    BS(tmp).ExclusiveSum(v, v, sum);
#pragma unroll
    for (int k = 0; k < kScanU; ++k)
      if (i0 + k < n) out[i0 + k] = run + v[k];
    run += sum;
  }
  for (int o = 16; o >= 1; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  mx = __reduce_max_sync(0xffffffffu, mx);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&s_tot, tot);
    atomicMax(&s_max, mx);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    out[n] = run;
    st->total = s_tot;
    st->largest = s_max;
  }
}

size_t scan_temp_bytes(int n) {
  size_t b = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, b, (const int*)nullptr, (int*)nullptr, n + 1);
  return b;
}
// in[0..n-1] -> out[0..n] with out[n] = total (in[n] is set to zero here: the
// caller's buffer holds n+1 entries)
cudaError_t scan_exclusive(Launch L, int* in, int* out, int n, void* temp, size_t temp_bytes) {
  const cudaError_t e = cudaMemsetAsync(in + n, 0, sizeof(int), L.st);
  if (e) return e;
  return cub::DeviceScan::ExclusiveSum(temp, temp_bytes, in, out, n + 1, L.st);
}
// One block up to 32,768 counts (15 us there, 4 us for a thousand, against
// four launches); the device-wide scan and a separate sum above
cudaError_t scan_counts(Launch L, int* cnt, int* out, int n, void* temp, size_t temp_bytes,
                        CountStats* st) {
  if (n <= 32768) {
    k_scan_short<<<1, kScanT, 0, L.st>>>(cnt, n, out, st);
    ++*L.launches;
    return cudaGetLastError();
  }
  cudaError_t e = cudaMemsetAsync(st, 0, sizeof(CountStats), L.st);
  if (e) return e;
  k_sum_counts<<<std::min((n + 255) / 256, 148 * 4), 256, 0, L.st>>>(cnt, n, st);
  ++*L.launches;
  if ((e = cudaGetLastError())) return e;
  return scan_exclusive(L, cnt, out, n, temp, temp_bytes);
}

// 1/sqrt(x) for a positive normal x (a squared distance between distinct
// points) in the N-body sums: the hardware estimate rsqrt.approx.ftz.f64,
// then one third-order Householder step y (1 + h/2 + 3h^2/8), h = 1 - x y^2
// (the binomial series of (1 - h)^(-1/2) to second order).  The step cubes
// the estimate's relative error, so the result carries only the rounding of
// its five FP64 operations; no special-value handling is needed for such x.
__device__ __forceinline__ double rsqrt_pos(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double h = fma(-x, y * y, 1.0);
  return fma(y * h, fma(h, 0.375, 0.5), y);
}
#define DDC_LMAX_CASES(X) \
  X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12)

__host__ __device__ constexpr int ls_nvals_m(int L, int m) { return m == 0 ? L + 1 : 2 * (L + 1 - m); }
// shared-memory fields per triple: ct, t2, then pmm[m], cos[m], sin[m]
__host__ __device__ constexpr int ls_nfields(int L) { return 2 + 3 * (L + 1); }

// column M of the normalised recurrence's accumulators, with its scale
template <int LMAX, int M, int OFF>
__device__ __forceinline__ void ls_store(const YlmTables& tb, const double* acc, double* yi,
                                         int lane) {
#pragma unroll
  for (int l = M; l <= LMAX; ++l) {
    const int ind = l * l + l;
    const double k = tb.Kg[lmi(l, M)];
    if (M == 0) {
      if (lane == 0) yi[ind] = -k * acc[OFF + (l - M)];
    } else if (lane == 0) {
      yi[ind + M] = -k * acc[OFF + (l - M)];
      yi[ind - M] = -k * acc[OFF + (LMAX + 1 - M) + (l - M)];
    }
  }
}

// ---------------------------------------------------------------------------
// Register-tiled SIMT GEMM, column-major C[M x N] = alpha * op(A) * B: the
// FP32 projection and expansion of the mixed path when the harmonics do not
// fit one 128-row tensor-core tile (lmax 11, 12).  BM x BN tile per block,
// BK deep, TM x TN outputs per thread, shared tiles double buffered with the
// next tile prefetched into registers.  Acc is the arithmetic/accumulation
// type; inputs are converted when staged.
// ---------------------------------------------------------------------------
template <bool TA, class TAin, class TBin, class TC, class Acc, int BM, int BN, int BK, int TM,
          int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) k_gemm2(int M, int N, int K, Acc alpha,
                                                                 const TAin* __restrict__ A,
                                                                 int lda,
                                                                 const TBin* __restrict__ B,
                                                                 int ldb, TC* C, int ldc) {
  constexpr int NT = (BM / TM) * (BN / TN);
  constexpr int NA = BM * BK / NT, NB = BK * BN / NT;  // staged elements per thread
  __shared__ __align__(16) Acc As[2][BK][BM];
  __shared__ __align__(16) Acc Bs[2][BK][BN];
  const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  Acc ra[NA], rb[NB];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int u = 0; u < NA; ++u) {
      const int e = threadIdx.x + u * NT;
      int mm, kk;
      if (TA) { kk = e % BK; mm = e / BK; } else { mm = e % BM; kk = e / BM; }
      const int m = m0 + mm, k = k0 + kk;
      Acc v = 0;
      if (m < M && k < K) v = (Acc)(TA ? A[(size_t)m * lda + k] : A[(size_t)k * lda + m]);
      ra[u] = v;
    }
#pragma unroll
    for (int u = 0; u < NB; ++u) {
      const int e = threadIdx.x + u * NT;
      const int kk = e % BK, nn = e / BK;
      const int n = n0 + nn, k = k0 + kk;
      rb[u] = (n < N && k < K) ? (Acc)B[(size_t)n * ldb + k] : Acc(0);
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int u = 0; u < NA; ++u) {
      const int e = threadIdx.x + u * NT;
      int mm, kk;
      if (TA) { kk = e % BK; mm = e / BK; } else { mm = e % BM; kk = e / BM; }
      As[buf][kk][mm] = ra[u];
    }
#pragma unroll
    for (int u = 0; u < NB; ++u) {
      const int e = threadIdx.x + u * NT;
      Bs[buf][e % BK][e / BK] = rb[u];
    }
  };
  Acc acc[TM][TN];
#pragma unroll
  for (int a = 0; a < TM; ++a)
#pragma unroll
    for (int b = 0; b < TN; ++b) acc[a][b] = 0;
  fetch(0);
  stash(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += BK) {
    const bool more = k0 + BK < K;
    if (more) fetch(k0 + BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      Acc a[TM], b[TN];
#pragma unroll
      for (int r = 0; r < TM; ++r) a[r] = As[buf][kk][ty * TM + r];
#pragma unroll
      for (int c = 0; c < TN; ++c) b[c] = Bs[buf][kk][tx * TN + c];
#pragma unroll
      for (int r = 0; r < TM; ++r)
#pragma unroll
        for (int c = 0; c < TN; ++c) acc[r][c] = fma(a[r], b[c], acc[r][c]);
    }
    if (more) {
      stash(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }
#pragma unroll
  for (int r = 0; r < TM; ++r)
#pragma unroll
    for (int c = 0; c < TN; ++c) {
      const int m = m0 + ty * TM + r, n = n0 + tx * TN + c;
      if (m < M && n < N) C[(size_t)n * ldc + m] = (TC)(alpha * acc[r][c]);
    }
}

template <bool TA, class TAin, class TBin, class TC, class Acc>
cudaError_t gemm2(Launch L, int M, int N, int K, Acc alpha, const TAin* A, int lda, const TBin* B,
                  int ldb, TC* C, int ldc) {
  if (M == 0 || N == 0) return cudaSuccess;
  // FP32: 128x64 tiles, 8x4 per thread; FP64: 128x32 tiles, 8x2 per thread
  constexpr bool D = sizeof(Acc) == 8;
  constexpr int BM = 128, BN = D ? 32 : 64, TM = 8, TN = D ? 2 : 4, BK = D ? 8 : 16;
  dim3 grid((M + BM - 1) / BM, (N + BN - 1) / BN);
  k_gemm2<TA, TAin, TBin, TC, Acc, BM, BN, BK, TM, TN>
      <<<grid, (BM / TM) * (BN / TN), 0, L.st>>>(M, N, K, alpha, A, lda, B, ldb, C, ldc);
  ++*L.launches;
  return cudaGetLastError();
}

// FP32 SIMT contractions of the mixed path where the tensor-core kernels do
// not apply (more than 128 harmonics): projection into FP64 y, and xi of the
// FP64 vector s
cudaError_t launch_proj_f32_simt(Launch L, int nylm, int nsph, int ngrid, float alpha,
                                 const float* bw_f, const float* pot, int ldp, double* y) {
  return gemm2<false, float, float, double, float>(L, nylm, nsph, ngrid, alpha, bw_f, nylm, pot,
                                                   ldp, y, nylm);
}
cudaError_t launch_xi_f32_simt(Launch L, int nylm, int nsph, int ngrid, const float* bw_f,
                               const double* s, float* xi) {
  return gemm2<true, float, double, float, float>(L, ngrid, nsph, nylm, 1.f, bw_f, nylm, s,
                                                  nylm, xi, ngrid);
}


// wghpot (ddcosmo.f90:1187-1224): g(n,i) = -ui * phi(cavity index)
__global__ void k_wghpot(long long np, const double* __restrict__ ui, const int* __restrict__ cavidx,
                         const double* __restrict__ phi, double* gb) {
  long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  int c = cavidx[p];
  gb[p] = c >= 0 ? -ui[p] * phi[c] : 0.0;
}
cudaError_t launch_wghpot(Launch L, const DevGeo& g, const double* phi, double* gbuf) {
  long long np = (long long)g.nsph * g.ngrid;
  if (np == 0) return cudaSuccess;
  k_wghpot<<<(unsigned)((np + 255) / 256), 256, 0, L.st>>>(np, g.ui, g.cavidx, phi, gbuf);
  ++*L.launches;
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// vector kernels of the Jacobi/DIIS solver (jacobi_diis.f90)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int l_of(int lm) {
  int l = (int)sqrtf((float)lm);
  while ((l + 1) * (l + 1) <= lm) ++l;
  while (l * l > lm) --l;
  return l;
}

// Grid-stride walk over the (nylm, nsph) vectors that keeps the harmonic
// index lm = q mod nylm incrementally (no 64-bit division per element).
struct LmWalk {
  long long q, stride;
  int lm, dlm, nylm;
  __device__ LmWalk(int nylm_) : nylm(nylm_) {
    q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    stride = (long long)gridDim.x * blockDim.x;
    lm = (int)(q % nylm);
    dlm = (int)(stride % nylm);
  }
  __device__ void next() {
    q += stride;
    lm += dlm;
    if (lm >= nylm) lm -= nylm;
  }
};

__global__ void k_ldm1x(const YlmTables tb, long long n, const double* __restrict__ x, double* y) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  int lm = (int)(e % tb.nylm);
  y[e] = tb.facl[l_of(lm)] * x[e];
}
cudaError_t launch_ldm1x(Launch L, const YlmTables& tb, long long n, const double* x, double* y) {
  if (n == 0) return cudaSuccess;
  k_ldm1x<<<(unsigned)((n + 255) / 256), 256, 0, L.st>>>(tb, n, x, y);
  ++*L.launches;
  return cudaGetLastError();
}
// mode 0: x = facl * rhs (cosmo.f90:136-138), 1: x = 0
__global__ void k_guess(const YlmTables tb, long long n, const double* __restrict__ rhs, double* x,
                        int mode) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  x[e] = mode == 0 ? tb.facl[l_of((int)(e % tb.nylm))] * rhs[e] : 0.0;
}
cudaError_t launch_guess(Launch L, const YlmTables& tb, long long n, const double* rhs, double* x,
                         int mode) {
  if (n == 0) return cudaSuccess;
  k_guess<<<(unsigned)((n + 255) / 256), 256, 0, L.st>>>(tb, n, rhs, x, mode);
  ++*L.launches;
  return cudaGetLastError();
}

int reduce_blocks() { return 148 * 4; }

// block sum of x into partials[blockIdx.x] (blocks of at most 256 threads)
__device__ __forceinline__ void block_sum_store(double x, double* partials) {
  __shared__ double sh[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  if (lane == 0) sh[w] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int ww = 0; ww < (int)(blockDim.x >> 5); ++ww) s += sh[ww];
    partials[blockIdx.x] = s;
  }
}

__global__ void __launch_bounds__(256) k_hnorm_partial(const YlmTables tb, long long n,
                                                       const double* __restrict__ x,
                                                       double* partials) {
  double acc = 0.0;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x) {
    int l = l_of((int)(q % tb.nylm));
    acc = fma(x[q] * x[q], 1.0 / (1.0 + l), acc);
  }
  block_sum_store(acc, partials);
}
cudaError_t launch_hnorm_partial(Launch L, const YlmTables& tb, long long n, const double* x,
                                 double* partials, int nblk) {
  k_hnorm_partial<<<nblk, 256, 0, L.st>>>(tb, n, x, partials);
  ++*L.launches;
  return cudaGetLastError();
}

__global__ void __launch_bounds__(256) k_dot_partial(long long n, const double* __restrict__ a,
                                                     const double* __restrict__ b,
                                                     double* partials) {
  double acc = 0.0;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x)
    acc = fma(a[q], b[q], acc);
  block_sum_store(acc, partials);
}
cudaError_t launch_dot_partial(Launch L, long long n, const double* a, const double* b,
                               double* partials, int nblk) {
  k_dot_partial<<<nblk, 256, 0, L.st>>>(n, a, b, partials);
  ++*L.launches;
  return cudaGetLastError();
}

// out[0] = sum over blocks of partials[b] in a fixed tree order
__global__ void k_reduce_partials(const double* __restrict__ partials, int nblk, double* out) {
  __shared__ double sh[256];
  double s = 0.0;
  for (int b = threadIdx.x; b < nblk; b += 256) s += partials[b];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int h = 128; h >= 1; h >>= 1) {
    if (threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = sh[0];
}
cudaError_t launch_reduce_partials(Launch L, const double* partials, int nblk, double* out) {
  k_reduce_partials<<<1, 256, 0, L.st>>>(partials, nblk, out);
  ++*L.launches;
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// solute electrostatics (mkrhs.f90:100-120, efld.f90:97-114): direct sums
// with source tiles staged in shared memory, summed in source order.
// ---------------------------------------------------------------------------
constexpr int kNbTile = 256;
// FP64 field: shortest chunk of sources
constexpr int kFieldChunk = 64;
// Source range of each thread's target ([0, nsrc) for one molecule; the
// target's own molecule in a batch) and the union over the block.
struct SrcRange {
  int lo, hi, ulo, uhi;
};
__device__ __forceinline__ SrcRange block_src_range(const int2* trange, int t, int ntrg,
                                                    int s0, int s1) {
  __shared__ int b_lo, b_hi;
  SrcRange r;
  r.lo = s0;
  r.hi = s1;
  if (trange) {
    if (t < ntrg) {
      int2 v = trange[t];
      r.lo = max(v.x, s0);
      r.hi = min(v.y, s1);
    } else {
      r.lo = s1;
      r.hi = s0;
    }
  }
  if (threadIdx.x == 0) {  // an empty range unless a thread has sources
    b_lo = s1;
    b_hi = min(s0, s1);
  }
  __syncthreads();
  if (r.lo < r.hi) {
    atomicMin(&b_lo, r.lo);
    atomicMax(&b_hi, r.hi);
  }
  __syncthreads();
  r.ulo = b_lo;
  r.uhi = b_hi;
  return r;
}
// Source range of part c of a field kernel's block: one molecule, chunk c of
// all sources; several, part c of gridDim.y of the tiles of the union of the
// block's ranges.  (The tiles start where the whole union does, whatever the
// number of parts: the FP32 sum of a tile is the same.)
__device__ __forceinline__ SrcRange field_src_range(const int2* trange, int t, int ntrg,
                                                    int nsrc, int chunk) {
  const int c = blockIdx.y;
  if (!trange)
    return block_src_range(nullptr, t, ntrg, c * chunk, min(nsrc, c * chunk + chunk));
  SrcRange r = block_src_range(trange, t, ntrg, 0, nsrc);
  const int tiles = (max(r.uhi - r.ulo, 0) + kNbTile - 1) / kNbTile;
  const int per = (tiles + gridDim.y - 1) / gridDim.y * kNbTile;
  r.ulo = min(r.ulo + c * per, max(r.uhi, r.ulo));
  r.uhi = min(r.uhi, r.ulo + per);
  return r;
}

// Potential of point charges; partial sums over chunks of the sources (grid y).
// Bound by the FP64 pipe, 12 operations per pair.  50,003 targets are 196
// blocks, one or two per SM: 30,001 sources took 1.86 ms in one piece and take
// 1.3 ms in seven.
__global__ void __launch_bounds__(kNbTile) k_coulomb_pot(int nsrc, const double* __restrict__ q,
                                                         const double* __restrict__ sx,
                                                         const double* __restrict__ sy,
                                                         const double* __restrict__ sz,
                                                         int ntrg, const double* __restrict__ ctrg,
                                                         int chunk, double* phi,
                                                         const int2* __restrict__ trange) {
  __shared__ double4 src[kNbTile];
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  double px = 0, py = 0, pz = 0;
  if (t < ntrg) {
    px = ctrg[3 * (size_t)t];
    py = ctrg[3 * (size_t)t + 1];
    pz = ctrg[3 * (size_t)t + 2];
  }
  const SrcRange rg = field_src_range(trange, t, ntrg, nsrc, chunk);
  double v = 0.0;
  for (int j0 = rg.ulo; j0 < rg.uhi; j0 += kNbTile) {
    const int j = j0 + threadIdx.x;
    __syncthreads();
    src[threadIdx.x] = j < rg.uhi ? make_double4(sx[j], sy[j], sz[j], q[j])
                              : make_double4(0, 0, 0, 0);
    __syncthreads();
    const int kb = max(rg.lo - j0, 0), ke = min(rg.hi - j0, min(kNbTile, rg.uhi - j0));
    auto pair = [&](const double4& s) {
      const double dx = px - s.x, dy = py - s.y, dz = pz - s.z;
      v = fma(s.w, rsqrt_pos(dx * dx + dy * dy + dz * dz), v);
    };
    if (kb == 0 && ke == kNbTile) {
#pragma unroll 8
      for (int k = 0; k < kNbTile; ++k) pair(src[k]);
    } else {
      for (int k = kb; k < ke; ++k) pair(src[k]);
    }
  }
  if (t < ntrg) phi[(size_t)blockIdx.y * ntrg + t] = v;
}
// The potential and, for the forces, the solute's field at the same targets
// (efld.f90:97-114 with the nuclei as sources) from one pass over the pairs:
// per pair the field adds q r^-3 (p - s) to the potential's q r^-1.
__global__ void __launch_bounds__(kNbTile) k_coulomb_pot_field(
    int nsrc, const double* __restrict__ q, const double* __restrict__ sx,
    const double* __restrict__ sy, const double* __restrict__ sz, int ntrg,
    const double* __restrict__ ctrg, double* phi, double* ef, const int2* __restrict__ trange) {
  __shared__ double4 src[kNbTile];
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  double px = 0, py = 0, pz = 0;
  if (t < ntrg) {
    px = ctrg[3 * (size_t)t];
    py = ctrg[3 * (size_t)t + 1];
    pz = ctrg[3 * (size_t)t + 2];
  }
  const SrcRange rg = block_src_range(trange, t, ntrg, 0, nsrc);
  double v = 0.0, ex = 0.0, ey = 0.0, ez = 0.0;
  auto pair = [&](const double4& s) {
    const double dx = px - s.x, dy = py - s.y, dz = pz - s.z;
    const double ri = rsqrt_pos(dx * dx + dy * dy + dz * dz);
    v = fma(s.w, ri, v);
    const double f = s.w * (ri * ri * ri);
    ex = fma(f, dx, ex);
    ey = fma(f, dy, ey);
    ez = fma(f, dz, ez);
  };
  for (int j0 = rg.ulo; j0 < rg.uhi; j0 += kNbTile) {
    int j = j0 + threadIdx.x;
    __syncthreads();
    src[threadIdx.x] = j < rg.uhi ? make_double4(sx[j], sy[j], sz[j], q[j])
                                  : make_double4(0, 0, 0, 0);
    __syncthreads();
    int cnt = min(kNbTile, rg.uhi - j0);
    const int kb = max(rg.lo - j0, 0), ke = min(rg.hi - j0, cnt);
    if (kb == 0 && ke == kNbTile) {
#pragma unroll 4
      for (int k = 0; k < kNbTile; ++k) pair(src[k]);
    } else {
      for (int k = kb; k < ke; ++k) pair(src[k]);
    }
  }
  if (t < ntrg) {
    phi[t] = v;
    ef[3 * (size_t)t] = ex;
    ef[3 * (size_t)t + 1] = ey;
    ef[3 * (size_t)t + 2] = ez;
  }
}
cudaError_t launch_coulomb_pot_field(Launch L, int nsrc, const double* q, const double* sx,
                                     const double* sy, const double* sz, int ntrg,
                                     const double* ctrg, double* phi, double* ef,
                                     const int2* trange) {
  if (ntrg == 0) return cudaSuccess;
  k_coulomb_pot_field<<<(ntrg + kNbTile - 1) / kNbTile, kNbTile, 0, L.st>>>(
      nsrc, q, sx, sy, sz, ntrg, ctrg, phi, ef, trange);
  ++*L.launches;
  return cudaGetLastError();
}
__global__ void k_psi(int n, int nylm, const double* __restrict__ q, double* psi) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)n * nylm) return;
  int i = (int)(e / nylm), lm = (int)(e - (long long)i * nylm);
  psi[e] = lm == 0 ? sqrt(16.0 * atan(1.0)) * q[i] : 0.0;
}
cudaError_t launch_psi(Launch L, int n, int nylm, const double* q, double* psi) {
  long long np = (long long)n * nylm;
  if (np == 0) return cudaSuccess;
  k_psi<<<(unsigned)((np + 255) / 256), 256, 0, L.st>>>(n, nylm, q, psi);
  ++*L.launches;
  return cudaGetLastError();
}

// Source chunks of the field kernels for few targets: enough blocks to fill the
// device, chunks of 1,024 sources or more, as every chunk costs a row of the
// reduction.  Up to 16 shorter ones are worth that where a chunk is walked
// alone: 12 targets and 587 sources in FP64 50 -> 15 us with chunks of 64.
static int field_chunks(int nsrc, int blocks, int shortest) {
  const int want = (148 * 8 + blocks - 1) / max(blocks, 1);
  const int maxc = max((nsrc + 4 * kNbTile - 1) / (4 * kNbTile),
                       min((nsrc + shortest - 1) / shortest, 16));
  return max(1, min(want, max(maxc, 1)));
}
int efield_chunks(int nsrc, int ntrg) {
  return field_chunks(nsrc, (ntrg + kNbTile - 1) / kNbTile, kFieldChunk);
}
// Parts of the sources when every target has its own range (batches): a block
// of 256 targets otherwise walks all sources of its molecules alone.  48
// molecules of 8 to 1,999 spheres, 18,000 targets in 70 blocks: 3.7 -> 0.7 ms.
int efield_parts(int ntrg) {
  const int tiles = (ntrg + kNbTile - 1) / kNbTile;
  return max(1, min((148 * 8 + tiles - 1) / max(tiles, 1), 64));
}
// source chunks for the FP32 field of one molecule: enough blocks of the
// two-targets-per-thread kernel (k_efield_f2) to fill the device
int efield_chunks_f32(int nsrc, int ntrg) {
  return field_chunks(nsrc, (ntrg + 2 * kNbTile - 1) / (2 * kNbTile), kNbTile);
}

__global__ void __launch_bounds__(kNbTile) k_efield(int nsrc, const double* __restrict__ q,
                                                    const double* __restrict__ csrc, int ntrg,
                                                    const double* __restrict__ ctrg, int chunk,
                                                    double* out,
                                                    const int2* __restrict__ trange) {
  __shared__ double4 src[kNbTile];
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.y;
  double px = 0, py = 0, pz = 0;
  if (t < ntrg) {
    px = ctrg[3 * (size_t)t];
    py = ctrg[3 * (size_t)t + 1];
    pz = ctrg[3 * (size_t)t + 2];
  }
  double ex = 0.0, ey = 0.0, ez = 0.0;
  const SrcRange rg = field_src_range(trange, t, ntrg, nsrc, chunk);
  for (int j0 = rg.ulo; j0 < rg.uhi; j0 += kNbTile) {
    int j = j0 + threadIdx.x;
    __syncthreads();
    src[threadIdx.x] = j < rg.uhi ? make_double4(csrc[3 * (size_t)j], csrc[3 * (size_t)j + 1],
                                                 csrc[3 * (size_t)j + 2], q[j])
                                  : make_double4(0, 0, 0, 0);
    __syncthreads();
    const int cnt = min(kNbTile, rg.uhi - j0);
    const int kb = max(rg.lo - j0, 0), ke = min(rg.hi - j0, cnt);
#pragma unroll 4
    for (int k = kb; k < ke; ++k) {
      double4 s = src[k];
      double dx = px - s.x, dy = py - s.y, dz = pz - s.z;
      double r2 = dx * dx + dy * dy + dz * dz;
      double ri = rsqrt_pos(r2);
      double f = s.w * (ri * ri * ri);
      ex = fma(f, dx, ex);
      ey = fma(f, dy, ey);
      ez = fma(f, dz, ez);
    }
  }
  if (t < ntrg) {
    double* o = out + ((size_t)c * ntrg + t) * 3;
    o[0] = ex;
    o[1] = ey;
    o[2] = ez;
  }
}
// the chunks' partial sums of n values, in chunk order
__global__ void k_efield_reduce(long long n, int nchunk, const double* __restrict__ scratch,
                                double* ef) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  double s = 0.0;
  for (int c = 0; c < nchunk; ++c) s += scratch[(size_t)c * n + e];
  ef[e] = s;
}
// FP32-pair variant (mixed precision, force terms only): coordinates are
// taken relative to the block's first target in FP64 and rounded once to
// FP32; each 256-source tile is summed in FP32 and added to FP64
// accumulators.  Same chunked partial-sum layout as k_efield.
__global__ void __launch_bounds__(kNbTile) k_efield_f(int nsrc, const double* __restrict__ q,
                                                      const double* __restrict__ csrc, int ntrg,
                                                      const double* __restrict__ ctrg, int chunk,
                                                      double* out,
                                                      const int2* __restrict__ trange) {
  __shared__ float4 src[kNbTile];
  __shared__ double org[3];
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.y;
  if (threadIdx.x == 0) {
    int t0 = blockIdx.x * blockDim.x;
    org[0] = ctrg[3 * (size_t)t0];
    org[1] = ctrg[3 * (size_t)t0 + 1];
    org[2] = ctrg[3 * (size_t)t0 + 2];
  }
  __syncthreads();
  const double ox = org[0], oy = org[1], oz = org[2];
  float px = 0.f, py = 0.f, pz = 0.f;
  if (t < ntrg) {
    px = (float)(ctrg[3 * (size_t)t] - ox);
    py = (float)(ctrg[3 * (size_t)t + 1] - oy);
    pz = (float)(ctrg[3 * (size_t)t + 2] - oz);
  }
  double ex = 0.0, ey = 0.0, ez = 0.0;
  const SrcRange rg = field_src_range(trange, t, ntrg, nsrc, chunk);
  for (int j0 = rg.ulo; j0 < rg.uhi; j0 += kNbTile) {
    int j = j0 + threadIdx.x;
    __syncthreads();
    src[threadIdx.x] = j < rg.uhi ? make_float4((float)(csrc[3 * (size_t)j] - ox),
                                                (float)(csrc[3 * (size_t)j + 1] - oy),
                                                (float)(csrc[3 * (size_t)j + 2] - oz),
                                                (float)q[j])
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    const int cnt = min(kNbTile, rg.uhi - j0);
    const int kb = max(rg.lo - j0, 0), ke = min(rg.hi - j0, cnt);
    float fx = 0.f, fy = 0.f, fz = 0.f;
#pragma unroll 8
    for (int k = kb; k < ke; ++k) {
      float4 s = src[k];
      float dx = px - s.x, dy = py - s.y, dz = pz - s.z;
      float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      float ri = rsqrtf(r2);
      float f = s.w * (ri * ri * ri);
      fx = fmaf(f, dx, fx);
      fy = fmaf(f, dy, fy);
      fz = fmaf(f, dz, fz);
    }
    ex += fx;
    ey += fy;
    ez += fz;
  }
  if (t < ntrg) {
    double* o = out + ((size_t)c * ntrg + t) * 3;
    o[0] = ex;
    o[1] = ey;
    o[2] = ez;
  }
}
// One molecule: two targets per thread (targets t and t + kNbTile of a
// 2*kNbTile block), so each broadcast source read serves both.  Same
// arithmetic per pair and the same summation order per target as k_efield_f.
__global__ void __launch_bounds__(kNbTile) k_efield_f2(int nsrc, const double* __restrict__ q,
                                                       const double* __restrict__ csrc, int ntrg,
                                                       const double* __restrict__ ctrg,
                                                       int chunk, double* out) {
  __shared__ float4 src[kNbTile];
  const int tb0 = blockIdx.x * 2 * kNbTile;
  const int c = blockIdx.y;
  const double ox = ctrg[3 * (size_t)tb0], oy = ctrg[3 * (size_t)tb0 + 1],
               oz = ctrg[3 * (size_t)tb0 + 2];
  float p[2][3];
  int tt[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int t = tb0 + h * kNbTile + threadIdx.x;
    tt[h] = t;
    p[h][0] = p[h][1] = p[h][2] = 0.f;
    if (t < ntrg) {
      p[h][0] = (float)(ctrg[3 * (size_t)t] - ox);
      p[h][1] = (float)(ctrg[3 * (size_t)t + 1] - oy);
      p[h][2] = (float)(ctrg[3 * (size_t)t + 2] - oz);
    }
  }
  double e[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
  const int s0 = c * chunk, s1 = min(nsrc, c * chunk + chunk);
  for (int j0 = s0; j0 < s1; j0 += kNbTile) {
    const int j = j0 + threadIdx.x;
    __syncthreads();
    src[threadIdx.x] = j < s1 ? make_float4((float)(csrc[3 * (size_t)j] - ox),
                                            (float)(csrc[3 * (size_t)j + 1] - oy),
                                            (float)(csrc[3 * (size_t)j + 2] - oz), (float)q[j])
                              : make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    const int cnt = min(kNbTile, s1 - j0);
    float f[2][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
#pragma unroll 4
    for (int k = 0; k < cnt; ++k) {
      const float4 sv = src[k];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float dx = p[h][0] - sv.x, dy = p[h][1] - sv.y, dz = p[h][2] - sv.z;
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        const float ri = rsqrtf(r2);
        const float w = sv.w * (ri * ri * ri);
        f[h][0] = fmaf(w, dx, f[h][0]);
        f[h][1] = fmaf(w, dy, f[h][1]);
        f[h][2] = fmaf(w, dz, f[h][2]);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      e[h][0] += f[h][0];
      e[h][1] += f[h][1];
      e[h][2] += f[h][2];
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (tt[h] < ntrg) {
      double* o = out + ((size_t)c * ntrg + tt[h]) * 3;
      o[0] = e[h][0];
      o[1] = e[h][1];
      o[2] = e[h][2];
    }
}

cudaError_t launch_efield_f32(Launch L, int nsrc, const double* q, const double* csrc, int ntrg,
                              const double* ctrg, double* ef, double* scratch, int nchunk,
                              const int2* trange) {
  if (ntrg == 0) return cudaSuccess;
  int chunk = (nsrc + nchunk - 1) / max(nchunk, 1);
  chunk = max((chunk + kNbTile - 1) / kNbTile, 1) * kNbTile;
  if (!trange)  // rounding up may leave chunks without sources
    nchunk = max(1, (nsrc + chunk - 1) / chunk);
  double* out = nchunk == 1 ? ef : scratch;
  const int tiles2 = (ntrg + 2 * kNbTile - 1) / (2 * kNbTile);
  if (!trange && (long long)tiles2 * nchunk >= 148 * 8) {  // enough blocks to fill the GPU
    dim3 grid2(tiles2, nchunk);
    k_efield_f2<<<grid2, kNbTile, 0, L.st>>>(nsrc, q, csrc, ntrg, ctrg, chunk, out);
  } else {
    dim3 grid((ntrg + kNbTile - 1) / kNbTile, nchunk);
    k_efield_f<<<grid, kNbTile, 0, L.st>>>(nsrc, q, csrc, ntrg, ctrg, chunk, out, trange);
  }
  ++*L.launches;
  cudaError_t e = cudaGetLastError();
  if (e || nchunk == 1) return e;
  k_efield_reduce<<<(unsigned)((3LL * ntrg + 255) / 256), 256, 0, L.st>>>(3LL * ntrg, nchunk, scratch, ef);
  ++*L.launches;
  return cudaGetLastError();
}

cudaError_t launch_efield(Launch L, int nsrc, const double* q, const double* csrc, int ntrg,
                          const double* ctrg, double* ef, double* scratch, int nchunk,
                          const int2* trange) {
  if (ntrg == 0) return cudaSuccess;
  int chunk = (nsrc + nchunk - 1) / max(nchunk, 1);
  chunk = max((chunk + kFieldChunk - 1) / kFieldChunk, 1) * kFieldChunk;
  if (!trange)  // rounding up may leave chunks without sources
    nchunk = max(1, (nsrc + chunk - 1) / chunk);
  dim3 grid((ntrg + kNbTile - 1) / kNbTile, nchunk);
  double* out = nchunk == 1 ? ef : scratch;
  k_efield<<<grid, kNbTile, 0, L.st>>>(nsrc, q, csrc, ntrg, ctrg, chunk, out, trange);
  ++*L.launches;
  cudaError_t e = cudaGetLastError();
  if (e || nchunk == 1) return e;
  k_efield_reduce<<<(unsigned)((3LL * ntrg + 255) / 256), 256, 0, L.st>>>(3LL * ntrg, nchunk, scratch, ef);
  ++*L.launches;
  return cudaGetLastError();
}
cudaError_t launch_coulomb_pot(Launch L, int nsrc, const double* q, const double* sx,
                               const double* sy, const double* sz, int ntrg, const double* ctrg,
                               double* phi, double* scratch, int nchunk, const int2* trange) {
  if (ntrg == 0) return cudaSuccess;
  int chunk = (nsrc + nchunk - 1) / max(nchunk, 1);
  chunk = max((chunk + kFieldChunk - 1) / kFieldChunk, 1) * kFieldChunk;
  if (!trange) nchunk = max(1, (nsrc + chunk - 1) / chunk);
  double* out = nchunk == 1 ? phi : scratch;
  k_coulomb_pot<<<dim3((ntrg + kNbTile - 1) / kNbTile, nchunk), kNbTile, 0, L.st>>>(
      nsrc, q, sx, sy, sz, ntrg, ctrg, chunk, out, trange);
  ++*L.launches;
  cudaError_t e = cudaGetLastError();
  if (e || nchunk == 1) return e;
  k_efield_reduce<<<(ntrg + 255) / 256, 256, 0, L.st>>>(ntrg, nchunk, scratch, phi);
  ++*L.launches;
  return cudaGetLastError();
}
// Loads the FP64 field kernels' code onto the current device now, rather than
// at their first launch (CUDA loads modules lazily by default).
cudaError_t preload_efield() {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, k_efield);
  if (e != cudaSuccess) return e;
  return cudaFuncGetAttributes(&a, k_efield_reduce);
}

// ---------------------------------------------------------------------------
// forces (fdoka ddcosmo.f90:1436-1504, fdokb :1511-1607, fdoga :1614-1650)
// ---------------------------------------------------------------------------
// alp = sum_{l>=1} t^{l-1}/facl_l sum_m sig_lm (l Y_lm s + dY_lm) and
// beta = sum_l t^l/facl_l sum_m sig_lm Y_lm, with Y and its surface gradient
// as dbasis (ddcosmo.f90:904-1043) computes them, pole branches included.
template <int LMAX>
__device__ void dbasis_contract(const YlmTables& tb, double sx, double sy, double sz, double t,
                                const double* __restrict__ sig, double alp[3], double& beta) {
  constexpr int NY = (LMAX + 1) * (LMAX + 1);
  double vplm[NY];
  double vc[LMAX + 2], vs[LMAX + 2];
  double cthe = sz;
  double sthe = sqrt(fmax(0.0, 1.0 - cthe * cthe));
  double cphi, sphi, et[3], ep[3];
  const bool pole = !(sthe != 0.0);
  if (!pole) {
    cphi = sx / sthe;
    sphi = sy / sthe;
  } else {
    cphi = 1.0;
    sphi = 0.0;
  }
  et[0] = cthe * cphi;
  et[1] = cthe * sphi;
  et[2] = -sthe;
  if (!pole) {
    ep[0] = -sphi / sthe;
    ep[1] = cphi / sthe;
  } else {
    ep[0] = 0.0;
    ep[1] = 1.0;
  }
  ep[2] = 0.0;
  vc[0] = 1.0; vs[0] = 0.0;
  if (!pole) {
    vc[1] = cphi; vs[1] = sphi;
    for (int m = 2; m <= LMAX; ++m) {
      vc[m] = 2.0 * cphi * vc[m - 1] - vc[m - 2];
      vs[m] = 2.0 * cphi * vs[m - 1] - vs[m - 2];
    }
  } else {
    for (int m = 1; m <= LMAX; ++m) { vc[m] = 1.0; vs[m] = 0.0; }
  }
  const double VC = 0.0, VS = (double)(int)cthe;  // integer VC/VS (ddcosmo.f90:912)
  {  // polleg
    double fact = 1.0, pmm = 1.0;
    for (int m = 0; m <= LMAX; ++m) {
      int ind = (m + 1) * (m + 1) - 1;
      vplm[ind] = pmm;
      if (m == LMAX) break;
      double pmm1 = cthe * (2.0 * m + 1.0) * pmm;
      vplm[ind + 2 * m + 2] = pmm1;
      double pmmo = pmm;
      for (int l = m + 2; l <= LMAX; ++l) {
        double pll = tb.A[lmi(l, m)] * cthe * pmm1 - tb.B[lmi(l, m)] * pmm;
        vplm[l * l + l + m] = pll;
        pmm = pmm1;
        pmm1 = pll;
      }
      pmm = -pmmo * fact * sthe;
      fact += 2.0;
    }
  }
  alp[0] = alp[1] = alp[2] = 0.0;
  beta = 0.0;
  double tl = 1.0;  // t^l
  for (int l = 0; l <= LMAX; ++l) {
    const int ind = l * l + l;
    const double fl = (double)l;
    double bl = 0.0, a0 = 0.0, a1 = 0.0, a2 = 0.0;
    {
      double fln = tb.facs[lmi(l, 0)];
      double Y = fln * vplm[ind];
      double sg = sig[ind];
      bl += Y * sg;
      if (l > 0) {
        double d = fln * vplm[ind + 1];
        a0 += sg * (fl * Y * sx + d * et[0]);
        a1 += sg * (fl * Y * sy + d * et[1]);
        a2 += sg * (fl * Y * sz + d * et[2]);
      }
    }
    for (int m = 1; m <= l; ++m) {
      double fln = tb.facs[lmi(l, m)];
      double plm = fln * vplm[ind + m];
      double pp1 = (m < l) ? -0.5 * vplm[ind + m + 1] : 0.0;
      double pm1 = 0.5 * ((double)(l + m) * (double)(l - m + 1) * vplm[ind + m - 1]);
      double pp = pp1 + pm1;
      double Yc = plm * vc[m], Ys = plm * vs[m];
      double dc[3], ds[3];
      for (int k = 0; k < 3; ++k) {
        if (!pole) {
          dc[k] = -fln * pp * vc[m] * et[k] - (double)m * plm * vs[m] * ep[k];
          ds[k] = -fln * pp * vs[m] * et[k] + (double)m * plm * vc[m] * ep[k];
        } else {
          dc[k] = -fln * pp * vc[m] * et[k] - fln * pp * ep[k] * VC;
          ds[k] = -fln * pp * vs[m] * et[k] - fln * pp * ep[k] * VS;
        }
      }
      double sc = sig[ind + m], ss = sig[ind - m];
      bl += Yc * sc + Ys * ss;
      a0 += sc * (fl * Yc * sx + dc[0]) + ss * (fl * Ys * sx + ds[0]);
      a1 += sc * (fl * Yc * sy + dc[1]) + ss * (fl * Ys * sy + ds[1]);
      a2 += sc * (fl * Yc * sz + dc[2]) + ss * (fl * Ys * sz + ds[2]);
    }
    const double ifl = 1.0 / tb.facl[l];
    if (l >= 1) {
      double f = (tl / t) * ifl;  // t^{l-1}/facl_l
      if (t == 0.0) f = (l == 1) ? ifl : 0.0;
      alp[0] += f * a0;
      alp[1] += f * a1;
      alp[2] += f * a2;
    }
    beta += tl * ifl * bl;
    tl *= t;
  }
}

// The same alp and beta from the normalised recurrence (YlmTables::Bn).  With
// u = v / r_i (|u| = t, u / |u| = s) and the real solid harmonics
// R_lm(u) = t^l Y_lm(s), the contraction above is
//   beta  = sum_lm w_lm R_lm(u),   alp_k = sum_lm w_lm d_k R_lm(u),
// w = sigma / facl, and d_k R_lm is a harmonic polynomial of degree l - 1,
// so alp_k = sum_{l'm'} G^k_{l'm'} R_{l'm'}(u) with l' = l - 1.  G follows
// from the ladder relations of the complex solid harmonics without the
// Condon-Shortley phase, S_l^m = |u|^l Pt_l^m(cos theta) e^{i m phi}:
//   d_z S_l^m = (l+m) S_{l-1}^m,   (d_x + i d_y) S_l^m = -S_{l-1}^{m+1},
//   (d_x - i d_y) S_l^m = (l+m)(l+m-1) S_{l-1}^{m-1}   (m >= 1),
//   (d_x - i d_y) S_l^0 = -conj(S_{l-1}^1),
// with R_{l,+m} = nu_lm Re S_l^m, R_{l,-m} = nu_lm Im S_l^m, nu_lm = |facs_lm|.
// k_force_vec writes per sphere the four vectors (beta, G^x, G^y, G^z) in
// the (l, m >= 0) pair layout, scaled by Kg facl so that they contract the
// normalised recurrence values Q_l^m (prefix 1) times cos / sin m phi.
template <int LMAX>
__global__ void k_force_vec(const YlmTables tb, int nsph, const double* __restrict__ sigma,
                            double2* __restrict__ fv) {
  constexpr int NLM = (LMAX + 1) * (LMAX + 2) / 2;
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)nsph * NLM) return;
  const int i = (int)(e / NLM), le = (int)(e - (long long)i * NLM);
  int lp = 0;
  while (lmi(lp + 1, 0) <= le) ++lp;
  const int m = le - lmi(lp, 0);
  const double* sg = sigma + (size_t)i * tb.nylm;
  auto nu = [&](int l, int mm) { return fabs(tb.facs[lmi(l, mm)]); };
  auto wc = [&](int l, int mm) { return sg[l * l + l + mm] / tb.facl[l]; };
  auto ws = [&](int l, int mm) { return sg[l * l + l - mm] / tb.facl[l]; };
  double2* out = fv + 4 * (size_t)e;
  out[0] = make_double2(tb.Kg[le] * sg[lp * lp + lp + m], m ? tb.Kg[le] * sg[lp * lp + lp - m] : 0.0);
  double gxc = 0.0, gxs = 0.0, gyc = 0.0, gys = 0.0, gzc = 0.0, gzs = 0.0;
  if (lp < LMAX) {
    const int l = lp + 1;
    gzc = (double)(l + m) * nu(l, m) * wc(l, m);
    if (m >= 1) gzs = (double)(l + m) * nu(l, m) * ws(l, m);
    if (m + 1 <= l) {  // lowering from m + 1
      const double f = 0.5 * nu(l, m + 1) * ((double)(l + m + 1) * (double)(l + m));
      gxc += f * wc(l, m + 1);
      gyc += f * ws(l, m + 1);
      if (m >= 1) {
        gxs += f * ws(l, m + 1);
        gys -= f * wc(l, m + 1);
      }
    }
    if (m >= 2) {  // raising from m - 1
      const double f = 0.5 * nu(l, m - 1);
      gxc -= f * wc(l, m - 1);
      gyc += f * ws(l, m - 1);
      gxs -= f * ws(l, m - 1);
      gys -= f * wc(l, m - 1);
    } else if (m == 1) {  // raising from m = 0
      gxc -= nu(l, 0) * wc(l, 0);
      gys -= nu(l, 0) * wc(l, 0);
    }
    const double sc = tb.Kg[le] * tb.facl[lp] / nu(lp, m);
    gxc *= sc; gxs *= sc; gyc *= sc; gys *= sc; gzc *= sc; gzs *= sc;
  }
  out[1] = make_double2(gxc, gxs);
  out[2] = make_double2(gyc, gys);
  out[3] = make_double2(gzc, gzs);
}
cudaError_t launch_force_vec(Launch L, const YlmTables& tb, int nsph, const double* sigma,
                             double2* fv) {
  const int nlm = (tb.lmax + 1) * (tb.lmax + 2) / 2;
  const long long n = (long long)nsph * nlm;
  if (n == 0) return cudaSuccess;
#define CASE(LV)                                                                              \
  case LV:                                                                                    \
    k_force_vec<LV><<<(unsigned)((n + 127) / 128), 128, 0, L.st>>>(tb, nsph, sigma, fv);       \
    break;
  switch (tb.lmax) {
    DDC_LMAX_CASES(CASE)
    default:
      return cudaErrorInvalidValue;
  }
#undef CASE
  ++*L.launches;
  return cudaGetLastError();
}
// beta and alp of one triple (s off the poles) from the vectors V of its
// sphere: ct = t cos theta, t2 = t^2, st = t sin theta, (cp, sp) = (cos, sin)
// phi.  The column loop is not unrolled (register pressure); (l, m) is warp
// uniform, so the table and shared-memory reads are broadcasts.
template <int LMAX>
__device__ __forceinline__ void force_contract(const YlmTables& tb, double ct, double t2,
                                               double st, double cp, double sp,
                                               const double2* V, double alp[3], double& beta) {
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  double pmm = 1.0, cm = 1.0, sm = 0.0, cmm1 = 1.0, smm1 = 0.0;
#pragma unroll 1
  for (int m = 0; m <= LMAX; ++m) {
    if (m == 1) {
      cm = cp;
      sm = sp;
    } else if (m >= 2) {
      const double cn = 2.0 * cp * cm - cmm1, sn = 2.0 * cp * sm - smm1;
      cmm1 = cm; smm1 = sm; cm = cn; sm = sn;
    }
    double dc[4] = {0.0, 0.0, 0.0, 0.0}, ds[4] = {0.0, 0.0, 0.0, 0.0};
    // value Q of degree l: beta for every l, the gradient vectors below lmax
    auto add = [&](double Q, int l) {
      const double2* v = V + 4 * lmi(l, m);
      const int nv = l < LMAX ? 4 : 1;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < nv) {
          const double2 c = v[k];
          dc[k] = fma(Q, c.x, dc[k]);
          ds[k] = fma(Q, c.y, ds[k]);
        }
    };
    double q0 = pmm, q1 = ct * pmm;
    add(q0, m);
    if (m < LMAX) {
      add(q1, m + 1);
#pragma unroll 2
      for (int l = m + 2; l <= LMAX; ++l) {
        const double Q = fma(ct, q1, -(tb.Bn[lmi(l, m)] * t2) * q0);
        q0 = q1;
        q1 = Q;
        add(Q, l);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[k] = fma(cm, dc[k], fma(sm, ds[k], acc[k]));
    pmm = -pmm * (double)(2 * m + 1) * st;
  }
  beta = acc[0];
  alp[0] = acc[1];
  alp[1] = acc[2];
  alp[2] = acc[3];
}

// Forces, kernel A: block per sphere i over its gather list, i.e. the
// triples (j, n, i) with point n of neighbour j inside i.  fdoka(j)
// (ddcosmo.f90:1436-1504) and fdokb(i) (:1511-1607) both contract
// dbasis(s_n^ji) with sigma_i at such a triple, so alp and beta are computed
// once per triple: the fdokb and fdoga-neighbour terms accumulate into
// fxa(:,i), the fdoka term of sphere j goes to the per-triple slot fda(:,q).
// fdokb's inner loop over k in N_j (:1575-1590) is u_chi(j,n) - chi_ji*beta
// with u_chi = sum_k chi_jk intmlp_k (an extra k_lx pass on sigma).
// alp and beta come from force_contract off the poles and from the
// reference's dbasis restatement at them.
template <int LMAX>
__global__ void __launch_bounds__(128) k_forces_a(const YlmTables tb, const DevGeo g,
                                                  const double* __restrict__ sigma,
                                                  const double2* __restrict__ fv,
                                                  const double* __restrict__ xs,
                                                  const double* __restrict__ uchi,
                                                  const double* __restrict__ phi, double* fxa,
                                                  double* fda) {
  constexpr int NLM = (LMAX + 1) * (LMAX + 2) / 2;
  __shared__ double2 sv[4 * NLM];
  const int i = blockIdx.x;
  for (int k = threadIdx.x; k < 4 * NLM; k += blockDim.x) sv[k] = fv[4 * (size_t)i * NLM + k];
  __syncthreads();
  const int G = g.ngrid, NY = g.nylm;
  const double4 ci = g.sph[i];
  const double eta = tb.eta, tlow = 1.0 - eta;
  double f0 = 0.0, f1 = 0.0, f2 = 0.0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const double* si = sigma + (size_t)i * NY;
  const int q0 = g.ls_ptr[i], nq = g.ls_ptr[i + 1] - q0;
  for (int t = threadIdx.x; t < nq; t += blockDim.x) {
    const int q = q0 + t;
    const int pj = g.ls[q], j = pj / G, n = pj - j * G;
    const double4 cj = g.sph[j];
    const double4 gn = g.grid[n];
    Rel r = rel_exact(cj, gn, ci);
    double sx = r.vx / r.vv, sy = r.vy / r.vv, sz = r.vz / r.vv;
    double alp[3], beta;
    const double sthe = sqrt(fmax(0.0, 1.0 - sz * sz));
    if (sthe != 0.0)
      force_contract<LMAX>(tb, r.t * sz, r.t * r.t, r.t * sthe, sx / sthe, sy / sthe, sv, alp,
                           beta);
    else
      dbasis_contract<LMAX>(tb, sx, sy, sz, r.t, si, alp, beta);
    double xji = fsw_exact(r.t, eta), fj = g.fi[pj];
    double xij = xs[pj];
    double dsw = (r.t > tlow) ? dfsw_exact(r.t, eta) : 0.0;
    // fdoka term of sphere j at its point n (neighbour i): -w xi_j(n) va
    {
      double oij, fb;
      if (fj > 1.0) {
        oij = xji / fj;
        fb = -oij / fj;
      } else {
        oij = xji;
        fb = 0.0;
      }
      double fa = oij / ci.w;
      double va0 = fa * alp[0] + beta * fb * g.zi[3 * (size_t)pj];
      double va1 = fa * alp[1] + beta * fb * g.zi[3 * (size_t)pj + 1];
      double va2 = fa * alp[2] + beta * fb * g.zi[3 * (size_t)pj + 2];
      if (r.t > tlow) {
        double f3 = beta * dsw / ci.w;
        if (fj > 1.0) f3 = f3 / fj;
        va0 += f3 * sx;
        va1 += f3 * sy;
        va2 += f3 * sz;
      }
      double c = -gn.w * xij;
      fda[3 * (size_t)q + 0] = c * va0;
      fda[3 * (size_t)q + 1] = c * va1;
      fda[3 * (size_t)q + 2] = c * va2;
    }
    // fdokb and the neighbour part of fdoga for sphere i
    double oji = fj > 1.0 ? xji / fj : xji;
    double fa = oji / ci.w;
    double vb0 = fa * alp[0] * xij, vb1 = fa * alp[1] * xij, vb2 = fa * alp[2] * xij;
    double vc0 = 0.0, vc1 = 0.0, vc2 = 0.0;
    if (r.t > tlow) {
      double di, fac;
      if (fj > 1.0) {
        di = 1.0 / fj;
        fac = di * xji;
        if (g.ntri_pt[pj] >= 2) {
          double b = uchi[pj] - xji * beta;
          double g1 = di * di * dsw / ci.w;
          double g2 = g1 * xij * b;
          vc0 = g2 * sx;
          vc1 = g2 * sy;
          vc2 = g2 * sz;
        }
      } else {
        di = 1.0;
        fac = 0.0;
      }
      double fb2 = (1.0 - fac) * di * dsw / ci.w;
      vb0 += fb2 * xij * beta * sx;
      vb1 += fb2 * xij * beta * sy;
      vb2 += fb2 * xij * beta * sz;
      if (r.t < 1.0 && g.ui[pj] > 0.0) {
        int cidx = g.cavidx[pj];
        double ph = cidx >= 0 ? phi[cidx] : 0.0;
        double fg = dsw / ci.w * ph * xij;
        vb0 += fg * sx;
        vb1 += fg * sy;
        vb2 += fg * sz;
      }
    }
    f0 += gn.w * (vb0 - vc0);
    f1 += gn.w * (vb1 - vc1);
    f2 += gn.w * (vb2 - vc2);
  }
  __shared__ double sh[3][4];
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    f0 += __shfl_xor_sync(0xffffffffu, f0, o);
    f1 += __shfl_xor_sync(0xffffffffu, f1, o);
    f2 += __shfl_xor_sync(0xffffffffu, f2, o);
  }
  if (lane == 0) {
    sh[0][w] = f0;
    sh[1][w] = f1;
    sh[2][w] = f2;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double s = 0.0;
    for (int ww = 0; ww < nw; ++ww) s += sh[threadIdx.x][ww];
    fxa[3 * (size_t)i + threadIdx.x] = s;
  }
}

// Forces, kernel B: block per sphere j.  Sums the fdoka slots of j (its pair
// lists, found through lsstart), the fdoga point term (0 < U < 1) and the
// kernel-A part, in fixed order, and applies fep (forces_dd.f90:160-161).
__global__ void __launch_bounds__(128) k_forces_b(const DevGeo g, const double* __restrict__ xs,
                                                  const double* __restrict__ phi,
                                                  const double* __restrict__ fxa,
                                                  const double* __restrict__ fda,
                                                  const int* __restrict__ lsstart, double fep,
                                                  double* fx) {
  const int j = blockIdx.x;
  const int G = g.ngrid;
  double f0 = 0.0, f1 = 0.0, f2 = 0.0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int k = g.inl[j] + w; k < g.inl[j + 1]; k += nw) {
    const int base = lsstart[k], cnt = g.pn_ptr[k + 1] - g.pn_ptr[k];
    for (int t = lane; t < cnt; t += 32) {
      const double* d = fda + 3 * (size_t)(base + t);
      f0 += d[0];
      f1 += d[1];
      f2 += d[2];
    }
  }
  for (int n = threadIdx.x; n < G; n += blockDim.x) {
    const size_t p = (size_t)j * G + n;
    double u = g.ui[p];
    if (u > 0.0 && u < 1.0) {
      double ph = phi[g.cavidx[p]];
      double c = g.grid[n].w * ph * xs[p];
      f0 -= c * g.zi[3 * p];
      f1 -= c * g.zi[3 * p + 1];
      f2 -= c * g.zi[3 * p + 2];
    }
  }
  __shared__ double sh[3][4];
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    f0 += __shfl_xor_sync(0xffffffffu, f0, o);
    f1 += __shfl_xor_sync(0xffffffffu, f1, o);
    f2 += __shfl_xor_sync(0xffffffffu, f2, o);
  }
  if (lane == 0) {
    sh[0][w] = f0;
    sh[1][w] = f1;
    sh[2][w] = f2;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double s = fxa[3 * (size_t)j + threadIdx.x];
    for (int ww = 0; ww < nw; ++ww) s += sh[threadIdx.x][ww];
    fx[3 * (size_t)j + threadIdx.x] = fep * s;
  }
}

cudaError_t launch_forces(Launch L, const YlmTables& tb, const DevGeo& g, const double* sigma,
                          const double* s_xi, const double* u_chi, const double* phi,
                          double fep, double* fx, double* fxa, double* fda, double2* fv) {
  if (g.nsph == 0) return cudaSuccess;
  cudaError_t e0 = launch_force_vec(L, tb, g.nsph, sigma, fv);
  if (e0) return e0;
#define CASE(LV)                                                                               \
  case LV:                                                                                     \
    k_forces_a<LV><<<g.nsph, 128, 0, L.st>>>(tb, g, sigma, fv, s_xi, u_chi, phi, fxa, fda);    \
    break;
  switch (tb.lmax) {
    DDC_LMAX_CASES(CASE)
    default:
      return cudaErrorInvalidValue;
  }
#undef CASE
  ++*L.launches;
  cudaError_t e = cudaGetLastError();
  if (e) return e;
  k_forces_b<<<g.nsph, 128, 0, L.st>>>(g, s_xi, phi, fxa, fda, g.lsstart, fep, fx);
  ++*L.launches;
  return cudaGetLastError();
}

// ddmkxi / ddmkzeta (ddcosmo.f90:1758-1806): scale * w_n U_i(n) xi_i(n) at
// the cavity points, xi_grid = basis^T S on the full grid.
__global__ void k_mkxi(int ncav, int G, const int* __restrict__ cavpt,
                       const double4* __restrict__ grid, const double* __restrict__ ui,
                       const double* __restrict__ xig, double scale, double* out) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncav) return;
  int p = cavpt[c];
  int n = p % G;
  out[c] = scale * (grid[n].w * ui[p] * xig[p]);
}
cudaError_t launch_mkxi(Launch L, const YlmTables& tb, const DevGeo& g, const double* xi_grid,
                        double scale, double* out) {
  if (g.ncav == 0) return cudaSuccess;
  k_mkxi<<<(g.ncav + 255) / 256, 256, 0, L.st>>>(g.ncav, g.ngrid, g.cavpt, g.grid, g.ui, xi_grid,
                                                  scale, out);
  ++*L.launches;
  return cudaGetLastError();
}

// fx(:,i) -= sum_{cavity points of i} zeta * ef  (main.f90:245-253): warp per
// sphere, the lanes' sums by a fixed shuffle tree (a thread per sphere walked
// its points alone: 26 us at 12 spheres, 176 us at 5,000)
__global__ void __launch_bounds__(128) k_zeta_contract(int nsph, const int* __restrict__ cavoff,
                                                       const double* __restrict__ zeta,
                                                       const double* __restrict__ ef,
                                                       double* fx) {
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= nsph) return;
  double a[3] = {0.0, 0.0, 0.0};
  for (int c = cavoff[i] + lane; c < cavoff[i + 1]; c += 32) {
    const double z = zeta[c];
#pragma unroll
    for (int k = 0; k < 3; ++k) a[k] = fma(z, ef[3 * (size_t)c + k], a[k]);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
  }
  if (lane < 3) fx[3 * (size_t)i + lane] -= lane == 0 ? a[0] : lane == 1 ? a[1] : a[2];
}
cudaError_t launch_zeta_efld_contract(Launch L, const DevGeo& g, const double* zeta,
                                      const double* ef, double* fx) {
  if (g.nsph == 0) return cudaSuccess;
  k_zeta_contract<<<(g.nsph + 3) / 4, 128, 0, L.st>>>(g.nsph, g.cavoff, zeta, ef, fx);
  ++*L.launches;
  return cudaGetLastError();
}
// fx(:,i) -= ef(:,i) * q_i  (main.f90:263-265)
__global__ void k_charge_contract(int n, const double* __restrict__ q,
                                  const double* __restrict__ ef, double* fx) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 3 * n) return;
  fx[e] -= ef[e] * q[e / 3];
}
cudaError_t launch_charge_efld_contract(Launch L, int n, const double* q, const double* ef,
                                        double* fx) {
  if (n == 0) return cudaSuccess;
  k_charge_contract<<<(3 * n + 255) / 256, 256, 0, L.st>>>(n, q, ef, fx);
  ++*L.launches;
  return cudaGetLastError();
}
// csph(3,n) and SoA copies of the centres from the packed spheres
__global__ void k_csph_pack(int n, const double4* __restrict__ sph, double* csph, double* sx,
                            double* sy, double* sz) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4 s = sph[i];
  csph[3 * i] = s.x;
  csph[3 * i + 1] = s.y;
  csph[3 * i + 2] = s.z;
  sx[i] = s.x;
  sy[i] = s.y;
  sz[i] = s.z;
}
cudaError_t launch_csph_pack(Launch L, int n, const double4* sph, double* csph, double* sx,
                             double* sy, double* sz) {
  if (n == 0) return cudaSuccess;
  k_csph_pack<<<(n + 255) / 256, 256, 0, L.st>>>(n, sph, csph, sx, sy, sz);
  ++*L.launches;
  return cudaGetLastError();
}

// Roles of the local expansions (k_far_acc): the columns m shared out over the
// warps of a block, greedily by cost or in pairs m / L - m
__host__ __device__ constexpr int lxs_cost(int L, int m) {
  return m == 0 ? 5 * (L + 1) + 4 : 7 * (L + 1 - m) + 4;
}
__host__ __device__ constexpr int lxs_role_of(int L, int NR, int m, bool greedy) {
  if (!greedy) return m <= L - m ? m : L - m;
  int load[DDC_MAX_LMAX + 1] = {};
  int role[DDC_MAX_LMAX + 1] = {};
  bool done[DDC_MAX_LMAX + 1] = {};
  for (int k = 0; k <= L; ++k) {
    int best = -1;
    for (int c = 0; c <= L; ++c)
      if (!done[c] && (best < 0 || lxs_cost(L, c) > lxs_cost(L, best))) best = c;
    int r = 0;
    for (int s = 1; s < NR; ++s)
      if (load[s] < load[r]) r = s;
    done[best] = true;
    load[r] += lxs_cost(L, best);
    role[best] = r;
  }
  return role[m];
}
// offset of column m in its role's register arrays
__host__ __device__ constexpr int lxs_off_of(int L, int NR, int m, bool g) {
  int off = 0;
  for (int c = 0; c < m; ++c)
    if (lxs_role_of(L, NR, c, g) == lxs_role_of(L, NR, m, g)) off += ls_nvals_m(L, c);
  return off;
}
__host__ __device__ constexpr int lxs_role_nvals(int L, int NR, int r, bool g) {
  int n = 0;
  for (int c = 0; c <= L; ++c)
    if (lxs_role_of(L, NR, c, g) == r) n += ls_nvals_m(L, c);
  return n;
}
__host__ __device__ constexpr int lxs_max_nvals(int L, int NR, bool g) {
  int mx = 0;
  for (int r = 0; r < NR; ++r)
    mx = lxs_role_nvals(L, NR, r, g) > mx ? lxs_role_nvals(L, NR, r, g) : mx;
  return mx;
}
// the rows of role R: lane sums by a fixed shuffle tree, then its columns
// G: the greedy column map (else the pairing)
template <int LMAX, int NR, int R, int M, bool G>
__device__ __forceinline__ void lxs_store_cols(const YlmTables& tb, const double* acc, double* yi,
                                               int lane) {
  if constexpr (lxs_role_of(LMAX, NR, M, G) == R)
    ls_store<LMAX, M, lxs_off_of(LMAX, NR, M, G)>(tb, acc, yi, lane);
  if constexpr (M < LMAX) lxs_store_cols<LMAX, NR, R, M + 1, G>(tb, acc, yi, lane);
}
template <int LMAX, int NR, int R, bool G>
__device__ __forceinline__ void lxs_finish_role(int role, const YlmTables& tb, double* acc,
                                                double* yi, int lane) {
  if (role == R) {
    constexpr int NV = lxs_role_nvals(LMAX, NR, R, G);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], o);
    }
    lxs_store_cols<LMAX, NR, R, 0, G>(tb, acc, yi, lane);
    return;
  }
  if constexpr (R + 1 < NR)
    lxs_finish_role<LMAX, NR, R + 1, G>(role, tb, acc, yi, lane);
}

// ---------------------------------------------------------------------------
// point lists: for every (a, n) the positions, in the neighbours' gather
// lists, of the triples (a, n, b), in a's CSR order.  Sphere a's entries take
// the range of its pair lists; pt_ptr counts through it point by point.
// Warp per sphere: prefix sums of the points' triple counts, then the pairs
// one after the other (a pair's points are distinct).
// ---------------------------------------------------------------------------
constexpr int kPtWarps = 4;
constexpr int kMaxGrid = 5810;  // points of the largest Lebedev grid
__global__ void __launch_bounds__(32 * kPtWarps)
    k_pt_fill(int nsph, int ngrid, const int* __restrict__ inl, const int* __restrict__ pn_ptr,
              const uint16_t* __restrict__ pn, const int* __restrict__ lsstart,
              const uint8_t* __restrict__ ntri, int* pt_ptr, int* pt_idx) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a = blockIdx.x * kPtWarps + w;
  if (a >= nsph) return;  // warp-uniform; no block barriers
  int* cur = reinterpret_cast<int*>(smraw) + (size_t)w * ngrid;
  const size_t p0 = (size_t)a * ngrid;
  int run = pn_ptr[inl[a]];
  for (int n0 = 0; n0 < ngrid; n0 += 32) {
    const int n = n0 + lane, c = n < ngrid ? ntri[p0 + n] : 0;
    int v = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += t;
    }
    if (n < ngrid) {
      cur[n] = run + v - c;
      pt_ptr[p0 + n] = run + v - c;
    }
    run += __shfl_sync(0xffffffffu, v, 31);
  }
  if (a == nsph - 1 && lane == 0) pt_ptr[p0 + ngrid] = run;
  __syncwarp();
  for (int k = inl[a]; k < inl[a + 1]; ++k) {
    const int q0 = pn_ptr[k], cnt = pn_ptr[k + 1] - q0, base = lsstart[k];
    for (int t = lane; t < cnt; t += 32) {
      const int n = pn[q0 + t], at = cur[n];
      cur[n] = at + 1;
      pt_idx[at] = base + t;
    }
    __syncwarp();
  }
}
cudaError_t launch_pt_fill(Launch L, int nsph, int ngrid, const int* inl, const int* pn_ptr,
                           const uint16_t* pn, const int* lsstart, const uint8_t* ntri,
                           int* pt_ptr, int* pt_idx) {
  if (nsph == 0) return cudaSuccess;
  const size_t sm = sizeof(int) * kPtWarps * ngrid;
  if (sm > 48 * 1024) {
    // the limit belongs to the function: the same value whatever the grid, so
    // that another thread's context cannot lower it before the launch
    const cudaError_t e = cudaFuncSetAttribute(
        k_pt_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(int) * kPtWarps * kMaxGrid);
    if (e) return e;
  }
  k_pt_fill<<<(nsph + kPtWarps - 1) / kPtWarps, 32 * kPtWarps, sm, L.st>>>(
      nsph, ngrid, inl, pn_ptr, pn, lsstart, ntri, pt_ptr, pt_idx);
  ++*L.launches;
  return cudaGetLastError();
}

// pot_a(n) = sum of the lx values of the triples of (a, n), in CSR order.
// Thread per point: a list has 3 entries on average, and consecutive threads
// (neighbouring points: the grid is in patch order) lie inside nearly the
// same neighbours, whose values are adjacent.  chi: the sums times
// max(f_a(n), 1), i.e. with the weight chi(t) of u_chi in place of
// chi(t) / f_a(n).  Fixed order, no atomics.  Bound: latency of the chain
// list bounds -> positions -> values for few points, HBM for many (0.4 GB at
// 20,000 spheres, lmax 10, 590 points).  Two points per thread: one is 123
// us there, two 83 us, four 84 us.  The warp-per-sphere form that this
// replaces walked a sphere's 20 or so pairs one after the other: 113 us there
// (FP64 151, now 102), 37 us at 5,000 spheres and 302 points (now 19), 21 us
// at 600 spheres (now 9).
constexpr int kPtPoints = 2;
template <class Rl>
__global__ void __launch_bounds__(256)
    k_lx_gather(const DevGeo g, const Rl* val, Rl* pot, int ldp, bool chi) {
  chain_wait();
  constexpr int P = kPtPoints;
  constexpr int U = 4;  // triples of a point in flight
  const unsigned np = (unsigned)g.nsph * g.ngrid, G = g.ngrid;
  int q[P], q1[P];
  Rl v[P];
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const unsigned p = step_point(blockIdx.x, P, i, 256, threadIdx.x);
    q[i] = q1[i] = 0;
    v[i] = 0;
    if (p < np && !sweep_skip(g.act, p / G)) {
      q[i] = g.pt_ptr[p];
      q1[i] = g.pt_ptr[p + 1];
    }
  }
  for (bool more = true; more;) {
    int at[P][U];
    Rl x[P][U];
#pragma unroll
    for (int i = 0; i < P; ++i)
#pragma unroll
      for (int u = 0; u < U; ++u) at[i][u] = u < q1[i] - q[i] ? g.pt_idx[q[i] + u] : -1;
#pragma unroll
    for (int i = 0; i < P; ++i)
#pragma unroll
      for (int u = 0; u < U; ++u) x[i][u] = at[i][u] >= 0 ? val[at[i][u]] : Rl(0);
    more = false;
#pragma unroll
    for (int i = 0; i < P; ++i) {
#pragma unroll
      for (int u = 0; u < U; ++u) v[i] += x[i][u];
      q[i] = min(q[i], q1[i] - U) + U;  // at most q1
      more |= q[i] < q1[i];
    }
  }
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const unsigned p = step_point(blockIdx.x, P, i, 256, threadIdx.x);
    if (p >= np) continue;
    const unsigned a = p / G;
    if (sweep_skip(g.act, a)) continue;
    if (chi) v[i] *= (Rl)fmax(g.fi[p], 1.0);
    pot[(size_t)a * ldp + (p - a * G)] = v[i];
  }
}

template <class Rl>
static cudaError_t gather_launch(Launch L, const DevGeo& g, const Rl* val, Rl* pot, int ldp,
                                 bool chi) {
  if (g.nsph == 0) return cudaSuccess;
  const long long np = (long long)g.nsph * g.ngrid;
  ++*L.launches;
  return launch_chained(k_lx_gather<Rl>, dim3((unsigned)((np + 256 * kPtPoints - 1) / (256 * kPtPoints))),
                        256, 0, L.st, g, val, pot, ldp, chi);
}
cudaError_t launch_lx_gather(Launch L, const DevGeo& g, const double* val, double* pot,
                             bool chi) {
  return gather_launch<double>(L, g, val, pot, g.ngrid, chi);
}
cudaError_t launch_lx_gather_f32(Launch L, const DevGeo& g, const float* val, float* pot,
                                 int ldp) {
  return gather_launch<float>(L, g, val, pot, ldp, false);
}

__global__ void k_to_float(long long n, const double* __restrict__ x, float* y) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) y[e] = (float)x[e];
}
cudaError_t launch_to_float(Launch L, long long n, const double* x, float* y) {
  if (n == 0) return cudaSuccess;
  k_to_float<<<(unsigned)((n + 255) / 256), 256, 0, L.st>>>(n, x, y);
  ++*L.launches;
  return cudaGetLastError();
}
// ---------------------------------------------------------------------------
// batches of molecules
// ---------------------------------------------------------------------------
// per-molecule <a, b> (energy: fep * <X, psi>, cosmo.f90:155)
__global__ void k_batch_dot(const int* __restrict__ off, int nylm, const double* __restrict__ a,
                            const double* __restrict__ b, double scale, double* out) {
  const int k = blockIdx.x;
  const long long e0 = (long long)off[k] * nylm, e1 = (long long)off[k + 1] * nylm;
  double acc = 0.0;
  for (long long e = e0 + threadIdx.x; e < e1; e += blockDim.x) acc = fma(a[e], b[e], acc);
  __shared__ double sh[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) sh[w] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int ww = 0; ww < (int)(blockDim.x >> 5); ++ww) t += sh[ww];
    out[k] = scale * t;
  }
}
cudaError_t launch_batch_dot(Launch L, int nmol, const int* off, int nylm, const double* a,
                             const double* b, double scale, double* out) {
  if (nmol == 0) return cudaSuccess;
  k_batch_dot<<<nmol, 256, 0, L.st>>>(off, nylm, a, b, scale, out);
  ++*L.launches;
  return cudaGetLastError();
}

// source ranges of the batched N-body sums: a cavity point sums over the
// nuclei of its molecule, a nucleus over the cavity points of its molecule
__global__ void k_batch_ranges(int nsph, int ngrid, int ncav, const int2* __restrict__ mrange,
                               const int* __restrict__ cavpt, const int* __restrict__ cavoff,
                               int2* tr_cav, int2* tr_nuc) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < ncav) tr_cav[e] = mrange[cavpt[e] / ngrid];
  if (e < nsph) {
    int2 r = mrange[e];
    tr_nuc[e] = make_int2(cavoff[r.x], cavoff[r.y]);
  }
}
cudaError_t launch_batch_ranges(Launch L, int nsph, int ngrid, int ncav, const int2* mrange,
                                const int* cavpt, const int* cavoff, int2* tr_cav,
                                int2* tr_nuc) {
  long long n = max((long long)ncav, (long long)nsph);
  if (n == 0) return cudaSuccess;
  k_batch_ranges<<<(unsigned)((n + 255) / 256), 256, 0, L.st>>>(nsph, ngrid, ncav, mrange, cavpt,
                                                                 cavoff, tr_cav, tr_nuc);
  ++*L.launches;
  return cudaGetLastError();
}

// FP64 peak probe: 8 independent FMA chains per thread, register resident.
template <class T>
__global__ void __launch_bounds__(256) k_fma_probe(int iters, T* out) {
  T a[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = T(1) + T(1e-6) * T(threadIdx.x + k);
  const T b = T(0.999999), c = T(1e-7);
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = fma(a[k], b, c);
  }
  T s = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += a[k];
  if (s == T(12345)) out[0] = s;  // keeps the chains live
}
cudaError_t launch_fp64_probe(Launch L, int blocks, int iters, double* out) {
  k_fma_probe<double><<<blocks, 256, 0, L.st>>>(iters, out);
  ++*L.launches;
  return cudaGetLastError();
}
cudaError_t launch_fp32_probe(Launch L, int blocks, int iters, float* out) {
  k_fma_probe<float><<<blocks, 256, 0, L.st>>>(iters, out);
  ++*L.launches;
  return cudaGetLastError();
}

}  // namespace ddc

namespace ddc {
// ---------------------------------------------------------------------------
// Solute potential and field at the cavity points with a near / far split
// (mkrhs.f90:102-114 and the field of efld.f90:97-114 at the cavity,
// main.f90:241).  Every cavity point lies on its sphere's surface,
// p = c_i + r_i s_n.  A charge q_j farther than rho * r_i from c_i contributes,
// by the addition theorem (|p - c_j| > r_i = |p - c_i|),
//   q_j / |p - c_j| = sum_lm [q_j / d (4 pi / (2l+1)) t^l Y_lm(d^)] Y_lm(s_n),
//   t = r_i / d <= 1 / rho,  d = c_j - c_i,
// so the far charges of sphere i are summed once into its local expansion
//   A_lm(i) = sum_{far j} q_j / d (4 pi / (2l+1)) t^l Y_lm(d^)   (degree P)
// and evaluated at its cavity points: phi_far = sum_lm A_lm Y_lm(s_n) and
// E_far = -(1 / r_i) sum_lm A_lm grad R_lm(s_n), with R_lm(u) = |u|^l Y_lm(u^)
// the regular solid harmonic.  The accumulation of A is the L* machinery
// (the adjrhs sum "weight * 4 pi/(2l+1) t^l Y_lm(s)" over (point, source)
// pairs) with the weight -q_j / d.  The near charges (and the sphere's own)
// are summed directly.  Truncation: at most t^(P+1) / (1 - t) of each far
// term, 1e-10 for P = 10, rho = 8.
// ---------------------------------------------------------------------------
// The adjrhs sum by the normalised recurrence, FP64: Q_l = ct Q_{l-1}
// - Bn t^2 Q_{l-2} (three operations per value; the scale gam_lm sits in Kg,
// applied when the rows are stored), accumulated into the column's register rows
template <int LMAX, int M, int OFF>
__device__ __forceinline__ void fa_column(const YlmTables& tb, double ct, double t2, double q0,
                                          double cm, double sm, double* acc) {
  constexpr int NM = LMAX + 1 - M;
  double q1 = 0.0;
#pragma unroll
  for (int l = M; l <= LMAX; ++l) {
    double Q;
    if (l == M) {
      Q = q0;
    } else if (l == M + 1) {
      q1 = ct * q0;
      Q = q1;
    } else {
      Q = fma(ct, q1, -(tb.Bn[lmi(l, M)] * t2) * q0);
      q0 = q1;
      q1 = Q;
    }
    if (M == 0) {
      acc[OFF + l] += Q;
    } else {
      acc[OFF + (l - M)] = fma(Q, cm, acc[OFF + (l - M)]);
      acc[OFF + NM + (l - M)] = fma(Q, sm, acc[OFF + NM + (l - M)]);
    }
  }
}
// Roles of k_far_acc: at lmax 10 four roles of about three columns each
// (the greedy map: each role's per-source fixed cost paid four times instead
// of six), else the pairing m / lmax-m
__host__ __device__ constexpr bool fa_greedy(int L) { return L == 10; }
__host__ __device__ constexpr int fa_nroles(int L) { return fa_greedy(L) ? 4 : L / 2 + 1; }
template <int LMAX, int R, int M>
__device__ __forceinline__ void fa_cols(const YlmTables& tb, const double* sh, int stride, int q,
                                        double ct, double t2, double* acc) {
  constexpr int NR = fa_nroles(LMAX);
  constexpr bool G = fa_greedy(LMAX);
  if constexpr (lxs_role_of(LMAX, NR, M, G) == R)
    fa_column<LMAX, M, lxs_off_of(LMAX, NR, M, G)>(tb, ct, t2, sh[(2 + 3 * M) * stride + q],
                                                   sh[(3 + 3 * M) * stride + q],
                                                   sh[(4 + 3 * M) * stride + q], acc);
  if constexpr (M < LMAX) fa_cols<LMAX, R, M + 1>(tb, sh, stride, q, ct, t2, acc);
}
template <int LMAX, int R>
__device__ __forceinline__ void fa_role(const YlmTables& tb, const double* sh, int stride,
                                        int count, int lane, double* acc) {
  for (int q = lane; q < count; q += 32) {
    const double ct = sh[q], t2 = sh[stride + q];
    fa_cols<LMAX, R, 0>(tb, sh, stride, q, ct, t2, acc);
  }
}
template <int LMAX, int R>
__device__ __forceinline__ void fa_run_role(int role, const YlmTables& tb, const double* sh,
                                            int stride, int count, int lane, double* acc) {
  if (role == R) {
    fa_role<LMAX, R>(tb, sh, stride, count, lane, acc);
    return;
  }
  if constexpr (R + 1 < fa_nroles(LMAX))
    fa_run_role<LMAX, R + 1>(role, tb, sh, stride, count, lane, acc);
}

// A(i, lm) for every sphere with cavity points: block per sphere, role warps
// over chunks of the sources of its molecule.  Per source the thread forms
// 1/d and 1/sin(theta) with the refined hardware reciprocal square root
// (rsqrt_pos), the prefix and cos/sin(m phi); the
// roles run the normalised recurrence (fa_column) and store with Kg.
template <int LMAX>
__global__ void __launch_bounds__(32 * fa_nroles(LMAX), fa_greedy(LMAX) ? 4 : 1)
    k_far_acc(const YlmTables tb, int nsph,
                                                                   const double4* __restrict__ sph,
                                                                   const double* __restrict__ q,
                                                                   const int2* __restrict__ mrange,
                                                                   const int* __restrict__ cavoff,
                                                                   double rho, double* A) {
  constexpr int NR = fa_nroles(LMAX);
  constexpr int CH = 32 * NR;
  constexpr int NVM = lxs_max_nvals(LMAX, NR, fa_greedy(LMAX));
  extern __shared__ double sh[];  // [ls_nfields][CH]
  const int i = blockIdx.x;
  if (cavoff[i + 1] == cavoff[i]) return;  // buried: A(i) is never read
  const int role = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double4 ci = sph[i];
  const double cut2 = (rho * ci.w) * (rho * ci.w);
  const int lo = mrange ? mrange[i].x : 0, hi = mrange ? mrange[i].y : nsph;
  double acc[NVM];
#pragma unroll
  for (int v = 0; v < NVM; ++v) acc[v] = 0.0;
  for (int j0 = lo; j0 < hi; j0 += CH) {
    const int chunk = min(CH, hi - j0);
    {
      const int tt = threadIdx.x;
      double* col = sh + tt;
      double ct = 0.0, t2 = 0.0, st = 0.0, w = 0.0, cp = 1.0, sp = 0.0;
      if (tt < chunk) {
        const int j = j0 + tt;
        const double4 cj = sph[j];
        const double vx = cj.x - ci.x, vy = cj.y - ci.y, vz = cj.z - ci.z;
        const double d2 = vx * vx + vy * vy + vz * vz;
        if (j != i && d2 > cut2) {
          const double di = rsqrt_pos(d2);
          const double t = ci.w * di, c = vz * di;
          const double s2 = fma(-c, c, 1.0);
          double sn = 0.0;
          if (s2 > 1e-280) {  // off the pole (at a pole only m = 0 survives)
            const double rs = rsqrt_pos(s2);
            sn = s2 * rs;
            cp = vx * di * rs;
            sp = vy * di * rs;
          }
          ct = c * t;
          t2 = t * t;
          st = sn * t;
          w = -q[j] * di;
        }
      }
      col[0] = ct;
      col[CH] = t2;
      double pmm = w, cm = 1.0, sm = 0.0, cmm1 = 1.0, smm1 = 0.0;
#pragma unroll
      for (int m = 0; m <= LMAX; ++m) {
        if (m == 1) {
          cm = cp;
          sm = sp;
        } else if (m >= 2) {
          const double cn = 2.0 * cp * cm - cmm1, sn = 2.0 * cp * sm - smm1;
          cmm1 = cm; smm1 = sm; cm = cn; sm = sn;
        }
        col[(2 + 3 * m) * CH] = pmm;
        col[(3 + 3 * m) * CH] = cm;
        col[(4 + 3 * m) * CH] = sm;
        pmm = -pmm * (2.0 * m + 1.0) * st;
      }
    }
    __syncthreads();
    fa_run_role<LMAX, 0>(role, tb, sh, CH, chunk, lane, acc);
    __syncthreads();
  }
  lxs_finish_role<LMAX, NR, 0, fa_greedy(LMAX)>(role, tb, acc, A + (size_t)i * tb.nylm, lane);
}

// Tables on the grid, once per context: BT[lm][n] = Y_lm(s_n) and
// DT[k][lm][n] = d R_lm / d u_k at u = s_n (k = x, y, z), by fourth-order
// central differences of R_lm(u) = |u|^l Y_lm(u / |u|) with step 1e-4
// (truncation ~h^4 l^5 / 30 and rounding ~1e-16 / h: about 1e-12 relative)
__global__ void k_far_tables(const YlmTables tb, const double4* __restrict__ grid, int ngrid,
                             double* BT, double* DT) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 4 * ngrid) return;
  const int n = e % ngrid, k = e / ngrid;  // k = 0: values; 1..3: d/du_{k-1}
  const double4 g = grid[n];
  const int ny = tb.nylm;
  double y[(DDC_MAX_LMAX + 1) * (DDC_MAX_LMAX + 1)];
  if (k == 0) {
    ylmbas_ref(tb, g.x, g.y, g.z, y);
    for (int lm = 0; lm < ny; ++lm) BT[(size_t)lm * ngrid + n] = y[lm];
    return;
  }
  double acc[(DDC_MAX_LMAX + 1) * (DDC_MAX_LMAX + 1)];
  for (int lm = 0; lm < ny; ++lm) acc[lm] = 0.0;
  const double h = 1e-4;
  const double cst[4] = {1.0, -8.0, 8.0, -1.0};   // f(-2h), f(-h), f(h), f(2h)
  const double off[4] = {-2.0, -1.0, 1.0, 2.0};
  for (int s = 0; s < 4; ++s) {
    double u[3] = {g.x, g.y, g.z};
    u[k - 1] += off[s] * h;
    const double r = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
    ylmbas_ref(tb, u[0] / r, u[1] / r, u[2] / r, y);
    double rl = 1.0;
    for (int l = 0; l <= tb.lmax; ++l) {
      for (int m = -l; m <= l; ++m) acc[l * l + l + m] += cst[s] * rl * y[l * l + l + m];
      rl *= r;
    }
  }
  for (int lm = 0; lm < ny; ++lm)
    DT[((size_t)(k - 1) * ny + lm) * ngrid + n] = acc[lm] / (12.0 * h);
}

// Potential and field at the cavity points of sphere i (block per sphere):
// the near charges directly (compacted into shared memory in passes of at
// most kNearCap), the far ones from A(i).  With ef == nullptr only phi.  A
// sphere without cavity points (buried) has nothing to do; the others run
// with NU = ceil(points / 128) point slots per thread (a sphere has 90
// points on average at the 20k workload, up to 590), so no thread steps
// through empty slots in the pair loop.
constexpr int kNearCap = 1024;
constexpr int kCandGroups = 512;
template <int NU>
__device__ __forceinline__ void far_cav_body(int i, int ngrid, int ny, double4 ci, double cut2,
                                             int lo, int hi, int c0, int c1,
                                             const double4* __restrict__ sph,
                                             const double* __restrict__ q,
                                             const int* __restrict__ cavpt,
                                             const double* __restrict__ ccav,
                                             const double* __restrict__ BT,
                                             const double* __restrict__ DT, double* phi,
                                             double* ef, double4* near, const double* sA,
                                             int& s_cnt, int& s_scan, int* wbase,
                                             const int* cgl, const int* cpre, int ncg,
                                             const int* __restrict__ gsph,
                                             const int* __restrict__ gstart) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  // candidate f of the scan: sphere f of the molecule's range, or with cell
  // groups (ncg > 0) the member f - cpre[k] of candidate group cgl[k]
  auto cand = [&](int f) -> int {
    if (ncg == 0) return f;
    int a = 0, b = ncg;  // cpre[a] <= f < cpre[b]
    while (b - a > 1) {
      const int mid = (a + b) >> 1;
      if (cpre[mid] <= f) a = mid;
      else b = mid;
    }
    return gsph[gstart[cgl[a]] + (f - cpre[a])];
  };
  // thread tid owns cavity points c0 + tid + 128 u, u < NU
  double v[NU], ex[NU], ey[NU], ez[NU], px[NU], py[NU], pz[NU];
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    v[u] = ex[u] = ey[u] = ez[u] = 0.0;
    const int c = c0 + tid + 128 * u;
    px[u] = py[u] = pz[u] = 0.0;
    if (c < c1) {
      px[u] = ccav[3 * (size_t)c];
      py[u] = ccav[3 * (size_t)c + 1];
      pz[u] = ccav[3 * (size_t)c + 2];
    }
  }
  if (tid == 0) s_scan = lo;
  __syncthreads();
  // passes over the molecule: compact near charges, then sum them
  while (true) {
    if (tid == 0) s_cnt = 0;
    __syncthreads();
    const int start = s_scan;
    if (start >= hi) break;
    int j = start;
    // scan in steps of 128 candidates while the buffer has room for a step
    for (; j < hi; j += 128) {
      __syncthreads();
      if (s_cnt + 128 > kNearCap) break;
      const int jj = j + tid;
      bool nb = false;
      double4 cj = make_double4(0, 0, 0, 0);
      int js = 0;
      if (jj < hi) {
        js = cand(jj);
        cj = sph[js];
        const double dx = cj.x - ci.x, dy = cj.y - ci.y, dz = cj.z - ci.z;
        nb = js == i || dx * dx + dy * dy + dz * dz <= cut2;
      }
      const unsigned bal = __ballot_sync(0xffffffffu, nb);
      if (lane == 0) wbase[w] = __popc(bal);
      __syncthreads();
      if (tid == 0) {
        int b = s_cnt;
        for (int k = 0; k < 4; ++k) {
          const int c = wbase[k];
          wbase[k] = b;
          b += c;
        }
        s_cnt = b;
      }
      __syncthreads();
      if (nb) near[wbase[w] + __popc(bal & ((1u << lane) - 1u))] = make_double4(cj.x, cj.y, cj.z, q[js]);
    }
    __syncthreads();
    if (tid == 0) s_scan = j;
    const int cnt = s_cnt;
    for (int k = 0; k < cnt; ++k) {
      const double4 s = near[k];
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        if (c0 + tid + 128 * u < c1) {
          const double dx = px[u] - s.x, dy = py[u] - s.y, dz = pz[u] - s.z;
          const double ri = rsqrt_pos(dx * dx + dy * dy + dz * dz);
          v[u] = fma(s.w, ri, v[u]);
          const double f = s.w * (ri * ri * ri);
          ex[u] = fma(f, dx, ex[u]);
          ey[u] = fma(f, dy, ey[u]);
          ez[u] = fma(f, dz, ez[u]);
        }
      }
    }
    __syncthreads();
  }
  // far part from the local expansion
  const double iri = 1.0 / ci.w;
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    const int c = c0 + tid + 128 * u;
    if (c >= c1) continue;
    const int n = cavpt[c] - i * ngrid;
    double fp = 0.0, fx = 0.0, fy = 0.0, fz = 0.0;
    for (int lm = 0; lm < ny; ++lm) {
      const double a = sA[lm];
      fp = fma(a, BT[(size_t)lm * ngrid + n], fp);
      if (ef) {
        fx = fma(a, DT[(size_t)lm * ngrid + n], fx);
        fy = fma(a, DT[((size_t)ny + lm) * ngrid + n], fy);
        fz = fma(a, DT[((size_t)2 * ny + lm) * ngrid + n], fz);
      }
    }
    phi[c] = v[u] + fp;
    if (ef) {
      ef[3 * (size_t)c] = ex[u] - iri * fx;
      ef[3 * (size_t)c + 1] = ey[u] - iri * fy;
      ef[3 * (size_t)c + 2] = ez[u] - iri * fz;
    }
  }
}

__global__ void __launch_bounds__(128) k_far_cav(int nsph, int ngrid, int ny,
                                                 const double4* __restrict__ sph,
                                                 const double* __restrict__ q,
                                                 const int2* __restrict__ mrange, double rho,
                                                 const int* __restrict__ cavoff,
                                                 const int* __restrict__ cavpt,
                                                 const double* __restrict__ ccav,
                                                 const double* __restrict__ A,
                                                 const double* __restrict__ BT,
                                                 const double* __restrict__ DT, double* phi,
                                                 double* ef, const ZGroups zg) {
  __shared__ double4 near[kNearCap];
  __shared__ double sA[(DDC_MAX_LMAX + 1) * (DDC_MAX_LMAX + 1)];
  __shared__ int s_cnt, s_scan, wbase[4];
  __shared__ int cgl[kCandGroups], cpre[kCandGroups + 1];
  __shared__ int s_ncg;
  const int i = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int c0 = cavoff[i], c1 = cavoff[i + 1];
  if (c1 == c0) return;  // buried: no cavity points
  const double4 ci = sph[i];
  const double cut2 = (rho * ci.w) * (rho * ci.w);
  int lo = mrange ? mrange[i].x : 0, hi = mrange ? mrange[i].y : nsph;
  for (int lm = tid; lm < ny; lm += blockDim.x) sA[lm] = A[(size_t)i * ny + lm];
  // with cell groups (one molecule): the groups that can hold a near charge
  // (|c_i - c_g| <= rho r_i + R_g, R_g bounding the members' centres; 1e-6
  // bohr of margin for rounding), compacted in group order, and the prefix
  // sums of their sizes; more than kCandGroups keeps the full scan
  int ncg = 0;
  if (zg.ngroup > 0) {
    if (tid == 0) s_ncg = 0;
    __syncthreads();
    const double reach = rho * ci.w;
    for (int g0 = 0; g0 < zg.ngroup; g0 += 128) {
      const int g = g0 + tid;
      bool c = false;
      if (g < zg.ngroup) {
        const double4 cg = zg.gcen[g];
        const double dx = ci.x - cg.x, dy = ci.y - cg.y, dz = ci.z - cg.z;
        const double lim = reach + cg.w + 1e-6;
        c = dx * dx + dy * dy + dz * dz <= lim * lim;
      }
      const unsigned bal = __ballot_sync(0xffffffffu, c);
      if (lane == 0) wbase[w] = __popc(bal);
      __syncthreads();
      if (tid == 0) {
        int b = s_ncg;
        for (int k = 0; k < 4; ++k) {
          const int n = wbase[k];
          wbase[k] = b;
          b += n;
        }
        s_ncg = b;
      }
      __syncthreads();
      const int pos = wbase[w] + __popc(bal & ((1u << lane) - 1u));
      if (c && pos < kCandGroups) cgl[pos] = g;
      __syncthreads();
    }
    ncg = s_ncg;
    if (ncg <= kCandGroups) {
      // prefix sums of the candidate groups' sizes (warp 0, in order)
      if (w == 0) {
        int run = 0;
        for (int k0 = 0; k0 < ncg; k0 += 32) {
          const int k = k0 + lane;
          int v = k < ncg ? zg.gstart[cgl[k] + 1] - zg.gstart[cgl[k]] : 0;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += t;
          }
          if (k < ncg) cpre[k + 1] = run + v;
          run += __shfl_sync(0xffffffffu, v, 31);
        }
        if (lane == 0) cpre[0] = 0;
      }
      __syncthreads();
      lo = 0;
      hi = ncg > 0 ? cpre[ncg] : 0;
    } else {
      ncg = 0;  // too many candidates: scan the molecule
    }
  }
  // 5 * 128 = 640 >= ngrid up to 590 points
  switch ((c1 - c0 + 127) / 128) {
#define FAR_CAV_CASE(NU)                                                                        \
  case NU:                                                                                      \
    far_cav_body<NU>(i, ngrid, ny, ci, cut2, lo, hi, c0, c1, sph, q, cavpt, ccav, BT, DT, phi, \
                     ef, near, sA, s_cnt, s_scan, wbase, cgl, cpre, ncg, zg.gsph, zg.gstart);  \
    break;
    FAR_CAV_CASE(1)
    FAR_CAV_CASE(2)
    FAR_CAV_CASE(3)
    FAR_CAV_CASE(4)
    FAR_CAV_CASE(5)
#undef FAR_CAV_CASE
    default:
      break;
  }
}

cudaError_t launch_far_tables(Launch L, const YlmTables& tbP, const double4* grid, int ngrid,
                              double* BT, double* DT) {
  const int n = 4 * ngrid;
  k_far_tables<<<(n + 63) / 64, 64, 0, L.st>>>(tbP, grid, ngrid, BT, DT);
  ++*L.launches;
  return cudaGetLastError();
}

cudaError_t launch_far_pot_field(Launch L, const YlmTables& tbP, int nsph, int ngrid,
                                 const double4* sph, const double* q, const int2* mrange,
                                 double rho, const int* cavoff, const int* cavpt,
                                 const double* ccav, const double* BT, const double* DT,
                                 double* A, double* phi, double* ef, const ZGroups* zg) {
  if (nsph == 0) return cudaSuccess;
  if (ngrid > 640) return cudaErrorInvalidValue;  // k_far_cav holds 5 x 128 points per thread set
  cudaError_t e;
#define CASE(LV)                                                                              \
  case LV: {                                                                                  \
    constexpr int NR = fa_nroles(LV);                                                         \
    const size_t sm = sizeof(double) * ls_nfields(LV) * 32 * NR;                              \
    if (sm > 48 * 1024)                                                                       \
      if ((e = cudaFuncSetAttribute(k_far_acc<LV>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                    (int)sm)))                                                \
        return e;                                                                             \
    k_far_acc<LV><<<nsph, 32 * NR, sm, L.st>>>(tbP, nsph, sph, q, mrange, cavoff, rho, A);    \
    break;                                                                                    \
  }
  switch (tbP.lmax) {
    DDC_LMAX_CASES(CASE)
    default:
      return cudaErrorInvalidValue;
  }
#undef CASE
  ++*L.launches;
  if ((e = cudaGetLastError())) return e;
  ZGroups none;
  k_far_cav<<<nsph, 128, 0, L.st>>>(nsph, ngrid, tbP.nylm, sph, q, mrange, rho, cavoff, cavpt,
                                    ccav, A, BT, DT, phi, ef, zg && !mrange ? *zg : none);
  ++*L.launches;
  return cudaGetLastError();
}

}  // namespace ddc
