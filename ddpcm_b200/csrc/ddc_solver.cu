// ddc_solver.cu -- the Jacobi/DIIS iteration (jacobi_diis.f90:1-360) on the
// device, for one molecule or many, one system or the direct and the adjoint
// one side by side.
//
// Every molecule of every system runs the reference's algorithm on its own
// segment of the vectors: own history, Gram matrix, restarts and convergence
// test, all in device memory, so that the host only launches sweeps and looks
// now and then whether anything still runs (with the bordered system solved on
// the host an iteration would wait for two round trips).  The vectors are cut
// into chunks of CK consecutive elements; a chunk is a block.  Two kernels per
// iteration, each over the chunks of all running systems (grid y):
//   k_gram    Jacobi iterate, increment, the chunk's part of the Gram row; the
//             molecule's last chunk to arrive sums the parts in chunk order
//             and solves the bordered system (the whole block, one barrier
//             per pivot);
//   k_extrap  extrapolated iterate, the chunk's part of the increment norm;
//             the molecule's last chunk applies the stop test.
// Sums have a fixed order: the results are bit-reproducible.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "ddc_internal.h"

namespace ddc {
namespace {

constexpr int kT = 256;  // threads per block
constexpr int kW = kT / 32;

__device__ __forceinline__ int l_of(int lm) {
  int l = (int)sqrtf((float)lm);
  while ((l + 1) * (l + 1) <= lm) ++l;
  while (l * l > lm) --l;
  return l;
}
__device__ __forceinline__ int lm_add(int lm, int d, int nylm) {
  lm += d;
  return lm >= nylm ? lm - nylm : lm;
}
// chunk c's molecule, and the molecule's spheres and chunks (one molecule:
// no maps)
__device__ __forceinline__ int mol_of(const SolverArgs& a, int c) { return a.cmol ? a.cmol[c] : 0; }
__device__ __forceinline__ int2 spheres_of(const SolverArgs& a, int k) {
  return a.cmol ? make_int2(a.off[k], a.off[k + 1]) : make_int2(0, a.nsph);
}
__device__ __forceinline__ int2 chunks_of(const SolverArgs& a, int k) {
  return a.cmol ? make_int2(a.cfirst[k], a.cfirst[k + 1]) : make_int2(0, a.nchunk);
}
struct Segment {
  long long b0;  // first element
  int cnt;       // elements
};
// Blocks per chunk in k_extrap: its blocks want short segments, as many loads at
// once as there are vectors, while k_gram's wait longer for a short segment
// than they work on it.  5,000 spheres, lmax 10, FP64, both systems: k_gram
// 67 us by 512 elements and 53 by 2,048, k_extrap 41 and 70.
template <int CK>
constexpr int kSub = CK == 2048 ? 4 : 1;
template <int CK>
__device__ __forceinline__ Segment segment_of(const SolverArgs& a, int c, int k) {
  const int2 sp = spheres_of(a, k), ch = chunks_of(a, k);
  Segment s;
  s.b0 = (long long)sp.x * a.nylm + (long long)(c - ch.x) * CK;
  s.cnt = (int)min((long long)CK, (long long)sp.y * a.nylm - s.b0);
  return s;
}

// Last arriving chunk of molecule k (the counter is reset for the next
// kernel).  Every block of the molecule calls it after writing its parts.
__device__ __forceinline__ bool last_chunk(const SolverArgs& a, const SolverSys& s, int k, int sub = 1) {
  __shared__ unsigned s_last;
  __threadfence();
  __syncthreads();
  const int2 ch = chunks_of(a, k);
  if (threadIdx.x == 0) {
    s_last = atomicAdd(s.cnt + k, 1u) == (unsigned)((ch.y - ch.x) * sub) - 1 ? 1u : 0u;
    if (s_last) s.cnt[k] = 0u;
  }
  __syncthreads();
  if (s_last) __threadfence();
  return s_last != 0;
}
// sum over the block, valid in thread 0
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double sh[kW];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int ww = 0; ww < kW; ++ww) t += sh[ww];
  return t;
}

// Sums entries [0, nv) of molecule k's parts in a fixed order: warp w the
// chunks w, w + 8, ... (a lane per entry), then the warps in order; a single
// entry by thread.
__device__ __forceinline__ void sum_parts(const SolverArgs& a, const SolverSys& s, int k, int nv,
                                          double* out, int sub = 1) {
  __shared__ double acc[kW][kMaxHist + 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int2 ch = chunks_of(a, k);
  if (nv == 1) {
    double v = 0.0;
#pragma unroll 4
    for (int c = ch.x * sub + (int)threadIdx.x; c < ch.y * sub; c += kT)
      v += __ldcg(s.part + (size_t)c * (kMaxHist + 1));
    v = block_sum(v);
    if (threadIdx.x == 0) out[0] = v;
    __syncthreads();
    return;
  }
  for (int h = lane; h < nv; h += 32) {
    double v = 0.0;
#pragma unroll 16
    for (int c = ch.x + w; c < ch.y; c += kW) v += __ldcg(s.part + (size_t)c * (kMaxHist + 1) + h);
    acc[w][h] = v;
  }
  __syncthreads();
  if (threadIdx.x < nv) {
    double v = acc[0][threadIdx.x];
#pragma unroll
    for (int ww = 1; ww < kW; ++ww) v += acc[ww][threadIdx.x];
    out[threadIdx.x] = v;
  }
  __syncthreads();
}
// Gauss-Jordan with full pivoting (gjinv, jacobi_diis.f90:272-360) of an
// n x n system, n <= 32, by the whole block: thread (w, lane) holds column
// `lane` of the rows w, w + 8, w + 16, w + 24 in a[], the rows' right-hand
// sides in b[] (every lane).  The pivot is the largest |a| over free rows and
// columns, compared by its high word alone (20 bits of the mantissa), the first
// in the reference's scan order (rows outer, columns inner) among equals: a
// pivot within 2^-20 of the largest, so not always the reference's, nor its
// rounding bit for bit; singular, as there, only without a pivot (here: one of
// 2^-1042 or more).  Rows stay in place (myrow: the row that column `lane` was
// pivoted in) instead of being swapped, which changes no value.  A chain of n dependent
// pivots, each some hundred cycles of latency: one barrier per pivot, the
// rows mirrored in shared memory as they are updated, so that every warp
// reads the pivot row of whichever warp offers it; 650 cycles per pivot
// (1,500 when the warps compared and handed over FP64 candidates).  Solution
// in x[0..n); false when singular.
__device__ bool gauss_jordan(int n, double (&a)[4], double (&b)[4], double* x) {
  __shared__ double mir[2][32][33];  // the matrix and (column 32) the right-hand side
  __shared__ uint2 cand[2][kW];      // high word and position of each warp's candidate
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned rfree = 0;  // rows of this warp (bit u) not pivoted yet
#pragma unroll
  for (int u = 0; u < 4; ++u) rfree |= (w + 8 * u < n ? 1u : 0u) << u;
  bool cfree = lane < n;
  int myrow = -1;  // the row column `lane` was pivoted in
  for (int i = 0; i < n; ++i) {
    const int buf = i & 1;
    unsigned key = 0, code = 0xffffffffu;  // position: row * 32 + column
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      mir[buf][w + 8 * u][lane] = a[u];
      if (lane == 0) mir[buf][w + 8 * u][32] = b[u];
      const unsigned h = (rfree >> u) & 1u ? (unsigned)__double2hiint(a[u]) & 0x7fffffffu : 0u;
      if (h > key) {
        key = h;
        code = (w + 8 * u) * 32 + lane;
      }
    }
    if (!cfree) key = 0;
    const unsigned mk = __reduce_max_sync(0xffffffffu, key);
    const unsigned pos = __reduce_min_sync(0xffffffffu, key == mk && key ? code : 0xffffffffu);
    if (lane == 0) cand[buf][w] = make_uint2(mk, pos);
    __syncthreads();
    const uint2 cd = cand[buf][lane & (kW - 1)];
    const unsigned bk = __reduce_max_sync(0xffffffffu, cd.x);
    if (!bk) return false;  // no non-zero free entry
    const unsigned rc = __reduce_min_sync(0xffffffffu, cd.x == bk ? cd.y : 0xffffffffu);
    const int r = rc >> 5, c = rc & 31;
    const double pinv = 1.0 / mir[buf][r][c];
    const double pr = mir[buf][r][lane] * pinv, pb = mir[buf][r][32] * pinv;
    if ((r & (kW - 1)) == w) rfree &= ~(1u << (r >> 3));
    if (lane == c) {
      cfree = false;
      myrow = r;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const double dum = mir[buf][w + 8 * u][c];
      if (w + 8 * u == r) {
        a[u] = pr;
        b[u] = pb;
      } else {
        a[u] -= pr * dum;
        b[u] -= pb * dum;
      }
    }
  }
  __shared__ double sol[32];
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (lane == 0) sol[w + 8 * u] = b[u];
  __syncthreads();
  if (w == 0 && lane < n) x[lane] = sol[myrow];
  __syncthreads();
  return true;
}

template <class H, int CK>
__global__ void __launch_bounds__(kT, 4) k_gram(const __grid_constant__ SolverArgs a) {
  chain_wait();
  constexpr int TILE = CK < 2048 ? CK : 2048;
  constexpr int U = TILE / kT;
  constexpr int KS = (kMaxHist + kW - 1) / kW;  // history vectors per warp
  constexpr int HL = 16;                        // loads per lane in flight
  static_assert(CK % TILE == 0 && TILE % (32 * HL) == 0, "chunk tiling");
  const SolverSys& s = a.sys[a.first + blockIdx.y];
  const int c = blockIdx.x, k = mol_of(a, c), tid = threadIdx.x;
  __shared__ int pm[kMaxHist];  // logical to physical history slots
  __shared__ H es[TILE];
  __shared__ double red[kMaxHist + 1];
  __shared__ double row[kMaxHist + 1], sol[kMaxHist + 1];
  const int nd = max(a.ndiis, 1);
  const int st = s.status[k], nmo = s.nmat[k];
  const int sl = tid < nd ? s.slot[(size_t)k * nd + tid] : 0;
  if (st != 0) return;
  // after `nmat` reaches ndiis the ten oldest are dropped (jacobi_diis.f90:196-205)
  const bool shift = a.ndiis && nmo >= nd;
  const int nm = a.ndiis ? (shift ? nmo - 10 : nmo) : 1, nh = nm - 1;
  if (tid < nd) pm[shift ? (tid + nd - 10) % nd : tid] = sl;
  const int lane = tid & 31, w = tid >> 5;
  const long long N = a.n_total;
  const Segment sg = segment_of<CK>(a, c, k);
  H* xnew = static_cast<H*>(s.hx) + sg.b0;
  H* enew = static_cast<H*>(s.he) + sg.b0;
  const H* he = static_cast<const H*>(s.he) + sg.b0;
  double ee = 0.0, d[KS];
#pragma unroll
  for (int q = 0; q < KS; ++q) d[q] = 0.0;
  const int dt = kT % a.nylm;
  int lm = (int)((sg.b0 + tid) % a.nylm);
  for (int t0 = 0; t0 < sg.cnt; t0 += TILE) {
    double rv[U], yv[U], xv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = t0 + tid + u * kT;
      rv[u] = j < sg.cnt ? s.rhs[sg.b0 + j] : 0.0;
      yv[u] = j < sg.cnt ? s.y[sg.b0 + j] : 0.0;
      xv[u] = j < sg.cnt ? s.x[sg.b0 + j] : 0.0;
    }
    __syncthreads();  // pm is there; es is free
    const size_t pn = (size_t)pm[nm - 1] * N;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = t0 + tid + u * kT;
      H eh = 0;
      if (j < sg.cnt) {
        const double xn = a.facl[l_of(lm)] * (rv[u] - yv[u]);
        eh = (H)(xn - xv[u]);
        xnew[pn + j] = (H)xn;
        enew[pn + j] = eh;
      }
      es[tid + u * kT] = eh;
      ee = fma((double)eh, (double)eh, ee);
      lm = lm_add(lm, dt, a.nylm);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < KS; ++q) {
      const int kk = w + kW * q;
      if (kk < nh) {
        const H* hk = he + (size_t)pm[kk] * N + t0;
        const int left = sg.cnt - t0;
#pragma unroll 2
        for (int j0 = 0; j0 < TILE; j0 += 32 * HL) {
          H hv[HL];
#pragma unroll
          for (int u = 0; u < HL; ++u) {
            const int j = j0 + u * 32 + lane;
            hv[u] = j < left ? hk[j] : H(0);
          }
#pragma unroll
          for (int u = 0; u < HL; ++u)
            d[q] = fma((double)es[j0 + u * 32 + lane], (double)hv[u], d[q]);
        }
      }
    }
  }
  if (!a.ndiis) {  // plain Jacobi: no Gram row
    if (!last_chunk(a, s, k)) return;
    if (tid == 0) s.ext[k] = -1;
    return;
  }
  ee = block_sum(ee);  // in thread 0
#pragma unroll
  for (int q = 0; q < KS; ++q) {
    const int kk = w + kW * q;
    if (kk < nh) {
      double v = d[q];
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[kk] = v;
    }
  }
  if (tid == 0) red[nh] = ee;
  __syncthreads();
  if (tid <= nh) s.part[(size_t)c * (kMaxHist + 1) + tid] = red[tid];
  if (!last_chunk(a, s, k)) return;
  sum_parts(a, s, k, nh + 1, row);
  // bordered Gram matrix (makeb, jacobi_diis.f90:232-270): the inner products
  // are kept by physical slot, the new row is still in shared memory
  double* G = s.gram + (size_t)k * nd * nd;
  // scaled by powers of two to a diagonal in [0.5, 2): the increments of one
  // history span many decades and their products twice as many, and unscaled
  // the elimination loses the small ones to the rounding of the large; the
  // coefficients of the last iterations are then noise that slows the solve
  // and now and then stops it early.  200 chains of 12 spheres, lmax 6, to 1e-12,
  // both solutions against direct ones: unscaled (the reference's elimination) 24.5 and
  // 24.8 iterations on average, errors of 5e-13 and 1e-13 in the median, 89 of
  // 400 above 1e-10 and up to 1.2e-8; scaled 21.2 and 21.0 iterations, 9e-12 and
  // 2e-12, none above 4e-11.  (The median is larger because a solve stops where the
  // test says; with noise for coefficients it ran on and ended far below it.)
  // The border row's scale is the smallest, so that the border stays below 1.
  const int n1 = nm + 1, pn = pm[nm - 1];
  __shared__ int ex[kMaxHist + 1];  // row r is scaled by 2^-ex[r]
  if (w == 0) {
    int k = INT_MAX;
    if (lane >= 1 && lane < n1) {
      const double g = lane == nm ? row[nm - 1] : G[pm[lane - 1] * nd + pm[lane - 1]];
      k = g > 0.0 && g < 1e300 ? (((__double2hiint(g) >> 20) & 0x7ff) - 1022) >> 1 : 0;
    }
    const int k0 = __reduce_min_sync(0xffffffffu, k);
    if (lane < n1) ex[lane] = lane == 0 ? -k0 : k;
  }
  __syncthreads();
  auto pow2 = [](int k) { return __hiloint2double((1023 + k) << 20, 0); };
  const int exl = lane < n1 ? ex[lane] : 0;
  double ga[4], gb[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int r = w + 8 * u;
    double v = 0.0;
    if (r < n1 && lane < n1) {
      if (r == 0 || lane == 0) v = r == lane ? 0.0 : 1.0;
      else if (r == nm) v = row[lane - 1];
      else if (lane == nm) v = row[r - 1];
      else v = G[pm[r - 1] * nd + pm[lane - 1]];
    }
    const double sr = r < n1 ? pow2(-ex[r]) : 1.0;
    ga[u] = v * pow2(-exl) * sr;
    gb[u] = r == 0 ? sr : 0.0;
  }
  if (tid < nm) {
    G[pn * nd + pm[tid]] = row[tid];
    G[pm[tid] * nd + pn] = row[tid];
  }
  const bool ok = gauss_jordan(n1, ga, gb, sol);
  if (shift && tid < nd) s.slot[(size_t)k * nd + tid] = pm[tid];
  if (ok && tid < nm) s.coef[(size_t)k * kMaxHist + tid] = sol[tid + 1] * pow2(-ex[tid + 1]);
  if (tid == 0) {
    if (ok) {
      s.nmat[k] = nm + 1;
    } else {  // singular: restart the history (jacobi_diis.f90:214-217)
      s.nmat[k] = 1;
      s.restarts[k] += 1;
    }
    s.ext[k] = ok ? nm : -nm;
  }
}

// DIIS extrapolation (jacobi_diis.f90:222-226) or, after a singular Gram
// system, the Jacobi iterate; increment H-norm (hnorm, matvec.f90:281-323)
// and update.
template <class H, int CK>
__global__ void __launch_bounds__(kT) k_extrap(const __grid_constant__ SolverArgs a) {
  chain_wait();
  constexpr int SUB = kSub<CK>, LEN = CK / SUB;
  constexpr int U = LEN / kT < 4 ? LEN / kT : 4;  // elements per thread and step
  // history vectors loaded at a time, unconditionally: 4 to 16 loads of a
  // thread in flight.  With loads behind the range test one at a time went out
  // (5,000 spheres FP64 54 us, 41 now; 20,000 FP32 by 8,192 73 and 58; a read of
  // the history at the copy rate 34 and 60); 2 at a time 42 and 57, 8: 45 and 77
  constexpr int B = 4;
  const int q = a.first + blockIdx.y;
  const SolverSys& s = a.sys[q];
  const int c = blockIdx.x, k = mol_of(a, c / SUB), tid = threadIdx.x;
  __shared__ int pm[kMaxHist];
  __shared__ double cf[kMaxHist];
  __shared__ double tot[1];
  const int nd = max(a.ndiis, 1);
  const int st = s.status[k], ext = s.ext[k];
  const int sl = tid < nd ? s.slot[(size_t)k * nd + tid] : 0;
  const double cv = tid < kMaxHist ? s.coef[(size_t)k * kMaxHist + tid] : 0.0;
  if (st != 0) return;
  const int nm = ext > 0 ? ext : -ext;
  const bool ok = ext > 0;
  if (tid < nd) pm[tid] = sl;
  if (tid < kMaxHist) cf[tid] = cv;
  __syncthreads();
  const long long N = a.n_total;
  Segment sg = segment_of<CK>(a, c / SUB, k);
  sg.b0 += (c % SUB) * LEN;
  sg.cnt = min(sg.cnt - (c % SUB) * LEN, LEN);  // zero or less: nothing here
  const H* hx = static_cast<const H*>(s.hx) + sg.b0;
  const int dt = kT % a.nylm;
  int lm = (int)((sg.b0 + tid) % a.nylm);
  double acc = 0.0;
  for (int u0 = 0; u0 * kT < sg.cnt; u0 += U) {
    double xo[U], xold[U];
    int j[U];  // past the end: the last element again, not stored
#pragma unroll
    for (int u = 0; u < U; ++u) {
      j[u] = min(tid + (u0 + u) * kT, sg.cnt - 1);
      xold[u] = s.x[sg.b0 + j[u]];
      xo[u] = 0.0;
    }
    if (ok) {
      int h = 0;
      for (; h + B <= nm; h += B) {
        H hv[B][U];
#pragma unroll
        for (int g = 0; g < B; ++g)
#pragma unroll
          for (int u = 0; u < U; ++u) hv[g][u] = hx[(size_t)pm[h + g] * N + j[u]];
#pragma unroll
        for (int g = 0; g < B; ++g)
#pragma unroll
          for (int u = 0; u < U; ++u) xo[u] = fma(cf[h + g], (double)hv[g][u], xo[u]);
      }
      if (h < nm) {
        H hv[B][U];
#pragma unroll
        for (int g = 0; g < B; ++g)
#pragma unroll
          for (int u = 0; u < U; ++u) hv[g][u] = hx[(size_t)pm[min(h + g, nm - 1)] * N + j[u]];
#pragma unroll
        for (int g = 0; g < B; ++g)
          if (h + g < nm) {
#pragma unroll
            for (int u = 0; u < U; ++u) xo[u] = fma(cf[h + g], (double)hv[g][u], xo[u]);
          }
      }
    } else {
      const H* xjac = hx + (size_t)pm[nm - 1] * N;
#pragma unroll
      for (int u = 0; u < U; ++u) xo[u] = (double)xjac[j[u]];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (tid + (u0 + u) * kT < sg.cnt) {
        const double dd = xo[u] - xold[u];
        acc = fma(dd * dd, a.hw[l_of(lm)], acc);
        s.x[sg.b0 + j[u]] = xo[u];
      }
      lm = lm_add(lm, dt, a.nylm);
    }
  }
  acc = block_sum(acc);
  if (tid == 0) s.part[(size_t)c * (kMaxHist + 1)] = acc;
  if (!last_chunk(a, s, k, SUB)) return;
  sum_parts(a, s, k, 1, tot, SUB);
  if (tid == 0) {
    const int2 sp = spheres_of(a, k);
    const double nrm = sqrt(tot[0] / (double)max(sp.y - sp.x, 1));
    s.norm[k] = nrm;
    const int it = s.iters[k] + 1;
    s.iters[k] = it;
    if (s.its[k] + it <= a.nlog) s.log[s.its[k] + it - 1] = nrm;
    const int now = nrm < s.tolk[k] ? 1 : (it >= s.maxk[k] ? 2 : (isfinite(nrm) ? 0 : 3));
    if (now != 0) {
      s.status[k] = now;
      // the system's last molecule: tell the host the sweep (1, 2, ...)
      if (atomicSub(a.active + q, 1) == 1) {
        *(volatile int*)(a.hstop + q) = a.sweep;
        __threadfence_system();
      }
    }
  }
}

__device__ __forceinline__ void start_molecule(const SolverArgs& a, const SolverSys& s, int k,
                                               double tol, int budget) {
  s.status[k] = 0;
  s.nmat[k] = 1;
  s.iters[k] = 0;
  s.restarts[k] = 0;
  s.tolk[k] = tol;
  s.maxk[k] = budget;
}

// starting state of every molecule: an FP64 solve runs at once; a mixed one
// waits for its first residual
__global__ void k_begin(const __grid_constant__ SolverArgs a, bool mixed) {
  const int nd = max(a.ndiis, 1);
  const SolverSys& s = a.sys[blockIdx.y];
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < a.nmol * nd;
       e += gridDim.x * blockDim.x) {
    const int k = e / nd, j = e - k * nd;
    s.slot[e] = j;
    if (j) continue;
    const int2 sp = spheres_of(a, k);
    const bool empty = sp.y <= sp.x;
    start_molecule(a, s, k, a.tol, a.max_iter);
    s.cnt[k] = 0u;
    s.run[k] = empty ? 1 : 0;
    s.its[k] = s.outer[k] = s.rst[k] = s.upd[k] = 0;
    s.norm[k] = s.last[k] = 0.0;
    if (empty || mixed) s.status[k] = 1;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) a.active[blockIdx.y] = mixed ? 0 : a.nonempty;
}

// Mixed refinement, per molecule still refining: r = rhs - y - x / facl with
// y = O x, the FP64 Jacobi increment e = D^-1 r and its H-norm.  The
// molecule's last chunk applies the stop test (not after an FP32 residual)
// or starts the inner solve L e = r from that e, reducing the increment by
// rho (floor 0.3 tol) within the remaining budget.
// Every restart of the inner DIIS costs about ten iterations before the
// extrapolation has a subspace again, so the split between the inner solves
// matters: at the 20,000-sphere workload rho = 1e-5 took 88 / 86 iterations,
// 3e-5 86 / 80, 1e-4 80 / 79 (Esolv 2e-10 from the FP64 oracle; at most
// 3.9e-10 over eight smaller molecules, as with 1e-5), and 3e-4 84 / 71 but
// 1.7e-9 on the 600-sphere configuration.
template <int CK>
__global__ void __launch_bounds__(kT) k_residual(const __grid_constant__ SolverArgs a, bool f32_res) {
  const int q = blockIdx.y;
  const SolverSys& s = a.sys[q];
  const int c = blockIdx.x, k = mol_of(a, c), tid = threadIdx.x;
  if (s.run[k] != 0) return;
  __shared__ double tot[1];
  const Segment sg = segment_of<CK>(a, c, k);
  const int dt = kT % a.nylm;
  int lm = (int)((sg.b0 + tid) % a.nylm);
  double acc = 0.0;
#pragma unroll 2
  for (int j = tid; j < CK; j += kT) {
    if (j < sg.cnt) {
      const long long e = sg.b0 + j;
      const int l = l_of(lm);
      const double rr = s.orhs[e] - s.y[e] - s.ox[e] / a.facl[l];
      const double dd = a.facl[l] * rr;
      s.r[e] = rr;
      s.x[e] = dd;
      acc = fma(dd * dd, a.hw[l], acc);
    }
    lm = lm_add(lm, dt, a.nylm);
  }
  acc = block_sum(acc);
  if (tid == 0) s.part[(size_t)c * (kMaxHist + 1)] = acc;
  if (!last_chunk(a, s, k)) return;
  sum_parts(a, s, k, 1, tot);
  if (tid == 0) {
    const int2 sp = spheres_of(a, k);
    const double nrm = sqrt(tot[0] / (double)max(sp.y - sp.x, 1));
    s.outer[k] += 1;
    s.last[k] = nrm;
    int run = 0;
    if (!isfinite(nrm)) run = 3;
    else if (nrm < a.tol && !f32_res) run = 1;
    else if (s.its[k] >= a.max_iter) run = 2;
    s.run[k] = run;
    s.upd[k] = run == 0;
    if (run == 0) {
      start_molecule(a, s, k, fmax(1e-4 * nrm, 0.3 * a.tol), a.max_iter - s.its[k]);
      atomicAdd(a.active + q, 1);
    } else {
      s.status[k] = 1;
    }
  }
  const int nd = max(a.ndiis, 1);
  if (tid < nd) s.slot[(size_t)k * nd + tid] = tid;
}

// x += e over the molecules whose inner solve ran, and its account
template <int CK>
__global__ void __launch_bounds__(kT) k_update(const __grid_constant__ SolverArgs a) {
  const SolverSys& s = a.sys[blockIdx.y];
  const int c = blockIdx.x, k = mol_of(a, c);
  if (c == 0 && threadIdx.x == 0) a.active[blockIdx.y] = 0;
  if (!s.upd[k]) return;
  const Segment sg = segment_of<CK>(a, c, k);
  for (int j = threadIdx.x; j < sg.cnt; j += kT) s.ox[sg.b0 + j] += s.x[sg.b0 + j];
  if (c == chunks_of(a, k).x && threadIdx.x == 0) {
    // iterations that did not converge count their whole budget
    s.its[k] += s.status[k] == 1 ? s.iters[k] : s.maxk[k];
    s.rst[k] += s.restarts[k];
  }
}

template <class F>
cudaError_t by_chunk(const SolverArgs& a, F&& f) {
  if (a.chunk == 512) f(std::integral_constant<int, 512>{});
  else if (a.chunk == 2048) f(std::integral_constant<int, 2048>{});
  else if (a.chunk == 8192) f(std::integral_constant<int, 8192>{});
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
}

}  // namespace

// Rows of the partial sums: a block of k_extrap each
int solver_parts(int nchunk, int chunk) { return nchunk * (chunk == 2048 ? kSub<2048> : 1); }
// Chunk length of k_gram's blocks (k_gram us, both systems, FP64): 512 elements
// while 2,048 would leave half of the SMs without a block per system (154,000
// elements 33.4 by 512 and 32.8 by 2,048, 250,000 42.9 and 38.9, 605,000 67 and
// 53); 8,192 for one molecule that fills the device with those, so that the
// last chunk sums few parts (2.4 million, FP32: 140 by 2,048 and 83 by 8,192)
int solver_chunk(long long n_total, bool one) {
  return n_total < 148LL * 1024 ? 512 : one && n_total >= 148LL * 8192 ? 8192 : 2048;
}

cudaError_t launch_solver_begin(Launch L, const SolverArgs& a, int ns, bool mixed) {
  const int n = a.nmol * std::max(a.ndiis, 1);
  k_begin<<<dim3(std::min((n + 255) / 256, 1024), ns), 256, 0, L.st>>>(a, mixed);
  ++*L.launches;
  return cudaGetLastError();
}
cudaError_t launch_solver_step(Launch L, const SolverArgs& a, int ns, bool f32, int which) {
  if (a.nchunk == 0) return cudaSuccess;
  ++*L.launches;
  return by_chunk(a, [&](auto ck) {
    constexpr int CK = decltype(ck)::value;
    const dim3 g(a.nchunk * (which == 0 ? 1 : kSub<CK>), ns);
    if (which == 0) {
      launch_chained(f32 ? k_gram<float, CK> : k_gram<double, CK>, g, kT, 0, L.st, a);
    } else {
      launch_chained(f32 ? k_extrap<float, CK> : k_extrap<double, CK>, g, kT, 0, L.st, a);
    }
  });
}
cudaError_t launch_solver_residual(Launch L, const SolverArgs& a, int ns, bool f32_res) {
  if (a.nchunk == 0) return cudaSuccess;
  ++*L.launches;
  return by_chunk(a, [&](auto ck) {
    k_residual<decltype(ck)::value><<<dim3(a.nchunk, ns), kT, 0, L.st>>>(a, f32_res);
  });
}
cudaError_t launch_solver_update(Launch L, const SolverArgs& a, int ns) {
  if (a.nchunk == 0) return cudaSuccess;
  ++*L.launches;
  return by_chunk(
      a, [&](auto ck) { k_update<decltype(ck)::value><<<dim3(a.nchunk, ns), kT, 0, L.st>>>(a); });
}

}  // namespace ddc
