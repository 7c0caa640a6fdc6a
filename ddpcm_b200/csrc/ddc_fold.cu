// ddc_fold.cu -- the operators' two contractions between grid points and
// harmonics, folded by the grid's reflections:
//   projection  y(lm,i)  = alpha sum_n w_n Y_lm(s_n) f(n,i)   (matvec.f90:131-135)
//   expansion   xi(n,i)  = [w_n] sum_lm Y_lm(s_n) s(lm,i)     (matvec.f90:189-204)
//
// A Lebedev grid maps onto itself under the reflections x -> -x, y -> -y and
// z -> -z, with equal weights, and every real harmonic is even or odd under
// each: Y_lm changes sign under x by (-1)^m (cosines) or (-1)^(m+1) (sines),
// under y only if it is a sine, under z by (-1)^(l+m).  So the harmonics fall
// into eight classes, and a class needs of a field only its part of the same
// parities: the Walsh-Hadamard sum of the field over the eight images of a
// point, one value per orbit.  An eighth of the multiplications remains
// (lmax 10, 590 points: 85 orbits, classes of 10 to 21 harmonics; 10,285
// instead of 71,390 products per sphere), and what bounds the kernels is
// latency and the field's memory traffic, no longer the FP64 pipe.
//
// A block takes eight spheres; its eight warps are the spheres while fields
// are read or written (lanes along the orbits: the grid is kept octant by
// octant, so the images of consecutive orbits are consecutive) and the eight
// classes in the products (FP64 tensor cores, mma.sync m8n8k4: eight spheres
// are the eight columns; tcgen05 has no FP64 kind).  The folded field lies in
// shared memory between the two, its rows 9 doubles apart so that neither
// side's accesses collide.
//
// Projection / expansion us (with 4 us of events), unfolded on the same tensor
// cores (40 % of the FP64 peak at best) and folded:
//   12 spheres, lmax 6, 110 points      6.9 /  7.9    8.0 /  8.6
//   600, lmax 8, 302 (FP32 fields)     10.7 / 11.0    8.6 / 10.7
//   2,000, lmax 8, 302                   17 / 17.6   10.7 / 11.6
//   5,000, lmax 10, 590                  49 / 47     23.1 / 24.5
// (625 blocks, four per SM: a second wave of 33; 4,700 spheres, one wave, 19
// and 20).  A pass of the 5,000 over field and vectors at the copy rate takes
// 4 us; the L1 traffic of the operands, 96 KB per block, 4 us more.
#include <algorithm>
#include <array>
#include <map>

#include "ddc_internal.h"

namespace ddc {
namespace {

constexpr int kT = 256;
constexpr int kChunk = 96;  // orbits of a block's pass (shared memory: 55 KB)
constexpr int kLm = 32;     // room per class in the list of harmonics (28 at lmax 12)

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}
// Walsh-Hadamard transform over three bits: v[c] = sum_k (-1)^popc(c & k) v[k]
__device__ __forceinline__ void wht8(double (&v)[8]) {
#pragma unroll
  for (int b = 1; b < 8; b <<= 1)
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (!(k & b)) {
        const double p = v[k], q = v[k | b];
        v[k] = p + q;
        v[k | b] = p - q;
      }
}

// the grid points of an orbit's eight images
struct Images {
  int4 v;
  __device__ int operator[](int k) const {
    const int p = k < 2 ? v.x : k < 4 ? v.y : k < 6 ? v.z : v.w;
    return k & 1 ? (unsigned)p >> 16 : p & 0xffff;
  }
};
__device__ __forceinline__ Images images(const FoldTab& ft, int o) {
  return Images{__ldg(reinterpret_cast<const int4*>(ft.img) + o)};
}

// the part of a class's product that one chunk of folded orbits gives; F: the
// class's rows, a: its operand in fragment order, MT row tiles ks apart
template <int MT>
__device__ __forceinline__ void proj_class(double (&acc)[4][2], const double* F, const double* a,
                                           int ks, int steps) {
  constexpr int U = MT < 3 ? 4 : MT == 3 ? 3 : 2;
  const int lane = threadIdx.x & 31, fr = lane >> 2, fk = lane & 3;
  for (int t = 0; t < steps; t += U) {
    double av[U][MT], bv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = t + u < steps;
#pragma unroll
      for (int i = 0; i < MT; ++i) av[u][i] = in ? a[((size_t)i * ks + t + u) * 32 + lane] : 0.0;
      bv[u] = in ? F[(4 * (t + u) + fk) * 9 + fr] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < MT; ++i) dmma(acc[i], av[u][i], bv[u]);
  }
}

template <class TB>
__global__ void __launch_bounds__(kT, 4) k_fold_proj(const __grid_constant__ FoldTab ft, int N,
                                                     double alpha, const TB* B, int ldb, double* C,
                                                     const SweepMask act) {
  extern __shared__ __align__(16) double fold_smem[];  // [8][oc][9]; then [8][nylm]
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, n0 = blockIdx.x * 8;
  const int NO = ft.norb, oc = ft.oc, NY = ft.nylm;
  // the tables do not change: read before the wait for the field
  Images im = images(ft, min(lane, NO - 1));
  chain_wait();
  // a sweep skips a block whose spheres all belong to stopped molecules
  if (act.st0 && __syncthreads_and(tid >= 8 || n0 + tid >= N || sweep_skip(act, n0 + tid)))
    return;
  const TB* row = B + (size_t)min(n0 + w, N - 1) * ldb;
  double acc[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0.0;
  for (int o0 = 0; o0 < NO; o0 += oc) {
    if (o0) __syncthreads();
    for (int o = lane; o < oc; o += 32) {
      double v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = o0 + o < NO ? (double)row[im[k]] : 0.0;
      im = images(ft, min(o0 + o + 32 < o0 + oc ? o0 + o + 32 : o0 + oc + lane, NO - 1));
      wht8(v);
#pragma unroll
      for (int c = 0; c < 8; ++c) fold_smem[(c * oc + o) * 9 + w] = v[c];
    }
    __syncthreads();
    const int ks = ft.otiles * 2, steps = min(oc / 4, ks - o0 / 4);
    const double* F = fold_smem + w * oc * 9;
    const double* a = ft.pf + ft.poff[w] + (size_t)o0 / 4 * 32;
    switch ((ft.cnt[w] + 7) / 8) {
      case 1: proj_class<1>(acc, F, a, ks, steps); break;
      case 2: proj_class<2>(acc, F, a, ks, steps); break;
      case 3: proj_class<3>(acc, F, a, ks, steps); break;
      case 4: proj_class<4>(acc, F, a, ks, steps); break;
      default: break;  // a class without harmonics
    }
  }
  __syncthreads();
  // the block's result is contiguous: put it in order before it is stored
  // (5,000 spheres: 27 us stored from the fragments, 19 so)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int j = 8 * i + (lane >> 2);
    if (j < ft.cnt[w]) {
      const int lm = ft.lm[w * kLm + j];
#pragma unroll
      for (int h = 0; h < 2; ++h) fold_smem[(2 * (lane & 3) + h) * NY + lm] = alpha * acc[i][h];
    }
  }
  __syncthreads();
  const int cnt = min(8, N - n0) * NY;
  double* out = C + (size_t)n0 * NY;
  for (int e = tid; e < cnt; e += kT) out[e] = fold_smem[e];
}

template <class TC>
__global__ void __launch_bounds__(kT, 4) k_fold_xi(const __grid_constant__ FoldTab ft,
                                                   const double* __restrict__ xf, int N,
                                                   const double* s, TC* xi, int ldc,
                                                   const SweepMask act) {
  extern __shared__ __align__(16) double fold_smem[];  // [8][oc][9]
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, n0 = blockIdx.x * 8;
  const int NO = ft.norb, oc = ft.oc, NY = ft.nylm, o0 = blockIdx.y * oc;
  const int fr = lane >> 2, fk = lane & 3;
  constexpr int KJ = kLm / 4 - 1;  // 28 harmonics at most
  constexpr int U = 2;             // tiles at a time, all their operands loaded first
  const int cnt = ft.cnt[w], kj = (cnt + 3) / 4, nt = min(oc / 8, ft.otiles - o0 / 8);
  const double* a = xf + ft.xoff[w] + (size_t)(o0 / 8) * kj * 32 + lane;
  double av[U][KJ];
  auto load = [&](int t) {
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int q = 0; q < KJ; ++q)
        av[u][q] = q < kj && t + u < nt ? a[((t + u) * kj + q) * 32] : 0.0;
  };
  // the tables do not change: what is read of them first is read before the
  // wait for the kernel that writes s
  int lmq[KJ];
#pragma unroll
  for (int q = 0; q < KJ; ++q) lmq[q] = 4 * q + fk < cnt ? ft.lm[w * kLm + 4 * q + fk] : -1;
  load(0);
  chain_wait();
  if (act.st0 && __syncthreads_and(tid >= 8 || n0 + tid >= N || sweep_skip(act, n0 + tid)))
    return;
  {
    const double* col = s + (size_t)min(n0 + fr, N - 1) * NY;
    double b[KJ];
#pragma unroll
    for (int q = 0; q < KJ; ++q) b[q] = lmq[q] >= 0 ? col[lmq[q]] : 0.0;
    for (int t = 0; t < nt; t += U) {
      double acc[U][2];
#pragma unroll
      for (int u = 0; u < U; ++u) acc[u][0] = acc[u][1] = 0.0;
      if (t) load(t);
#pragma unroll
      for (int q = 0; q < KJ; ++q)
        if (q < kj) {
#pragma unroll
          for (int u = 0; u < U; ++u) dmma(acc[u], av[u][q], b[q]);
        }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (t + u < nt) {
          double* x = fold_smem + (w * oc + 8 * (t + u) + fr) * 9 + 2 * fk;
          x[0] = acc[u][0];
          x[1] = acc[u][1];
        }
    }
  }
  __syncthreads();
  if (n0 + w >= N) return;
  TC* row = xi + (size_t)(n0 + w) * ldc;
#pragma unroll 2
  for (int o = lane; o < min(oc, NO - o0); o += 32) {
    const Images im = images(ft, o0 + o);
    const unsigned first = ft.first[o0 + o];  // images that are other points
    double v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = fold_smem[(c * oc + o) * 9 + w];
    wht8(v);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if ((first >> k) & 1u) row[im[k]] = (TC)v[k];
  }
}

// The operands in the order in which the fragments are read: a lane's value of
// a step beside its neighbours'.  Row (lane >> 2) and k (lane & 3) of the tile
// are harmonic and orbit in the projection (times the orbit's points over
// eight: its sum runs over eight images), orbit and harmonic in the expansion.
__global__ void k_fold_pack(FoldTab ft, const double* __restrict__ basis,
                            const double* __restrict__ bw, double* pf, double* xw, double* xb) {
  const int c = blockIdx.y, cnt = ft.cnt[c], mt = (cnt + 7) / 8, kj = (cnt + 3) / 4;
  const int ks = ft.otiles * 2;
  const int e = blockIdx.x * blockDim.x + threadIdx.x, lane = e & 31, step = e >> 5;
  const int r = lane >> 2, k = lane & 3;
  if (step < mt * ks) {
    const int j = step / ks * 8 + r, o = step % ks * 4 + k;
    pf[ft.poff[c] + e] = j < cnt && o < ft.norb ? bw[(size_t)o * ft.nylm + ft.lm[c * kLm + j]] *
                                                      (0.125 * __popc(ft.first[o]))
                                                : 0.0;
  }
  if (step < ft.otiles * kj) {
    const int o = step / kj * 8 + r, j = step % kj * 4 + k;
    const bool in = j < cnt && o < ft.norb;
    const size_t at = in ? (size_t)o * ft.nylm + ft.lm[c * kLm + j] : 0;
    xw[ft.xoff[c] + e] = in ? bw[at] : 0.0;
    xb[ft.xoff[c] + e] = in ? basis[at] : 0.0;
  }
}

size_t fold_smem_size(const FoldTab& t) {
  return sizeof(double) * std::max(8 * t.oc * 9, 8 * t.nylm);
}
// the most that any context needs.  The kernels' limit belongs to the function,
// whatever context set it, so it is the same for all of them (it is a cap: a
// launch takes what it asks for)
constexpr int kSmemMost = (int)sizeof(double) * 8 * kChunk * 9;
static_assert((DDC_MAX_LMAX + 1) * (DDC_MAX_LMAX + 1) <= kChunk * 9, "the result's rows fit");

}  // namespace

// g4: the grid octant by octant, the first octant's points (no negative
// coordinate) first: one of each orbit.  False if the grid lacks an image.
bool fold_tables(const std::vector<double>& g4, int lmax, FoldTab& t, std::vector<short>& img,
                 std::vector<uint8_t>& first, std::vector<short>& lm) {
  const int G = (int)g4.size() / 4;
  std::map<std::array<double, 3>, int> at;
  // adding zero turns -0 into +0
  for (int i = 0; i < G; ++i)
    at[{g4[4 * i] + 0.0, g4[4 * i + 1] + 0.0, g4[4 * i + 2] + 0.0}] = i;
  int no = 0;
  while (no < G && g4[4 * no] >= 0.0 && g4[4 * no + 1] >= 0.0 && g4[4 * no + 2] >= 0.0) ++no;
  img.assign(8 * (size_t)no, 0);
  first.assign(no, 0);
  int points = 0;
  for (int o = 0; o < no; ++o)
    for (int k = 0; k < 8; ++k) {
      std::array<double, 3> p;
      for (int d = 0; d < 3; ++d) p[d] = ((k >> d) & 1 ? -g4[4 * o + d] : g4[4 * o + d]) + 0.0;
      const auto f = at.find(p);
      if (f == at.end() || g4[4 * f->second + 3] != g4[4 * o + 3]) return false;
      img[(size_t)o * 8 + k] = (short)f->second;
      bool seen = false;
      for (int q = 0; q < k; ++q) seen = seen || img[(size_t)o * 8 + q] == f->second;
      if (!seen) {
        first[o] |= (uint8_t)(1u << k);
        ++points;
      }
    }
  if (points != G) return false;
  t.norb = no;
  t.otiles = (no + 7) / 8;
  t.oc = std::min(kChunk, 8 * t.otiles);
  t.nylm = (lmax + 1) * (lmax + 1);
  lm.assign(8 * kLm, 0);
  for (int c = 0; c < 8; ++c) t.cnt[c] = 0;
  for (int l = 0; l <= lmax; ++l)
    for (int m = -l; m <= l; ++m) {
      const int a = std::abs(m), sine = m < 0 ? 1 : 0;
      const int c = ((a + sine) & 1) | sine << 1 | ((l + a) & 1) << 2;
      lm[c * kLm + t.cnt[c]++] = (short)(l * l + l + m);
    }
  int po = 0, xo = 0;
  for (int c = 0; c < 8; ++c) {
    t.poff[c] = po;
    t.xoff[c] = xo;
    po += (t.cnt[c] + 7) / 8 * t.otiles * 2 * 32;
    xo += (t.cnt[c] + 3) / 4 * t.otiles * 32;
  }
  t.psize = po;
  t.xsize = xo;
  return true;
}

cudaError_t launch_fold_pack(Launch L, const FoldTab& t, const double* basis, const double* bw,
                             double* pf, double* xw, double* xb) {
  cudaError_t e;
  for (auto f : {(const void*)k_fold_proj<double>, (const void*)k_fold_proj<float>,
                 (const void*)k_fold_xi<double>, (const void*)k_fold_xi<float>})
    if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMost)))
      return e;
  const int n = std::max(4 * t.otiles * 2, t.otiles * 7) * 32;
  k_fold_pack<<<dim3((n + kT - 1) / kT, 8), kT, 0, L.st>>>(t, basis, bw, pf, xw, xb);
  ++*L.launches;
  return cudaGetLastError();
}
template <class TB>
cudaError_t launch_fold_proj(Launch L, const FoldTab& t, int N, double alpha, const TB* B, int ldb,
                             double* C, const SweepMask& act) {
  if (N == 0) return cudaSuccess;
  ++*L.launches;
  return launch_chained(k_fold_proj<TB>, dim3((N + 7) / 8), kT, fold_smem_size(t), L.st, t, N, alpha, B,
                        ldb, C, act);
}
template <class TC>
cudaError_t launch_fold_xi(Launch L, const FoldTab& t, bool weighted, int N, const double* s,
                           TC* xi, int ldc, const SweepMask& act) {
  if (N == 0) return cudaSuccess;
  ++*L.launches;
  return launch_chained(k_fold_xi<TC>, dim3((N + 7) / 8, (t.norb + t.oc - 1) / t.oc), kT,
                        fold_smem_size(t), L.st, t, weighted ? t.xfw : t.xfb, N, s, xi, ldc, act);
}
template cudaError_t launch_fold_proj(Launch, const FoldTab&, int, double, const double*, int,
                                      double*, const SweepMask&);
template cudaError_t launch_fold_proj(Launch, const FoldTab&, int, double, const float*, int,
                                      double*, const SweepMask&);
template cudaError_t launch_fold_xi(Launch, const FoldTab&, bool, int, const double*, double*, int,
                                    const SweepMask&);
template cudaError_t launch_fold_xi(Launch, const FoldTab&, bool, int, const double*, float*, int,
                                    const SweepMask&);

}  // namespace ddc
