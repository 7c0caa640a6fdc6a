// ddc_lxs.cu -- the per-iteration operators L and L* over the (sphere, point,
// neighbour) triples (lx matvec.f90:94-148 with calcv ddcosmo.f90:1671-1746
// and intmlp :1140-1178; lstarx matvec.f90:161-235 with adjrhs
// ddcosmo.f90:1301-1384), FP64 and FP32.
//
// Both operators run over the same triples (a, n, b): grid point n of sphere
// a inside sphere b (t < 1).  They share the weight W = chi(t) / f_a(n) and
// the values t^l Y_lm(s), s the unit vector from c_b to c_a + r_a s_n:
//   lx     (output a):  pot_a(n) += W sum_lm K_lm t^l Y_lm(s) X_b,lm
//   lstarx (output b):  y_b,lm   -= K_lm w_n xi_a(n) W t^l Y_lm(s)
//
// t^l Y_lm(s) is a polynomial of the scaled position (u, v, z) = (p - c_b) / r_b:
//   t^l Y_l,+-m(s) ~ Q_l^m(z, t^2) { Re, Im } (u + i v)^m,
//   Q_m = 1, Q_{m+1} = z, Q_l = z Q_{l-1} - beta_lm t^2 Q_{l-2},
//   beta_lm = ((l-1)^2 - m^2) / ((2l-1)(2l-3)),
// the monic form of the associated Legendre recurrence; its scale
// (2m-1)!! / ... sits with the Y_lm normalisation in kp (YlmTables::Kp),
// applied once per block to X_b and to the finished L* rows.  So a triple
// needs no angles, no division by sin(theta) and no branch at the poles; W is
// folded into the powers (u + i v)^m.
//
// Block per sphere b over its gather list.  A lane works on a slot: one
// triple in FP64, two triples in FP32, whose values sit in the two halves of
// 64-bit registers and whose arithmetic is the packed fma.rn.f32x2 (one
// issued instruction for two FP32 operations; the scalar FP32 form of this
// pass issued 758 instructions per triple and was bound by that).  Per chunk
// of NT slots (NT threads per block) every thread writes the fields (powers)
// of its slot to shared memory, then the role warps run over the chunk's
// slots; the geometry of the next chunk (cp.async), its xi values and the
// gather-list entries after it are in flight meanwhile.  A role (warp) owns
// some of the columns m; its L* rows stay in registers, and its share of a
// triple's lx value goes to shared memory, from where the shares are summed
// in role order into val[q] (gather-list order).  k_lx_gather sums the
// triples of each point.  No atomics: the results are bit-reproducible.
//
// Bound: the FMA / FP64 pipe (about 390 multiply-adds per triple at lmax 10
// and 40 for its fields), then latency at 16 warps per SM.  One fields
// buffer with two barriers per chunk and 16 warps beats two buffers with one
// barrier and 12 warps (FP32, lmax 10: 0.85 against 0.91 ms).  Measured per
// launch, against the angular form with scalar arithmetic that this replaces:
//   20,000 spheres, lmax 10, 590 points: FP32 1.07 -> 0.85, FP64 2.57 -> 1.52 ms
//    5,000 spheres, lmax 9, 434 points:  FP32 0.222 -> 0.158, FP64 0.468 -> 0.318 ms
//    5,000 spheres, lmax 8, 302 points:  FP32 0.145 -> 0.105, FP64 0.380 -> 0.169 ms
//    5,000 spheres, lmax 6, 302 points:  FP32 0.101 -> 0.076, FP64 0.194 -> 0.130 ms
// The FP32 operator's error against FP64 falls from 1.7e-6 to 1.3e-7 (the
// geometry is rounded once from FP64 and no angles are formed).
#include <climits>

#include "ddc_internal.h"

namespace ddc {
namespace {

__host__ __device__ constexpr int lmi(int l, int m) { return l * (l + 1) / 2 + m; }

// ---------------------------------------------------------------------------
// arithmetic of a slot: one FP64 value, or two FP32 values packed in 64 bits
// ---------------------------------------------------------------------------
// Loads that stay where they are written: issued ahead of the role work that
// hides their latency (the compiler would sink them to their first use).
// ld_list goes through the read-only path and is for the lists and other tables
// of the molecule; what the preceding kernel of a sweep writes (X, xi) is not
// read-only while this one is resident (chain_wait), so it takes ordinary loads
// and its pointers carry no __restrict__.
__device__ __forceinline__ int ld_list(const int* p) {
  int v;
  asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_here(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ double ld_here(const double* p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}

template <class Rl>
struct Slot;
template <>
struct Slot<double> {
  typedef double V;
  typedef double4 G4;
  static constexpr int N = 1;  // triples per slot
  static __device__ __forceinline__ V fma(V a, V b, V c) { return ::fma(a, b, c); }
  static __device__ __forceinline__ V mul(V a, V b) { return a * b; }
  static __device__ __forceinline__ V add(V a, V b) { return a + b; }
  static __device__ __forceinline__ V fmas(V a, double b, V c) { return ::fma(a, b, c); }
  static __device__ __forceinline__ V muls(V a, double b) { return a * b; }
  static __device__ __forceinline__ V dup(double a) { return a; }
  static __device__ __forceinline__ V pack(const double* a) { return a[0]; }
  static __device__ __forceinline__ void unpack(V v, double* a) { a[0] = v; }
};
template <>
struct Slot<float> {
  typedef unsigned long long V;
  typedef float4 G4;
  static constexpr int N = 2;
  static __device__ __forceinline__ V fma(V a, V b, V c) {
    V d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
  }
  static __device__ __forceinline__ V mul(V a, V b) {
    V d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
  }
  static __device__ __forceinline__ V add(V a, V b) {
    V d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
  }
  static __device__ __forceinline__ V pack2(float a, float b) {
    V d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
  }
  // with a scalar operand: one scalar operation on each half (as many FMA
  // pipe cycles as the packed form, without moving the scalar into a pair)
  static __device__ __forceinline__ V fmas(V a, float b, V c) {
    float x[2], y[2];
    unpack(a, x);
    unpack(c, y);
    return pack2(fmaf(x[0], b, y[0]), fmaf(x[1], b, y[1]));
  }
  static __device__ __forceinline__ V muls(V a, float b) {
    float x[2];
    unpack(a, x);
    return pack2(x[0] * b, x[1] * b);
  }
  static __device__ __forceinline__ V dup(float a) { return pack2(a, a); }
  static __device__ __forceinline__ V pack(const float* a) { return pack2(a[0], a[1]); }
  static __device__ __forceinline__ void unpack(V v, float* a) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a[0]), "=f"(a[1]) : "l"(v));
  }
};
template <class V>
struct __align__(16) V2 {
  V x, y;
};
// a shared-memory pair read where it is written (kept out of registers: the
// compiler would hoist the loads out of the loop over the slots)
__device__ __forceinline__ V2<double> ld_pair(const V2<double>* p) {
  V2<double> v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];"
               : "=d"(v.x), "=d"(v.y)
               : "r"((unsigned)__cvta_generic_to_shared(p)));
  return v;
}
__device__ __forceinline__ V2<unsigned long long> ld_pair(const V2<unsigned long long>* p) {
  V2<unsigned long long> v;
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];"
               : "=l"(v.x), "=l"(v.y)
               : "r"((unsigned)__cvta_generic_to_shared(p)));
  return v;
}

// ---------------------------------------------------------------------------
// roles: the lmax+1 columns are shared out so that the role with the most
// values (accumulator and X registers) has as few as possible, by a search
// over assignments in order of decreasing column size; a role runs its
// columns in increasing m and holds them in that order in its register arrays
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int col_vals(int L, int m) { return m == 0 ? L + 1 : 2 * (L + 1 - m); }
struct RoleMap {
  int role[DDC_MAX_LMAX + 1];
};
__host__ __device__ constexpr bool role_fit(int L, int NR, int cap, const int* order, int k,
                                            int* load, RoleMap& map) {
  if (k > L) return true;
  const int m = order[k], v = col_vals(L, m);
  for (int r = 0; r < NR; ++r) {
    if (load[r] + v > cap) continue;
    load[r] += v;
    map.role[m] = r;
    if (role_fit(L, NR, cap, order, k + 1, load, map)) return true;
    load[r] -= v;
    if (load[r] == 0) break;  // empty roles are alike
  }
  return false;
}
__host__ __device__ constexpr RoleMap role_map(int L, int NR) {
  int order[DDC_MAX_LMAX + 1] = {};
  bool used[DDC_MAX_LMAX + 1] = {};
  for (int k = 0; k <= L; ++k) {
    int best = -1;
    for (int c = 0; c <= L; ++c)
      if (!used[c] && (best < 0 || col_vals(L, c) > col_vals(L, best))) best = c;
    used[best] = true;
    order[k] = best;
  }
  RoleMap map{};
  for (int cap = ((L + 1) * (L + 1) + NR - 1) / NR;; ++cap) {
    int load[DDC_MAX_LMAX + 1] = {};
    if (role_fit(L, NR, cap, order, 0, load, map)) return map;
  }
}
template <int L, int NR>
struct Roles {
  static constexpr RoleMap map = role_map(L, NR);
};
template <int L, int NR>
__host__ __device__ constexpr int role_of(int m) {
  return Roles<L, NR>::map.role[m];
}
template <int L, int NR>
__host__ __device__ constexpr int off_of(int m) {
  int off = 0;
  for (int c = 0; c < m; ++c)
    if (role_of<L, NR>(c) == role_of<L, NR>(m)) off += col_vals(L, c);
  return off;
}
template <int L, int NR>
__host__ __device__ constexpr int role_vals(int r) {
  int n = 0;
  for (int c = 0; c <= L; ++c)
    if (role_of<L, NR>(c) == r) n += col_vals(L, c);
  return n;
}
template <int L, int NR>
__host__ __device__ constexpr int max_vals() {
  int mx = 0;
  for (int r = 0; r < NR; ++r) mx = role_vals<L, NR>(r) > mx ? role_vals<L, NR>(r) : mx;
  return mx;
}
// Roles per degree: blocks of at most four warps, so that a warp scheduler
// runs one role's code (more roles, with one scheduler alternating between
// two of them, were slower: six / eight roles 1.08 / 1.49 ms per FP32 launch
// at 20,000 spheres and lmax 10 against 0.91 ms for four, X in registers),
// and few enough values per role for 128 registers a thread.
template <class Rl>
__host__ __device__ constexpr int nroles(int L) {
  return L >= 7 ? 4 : L >= 5 ? (sizeof(Rl) == 8 ? 3 : 2) : L >= 3 && sizeof(Rl) == 8 ? 2 : 1;
}
// blocks per SM for 128 registers a thread: 16 warps
template <class Rl>
__host__ __device__ constexpr int min_blocks(int L) {
  return 16 / nroles<Rl>(L);
}
// A role's columns of X_b: held in registers by the FP64 roles up to lmax 8,
// else read from shared memory at every use (one broadcast load per (l, m)).
// At 128 registers both do not fit: at lmax 10 the FP32 pass takes 0.85 ms
// with X in shared memory and 16 warps per SM, 0.91 ms with X in registers
// and 12 warps; FP64 at lmax 8 0.169 ms with X in registers, 0.191 ms not
// (5,000 spheres, 302 points).
template <class Rl>
__host__ __device__ constexpr bool x_in_regs(int L) {
  return sizeof(Rl) == 8 && L <= 8;
}

__host__ __device__ constexpr double beta_lm(int l, int m) {
  return (double)((l - 1) * (l - 1) - m * m) / (double)((2 * l - 1) * (2 * l - 3));
}

// ---------------------------------------------------------------------------
// shared fields of a chunk of NT slots, 16-byte pairs of slot values:
// [0] (z, t^2), [1] (c = w_n xi_a(n), W), [1 + m] Re and Im of W (u + i v)^m
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int nfields(int L) { return 2 + L; }

// One column of a slot: its L* rows take Q c {Re, Im}, its part of the lx
// value is returned added to part.
template <int LMAX, int M, class Rl, int MODE>
__device__ __forceinline__ typename Slot<Rl>::V lxs_column(
    typename Slot<Rl>::V z, typename Slot<Rl>::V t2, typename Slot<Rl>::V c,
    typename Slot<Rl>::V re, typename Slot<Rl>::V im, typename Slot<Rl>::V* acc,
    const V2<typename Slot<Rl>::V>* xs, typename Slot<Rl>::V part, bool first) {
  typedef Slot<Rl> S;
  typedef typename S::V V;
  constexpr int NM = LMAX + 1 - M;
  constexpr bool DOX = MODE != 2, DOS = MODE != 1;
  V q0{}, q1{}, dc{}, ds{}, rc{}, ic{};
  if (DOS) {
    rc = S::mul(re, c);
    if (M > 0) ic = S::mul(im, c);
  }
#pragma unroll
  for (int k = 0; k < NM; ++k) {
    if (k == 0) {  // Q = 1
      if (DOS) {
        acc[0] = S::add(acc[0], rc);
        if (M > 0) acc[NM] = S::add(acc[NM], ic);
      }
      if (DOX) {
        const V2<V> x = x_in_regs<Rl>(LMAX) ? xs[lmi(M, M)] : ld_pair(xs + lmi(M, M));
        dc = x.x;
        ds = x.y;
      }
      continue;
    }
    V Q;
    if (k == 1) {
      Q = z;
    } else {
      const V nb = S::muls(t2, (Rl)-beta_lm(M + k, M));
      Q = k == 2 ? S::fma(z, z, nb) : S::fma(z, q1, S::mul(nb, q0));
    }
    q0 = q1;
    q1 = Q;
    if (DOS) {
      acc[k] = S::fma(Q, rc, acc[k]);
      if (M > 0) acc[NM + k] = S::fma(Q, ic, acc[NM + k]);
    }
    if (DOX) {
      const V2<V> x = x_in_regs<Rl>(LMAX) ? xs[lmi(M + k, M)] : ld_pair(xs + lmi(M + k, M));
      dc = S::fma(Q, x.x, dc);
      if (M > 0) ds = S::fma(Q, x.y, ds);
    }
  }
  if (!DOX) return part;
  part = first ? S::mul(re, dc) : S::fma(re, dc, part);
  if (M > 0) part = S::fma(im, ds, part);
  return part;
}

template <int LMAX, int NR, int R, int M, class Rl, int MODE>
__device__ __forceinline__ void lxs_cols(const V2<typename Slot<Rl>::V>* fld, int j,
                                         typename Slot<Rl>::V z, typename Slot<Rl>::V t2,
                                         typename Slot<Rl>::V c, typename Slot<Rl>::V* acc,
                                         const V2<typename Slot<Rl>::V>* xs,
                                         typename Slot<Rl>::V& part, bool first) {
  constexpr int NT = 32 * NR;
  if constexpr (role_of<LMAX, NR>(M) == R) {
    constexpr int OFF = off_of<LMAX, NR>(M);
    if constexpr (M == 0) {
      const typename Slot<Rl>::V W = fld[NT + j].y;
      part = lxs_column<LMAX, 0, Rl, MODE>(z, t2, c, W, W, acc + OFF, xs, part, first);
    } else {
      const V2<typename Slot<Rl>::V> p = fld[(1 + M) * NT + j];
      part = lxs_column<LMAX, M, Rl, MODE>(z, t2, c, p.x, p.y, acc + OFF, xs, part, first);
    }
    first = false;
  }
  if constexpr (M < LMAX)
    lxs_cols<LMAX, NR, R, M + 1, Rl, MODE>(fld, j, z, t2, c, acc, xs, part, first);
}

// role R over the chunk's slots: lanes take slots j < count
template <int LMAX, int NR, int R, class Rl, int MODE>
__device__ __forceinline__ void lxs_run_role(int role, const V2<typename Slot<Rl>::V>* fld,
                                             int count, int lane, typename Slot<Rl>::V* acc,
                                             const V2<typename Slot<Rl>::V>* xs,
                                             typename Slot<Rl>::V* lxp) {
  constexpr int NT = 32 * NR;
  typedef typename Slot<Rl>::V V;
  if (role == R) {
    for (int j = lane; j < count; j += 32) {
      const V2<V> zt = fld[j];
      V c{};
      if (MODE != 1) c = fld[NT + j].x;
      V part{};
      lxs_cols<LMAX, NR, R, 0, Rl, MODE>(fld, j, zt.x, zt.y, c, acc, xs, part, true);
      if (MODE != 2) lxp[R * NT + j] = part;
    }
    return;
  }
  if constexpr (R + 1 < NR)
    lxs_run_role<LMAX, NR, R + 1, Rl, MODE>(role, fld, count, lane, acc, xs, lxp);
}

// the finished L* rows of role R: the halves of a slot, then the lanes by a
// fixed shuffle tree
template <int LMAX, int NR, int R, int M, class Rl>
__device__ __forceinline__ void lxs_store_cols(const LxsTab& tb, const Rl* acc, double* yb) {
  if constexpr (role_of<LMAX, NR>(M) == R) {
    constexpr int OFF = off_of<LMAX, NR>(M), NM = LMAX + 1 - M;
#pragma unroll
    for (int k = 0; k < NM; ++k) {
      const int l = M + k, ind = l * l + l;
      const double s = -tb.kp[lmi(l, M)];
      yb[ind + M] = s * (double)acc[OFF + k];
      if (M > 0) yb[ind - M] = s * (double)acc[OFF + NM + k];
    }
  }
  if constexpr (M < LMAX) lxs_store_cols<LMAX, NR, R, M + 1, Rl>(tb, acc, yb);
}
template <int LMAX, int NR, int R, class Rl>
__device__ __forceinline__ void lxs_finish_role(int role, const LxsTab& tb,
                                                const typename Slot<Rl>::V* acc, double* yb,
                                                int lane) {
  if (role == R) {
    constexpr int NV = role_vals<LMAX, NR>(R);
    Rl sum[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      Rl a[Slot<Rl>::N];
      Slot<Rl>::unpack(acc[v], a);
      sum[v] = Slot<Rl>::N == 2 ? a[0] + a[Slot<Rl>::N - 1] : a[0];
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) sum[v] += __shfl_xor_sync(0xffffffffu, sum[v], o);
    }
    if (lane == 0) lxs_store_cols<LMAX, NR, R, 0, Rl>(tb, sum, yb);
    return;
  }
  if constexpr (R + 1 < NR) lxs_finish_role<LMAX, NR, R + 1, Rl>(role, tb, acc, yb, lane);
}

// ---------------------------------------------------------------------------
// geometry of one triple in FP64: (u, v, z) and W = chi(t) / f_a(n)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double4 lxs_geom(const LxsTab& tb, double4 ca, double4 gn, double f,
                                            double4 cb, double irb) {
  const double eta = tb.eta;
  const double fa = 15.0 * eta - 12.0, fb = 10.0 * eta * eta - 15.0 * eta + 6.0;
  double4 o;
  o.x = (fma(ca.w, gn.x, ca.x) - cb.x) * irb;
  o.y = (fma(ca.w, gn.y, ca.y) - cb.y) * irb;
  o.z = (fma(ca.w, gn.z, ca.z) - cb.z) * irb;
  const double t = sqrt(fma(o.x, o.x, fma(o.y, o.y, o.z * o.z)));
  double chi;
  if (t >= 1.0) chi = 0.0;
  else if (t <= 1.0 - eta) chi = 1.0;
  else {
    const double xm = t - 1.0;
    chi = (xm * xm * (1.0 - t)) * ((6.0 * t + fa) * t + fb) * tb.ie5;
  }
  o.w = f > 1.0 ? chi / f : chi;
  return o;
}
__device__ __forceinline__ void set4(float4& d, const double4& s) {
  d = make_float4((float)s.x, (float)s.y, (float)s.z, (float)s.w);
}
__device__ __forceinline__ void set4(double4& d, const double4& s) { d = s; }

// the geometry of every triple, once per molecule: block per sphere b
template <class Rl>
__global__ void __launch_bounds__(128) k_lxs_geo(const LxsTab tb, const DevGeo g,
                                                 typename Slot<Rl>::G4* tg) {
  const int b = blockIdx.x;
  const double4 cb = g.sph[b];
  const double irb = 1.0 / cb.w;
  const int q0 = g.ls_ptr[b], n1 = g.ls_ptr[b + 1] - q0;
  for (int k = threadIdx.x; k < n1; k += blockDim.x) {
    const int q = q0 + k;
    const int pa = g.ls[q], a = pa / g.ngrid, n = pa - a * g.ngrid;
    set4(tg[q], lxs_geom(tb, g.sph[a], g.grid[n], g.fi[pa], cb, irb));
  }
}

__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int LMAX, class Rl>
constexpr size_t lxs_smem(bool pre) {
  constexpr int NR = nroles<Rl>(LMAX), NT = 32 * NR;
  return (size_t)NT * (16 * nfields(LMAX) + 8 * NR) +
         (pre ? (size_t)NT * Slot<Rl>::N * sizeof(typename Slot<Rl>::G4) : 0) +
         16 * (LMAX + 1) * (LMAX + 2) / 2;
}

// MODE 0: val = lx values and y = L* xi; 1: lx values only; 2: L* only.
// PRE: the geometry comes from tg (built by k_lxs_geo), else it is evaluated
// per pass (the few FP64 passes of the mixed path).
template <int LMAX, class Rl, bool PRE, int MODE>
__device__ __forceinline__ void lxs_block(const LxsTab& tb, const DevGeo& g,
                                          const typename Slot<Rl>::G4* __restrict__ tg,
                                          const double* X, const Rl* xi, Rl* val, double* y) {
  typedef Slot<Rl> S;
  typedef typename S::V V;
  typedef typename S::G4 G4;
  constexpr int NR = nroles<Rl>(LMAX), NT = 32 * NR, NP = S::N;
  constexpr int NF = nfields(LMAX), NY = (LMAX + 1) * (LMAX + 1);
  constexpr int NVM = max_vals<LMAX, NR>();
  extern __shared__ __align__(16) unsigned char smraw[];
  V2<V>* fld = reinterpret_cast<V2<V>*>(smraw);         // [NF][NT]
  V2<V>* xs = fld + NF * NT;                             // [(l, m)]
  G4* gs = reinterpret_cast<G4*>(xs + lmi(LMAX + 1, 0)); // [NP][NT] (PRE)
  V* lxp = reinterpret_cast<V*>(gs + (PRE ? NP * NT : 0));  // [NR][NT]
  const int b = g.ls_order ? g.ls_order[blockIdx.x] : (int)blockIdx.x, tid = threadIdx.x;
  if (sweep_skip(g.act, b)) return;
  const int role = tid >> 5, lane = tid & 31;
  const int q0 = g.ls_ptr[b], q1 = g.ls_ptr[b + 1];
  constexpr int CH = NT * NP;
  const int nch = (q1 - q0 + CH - 1) / CH;
  // slots of chunk k: NT, fewer (packed: whole warps) in the last; slot j
  // holds the triples c0 + j and, packed, c0 + j + slots.  Threads without a
  // triple read the list's last one and give it the weight zero.
  const int left = q1 - q0 - (nch - 1) * CH;
  const int hlast = NP == 1 ? left : min(NT, ((left + 1) / 2 + 31) & ~31);
  auto slots = [&](int k) { return k == nch - 1 ? hlast : NT; };
  auto entry = [&](int k, int p) { return k * CH + tid + p * slots(k); };
  auto triple = [&](int k, int p) { return list_entry(q0, q1, entry(k, p)); };
  auto mine = [&](int k, int p) { return tid < slots(k) && entry(k, p) < q1 - q0; };
  auto geo_copy = [&](int k) {  // chunk k's geometry into this thread's slots of gs
    if (PRE && k < nch) {
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const G4* src = tg + triple(k, p);
        G4* d = gs + p * NT + tid;
        cp_async16(d, src);
        if (sizeof(G4) == 32)
          cp_async16(reinterpret_cast<char*>(d) + 16, reinterpret_cast<const char*>(src) + 16);
      }
    }
  };
  // gather-list entries (a, n) of this thread's triples of chunk k
  auto points = [&](int k, int* pa) {
    if (k < nch) {
#pragma unroll
      for (int p = 0; p < NP; ++p) pa[p] = ld_list(g.ls + triple(k, p));
    }
  };
  struct In {
    Rl c[NP];
    double4 ca, gn;  // on-the-fly geometry (one triple per slot)
    double f;
  };
  auto load = [&](const int* pa, In& in) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      if (MODE != 1) in.c[p] = ld_here(xi + pa[p]);
      if constexpr (!PRE) {
        const int a = pa[p] / g.ngrid;
        in.ca = g.sph[a];
        in.gn = g.grid[pa[p] - a * g.ngrid];
        in.f = g.fi[pa[p]];
      }
    }
  };
  const double4 cb = g.sph[b];
  const double irb = 1.0 / cb.w;
  // the fields of this thread's slot of chunk k
  auto fields = [&](int k, const In& in) {
    V2<V>* f = fld + tid;
    Rl gu[NP], gv[NP], gz[NP], gw[NP], gc[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      G4 v;
      if constexpr (PRE) v = gs[p * NT + tid];
      else set4(v, lxs_geom(tb, in.ca, in.gn, in.f, cb, irb));
      gu[p] = v.x;
      gv[p] = v.y;
      gz[p] = v.z;
      gw[p] = v.w;
      gc[p] = MODE != 1 ? in.c[p] : Rl(0);
      if (k == nch - 1 && !mine(k, p)) gw[p] = gc[p] = Rl(0);
    }
    const V u = S::pack(gu), v = S::pack(gv), z = S::pack(gz), W = S::pack(gw);
    const V nv = S::mul(v, S::dup(Rl(-1)));
    f[0] = V2<V>{z, S::fma(u, u, S::fma(v, v, S::mul(z, z)))};
    f[NT] = V2<V>{S::pack(gc), W};
    V re = S::mul(W, u), im = S::mul(W, v);
#pragma unroll
    for (int m = 1; m <= LMAX; ++m) {
      f[(1 + m) * NT] = V2<V>{re, im};
      const V rn = S::fma(re, u, S::mul(im, nv));
      im = S::fma(re, v, S::mul(im, u));
      re = rn;
    }
  };
  auto values = [&](int k) {  // lx values of chunk k: the roles' shares in role order
    if (MODE == 2) return;
    const V* lp = lxp + tid;
    V sv = lp[0];
#pragma unroll
    for (int r = 1; r < NR; ++r) sv = S::add(sv, lp[r * NT]);
    Rl o[NP];
    S::unpack(sv, o);
#pragma unroll
    for (int p = 0; p < NP; ++p)
      if (k < nch - 1 || mine(k, p)) val[q0 + entry(k, p)] = o[p];
  };
  geo_copy(0);
  int pa[NP] = {};
  In in;
  points(0, pa);
  if (MODE != 2)
    for (int e = tid; e < lmi(LMAX + 1, 0); e += NT) {
      int l = 0;
      while (lmi(l + 1, 0) <= e) ++l;
      const int m = e - lmi(l, 0), ind = l * l + l;
      const double* xb = X + (size_t)b * NY + ind;
      xs[e] = V2<V>{S::dup((Rl)(tb.kp[e] * xb[m])), S::dup((Rl)(tb.kp[e] * xb[-m]))};
    }
  if (nch > 0) load(pa, in);
  points(1, pa);
  V acc[NVM];
#pragma unroll
  for (int v = 0; v < NVM; ++v) acc[v] = S::dup(Rl(0));
  for (int k = 0; k < nch; ++k) {
    cp_async_wait_all();
    fields(k, in);
    __syncthreads();
    // in flight while the roles work: the geometry and xi of chunk k+1 and
    // the gather-list entries of chunk k+2
    geo_copy(k + 1);
    if (k + 1 < nch) load(pa, in);
    points(k + 2, pa);
    lxs_run_role<LMAX, NR, 0, Rl, MODE>(role, fld, slots(k), lane, acc, xs, lxp);
    __syncthreads();
    values(k);
  }
  if (MODE != 1) lxs_finish_role<LMAX, NR, 0, Rl>(role, tb, acc, y + (size_t)b * NY, lane);
}

// MODE 3: lx and L* by blocks of their own (grid y)
template <int LMAX, class Rl, bool PRE, int MODE>
__global__ void __launch_bounds__(32 * nroles<Rl>(LMAX), min_blocks<Rl>(LMAX))
    k_lxs(const __grid_constant__ LxsTab tb, const DevGeo g,
          const typename Slot<Rl>::G4* __restrict__ tg, const double* X, const Rl* xi, Rl* val,
          double* y) {
  chain_wait();
  if constexpr (MODE < 3) {
    lxs_block<LMAX, Rl, PRE, MODE>(tb, g, tg, X, xi, val, y);
  } else if (blockIdx.y == 0) {
    lxs_block<LMAX, Rl, PRE, 1>(tb, g, tg, X, xi, val, y);
  } else {
    lxs_block<LMAX, Rl, PRE, 2>(tb, g, tg, X, xi, val, y);
  }
}

LxsTab lxs_tab(const YlmTables& tb) {
  LxsTab t;
  for (int e = 0; e < DDC_NLM_CAP; ++e) t.kp[e] = tb.Kp[e];
  t.eta = tb.eta;
  t.ie5 = 1.0 / (tb.eta * tb.eta * tb.eta * tb.eta * tb.eta);
  return t;
}

#define DDC_LMAX_CASES(X) \
  X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12)

template <class Rl, bool PRE, int MODE>
cudaError_t lxs_launch(Launch L, const YlmTables& tb, const DevGeo& g,
                       const typename Slot<Rl>::G4* tg, const double* X, const Rl* xi, Rl* val,
                       double* y) {
  if (g.nsph == 0) return cudaSuccess;
  const LxsTab t = lxs_tab(tb);
  cudaError_t e = cudaSuccess;
#define CASE(LV)                                                                               \
  case LV: {                                                                                   \
    e = launch_chained(k_lxs<LV, Rl, PRE, MODE>, dim3(g.nsph, MODE == 3 ? 2 : 1),              \
                       32 * nroles<Rl>(LV),                                                    \
                       lxs_smem<LV, Rl>(PRE), L.st, t, g, tg, X, xi, val, y);                  \
    break;                                                                                     \
  }
  switch (tb.lmax) {
    DDC_LMAX_CASES(CASE)
    default:
      return cudaErrorInvalidValue;
  }
#undef CASE
  ++*L.launches;
  return e ? e : cudaGetLastError();
}
template <int LV, class Rl, bool PRE, int MODE>
cudaError_t lxs_attributes() {
  constexpr size_t sm = lxs_smem<LV, Rl>(PRE);
  auto kfn = k_lxs<LV, Rl, PRE, MODE>;
  cudaError_t e = cudaSuccess;
  if (sm > 48 * 1024)
    e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  return e ? e : cudaFuncSetAttribute(kfn, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
}
template <int LV, int MODE>
cudaError_t lxs_attributes_mode() {
  cudaError_t e = lxs_attributes<LV, double, true, MODE>();
  if (!e) e = lxs_attributes<LV, double, false, MODE>();
  return e ? e : lxs_attributes<LV, float, true, MODE>();
}
// FP64: with the stored geometry when there is one
template <int MODE>
cudaError_t lxs_launch64(Launch L, const YlmTables& tb, const DevGeo& g, const double* X,
                         const double* xi, double* val, double* y) {
  return g.tgeo4d ? lxs_launch<double, true, MODE>(L, tb, g, g.tgeo4d, X, xi, val, y)
                  : lxs_launch<double, false, MODE>(L, tb, g, nullptr, X, xi, val, y);
}

// Few spheres: the two operators by blocks of their own, which takes both
// halves' latency side by side; with more the shared geometry and powers are worth
// more.  us of a call of lx and lstarx on device vectors (some 25 of them the call and
// the other kernels), by one pass / by halves:
//   lmax 10, 302 points, FP64   12 spheres 41.8 / 38.0, 60 54.5 / 47.3, 200 63.8 / 62.8,
//                               296 68.2 / 69.2, 450 77.3 / 77.3, 900 100 / 108
//   lmax 10, mixed              60 44.8 / 42.1, 200 49.6 / 50.3, 450 59.1 / 58.2, 900 71.7 / 77.5
//   lmax 8, 302 points, FP64    60 49.4 / 45.2, 200 53.7 / 51.5, 296 55.5 / 61.4, 900 79.7 / 86.4
//   lmax 6, 302 points, mixed   60 43.0 / 40.3, 296 46.5 / 46.6, 900 54.2 / 59.9
//   lmax 6, 110 points, FP64    113 39.5 / 35.7, 296 38.7 / 38.4, 450 38.7 / 43.5
// and ms of energy and forces, lmax 10, FP64: 60 spheres 2.09 / 1.93, 296 3.73 / 3.62,
// 600 4.86 / 4.97, 900 7.12 / 7.46.
bool split_pass(const DevGeo& g) { return g.nsph <= 2 * 148; }

}  // namespace

cudaError_t prepare_lxs(int lmax) {
  cudaError_t e = cudaErrorInvalidValue;
#define CASE(LV)                                       \
  case LV:                                             \
    e = lxs_attributes_mode<LV, 0>();                  \
    if (!e) e = lxs_attributes_mode<LV, 1>();          \
    if (!e) e = lxs_attributes_mode<LV, 2>();          \
    if (!e) e = lxs_attributes_mode<LV, 3>();          \
    break;
  switch (lmax) { DDC_LMAX_CASES(CASE) }
#undef CASE
  return e;
}
cudaError_t launch_lxs(Launch L, const YlmTables& tb, const DevGeo& g, const double* X,
                       const double* xi, double* val, double* y) {
  return split_pass(g) ? lxs_launch64<3>(L, tb, g, X, xi, val, y)
                       : lxs_launch64<0>(L, tb, g, X, xi, val, y);
}
cudaError_t launch_lx_vals(Launch L, const YlmTables& tb, const DevGeo& g, const double* X,
                           double* val) {
  return lxs_launch64<1>(L, tb, g, X, nullptr, val, nullptr);
}
cudaError_t launch_lstarx_acc(Launch L, const YlmTables& tb, const DevGeo& g, const double* xi,
                              double* y) {
  return lxs_launch64<2>(L, tb, g, nullptr, xi, nullptr, y);
}
cudaError_t launch_lxs_f32(Launch L, const YlmTables& tb, const DevGeo& g, const double* X,
                           const float* xi, float* val, double* y) {
  return split_pass(g) ? lxs_launch<float, true, 3>(L, tb, g, g.tgeo4, X, xi, val, y)
                       : lxs_launch<float, true, 0>(L, tb, g, g.tgeo4, X, xi, val, y);
}
cudaError_t launch_lx_vals_f32(Launch L, const YlmTables& tb, const DevGeo& g, const double* X,
                               float* val) {
  return lxs_launch<float, true, 1>(L, tb, g, g.tgeo4, X, nullptr, val, nullptr);
}
cudaError_t launch_lstarx_acc_f32(Launch L, const YlmTables& tb, const DevGeo& g,
                                  const float* xi, double* y) {
  return lxs_launch<float, true, 2>(L, tb, g, g.tgeo4, nullptr, xi, nullptr, y);
}
cudaError_t launch_lxs_geo(Launch L, const YlmTables& tb, const DevGeo& g, float4* tg) {
  if (g.nsph == 0) return cudaSuccess;
  k_lxs_geo<float><<<g.nsph, 128, 0, L.st>>>(lxs_tab(tb), g, tg);
  ++*L.launches;
  return cudaGetLastError();
}
cudaError_t launch_lxs_geo_f64(Launch L, const YlmTables& tb, const DevGeo& g, double4* tg) {
  if (g.nsph == 0) return cudaSuccess;
  k_lxs_geo<double><<<g.nsph, 128, 0, L.st>>>(lxs_tab(tb), g, tg);
  ++*L.launches;
  return cudaGetLastError();
}

}  // namespace ddc
