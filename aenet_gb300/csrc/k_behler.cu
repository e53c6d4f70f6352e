// Behler-Parrinello symmetry functions G1-G5 and their adjoint (replaces
// sf_fingerprint and the G*_update routines of src/ext/symmfunc.f90:311-811).
//
// One warp per central atom.  The neighbours are first staged in shared
// memory grouped by species (buckets), so that every radial list
// (functions of the central species for one neighbour species) and every
// angular list (one unordered pair of neighbour species) sees neighbours,
// or neighbour pairs, of a single kind:
//   radial  : lanes over the neighbours of a bucket, the list's functions
//             accumulated in registers (chunks of 16), warp reduction;
//   angular : the pairs of a bucket or of two buckets, offset by offset,
//             compacted through a queue so that 32 live pairs are evaluated
//             at a time (run_pairs).
// Angular lists that form a product grid (one kind and Rc, lambda = +-1,
// every (lambda, zeta) x eta combination; BehlerGrid) are evaluated per
// pair with one exponential per eta and one power per (lambda, zeta), the
// functions being their products; the factors of one neighbour alone,
// exp(-eta r^2) fc(r), are staged with it.  Other lists go function by
// function.
//
// What bounds them: instruction issue in FP32 and the FP64 pipe (two lanes
// per clock and SM, 75-80 % busy) in FP64; the neighbour rows fit L2.
// Measured on rutile Ti/O with 64 functions, before (an exponential of the
// whole sum per eta and pair, sin/cos of r_jk, shared-memory atomics in the
// adjoint) and now: 9,000 atoms mixed, forward 324 -> 238 us, adjoint 717 ->
// 429 us; 763 atoms FP64, forward 1160 -> 487 us, adjoint 1733 -> 889 us.
// The tables come from build_behler (capi.cpp): they already encode the
// reference's indexing (functions registered under the global species
// index, evaluated with the central atom's local one) and the feature
// index of every function.
//
// Functions (symmfunc.f90:445-838, PI truncated as there):
//   fc(r)  = 0.5 (cos(pi r/Rc) + 1)                 r < Rc, else 0
//   G1     = fc(r_ij)
//   G2     = exp(-eta (r_ij - Rs)^2) fc(r_ij)
//   G3     = cos(kappa r_ij) fc(r_ij)
//   G4     = 2 [(1 + lambda cos)/2]^zeta e^{-eta(r_ij^2 + r_ik^2 + r_jk^2)} fc_ij fc_ik fc_jk
//   G5     = 2 [(1 + lambda cos)/2]^zeta e^{-eta(r_ij^2 + r_ik^2)} fc_ij fc_ik
// (the factor 2 accounts for k < j, symmfunc.f90:724), cos clamped to
// [-1, 1] (symmfunc.f90:409-411).
//
// Adjoint: one-sided -- each pair (j, k) once, its gradient with respect to
// both neighbours added to per-neighbour accumulators in shared memory;
// the central atom's force and the virial follow from those sums.
#include <cmath>

#include "common.h"
#include "cutoff64.cuh"
#include "exp64.cuh"

namespace {

constexpr double SF_PI = 3.14159265358979;   // symmfunc.f90:38
constexpr int FCH = 16;                      // functions per register chunk
// resident one-warp blocks per SM asked of the register allocator (FP32);
// 9,000 rutile atoms: forward 243 us at 24, 270 at 20, 251 at 28; adjoint
// 431 us at 16, 464 at 20, 440 at 24
constexpr int FWD_BLOCKS = 24, ADJ_BLOCKS = 16;

template <typename T>
struct V4;
template <>
struct V4<float> {
  using type = float4;
};
template <>
struct V4<double> {
  using type = double4_32a;
};

__device__ __forceinline__ void sincos_t(float x, float* s, float* c) { __sincosf(x, s, c); }
__device__ __forceinline__ void sincos_t(double x, double* s, double* c) { sincos(x, s, c); }
__device__ __forceinline__ float exp_t(float x) { return __expf(x); }
__device__ __forceinline__ double exp_t(double x) { return exp(x); }
__device__ __forceinline__ float pow_t(float a, float b) { return powf(a, b); }
__device__ __forceinline__ double pow_t(double a, double b) { return pow(a, b); }

template <typename T>
struct Fn {
  T Rc, p1, p2, p3;
  int kind, out, izeta;
};

__device__ __forceinline__ Fn<float> load_fn_f(const BehlerFn* f) {
  Fn<float> r;
  r.Rc = f->fRc;
  r.p1 = f->fp1;
  r.p2 = f->fp2;
  r.p3 = f->fp3;
  r.kind = f->kind;
  r.out = f->out;
  r.izeta = f->izeta;
  return r;
}
__device__ __forceinline__ Fn<double> load_fn_d(const BehlerFn* f) {
  Fn<double> r;
  r.Rc = f->Rc;
  r.p1 = f->p1;
  r.p2 = f->p2;
  r.p3 = f->p3;
  r.kind = f->kind;
  r.out = f->out;
  r.izeta = f->izeta;
  return r;
}
template <typename T>
__device__ __forceinline__ Fn<T> load_fn(const BehlerFn* f);
template <>
__device__ __forceinline__ Fn<float> load_fn<float>(const BehlerFn* f) { return load_fn_f(f); }
template <>
__device__ __forceinline__ Fn<double> load_fn<double>(const BehlerFn* f) { return load_fn_d(f); }

// sf_cut (symmfunc.f90:823-838)
template <typename T>
__device__ __forceinline__ void cutfn(T r, T Rc, T& fc, T& dfc) {
  if (r >= Rc) {
    fc = T(0);
    dfc = T(0);
    return;
  }
  const T a = T(SF_PI) / Rc;
  T s, c;
  sincos_t(a * r, &s, &c);
  fc = T(0.5) * (c + T(1));
  dfc = T(-0.5) * a * s;
}

// a^n for a small non-negative integer n (binary exponentiation)
template <typename T>
__device__ __forceinline__ T ipow(T a, int n) {
  T r = T(1);
  while (n) {
    if (n & 1) r *= a;
    a *= a;
    n >>= 1;
  }
  return r;
}

// radial value and d/dr (sf_G1_ij, sf_G2_ij, sf_G3_ij)
// A: the staged (dfc, fc, 1/r), used when the function's cut-off is theirs
template <typename T>
__device__ __forceinline__ void radial_fn(const Fn<T>& f, T r, bool cached,
                                          const typename V4<T>::type& A, T& v, T& dv) {
  T fc = A.y, dfc = A.x;
  if (!cached) cutfn(r, f.Rc, fc, dfc);
  if (f.kind == 2) {
    const T a = r - f.p1;
    const T e = exp_t(-f.p2 * a * a);
    v = e * fc;
    dv = e * (dfc - T(2) * f.p2 * a * fc);
  } else if (f.kind == 3) {
    T s, c;
    sincos_t(f.p1 * r, &s, &c);
    v = c * fc;
    dv = c * dfc - f.p1 * s * fc;
  } else {
    v = fc;
    dv = dfc;
  }
}

// F1 = ((1 + lambda cos)/2)^zeta and dF1/dcos (sf_F1_ijk)
template <typename T>
__device__ __forceinline__ void f1(const Fn<T>& f, T cosv, T& F, T& dF) {
  const T a = T(0.5) * (T(1) + f.p1 * cosv);
  T pz, pz1;
  if (f.izeta > 0) {
    pz1 = ipow(a, f.izeta - 1);
    pz = pz1 * a;
  } else {
    pz = pow_t(a, f.p2);
    pz1 = pow_t(a, f.p2 - T(1));
  }
  F = pz;
  dF = T(0.5) * f.p2 * f.p1 * pz1;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

__device__ __forceinline__ double normalise(double g, const PotDevice& pd, size_t k) {
  return (g - pd.shift[k]) * pd.scale[k];
}
__device__ __forceinline__ float normalise(float g, const PotDevice& pd, size_t k) {
  const float2 sh = pd.shift2[k];
  return ((g - sh.x) - sh.y) * pd.scale32[k];
}

// Stage the neighbours inside rc into shared memory grouped by species.
// bstart[s] .. bstart[s+1] is bucket s; returns the number staged.  sA
// (optional) receives dfc(r), fc(r) (cut-off rc) and 1/r.
template <typename T>
__device__ int stage_buckets(const typename V4<T>::type* __restrict__ vec,
                             const int* __restrict__ jt, int n, int nt, T rc,
                             typename V4<T>::type* sR, typename V4<T>::type* sA, int* sslot,
                             int* bstart, int lane) {
  using T4 = typename V4<T>::type;
  int cnt = 0;
  for (int s = 0; s < nt; ++s) {
    bstart[s] = cnt;
    for (int base = 0; base < n; base += 32) {
      const int j = base + lane;
      bool in = false;
      T4 v;
      if (j < n) {
        v = vec[j];
        in = ((jt[j] >> AE_TYPE_SHIFT) == s) && v.w < rc && v.w > T(1e-8);
      }
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (in) {
        const int k = cnt + __popc(m & ((1u << lane) - 1u));
        sR[k] = v;
        sslot[k] = j;
        if (sA) {
          T4 a;
          a.z = T(1) / v.w;
          cutfn(v.w, rc, a.y, a.x);
          a.w = T(0);
          sA[k] = a;
        }
      }
      cnt += __popc(m);
    }
  }
  bstart[nt] = cnt;
  __syncwarp();
  return cnt;
}

template <typename T>
__device__ __forceinline__ const BehlerTable* table_of(const PotDevice& pd, int t) {
  return reinterpret_cast<const BehlerTable*>(pd.behler_blob + pd.sp[t].behler_off);
}
__device__ __forceinline__ const BehlerGrid* grids_of(const BehlerTable* tab) {
  return reinterpret_cast<const BehlerGrid*>(reinterpret_cast<const unsigned char*>(tab) +
                                             tab->grid_off);
}

// ---- pairs of staged neighbours, walked by the offset q between the row r
// of one bucket and its partner:
//   unordered pairs of one bucket of m : (r, (r + q) mod m), q = 1 .. m/2
//     (q = m/2 from the lower half only when m is even)
//   pairs of two buckets (mr >= mc)    : (r, (r + q) mod mc), q = 0 .. mc - 1
// so that every pair occurs once and the rows of one offset have distinct
// partners (in runs of mc rows).  Such a run is a pair's key.
//
// G4 pairs with r_jk >= Rc contribute nothing (fc(r_jk) = 0): an FP32 test
// drops them (with a margin when the pair itself is evaluated in FP64, which
// then decides), and the survivors go through a per-warp queue in shared
// memory, so that the body runs on 32 live pairs instead of the ~45 % that
// the loop leaves.  A queue entry carries its key: pairs with the same key
// touch distinct rows and distinct partners, which lets the adjoint add to
// the neighbours' accumulators without atomics.
struct PairList {
  int r0, mr, c0, mc;   // rows and partners (bucket start and size)
  int rs, cs;           // their buckets
  bool tri;
};

__device__ __forceinline__ PairList pair_list(const int* bstart, int a, int c) {
  PairList L;
  L.tri = a == c;
  const int na = bstart[a + 1] - bstart[a], nc = bstart[c + 1] - bstart[c];
  const int rows = na >= nc ? a : c, part = na >= nc ? c : a;
  L.rs = rows;
  L.cs = part;
  L.r0 = bstart[rows];
  L.mr = bstart[rows + 1] - bstart[rows];
  L.c0 = bstart[part];
  L.mc = bstart[part + 1] - bstart[part];
  return L;
}
__device__ __forceinline__ bool empty(const PairList& L) {
  return L.tri ? L.mr < 2 : L.mr < 1 || L.mc < 1;
}

// body(live, j, k, key): called by the whole warp; lanes without a pair get
// live = false and the indices of some staged pair.  The rows are cut into
// blocks of equal width, so that no block leaves steps of a few lanes (each
// step of a batch costs the adjoint one pass of add_pair).
template <typename Body>
__device__ __forceinline__ void run_pairs(const PairList& L, const float4* sP, bool filter,
                                          float Rc2, int2* queue, int lane, Body body) {
  const unsigned lt = (1u << lane) - 1u;
  const int sub = !L.tri && L.mc < 32 ? lane / L.mc : 0;
  const int qfirst = L.tri ? 1 : 0, qlast = L.tri ? L.mr / 2 : L.mc - 1;
  const int nb = (L.mr + 31) / 32, width = (L.mr + nb - 1) / nb;
  if (!filter) Rc2 = 3e38f;
  int head = 0, key = sub;
  for (int rb = 0; rb < L.mr; rb += width) {
    const int r = rb + lane;
    const bool row = lane < width && r < L.mr;
    const float4 P = sP[L.r0 + (row ? r : rb)];
    const int k0 = row ? (L.tri ? r + 1 : r % L.mc) : 0;
    // the last offset of an even bucket pairs its lower half only
    const int qend = !row ? 0 : (L.tri && !(L.mr & 1) && r >= L.mr / 2 ? qlast : qlast + 1);
    const int jr = L.r0 + r;
    int kc = L.c0 + (k0 < L.mc ? k0 : 0);
    const int kend = L.c0 + L.mc;
    for (int q = qfirst; q <= qlast; ++q, key += 32) {
      const float4 O = sP[kc];
      const float dx = O.x - P.x, dy = O.y - P.y, dz = O.z - P.z;
      const bool ok = q < qend && dx * dx + dy * dy + dz * dz < Rc2;
      const unsigned m = __ballot_sync(0xffffffffu, ok);
      if (ok) queue[head + __popc(m & lt)] = make_int2(jr | (kc << 16), key);
      head += __popc(m);
      if (++kc == kend) kc = L.c0;
      const bool last = q == qlast && rb + width >= L.mr;
      while (head >= 32 || (last && head > 0)) {
        __syncwarp();
        const int n = min(head, 32);
        head -= n;
        const bool live = lane < n;
        const int2 e = queue[head + (live ? lane : 0)];
        __syncwarp();
        body(live, e.x & 0xffff, e.x >> 16, e.y);
      }
    }
  }
}

// ---- powers of the grid path: F = u^zeta, D = dF/du, u = (1 +- cos)/2
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float lg2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsq_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// e^(-eta x) from rate = -eta (FP64) or -eta log2 e (FP32)
__device__ __forceinline__ float decay_rate(float eta) { return -1.4426950408889634f * eta; }
__device__ __forceinline__ double decay_rate(double eta) { return -eta; }
__device__ __forceinline__ float decay(float rate, float x) { return ex2_approx(rate * x); }
__device__ __forceinline__ double decay(double rate, double x) { return exp_table(rate * x); }
template <typename T>
__device__ __forceinline__ T gval(const double* d, const float* f, int i);
template <>
__device__ __forceinline__ float gval<float>(const double*, const float* f, int i) {
  return f[i];
}
template <>
__device__ __forceinline__ double gval<double>(const double* d, const float*, int i) {
  return d[i];
}

constexpr int BE = 2;   // eta values per grid block

// fc(sqrt(x)) and d fc / dx; beyond Rc zero (FP64) or at the value of Rc,
// which rounds to zero (FP32, whose pairs are inside).  a2 = (pi/Rc)^2,
// a = pi/Rc
template <bool DERIV>
__device__ __forceinline__ void cut_x(double x, double Rc2, double a2, double, double& fc,
                                      double& dfc) {
  const double z = fma(a2, x, -FC_Y0);
  fc = x < Rc2 ? fc_series(z) : 0.0;
  if (DERIV) dfc = x < Rc2 ? a2 * fc_series_d(z) : 0.0;
}
template <bool DERIV>
__device__ __forceinline__ void cut_x(float x, float Rc2, float, float a, float& fc, float& dfc) {
  // the root and its reciprocal to their last rounding: one Newton step each
  // from the approximate reciprocal root
  x = fminf(fmaxf(x, 1e-16f), Rc2);
  const float y = rsq_approx(x), g = x * y, e = fmaf(-g, y, 1.f);
  float s, c;
  __sincosf(a * fmaf(0.5f * g, e, g), &s, &c);
  fc = fmaf(0.5f, c, 0.5f);
  if (DERIV) dfc = -0.25f * a * s * fmaf(0.5f * y, e, y);
}
// the same of a staged neighbour at r, d fc / dr
template <bool DERIV>
__device__ __forceinline__ void cut_r(double r, double Rc2, double a2, double, double& fc,
                                      double& dfc) {
  cut_x<DERIV>(r * r, Rc2, a2, 0.0, fc, dfc);
  if (DERIV) dfc *= 2.0 * r;
}
template <bool DERIV>
__device__ __forceinline__ void cut_r(float r, float, float, float a, float& fc, float& dfc) {
  float s, c;
  __sincosf(a * r, &s, &c);
  fc = fmaf(0.5f, c, 0.5f);
  if (DERIV) dfc = -0.5f * a * s;
}

// Per-neighbour factors of a grid block: h_e = exp(-eta_e r^2) fc(r), 1/r
// and fc'/fc (whose products with h_e and -2 eta_e r h_e give dh_e/dr; fc is
// kept away from zero so that h_e fc'/fc stays exp(-eta_e r^2) fc' up to the
// cut-off).  Filled per bucket and kept while the etas and Rc stay the same.
template <typename T>
struct FactorKey {
  T eta0, eta1, Rc;
  unsigned filled;   // buckets whose factors are in place
};
__device__ __forceinline__ double fc_floor(double fc) { return fmax(fc, 1e-30); }
__device__ __forceinline__ float fc_floor(float fc) { return fmaxf(fc, 1e-12f); }
// a / b with b > 0 normal in FP32: FP64 by Newton's iteration for 1/b from an
// FP32 seed and one correction of the quotient
__device__ __forceinline__ float quotient(float a, float b) { return a / b; }
__device__ __forceinline__ double quotient(double a, double b) {
  float f;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"((float)b));
  double y = (double)f;
  y = fma(y, fma(-b, y, 1.0), y);
  const double q = a * y;
  return fma(fma(-q, b, a), y, q);
}
__device__ __forceinline__ float exp_fill(float x) { return expf(x); }
__device__ __forceinline__ double exp_fill(double x) { return exp_table(x); }

// The factors of a list's two buckets, filled together: lists of a few
// neighbours are many where there are many species, and each round costs a
// warp's FP64 instructions whatever lanes it uses.  (Calls of one row, five species
// whose lists have etas of their own: 6 neighbours 333 -> 248 us, 27 neighbours
// 483 -> 387 us.)
// DERIV: fc'/fc too (the adjoint).  sH comes with 1/r in place (stage_buckets).
template <typename T, bool DERIV>
__device__ __forceinline__ void need_factors(FactorKey<T>& key, const PairList& L,
                                             const typename V4<T>::type* sR, T Rc, T a, T a2,
                                             const T (&eta)[BE], typename V4<T>::type* sH,
                                             int lane) {
  using T4 = typename V4<T>::type;
  if (key.eta0 != eta[0] || key.eta1 != eta[1] || key.Rc != Rc) {
    key.eta0 = eta[0];
    key.eta1 = eta[1];
    key.Rc = Rc;
    key.filled = 0u;
  }
  const int nr = key.filled >> L.rs & 1u ? 0 : L.mr;
  const int n = nr + (L.tri || (key.filled >> L.cs & 1u) ? 0 : L.mc);
  __syncwarp();   // the previous list's readers are done
  for (int q = lane; q < n; q += 32) {
    const int j = q < nr ? L.r0 + q : L.c0 + q - nr;
    const T r = sR[j].w, x = r * r;
    T fc, dfc;
    cut_r<DERIV>(r, Rc * Rc, a2, a, fc, dfc);
    fc = fc_floor(fc);
    T4 h = sH[j];
    h.x = exp_fill(-eta[0] * x) * fc;
    h.y = exp_fill(-eta[1] * x) * fc;
    if (DERIV) h.w = quotient(dfc, fc);
    if (!(x < Rc * Rc)) h.x = h.y = T(0);
    sH[j] = h;
  }
  key.filled |= (1u << L.rs) | (1u << L.cs);
  __syncwarp();
}

// sum over the warp of 16 values per lane: lane l returns the sum of value
// l >> 1 (each step hands half of the values to the partner: 16 additions
// instead of the 80 of 16 butterflies)
template <typename T>
__device__ __forceinline__ T reduce16(T (&v)[16], int lane) {
#pragma unroll
  for (int h = 8, d = 16; h > 0; h >>= 1, d >>= 1) {
    const bool up = lane & d;
#pragma unroll
    for (int q = 0; q < h; ++q) {
      const T give = up ? v[q] : v[q + h];
      const T keep = up ? v[q + h] : v[q];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, give, d);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// The (lambda, zeta) entries of a grid handled together: slot [s][i] is sign
// s (0: lambda = +1, 1: -1) and the i-th zeta.  CHAIN: the zetas of the grid
// are z_0 = 2^s_0, z_i = z_{i-1} 2^{s_i} (BehlerGrid::chain), so that a
// sign's powers are a run of squarings; otherwise up to four entries of any
// zeta per pass, in list order (always in FP32, where CHAIN instances are those
// for zetas of one at least).
constexpr int NZ = AE_BG_NZ;

// ----------------------------------------------------------------------
// forward
// ----------------------------------------------------------------------
template <typename T>
struct WarpMem {
  typename V4<T>::type *sR, *sH, *sF;   // neighbours, factors, accumulators
  float4* sP;                                // FP32 positions (aliases sR in the FP32 kernels)
  T* sg;
  T* sB;                                     // [2][NZ] (g_0, g_1) of a grid block
  int* sslot;
  int2* queue;
};

// Shared memory of one warp: the staged neighbours (x, y, z, r), their
// factors (first dfc, fc, 1/r at the table's largest Rc for the radial
// functions, then those of the grids), FP32 positions for the pair test (FP64
// kernels), in the adjoint the accumulators and the scaled dE/dG row, the
// table slot of each staged neighbour and the pair queue.
constexpr int QCAP = 64;
template <typename T>
__host__ __device__ inline size_t behler_smem_per_warp(int cap, int nsf_pad, bool adjoint) {
  using T4 = typename V4<T>::type;
  size_t per = (adjoint ? 3 : 2) * sizeof(T4) * (size_t)cap + 4 * (size_t)cap + 8 * QCAP +
               (sizeof(T) == 8 ? sizeof(float4) * (size_t)cap : 0) +
               (adjoint ? sizeof(T) * ((size_t)nsf_pad + 2 * NZ * BE) : 0);
  return (per + 31) & ~size_t(31);
}
template <typename T>
__device__ __forceinline__ WarpMem<T> warp_mem(unsigned char* base, int cap, int nsf_pad,
                                               bool adjoint) {
  using T4 = typename V4<T>::type;
  WarpMem<T> w;
  w.sR = reinterpret_cast<T4*>(base);
  w.sH = w.sR + cap;
  w.sF = w.sH + cap;
  T4* next = adjoint ? w.sF + cap : w.sF;
  if (sizeof(T) == 8) {
    w.sP = reinterpret_cast<float4*>(next);
    w.sg = reinterpret_cast<T*>(w.sP + cap);
  } else {
    w.sP = reinterpret_cast<float4*>(w.sR);
    w.sg = reinterpret_cast<T*>(next);
  }
  w.sB = w.sg;
  if (adjoint) w.sg += 2 * NZ * BE;
  w.queue = reinterpret_cast<int2*>(w.sg + (adjoint ? nsf_pad : 0));
  w.sslot = reinterpret_cast<int*>(w.queue + QCAP);
  return w;
}
__device__ __forceinline__ void fill_positions(const double4_32a* sR, float4* sP, int n, int lane) {
  for (int j = lane; j < n; j += 32) {
    const double4_32a R = sR[j];
    sP[j] = make_float4((float)R.x, (float)R.y, (float)R.z, 0.f);
  }
  __syncwarp();
}
__device__ __forceinline__ void fill_positions(const float4*, float4*, int, int) {}

// squared cut-off of the FP32 pair test: exact for FP32 pairs, wider than any
// rounding of the FP32 positions for FP64 ones
__device__ __forceinline__ float filter_rc2(float Rc) { return Rc * Rc; }
__device__ __forceinline__ float filter_rc2(double Rc) {
  return (float)(Rc * Rc) * 1.0001f + 1e-4f;
}

// Block of a grid: the etas e0, e0 + 1 and the zeta entries of pass l0.
template <typename T>
struct GridBlock {
  T eta[BE], rate[BE];
  int iz[2][NZ];
  T zeta[2][NZ];
  int sq[NZ];
  // the grid entry of slot (s, i), or -1
  static __device__ __forceinline__ int entry(const BehlerGrid* gr, bool chain, int l0, int s,
                                              int i) {
    return chain ? gr->slot[s][i] : gr->general[s][l0 + i];
  }
  // the feature of slot (s, i) and eta e, or -1
  static __device__ __forceinline__ int feature(const BehlerGrid* gr, bool chain, int l0, int e0,
                                                int s, int i, int e) {
    const int l = entry(gr, chain, l0, s, i);
    return l >= 0 && e0 + e < gr->ne ? gr->out[l * AE_BG_NE + e0 + e] : -1;
  }
  __device__ __forceinline__ void load(const BehlerGrid* gr, bool chain, int l0, int e0) {
#pragma unroll
    for (int e = 0; e < BE; ++e)
      eta[e] = e0 + e < gr->ne ? gval<T>(gr->eta, gr->feta, e0 + e) : T(0);
#pragma unroll
    for (int e = 0; e < BE; ++e) rate[e] = decay_rate(eta[e]);
#pragma unroll
    for (int i = 0; i < NZ; ++i) sq[i] = gr->sq[i];
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int i = 0; i < NZ; ++i) {
        const int l = entry(gr, chain, l0, s, i);
        iz[s][i] = l >= 0 ? gr->izeta[l] : 1;
        zeta[s][i] = l >= 0 ? gval<T>(gr->zeta, gr->fzeta, l) : T(1);
      }
  }
};

// F (and D = dF/du) of one sign's entries at u: squarings along the chain
// (FP64: 8 multiplications for the zetas 1, 2, 4, 16 of both signs), or one
// power per entry (FP32: u^zeta = 2^(zeta log2 u) on the special-function
// unit, which the pair's work leaves idle, costs fewer instructions than the
// uniform loops of a chain)
template <bool CHAIN, bool DERIV>
__device__ __forceinline__ void powers(double u, const GridBlock<double>& B, int s, int nz,
                                       double (&F)[NZ], double (&D)[NZ]) {
  if (CHAIN) {
    double f = u, d = 1.0;
#pragma unroll
    for (int i = 0; i < NZ; ++i) {
      if (i < nz) {
        for (int t = B.sq[i]; t > 0; --t) {
          if (DERIV) d *= f + f;
          f *= f;
        }
      }
      F[i] = f;
      if (DERIV) D[i] = d;
    }
  } else {
#pragma unroll
    for (int i = 0; i < NZ; ++i)
      if (i < nz) {
        if (B.iz[s][i] > 0) {
          const double p = ipow(u, B.iz[s][i] - 1);
          F[i] = p * u;
          D[i] = B.zeta[s][i] * p;
        } else {
          F[i] = pow(u, B.zeta[s][i]);
          if (DERIV) D[i] = B.zeta[s][i] * pow(u, B.zeta[s][i] - 1.0);
        }
      }
  }
}
template <bool CHAIN>
__device__ __forceinline__ void powers(float u, const GridBlock<float>& B, int s, int nz,
                                       float (&F)[NZ]) {
  const float l = lg2_approx(u);
#pragma unroll
  for (int i = 0; i < NZ; ++i) F[i] = ex2_approx(B.zeta[s][i] * l);   // absent entries too
}

// A_e += sum_i g_ie F_i and d_e = sum_i g_ie D_i of one sign
template <bool CHAIN>
__device__ __forceinline__ void power_sums(double u, const GridBlock<double>& B, int s, int nz,
                                           const double* g, double (&A)[BE], double (&d)[BE]) {
  double F[NZ], D[NZ];
  powers<CHAIN, true>(u, B, s, nz, F, D);
#pragma unroll
  for (int e = 0; e < BE; ++e) d[e] = 0.0;
#pragma unroll
  for (int i = 0; i < NZ; ++i)
    if (i < nz) {
#pragma unroll
      for (int e = 0; e < BE; ++e) {
        const double ge = g[(s * NZ + i) * BE + e];
        A[e] = fma(ge, F[i], A[e]);
        d[e] = fma(ge, D[i], d[e]);
      }
    }
}
// FP32: D = zeta P with P = u^(zeta - 1), F = P u: exact at zeta = 1, and at u =
// 0 too (of two neighbours in line u rounds to zero before the gradient of
// the cosine that D multiplies does).  Zetas below one have no D there and
// take zero (CHAIN: there are none).
template <bool CHAIN>
__device__ __forceinline__ void power_sums(float u, const GridBlock<float>& B, int s, int nz,
                                           const float* g, float (&A)[BE], float (&d)[BE]) {
  float F[NZ], z[NZ];
  const float l = lg2_approx(CHAIN ? fmaxf(u, 1.2e-38f) : u);
  const float inv = CHAIN || !(u > 0.f) ? 0.f : __frcp_rn(u);
#pragma unroll
  for (int i = 0; i < NZ; ++i) {
    const float zeta = B.zeta[s][i];
    if (CHAIN) {
      const float P = ex2_approx(fmaf(zeta, l, -l));
      F[i] = P * u;
      z[i] = P * zeta;
    } else {
      F[i] = ex2_approx(zeta * l);
      z[i] = zeta == 1.f ? 1.f : zeta * (F[i] * inv);
    }
  }
#pragma unroll
  for (int e = 0; e < BE; ++e) d[e] = 0.f;
  const float4* g4 = reinterpret_cast<const float4*>(g + s * NZ * BE);
#pragma unroll
  for (int i = 0; i < NZ; i += 2) {
    const float4 q = g4[i / 2];
    A[0] = fmaf(q.z, F[i + 1], fmaf(q.x, F[i], A[0]));
    A[1] = fmaf(q.w, F[i + 1], fmaf(q.y, F[i], A[1]));
    d[0] = fmaf(q.z, z[i + 1], fmaf(q.x, z[i], d[0]));
    d[1] = fmaf(q.w, z[i + 1], fmaf(q.y, z[i], d[1]));
  }
}

template <bool CHAIN>
__device__ __forceinline__ void powers(double u, const GridBlock<double>& B, int s, int nz,
                                       double (&F)[NZ]) {
  double D[NZ];
  powers<CHAIN, false>(u, B, s, nz, F, D);
}

template <typename T, bool CHAIN>
__device__ void forward_grid(const BehlerGrid* gr, const PairList& L, const WarpMem<T>& w,
                             FactorKey<T>& key, T* G, const PotDevice& pd, size_t nrow, int lane) {
  using T4 = typename V4<T>::type;
  const bool g4 = gr->kind == 4;
  const T Rc = gval<T>(&gr->Rc, &gr->fRc, 0);
  const T a = T(SF_PI) / Rc, a2 = a * a, Rc2 = Rc * Rc;
  const int npass = CHAIN ? 1 : (gr->ngeneral + NZ - 1) / NZ;
  for (int e0 = 0; e0 < gr->ne; e0 += BE)
    for (int pass = 0; pass < npass; ++pass) {
      GridBlock<T> B;
      B.load(gr, CHAIN, NZ * pass, e0);
      const int nz = CHAIN ? gr->chain : min(NZ, gr->ngeneral - NZ * pass);
      need_factors<T, false>(key, L, w.sR, Rc, a, a2, B.eta, w.sH, lane);
      T acc[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) acc[q] = T(0);
      run_pairs(L, w.sP, g4, filter_rc2(Rc), w.queue, lane, [&](bool live, int j, int k, int) {
        const T4 Rj = w.sR[j], Rk = w.sR[k], Hj = w.sH[j], Hk = w.sH[k];
        T E[BE] = {Hj.x * Hk.x, Hj.y * Hk.y};
        if (g4) {
          const T dx = Rk.x - Rj.x, dy = Rk.y - Rj.y, dz = Rk.z - Rj.z;
          const T x = dx * dx + dy * dy + dz * dz;
          T fc, dum;
          cut_x<false>(x, Rc2, a2, a, fc, dum);
#pragma unroll
          for (int e = 0; e < BE; ++e) E[e] *= decay(B.rate[e], x) * fc;
        }
        if (!live) E[0] = E[1] = T(0);
        const T c = (Rj.x * Rk.x + Rj.y * Rk.y + Rj.z * Rk.z) * (Hj.z * Hk.z);
        const T ch = fmax(T(-0.5), fmin(T(0.5), T(0.5) * c));
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          T F[NZ];
          powers<CHAIN>(s ? T(0.5) - ch : T(0.5) + ch, B, s, nz, F);
#pragma unroll
          for (int i = 0; i < NZ; ++i)
            if (sizeof(T) == 4 || i < nz) {
#pragma unroll
              for (int e = 0; e < BE; ++e)
                acc[(s * NZ + i) * BE + e] = fma(F[i], E[e], acc[(s * NZ + i) * BE + e]);
            }
        }
      });
      const T v = T(2) * reduce16(acc, lane);   // the factor 2 of symmfunc.f90:724
      const int out = GridBlock<T>::feature(gr, CHAIN, NZ * pass, e0, lane >> 4, (lane >> 2) & 3,
                                            (lane >> 1) & 1);
      if (!(lane & 1) && out >= 0) G[out] = normalise(v, pd, nrow + out);
    }
}

template <typename T>
__device__ void forward_generic(const BehlerTable* tab, int f0, int f1e, const PairList& L,
                                const WarpMem<T>& w, T* G, const PotDevice& pd, size_t nrow,
                                int lane) {
  using T4 = typename V4<T>::type;
  for (int c0 = f0; c0 < f1e; c0 += FCH) {
    const int nf = min(FCH, f1e - c0);
    T acc[FCH];
#pragma unroll
    for (int q = 0; q < FCH; ++q) acc[q] = T(0);
    run_pairs(L, w.sP, false, 0.f, w.queue, lane, [&](bool live, int j, int k, int) {
      const T4 Rj = w.sR[j], Rk = w.sR[k];
      const T dxx = Rk.x - Rj.x, dyy = Rk.y - Rj.y, dzz = Rk.z - Rj.z;
      const T rjk2 = dxx * dxx + dyy * dyy + dzz * dzz;
      const T rjk = sqrt(rjk2);
      T cosv = (Rj.x * Rk.x + Rj.y * Rk.y + Rj.z * Rk.z) / (Rj.w * Rk.w);
      cosv = fmax(T(-1), fmin(T(1), cosv));
      const T rij2 = Rj.w * Rj.w, rik2 = Rk.w * Rk.w;
      T rc_cur = T(-1), fij = T(0), fik = T(0), fjk = T(0), dum;
#pragma unroll
      for (int q = 0; q < FCH; ++q) {
        if (q < nf) {
          const Fn<T> f = load_fn<T>(&tab->fn[c0 + q]);
          if (f.Rc != rc_cur) {
            rc_cur = f.Rc;
            cutfn(Rj.w, rc_cur, fij, dum);
            cutfn(Rk.w, rc_cur, fik, dum);
            cutfn(rjk, rc_cur, fjk, dum);
          }
          T F, dF;
          f1(f, cosv, F, dF);
          if (!live) F = T(0);
          if (f.kind == 4)
            acc[q] += T(2) * F * exp_t(-f.p3 * (rij2 + rik2 + rjk2)) * fij * fik * fjk;
          else
            acc[q] += T(2) * F * exp_t(-f.p3 * (rij2 + rik2)) * fij * fik;
        }
      }
    });
#pragma unroll
    for (int q = 0; q < FCH; ++q) {
      if (q < nf) {
        const T v = warp_sum(acc[q]);
        if (lane == q) {
          const int out = tab->fn[c0 + q].out;
          G[out] = normalise(v, pd, nrow + out);
        }
      }
    }
  }
}

// The pair lists of a block: all of its atom's, or (SPLIT) the one of number
// blockIdx.y among the species pairs a <= c, the first with the radial
// functions.
template <bool SPLIT>
struct ListOf {
  int a, c;   // the one list
  __device__ __forceinline__ explicit ListOf(int nt) {
    if (!SPLIT) return;
    int u = blockIdx.y;
    a = 0;
    while (u >= nt - a) u -= nt - a++;
    c = a + u;
  }
  __device__ __forceinline__ bool first() const { return !SPLIT || blockIdx.y == 0; }
  __device__ __forceinline__ bool list(int x, int y) const { return !SPLIT || (x == a && y == c); }
  // whether this block sets feature k
  __device__ __forceinline__ bool mine(const BehlerTable* tab, int k) const {
    if (!SPLIT) return true;
    const int u = tab->list_of[k];
    return u < 0 ? first() : u == (int)blockIdx.y;
  }
  // whether staged neighbour j can have a force from this block
  __device__ __forceinline__ bool touches(const int* bstart, int j) const {
    return first() || (j >= bstart[a] && j < bstart[a + 1]) || (j >= bstart[c] && j < bstart[c + 1]);
  }
};

// Whether the lists of an atom go to blocks of their own.  One warp takes an
// atom's lists in turn, as long as four to five (FP64) or many more (mixed)
// atoms in flight on an SM take together, so a few atoms an SM, or few left
// over after full SMs, leave it waiting; but every block stages the
// neighbours anew.  Rutile (three lists), forward and adjoint (us), one block
// an atom and split:
//   FP64   72 atoms 403 + 682 and 188 + 310, 270 atoms 402 + 682 and 217 +
//          389, 750 atoms 454 + 815 and 510 + 901, 1,512 atoms 1,212 + 2,257
//          and 977 + 1,739, 3,072 atoms 1,837 + 3,419 and 1,857 + 3,301
//   mixed  72 atoms 69 + 85 and 45 + 44, 750 atoms 70 + 92 and 50 + 55, 1,512
//          atoms 75 + 102 and 88 + 98, 3,072 atoms 96 + 197 and 137 + 172
// FP64: in units of an atom's time on a full SM (eight blocks), the last round
// of fewer takes 4.4 at least, and splitting costs 0.65.
template <typename T>
bool split_lists(int natoms, int lists) {
  if (lists < 2 || lists > 6) return false;
  int dev = 0, nsm = 152;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const double per = (double)natoms / nsm;
  if (sizeof(T) == 4) return per <= 7.0;
  const double full = 8.0 * std::floor(per / 8.0), rest = per - full;
  return per + 0.65 < full + (rest > 0.0 ? std::fmax(4.4, rest) : 0.0);
}

// GRID: every angular list is a BehlerGrid (the generic path is left out,
// which frees its registers).  One warp per block: the warps of a block
// share nothing, and small blocks spread a few hundred atoms evenly.
template <typename T, bool GRID, bool SPLIT>
__global__ void __launch_bounds__(32, sizeof(T) == 4 ? FWD_BLOCKS : 1) k_behler_forward(PotDevice pd, DescBuffers b) {
  using T4 = typename V4<T>::type;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  const int lane = threadIdx.x;
  const int i = blockIdx.x;
  const WarpMem<T> w = warp_mem<T>(smem_raw, b.cap, pd.nsf_pad, false);
  const ListOf<SPLIT> of(pd.ntypes);
  const int ti = b.types[i];
  const BehlerTable* tab = table_of<T>(pd, ti);
  const int nt = pd.ntypes;
  const int n = b.nb_cnt[i];
  const T4* __restrict__ vec = reinterpret_cast<const T4*>(b.nb_vec) + (size_t)i * b.cap;
  const int* __restrict__ jt = b.nb_jt + (size_t)i * b.cap;
  int bstart[AE_MAXT + 1];
  const int nst = stage_buckets<T>(vec, jt, n, nt, T(tab->rc_max), w.sR, w.sH, w.sslot, bstart,
                                   lane);
  fill_positions(w.sR, w.sP, nst, lane);
  if (b.zero_F && lane == 0 && of.first()) {
    T4 z;
    z.x = z.y = z.z = z.w = T(0);
    reinterpret_cast<T4*>(b.F)[i] = z;
  }
  const size_t nrow = (size_t)ti * pd.nsf_pad;
  T* G = reinterpret_cast<T*>(b.G) + (size_t)i * pd.nsf_pad;
  const int nsf = pd.sp[ti].nsf;
  // features that no function feeds are normalised zeros (symmfunc.f90:367);
  // a block with one list of its own leaves the other lists' alone
  for (int k = lane; k < nsf; k += 32)
    if (of.mine(tab, k)) G[k] = normalise(T(0), pd, nrow + k);
  __syncwarp();

  // ---- radial lists: function by function, lanes over the bucket's
  // neighbours (a few per lane), warp sum
  for (int s = 0; s < nt && of.first(); ++s) {
    const int f0 = tab->rad_off[s], f1e = tab->rad_off[s + 1];
    for (int q = f0; q < f1e; ++q) {
      const Fn<T> f = load_fn<T>(&tab->fn[q]);
      const bool cached = f.Rc == T(tab->rc_max);
      T acc = T(0);
      for (int j = bstart[s] + lane; j < bstart[s + 1]; j += 32) {
        T v, dv;
        radial_fn(f, w.sR[j].w, cached, w.sH[j], v, dv);
        acc += v;
      }
      acc = warp_sum(acc);
      if (lane == 0) G[f.out] = normalise(acc, pd, nrow + f.out);
    }
  }

  // ---- angular lists (one per unordered pair of neighbour species)
  FactorKey<T> key{T(-1), T(-1), T(-1), 0u};
  const BehlerGrid* grids = grids_of(tab);
  for (int a = 0; a < nt; ++a) {
    for (int c = a; c < nt; ++c) {
      const int f0 = tab->ang_off[a * nt + c], f1e = tab->ang_off[a * nt + c + 1];
      if (f0 == f1e || !of.list(a, c)) continue;
      const PairList L = pair_list(bstart, a, c);
      if (empty(L)) continue;
      const int gi = tab->grid_of[a * nt + c];
      if (GRID || gi >= 0) {
        const BehlerGrid* gr = grids + gi;
        if (sizeof(T) == 8 && gr->chain)
          forward_grid<T, sizeof(T) == 8>(gr, L, w, key, G, pd, nrow, lane);
        else
          forward_grid<T, false>(gr, L, w, key, G, pd, nrow, lane);
      } else {
        if constexpr (!GRID) forward_generic<T>(tab, f0, f1e, L, w, G, pd, nrow, lane);
      }
    }
  }
}

// ----------------------------------------------------------------------
// adjoint
// ----------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void atomic_add3(T* F, int atom, T fx, T fy, T fz);
template <>
__device__ __forceinline__ void atomic_add3<float>(float* F, int atom, float fx, float fy, float fz) {
  atomicAdd(reinterpret_cast<float4*>(F) + atom, make_float4(fx, fy, fz, 0.f));
}
template <>
__device__ __forceinline__ void atomic_add3<double>(double* F, int atom, double fx, double fy,
                                                    double fz) {
  atomicAdd(F + 4 * atom, fx);
  atomicAdd(F + 4 * atom + 1, fy);
  atomicAdd(F + 4 * atom + 2, fz);
}

// The gradient of one pair's terms with respect to R_j and R_k from the
// partials Sc (cos), Sj and Sk (r_ij, r_ik) and Sx (twice that in r_jk^2),
// added to the neighbours' accumulators in shared memory.  Step by step of
// the pair schedule the lanes hold distinct rows and distinct partners, so
// plain adds are enough (shared-memory atomics, six per pair, are loops).
//   FP32: the vector gradients, as
//     Sc/r_j (v - cos u) + Sj u - Sx (R_k - R_j)
//   FP64: their coefficients of the two position vectors, alpha R_k + beta_j
//     R_j and alpha R_j + beta_k R_k, with beta summed per neighbour (10
//     multiply-adds less per pair; the sums cancel to the vectors, which
//     costs FP32 a digit and FP64 nothing that its results show)
template <typename T>
struct PairGrad;
template <>
struct PairGrad<float> {
  float gx, gy, gz, hx, hy, hz;
  __device__ __forceinline__ PairGrad(const float4& Rj, const float4& Rk, float invj, float invk,
                                      float c, float Sc, float Sj, float Sk, float Sx) {
    const float ux = Rj.x * invj, uy = Rj.y * invj, uz = Rj.z * invj;
    const float vx = Rk.x * invk, vy = Rk.y * invk, vz = Rk.z * invk;
    const float dx = Sx * (Rk.x - Rj.x), dy = Sx * (Rk.y - Rj.y), dz = Sx * (Rk.z - Rj.z);
    const float cj = Sc * invj, ck = Sc * invk;
    const float bj = fmaf(-cj, c, Sj), bk = fmaf(-ck, c, Sk);
    gx = fmaf(cj, vx, fmaf(bj, ux, -dx));
    gy = fmaf(cj, vy, fmaf(bj, uy, -dy));
    gz = fmaf(cj, vz, fmaf(bj, uz, -dz));
    hx = fmaf(ck, ux, fmaf(bk, vx, dx));
    hy = fmaf(ck, uy, fmaf(bk, vy, dy));
    hz = fmaf(ck, uz, fmaf(bk, vz, dz));
  }
  __device__ __forceinline__ void add_j(float4& f, const float4&) const {
    f.x += gx;
    f.y += gy;
    f.z += gz;
  }
  __device__ __forceinline__ void add_k(float4& f, const float4&) const {
    f.x += hx;
    f.y += hy;
    f.z += hz;
  }
};
template <>
struct PairGrad<double> {
  double alpha, bj, bk;
  __device__ __forceinline__ PairGrad(const double4_32a&, const double4_32a&, double invj,
                                      double invk, double c, double Sc, double Sj, double Sk,
                                      double Sx) {
    alpha = fma(Sc, invj * invk, -Sx);
    const double scc = Sc * c;
    bj = fma(invj, fma(-scc, invj, Sj), Sx);
    bk = fma(invk, fma(-scc, invk, Sk), Sx);
  }
  __device__ __forceinline__ void add_j(double4_32a& f, const double4_32a& Rk) const {
    f.x = fma(alpha, Rk.x, f.x);
    f.y = fma(alpha, Rk.y, f.y);
    f.z = fma(alpha, Rk.z, f.z);
    f.w += bj;
  }
  __device__ __forceinline__ void add_k(double4_32a& f, const double4_32a& Rj) const {
    f.x = fma(alpha, Rj.x, f.x);
    f.y = fma(alpha, Rj.y, f.y);
    f.z = fma(alpha, Rj.z, f.z);
    f.w += bk;
  }
};

template <typename T>
__device__ __forceinline__ void add_pair(typename V4<T>::type* sF, bool live, int j, int k, int key,
                                         const typename V4<T>::type& Rj,
                                         const typename V4<T>::type& Rk, const PairGrad<T>& p) {
  using T4 = typename V4<T>::type;
  // runs of equal keys, in lane order
  const int lane = threadIdx.x;
  const int before = __shfl_up_sync(0xffffffffu, key, 1);
  const unsigned first = __ballot_sync(0xffffffffu, live && (lane == 0 || key != before));
  const int run = live ? __popc(first & (0xffffffffu >> (31 - lane))) : 0;
  const int nrun = __popc(first);
  for (int q = 1; q <= nrun; ++q) {
    if (run == q) {
      T4 f = sF[j];
      p.add_j(f, Rk);
      sF[j] = f;
    }
    __syncwarp();
    if (run == q) {
      T4 f = sF[k];
      p.add_k(f, Rj);
      sF[k] = f;
    }
    __syncwarp();
  }
}

template <typename T, bool CHAIN>
__device__ void adjoint_grid(const BehlerGrid* gr, const PairList& L, const WarpMem<T>& w,
                             FactorKey<T>& key, int lane) {
  using T4 = typename V4<T>::type;
  const bool g4 = gr->kind == 4;
  const T Rc = gval<T>(&gr->Rc, &gr->fRc, 0);
  const T a = T(SF_PI) / Rc, a2 = a * a, Rc2 = Rc * Rc;
  constexpr bool ORDER = CHAIN && sizeof(T) == 8;   // the entries in the chain's order
  const int npass = ORDER ? 1 : (gr->ngeneral + NZ - 1) / NZ;
  for (int e0 = 0; e0 < gr->ne; e0 += BE)
    for (int pass = 0; pass < npass; ++pass) {
      GridBlock<T> B;
      B.load(gr, ORDER, NZ * pass, e0);
      const int nz = ORDER ? gr->chain : min(NZ, gr->ngeneral - NZ * pass);
      __syncwarp();
      if (lane < 2 * NZ * BE) {
        const int f = GridBlock<T>::feature(gr, ORDER, NZ * pass, e0, lane / (NZ * BE),
                                            lane / BE % NZ, lane % BE);
        w.sB[lane] = f >= 0 ? T(2) * w.sg[f] : T(0);
      }
      need_factors<T, true>(key, L, w.sR, Rc, a, a2, B.eta, w.sH, lane);
      run_pairs(L, w.sP, g4, filter_rc2(Rc), w.queue, lane, [&](bool live, int j, int k, int step) {
        const T4 Rj = w.sR[j], Rk = w.sR[k], Hj = w.sH[j], Hk = w.sH[k];
        const T invj = Hj.z, invk = Hk.z;
        const T c = (Rj.x * Rk.x + Rj.y * Rk.y + Rj.z * Rk.z) * (invj * invk);
        const T ch = fmax(T(-0.5), fmin(T(0.5), T(0.5) * c));
        T A[BE] = {T(0), T(0)}, C[BE] = {T(0), T(0)};   // sum of g F, twice its d/dcos
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          T d[BE];
          power_sums<CHAIN>(s ? T(0.5) - ch : T(0.5) + ch, B, s, nz, w.sB, A, d);
#pragma unroll
          for (int e = 0; e < BE; ++e) C[e] = s ? C[e] - d[e] : d[e];
        }
        T h[BE] = {Hj.x * Hk.x, Hj.y * Hk.y};
        T fc = T(1), dfc = T(0);
        if (g4) {
          const T dx = Rk.x - Rj.x, dy = Rk.y - Rj.y, dz = Rk.z - Rj.z;
          const T x = dx * dx + dy * dy + dz * dz;
          cut_x<true>(x, Rc2, a2, a, fc, dfc);
#pragma unroll
          for (int e = 0; e < BE; ++e) h[e] *= decay(B.rate[e], x);
        }
        // with s_e = A_e h_e fc(r_jk): the partials in r_ij, r_ik and r_jk^2
        // from the sums of s_e and eta_e s_e
        const T s0 = A[0] * h[0], s1 = A[1] * h[1];
        const T sum = s0 + s1;
        const T S = sum * fc, Se = fma(B.eta[0], s0, B.eta[1] * s1) * fc;
        const T Sc = T(0.5) * fc * fma(C[0], h[0], C[1] * h[1]);
        const T e2 = Se + Se;
        const T Sj = fma(S, Hj.w, -e2 * Rj.w), Sk = fma(S, Hk.w, -e2 * Rk.w);
        const T Sx = g4 ? T(2) * fma(sum, dfc, -Se) : T(0);
        const PairGrad<T> p(Rj, Rk, invj, invk, ch + ch, Sc, Sj, Sk, Sx);
        add_pair<T>(w.sF, live, j, k, step, Rj, Rk, p);
      });
    }
}

template <typename T>
__device__ void adjoint_generic(const BehlerTable* tab, int f0, int f1e, const PairList& L,
                                const WarpMem<T>& w, int lane) {
  using T4 = typename V4<T>::type;
  run_pairs(L, w.sP, false, 0.f, w.queue, lane, [&](bool live, int j, int k, int key) {
    const T4 Rj = w.sR[j], Rk = w.sR[k];
    const T invj = T(1) / Rj.w, invk = T(1) / Rk.w;
    const T dx = Rk.x - Rj.x, dy = Rk.y - Rj.y, dz = Rk.z - Rj.z;
    const T rjk2 = dx * dx + dy * dy + dz * dz;
    const T rjk = sqrt(rjk2);
    T cosv = (Rj.x * Rk.x + Rj.y * Rk.y + Rj.z * Rk.z) * invj * invk;
    cosv = fmax(T(-1), fmin(T(1), cosv));
    const T rij2 = Rj.w * Rj.w, rik2 = Rk.w * Rk.w;
    T rc_cur = T(-1), fij = 0, dfij = 0, fik = 0, dfik = 0, fjk = 0, dfjk = 0;
    T Sc = T(0), Sij = T(0), Sik = T(0), Sjk = T(0);
    for (int q = f0; q < f1e; ++q) {
      const Fn<T> f = load_fn<T>(&tab->fn[q]);
      if (f.Rc != rc_cur) {
        rc_cur = f.Rc;
        cutfn(Rj.w, rc_cur, fij, dfij);
        cutfn(Rk.w, rc_cur, fik, dfik);
        cutfn(rjk, rc_cur, fjk, dfjk);
      }
      const T g2 = T(2) * w.sg[f.out];
      T F1v, dF1v;
      f1(f, cosv, F1v, dF1v);
      if (f.kind == 4) {
        const T base3 = g2 * exp_t(-f.p3 * (rij2 + rik2 + rjk2));
        Sc += base3 * dF1v * fij * fik * fjk;
        Sij += base3 * F1v * fik * fjk * (dfij - T(2) * f.p3 * Rj.w * fij);
        Sik += base3 * F1v * fij * fjk * (dfik - T(2) * f.p3 * Rk.w * fik);
        Sjk += base3 * F1v * fij * fik * (dfjk - T(2) * f.p3 * rjk * fjk);
      } else {
        const T base3 = g2 * exp_t(-f.p3 * (rij2 + rik2));
        Sc += base3 * dF1v * fij * fik;
        Sij += base3 * F1v * fik * (dfij - T(2) * f.p3 * Rj.w * fij);
        Sik += base3 * F1v * fij * (dfik - T(2) * f.p3 * Rk.w * fik);
      }
    }
    const T Sx = rjk > T(1e-8) ? Sjk / rjk : T(0);   // 2 dE/d(r_jk^2)
    const PairGrad<T> p(Rj, Rk, invj, invk, cosv, Sc, Sij, Sik, Sx);
    add_pair<T>(w.sF, live, j, k, key, Rj, Rk, p);
  });
}

// One-sided adjoint: every pair (j, k) is evaluated once, by one lane, and
// its gradient goes to both staged neighbours' accumulators in shared
// memory (add_pair).  The central atom's gradient is minus the
// sum over its neighbours (the energy depends on R_j - R_i only), and the
// atom's virial contribution is -sum_j R_ij (x) dE_i/dR_j.
template <typename T, bool GRID, bool SPLIT>
__global__ void __launch_bounds__(32, sizeof(T) == 4 ? ADJ_BLOCKS : 1) k_behler_adjoint(PotDevice pd, DescBuffers b) {
  using T4 = typename V4<T>::type;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  const int lane = threadIdx.x;
  const int i = blockIdx.x;
  const WarpMem<T> w = warp_mem<T>(smem_raw, b.cap, pd.nsf_pad, true);
  const ListOf<SPLIT> of(pd.ntypes);
  const int ti = b.types[i];
  const BehlerTable* tab = table_of<T>(pd, ti);
  const int nt = pd.ntypes;
  const int n = b.nb_cnt[i];
  const T4* __restrict__ vec = reinterpret_cast<const T4*>(b.nb_vec) + (size_t)i * b.cap;
  const int* __restrict__ jt = b.nb_jt + (size_t)i * b.cap;
  const int sid = b.atom_struct[i];
  const T gs = b.grad_scale ? T(b.grad_scale[sid]) : T(1);
  const T* gsrc = reinterpret_cast<const T*>(b.dEdG) + (size_t)i * pd.nsf_pad;
  const int nsf = pd.sp[ti].nsf;
  for (int k = lane; k < nsf; k += 32) w.sg[k] = gs * gsrc[k];
  int bstart[AE_MAXT + 1];
  const int nst = stage_buckets<T>(vec, jt, n, nt, T(tab->rc_max), w.sR, w.sH, w.sslot, bstart,
                                   lane);
  fill_positions(w.sR, w.sP, nst, lane);

  // radial terms: d/dr_ij of sum_f g_f G_f(r_ij) along Rhat_ij (initialises
  // each staged neighbour's accumulator)
  for (int j = lane; j < nst; j += 32) {
    int tj = 0;
    for (int s = 0; s < nt; ++s)
      if (j >= bstart[s + 1]) tj = s + 1;
    const T r = w.sR[j].w;
    const T4 A = w.sH[j];
    const int f0 = tab->rad_off[tj], f1e = of.first() ? tab->rad_off[tj + 1] : f0;
    T c = T(0);
    for (int q = f0; q < f1e; ++q) {
      const Fn<T> f = load_fn<T>(&tab->fn[q]);
      T v, dv;
      radial_fn(f, r, f.Rc == T(tab->rc_max), A, v, dv);
      c += w.sg[f.out] * dv;
    }
    // FP64 sums coefficients of R_j, FP32 the vector
    T4 acc = w.sR[j];
    c *= A.z;
    const T cv = sizeof(T) == 8 ? T(0) : c;
    acc.x *= cv;
    acc.y *= cv;
    acc.z *= cv;
    acc.w = sizeof(T) == 8 ? c : T(0);
    w.sF[j] = acc;
  }
  __syncwarp();

  // angular terms, each pair once
  FactorKey<T> key{T(-1), T(-1), T(-1), 0u};
  const BehlerGrid* grids = grids_of(tab);
  for (int a = 0; a < nt; ++a) {
    for (int c = a; c < nt; ++c) {
      const int f0 = tab->ang_off[a * nt + c], f1e = tab->ang_off[a * nt + c + 1];
      if (f0 == f1e || !of.list(a, c)) continue;
      const PairList L = pair_list(bstart, a, c);
      if (empty(L)) continue;
      const int gi = tab->grid_of[a * nt + c];
      if (GRID || gi >= 0) {
        const BehlerGrid* gr = grids + gi;
        if (sizeof(T) == 8 ? gr->chain > 0 : gr->steep)
          adjoint_grid<T, true>(gr, L, w, key, lane);
        else
          adjoint_grid<T, false>(gr, L, w, key, lane);
      } else {
        if constexpr (!GRID) adjoint_generic<T>(tab, f0, f1e, L, w, lane);
      }
    }
  }
  __syncwarp();

  // forces: F_j -= dE_i/dR_j, F_i += sum_j dE_i/dR_j; virial
  T* F = reinterpret_cast<T*>(b.F);
  const bool want_virial = b.virial != nullptr;
  T fix = T(0), fiy = T(0), fiz = T(0);
  T w00 = 0, w01 = 0, w02 = 0, w10 = 0, w11 = 0, w12 = 0, w20 = 0, w21 = 0, w22 = 0;
  for (int j = lane; j < nst; j += 32) {
    if (!of.touches(bstart, j)) continue;
    const T4 Rj = w.sR[j], f = w.sF[j];
    const T gx = fma(f.w, Rj.x, f.x), gy = fma(f.w, Rj.y, f.y), gz = fma(f.w, Rj.z, f.z);
    atomic_add3<T>(F, jt[w.sslot[j]] & AE_INDEX_MASK, -gx, -gy, -gz);
    if (want_virial) {
      w00 -= Rj.x * gx; w01 -= Rj.x * gy; w02 -= Rj.x * gz;
      w10 -= Rj.y * gx; w11 -= Rj.y * gy; w12 -= Rj.y * gz;
      w20 -= Rj.z * gx; w21 -= Rj.z * gy; w22 -= Rj.z * gz;
    }
    fix += gx;
    fiy += gy;
    fiz += gz;
  }
  fix = warp_sum(fix);
  fiy = warp_sum(fiy);
  fiz = warp_sum(fiz);
  if (lane == 0) atomic_add3<T>(F, i, fix, fiy, fiz);
  if (want_virial) {
    T wv[9] = {w00, w01, w02, w10, w11, w12, w20, w21, w22};
#pragma unroll
    for (int q = 0; q < 9; ++q) wv[q] = warp_sum(wv[q]);
    if (lane == 0) {
      double* V = b.virial + 9 * sid;
#pragma unroll
      for (int q = 0; q < 9; ++q) atomicAdd(V + q, (double)wv[q]);
    }
  }
}

template <typename T>
int launch(const PotDevice& pd, const DescBuffers& b, bool adjoint, cudaStream_t s) {
  const size_t smem = behler_smem_per_warp<T>(b.cap, pd.nsf_pad, adjoint);
  if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
  const int lists = pd.ntypes * (pd.ntypes + 1) / 2;
  // (a single row's neighbours get their forces in one addition each, the same
  // bits every time)
  const bool split = split_lists<T>(b.natoms, lists) && !(adjoint && b.natoms == 1);
  const bool grid = pd.behler_grid_only;
  auto pick = [&](auto one, auto each) { return split ? each : one; };
  auto kern = adjoint ? (grid ? pick(k_behler_adjoint<T, true, false>, k_behler_adjoint<T, true, true>)
                              : pick(k_behler_adjoint<T, false, false>, k_behler_adjoint<T, false, true>))
                      : (grid ? pick(k_behler_forward<T, true, false>, k_behler_forward<T, true, true>)
                              : pick(k_behler_forward<T, false, false>, k_behler_forward<T, false, true>));
  allow_smem(kern, smem, 200 * 1024);
  kern<<<dim3(b.natoms, split ? lists : 1), 32, smem, s>>>(pd, b);
  return (int)cudaGetLastError();
}

// ----------------------------------------------------------------------
// descriptor Jacobians (FP64) for generate.x's PyTorch export: a
// two-sided sweep without the contraction with dE/dG -- the lane owning
// staged neighbour j adds dG_f/dR_j of every radial function of its bucket
// and of every angular function of every pair (j, k) to its own slot row
// (G4/G5 carry the factor 2 of symmfunc.f90:724); the central atom's row is
// minus the sum over the neighbours.
// ----------------------------------------------------------------------
// shared memory of one warp: the staged neighbours and their table slots
__host__ __device__ inline size_t jacobian_smem_per_warp(int cap) {
  return ((sizeof(double4_32a) + sizeof(int)) * (size_t)cap + 31) & ~size_t(31);
}
__global__ void __launch_bounds__(128) k_behler_jacobian(PotDevice pd, DescBuffers b, int atom0,
                                                         int count, int nsf_max,
                                                         double* __restrict__ Ji,
                                                         double* __restrict__ Jj,
                                                         int* __restrict__ nbl,
                                                         int* __restrict__ nnb) {
  using T = double;
  using T4 = double4_32a;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int r = blockIdx.x * (blockDim.x >> 5) + warp;
  if (r >= count) return;
  const int i = atom0 + r;
  unsigned char* base = smem_raw + jacobian_smem_per_warp(b.cap) * warp;
  T4* sR = reinterpret_cast<T4*>(base);
  int* sslot = reinterpret_cast<int*>(sR + b.cap);
  const int ti = b.types[i];
  const BehlerTable* tab = table_of<T>(pd, ti);
  const int nt = pd.ntypes;
  const int n = b.nb_cnt[i];
  const T4* __restrict__ vec = reinterpret_cast<const T4*>(b.nb_vec) + (size_t)i * b.cap;
  const int* __restrict__ jt = b.nb_jt + (size_t)i * b.cap;
  const size_t rs = (size_t)nsf_max * 3;
  double* __restrict__ Jrow = Jj + (size_t)r * b.cap * rs;
  if (lane == 0) nnb[r] = n;
  for (int a = lane; a < n; a += 32) {
    for (size_t q = 0; q < rs; ++q) Jrow[(size_t)a * rs + q] = 0.0;
    nbl[(size_t)r * b.cap + a] = jt[a] & AE_INDEX_MASK;
  }
  int bstart[AE_MAXT + 1];
  const int nst = stage_buckets<T>(vec, jt, n, nt, T(tab->rc_max), sR, nullptr, sslot, bstart,
                                   lane);
  __syncwarp();
  for (int j = lane; j < nst; j += 32) {
    int tj = 0;
    for (int s2 = 0; s2 < nt; ++s2)
      if (j >= bstart[s2 + 1]) tj = s2 + 1;
    if (tj >= nt) tj = nt - 1;
    const T4 Rj = sR[j];
    const T invj = T(1) / Rj.w;
    const T ux = Rj.x * invj, uy = Rj.y * invj, uz = Rj.z * invj;
    double* Ja = Jrow + (size_t)sslot[j] * rs;
    // radial functions of bucket tj
    for (int q = tab->rad_off[tj]; q < tab->rad_off[tj + 1]; ++q) {
      const Fn<T> f = load_fn<T>(&tab->fn[q]);
      T v, dv;
      radial_fn(f, Rj.w, false, T4{}, v, dv);
      Ja[f.out * 3] += dv * ux;
      Ja[f.out * 3 + 1] += dv * uy;
      Ja[f.out * 3 + 2] += dv * uz;
    }
    // angular functions of every pair (j, k)
    for (int k = 0; k < nst; ++k) {
      if (k == j) continue;
      int tk = 0;
      for (int s2 = 0; s2 < nt; ++s2)
        if (k >= bstart[s2 + 1]) tk = s2 + 1;
      const int lo = min(tj, tk), hi = max(tj, tk);
      const int f0 = tab->ang_off[lo * nt + hi], f1e = tab->ang_off[lo * nt + hi + 1];
      if (f0 == f1e) continue;
      const T4 Rk = sR[k];
      const T dxx = Rk.x - Rj.x, dyy = Rk.y - Rj.y, dzz = Rk.z - Rj.z;
      const T rjk2 = dxx * dxx + dyy * dyy + dzz * dzz;
      const T rjk = sqrt(rjk2);
      const T invk = T(1) / Rk.w;
      const T vx = Rk.x * invk, vy = Rk.y * invk, vz = Rk.z * invk;
      T cosv = ux * vx + uy * vy + uz * vz;
      cosv = fmax(T(-1), fmin(T(1), cosv));
      const T rij2 = Rj.w * Rj.w, rik2 = Rk.w * Rk.w;
      const T ijk = rjk > T(1e-8) ? T(1) / rjk : T(0);
      T rc_cur = T(-1), fij = 0, dfij = 0, fik = 0, dfik = 0, fjk = 0, dfjk = 0;
      for (int q = f0; q < f1e; ++q) {
        const Fn<T> f = load_fn<T>(&tab->fn[q]);
        if (f.Rc != rc_cur) {
          rc_cur = f.Rc;
          cutfn(Rj.w, rc_cur, fij, dfij);
          cutfn(Rk.w, rc_cur, fik, dfik);
          cutfn(rjk, rc_cur, fjk, dfjk);
        }
        T F1v, dF1v;
        f1(f, cosv, F1v, dF1v);
        T Sc, Sij, Sjk = T(0);
        if (f.kind == 4) {
          const T E = T(2) * exp_t(-f.p3 * (rij2 + rik2 + rjk2));
          Sc = E * dF1v * fij * fik * fjk;
          Sij = E * F1v * fik * fjk * (dfij - T(2) * f.p3 * Rj.w * fij);
          Sjk = E * F1v * fij * fik * (dfjk - T(2) * f.p3 * rjk * fjk);
        } else {
          const T E = T(2) * exp_t(-f.p3 * (rij2 + rik2));
          Sc = E * dF1v * fij * fik;
          Sij = E * F1v * fik * (dfij - T(2) * f.p3 * Rj.w * fij);
        }
        // grad_j = Sc (Rhat_k - cos Rhat_j)/r_ij + Sij Rhat_j - Sjk Rhat_jk
        const T cj = Sc * invj;
        Ja[f.out * 3] += cj * (vx - cosv * ux) + Sij * ux - Sjk * ijk * dxx;
        Ja[f.out * 3 + 1] += cj * (vy - cosv * uy) + Sij * uy - Sjk * ijk * dyy;
        Ja[f.out * 3 + 2] += cj * (vz - cosv * uz) + Sij * uz - Sjk * ijk * dzz;
      }
    }
  }
  __syncwarp();
  const int nq = pd.sp[ti].nsf * 3;
  for (int q = lane; q < (int)rs; q += 32) {
    double acc = 0.0;
    if (q < nq)
      for (int a = 0; a < n; ++a) acc -= Jrow[(size_t)a * rs + q];
    Ji[(size_t)r * rs + q] = acc;
  }
}

}  // namespace

int ae_launch_behler_forward(const PotDevice& pd, const DescBuffers& b, int fp64, cudaStream_t s) {
  if (b.natoms <= 0) return 0;
  return fp64 ? launch<double>(pd, b, false, s) : launch<float>(pd, b, false, s);
}

int ae_launch_behler_adjoint(const PotDevice& pd, const DescBuffers& b, int fp64, cudaStream_t s) {
  if (b.natoms <= 0) return 0;
  return fp64 ? launch<double>(pd, b, true, s) : launch<float>(pd, b, true, s);
}

int ae_launch_behler_jacobian(const PotDevice& pd, const DescBuffers& b, int atom0, int count,
                              int nsf_max, double* Ji, double* Jj, int* nbl, int* nnb,
                              cudaStream_t s) {
  if (count <= 0) return 0;
  const int warps = 4;
  const size_t smem = jacobian_smem_per_warp(b.cap) * warps;
  if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
  allow_smem(k_behler_jacobian, smem, 200 * 1024);
  k_behler_jacobian<<<(count + warps - 1) / warps, warps * 32, smem, s>>>(pd, b, atom0, count,
                                                                         nsf_max, Ji, Jj, nbl, nnb);
  return (int)cudaGetLastError();
}
