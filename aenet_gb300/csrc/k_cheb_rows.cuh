// Chebyshev descriptor and adjoint kernels of both precisions (the formulas and
// the feature layout are those of k_cheb_impl.cuh).
//
// FP64: the FP64 pipe of this GPU takes two lanes per clock and SM, 64 times
// fewer than FP32, and bounds these kernels (85 % busy); loads, shared memory
// and integer work run beside it for free.  FP32: instruction issue bounds
// them (83 % busy in the pair forward of 256,000 atoms), in the pair adjoint the
// shared-memory pipe (82 %: coefficient tables, staged neighbours and their
// sums).  For both the work is arranged for few instructions, each with all its
// lanes in use:
//   * FP64: the cut-off is a series in r^2 (no square root, sine or division:
//     14 multiply-adds for fc, 13 more for fc'), reciprocals come by Newton
//     steps from an FP32 seed;
//   * the neighbours inside the angular cut-off are compacted first and then
//     prepared (unit vector, fc, fc') densely;
//   * sums over a group's lanes are scattered while they are reduced: V
//     values cost about V additions per lane instead of V log2(lanes);
//   * sum_q c_q T_q and its derivative share the T_q (the derivative's
//     coefficients follow from the c_q once per atom and neighbour species):
//     three multiply-adds per order;
//   * the pairs a < k of staged neighbours are flattened over the lanes in
//     circulant order.  A pair's gradient needs five multiply-adds per side:
//     each neighbour sums V_a = sum_k fc_k A'(cos) u_k and S_a = sum_k fc_k
//     A(cos), from which its force follows at the end.  min(lanes, na - 1)
//     consecutive pairs have distinct a and distinct k, so both sums live in
//     shared memory without atomics;
//   * where the moments fit the registers the angular terms take the moment
//     form of k_cheb_mom.cuh with monic polynomials: linear in the angular
//     neighbours.
// Measured, before and now.  FP64: 512 Li/Si/O cells (72,513 atoms, 72
// neighbours, 21 angular) forward 2481 -> 1138 us, adjoint 4527 -> 1516 us;
// 2,765 Au/Cu atoms forward 144 -> 80 us, adjoint 323 -> 109 us.  The error
// against 64-bit automatic differentiation is that of the pair sums (1.6e-14
// of the forces of the batch, 1.7e-14 before).  FP32: 256,000 Cu/Au atoms (78
// neighbours, 18 angular, pair sums) forward 645 -> 235 us, adjoint 614 -> 444
// us; 4,096 Li/Si/O cells (597,000 atoms, moments) forward 569 -> 460 us.
#pragma once
#include "common.h"
#include "chain.cuh"
#include "cutoff64.cuh"
#include "k_cheb_mom.cuh"

namespace chebr {

constexpr double SFB_PI = 3.14159265358979;   // sfbasis.f90:72
constexpr double SFB_EPS = 1.0e-12;

template <typename T>
struct Num;
template <>
struct Num<float> {
  using v4 = float4;
  using v2 = float2;
};
template <>
struct Num<double> {
  using v4 = double4_32a;
  using v2 = double2;
};

// an empty row slot: beyond every cut-off
template <typename T>
__device__ __forceinline__ typename Num<T>::v4 far_row() {
  typename Num<T>::v4 v;
  v.x = v.y = v.z = T(0);
  v.w = T(1e30);
  return v;
}

// spin weights of the neighbours: none (single species), all within -1 .. 1
// (tables per spin), any
enum { SPIN_NONE = 0, SPIN_UNIT = 1, SPIN_ANY = 2 };

// 1 / d: FP64 by Newton's iteration from an FP32 seed (relative error 2^-23,
// then 2^-46, then rounding)
__device__ __forceinline__ double recip(double d) {
  float f;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"((float)d));
  double y = (double)f;
  y = fma(y, fma(-d, y, 1.0), y);
  return fma(y, fma(-d, y, 1.0), y);
}
__device__ __forceinline__ float recip(float d) { return __fdividef(1.0f, d); }

// fc(d) = (1 + cos(a d)) / 2 and fc' (over d: OVER_D), a = pi / Rc, zero from
// Rc on (sfb_fc / sfb_fc_d1, sfbasis.f90:719-752); inv = 1/d (FP32, OVER_D)
template <bool DERIV, bool OVER_D>
__device__ __forceinline__ void cutoff(double d, double Rc, double a, double, double& fc,
                                       double& dfc) {
  const double a2 = a * a, z = fma(a2 * d, d, -FC_Y0);
  fc = d < Rc ? fc_series(z) : 0.0;
  if (DERIV) dfc = d < Rc ? (OVER_D ? 2.0 * a2 : 2.0 * a2 * d) * fc_series_d(z) : 0.0;
}
template <bool DERIV, bool OVER_D>
__device__ __forceinline__ void cutoff(float d, float Rc, float a, float inv, float& fc,
                                       float& dfc) {
  float s, c;
  __sincosf(a * d, &s, &c);
  fc = d < Rc ? fmaf(0.5f, c, 0.5f) : 0.f;
  if (DERIV) dfc = d < Rc ? -0.5f * a * s * (OVER_D ? inv : 1.f) : 0.f;
}

__device__ __forceinline__ double normalise(double g, const PotDevice& pd, size_t k) {
  return (g - pd.shift[k]) * pd.scale[k];
}
__device__ __forceinline__ float normalise(float g, const PotDevice& pd, size_t k) {
  const float2 sh = pd.shift2[k];
  return ((g - sh.x) - sh.y) * pd.scale32[k];
}

__device__ __forceinline__ int warp_max(int v) {
  return __reduce_max_sync(0xffffffffu, v);
}

template <int LPA, typename T>
__device__ __forceinline__ T gsum(T v) {
#pragma unroll
  for (int d = LPA / 2; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

// Sums of N values per lane over a group of 2 D lanes, scattered: every lane
// ends with some of the sums and hands them to sink(index, sum).
template <int N, int D, typename T, int V, typename Sink>
__device__ __forceinline__ void reduce_scatter(T (&v)[V], int sl, int off, int lim, Sink sink) {
  if constexpr (D == 0) {
#pragma unroll
    for (int q = 0; q < N; ++q)
      if (q < lim) sink(off + q, v[q]);
  } else {
    constexpr int H = (N + 1) / 2;
    const bool up = sl & D;
#pragma unroll
    for (int q = 0; q < H; ++q) {
      const T hi = q + H < N ? v[q + H] : T(0);
      const T give = up ? v[q] : hi, keep = up ? hi : v[q];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, give, D);
    }
    reduce_scatter<H, D / 2>(v, sl, off + (up ? H : 0), up ? lim - H : min(lim, H), sink);
  }
}

// sum_q c_q T_q(x) and sum_q c'_q T_q(x), tab[q] = (c_q, c'_q); the
// derivative's last coefficient is zero.  (Two entries per load were slower in
// FP32: 541 against 477 us for the adjoint of 256,000 Cu/Au atoms.)
template <int N, bool GUARD, typename T>
__device__ __forceinline__ void series(const typename Num<T>::v2* tab, T x, int n, T& A, T& B) {
  const T x2 = x + x;
  T tm1 = T(1), t0 = x;
  A = tab[0].x;
  B = tab[0].y;
#pragma unroll
  for (int q = 1; q < N; ++q) {
    if (!GUARD || q < n) {
      const typename Num<T>::v2 c = tab[q];
      A = fma(c.x, t0, A);
      if (q + 1 < N) {
        B = fma(c.y, t0, B);
        const T tn = fma(x2, t0, -tm1);
        tm1 = t0;
        t0 = tn;
      }
    }
  }
}

// Shared memory of one group (one atom): staged angular neighbours (unit
// vector and 1/d; fc and fc'; table slot and species), in the adjoint their
// sums (V, S) and radial term and the coefficient tables; in the moment form
// the moments and, in the adjoint, their tables.
// info: table slot << 5 | spin + 1 (adjoint, unit spins) << 3 | species
struct Layout {
  int sf, info, acc, rad, g, tab_r, tab_a, mom, bytes;
};
template <typename T>
__host__ __device__ inline Layout layout(int cap_a, int nsf_pad, int nt_tab, int R, int ncls, int A,
                                         bool adjoint, bool mom) {
  const int z = sizeof(T);
  Layout L;
  int o = 4 * z * cap_a;                       // su at 0
  // the sums start when the dE/dG row and the radial tables are done with
  L.acc = L.tab_r = o;
  L.g = o + 2 * z * nt_tab * R;
  if (adjoint) {
    const int early = 2 * z * nt_tab * R + z * nsf_pad, late = mom ? 0 : 4 * z * cap_a;
    o += ((early > late ? early : late) + 15) & ~15;
  }
  L.sf = o;
  o += 2 * z * cap_a;
  L.tab_a = o;
  if (adjoint && !mom) o += 2 * z * ncls * A;
  L.mom = o;
  if (mom) o += adjoint ? 2 * z * (ncls * A * A + A + 1) : z * (2 * A * A + 2);
  // FP32 keeps the radial term in the place of fc' and recomputes that
  L.rad = o;
  if (adjoint && z == 8) o += z * cap_a;
  L.info = o;
  o += 4 * cap_a;
  // 32 bytes past a multiple of 128: the groups of a warp read their tables at
  // the same offsets, which then lie in different banks
  L.bytes = ((o + 95) & ~127) + 32;
  return L;
}

template <typename T>
struct Group {
  using T4 = typename Num<T>::v4;
  using T2 = typename Num<T>::v2;
  T4 *su, *acc;
  T2 *sf, *tab_r, *tab_a;
  T *mom, *rad, *g;
  int* info;
  __device__ __forceinline__ Group(unsigned char* p, const Layout& L)
      : su((T4*)p), acc((T4*)(p + L.acc)), sf((T2*)(p + L.sf)), tab_r((T2*)(p + L.tab_r)),
        tab_a((T2*)(p + L.tab_a)), mom((T*)(p + L.mom)), rad((T*)(p + L.rad)), g((T*)(p + L.g)),
        info((int*)(p + L.info)) {}
};

// entries of the angular coefficient table: one, one per spin product -1 ..
// 1, or the two blocks
template <int SPIN>
__host__ __device__ constexpr int classes() {
  return SPIN == SPIN_NONE ? 1 : SPIN == SPIN_UNIT ? 3 : 2;
}

// Chebyshev series of a derivative: d/dx sum c_q T_q = sum c'_q T_q,
// c'_{q-1} = c'_{q+1} + 2 q c_q (halved at q = 1); tab[q] = (c_q, c'_q)
template <typename T2>
__device__ __forceinline__ void derivative_series(T2* tab, int n) {
  using T = decltype(tab->x);
  T d1 = 0, d2 = 0;   // c'_{q}, c'_{q+1}
  for (int q = n - 1; q >= 0; --q) {
    tab[q].y = q ? d1 : T(0.5) * d1;
    const T d0 = fma(T(2 * q), tab[q].x, d2);
    d2 = d1;
    d1 = d0;
  }
}

// The group's angular neighbours from raw rows (vector and distance in su):
// unit vectors, 1/d, fc and fc'
template <bool DERIV, int LPA, typename T>
__device__ __forceinline__ void prepare_angular(const Group<T>& w, int na, int sl, T Rc) {
  const T a = T(SFB_PI) / Rc;
  for (int k = sl; k < na; k += LPA) {
    typename Num<T>::v4 u = w.su[k];
    const T d = u.w, inv = recip(d);
    T fc, dfc = T(0);
    cutoff<DERIV && sizeof(T) == 8, false>(d, Rc, a, inv, fc, dfc);
    u.x *= inv;
    u.y *= inv;
    u.z *= inv;
    u.w = inv;
    w.su[k] = u;
    w.sf[k].x = fc;
    if (sizeof(T) == 8) w.sf[k].y = dfc;
  }
}

// radial term (dE_radial/dd) of a staged neighbour, and fc' of its angular
// cut-off
__device__ __forceinline__ void put_radial(const Group<double>& w, int k, double c) { w.rad[k] = c; }
__device__ __forceinline__ void put_radial(const Group<float>& w, int k, float c) { w.sf[k].y = c; }
__device__ __forceinline__ void get_radial(const Group<double>& w, int k, double, double, double& c,
                                           double& dfc) {
  c = w.rad[k];
  dfc = w.sf[k].y;
}
__device__ __forceinline__ void get_radial(const Group<float>& w, int k, float inv, float Rc,
                                           float& c, float& dfc) {
  c = w.sf[k].y;
  const float d = recip(inv);
  float fc;
  cutoff<true, false>(d, Rc, float(SFB_PI) / Rc, inv, fc, dfc);
}

// flattened circulant walk over the pairs (a, a + t mod na), t = 1 .. na/2
struct PairWalk {
  int a, t, p;
  __device__ __forceinline__ void start(int lane, int na) {
    a = lane;
    t = 1;
    p = lane;
    wrap(na);
  }
  __device__ __forceinline__ void wrap(int na) {
    while (a >= na && na > 0) {
      a -= na;
      ++t;
    }
  }
  __device__ __forceinline__ int partner(int na) const {
    const int k = a + t;
    return k >= na ? k - na : k;
  }
  __device__ __forceinline__ void advance(int na, int stride) {
    p += stride;
    a += stride;
    wrap(na);
  }
};

// spin weight of a pair with the reference's stale s_j (sfbasis.f90:514,
// 556): the member first in the reference's neighbour order contributes
// s_eff, the other its own spin
__device__ __forceinline__ float ordered_spin(const DescBuffers& b, int i, int sa, int sk,
                                              float spin_a, float spin_k) {
  const size_t rb = (size_t)i * b.cap;
  return b.nb_rank[rb + sa] < b.nb_rank[rb + sk] ? b.nb_seff[rb + sa] * spin_k
                                                 : b.nb_seff[rb + sk] * spin_a;
}

// Monic forms of the moment polynomials: q_l^m = n_lm x (monic polynomial of
// degree l - m in z), p_l = z p_{l-1} - beta_lm p_{l-2}.
template <typename T>
struct MonicConsts {
  T norm[AE_MOMA * AE_MOMA];          // by component k
  T beta[AE_MOMA][AE_MOMA];           // [l][m]
};
template <typename T>
__host__ __device__ constexpr MonicConsts<T> monic_consts() {
  MonicConsts<T> c{};
  for (int m = 0; m < AE_MOMA; ++m) {
    double lead = m == 0 ? 1.0 : cheb::mc_sqrt(2.0 / cheb::mc_fact(2 * m)) * cheb::mc_dfact(2 * m - 1);
    for (int l = m; l < AE_MOMA; ++l) {
      if (l == m + 1) lead *= cheb::mc_sqrt(2.0 * m + 1.0);
      if (l >= m + 2) {
        lead *= (2.0 * l - 1.0) / cheb::mc_sqrt((double)(l - m) * (l + m));
        // b_l lead_{l-2} / lead_l of the normalised recurrence
        c.beta[l][m] = (T)((double)(l + m - 1) * (l - m - 1) / ((2.0 * l - 1.0) * (2.0 * l - 3.0)));
      }
      const int k = l * l + (m ? 2 * m - 1 : 0);
      c.norm[k] = (T)lead;
      if (m) c.norm[k + 1] = (T)lead;
    }
  }
  return c;
}
static __constant__ MonicConsts<double> c_monic64 = monic_consts<double>();
static __constant__ MonicConsts<float> c_monic32 = monic_consts<float>();
template <typename T>
__device__ __forceinline__ const MonicConsts<T>& monic();
template <>
__device__ __forceinline__ const MonicConsts<double>& monic<double>() { return c_monic64; }
template <>
__device__ __forceinline__ const MonicConsts<float>& monic<float>() { return c_monic32; }

// M0 += w0 Y, M1 += w1 Y over all components up to degree L, unnormalised
template <int L, bool MULTI, typename T>
__device__ __forceinline__ void monic_accumulate(T x, T y, T z, T w0, T w1, T* M0, T* M1) {
  T cm = T(1), sm = T(0);
#pragma unroll
  for (int m = 0; m <= L; ++m) {
    if (m == 1) {
      cm = x;
      sm = y;
    } else if (m > 1) {
      const T cn = fma(x, cm, -y * sm);
      sm = fma(x, sm, y * cm);
      cm = cn;
    }
    const T c0 = m ? w0 * cm : w0, s0 = w0 * sm;
    const T c1 = m ? w1 * cm : w1, s1 = w1 * sm;
    T q1 = T(0), q2 = T(0);
#pragma unroll
    for (int l = m; l <= L; ++l) {
      T q = T(1);
      if (l == m + 1) q = z;
      else if (l == m + 2) q = fma(z, z, -monic<T>().beta[l][m]);
      else if (l > m + 2) q = fma(z, q1, -monic<T>().beta[l][m] * q2);
      q2 = q1;
      q1 = q;
      const int k = l * l + (m ? 2 * m - 1 : 0);
      M0[k] = l == m ? M0[k] + c0 : fma(q, c0, M0[k]);
      if (m) M0[k + 1] = l == m ? M0[k + 1] + s0 : fma(q, s0, M0[k + 1]);
      if (MULTI) {
        M1[k] = l == m ? M1[k] + c1 : fma(q, c1, M1[k]);
        if (m) M1[k + 1] = l == m ? M1[k + 1] + s1 : fma(q, s1, M1[k + 1]);
      }
    }
  }
}

// F = sum_k C_k Y_k(u) and the gradient of its polynomial extension; tab[k] =
// (C_k n_k, (l - m) C_k n_k)
template <int L, typename T>
__device__ __forceinline__ void monic_gradient(T x, T y, T z, const typename Num<T>::v2* tab, T& F,
                                               T& px, T& py, T& pz) {
  T E[L + 1];   // z derivatives' factors of the order before
  F = px = py = pz = T(0);
  T cm = T(1), sm = T(0), cb = T(0), sb = T(0);   // Re, Im (x + iy)^m and of the power before
#pragma unroll
  for (int m = 0; m <= L; ++m) {
    if (m > 0) {
      cb = cm;
      sb = sm;
      if (m == 1) {
        cm = x;
        sm = y;
      } else {
        cm = fma(x, cb, -y * sb);
        sm = fma(x, sb, y * cb);
      }
    }
    T gam = T(0), del = T(0), q1 = T(0), q2 = T(0);
#pragma unroll
    for (int l = m; l <= L; ++l) {
      T q = T(1);
      if (l == m + 1) q = z;
      else if (l == m + 2) q = fma(z, z, -monic<T>().beta[l][m]);
      else if (l > m + 2) q = fma(z, q1, -monic<T>().beta[l][m] * q2);
      q2 = q1;
      q1 = q;
      const int k = l * l + (m ? 2 * m - 1 : 0);
      const typename Num<T>::v2 C = tab[k];
      if (m == 0) {
        F = l ? fma(C.x, q, F) : C.x;
        E[l] = C.y;
      } else {
        const typename Num<T>::v2 S = tab[k + 1];
        gam = l == m ? C.x : fma(C.x, q, gam);
        del = l == m ? S.x : fma(S.x, q, del);
        pz = l == m ? pz + E[l] : fma(E[l], q, pz);
        if (l > m) E[l] = fma(C.y, cm, S.y * sm);
      }
    }
    if (m > 0) {
      F = fma(gam, cm, fma(del, sm, F));
      if (m == 1) {
        px += gam;
        py += del;
      } else {
        gam *= T(m);
        del *= T(m);
        px = fma(gam, cb, fma(del, sb, px));
        py = fma(del, cb, fma(-gam, sb, py));
      }
    }
  }
}

// Bulk prefetch of an atom's neighbour rows into L2 (one instruction per row,
// issued by the group's first lane): the radial rounds then wait on L2 instead
// of DRAM.  Rows start 16-byte aligned (the ELL capacity is a multiple of 32)
// and the sizes are rounded up to 16 bytes inside the row.  FP32 only: the
// FP64 kernels wait on their pipe.
__device__ __forceinline__ void prefetch_rows(const float4* vec, const int* jt, int n) {
  if (n <= 0) return;
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(vec)),
               "r"(16 * n)
               : "memory");
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(jt)),
               "r"((4 * n + 15) & ~15)
               : "memory");
}
__device__ __forceinline__ void prefetch_rows(const double4_32a*, const int*, int) {}

// the moment rows and the Legendre tables of a precision
template <typename T>
struct MomRows;
template <>
struct MomRows<float> {
  static __host__ __device__ __forceinline__ float* rows(const DescBuffers& b) { return b.M; }
  static __host__ __device__ __forceinline__ const float* q(const PotDevice& pd) { return pd.qleg; }
};
template <>
struct MomRows<double> {
  static __host__ __device__ __forceinline__ double* rows(const DescBuffers& b) { return b.M64; }
  static __host__ __device__ __forceinline__ const double* q(const PotDevice& pd) { return pd.qleg64; }
};

// warps per block (they share only the spin table) and the resident blocks
// asked of the register allocator: FP64 leaves it to one-warp blocks, which
// spread few atoms evenly; FP32 asks for the occupancy that its latencies need
// (256,000 Cu/Au atoms: forward 279, 250, 239 and 241 us at 5, 6, 7 and 8
// blocks, adjoint 477 and 487 us at 6 and 7; 4,096 Li/Si/O cells: forward 494,
// 480 and 501 us at 6, 7 and 8)
template <typename T>
constexpr int max_threads() {
  return sizeof(T) == 8 ? 32 : 128;
}
template <typename T, int R, int A, int SPIN, bool MOM>
constexpr int fwd_blocks() {
  return sizeof(T) == 8 ? 1 : MOM ? (A <= 5 ? 7 : 3) : R <= 17 ? 7 : 4;
}
template <typename T>
constexpr int adj_blocks() {
  return sizeof(T) == 8 ? 1 : 6;
}

// ----------------------------------------------------------------------
// forward
// ----------------------------------------------------------------------
template <typename T, int R, int A, int LPA, bool GUARD, int SPIN, bool MOM>
__global__ void __launch_bounds__(max_threads<T>(), fwd_blocks<T, R, A, SPIN, MOM>())
    k_forward_rows(PotDevice pd, DescBuffers b) {
  using T4 = typename Num<T>::v4;
  using T2 = typename Num<T>::v2;
  constexpr int GPW = 32 / LPA;
  constexpr bool MULTI = SPIN != SPIN_NONE;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  __shared__ float s_spin[AE_MAXT * AE_MAXT];
  wait_for_previous();
  const int lane = threadIdx.x & 31, grp = lane / LPA, sl = lane % LPA;
  if (MULTI) {
    for (int q = threadIdx.x; q < pd.ntypes * AE_MAXT; q += blockDim.x)
      s_spin[q] = pd.sp[q / AE_MAXT].cheb.spin[q % AE_MAXT];
    __syncthreads();
  }
  const Layout lay = layout<T>(b.cap_a, pd.nsf_pad, 0, R, 0, A, false, MOM);
  const Group<T> w(smem_raw + (size_t)(threadIdx.x / LPA) * lay.bytes, lay);
  const int first = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * GPW;
  if (first >= b.natoms) return;   // whole warp idle
  const int gid = first + grp;
  const bool active = gid < b.natoms;
  const int i = active ? gid : b.natoms - 1;
  const int ti = b.types[i];
  const ChebTable& ct = pd.sp[ti].cheb;
  const int n = active ? b.nb_cnt[i] : 0;
  const T4* __restrict__ vec =
      reinterpret_cast<const T4*>(b.nb_vec) + (size_t)i * b.cap;
  const int* __restrict__ jt = b.nb_jt + (size_t)i * b.cap;
  if (sl == 0) prefetch_rows(vec, jt, n);
  const int nloop = warp_max(n);
  const T r_Rc = T(ct.r_Rc), a_Rc = T(ct.a_Rc);
  const T two_over_rc = T(2) / r_Rc, r_a = T(SFB_PI) / r_Rc;
  const int rN = GUARD ? ct.r_N : R, aN = GUARD ? ct.a_N : A;
  const bool multi = MULTI && ct.multi;
  const unsigned gmask = (LPA == 32) ? 0xffffffffu : (((1u << LPA) - 1u) << (grp * LPA));

  if (b.zero_F && active && sl == 0) {
    T4 z;
    z.x = z.y = z.z = z.w = T(0);
    reinterpret_cast<T4*>(b.F)[i] = z;
  }

  // ---- radial terms, compaction of the angular neighbours
  T acc[MULTI ? 2 * R : R];
#pragma unroll
  for (int q = 0; q < (MULTI ? 2 * R : R); ++q) acc[q] = T(0);
  int na = 0;
  // the table row is read one iteration ahead (its load latency overlaps the
  // previous neighbour's work)
  T4 vn = far_row<T>();
  int qn = 0;
  if (sl < n) {
    vn = vec[sl];
    qn = jt[sl];
  }
  for (int base = 0; base < nloop; base += LPA) {
    const int j = base + sl;
    const T4 v = vn;
    const int t = qn >> AE_TYPE_SHIFT;
    vn = far_row<T>();
    qn = 0;
    if (j + LPA < n) {
      vn = vec[j + LPA];
      qn = jt[j + LPA];
    }
    const T d = v.w;
    const float s = MULTI ? s_spin[ti * AE_MAXT + t] : 0.f;
    if (d <= r_Rc && d > T(SFB_EPS)) {
      T fc, none;
      cutoff<false, false>(d, r_Rc, r_a, T(0), fc, none);
      const T x = fma(d, two_over_rc, T(-1)), x2 = x + x;
      T sfc = T(0);
      if (MULTI) sfc = (T)s * fc;
      T tm1 = T(1), t0 = x;
      acc[0] += fc;
      if (MULTI) acc[R] += sfc;
#pragma unroll
      for (int q = 1; q < R; ++q) {
        if (!GUARD || q < rN) {
          acc[q] = fma(fc, t0, acc[q]);
          if (MULTI) acc[R + q] = fma(sfc, t0, acc[R + q]);
          if (q + 1 < R) {
            const T tn = fma(x2, t0, -tm1);
            tm1 = t0;
            t0 = tn;
          }
        }
      }
    }
    const bool inA = d <= a_Rc && d >= T(SFB_EPS);
    const unsigned m = __ballot_sync(0xffffffffu, inA) & gmask;
    if (inA) {
      const int k = na + __popc(m & ((1u << lane) - 1u));
      if (k < b.cap_a) {
        w.su[k] = v;
        w.info[k] = (j << 5) | t;
      }
    }
    na += __popc(m);
  }
  if (na > b.cap_a) {
    if (sl == 0 && active) atomicOr(b.status, AE_ST_NB_OVERFLOW);
    na = b.cap_a;
  }
  const size_t nrow = (size_t)ti * pd.nsf_pad;
  T* G = reinterpret_cast<T*>(b.G) + (size_t)i * pd.nsf_pad;
  constexpr int NR = MULTI ? 2 * R : R;
  reduce_scatter<NR, LPA / 2>(acc, sl, 0, NR, [&](int q, T s) {
    const bool spin = MULTI && q >= R;
    const int f = spin ? q - R : q;
    if (active && f < rN && (!spin || multi)) {
      const int k = (spin ? ct.r_i2 : ct.r_i1) + f;
      G[k] = normalise(s, pd, nrow + k);
    }
  });
  __syncwarp();
  prepare_angular<false, LPA, T>(w, na, sl, a_Rc);
  __syncwarp();

  // ---- angular terms
  if constexpr (MOM) {
    constexpr int K = A * A, NV = MULTI ? 2 * K + 2 : K + 1;
    T M[NV];   // plain moments, sum of w^2, then the spin block's
#pragma unroll
    for (int k = 0; k < NV; ++k) M[k] = T(0);
    for (int a = sl; a < na; a += LPA) {
      const T4 u = w.su[a];
      const T fc = w.sf[a].x;
      T fs = T(0);
      if (MULTI) fs = fc * (T)s_spin[ti * AE_MAXT + (w.info[a] & 7)];
      monic_accumulate<A - 1, MULTI, T>(u.x, u.y, u.z, fc, fs, M, M + (MULTI ? K + 1 : 0));
      M[K] = fma(fc, fc, M[K]);
      if (MULTI) M[NV - 1] = fma(fs, fs, M[NV - 1]);
    }
    T* Mg = MomRows<T>::rows(b) + (size_t)i * b.mom_pad;
    T* sq = w.mom;
    reduce_scatter<NV, LPA / 2>(M, sl, 0, NV, [&](int q, T s) {
      const int blk = q > K ? 1 : 0, k = q - blk * (K + 1);
      if (k < K) {
        s *= monic<T>().norm[k];
        if (active) Mg[blk * K + k] = s;
        s *= s;
      }
      sq[q] = s;
    });
    __syncwarp();
    // G_n = 1/2 (sum_l q_nl p_l - T_n(x(1)) W), a lane per feature
    const T* ql = MomRows<T>::q(pd) + (size_t)ti * AE_MOMA * AE_MOMA;
    for (int f = sl; f < (MULTI ? 2 : 1) * A; f += LPA) {
      const int blk = f / A, nn = f - blk * A;
      const T* s = sq + blk * (K + 1);
      T g = T(0), t1 = T(0);
      for (int l = 0; l <= nn; ++l) {
        T p = T(0);
        for (int k = l * l; k < (l + 1) * (l + 1); ++k) p += s[k];
        g = fma(ql[nn * AE_MOMA + l], p, g);
        t1 += ql[nn * AE_MOMA + l];
      }
      if (active && (!blk || multi)) {
        const int k = (blk ? ct.a_i2 : ct.a_i1) + nn;
        G[k] = normalise(T(0.5) * fma(-t1, s[K], g), pd, nrow + k);
      }
    }
  } else {
    constexpr int NA = MULTI ? 2 * A : A;
    T ang[NA];
#pragma unroll
    for (int q = 0; q < NA; ++q) ang[q] = T(0);
    const int P = active ? na * (na - 1) / 2 : 0;
    PairWalk pw;
    pw.start(sl, na);
    for (; pw.p < P; pw.advance(na, LPA)) {
      const int a = pw.a, k = pw.partner(na);
      const T4 ua = w.su[a], uk = w.su[k];
      const T wt = w.sf[a].x * w.sf[k].x;
      T sw = T(0);
      if (MULTI) {
        const int ia = w.info[a], ik = w.info[k];
        const T sa = s_spin[ti * AE_MAXT + (ia & 7)], sk = s_spin[ti * AE_MAXT + (ik & 7)];
        T ss = sa * sk;
        if constexpr (GUARD) {
          if (b.nb_rank) ss = ordered_spin(b, i, ia >> 5, ik >> 5, sa, sk);
        }
        sw = ss * wt;
      }
      T x = ua.x * uk.x + ua.y * uk.y + ua.z * uk.z;
      if (ct.angular_legacy) x = fma(x, T(2.0 / SFB_PI), T(-1));
      const T x2 = x + x;
      T tm1 = T(1), t0 = x;
      ang[0] += wt;
      if (MULTI) ang[A] += sw;
#pragma unroll
      for (int q = 1; q < A; ++q) {
        if (!GUARD || q < aN) {
          ang[q] = fma(wt, t0, ang[q]);
          if (MULTI) ang[A + q] = fma(sw, t0, ang[A + q]);
          if (q + 1 < A) {
            const T tn = fma(x2, t0, -tm1);
            tm1 = t0;
            t0 = tn;
          }
        }
      }
    }
    __syncwarp();
    reduce_scatter<NA, LPA / 2>(ang, sl, 0, NA, [&](int q, T s) {
      const bool spin = MULTI && q >= A;
      const int f = spin ? q - A : q;
      if (active && f < aN && (!spin || multi)) {
        const int k = (spin ? ct.a_i2 : ct.a_i1) + f;
        G[k] = normalise(s, pd, nrow + k);
      }
    });
  }
}

// ----------------------------------------------------------------------
// adjoint
// ----------------------------------------------------------------------
__device__ __forceinline__ void add_force(double* F, int atom, double fx, double fy, double fz) {
  atomicAdd(F + 4 * (size_t)atom, fx);
  atomicAdd(F + 4 * (size_t)atom + 1, fy);
  atomicAdd(F + 4 * (size_t)atom + 2, fz);
}
__device__ __forceinline__ void add_force(float* F, int atom, float fx, float fy, float fz) {
  atomicAdd(reinterpret_cast<float4*>(F) + atom, make_float4(fx, fy, fz, 0.f));
}

// FP64 pair form, a warp per atom: the adjoint of an atom may be shared out
template <typename T, int LPA, bool MOM>
constexpr bool ADJ_PARTS = sizeof(T) == 8 && LPA == 32 && !MOM;

template <typename T, int R, int A, int LPA, bool GUARD, int SPIN, bool MOM>
__global__ void __launch_bounds__(max_threads<T>(), adj_blocks<T>())
    k_adjoint_rows(PotDevice pd, DescBuffers b) {
  using T4 = typename Num<T>::v4;
  using T2 = typename Num<T>::v2;
  constexpr int GPW = 32 / LPA;
  constexpr bool MULTI = SPIN != SPIN_NONE;
  constexpr int NC = classes<SPIN>();
  // blocks per atom: each takes some of the radial rounds and pair steps
  constexpr bool PARTS = ADJ_PARTS<T, LPA, MOM>;
  const int part = PARTS ? blockIdx.y : 0, pmask = PARTS ? gridDim.y - 1 : 0;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  __shared__ float s_spin[AE_MAXT * AE_MAXT];
  wait_for_previous();
  const int lane = threadIdx.x & 31, grp = lane / LPA, sl = lane % LPA;
  if (MULTI) {
    for (int q = threadIdx.x; q < pd.ntypes * AE_MAXT; q += blockDim.x)
      s_spin[q] = pd.sp[q / AE_MAXT].cheb.spin[q % AE_MAXT];
    __syncthreads();
  }
  const int nt = MULTI ? pd.ntypes : 1;
  const Layout lay = layout<T>(b.cap_a, pd.nsf_pad, nt, R, NC, A, true, MOM);
  const Group<T> w(smem_raw + (size_t)(threadIdx.x / LPA) * lay.bytes, lay);
  const int first = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * GPW;
  if (first >= b.natoms) return;
  const int gid = first + grp;
  const bool active = gid < b.natoms;
  const int i = active ? gid : b.natoms - 1;
  const int ti = b.types[i];
  const ChebTable& ct = pd.sp[ti].cheb;
  const int n = active ? b.nb_cnt[i] : 0;
  const T4* __restrict__ vec =
      reinterpret_cast<const T4*>(b.nb_vec) + (size_t)i * b.cap;
  const int* __restrict__ jt = b.nb_jt + (size_t)i * b.cap;
  if (sl == 0) prefetch_rows(vec, jt, n);
  const int nloop = warp_max(n);
  const T r_Rc = T(ct.r_Rc), a_Rc = T(ct.a_Rc);
  const T two_over_rc = T(2) / r_Rc, r_a = T(SFB_PI) / r_Rc;
  const int rN = GUARD ? ct.r_N : R, aN = GUARD ? ct.a_N : A;
  const bool multi = MULTI && ct.multi;
  const unsigned gmask = (LPA == 32) ? 0xffffffffu : (((1u << LPA) - 1u) << (grp * LPA));
  const int sid = b.atom_struct[i];
  const T gs = b.grad_scale ? T(b.grad_scale[sid]) : T(1);
  const bool want_virial = b.virial != nullptr;
  T* F = reinterpret_cast<T*>(b.F);
  const T* gsrc = reinterpret_cast<const T*>(b.dEdG) + (size_t)i * pd.nsf_pad;
  for (int k = sl; k < ct.nsf; k += LPA) w.g[k] = gs * gsrc[k];
  __syncwarp();
  // coefficient tables: radial per neighbour species, angular per spin
  // product (or per block)
  for (int q = sl; q < nt * R; q += LPA) {
    const int t = q / R, f = q - t * R;
    T c = f < rN ? w.g[ct.r_i1 + f] : T(0);
    if (MULTI && multi && f < rN) c = fma((T)s_spin[ti * AE_MAXT + t], w.g[ct.r_i2 + f], c);
    w.tab_r[q].x = c;
  }
  if (!MOM)
    for (int q = sl; q < NC * A; q += LPA) {
      const int cl = q / A, f = q - cl * A;
      const T g0 = f < aN ? w.g[ct.a_i1 + f] : T(0);
      const T g1 = MULTI && multi && f < aN ? w.g[ct.a_i2 + f] : T(0);
      w.tab_a[q].x = SPIN == SPIN_NONE ? g0 : SPIN == SPIN_UNIT ? fma((T)(cl - 1), g1, g0)
                                                                : (cl ? g1 : g0);
    }
  __syncwarp();
  {
    // one lane per table (a group of eight lanes holds at most eight radial
    // tables and takes the angular ones in turn)
    if (sl < nt) derivative_series(w.tab_r + sl * R, R);
    if (!MOM && sl < NC) derivative_series(w.tab_a + sl * A, A);
  }
  __syncwarp();

  T fix = T(0), fiy = T(0), fiz = T(0);
  T w00 = 0, w01 = 0, w02 = 0, w10 = 0, w11 = 0, w12 = 0, w20 = 0, w21 = 0, w22 = 0;
  int na = 0;
  T4 vn = far_row<T>();
  int qn = 0;
  if (sl < n) {
    vn = vec[sl];
    qn = jt[sl];
  }
  for (int base = 0; base < nloop; base += LPA) {
    const int j = base + sl;
    const T4 v = vn;
    const int t = qn >> AE_TYPE_SHIFT, jatom = qn & AE_INDEX_MASK;
    vn = far_row<T>();
    qn = 0;
    if (j + LPA < n) {
      vn = vec[j + LPA];
      qn = jt[j + LPA];
    }
    const T d = v.w;
    const float s = SPIN == SPIN_UNIT ? s_spin[ti * AE_MAXT + t] : 0.f;
    T c = T(0);   // (dE/dd) / d
    const bool own = !PARTS || ((base / LPA) & pmask) == part;
    if (own && d <= r_Rc && d > T(SFB_EPS)) {
      const T inv = recip(d);
      T fc, dfc;   // dfc: fc' / d
      cutoff<true, true>(d, r_Rc, r_a, inv, fc, dfc);
      const T x = fma(d, two_over_rc, T(-1));
      const T2* tab = w.tab_r + (MULTI ? t * R : 0);
      T Av, Bv;
      series<R, GUARD, T>(tab, x, rN, Av, Bv);
      c = fma(dfc, Av, fc * two_over_rc * inv * Bv);
    }
    const bool inA = d <= a_Rc && d >= T(SFB_EPS);
    const unsigned m = __ballot_sync(0xffffffffu, inA) & gmask;
    bool staged = false;
    if (inA) {
      const int k = na + __popc(m & ((1u << lane) - 1u));
      if (k < b.cap_a) {
        w.su[k] = v;
        w.info[k] = (j << 5) | (SPIN == SPIN_UNIT ? ((int)s + 1) << 3 : 0) | t;
        put_radial(w, k, c * d);
        staged = true;
      }
    }
    if (!staged && c != T(0)) {
      // dE/dR_j = c R_ij: the force on j is minus that (staged neighbours
      // hand theirs over at the end)
      const T gx = c * v.x, gy = c * v.y, gz = c * v.z;
      fix += gx;
      fiy += gy;
      fiz += gz;
      add_force(F, jatom, -gx, -gy, -gz);
      if (want_virial) {
        w00 -= v.x * gx; w01 -= v.x * gy; w02 -= v.x * gz;
        w10 -= v.y * gx; w11 -= v.y * gy; w12 -= v.y * gz;
        w20 -= v.z * gx; w21 -= v.z * gy; w22 -= v.z * gz;
      }
    }
    na += __popc(m);
  }
  if (na > b.cap_a) {
    if (sl == 0 && active) atomicOr(b.status, AE_ST_NB_OVERFLOW);
    na = b.cap_a;
  }
  __syncwarp();
  prepare_angular<true, LPA, T>(w, na, sl, a_Rc);

  if constexpr (MOM) {
    // B_l = sum_n g_n q_nl, D = B M, and per spin the tables of
    // C = D0 + s D1 (times the monic norm), tau = sum_l B_l
    constexpr int K = A * A;
    T* Bl = w.mom + 2 * NC * K;   // B of both blocks, then tau of both
    const T* ql = MomRows<T>::q(pd) + (size_t)ti * AE_MOMA * AE_MOMA;
    for (int f = sl; f < 2 * A; f += LPA) {
      const int blk = f / A, l = f - blk * A;
      T s = T(0);
      if (!blk || multi)
        for (int nn = l; nn < A; ++nn)
          s = fma(w.g[(blk ? ct.a_i2 : ct.a_i1) + nn], ql[nn * AE_MOMA + l], s);
      Bl[f] = s;
    }
    __syncwarp();
    if (sl < 2) {
      T s = T(0);
      for (int l = 0; l < A; ++l) s += Bl[sl * A + l];
      Bl[2 * A + sl] = s;
    }
    const T* Mg = MomRows<T>::rows(b) + (size_t)i * b.mom_pad;
    T2* tab = reinterpret_cast<T2*>(w.mom);
    for (int k = sl; k < K; k += LPA) {
      int l = 0;
      while ((l + 1) * (l + 1) <= k) ++l;
      const int m = (k - l * l + 1) / 2;
      const T nk = monic<T>().norm[k], D0 = nk * Bl[l] * Mg[k];
      const T D1 = MULTI ? nk * Bl[A + l] * Mg[K + k] : T(0);
#pragma unroll
      for (int cl = 0; cl < NC; ++cl) {
        const T C = NC == 1 ? D0 : fma((T)(cl - 1), D1, D0);
        T2 e;
        e.x = C;
        e.y = T(l - m) * C;
        tab[cl * K + k] = e;
      }
    }
    __syncwarp();
    const T tau0 = Bl[2 * A], tau1 = Bl[2 * A + 1];
    for (int a = sl; a < na; a += LPA) {
      if (!active) break;
      const T4 u = w.su[a];
      const T fc = w.sf[a].x;
      T rad, dfc;
      get_radial(w, a, u.w, a_Rc, rad, dfc);
      const int info = w.info[a], slot = info >> 5;
      const T s = MULTI ? (T)s_spin[ti * AE_MAXT + (info & 7)] : T(0);
      T Fv, px, py, pz;
      monic_gradient<A - 1, T>(u.x, u.y, u.z, tab + (MULTI ? ((int)s + 1) * K : 0), Fv, px, py, pz);
      const T up = u.x * px + u.y * py + u.z * pz;
      const T wd = fc * u.w;
      const T tau = MULTI ? fma(tau1 * s, s, tau0) : tau0;
      const T cu = fma(dfc, fma(-tau, fc, Fv), fma(-wd, up, rad));
      const T fx = -fma(cu, u.x, wd * px), fy = -fma(cu, u.y, wd * py),
                   fz = -fma(cu, u.z, wd * pz);
      add_force(F, jt[slot] & AE_INDEX_MASK, fx, fy, fz);
      fix -= fx;
      fiy -= fy;
      fiz -= fz;
      if (want_virial) {
        const T4 v = vec[slot];
        w00 += v.x * fx; w01 += v.x * fy; w02 += v.x * fz;
        w10 += v.y * fx; w11 += v.y * fy; w12 += v.y * fz;
        w20 += v.z * fx; w21 += v.z * fy; w22 += v.z * fz;
      }
    }
  } else {
    for (int k = sl; k < na; k += LPA) {
      T4 o;
      o.x = o.y = o.z = o.w = T(0);
      w.acc[k] = o;
    }
    __syncwarp();
    const int P = active ? na * (na - 1) / 2 : 0;
    const int stride = max(1, min(LPA, na - 1));
    const int steps = warp_max((P + stride - 1) / stride);
    PairWalk pw;
    pw.start(sl, na);
    for (int q0 = 0; q0 < steps; ++q0, pw.advance(na, stride)) {
      if (PARTS && ((q0 + 1) & pmask) != part) continue;
      const bool live = sl < stride && pw.p < P;
      const int a = live ? pw.a : 0, k = live ? pw.partner(na) : 0;
      const T4 ua = w.su[a], uk = w.su[k];
      T Av = T(0), Bv = T(0);
      if (live) {
        T x = ua.x * uk.x + ua.y * uk.y + ua.z * uk.z;
        if (ct.angular_legacy) x = fma(x, T(2.0 / SFB_PI), T(-1));
        if constexpr (SPIN == SPIN_ANY) {
          const T x2 = x + x;
          T tm1 = T(1), t0 = x;
          const int ia = w.info[a], ik = w.info[k];
          const T sa = s_spin[ti * AE_MAXT + (ia & 7)], sk = s_spin[ti * AE_MAXT + (ik & 7)];
          T ss = sa * sk;
          if (b.nb_rank) ss = ordered_spin(b, i, ia >> 5, ik >> 5, sa, sk);
          const T2 *t0p = w.tab_a, *t1p = w.tab_a + A;
          T A1 = t1p[0].x, B1 = t1p[0].y;
          Av = t0p[0].x;
          Bv = t0p[0].y;
#pragma unroll
          for (int q = 1; q < A; ++q) {
            if (!GUARD || q < aN) {
              const T2 c0 = t0p[q], c1 = t1p[q];
              Av = fma(c0.x, t0, Av);
              A1 = fma(c1.x, t0, A1);
              Bv = fma(c0.y, t0, Bv);
              B1 = fma(c1.y, t0, B1);
              const T tn = fma(x2, t0, -tm1);
              tm1 = t0;
              t0 = tn;
            }
          }
          Av = fma(ss, A1, Av);
          Bv = fma(ss, B1, Bv);
        } else {
          const T2* tab = w.tab_a;
          if (SPIN == SPIN_UNIT) {
            const int ss = ((w.info[a] >> 3 & 3) - 1) * ((w.info[k] >> 3 & 3) - 1);
            tab += (ss + 1) * A;
          }
          series<A, GUARD, T>(tab, x, aN, Av, Bv);
        }
        const T fk = w.sf[k].x, cb = fk * Bv;
        T4 s = w.acc[a];
        s.x = fma(cb, uk.x, s.x);
        s.y = fma(cb, uk.y, s.y);
        s.z = fma(cb, uk.z, s.z);
        s.w = fma(fk, Av, s.w);
        w.acc[a] = s;
      }
      __syncwarp();
      if (live) {
        const T fa = w.sf[a].x, cb = fa * Bv;
        T4 s = w.acc[k];
        s.x = fma(cb, ua.x, s.x);
        s.y = fma(cb, ua.y, s.y);
        s.z = fma(cb, ua.z, s.z);
        s.w = fma(fa, Av, s.w);
        w.acc[k] = s;
      }
      __syncwarp();
    }
    // forces on the staged neighbours (radial + angular), one scatter each
    const T dxdc = ct.angular_legacy ? T(2.0 / SFB_PI) : T(1);
    for (int a = sl; a < na; a += LPA) {
      if (!active) break;
      const T4 u = w.su[a], V = w.acc[a];
      T rad, dfc;
      get_radial(w, a, u.w, a_Rc, rad, dfc);
      const int slot = w.info[a] >> 5;
      const T wd = w.sf[a].x * u.w * dxdc;
      const T vu = V.x * u.x + V.y * u.y + V.z * u.z;
      const T cu = fma(dfc, V.w, fma(-wd, vu, rad));
      const T fx = -fma(cu, u.x, wd * V.x), fy = -fma(cu, u.y, wd * V.y),
                   fz = -fma(cu, u.z, wd * V.z);
      add_force(F, jt[slot] & AE_INDEX_MASK, fx, fy, fz);
      fix -= fx;
      fiy -= fy;
      fiz -= fz;
      if (want_virial) {
        const T4 v = vec[slot];
        w00 += v.x * fx; w01 += v.x * fy; w02 += v.x * fz;
        w10 += v.y * fx; w11 += v.y * fy; w12 += v.y * fz;
        w20 += v.z * fx; w21 += v.z * fy; w22 += v.z * fz;
      }
    }
  }
  __syncwarp();
  fix = gsum<LPA>(fix);
  fiy = gsum<LPA>(fiy);
  fiz = gsum<LPA>(fiz);
  if (active && sl == 0) add_force(F, i, fix, fiy, fiz);
  if (want_virial) {
    T wv[9] = {w00, w01, w02, w10, w11, w12, w20, w21, w22};
    reduce_scatter<9, LPA / 2>(wv, sl, 0, 9, [&](int q, T s) {
      if (active) atomicAdd(b.virial + 9 * (size_t)sid + q, (double)s);
    });
  }
}

// Shared memory of one atom's group
template <typename T, int R, int A, int SPIN, bool MOM>
size_t group_smem(const PotDevice& pd, const DescBuffers& b, bool adjoint) {
  const int nt = SPIN == SPIN_NONE ? 1 : pd.ntypes;
  return (size_t)layout<T>(b.cap_a, pd.nsf_pad, nt, R, classes<SPIN>(), A, adjoint, MOM).bytes;
}

constexpr size_t SMEM_MAX = AE_SMEM_MAX;
// the FP32 adjoint in moment form is k_cheb_impl.cuh's, which keeps its
// coefficients in registers: 576 us for 4,096 Li/Si/O cells against 625 us
// with the tables of this file's and 620 us with registers in it
template <typename T, bool MOM>
constexpr bool HAS_ADJOINT = sizeof(T) == 8 || !MOM;
// the unguarded forward of SPIN_UNIT takes any spins (launch_spin)
template <bool GUARD, int SPIN>
constexpr bool HAS_FORWARD = GUARD || SPIN != SPIN_ANY;

template <typename T, int R, int A, int LPA, bool GUARD, int SPIN, bool MOM>
int launch_lanes(const PotDevice& pd, const DescBuffers& b, bool adjoint, int warps, int parts,
                 cudaStream_t s) {
  const int atoms = warps * (32 / LPA);
  const size_t smem = group_smem<T, R, A, SPIN, MOM>(pd, b, adjoint) * atoms;
  if (smem > SMEM_MAX) return (int)cudaErrorInvalidValue;
  const int blocks = (b.natoms + atoms - 1) / atoms;
  void (*kern)(PotDevice, DescBuffers) = nullptr;
  if constexpr (HAS_FORWARD<GUARD, SPIN>) {
    if (!adjoint) kern = k_forward_rows<T, R, A, LPA, GUARD, SPIN, MOM>;
  }
  if constexpr (HAS_ADJOINT<T, MOM>) {
    if (adjoint) kern = k_adjoint_rows<T, R, A, LPA, GUARD, SPIN, MOM>;
  }
  if (!kern) return (int)cudaErrorInvalidValue;
  allow_smem(kern, smem, SMEM_MAX);
  const int split = adjoint && ADJ_PARTS<T, LPA, MOM> ? parts : 1;
  launch_next(kern, dim3(blocks, split), 32 * warps, smem, s, pd, b);
  return (int)cudaGetLastError();
}

// Lanes per atom, as asked or by the number of atoms: 8 use every lane best (a
// whole number of rounds over the neighbours, cheap group sums), 32 spread few
// atoms over more SMs (one warp each) and take rows too long for several
// groups' shared memory.  Whole FP64 passes with 32, 16 and 8 lanes: 864 Au/Cu
// atoms 148, 158 and 217 us; 1,176 168, 165 and 224; 1,792 239, 222 and 253;
// 2,772 361, 331 and 337; 4,840 Cu/Au atoms 541, 464 and 442.  Hence below 8
// atoms per SM 32, below 20 16.  The moment form in FP32 follows the same line
// (864 Au/Cu atoms 56, 59 and 65 us; 2,304 71, 64 and 69; 4,000 84, 81 and 73);
// its pair sums, whose warps wait for the longest of their rows, gain from more
// lanes for longer: 2,048 Cu/Au atoms 58, 59 and 66 us, 2,304 Cu atoms 55, 56 and
// 62, 3,240 69, 67 and 74, 5,324 86, 80 and 84, 6,336 81, 77 and 79, 7,488 100, 96
// and 94, hence 32 below 16 atoms per SM and 16 below 42.
template <typename T, int R, int A, bool GUARD, int SPIN, bool MOM>
int launch(const PotDevice& pd, const DescBuffers& b, bool adjoint, cudaStream_t s) {
  int dev = 0, nsm = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  // long rows leave room for few warps on an SM, and few warps wait for each
  // other's latencies: groups share a warp while 16 warps (FP64 8) still fit (as
  // asked: while one does).  21,658 atoms of 64 neighbours, nearly all angular,
  // mixed, descriptor and adjoint with 8, 16 and 32 lanes (24, 12 and 6 KB a
  // warp): 619 + 725, - + 449 and 404 + 377 us
  const size_t one = group_smem<T, R, A, SPIN, MOM>(pd, b, true);
  const size_t room = b.lpa ? SMEM_MAX : SMEM_MAX / (sizeof(T) == 4 ? 16 : 8);
  constexpr bool PAIRS32 = sizeof(T) == 4 && !MOM;
  constexpr int LINE16 = PAIRS32 ? 16 : 8, LINE8 = PAIRS32 ? 42 : 20;   // atoms per SM
  int lanes = b.lpa ? b.lpa : b.natoms >= LINE8 * nsm ? 8 : b.natoms >= LINE16 * nsm ? 16 : 32;
  while (lanes < 32 && 32 / lanes * one > room) lanes *= 2;
  // four warps per block once they fill the SMs (FP32)
  const int warps = sizeof(T) == 4 && b.natoms >= 64 * nsm && 16 * one <= SMEM_MAX / 3 ? 4 : 1;
  if (lanes == 8) return launch_lanes<T, R, A, 8, GUARD, SPIN, MOM>(pd, b, adjoint, warps, 1, s);
  if (lanes == 16) return launch_lanes<T, R, A, 16, GUARD, SPIN, MOM>(pd, b, adjoint, 1, 1, s);
  // Blocks per atom in the FP64 pair adjoint: a scheduler starts one FP64
  // instruction in 64 cycles, so that up to two atoms an SM leave it waiting
  // on their chains.  Adjoint with 1, 2 and 4 (us): 108 atoms 35.8, 25.6 and
  // 21.5, 256 36.9, 28.7 and 28.6, 400 36.9, 34.8 and 41.0, 500 36.9, 36.9
  // and 45.0, 864 49.1, 57.3 and 75.8.  A single row keeps one block: its
  // neighbours' forces are one addition each, the same bits every time.
  const int parts = b.natoms == 1 ? 1 : b.natoms <= nsm ? 4 : 2 * b.natoms <= 5 * nsm ? 2 : 1;
  return launch_lanes<T, R, A, 32, GUARD, SPIN, MOM>(pd, b, adjoint, 1, parts, s);
}

// (the forward takes any spins in its SPIN_UNIT instance)
template <typename T, int R, int A, bool MOM>
int launch_spin(const PotDevice& pd, const DescBuffers& b, int spin, bool adjoint, cudaStream_t s) {
  if (spin == SPIN_NONE) return launch<T, R, A, false, SPIN_NONE, MOM>(pd, b, adjoint, s);
  if constexpr (!MOM) {
    if (adjoint && spin == SPIN_ANY)
      return launch<T, R, A, false, SPIN_ANY, false>(pd, b, adjoint, s);
  }
  return launch<T, R, A, false, SPIN_UNIT, MOM>(pd, b, adjoint, s);
}

// common sizes and spin range of a set of potentials
struct Sizes {
  int rN = 0, aN = 0, spin = SPIN_NONE;
  bool same = true;
};
inline Sizes sizes(const PotDevice& pd) {
  Sizes z;
  for (int t = 0; t < pd.ntypes; ++t) {
    const ChebTable& ct = pd.sp[t].cheb;
    if (t > 0 && (ct.r_N != z.rN || ct.a_N != z.aN)) z.same = false;
    z.rN = max(z.rN, ct.r_N);
    z.aN = max(z.aN, ct.a_N);
    if (!ct.multi) continue;
    z.spin = max(z.spin, (int)SPIN_UNIT);
    for (int q = 0; q < pd.ntypes; ++q)
      if (ct.spin[q] < -1.f || ct.spin[q] > 1.f) z.spin = SPIN_ANY;
  }
  return z;
}
inline bool exact(const Sizes& z, const DescBuffers& b) {
  return z.same && !b.nb_rank;
}
// whether the potentials have a moment form: an instantiated size, and in
// FP64 spins that the adjoint's tables cover
template <typename T>
bool moment_sizes(const Sizes& z) {
  if (!z.same || (sizeof(T) == 8 && z.spin == SPIN_ANY)) return false;
  return (z.rN == 11 && z.aN == 5) || (z.rN == 17 && z.aN == 5) ||
         (sizeof(T) == 4 && z.rN == 13 && z.aN == 7);
}
// whether the angular terms of a pass take it: there is a moment buffer, and
// every neighbour carries its own spin
template <typename T>
bool moment_form(const PotDevice& pd, const DescBuffers& b) {
  const Sizes z = sizes(pd);
  return moment_sizes<T>(z) && !b.nb_rank && MomRows<T>::rows(b) && MomRows<T>::q(pd) &&
         b.mom_pad >= 2 * z.aN * z.aN;
}

// The instances for a set of potentials: exact ones for the common (radial,
// angular) sizes, guarded ones for everything else.
template <typename T>
int dispatch_rows(const PotDevice& pd, const DescBuffers& b, bool adjoint, cudaStream_t s) {
  const Sizes z = sizes(pd);
  const bool mom = moment_form<T>(pd, b);
  if (exact(z, b)) {
    if (z.rN == 11 && z.aN == 5)
      return mom ? launch_spin<T, 11, 5, true>(pd, b, z.spin, adjoint, s)
                 : launch_spin<T, 11, 5, false>(pd, b, z.spin, adjoint, s);
    if (z.rN == 17 && z.aN == 5)
      return mom ? launch_spin<T, 17, 5, true>(pd, b, z.spin, adjoint, s)
                 : launch_spin<T, 17, 5, false>(pd, b, z.spin, adjoint, s);
    if (z.rN == 13 && z.aN == 7) {
      if constexpr (sizeof(T) == 4) {
        if (mom) return launch_spin<T, 13, 7, true>(pd, b, z.spin, adjoint, s);
      }
      return launch_spin<T, 13, 7, false>(pd, b, z.spin, adjoint, s);
    }
    if (z.rN == 17 && z.aN == 9) return launch_spin<T, 17, 9, false>(pd, b, z.spin, adjoint, s);
  }
  if (z.rN <= 24 && z.aN <= 16) return launch<T, 24, 16, true, SPIN_ANY, false>(pd, b, adjoint, s);
  if (z.rN <= 32 && z.aN <= 32) return launch<T, 32, 32, true, SPIN_ANY, false>(pd, b, adjoint, s);
  return (int)cudaErrorInvalidValue;
}

}  // namespace chebr
