// FP64 Chebyshev descriptor and adjoint (the plain path; the formulas and
// the feature layout are those of k_cheb_impl.cuh).
//
// The FP64 pipe of this GPU takes two lanes per clock and SM, 64 times fewer
// than FP32, and bounds these kernels (85 % busy); loads, shared memory and
// integer work run beside it for free.  So the work is arranged for few FP64
// instructions, each with all its lanes in use:
//   * the cut-off is a series in r^2 (no square root, sine or division:
//     14 multiply-adds for fc, 13 more for fc');
//   * reciprocals by Newton steps from an FP32 seed;
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
//   * angular orders up to 4 (where the moments fit the registers) use the
//     moment form of k_cheb_mom.cuh with monic polynomials: linear in the
//     angular neighbours.
// Measured, pair sums with two lanes' rows per warp before and now: 512 Li/Si/O
// cells (72,513 atoms, 72 neighbours, 21 angular) forward 2481 -> 1138 us,
// adjoint 4527 -> 1516 us; 2,765 Au/Cu atoms forward 144 -> 80 us, adjoint
// 323 -> 109 us.  The error against 64-bit automatic differentiation is that
// of the pair sums (1.6e-14 of the forces of the batch, 1.7e-14 before).
#pragma once
#include "common.h"
#include "cutoff64.cuh"
#include "k_cheb_mom.cuh"

namespace cheb64 {

constexpr double SFB_PI = 3.14159265358979;   // sfbasis.f90:72
constexpr double SFB_EPS = 1.0e-12;

// spin weights of the neighbours: none (single species), all within -1 .. 1
// (tables per spin), any
enum { SPIN_NONE = 0, SPIN_UNIT = 1, SPIN_ANY = 2 };

// 1 / d by Newton's iteration from an FP32 seed (relative error 2^-23, then
// 2^-46, then rounding)
__device__ __forceinline__ double recip(double d) {
  float f;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"((float)d));
  double y = (double)f;
  y = fma(y, fma(-d, y, 1.0), y);
  return fma(y, fma(-d, y, 1.0), y);
}

__device__ __forceinline__ int warp_max(int v) {
  return __reduce_max_sync(0xffffffffu, v);
}

template <int LPA>
__device__ __forceinline__ double gsum(double v) {
#pragma unroll
  for (int d = LPA / 2; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

// Sums of N values per lane over a group of 2 D lanes, scattered: every lane
// ends with some of the sums and hands them to sink(index, sum).
template <int N, int D, int V, typename Sink>
__device__ __forceinline__ void reduce_scatter(double (&v)[V], int sl, int off, int lim, Sink sink) {
  if constexpr (D == 0) {
#pragma unroll
    for (int q = 0; q < N; ++q)
      if (q < lim) sink(off + q, v[q]);
  } else {
    constexpr int H = (N + 1) / 2;
    const bool up = sl & D;
#pragma unroll
    for (int q = 0; q < H; ++q) {
      const double hi = q + H < N ? v[q + H] : 0.0;
      const double give = up ? v[q] : hi, keep = up ? hi : v[q];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, give, D);
    }
    reduce_scatter<H, D / 2>(v, sl, off + (up ? H : 0), up ? lim - H : min(lim, H), sink);
  }
}

// Shared memory of one group (one atom): staged angular neighbours (unit
// vector and 1/d; fc and fc'; table slot and species), in the adjoint their
// sums (V, S) and radial term and the coefficient tables; in the moment form
// the moments and, in the adjoint, their tables.
struct Layout {
  int sf, info, acc, rad, g, tab_r, tab_a, mom, bytes;
};
__host__ __device__ inline Layout layout(int cap_a, int nsf_pad, int nt_tab, int R, int ncls, int A,
                                         bool adjoint, bool mom) {
  Layout L;
  int o = 32 * cap_a;                       // su at 0
  L.acc = o;
  if (adjoint) o += 32 * cap_a;
  L.sf = o;
  o += 16 * cap_a;
  L.tab_r = o;
  if (adjoint) o += 16 * nt_tab * R;
  L.tab_a = o;
  if (adjoint && !mom) o += 16 * ncls * A;
  L.mom = o;
  if (mom) o += adjoint ? 16 * ncls * A * A + 16 * A + 16 : 8 * (2 * A * A + 2);
  L.rad = o;
  if (adjoint) o += 8 * cap_a;
  L.g = o;
  if (adjoint) o += 8 * nsf_pad;
  L.info = o;
  o += 4 * cap_a;
  L.bytes = (o + 31) & ~31;
  return L;
}

struct Group {
  double4_32a *su, *acc;
  double2* sf;
  double2 *tab_r, *tab_a;
  double *mom, *rad, *g;
  int* info;
  __device__ __forceinline__ Group(unsigned char* p, const Layout& L)
      : su((double4_32a*)p), acc((double4_32a*)(p + L.acc)), sf((double2*)(p + L.sf)),
        tab_r((double2*)(p + L.tab_r)), tab_a((double2*)(p + L.tab_a)), mom((double*)(p + L.mom)),
        rad((double*)(p + L.rad)), g((double*)(p + L.g)), info((int*)(p + L.info)) {}
};

// entries of the angular coefficient table: one, one per spin product -1 ..
// 1, or the two blocks
template <int SPIN>
__host__ __device__ constexpr int classes() {
  return SPIN == SPIN_NONE ? 1 : SPIN == SPIN_UNIT ? 3 : 2;
}

// Chebyshev series of a derivative: d/dx sum c_q T_q = sum c'_q T_q,
// c'_{q-1} = c'_{q+1} + 2 q c_q (halved at q = 1); tab[q] = (c_q, c'_q)
__device__ __forceinline__ void derivative_series(double2* tab, int n) {
  double d1 = 0.0, d2 = 0.0;   // c'_{q}, c'_{q+1}
  for (int q = n - 1; q >= 0; --q) {
    tab[q].y = q ? d1 : 0.5 * d1;
    const double d0 = fma(2.0 * q, tab[q].x, d2);
    d2 = d1;
    d1 = d0;
  }
}

// The group's angular neighbours from raw rows (vector and distance in su):
// unit vectors, 1/d, fc and fc'
template <bool DERIV, int LPA>
__device__ __forceinline__ void prepare_angular(const Group& w, int na, int sl, double Rc) {
  const double a = SFB_PI / Rc, a2 = a * a;
  for (int k = sl; k < na; k += LPA) {
    double4_32a u = w.su[k];
    const double d = u.w, inv = recip(d);
    const double z = fma(a2 * d, d, -FC_Y0);
    double2 f;
    f.x = d < Rc ? fc_series(z) : 0.0;
    f.y = DERIV ? (d < Rc ? 2.0 * a2 * d * fc_series_d(z) : 0.0) : 0.0;
    u.x *= inv;
    u.y *= inv;
    u.z *= inv;
    u.w = inv;
    w.su[k] = u;
    w.sf[k] = f;
  }
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
__device__ __forceinline__ double ordered_spin(const DescBuffers& b, int i, int sa, int sk,
                                               double spin_a, double spin_k) {
  const size_t rb = (size_t)i * b.cap;
  return b.nb_rank[rb + sa] < b.nb_rank[rb + sk] ? (double)b.nb_seff[rb + sa] * spin_k
                                                 : (double)b.nb_seff[rb + sk] * spin_a;
}

// Monic forms of the moment polynomials: q_l^m = n_lm x (monic polynomial of
// degree l - m in z), p_l = z p_{l-1} - beta_lm p_{l-2}.
struct MonicConsts {
  double norm[AE_MOMA * AE_MOMA];          // by component k
  double beta[AE_MOMA][AE_MOMA];           // [l][m]
};
__host__ __device__ constexpr MonicConsts monic_consts() {
  MonicConsts c{};
  for (int m = 0; m < AE_MOMA; ++m) {
    double lead = m == 0 ? 1.0 : cheb::mc_sqrt(2.0 / cheb::mc_fact(2 * m)) * cheb::mc_dfact(2 * m - 1);
    for (int l = m; l < AE_MOMA; ++l) {
      if (l == m + 1) lead *= cheb::mc_sqrt(2.0 * m + 1.0);
      if (l >= m + 2) {
        lead *= (2.0 * l - 1.0) / cheb::mc_sqrt((double)(l - m) * (l + m));
        // b_l lead_{l-2} / lead_l of the normalised recurrence
        c.beta[l][m] = (double)(l + m - 1) * (l - m - 1) / ((2.0 * l - 1.0) * (2.0 * l - 3.0));
      }
      const int k = l * l + (m ? 2 * m - 1 : 0);
      c.norm[k] = lead;
      if (m) c.norm[k + 1] = lead;
    }
  }
  return c;
}
static __constant__ MonicConsts c_monic = monic_consts();

// M0 += w0 Y, M1 += w1 Y over all components up to degree L, unnormalised
template <int L, bool MULTI>
__device__ __forceinline__ void monic_accumulate(double x, double y, double z, double w0, double w1,
                                                 double* M0, double* M1) {
  double cm = 1.0, sm = 0.0;
#pragma unroll
  for (int m = 0; m <= L; ++m) {
    if (m == 1) {
      cm = x;
      sm = y;
    } else if (m > 1) {
      const double cn = fma(x, cm, -y * sm);
      sm = fma(x, sm, y * cm);
      cm = cn;
    }
    const double c0 = m ? w0 * cm : w0, s0 = w0 * sm;
    const double c1 = m ? w1 * cm : w1, s1 = w1 * sm;
    double q1 = 0.0, q2 = 0.0;
#pragma unroll
    for (int l = m; l <= L; ++l) {
      double q = 1.0;
      if (l == m + 1) q = z;
      else if (l == m + 2) q = fma(z, z, -c_monic.beta[l][m]);
      else if (l > m + 2) q = fma(z, q1, -c_monic.beta[l][m] * q2);
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
template <int L>
__device__ __forceinline__ void monic_gradient(double x, double y, double z, const double2* tab,
                                               double& F, double& px, double& py, double& pz) {
  double E[L + 1];   // z derivatives' factors of the order before
  F = px = py = pz = 0.0;
  double cm = 1.0, sm = 0.0, cb = 0.0, sb = 0.0;   // Re, Im (x + iy)^m and of the power before
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
    double gam = 0.0, del = 0.0, q1 = 0.0, q2 = 0.0;
#pragma unroll
    for (int l = m; l <= L; ++l) {
      double q = 1.0;
      if (l == m + 1) q = z;
      else if (l == m + 2) q = fma(z, z, -c_monic.beta[l][m]);
      else if (l > m + 2) q = fma(z, q1, -c_monic.beta[l][m] * q2);
      q2 = q1;
      q1 = q;
      const int k = l * l + (m ? 2 * m - 1 : 0);
      const double2 C = tab[k];
      if (m == 0) {
        F = l ? fma(C.x, q, F) : C.x;
        E[l] = C.y;
      } else {
        const double2 S = tab[k + 1];
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
        gam *= (double)m;
        del *= (double)m;
        px = fma(gam, cb, fma(del, sb, px));
        py = fma(del, cb, fma(-gam, sb, py));
      }
    }
  }
}

// ----------------------------------------------------------------------
// forward
// ----------------------------------------------------------------------
template <int R, int A, int LPA, bool GUARD, int SPIN, bool MOM>
__global__ void __launch_bounds__(32) k_forward64(PotDevice pd, DescBuffers b) {
  constexpr int GPW = 32 / LPA;
  constexpr bool MULTI = SPIN != SPIN_NONE;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  __shared__ float s_spin[AE_MAXT * AE_MAXT];
  const int lane = threadIdx.x, grp = lane / LPA, sl = lane % LPA;
  if (MULTI)
    for (int q = lane; q < pd.ntypes * AE_MAXT; q += 32)
      s_spin[q] = pd.sp[q / AE_MAXT].cheb.spin[q % AE_MAXT];
  __syncwarp();
  const Layout lay = layout(b.cap_a, pd.nsf_pad, 0, R, 0, A, false, MOM);
  const Group w(smem_raw + (size_t)grp * lay.bytes, lay);
  const int gid = blockIdx.x * GPW + grp;
  const bool active = gid < b.natoms;
  const int i = active ? gid : b.natoms - 1;
  const int ti = b.types[i];
  const ChebTable& ct = pd.sp[ti].cheb;
  const int n = active ? b.nb_cnt[i] : 0;
  const double4_32a* __restrict__ vec =
      reinterpret_cast<const double4_32a*>(b.nb_vec) + (size_t)i * b.cap;
  const int* __restrict__ jt = b.nb_jt + (size_t)i * b.cap;
  const int nloop = warp_max(n);
  const double r_Rc = ct.r_Rc, a_Rc = ct.a_Rc;
  const double two_over_rc = 2.0 / r_Rc, r_a = SFB_PI / r_Rc, r_a2 = r_a * r_a;
  const int rN = GUARD ? ct.r_N : R, aN = GUARD ? ct.a_N : A;
  const bool multi = MULTI && ct.multi;
  const unsigned gmask = (LPA == 32) ? 0xffffffffu : (((1u << LPA) - 1u) << (grp * LPA));

  if (b.zero_F && active && sl == 0) {
    double4_32a z;
    z.x = z.y = z.z = z.w = 0.0;
    reinterpret_cast<double4_32a*>(b.F)[i] = z;
  }

  // ---- radial terms, compaction of the angular neighbours
  double acc[MULTI ? 2 * R : R];
#pragma unroll
  for (int q = 0; q < (MULTI ? 2 * R : R); ++q) acc[q] = 0.0;
  int na = 0;
  for (int base = 0; base < nloop; base += LPA) {
    const int j = base + sl;
    double4_32a v;
    v.x = v.y = v.z = 0.0;
    v.w = 1e30;
    int t = 0;
    if (j < n) {
      v = vec[j];
      t = jt[j] >> AE_TYPE_SHIFT;
    }
    const double d = v.w;
    if (d <= r_Rc && d > SFB_EPS) {
      const double fc = d < r_Rc ? fc_series(fma(r_a2 * d, d, -FC_Y0)) : 0.0;
      const double x = fma(d, two_over_rc, -1.0), x2 = x + x;
      double sfc = 0.0;
      if (MULTI) sfc = (double)s_spin[ti * AE_MAXT + t] * fc;
      double tm1 = 1.0, t0 = x;
      acc[0] += fc;
      if (MULTI) acc[R] += sfc;
#pragma unroll
      for (int q = 1; q < R; ++q) {
        if (!GUARD || q < rN) {
          acc[q] = fma(fc, t0, acc[q]);
          if (MULTI) acc[R + q] = fma(sfc, t0, acc[R + q]);
          if (q + 1 < R) {
            const double tn = fma(x2, t0, -tm1);
            tm1 = t0;
            t0 = tn;
          }
        }
      }
    }
    const bool inA = d <= a_Rc && d >= SFB_EPS;
    const unsigned m = __ballot_sync(0xffffffffu, inA) & gmask;
    if (inA) {
      const int k = na + __popc(m & ((1u << lane) - 1u));
      if (k < b.cap_a) {
        w.su[k] = v;
        w.info[k] = (j << 3) | t;
      }
    }
    na += __popc(m);
  }
  if (na > b.cap_a) {
    if (sl == 0 && active) atomicOr(b.status, AE_ST_NB_OVERFLOW);
    na = b.cap_a;
  }
  const size_t nrow = (size_t)ti * pd.nsf_pad;
  double* G = reinterpret_cast<double*>(b.G) + (size_t)i * pd.nsf_pad;
  const double *shift = pd.shift + nrow, *scale = pd.scale + nrow;
  constexpr int NR = MULTI ? 2 * R : R;
  reduce_scatter<NR, LPA / 2>(acc, sl, 0, NR, [&](int q, double s) {
    const bool spin = MULTI && q >= R;
    const int f = spin ? q - R : q;
    if (active && f < rN && (!spin || multi)) {
      const int k = (spin ? ct.r_i2 : ct.r_i1) + f;
      G[k] = (s - shift[k]) * scale[k];
    }
  });
  __syncwarp();
  prepare_angular<false, LPA>(w, na, sl, a_Rc);
  __syncwarp();

  // ---- angular terms
  if constexpr (MOM) {
    constexpr int K = A * A, NV = MULTI ? 2 * K + 2 : K + 1;
    double M[NV];   // plain moments, sum of w^2, then the spin block's
#pragma unroll
    for (int k = 0; k < NV; ++k) M[k] = 0.0;
    for (int a = sl; a < na; a += LPA) {
      const double4_32a u = w.su[a];
      const double fc = w.sf[a].x;
      double fs = 0.0;
      if (MULTI) fs = fc * (double)s_spin[ti * AE_MAXT + (w.info[a] & 7)];
      monic_accumulate<A - 1, MULTI>(u.x, u.y, u.z, fc, fs, M, M + (MULTI ? K + 1 : 0));
      M[K] = fma(fc, fc, M[K]);
      if (MULTI) M[NV - 1] = fma(fs, fs, M[NV - 1]);
    }
    double* Mg = b.M64 + (size_t)i * b.mom_pad;
    double* sq = w.mom;
    reduce_scatter<NV, LPA / 2>(M, sl, 0, NV, [&](int q, double s) {
      const int blk = q > K ? 1 : 0, k = q - blk * (K + 1);
      if (k < K) {
        s *= c_monic.norm[k];
        if (active) Mg[blk * K + k] = s;
        s *= s;
      }
      sq[q] = s;
    });
    __syncwarp();
    // G_n = 1/2 (sum_l q_nl p_l - T_n(x(1)) W), a lane per feature
    const double* ql = pd.qleg64 + (size_t)ti * AE_MOMA * AE_MOMA;
    for (int f = sl; f < (MULTI ? 2 : 1) * A; f += LPA) {
      const int blk = f / A, nn = f - blk * A;
      const double* s = sq + blk * (K + 1);
      double g = 0.0, t1 = 0.0;
      for (int l = 0; l <= nn; ++l) {
        double p = 0.0;
        for (int k = l * l; k < (l + 1) * (l + 1); ++k) p += s[k];
        g = fma(ql[nn * AE_MOMA + l], p, g);
        t1 += ql[nn * AE_MOMA + l];
      }
      if (active && (!blk || multi)) {
        const int k = (blk ? ct.a_i2 : ct.a_i1) + nn;
        G[k] = (0.5 * fma(-t1, s[K], g) - shift[k]) * scale[k];
      }
    }
  } else {
    constexpr int NA = MULTI ? 2 * A : A;
    double ang[NA];
#pragma unroll
    for (int q = 0; q < NA; ++q) ang[q] = 0.0;
    const int P = active ? na * (na - 1) / 2 : 0;
    PairWalk pw;
    pw.start(sl, na);
    for (; pw.p < P; pw.advance(na, LPA)) {
      const int a = pw.a, k = pw.partner(na);
      const double4_32a ua = w.su[a], uk = w.su[k];
      const double wt = w.sf[a].x * w.sf[k].x;
      double sw = 0.0;
      if (MULTI) {
        const int ia = w.info[a], ik = w.info[k];
        const double sa = s_spin[ti * AE_MAXT + (ia & 7)], sk = s_spin[ti * AE_MAXT + (ik & 7)];
        double ss = sa * sk;
        if constexpr (GUARD) {
          if (b.nb_rank) ss = ordered_spin(b, i, ia >> 3, ik >> 3, sa, sk);
        }
        sw = ss * wt;
      }
      double x = ua.x * uk.x + ua.y * uk.y + ua.z * uk.z;
      if (ct.angular_legacy) x = fma(x, 2.0 / SFB_PI, -1.0);
      const double x2 = x + x;
      double tm1 = 1.0, t0 = x;
      ang[0] += wt;
      if (MULTI) ang[A] += sw;
#pragma unroll
      for (int q = 1; q < A; ++q) {
        if (!GUARD || q < aN) {
          ang[q] = fma(wt, t0, ang[q]);
          if (MULTI) ang[A + q] = fma(sw, t0, ang[A + q]);
          if (q + 1 < A) {
            const double tn = fma(x2, t0, -tm1);
            tm1 = t0;
            t0 = tn;
          }
        }
      }
    }
    __syncwarp();
    reduce_scatter<NA, LPA / 2>(ang, sl, 0, NA, [&](int q, double s) {
      const bool spin = MULTI && q >= A;
      const int f = spin ? q - A : q;
      if (active && f < aN && (!spin || multi)) {
        const int k = (spin ? ct.a_i2 : ct.a_i1) + f;
        G[k] = (s - shift[k]) * scale[k];
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

template <int R, int A, int LPA, bool GUARD, int SPIN, bool MOM>
__global__ void __launch_bounds__(32) k_adjoint64(PotDevice pd, DescBuffers b) {
  constexpr int GPW = 32 / LPA;
  constexpr bool MULTI = SPIN != SPIN_NONE;
  constexpr int NC = classes<SPIN>();
  extern __shared__ __align__(32) unsigned char smem_raw[];
  __shared__ float s_spin[AE_MAXT * AE_MAXT];
  const int lane = threadIdx.x, grp = lane / LPA, sl = lane % LPA;
  if (MULTI)
    for (int q = lane; q < pd.ntypes * AE_MAXT; q += 32)
      s_spin[q] = pd.sp[q / AE_MAXT].cheb.spin[q % AE_MAXT];
  const int nt = MULTI ? pd.ntypes : 1;
  const Layout lay = layout(b.cap_a, pd.nsf_pad, nt, R, NC, A, true, MOM);
  const Group w(smem_raw + (size_t)grp * lay.bytes, lay);
  const int gid = blockIdx.x * GPW + grp;
  const bool active = gid < b.natoms;
  const int i = active ? gid : b.natoms - 1;
  const int ti = b.types[i];
  const ChebTable& ct = pd.sp[ti].cheb;
  const int n = active ? b.nb_cnt[i] : 0;
  const double4_32a* __restrict__ vec =
      reinterpret_cast<const double4_32a*>(b.nb_vec) + (size_t)i * b.cap;
  const int* __restrict__ jt = b.nb_jt + (size_t)i * b.cap;
  const int nloop = warp_max(n);
  const double r_Rc = ct.r_Rc, a_Rc = ct.a_Rc;
  const double two_over_rc = 2.0 / r_Rc, r_a = SFB_PI / r_Rc, r_a2 = r_a * r_a;
  const int rN = GUARD ? ct.r_N : R, aN = GUARD ? ct.a_N : A;
  const bool multi = MULTI && ct.multi;
  const unsigned gmask = (LPA == 32) ? 0xffffffffu : (((1u << LPA) - 1u) << (grp * LPA));
  const int sid = b.atom_struct[i];
  const double gs = b.grad_scale ? b.grad_scale[sid] : 1.0;
  const bool want_virial = b.virial != nullptr;
  double* F = reinterpret_cast<double*>(b.F);
  const double* gsrc = reinterpret_cast<const double*>(b.dEdG) + (size_t)i * pd.nsf_pad;
  for (int k = sl; k < ct.nsf; k += LPA) w.g[k] = gs * gsrc[k];
  __syncwarp();
  // coefficient tables: radial per neighbour species, angular per spin
  // product (or per block)
  for (int q = sl; q < nt * R; q += LPA) {
    const int t = q / R, f = q - t * R;
    double c = f < rN ? w.g[ct.r_i1 + f] : 0.0;
    if (MULTI && multi && f < rN) c = fma((double)s_spin[ti * AE_MAXT + t], w.g[ct.r_i2 + f], c);
    w.tab_r[q].x = c;
  }
  if (!MOM)
    for (int q = sl; q < NC * A; q += LPA) {
      const int cl = q / A, f = q - cl * A;
      const double g0 = f < aN ? w.g[ct.a_i1 + f] : 0.0;
      const double g1 = MULTI && multi && f < aN ? w.g[ct.a_i2 + f] : 0.0;
      w.tab_a[q].x = SPIN == SPIN_NONE ? g0 : SPIN == SPIN_UNIT ? fma((double)(cl - 1), g1, g0)
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

  double fix = 0.0, fiy = 0.0, fiz = 0.0;
  double w00 = 0, w01 = 0, w02 = 0, w10 = 0, w11 = 0, w12 = 0, w20 = 0, w21 = 0, w22 = 0;
  int na = 0;
  for (int base = 0; base < nloop; base += LPA) {
    const int j = base + sl;
    double4_32a v;
    v.x = v.y = v.z = 0.0;
    v.w = 1e30;
    int t = 0, jatom = 0;
    if (j < n) {
      v = vec[j];
      const int q = jt[j];
      t = q >> AE_TYPE_SHIFT;
      jatom = q & AE_INDEX_MASK;
    }
    const double d = v.w;
    double c = 0.0;   // (dE/dd) / d
    if (d <= r_Rc && d > SFB_EPS) {
      const double z = fma(r_a2 * d, d, -FC_Y0);
      const bool in = d < r_Rc;
      const double fc = in ? fc_series(z) : 0.0;
      const double dfc = in ? 2.0 * r_a2 * fc_series_d(z) : 0.0;   // fc' / d
      const double x = fma(d, two_over_rc, -1.0), x2 = x + x;
      const double2* tab = w.tab_r + (MULTI ? t * R : 0);
      double tm1 = 1.0, t0 = x;
      double Av = tab[0].x, Bv = tab[0].y;
#pragma unroll
      for (int q = 1; q < R; ++q) {
        if (!GUARD || q < rN) {
          const double2 cq = tab[q];
          Av = fma(cq.x, t0, Av);
          if (q + 1 < R) {
            Bv = fma(cq.y, t0, Bv);
            const double tn = fma(x2, t0, -tm1);
            tm1 = t0;
            t0 = tn;
          }
        }
      }
      c = fma(dfc, Av, fc * two_over_rc * recip(d) * Bv);
    }
    const bool inA = d <= a_Rc && d >= SFB_EPS;
    const unsigned m = __ballot_sync(0xffffffffu, inA) & gmask;
    bool staged = false;
    if (inA) {
      const int k = na + __popc(m & ((1u << lane) - 1u));
      if (k < b.cap_a) {
        w.su[k] = v;
        w.info[k] = (j << 3) | t;
        w.rad[k] = c * d;
        staged = true;
      }
    }
    if (!staged && c != 0.0) {
      // dE/dR_j = c R_ij: the force on j is minus that (staged neighbours
      // hand theirs over at the end)
      const double gx = c * v.x, gy = c * v.y, gz = c * v.z;
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
  prepare_angular<true, LPA>(w, na, sl, a_Rc);

  if constexpr (MOM) {
    // B_l = sum_n g_n q_nl, D = B M, and per spin the tables of
    // C = D0 + s D1 (times the monic norm), tau = sum_l B_l
    constexpr int K = A * A;
    double* Bl = w.mom + 2 * NC * K;   // B of both blocks, then tau of both
    const double* ql = pd.qleg64 + (size_t)ti * AE_MOMA * AE_MOMA;
    for (int f = sl; f < 2 * A; f += LPA) {
      const int blk = f / A, l = f - blk * A;
      double s = 0.0;
      if (!blk || multi)
        for (int nn = l; nn < A; ++nn)
          s = fma(w.g[(blk ? ct.a_i2 : ct.a_i1) + nn], ql[nn * AE_MOMA + l], s);
      Bl[f] = s;
    }
    __syncwarp();
    if (sl < 2) {
      double s = 0.0;
      for (int l = 0; l < A; ++l) s += Bl[sl * A + l];
      Bl[2 * A + sl] = s;
    }
    const double* Mg = b.M64 + (size_t)i * b.mom_pad;
    double2* tab = reinterpret_cast<double2*>(w.mom);
    for (int k = sl; k < K; k += LPA) {
      int l = 0;
      while ((l + 1) * (l + 1) <= k) ++l;
      const int m = (k - l * l + 1) / 2;
      const double nk = c_monic.norm[k], D0 = nk * Bl[l] * Mg[k];
      const double D1 = MULTI ? nk * Bl[A + l] * Mg[K + k] : 0.0;
#pragma unroll
      for (int cl = 0; cl < NC; ++cl) {
        const double C = NC == 1 ? D0 : fma((double)(cl - 1), D1, D0);
        tab[cl * K + k] = make_double2(C, (double)(l - m) * C);
      }
    }
    __syncwarp();
    const double tau0 = Bl[2 * A], tau1 = Bl[2 * A + 1];
    for (int a = sl; a < na; a += LPA) {
      if (!active) break;
      const double4_32a u = w.su[a];
      const double2 f = w.sf[a];
      const int info = w.info[a], slot = info >> 3;
      const double s = MULTI ? (double)s_spin[ti * AE_MAXT + (info & 7)] : 0.0;
      double Fv, px, py, pz;
      monic_gradient<A - 1>(u.x, u.y, u.z, tab + (MULTI ? ((int)s + 1) * K : 0), Fv, px, py, pz);
      const double up = u.x * px + u.y * py + u.z * pz;
      const double wd = f.x * u.w;
      const double tau = MULTI ? fma(tau1 * s, s, tau0) : tau0;
      const double cu = fma(f.y, fma(-tau, f.x, Fv), fma(-wd, up, w.rad[a]));
      const double fx = -fma(cu, u.x, wd * px), fy = -fma(cu, u.y, wd * py),
                   fz = -fma(cu, u.z, wd * pz);
      add_force(F, jt[slot] & AE_INDEX_MASK, fx, fy, fz);
      fix -= fx;
      fiy -= fy;
      fiz -= fz;
      if (want_virial) {
        const double4_32a v = vec[slot];
        w00 += v.x * fx; w01 += v.x * fy; w02 += v.x * fz;
        w10 += v.y * fx; w11 += v.y * fy; w12 += v.y * fz;
        w20 += v.z * fx; w21 += v.z * fy; w22 += v.z * fz;
      }
    }
  } else {
    for (int k = sl; k < na; k += LPA) {
      double4_32a o;
      o.x = o.y = o.z = o.w = 0.0;
      w.acc[k] = o;
    }
    __syncwarp();
    const int P = active ? na * (na - 1) / 2 : 0;
    const int stride = max(1, min(LPA, na - 1));
    const int steps = warp_max((P + stride - 1) / stride);
    PairWalk pw;
    pw.start(sl, na);
    for (int q0 = 0; q0 < steps; ++q0, pw.advance(na, stride)) {
      const bool live = sl < stride && pw.p < P;
      const int a = live ? pw.a : 0, k = live ? pw.partner(na) : 0;
      const double4_32a ua = w.su[a], uk = w.su[k];
      double Av = 0.0, Bv = 0.0;
      if (live) {
        double x = ua.x * uk.x + ua.y * uk.y + ua.z * uk.z;
        if (ct.angular_legacy) x = fma(x, 2.0 / SFB_PI, -1.0);
        const double x2 = x + x;
        double tm1 = 1.0, t0 = x;
        if constexpr (SPIN == SPIN_ANY) {
          const int ia = w.info[a], ik = w.info[k];
          const double sa = s_spin[ti * AE_MAXT + (ia & 7)], sk = s_spin[ti * AE_MAXT + (ik & 7)];
          double ss = sa * sk;
          if (b.nb_rank) ss = ordered_spin(b, i, ia >> 3, ik >> 3, sa, sk);
          const double2 *t0p = w.tab_a, *t1p = w.tab_a + A;
          double A1 = t1p[0].x, B1 = t1p[0].y;
          Av = t0p[0].x;
          Bv = t0p[0].y;
#pragma unroll
          for (int q = 1; q < A; ++q) {
            if (!GUARD || q < aN) {
              const double2 c0 = t0p[q], c1 = t1p[q];
              Av = fma(c0.x, t0, Av);
              A1 = fma(c1.x, t0, A1);
              Bv = fma(c0.y, t0, Bv);
              B1 = fma(c1.y, t0, B1);
              const double tn = fma(x2, t0, -tm1);
              tm1 = t0;
              t0 = tn;
            }
          }
          Av = fma(ss, A1, Av);
          Bv = fma(ss, B1, Bv);
        } else {
          const double2* tab = w.tab_a;
          if (SPIN == SPIN_UNIT) {
            const float ss = s_spin[ti * AE_MAXT + (w.info[a] & 7)] *
                             s_spin[ti * AE_MAXT + (w.info[k] & 7)];
            tab += ((int)ss + 1) * A;
          }
          Av = tab[0].x;
          Bv = tab[0].y;
#pragma unroll
          for (int q = 1; q < A; ++q) {
            if (!GUARD || q < aN) {
              const double2 cq = tab[q];
              Av = fma(cq.x, t0, Av);
              if (q + 1 < A) {
                Bv = fma(cq.y, t0, Bv);
                const double tn = fma(x2, t0, -tm1);
                tm1 = t0;
                t0 = tn;
              }
            }
          }
        }
        const double fk = w.sf[k].x, cb = fk * Bv;
        double4_32a s = w.acc[a];
        s.x = fma(cb, uk.x, s.x);
        s.y = fma(cb, uk.y, s.y);
        s.z = fma(cb, uk.z, s.z);
        s.w = fma(fk, Av, s.w);
        w.acc[a] = s;
      }
      __syncwarp();
      if (live) {
        const double fa = w.sf[a].x, cb = fa * Bv;
        double4_32a s = w.acc[k];
        s.x = fma(cb, ua.x, s.x);
        s.y = fma(cb, ua.y, s.y);
        s.z = fma(cb, ua.z, s.z);
        s.w = fma(fa, Av, s.w);
        w.acc[k] = s;
      }
      __syncwarp();
    }
    // forces on the staged neighbours (radial + angular), one scatter each
    const double dxdc = ct.angular_legacy ? 2.0 / SFB_PI : 1.0;
    for (int a = sl; a < na; a += LPA) {
      if (!active) break;
      const double4_32a u = w.su[a], V = w.acc[a];
      const double2 f = w.sf[a];
      const int slot = w.info[a] >> 3;
      const double wd = f.x * u.w * dxdc;
      const double vu = V.x * u.x + V.y * u.y + V.z * u.z;
      const double cu = fma(f.y, V.w, fma(-wd, vu, w.rad[a]));
      const double fx = -fma(cu, u.x, wd * V.x), fy = -fma(cu, u.y, wd * V.y),
                   fz = -fma(cu, u.z, wd * V.z);
      add_force(F, jt[slot] & AE_INDEX_MASK, fx, fy, fz);
      fix -= fx;
      fiy -= fy;
      fiz -= fz;
      if (want_virial) {
        const double4_32a v = vec[slot];
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
    double wv[9] = {w00, w01, w02, w10, w11, w12, w20, w21, w22};
    reduce_scatter<9, LPA / 2>(wv, sl, 0, 9, [&](int q, double s) {
      if (active) atomicAdd(b.virial + 9 * (size_t)sid + q, s);
    });
  }
}

// Shared memory of a block (32 / LPA groups)
template <int R, int A, int LPA, int SPIN, bool MOM>
size_t block_smem(const PotDevice& pd, const DescBuffers& b, bool adjoint) {
  const int nt = SPIN == SPIN_NONE ? 1 : pd.ntypes;
  return (size_t)layout(b.cap_a, pd.nsf_pad, nt, R, classes<SPIN>(), A, adjoint, MOM).bytes *
         (32 / LPA);
}

constexpr size_t SMEM_MAX = 226 * 1024;

// Lanes per atom: 8 use every lane best (a whole number of rounds over the
// neighbours, cheap group sums), 32 spread few atoms over more SMs (one warp
// each) and take rows too long for several groups' shared memory.  Whole FP64
// passes with 32, 16 and 8 lanes: 864 Au/Cu atoms 148, 158 and 217 us; 1,176
// 168, 165 and 224; 1,792 239, 222 and 253; 2,772 361, 331 and 337; 4,840
// Cu/Au atoms 541, 464 and 442.  Hence below 8 atoms per SM 32, below 20 16.
template <int R, int A, int LPA, bool GUARD, int SPIN, bool MOM>
int launch_lanes(const PotDevice& pd, const DescBuffers& b, bool adjoint, cudaStream_t s) {
  const size_t smem = block_smem<R, A, LPA, SPIN, MOM>(pd, b, adjoint);
  if (smem > SMEM_MAX) return (int)cudaErrorInvalidValue;
  const int blocks = (b.natoms + 32 / LPA - 1) / (32 / LPA);
  auto kern = adjoint ? k_adjoint64<R, A, LPA, GUARD, SPIN, MOM>
                      : k_forward64<R, A, LPA, GUARD, SPIN, MOM>;
  if (smem + AE_STATIC_SMEM > 48 * 1024)
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  kern<<<blocks, 32, smem, s>>>(pd, b);
  return (int)cudaGetLastError();
}
template <int R, int A, bool GUARD, int SPIN, bool MOM>
int launch(const PotDevice& pd, const DescBuffers& b, bool adjoint, cudaStream_t s) {
  int dev = 0, nsm = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  // several groups share a block while three blocks still fit an SM
  const size_t most = SMEM_MAX / 3;
  if (b.natoms >= 20 * nsm && block_smem<R, A, 8, SPIN, MOM>(pd, b, true) <= most)
    return launch_lanes<R, A, 8, GUARD, SPIN, MOM>(pd, b, adjoint, s);
  if (b.natoms >= 8 * nsm && block_smem<R, A, 16, SPIN, MOM>(pd, b, true) <= most)
    return launch_lanes<R, A, 16, GUARD, SPIN, MOM>(pd, b, adjoint, s);
  return launch_lanes<R, A, 32, GUARD, SPIN, MOM>(pd, b, adjoint, s);
}

template <int R, int A, bool MOM>
int launch_spin(const PotDevice& pd, const DescBuffers& b, int spin, bool adjoint, cudaStream_t s) {
  return spin == SPIN_NONE ? launch<R, A, false, SPIN_NONE, MOM>(pd, b, adjoint, s)
                           : launch<R, A, false, SPIN_UNIT, MOM>(pd, b, adjoint, s);
}

}  // namespace cheb64
