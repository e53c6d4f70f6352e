// Chebyshev descriptor: the FP32 adjoint with the angular terms in moment form
// (k_cheb_mom.cuh), and helpers of both precisions for the tangent and
// Jacobian kernels.  k_cheb_rows.cuh has the forward of both precisions, the
// FP64 adjoint and the pair sums.  The descriptor replaces sfb_eval /
// sfb_radial / sfb_angular of src/ext/sfbasis.f90:440-571, 762-858 and
// chebyshev.f90:41-128, the adjoint is the force chain rule of
// src/aenet.f90:471-477 without ever materialising the descriptor Jacobian.
//
// Feature layout per atom (sfbasis.f90:114-131):
//   [radial R][angular A][radial x spin R][angular x spin A]
// The spin block exists when the setup has more than one species;
// typespin follows sfbasis.f90:142-147.
#pragma once
#include "common.h"
#include "k_cheb_mom.cuh"

namespace cheb {

template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
  using type = float4;
};
template <>
struct Vec4<double> {
  using type = double4_32a;
};

// PI as written in sfbasis.f90:72
constexpr double SFB_PI = 3.14159265358979;
constexpr double SFB_EPS = 1.0e-12;

__device__ __forceinline__ void sincos_t(float x, float* s, float* c) { __sincosf(x, s, c); }
__device__ __forceinline__ void sincos_t(double x, double* s, double* c) { sincos(x, s, c); }

template <typename T, int LPA>
__device__ __forceinline__ T gsum(T v) {
#pragma unroll
  for (int d = LPA / 2; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

__device__ __forceinline__ int warp_max(int v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, d));
  return v;
}

// fc(d) = 0.5 (cos(pi d / Rc) + 1), fc' = -0.5 (pi/Rc) sin(pi d / Rc), zero
// beyond Rc (sfb_fc / sfb_fc_d1, sfbasis.f90:719-752); a = pi/Rc
template <typename T>
__device__ __forceinline__ void cutoff_a(T d, T Rc, T a, T& fc, T& dfc) {
  if (d >= Rc) {
    fc = T(0);
    dfc = T(0);
    return;
  }
  T s, c;
  sincos_t(a * d, &s, &c);
  fc = T(0.5) * (c + T(1));
  dfc = T(-0.5) * a * s;
}
template <typename T>
__device__ __forceinline__ void cutoff(T d, T Rc, T& fc, T& dfc) {
  cutoff_a(d, Rc, T(SFB_PI) / Rc, fc, dfc);
}

// x / y: IEEE division in FP64; in FP32 the hardware reciprocal (~2 ulp,
// far inside the mixed path's error budget)
__device__ __forceinline__ double div_t(double x, double y) { return x / y; }
__device__ __forceinline__ float div_t(float x, float y) { return __fdividef(x, y); }

// radial argument x = (2 d - Rc)/Rc of chebyshev_polynomial(d, 0, Rc)
__device__ __forceinline__ double radial_x(double d, double Rc, double) { return (2.0 * d - Rc) / Rc; }
__device__ __forceinline__ float radial_x(float d, float, float two_over_rc) {
  return fmaf(d, two_over_rc, -1.0f);
}

// angular argument and dx/dcos: current domain [-1, 1] or legacy [0, pi]
template <typename T>
__device__ __forceinline__ void angular_arg(T cosv, int legacy, T& x, T& dxdc) {
  if (legacy) {
    x = (T(2) * cosv - T(SFB_PI)) / T(SFB_PI);
    dxdc = T(2) / T(SFB_PI);
  } else {
    x = cosv;
    dxdc = T(1);
  }
}

// (G - shift) * scale (sfsetup.f90:985-1035).  FP32 kernels hold the shift
// as hi + lo floats (FP64 precision); G - hi is exact whenever G and the
// shift are within a factor two of each other (Sterbenz).
__device__ __forceinline__ double normalise(double g, const PotDevice& pd, size_t k) {
  return (g - pd.shift[k]) * pd.scale[k];
}
__device__ __forceinline__ float normalise(float g, const PotDevice& pd, size_t k) {
  const float2 sh = pd.shift2[k];
  return ((g - sh.x) - sh.y) * pd.scale32[k];
}

// row-major walk of the upper triangle a < b < na with a fixed stride
struct PairWalk {
  int a, b;
  __device__ __forceinline__ void start(int p, int na) {
    a = 0;
    int rem = p;
    while (a < na - 1 && rem >= na - 1 - a) {
      rem -= na - 1 - a;
      ++a;
    }
    b = a + 1 + rem;
  }
  __device__ __forceinline__ void advance(int na, int stride) {
    b += stride;
    while (a < na - 1 && b >= na) {
      b = b - na + a + 2;
      ++a;
    }
  }
};

// Bulk prefetch of an atom's neighbour rows into L2 (one instruction per
// row, issued by the group's first lane): the radial rounds then wait on L2
// instead of DRAM.  Rows start 16-byte aligned (the ELL capacity is a
// multiple of 32) and the sizes are rounded up to 16 bytes inside the row.
template <typename T4>
__device__ __forceinline__ void prefetch_rows(const T4* vec, const int* jt, int n) {
  if (n <= 0) return;
  const unsigned bv = (unsigned)(sizeof(T4) * n);
  const unsigned bj = (unsigned)((4 * n + 15) & ~15);
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(vec)),
               "r"(bv)
               : "memory");
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(jt)),
               "r"(bj)
               : "memory");
}

// Adjoint, one group of LPA lanes (8, 16 or 32) per central atom: contracts
// dE/dG (already multiplied by E_scale and the normalisation scale) with
//   radial:  dE/dd_ij = sum_n g_n (fc' T_n + fc T_n')       along R_ij/d_ij
//   angular: k_cheb_mom.cuh
// Bound by instruction issue and by the latency of the table rows.  The
// angular neighbours are compacted in the radial pass and prepared (unit
// vector, fc, fc') densely in the angular one, where each scatters its whole
// force once; the moments' coefficients stay in registers.  4,096 Li/Si/O
// cells (597,000 atoms): 576 us with both done in the radial pass, 528 us now
// (580 and 549 us at four and six resident blocks).
#ifndef AE_MOM_ADJ_BLOCKS
#define AE_MOM_ADJ_BLOCKS 5
#endif
// shared memory of a group: staged rows (vector, distance), radial terms,
// table slot and species, and the dE/dG row; groups 16 bytes apart in banks
__host__ __device__ inline size_t adjoint_mom_smem(int cap_a, int nsf_pad) {
  const size_t per = 24 * (size_t)cap_a + 4 * (size_t)nsf_pad;
  return ((per + 111) & ~size_t(127)) + 16;
}
template <int R, int A, int LPA>
__global__ void __launch_bounds__(128, A <= 5 ? AE_MOM_ADJ_BLOCKS : 3)
    k_adjoint_mom(PotDevice pd, DescBuffers b) {
  constexpr int GPW = 32 / LPA;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  // typespin of (central species, neighbour species): a shared table, as
  // the per-neighbour lookups in the parameter bank would serialise
  __shared__ float s_spin[AE_MAXT * AE_MAXT];
  for (int q = threadIdx.x; q < pd.ntypes * AE_MAXT; q += blockDim.x)
    s_spin[q] = pd.sp[q / AE_MAXT].cheb.spin[q % AE_MAXT];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int grp = lane / LPA, sl = lane % LPA;
  const int first = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * GPW;
  if (first >= b.natoms) return;
  const int gid = first + grp;
  const bool active = gid < b.natoms;
  const int i = active ? gid : b.natoms - 1;
  unsigned char* base = smem_raw + adjoint_mom_smem(b.cap_a, pd.nsf_pad) * (threadIdx.x / LPA);
  float4* au = reinterpret_cast<float4*>(base);
  float* rad = reinterpret_cast<float*>(au + b.cap_a);
  int* info = reinterpret_cast<int*>(rad + b.cap_a);
  float* sg = reinterpret_cast<float*>(info + b.cap_a);
  const int ti = b.types[i];
  const ChebTable& ct = pd.sp[ti].cheb;
  const int n = active ? b.nb_cnt[i] : 0;
  const float4* __restrict__ vec = reinterpret_cast<const float4*>(b.nb_vec) + (size_t)i * b.cap;
  const int* __restrict__ jt = b.nb_jt + (size_t)i * b.cap;
  if (sl == 0) prefetch_rows(vec, jt, n);
  const int nloop = warp_max(n);
  const float r_Rc = float(ct.r_Rc), a_Rc = float(ct.a_Rc);
  const float two_over_rc = 2.f / r_Rc;
  const float r_a = float(SFB_PI) / r_Rc, a_a = float(SFB_PI) / a_Rc;
  const bool multi = ct.multi;
  const unsigned gmask = (LPA == 32) ? 0xffffffffu : (((1u << LPA) - 1u) << (grp * LPA));
  const int sid = b.atom_struct[i];
  const float gs = b.grad_scale ? float(b.grad_scale[sid]) : 1.f;
  const bool want_virial = b.virial != nullptr;
  float* F = reinterpret_cast<float*>(b.F);

  const float* gsrc = reinterpret_cast<const float*>(b.dEdG) + (size_t)i * pd.nsf_pad;
  for (int k = sl; k < ct.nsf; k += LPA) sg[k] = gs * gsrc[k];
  __syncwarp();
  // radial coefficients in registers
  float gr[R], grs[R];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    gr[q] = sg[ct.r_i1 + q];
    grs[q] = multi ? sg[ct.r_i2 + q] : 0.f;
  }

  float fix = 0.f, fiy = 0.f, fiz = 0.f;
  float w00 = 0, w01 = 0, w02 = 0, w10 = 0, w11 = 0, w12 = 0, w20 = 0, w21 = 0, w22 = 0;
  int na = 0;
  // the table row is read one iteration ahead (its load latency overlaps the
  // previous neighbour's work)
  float4 vn = make_float4(0.f, 0.f, 0.f, 1e30f);
  int qn = 0;
  if (sl < n) {
    vn = vec[sl];
    qn = jt[sl];
  }
  for (int base_j = 0; base_j < nloop; base_j += LPA) {
    const int j = base_j + sl;
    const float4 v = vn;
    const int t = qn >> AE_TYPE_SHIFT, jatom = qn & AE_INDEX_MASK;
    vn = make_float4(0.f, 0.f, 0.f, 1e30f);
    qn = 0;
    if (j + LPA < n) {
      vn = vec[j + LPA];
      qn = jt[j + LPA];
    }
    const float d = v.w;
    float c = 0.f;   // (dE/dd) / d
    if (d <= r_Rc && d > float(SFB_EPS)) {
      const float s = multi ? s_spin[ti * AE_MAXT + t] : 0.f;
      float fc, dfc;
      cutoff_a(d, r_Rc, r_a, fc, dfc);
      const float x = fmaf(d, two_over_rc, -1.f), x2 = x + x;
      // sum g_q T_q and sum g_q q U_{q-1} (chebyshev_polynomial_d1)
      float tm1 = 1.f, t0 = x, um1 = 1.f, u0 = x2;
      float Av = fmaf(s, grs[0], gr[0]), Bv = 0.f;
#pragma unroll
      for (int q = 1; q < R; ++q) {
        const float gq = fmaf(s, grs[q], gr[q]);
        Av = fmaf(gq, t0, Av);
        Bv = fmaf(q == 1 ? gq : float(q) * gq, um1, Bv);
        const float tn = fmaf(x2, t0, -tm1);
        tm1 = t0;
        t0 = tn;
        const float un = fmaf(x2, u0, -um1);
        um1 = u0;
        u0 = un;
      }
      c = __fdividef(fmaf(dfc, Av, fc * two_over_rc * Bv), d);
    }
    const bool inA = d <= a_Rc && d >= float(SFB_EPS);
    const unsigned m = __ballot_sync(0xffffffffu, inA) & gmask;
    bool staged = false;
    if (inA) {
      const int k = na + __popc(m & ((1u << lane) - 1u));
      if (k < b.cap_a) {
        au[k] = v;
        rad[k] = c * d;
        info[k] = (j << 3) | t;
        staged = true;
      }
    }
    if (!staged && c != 0.f) {
      // dE/dR_j = c R_ij: the force on j is minus that
      const float gx = c * v.x, gy = c * v.y, gz = c * v.z;
      fix += gx;
      fiy += gy;
      fiz += gz;
      atomicAdd(reinterpret_cast<float4*>(F) + jatom, make_float4(-gx, -gy, -gz, 0.f));
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

  // ---- angular terms: D = B_l M (plain and spin blocks), then one pass over
  // the staged neighbours, each adding its angular gradient to its radial
  // force and scattering the total once
  constexpr int L = A - 1;
  constexpr int K = A * A;
  const float* q = pd.qleg + (size_t)ti * AE_MOMA * AE_MOMA;
  float B0[A], B1[A];
#pragma unroll
  for (int l = 0; l < A; ++l) {
    B0[l] = 0.f;
    B1[l] = 0.f;
  }
#pragma unroll
  for (int nn = 0; nn < A; ++nn) {
    const float g0 = sg[ct.a_i1 + nn], g1 = multi ? sg[ct.a_i2 + nn] : 0.f;
#pragma unroll
    for (int l = 0; l <= nn; ++l) {
      const float ql = q[nn * AE_MOMA + l];
      B0[l] = fmaf(g0, ql, B0[l]);
      B1[l] = fmaf(g1, ql, B1[l]);
    }
  }
  float tau0 = 0.f, tau1 = 0.f;
#pragma unroll
  for (int l = 0; l < A; ++l) {
    tau0 += B0[l];
    tau1 += B1[l];
  }
  float Mv[4 * ((2 * K + 3) / 4)];
  const float4* M4 = reinterpret_cast<const float4*>(b.M + (size_t)i * b.mom_pad);
#pragma unroll
  for (int c4 = 0; c4 < (2 * K + 3) / 4; ++c4) {
    const float4 t4 = M4[c4];
    Mv[4 * c4] = t4.x;
    Mv[4 * c4 + 1] = t4.y;
    Mv[4 * c4 + 2] = t4.z;
    Mv[4 * c4 + 3] = t4.w;
  }
  float D0[K], D1[K];
#pragma unroll
  for (int l = 0; l < A; ++l) {
#pragma unroll
    for (int k = l * l; k < (l + 1) * (l + 1); ++k) {
      D0[k] = B0[l] * Mv[k];
      D1[k] = multi ? B1[l] * Mv[K + k] : 0.f;
    }
  }
  for (int a = sl; a < na; a += LPA) {
    if (!active) break;
    const float4 v = au[a];
    const int slot = info[a] >> 3;
    const float s = multi ? s_spin[ti * AE_MAXT + (info[a] & 7)] : 0.f;
    const float inv = __fdividef(1.f, v.w);
    const float ux = v.x * inv, uy = v.y * inv, uz = v.z * inv;
    float fc, dfc;
    cutoff_a(v.w, a_Rc, a_a, fc, dfc);
    float Fv, px, py, pz;
    mom_gradient<L, true>(ux, uy, uz, s, D0, D1, Fv, px, py, pz);
    const float up = ux * px + uy * py + uz * pz;
    const float wd = fc * inv;
    const float cu = fmaf(dfc, fmaf(-fmaf(tau1 * s, s, tau0), fc, Fv), fmaf(-wd, up, rad[a]));
    const float fx = -fmaf(cu, ux, wd * px), fy = -fmaf(cu, uy, wd * py),
                fz = -fmaf(cu, uz, wd * pz);
    atomicAdd(reinterpret_cast<float4*>(F) + (jt[slot] & AE_INDEX_MASK),
              make_float4(fx, fy, fz, 0.f));
    fix -= fx;
    fiy -= fy;
    fiz -= fz;
    if (want_virial) {
      w00 += v.x * fx; w01 += v.x * fy; w02 += v.x * fz;
      w10 += v.y * fx; w11 += v.y * fy; w12 += v.y * fz;
      w20 += v.z * fx; w21 += v.z * fy; w22 += v.z * fz;
    }
  }
  fix = gsum<float, LPA>(fix);
  fiy = gsum<float, LPA>(fiy);
  fiz = gsum<float, LPA>(fiz);
  if (active && sl == 0)
    atomicAdd(reinterpret_cast<float4*>(F) + i, make_float4(fix, fiy, fiz, 0.f));
  if (want_virial) {
    float wv[9] = {w00, w01, w02, w10, w11, w12, w20, w21, w22};
#pragma unroll
    for (int k = 0; k < 9; ++k) wv[k] = gsum<float, LPA>(wv[k]);
    if (active && sl == 0) {
      double* V = b.virial + 9 * (size_t)sid;
#pragma unroll
      for (int k = 0; k < 9; ++k) atomicAdd(V + k, (double)wv[k]);
    }
  }
}

template <int R, int A, int LPA>
int launch_adjoint_mom(const PotDevice& pd, const DescBuffers& b, cudaStream_t s) {
  // four warps per block, fewer when the atoms do not fill them (the
  // per-atom calls: one group, so long rows still fit shared memory)
  const int gpw = 32 / LPA;
  const int warps = b.natoms >= 4 * gpw ? 4 : (b.natoms + gpw - 1) / gpw;
  const int groups = warps * gpw;
  const size_t smem = adjoint_mom_smem(b.cap_a, pd.nsf_pad) * groups;
  if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
  const int blocks = (b.natoms + groups - 1) / groups;
  auto kern = k_adjoint_mom<R, A, LPA>;
  allow_smem(kern, smem, 200 * 1024);
  kern<<<blocks, warps * 32, smem, s>>>(pd, b);
  return (int)cudaGetLastError();
}
// Lanes per atom: as asked, else 8 from 20 atoms per SM on and 16
// below.  Whole mixed passes with 8, 16 and 32 lanes: 864 Au/Cu atoms 74, 72
// and 72 us, 4,000 90, 94 and 97, 32,000 246, 261 and 290; 512 Li/Si/O cells
// (72,513 atoms) 359, 380 and 418 us.  More lanes where a block's rows would
// not fit its shared memory.
template <int R, int A>
int adjoint_mom(const PotDevice& pd, const DescBuffers& b, cudaStream_t s) {
  int dev = 0, nsm = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  int lanes = b.lpa ? b.lpa : b.natoms >= 20 * nsm ? 8 : 16;
  while (lanes < 32 &&
         adjoint_mom_smem(b.cap_a, pd.nsf_pad) * (size_t)(4 * 32 / lanes) > 200 * 1024)
    lanes *= 2;
  return lanes == 8    ? launch_adjoint_mom<R, A, 8>(pd, b, s)
         : lanes == 16 ? launch_adjoint_mom<R, A, 16>(pd, b, s)
                       : launch_adjoint_mom<R, A, 32>(pd, b, s);
}

// common (radial, angular) sizes of every species, or false
inline bool uniform_sizes(const PotDevice& pd, int& rN, int& aN) {
  rN = aN = 0;
  bool same = true;
  for (int t = 0; t < pd.ntypes; ++t) {
    if (t > 0 && (pd.sp[t].cheb.r_N != rN || pd.sp[t].cheb.a_N != aN)) same = false;
    rN = max(rN, pd.sp[t].cheb.r_N);
    aN = max(aN, pd.sp[t].cheb.a_N);
  }
  return same;
}

// FP32 adjoint in moment form (k_cheb_mom.cu); AE_MOM_NA when the sizes have
// no moment instantiation
constexpr int AE_MOM_NA = -1;
int dispatch_adjoint_mom(const PotDevice& pd, const DescBuffers& b, cudaStream_t s);

}  // namespace cheb
