// One atom per call for FP64 Chebyshev potentials: the libaenet per-atom
// entry points (aenet_atomic_energy / aenet_atomic_energy_and_forces,
// src/aenet.f90:359-486) evaluate one central atom with the caller's
// neighbour list.  A warp per atom leaves an SM's FP64 pipe waiting on the
// dependent chains of one lane group, so the whole call is one launch of
// either one block of AT_THREADS threads (k_atom) or a cluster of AC_CTAS
// such blocks on as many SMs (k_atom_cluster), phase after phase:
//
//   stage    thread per neighbour: radial argument and cut-off, angular
//            cut-off and unit vector (the per-neighbour values of sfb_eval,
//            src/ext/sfbasis.f90:488-512); angular neighbours compacted in
//            list order;
//   forward  warps 0-2 over the neighbours (radial T_n, chebyshev.f90:41-128),
//            the other warps over the pairs j < k of angular neighbours;
//            the per-thread sums are reduced column by column through
//            shared memory, eight lanes per feature;
//   network  a few lanes per node for its sum and activation, forward and
//            back (ff_eval / ff_deriv, src/ext/feedforward.f90:586-757);
//   adjoint  thread per neighbour (radial, warps 0-2) and per pair
//            (angular, warps 3-7, at the same time); the pairs leave three
//            numbers each, which four lanes per neighbour gather in a
//            fixed order; the central atom takes minus the sum of the
//            neighbour forces (aenet.f90:471-477).
//
// Bound by chains of FP64 instructions, of which a scheduler of the SM starts
// one in 64 cycles: the phases of a row of 78 neighbours and 153 pairs
// (26-20-20-1) take 7,000 cycles (the row's way from host memory among them),
// 6,700, 14,500, 13,500 and 2,000 for the output.  Cut-offs as a series in d^2
// (cutoff64.cuh), constants divided on the host, spin sums only where there
// are spins, derivatives as sums over q U_(q-1) with the order multiplied
// into the coefficients once, tanh without branches and pair gradients from
// sums of scalars instead of two vectors a pair: the kernel 41 -> 31 us, the
// phases before 7,600, 8,900, 19,000, 27,500 and 2,300 cycles.
//
// In the cluster each block stages a contiguous slice of the rows and takes
// a contiguous slice of the pair index space; the blocks exchange their
// angular records, their partial descriptor sums and their partial pair
// gradients through distributed shared memory between cluster barriers,
// and every block runs the (small) network itself.  Every sum runs in a
// fixed order, so repeated calls give identical bits.  The call's row is
// read from, and its outputs written to, mapped pinned host memory (the
// row length, species and forces flag come as launch arguments): a call is
// one launch and one stream synchronisation.
#include <cooperative_groups.h>

#include <type_traits>

#include "common.h"
#include "activate.cuh"
#include "cutoff64.cuh"
#include "exp64.cuh"
#include "k_cheb_impl.cuh"

namespace cg = cooperative_groups;

namespace {

using cheb::PairWalk;
using cheb::SFB_EPS;
using cheb::SFB_PI;

constexpr int AT_THREADS = 256;
constexpr int AT_WARPS = AT_THREADS / 32;
// FP64 runs at 2 lanes per clock per SM, so every phase spreads its FP64
// work over as many warps as it can: radial terms on warps 0-2, pairs on
// warps 3-7 (forward and adjoint at the same time), radial and angular
// cut-offs of a row on two threads, activations on one warp
constexpr int AT_RAD = 96;                    // radial threads (warps 0-2)
constexpr int AT_ANG = AT_THREADS - AT_RAD;   // pair threads (warps 3-7)
constexpr int AT_HALF = AT_THREADS / 2;       // rows per staging pass
constexpr int AT_LPF = 8;                     // lanes per feature sum
constexpr int AT_LPA = 4;                     // lanes per angular neighbour's gradient
constexpr int AT_NSTRIDE = AE_MAXNODES + 1;
constexpr int AC_CTAS = 8;                    // blocks of the cluster form
constexpr int AT_WMAX = 8192;                 // network weights staged in shared memory
                                              // (doubles; larger networks read L2: calls
                                              // of 12 neighbours, 32-40-56-51-1 and eight
                                              // species, 62 us from there and 53 staged)

template <int RB, int AB>
__host__ __device__ constexpr size_t at_red_elems() {
  return (2 * RB * AT_RAD + 2 * AB * AT_ANG) > 6 * AT_THREADS ? (2 * RB * AT_RAD + 2 * AB * AT_ANG)
                                                              : 6 * AT_THREADS;
}

// shared memory of a call with n neighbours: rows (sv, sr), angular list
// (au, af), in the cluster form also the block's own angular records and
// the row -> angular index map; forces, angular gradients, reduction and
// network scratch
template <int RB, int AB>
__host__ __device__ size_t at_smem_bytes(int n, int nsf_pad, bool cluster, int wcount) {
  return (cluster ? 6 : 4) * sizeof(double4_32a) * (size_t)n + 6 * sizeof(double) * (size_t)n +
         (cluster ? 4 * (size_t)n : 0) +
         sizeof(double) * (at_red_elems<RB, AB>() + 3 * (size_t)nsf_pad +
                           2 * (size_t)AE_MAXLAYERS * AT_NSTRIDE + 4 + (size_t)wcount) +
         64;
}

// first and one-past-last weight of species t's network in the weight array
__host__ __device__ inline void net_range(const NetTable& net, int& w0, int& w1) {
  const int L = net.nlayers;
  w0 = net.w_off[0];
  w1 = net.w_off[L - 2] + net.pitch[L - 2] * net.nnodes[L - 1];
}

__device__ __forceinline__ int tri_index(int a, int b, int na) {
  // row-major index of pair (a, b), a < b, in the upper triangle
  return a * (2 * na - a - 1) / 2 + (b - a - 1);
}

// constants of the central atom's basis, divided out on the host, and the
// lanes per node of its network's layers
struct AtomConst {
  double two_over_rc, r_a2, a_a2;   // 2 / Rc; (pi / Rc)^2, radial and angular
  unsigned char fwd[AE_MAXLAYERS], back[AE_MAXLAYERS];
};

// Lanes per node for sums of n terms over `nodes` nodes, `after` instructions
// on each sum: the FP64 instructions of the busiest of the four schedulers.
int node_lanes(int nodes, int n, int after) {
  int best = 16, cost = 1 << 30;
  for (int lg = 4; lg >= 1; --lg) {
    const int k = (((nodes << lg) + 127) >> 7) * (((n + (1 << lg) - 1) >> lg) + lg + after);
    if (k < cost) {
      cost = k;
      best = 1 << lg;
    }
  }
  return best;
}

// per-call constants of the central atom's basis
struct AtomCtx {
  double r_Rc, a_Rc, two_over_rc, r_a2, a_a2;
  int rN, aN, legacy;
  bool multi;
  __device__ void init(const ChebTable& ct, const AtomConst& k) {
    r_Rc = ct.r_Rc;
    a_Rc = ct.a_Rc;
    two_over_rc = k.two_over_rc;
    r_a2 = k.r_a2;
    a_a2 = k.a_a2;
    rN = ct.r_N;
    aN = ct.a_N;
    legacy = ct.angular_legacy;
    multi = ct.multi;
  }
  // angular argument, current domain [-1, 1] or legacy (2 cos - pi) / pi
  __device__ double angular_x(double cosv) const {
    return legacy ? fma(cosv, 2.0 / SFB_PI, -1.0) : cosv;
  }
  __device__ double angular_dx() const { return legacy ? 2.0 / SFB_PI : 1.0; }
};

// cosine cut-off and its derivative over d, zero from Rc on (a2 = (pi/Rc)^2)
__device__ __forceinline__ void cutoff_series(double d, double Rc, double a2, double& fc,
                                              double& dfc) {
  const double ad = a2 * d, z = fma(ad, d, -FC_Y0);
  fc = d < Rc ? fc_series(z) : 0.0;
  dfc = d < Rc ? 2.0 * ad * fc_series_d(z) : 0.0;
}

// 1 / d by Newton's iteration from an FP32 seed
__device__ __forceinline__ double recip(double d) {
  float f;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"((float)d));
  double y = (double)f;
  y = fma(y, fma(-d, y, 1.0), y);
  return fma(y, fma(-d, y, 1.0), y);
}

// Rows [j0, j1) of the call: sv (vector and 1 / d, zero beyond the radial
// cut-off) and sr (argument, cut-off, its derivative, spin) at j - j0, the angular ones compacted in
// row order into au/af (slot = the row's index j), amap[j - j0] = the
// compacted index or -1 (when amap is given).  AT_HALF rows per pass: the
// first half of the block computes their radial records, the second half
// their angular ones.  Block-wide; returns the number of angular rows.
__device__ int stage_rows(const AtomCtx& c, const ChebTable& ct, const double4_32a* vin,
                          const int* tin, int j0, int j1, double4_32a* sv, double4_32a* sr,
                          double4_32a* au, double4_32a* af, int* amap, int* s_wcnt) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool ang_half = tid >= AT_HALF;
  const int h = ang_half ? tid - AT_HALF : tid;
  int na = 0;
  for (int c0 = j0; c0 < j1; c0 += AT_HALF) {
    const int j = c0 + h;
    bool inA = false;
    double4_32a v;
    v.x = v.y = v.z = v.w = 0.0;
    double s = 0.0;
    if (j < j1) {
      v = vin[j];
      const int t = tin[j];
      s = c.multi ? (double)ct.spin[t] : 0.0;
      const double d = v.w;
      if (!ang_half) {
        double4_32a r;
        r.x = r.y = r.z = 0.0;
        r.w = s;
        v.w = 0.0;
        if (d <= c.r_Rc && d > SFB_EPS) {
          cutoff_series(d, c.r_Rc, c.r_a2, r.y, r.z);
          r.x = fma(d, c.two_over_rc, -1.0);
          v.w = recip(d);
        }
        sv[j - j0] = v;
        sr[j - j0] = r;
      } else {
        inA = d <= c.a_Rc && d >= SFB_EPS;
      }
    }
    // compaction over the angular half's warps
    const unsigned m = __ballot_sync(0xffffffffu, inA);
    if (ang_half && lane == 0) s_wcnt[warp - AT_HALF / 32] = __popc(m);
    __syncthreads();
    int off = na, tot = 0;
    for (int w = 0; w < AT_HALF / 32; ++w) {
      if (w < warp - AT_HALF / 32) off += s_wcnt[w];
      tot += s_wcnt[w];
    }
    const int k = off + __popc(m & ((1u << lane) - 1u));
    if (inA) {
      const double d = v.w, invd = recip(d);
      double4_32a u, f;
      u.x = v.x * invd;
      u.y = v.y * invd;
      u.z = v.z * invd;
      u.w = invd;
      cutoff_series(d, c.a_Rc, c.a_a2, f.x, f.y);
      f.z = s;
      f.w = (double)j;
      au[k] = u;
      af[k] = f;
    }
    if (ang_half && amap && j < j1) amap[j - j0] = inA ? k : -1;
    na += tot;
    __syncthreads();   // s_wcnt is rewritten by the next pass
  }
  return na;
}

// Raw descriptor sums of rows [0, nl) of sv/sr (radial, warp 0) and of the
// pairs [p_lo, p_hi) of the angular list (warps 1 ..), written to
// fsum[feature index].  Block-wide.
template <int RB, int AB>
__device__ void forward_sums(const AtomCtx& c, const ChebTable& ct, const double4_32a* sv,
                             const double4_32a* sr, int nl, const double4_32a* au,
                             const double4_32a* af, int na, int p_lo, int p_hi, double* red,
                             double* fsum) {
  const int tid = threadIdx.x;
  double* red_r = red;                       // [2 RB][AT_RAD]
  double* red_a = red + 2 * RB * AT_RAD;     // [2 AB][AT_ANG]
  const int rN = c.rN, aN = c.aN;
  if (tid < AT_RAD) {
    double acc[RB], accs[RB];
#pragma unroll
    for (int q = 0; q < RB; ++q) acc[q] = accs[q] = 0.0;
    // (rows beyond the cut-off have fc = 0)
    auto rows = [&](auto flag) {
      constexpr bool spin = decltype(flag)::value;
      for (int j = tid; j < nl; j += AT_RAD) {
        const double4_32a r = sr[j];
        const double fc = r.y, x = r.x, x2 = x + x, sfc = spin ? r.w * fc : 0.0;
        double tm1 = 1.0, t0 = x;
        acc[0] += fc;
        if (spin) accs[0] += sfc;
#pragma unroll
        for (int q = 1; q < RB; ++q) {
          if (q < rN) {
            acc[q] = fma(fc, t0, acc[q]);
            if (spin) accs[q] = fma(sfc, t0, accs[q]);
            const double tn = fma(x2, t0, -tm1);
            tm1 = t0;
            t0 = tn;
          }
        }
      }
    };
    if (c.multi) rows(std::true_type{});
    else rows(std::false_type{});
#pragma unroll
    for (int q = 0; q < RB; ++q) {
      red_r[q * AT_RAD + tid] = acc[q];
      if (c.multi) red_r[(RB + q) * AT_RAD + tid] = accs[q];
    }
  } else {
    const int p0 = tid - AT_RAD;
    double ang[AB], angs[AB];
#pragma unroll
    for (int q = 0; q < AB; ++q) ang[q] = angs[q] = 0.0;
    auto pairs = [&](auto flag) {
      constexpr bool spin = decltype(flag)::value;
      PairWalk pw;
      pw.start(p_lo + p0, na);
      for (int p = p_lo + p0; p < p_hi; p += AT_ANG) {
        const double4_32a ua = au[pw.a], ub = au[pw.b], fa = af[pw.a], fb = af[pw.b];
        const double cosv = ua.x * ub.x + ua.y * ub.y + ua.z * ub.z;
        const double w = fa.x * fb.x;
        const double sw = spin ? fa.z * fb.z * w : 0.0;
        const double x = c.angular_x(cosv), x2 = x + x;
        double tm1 = 1.0, t0 = x;
        ang[0] += w;
        if (spin) angs[0] += sw;
#pragma unroll
        for (int q = 1; q < AB; ++q) {
          if (q < aN) {
            ang[q] = fma(w, t0, ang[q]);
            if (spin) angs[q] = fma(sw, t0, angs[q]);
            const double tn = fma(x2, t0, -tm1);
            tm1 = t0;
            t0 = tn;
          }
        }
        pw.advance(na, AT_ANG);
      }
    };
    if (p_lo + p0 < p_hi) {
      if (c.multi) pairs(std::true_type{});
      else pairs(std::false_type{});
    }
#pragma unroll
    for (int q = 0; q < AB; ++q) {
      red_a[q * AT_ANG + p0] = ang[q];
      if (c.multi) red_a[(AB + q) * AT_ANG + p0] = angs[q];
    }
  }
  __syncthreads();
  // feature f: radial, radial x spin, angular, angular x spin
  const int nfr = c.multi ? 2 * rN : rN, nfa = c.multi ? 2 * aN : aN;
  const int ncol_r = min(nl, AT_RAD), ncol_a = max(0, min(p_hi - p_lo, AT_ANG));
  for (int f0 = 0; f0 < nfr + nfa; f0 += AT_THREADS / AT_LPF) {
    const int f = f0 + tid / AT_LPF, sub = tid % AT_LPF;
    if (f0 + (tid & ~31) / AT_LPF >= nfr + nfa) continue;   // nothing for this warp
    double sum = 0.0;
    int gk = -1;
    if (f < nfr) {
      const int q = f < rN ? f : f - rN;
      const double* col = red_r + (f < rN ? q : RB + q) * AT_RAD;
      for (int k = sub; k < ncol_r; k += AT_LPF) sum += col[k];
      gk = (f < rN ? ct.r_i1 : ct.r_i2) + q;
    } else if (f < nfr + nfa) {
      const int fa = f - nfr;
      const int q = fa < aN ? fa : fa - aN;
      const double* col = red_a + (fa < aN ? q : AB + q) * AT_ANG;
      for (int k = sub; k < ncol_a; k += AT_LPF) sum += col[k];
      gk = (fa < aN ? ct.a_i1 : ct.a_i2) + q;
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 4);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    if (gk >= 0 && sub == 0) fsum[gk] = sum;
  }
  __syncthreads();
}

__device__ __noinline__ void activate_other(int t, double x, double& y, double& dy) {
  activate<double>(t, x, y, dy);
}

// activate<double> with the branch-free tanh
__device__ __forceinline__ void activate_even(int t, double x, double& y, double& dy) {
  if (t == 1) {
    y = tanh_even(x);
    dy = 1.0 - y * y;
  } else if (t == 3 || t == 4) {
    const double a = 1.7159, b = 0.666666666666667, c = t == 4 ? 0.1 : 0.0;
    const double tb = tanh_even(b * x);
    y = fma(c, x, a * tb);
    dy = a * (1.0 - tb * tb) * b + c;
  } else {
    activate_other(t, x, y, dy);
  }
}

__device__ __forceinline__ double lanes_sum(double v, int lpn) {
  if (lpn > 8) v += __shfl_xor_sync(0xffffffffu, v, 8);
  if (lpn > 4) v += __shfl_xor_sync(0xffffffffu, v, 4);
  if (lpn > 2) v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v + __shfl_xor_sync(0xffffffffu, v, 1);
}

// Network of species ti on the normalised descriptor G: returns the output
// node y and leaves dE/dG of the raw descriptor (times E_scale and the
// normalisation scale) in D, and the same times the order of its polynomial in
// G.  Block-wide.  A warp's FP64 instruction keeps its
// scheduler's unit for many cycles whatever its lanes do, so the lanes of a
// node go by node_lanes, warps without nodes take no part, and the activation
// follows the sum on the lanes that hold it.
__device__ double atom_network(const PotDevice& pd, const SpeciesTable& sp, int ti,
                               const AtomConst& kc, double* G, double* D, double* act, double* der,
                               const double* wsm, double scale0) {
  const int tid = threadIdx.x;
  const NetTable& net = sp.net;
  const int L = net.nlayers;
  // the species' weights: staged in shared memory (wsm, from its first
  // weight on) or read from the global table
  int w0, w1;
  net_range(net, w0, w1);
  auto layer = [&](int l) { return wsm ? wsm + (net.w_off[l] - w0) : pd.w64 + net.w_off[l]; };
  for (int l = 0; l < L - 1; ++l) {
    const int nin = net.nnodes[l], nout = net.nnodes[l + 1];
    const double* Wl = layer(l);
    const int pitch = net.pitch[l];
    const double* hin = (l == 0) ? G : act + l * AT_NSTRIDE;
    double* hout = act + (l + 1) * AT_NSTRIDE;
    double* dout = der + (l + 1) * AT_NSTRIDE;
    const int fa = net.f_a[l + 1];
    const int lpn = kc.fwd[l], step = AT_THREADS / lpn;
    const int sub = tid & (lpn - 1);
    for (int ob = 0; ob < nout; ob += step) {
      const int o = ob + tid / lpn;
      if (ob + (tid & ~31) / lpn >= nout) break;   // (the whole warp)
      double part = 0.0;
      if (o < nout) {
        const double* row = Wl + (size_t)o * pitch;
        if (sub == 0) part = row[nin];
        for (int k = sub; k < nin; k += lpn) part = fma(row[k], hin[k], part);
      }
      double y, dy;
      activate_even(fa, lanes_sum(part, lpn), y, dy);
      if (o < nout && sub == 0) {
        hout[o] = y;
        dout[o] = dy;
      }
    }
    __syncthreads();
  }
  const double y = act[(L - 1) * AT_NSTRIDE];
  // back: delta_l = (W_l^T delta_{l+1}) f'_l, from the output node down
  const double* delta = der + (L - 1) * AT_NSTRIDE;
  const size_t nrow = (size_t)ti * pd.nsf_pad;
  for (int l = L - 2; l >= 0; --l) {
    const int nin = net.nnodes[l], nout = net.nnodes[l + 1];
    const double* Wl = layer(l);
    const int pitch = net.pitch[l];
    double* dl = (l == 0) ? D : der + l * AT_NSTRIDE;
    const int lpn = kc.back[l], step = AT_THREADS / lpn;
    const int sub = tid & (lpn - 1);
    for (int kb = 0; kb < nin; kb += step) {
      const int k = kb + tid / lpn;
      if (kb + (tid & ~31) / lpn >= nin) break;
      double part = 0.0;
      if (k < nin)
        for (int o = sub; o < nout; o += lpn) part = fma(Wl[(size_t)o * pitch + k], delta[o], part);
      part = lanes_sum(part, lpn);
      if (k < nin && sub == 0) dl[k] = (l > 0) ? part * dl[k] : part;
    }
    __syncthreads();
    delta = dl;
  }
  const ChebTable& ct = sp.cheb;
  for (int k = tid; k < sp.nsf; k += AT_THREADS) {
    const double d = sp.E_scale * D[k] * (k == tid ? scale0 : pd.scale[nrow + k]);
    // feature order: radial, angular and, with several species, both again
    const int r = k - (k < ct.r_i2 || !ct.multi ? ct.r_i1 : ct.r_i2);
    const int a = k - (k < ct.a_i2 || !ct.multi ? ct.a_i1 : ct.a_i2);
    D[k] = d;
    G[k] = (double)(r >= 0 && r < ct.r_N ? r : a) * d;
  }
  __syncthreads();
  return y;
}

// The adjoint: radial part of the force on rows [0, nl) (-c R_ij / d into
// sF) on warps 0-2 while warps 3-7 take the pairs [p_lo, p_hi) in rounds of
// AT_ANG (Dq: D times the order q, T_q' = q U_(q-1)).  With A = sum c_q T_q and B = sum c_q T_q' of a pair (a, b), both
// symmetric, the gradient on neighbour a is
//   u_a (fc'_a sum_b fc_b A - sum_b Q cos / d_a) + sum_b Q u_b / d_a,  Q = fc_a fc_b B:
// a pair leaves three numbers (A, Q, Q cos) in pbuf, and AT_LPA lanes per
// neighbour sum five over its partners in a fixed order, into aF[3 a] (the
// vector) and a2[2 a].  Block-wide; aF[3 a] ends as the gradient.
template <int RB, int AB>
__device__ void adjoint_rows_pairs(const AtomCtx& c, const ChebTable& ct, const double* D,
                                   const double* Dq, const double4_32a* sv, const double4_32a* sr, int nl,
                                   double* sF, const double4_32a* au, const double4_32a* af,
                                   int na, int p_lo, int p_hi, double* pbuf, double* aF) {
  const int tid = threadIdx.x, rN = c.rN, aN = c.aN;
  double* a2 = pbuf + 3 * AT_ANG;
  for (int a = tid; a < na; a += AT_THREADS)
    aF[3 * a] = aF[3 * a + 1] = aF[3 * a + 2] = a2[2 * a] = a2[2 * a + 1] = 0.0;
  __syncthreads();
  if (tid < AT_RAD) {
    auto rows = [&](auto flag) {
      constexpr bool spin = decltype(flag)::value;
      for (int j = tid; j < nl; j += AT_RAD) {
        const double4_32a v = sv[j], r = sr[j];
        const double fc = r.y, dfc = r.z, s = r.w, x = r.x, x2 = x + x;
        const double* gr = D + ct.r_i1;
        const double* grs = D + ct.r_i2;
        const double* hr = Dq + ct.r_i1;
        const double* hrs = Dq + ct.r_i2;
        double tm1 = 1.0, t0 = x, um1 = 1.0, u0 = x2;
        double A = spin ? fma(s, grs[0], gr[0]) : gr[0], B = 0.0;
#pragma unroll
        for (int q = 1; q < RB; ++q) {
          if (q < rN) {
            A = fma(spin ? fma(s, grs[q], gr[q]) : gr[q], t0, A);
            B = fma(spin ? fma(s, hrs[q], hr[q]) : hr[q], um1, B);
            const double tn = fma(x2, t0, -tm1);
            tm1 = t0;
            t0 = tn;
            const double un = fma(x2, u0, -um1);
            um1 = u0;
            u0 = un;
          }
        }
        const bool in = __double_as_longlong(v.w) != 0;
        const double cc = in ? fma(dfc, A, fc * c.two_over_rc * B) * v.w : 0.0;
        sF[3 * j] = -(cc * v.x);
        sF[3 * j + 1] = -(cc * v.y);
        sF[3 * j + 2] = -(cc * v.z);
      }
    };
    if (c.multi) rows(std::true_type{});
    else rows(std::false_type{});
  }
  const int pt = tid - AT_RAD;   // pair thread
  PairWalk pw;
  if (pt >= 0 && p_lo + pt < p_hi) pw.start(p_lo + pt, na);
  for (int P0 = p_lo; P0 < p_hi; P0 += AT_ANG) {
    const int p = P0 + pt;
    auto pair = [&](auto flag) {
      constexpr bool spin = decltype(flag)::value;
      const double4_32a ua = au[pw.a], uk = au[pw.b], fa = af[pw.a], fk = af[pw.b];
      const double cosv = ua.x * uk.x + ua.y * uk.y + ua.z * uk.z;
      const double w = fa.x * fk.x;
      const double ss = spin ? fa.z * fk.z : 0.0;
      const double x = c.angular_x(cosv), x2 = x + x;
      const double* ga = D + ct.a_i1;
      const double* gas = D + ct.a_i2;
      const double* ha = Dq + ct.a_i1;
      const double* has = Dq + ct.a_i2;
      double tm1 = 1.0, t0 = x, um1 = 1.0, u0 = x2;
      double Av = spin ? fma(ss, gas[0], ga[0]) : ga[0], Bv = 0.0;
#pragma unroll
      for (int q = 1; q < AB; ++q) {
        if (q < aN) {
          Av = fma(spin ? fma(ss, gas[q], ga[q]) : ga[q], t0, Av);
          Bv = fma(spin ? fma(ss, has[q], ha[q]) : ha[q], um1, Bv);
          const double tn = fma(x2, t0, -tm1);
          tm1 = t0;
          t0 = tn;
          const double un = fma(x2, u0, -um1);
          um1 = u0;
          u0 = un;
        }
      }
      const double Q = w * Bv * c.angular_dx();
      pbuf[3 * pt] = Av;
      pbuf[3 * pt + 1] = Q;
      pbuf[3 * pt + 2] = Q * cosv;
      pw.advance(na, AT_ANG);
    };
    if (pt >= 0 && p < p_hi) {
      if (c.multi) pair(std::true_type{});
      else pair(std::false_type{});
    }
    __syncthreads();
    const int P1 = min(p_hi, P0 + AT_ANG);
    for (int ab = 0; ab < na; ab += AT_THREADS / AT_LPA) {
      const int a = ab + tid / AT_LPA, sub = tid % AT_LPA;
      if (ab + (tid & ~31) / AT_LPA >= na) break;   // (the whole warp)
      double s1 = 0.0, s2 = 0.0, vx = 0.0, vy = 0.0, vz = 0.0;
      if (a < na)
        for (int b = sub; b < na; b += AT_LPA) {
          const int q = a < b ? tri_index(a, b, na) : tri_index(b, a, na);
          if (b != a && q >= P0 && q < P1) {
            const double* e = pbuf + 3 * (q - P0);
            const double4_32a ub = au[b];
            s1 = fma(af[b].x, e[0], s1);
            s2 += e[2];
            vx = fma(e[1], ub.x, vx);
            vy = fma(e[1], ub.y, vy);
            vz = fma(e[1], ub.z, vz);
          }
        }
      s1 = lanes_sum(s1, AT_LPA);
      s2 = lanes_sum(s2, AT_LPA);
      vx = lanes_sum(vx, AT_LPA);
      vy = lanes_sum(vy, AT_LPA);
      vz = lanes_sum(vz, AT_LPA);
      if (a < na && sub == 0) {
        aF[3 * a] += vx;
        aF[3 * a + 1] += vy;
        aF[3 * a + 2] += vz;
        a2[2 * a] += s1;
        a2[2 * a + 1] += s2;
      }
    }
    __syncthreads();   // pbuf is rewritten by the next round
  }
  for (int a = tid; a < na; a += AT_THREADS) {
    const double4_32a ua = au[a];
    const double k = fma(af[a].y, a2[2 * a], -(ua.w * a2[2 * a + 1]));
    aF[3 * a] = fma(k, ua.x, ua.w * aF[3 * a]);
    aF[3 * a + 1] = fma(k, ua.y, ua.w * aF[3 * a + 1]);
    aF[3 * a + 2] = fma(k, ua.z, ua.w * aF[3 * a + 2]);
  }
  __syncthreads();
}

// The species' network weights into shared memory (when there is room for
// them): issued at the start of the call, so that their loads overlap the
// row reads; the block's later barriers order them before the network.
__device__ __forceinline__ void stage_weights(const NetTable& net, const double* W, double* wsm) {
  if (!wsm) return;
  int w0, w1;
  net_range(net, w0, w1);
  for (int q = threadIdx.x; q < w1 - w0; q += AT_THREADS) wsm[q] = W[w0 + q];
}

// shared-memory carve-up of a call
struct AtomSmem {
  double4_32a *sv, *sr, *au, *af, *lau, *laf;
  double *sF, *aF, *red, *fsum, *G, *D, *act, *der, *cen, *wsm;
  int* amap;
  template <int RB, int AB>
  __device__ void carve(unsigned char* base, int n, int nsf_pad, bool cluster, int wcount) {
    double4_32a* p = reinterpret_cast<double4_32a*>(base);
    sv = p;
    sr = sv + n;
    au = sr + n;
    af = au + n;
    lau = cluster ? af + n : nullptr;
    laf = cluster ? lau + n : nullptr;
    double* q = reinterpret_cast<double*>(af + (cluster ? 3 : 1) * (size_t)n);
    sF = q;
    aF = sF + 3 * (size_t)n;
    red = aF + 3 * (size_t)n;
    fsum = red + at_red_elems<RB, AB>();
    G = fsum + nsf_pad;
    D = G + nsf_pad;
    act = D + nsf_pad;
    der = act + AE_MAXLAYERS * AT_NSTRIDE;
    cen = der + AE_MAXLAYERS * AT_NSTRIDE;
    wsm = wcount > 0 ? cen + 4 : nullptr;
    amap = cluster ? reinterpret_cast<int*>(cen + 4 + wcount) : nullptr;
  }
};

template <int RB, int AB>
__global__ void __launch_bounds__(AT_THREADS, 1)
    k_atom(PotDevice pd, AtomCallHeader hd, AtomConst kc, int wcount, const unsigned char* __restrict__ in,
           unsigned char* __restrict__ out) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  __shared__ int s_wcnt[AT_WARPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = hd.n, ti = hd.ti;
  const double4_32a* __restrict__ vin = reinterpret_cast<const double4_32a*>(in + AE_ATOM_IN_VEC);
  const int* __restrict__ tin =
      reinterpret_cast<const int*>(in + AE_ATOM_IN_VEC + sizeof(double4_32a) * (size_t)n);
  const SpeciesTable& sp = pd.sp[ti];
  const ChebTable& ct = sp.cheb;
  AtomCtx c;
  c.init(ct, kc);
  AtomSmem sm{};
  sm.carve<RB, AB>(smem_raw, n, pd.nsf_pad, false, wcount);
  stage_weights(sp.net, pd.w64, sm.wsm);
  // the normalisation of this thread's feature, read while the rows come
  const size_t nrow = (size_t)ti * pd.nsf_pad;
  const double shift0 = tid < sp.nsf ? pd.shift[nrow + tid] : 0.0;
  const double scale0 = tid < sp.nsf ? pd.scale[nrow + tid] : 0.0;

  const int na = stage_rows(c, ct, vin, tin, 0, n, sm.sv, sm.sr, sm.au, sm.af, nullptr, s_wcnt);
  const int np = na * (na - 1) / 2;
  forward_sums<RB, AB>(c, ct, sm.sv, sm.sr, n, sm.au, sm.af, na, 0, np, sm.red, sm.fsum);
  for (int k = tid; k < sp.nsf; k += AT_THREADS)
    sm.G[k] = k == tid ? (sm.fsum[k] - shift0) * scale0
                       : (sm.fsum[k] - pd.shift[nrow + k]) * pd.scale[nrow + k];
  __syncthreads();
  const double y = atom_network(pd, sp, ti, kc, sm.G, sm.D, sm.act, sm.der, sm.wsm, scale0);
  if (tid == 0) {
    *reinterpret_cast<double*>(out) = sp.E_scale * y + sp.E_shift + sp.E_atom;
    *reinterpret_cast<unsigned*>(out + 8) = 0u;
  }
  if (!hd.forces) return;

  adjoint_rows_pairs<RB, AB>(c, ct, sm.D, sm.G, sm.sv, sm.sr, n, sm.sF, sm.au, sm.af, na, 0, np, sm.red,
                             sm.aF);
  for (int a = tid; a < na; a += AT_THREADS) {
    const int slot = (int)sm.af[a].w;
    sm.sF[3 * slot] -= sm.aF[3 * a];
    sm.sF[3 * slot + 1] -= sm.aF[3 * a + 1];
    sm.sF[3 * slot + 2] -= sm.aF[3 * a + 2];
  }
  __syncthreads();

  // outputs: row 0 the central atom (minus the neighbours' sum), then the
  // neighbours in list order
  double* Fo = reinterpret_cast<double*>(out + AE_ATOM_OUT_F);
  if (warp < 3) {
    double s = 0.0;
    for (int j = lane; j < n; j += 32) s += sm.sF[3 * j + warp];
#pragma unroll
    for (int dd = 16; dd > 0; dd >>= 1) s += __shfl_xor_sync(0xffffffffu, s, dd);
    if (lane == 0) Fo[warp] = -s;
  }
  for (int q = tid; q < 3 * n; q += AT_THREADS) Fo[3 + q] = sm.sF[q];
}

template <int RB, int AB>
__global__ void __cluster_dims__(AC_CTAS, 1, 1) __launch_bounds__(AT_THREADS, 1)
    k_atom_cluster(PotDevice pd, AtomCallHeader hd, AtomConst kc, int wcount,
                   const unsigned char* __restrict__ in, unsigned char* __restrict__ out) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  __shared__ int s_wcnt[AT_WARPS];
  __shared__ int s_na;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = hd.n, ti = hd.ti;
  const double4_32a* __restrict__ vin = reinterpret_cast<const double4_32a*>(in + AE_ATOM_IN_VEC);
  const int* __restrict__ tin =
      reinterpret_cast<const int*>(in + AE_ATOM_IN_VEC + sizeof(double4_32a) * (size_t)n);
  const SpeciesTable& sp = pd.sp[ti];
  const ChebTable& ct = sp.cheb;
  AtomCtx c;
  c.init(ct, kc);
  AtomSmem sm{};
  sm.carve<RB, AB>(smem_raw, n, pd.nsf_pad, true, wcount);
  stage_weights(sp.net, pd.w64, sm.wsm);
  // the normalisation of this thread's feature, read while the rows come
  const size_t nrow = (size_t)ti * pd.nsf_pad;
  const double shift0 = tid < sp.nsf ? pd.shift[nrow + tid] : 0.0;
  const double scale0 = tid < sp.nsf ? pd.scale[nrow + tid] : 0.0;
  // this block's rows
  const int j0 = (int)((long long)n * rank / AC_CTAS);
  const int j1 = (int)((long long)n * (rank + 1) / AC_CTAS);
  const int nl = j1 - j0;

  const int nal = stage_rows(c, ct, vin, tin, j0, j1, sm.sv, sm.sr, sm.lau, sm.laf, sm.amap, s_wcnt);
  if (tid == 0) s_na = nal;
  cl.sync();
  // every block's angular records, in row order
  int na = 0, myoff = 0;
  for (int r = 0; r < AC_CTAS; ++r) {
    const int nr = *cl.map_shared_rank(&s_na, r);
    const double4_32a* ru = cl.map_shared_rank(sm.lau, r);
    const double4_32a* rf = cl.map_shared_rank(sm.laf, r);
    for (int k = tid; k < nr; k += AT_THREADS) {
      sm.au[na + k] = ru[k];
      sm.af[na + k] = rf[k];
    }
    if (r == rank) myoff = na;
    na += nr;
  }
  for (int jl = tid; jl < nl; jl += AT_THREADS)
    if (sm.amap[jl] >= 0) sm.amap[jl] += myoff;
  __syncthreads();
  const int np = na * (na - 1) / 2;
  const int p_lo = (int)((long long)np * rank / AC_CTAS);
  const int p_hi = (int)((long long)np * (rank + 1) / AC_CTAS);
  forward_sums<RB, AB>(c, ct, sm.sv, sm.sr, nl, sm.au, sm.af, na, p_lo, p_hi, sm.red, sm.fsum);
  cl.sync();
  // the descriptor: every block's partial sums, in block order
  for (int k = tid; k < sp.nsf; k += AT_THREADS) {
    double s = 0.0;
    for (int r = 0; r < AC_CTAS; ++r) s += cl.map_shared_rank(sm.fsum, r)[k];
    sm.G[k] = k == tid ? (s - shift0) * scale0 : (s - pd.shift[nrow + k]) * pd.scale[nrow + k];
  }
  cl.sync();   // no block reads another's partial sums after this
  const double y = atom_network(pd, sp, ti, kc, sm.G, sm.D, sm.act, sm.der, sm.wsm, scale0);
  if (rank == 0 && tid == 0) {
    *reinterpret_cast<double*>(out) = sp.E_scale * y + sp.E_shift + sp.E_atom;
    *reinterpret_cast<unsigned*>(out + 8) = 0u;
  }
  if (!hd.forces) return;

  adjoint_rows_pairs<RB, AB>(c, ct, sm.D, sm.G, sm.sv, sm.sr, nl, sm.sF, sm.au, sm.af, na, p_lo, p_hi,
                             sm.red, sm.aF);
  cl.sync();
  // this block's rows: radial part minus every block's angular gradients
  double* Fo = reinterpret_cast<double*>(out + AE_ATOM_OUT_F);
  for (int jl = tid; jl < nl; jl += AT_THREADS) {
    double fx = sm.sF[3 * jl], fy = sm.sF[3 * jl + 1], fz = sm.sF[3 * jl + 2];
    const int a = sm.amap[jl];
    if (a >= 0) {
      for (int r = 0; r < AC_CTAS; ++r) {
        const double* g = cl.map_shared_rank(sm.aF, r) + 3 * a;
        fx -= g[0];
        fy -= g[1];
        fz -= g[2];
      }
    }
    sm.sF[3 * jl] = fx;
    sm.sF[3 * jl + 1] = fy;
    sm.sF[3 * jl + 2] = fz;
    Fo[3 * (1 + j0 + jl)] = fx;
    Fo[3 * (1 + j0 + jl) + 1] = fy;
    Fo[3 * (1 + j0 + jl) + 2] = fz;
  }
  __syncthreads();
  if (warp < 3) {
    double s = 0.0;
    for (int j = lane; j < nl; j += 32) s += sm.sF[3 * j + warp];
#pragma unroll
    for (int dd = 16; dd > 0; dd >>= 1) s += __shfl_xor_sync(0xffffffffu, s, dd);
    if (lane == 0) sm.cen[warp] = s;
  }
  cl.sync();
  // the central atom: minus the sum of every block's rows
  if (rank == 0 && tid < 3) {
    double s = 0.0;
    for (int r = 0; r < AC_CTAS; ++r) s += cl.map_shared_rank(sm.cen, r)[tid];
    Fo[tid] = -s;
  }
  cl.sync();   // block 0 has read the others' sums before they exit
}

template <int RB, int AB>
int launch_atom(const PotDevice& pd, const AtomCallHeader& hd, const void* in, void* out,
                bool cluster, cudaStream_t s) {
  // room for the largest species' weights, unless some network exceeds
  // AT_WMAX (then every call reads them from L2)
  int wcount = 0;
  for (int t = 0; t < pd.ntypes; ++t) {
    int w0, w1;
    net_range(pd.sp[t].net, w0, w1);
    wcount = max(wcount, w1 - w0);
  }
  if (wcount > AT_WMAX) wcount = 0;
  size_t smem = at_smem_bytes<RB, AB>(hd.n, pd.nsf_pad, cluster, wcount);
  if (smem > 200 * 1024 && wcount > 0) {
    wcount = 0;
    smem = at_smem_bytes<RB, AB>(hd.n, pd.nsf_pad, cluster, 0);
  }
  if (smem > 200 * 1024) return AE_ATOM_NA;
  const ChebTable& ct = pd.sp[hd.ti].cheb;
  AtomConst kc{2.0 / ct.r_Rc, (SFB_PI / ct.r_Rc) * (SFB_PI / ct.r_Rc),
               (SFB_PI / ct.a_Rc) * (SFB_PI / ct.a_Rc), {}, {}};
  const NetTable& net = pd.sp[hd.ti].net;
  for (int l = 0; l + 1 < net.nlayers; ++l) {
    kc.fwd[l] = (unsigned char)node_lanes(net.nnodes[l + 1], net.nnodes[l], net.f_a[l + 1] ? 30 : 0);
    kc.back[l] = (unsigned char)node_lanes(net.nnodes[l], net.nnodes[l + 1], 1);
  }
  const unsigned char* pin = static_cast<const unsigned char*>(in);
  unsigned char* pout = static_cast<unsigned char*>(out);
  // the opt-in limit is raised once per kernel (callers hold the library
  // lock)
  if (cluster) {
    static bool opted = false;
    if (!opted) {
      const cudaError_t e = cudaFuncSetAttribute(
          k_atom_cluster<RB, AB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
      if (e != cudaSuccess) return (int)e;
      opted = true;
    }
    k_atom_cluster<RB, AB><<<AC_CTAS, AT_THREADS, smem, s>>>(pd, hd, kc, wcount, pin, pout);
  } else {
    static bool opted = false;
    if (!opted) {
      const cudaError_t e = cudaFuncSetAttribute(
          k_atom<RB, AB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
      if (e != cudaSuccess) return (int)e;
      opted = true;
    }
    k_atom<RB, AB><<<1, AT_THREADS, smem, s>>>(pd, hd, kc, wcount, pin, pout);
  }
  return (int)cudaGetLastError();
}

}  // namespace

int ae_launch_atom(const PotDevice& pd, const AtomCallHeader& hd, const void* in, void* out,
                   int cluster, cudaStream_t s) {
  if (hd.n < 0 || hd.n > AE_ATOM_NMAX) return AE_ATOM_NA;
  int rN = 0, aN = 0;
  for (int t = 0; t < pd.ntypes; ++t) {
    if (pd.sp[t].sftype != AE_SF_CHEBYSHEV) return AE_ATOM_NA;
    rN = max(rN, pd.sp[t].cheb.r_N);
    aN = max(aN, pd.sp[t].cheb.a_N);
    for (int l = 1; l < pd.sp[t].net.nlayers; ++l)
      if (pd.sp[t].net.nnodes[l] > AE_MAXNODES) return AE_ATOM_NA;
  }
  if (rN <= 17 && aN <= 9) return launch_atom<17, 9>(pd, hd, in, out, cluster != 0, s);
  if (rN <= 24 && aN <= 16) return launch_atom<24, 16>(pd, hd, in, out, cluster != 0, s);
  return AE_ATOM_NA;
}
