// Per-species feed-forward networks: energy and dE/dG (replaces ff_eval /
// ff_deriv of src/ext/feedforward.f90:586-757 and the energy assembly of
// src/aenet.f90:464-469), plus the per-structure energy reduction and the
// force output conversion.
//
// Weights of every species are staged once per block in shared memory;
// blocks are persistent (grid-stride over atoms), one warp per atom, lane o
// computing node o of a layer, or (FP64, networks_in_tiles) a warp per eight
// atoms.  Rows of a layer's weight matrix are stored
// W[o][k] with the bias in column n_in and an odd row pitch, so that both
// the forward pass (lanes over rows) and the backward pass (lanes over
// columns) read shared memory without bank conflicts.
//
// dE/dG is written already multiplied by E_scale and by the descriptor
// normalisation scale 1/s (sfsetup.f90:1010-1031): the adjoint kernels
// contract it with the derivatives of the raw descriptor.
#include "common.h"
#include "chain.cuh"
#include "activate.cuh"
#include "exp64.cuh"

namespace {

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

constexpr int MLP_WARPS = 8;
__host__ __device__ constexpr int mlp_warp_elems() {
  return 2 * (AE_MAXNSF + 1) + 2 * AE_MAXLAYERS * (AE_MAXNODES + 1) + 1;
}

// 1/s of a feature (the FP32 kernels' copy)
template <typename T>
__device__ __forceinline__ T nscale(const PotDevice& pd, size_t k);
template <>
__device__ __forceinline__ float nscale<float>(const PotDevice& pd, size_t k) { return pd.scale32[k]; }
template <>
__device__ __forceinline__ double nscale<double>(const PotDevice& pd, size_t k) { return pd.scale[k]; }

// a warp per atom: FP32 networks that the tensor-core kernel does not take,
// and FP64 networks (networks_in_tiles)
template <typename T>
__global__ void __launch_bounds__(256) k_mlp(PotDevice pd, DescBuffers b, const T* __restrict__ W,
                                             int wtotal) {
  wait_for_previous();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sW = reinterpret_cast<T*>(smem_raw);
  const int warps = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  for (int q = threadIdx.x; q < wtotal; q += blockDim.x) sW[q] = W[q];
  // per warp: input features and their gradient (up to AE_MAXNSF), then
  // activations and derivatives of layers 1 .. L-1 (up to AE_MAXNODES)
  const int stride = AE_MAXNODES + 1;
  T* xin = sW + ((wtotal + 1) & ~1) + (size_t)warp * mlp_warp_elems();
  T* gin = xin + (AE_MAXNSF + 1);
  T* act = gin + (AE_MAXNSF + 1);
  T* der = act + AE_MAXLAYERS * stride;
  __syncthreads();

  for (int i = blockIdx.x * warps + warp; i < b.natoms; i += gridDim.x * warps) {
    const int ti = b.types[i];
    const SpeciesTable& sp = pd.sp[ti];
    const NetTable& net = sp.net;
    const int nsf = sp.nsf;
    const T* G = reinterpret_cast<const T*>(b.G) + (size_t)i * pd.nsf_pad;
    for (int k = lane; k < nsf; k += 32) xin[k] = G[k];
    __syncwarp();
    T y = T(0);
    const int L = net.nlayers;
    for (int l = 0; l < L - 1; ++l) {
      const int nin = net.nnodes[l], nout = net.nnodes[l + 1];
      const T* Wl = sW + net.w_off[l];
      const int pitch = net.pitch[l];
      const T* hin = (l == 0) ? xin : act + l * stride;
      T* hout = act + (l + 1) * stride;
      T* dout = der + (l + 1) * stride;
      if (nout == 1) {
        T part = T(0);
        for (int k = lane; k < nin; k += 32) part += Wl[k] * hin[k];
        part = warp_sum(part) + Wl[nin];
        T yy, dy;
        activate<T>(net.f_a[l + 1], part, yy, dy);
        if (lane == 0) {
          hout[0] = yy;
          dout[0] = dy;
        }
        y = yy;
      } else {
        for (int o = lane; o < nout; o += 32) {
          const T* row = Wl + o * pitch;
          T z = row[nin];
          for (int k = 0; k < nin; ++k) z += row[k] * hin[k];
          T yy, dy;
          activate<T>(net.f_a[l + 1], z, yy, dy);
          hout[o] = yy;
          dout[o] = dy;
        }
      }
      __syncwarp();
    }
    // backward: delta of the output node (dE/dy = 1 times f'(z_out)), then
    // delta_l = (W_l^T delta_{l+1}) * f'_l down to the inputs
    const T* delta_cur = der + (L - 1) * stride;
    for (int l = L - 2; l >= 0; --l) {
      const int nin = net.nnodes[l], nout = net.nnodes[l + 1];
      const T* Wl = sW + net.w_off[l];
      const int pitch = net.pitch[l];
      T* dl = (l == 0) ? gin : der + l * stride;
      for (int k = lane; k < nin; k += 32) {
        T s = T(0);
        for (int o = 0; o < nout; ++o) s += Wl[o * pitch + k] * delta_cur[o];
        dl[k] = (l > 0) ? s * dl[k] : s;
      }
      __syncwarp();
      delta_cur = dl;
    }
    // delta_cur = dE/dG (normalised inputs)
    T* out = reinterpret_cast<T*>(b.dEdG) + (size_t)i * pd.nsf_pad;
    const T es = T(sp.E_scale);
    for (int k = lane; k < nsf; k += 32)
      out[k] = es * delta_cur[k] * nscale<T>(pd, (size_t)ti * pd.nsf_pad + k);
    if (lane == 0) b.E_atom[i] = sp.E_scale * (double)y + sp.E_shift + sp.E_atom;
    __syncwarp();
  }
}

// FP64 networks by tiles (networks_in_tiles).  The FP64 pipe (two lanes per
// clock and SM) bounds them, so a warp takes `tile` atoms at once and spreads
// their (atom, node) pairs over its lanes: 20 or 25 nodes fill as many lanes as
// 32, and tanh is evaluated without branches.  The activations of a tile live
// in shared memory beside the weights.
constexpr int MLP64_WARPS = 4;
struct Mlp64Shape {
  int tile;       // atoms per warp
  int hmax;       // widest hidden layer (odd pitch)
  int in;         // input pitch (odd)
  int per;        // doubles per atom
};
__global__ void __launch_bounds__(32 * MLP64_WARPS) k_mlp64(PotDevice pd, DescBuffers b, int wtotal,
                                                            Mlp64Shape sh) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  wait_for_previous();
  double* sW = reinterpret_cast<double*>(smem_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int q = threadIdx.x; q < wtotal; q += blockDim.x) sW[q] = pd.w64[q];
  double* mine = sW + wtotal + (size_t)warp * sh.tile * sh.per;
  __syncthreads();
  // an atom's block: inputs, then activations and derivatives of the hidden
  // layers (l = 1 .. L - 2)
  auto act = [&](int a, int l) { return mine + a * sh.per + sh.in + 2 * (l - 1) * sh.hmax; };
  const int ntile = (b.natoms + sh.tile - 1) / sh.tile;
  for (int tl = blockIdx.x * MLP64_WARPS + warp; tl < ntile; tl += gridDim.x * MLP64_WARPS) {
    const int i0 = tl * sh.tile, na = min(sh.tile, b.natoms - i0);
    for (int a = 0; a < na; ++a) {
      const int nsf = pd.sp[b.types[i0 + a]].nsf;
      const double* G = reinterpret_cast<const double*>(b.G) + (size_t)(i0 + a) * pd.nsf_pad;
      for (int k = lane; k < nsf; k += 32) mine[a * sh.per + k] = G[k];
    }
    __syncwarp();
    // the tile's deepest network and widest layers (species may differ)
    int L = 0;
    for (int a = 0; a < na; ++a) L = max(L, pd.sp[b.types[i0 + a]].net.nlayers);
    for (int l = 0; l < L - 2; ++l) {
      int wide = 1;
      for (int a = 0; a < na; ++a) {
        const NetTable& net = pd.sp[b.types[i0 + a]].net;
        if (l < net.nlayers - 2) wide = max(wide, net.nnodes[l + 1]);
      }
      int a = lane / wide, o = lane - a * wide;
      const int da = 32 / wide, dr = 32 - da * wide;
      for (; a < na; a += da, o += dr) {
        if (o >= wide) {
          o -= wide;
          if (++a >= na) break;
        }
        const NetTable& net = pd.sp[b.types[i0 + a]].net;
        if (l >= net.nlayers - 2 || o >= net.nnodes[l + 1]) continue;
        const int nin = net.nnodes[l];
        const double* row = sW + net.w_off[l] + o * net.pitch[l];
        const double* x = l == 0 ? mine + a * sh.per : act(a, l);
        double z = row[nin];
#pragma unroll 4
        for (int k = 0; k < nin; ++k) z = fma(row[k], x[k], z);
        double y, dy;
        const int f = net.f_a[l + 1];
        if (f == 1) {
          y = tanh_even(z);
          dy = fma(-y, y, 1.0);
        } else {
          activate<double>(f, z, y, dy);
        }
        double* h = act(a, l + 1);
        h[o] = y;
        h[sh.hmax + o] = dy;
      }
      __syncwarp();
    }
    // output node, four lanes per atom: energy, and its derivative times the
    // weights into the last hidden layer's derivatives (networks without one:
    // into the gradient)
    for (int a0 = 0; a0 < na; a0 += 8) {
      const int a = a0 + (lane >> 2);
      const bool on = a < na;
      const int i = i0 + (on ? a : 0);
      const SpeciesTable& sp = pd.sp[b.types[i]];
      const NetTable& net = sp.net;
      const int l = net.nlayers - 2, nin = net.nnodes[l];
      const double* row = sW + net.w_off[l];
      const double* x = l == 0 ? mine + (on ? a : 0) * sh.per : act(on ? a : 0, l);
      double part = (lane & 3) ? 0.0 : row[nin];
      for (int k = lane & 3; k < nin; k += 4) part = fma(row[k], x[k], part);
      part += __shfl_xor_sync(0xffffffffu, part, 1);
      part += __shfl_xor_sync(0xffffffffu, part, 2);
      double y, dy;
      activate<double>(net.f_a[l + 1], part, y, dy);
      if (on) {
        if (!(lane & 3)) b.E_atom[i] = sp.E_scale * y + sp.E_shift + sp.E_atom;
        if (l == 0) {
          double* out = reinterpret_cast<double*>(b.dEdG) + (size_t)i * pd.nsf_pad;
          const double* sc = pd.scale + (size_t)b.types[i] * pd.nsf_pad;
          for (int k = lane & 3; k < nin; k += 4) out[k] = sp.E_scale * (row[k] * dy) * sc[k];
        } else {
          double* d = act(a, l) + sh.hmax;
          for (int k = lane & 3; k < nin; k += 4) d[k] *= row[k] * dy;
        }
      }
    }
    __syncwarp();
    // delta_l = (W_l^T delta_{l+1}) f'_l, down to the inputs (dE/dG)
    for (int l = L - 3; l >= 0; --l) {
      int wide = 1;
      for (int a = 0; a < na; ++a) {
        const NetTable& net = pd.sp[b.types[i0 + a]].net;
        if (l < net.nlayers - 2) wide = max(wide, net.nnodes[l]);
      }
      int a = lane / wide, k = lane - a * wide;
      const int da = 32 / wide, dr = 32 - da * wide;
      for (; a < na; a += da, k += dr) {
        if (k >= wide) {
          k -= wide;
          if (++a >= na) break;
        }
        const int i = i0 + a, ti = b.types[i];
        const SpeciesTable& sp = pd.sp[ti];
        const NetTable& net = sp.net;
        if (l >= net.nlayers - 2 || k >= net.nnodes[l]) continue;
        const int nout = net.nnodes[l + 1], pitch = net.pitch[l];
        const double* col = sW + net.w_off[l] + k;
        const double* d = act(a, l + 1) + sh.hmax;
        double s = 0.0;
#pragma unroll 4
        for (int o = 0; o < nout; ++o) s = fma(col[o * pitch], d[o], s);
        if (l > 0)
          act(a, l)[sh.hmax + k] *= s;
        else
          reinterpret_cast<double*>(b.dEdG)[(size_t)i * pd.nsf_pad + k] =
              sp.E_scale * s * pd.scale[(size_t)ti * pd.nsf_pad + k];
      }
      __syncwarp();
    }
  }
}

// Per-structure energy with Neumaier-compensated FP64 summation: one warp
// per structure, each lane sums a strided subset, then the (sum,
// compensation) pairs are combined by a butterfly of two-sums.
__device__ __forceinline__ void two_sum(double a, double b, double& s, double& e) {
  s = a + b;
  double bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

__global__ void k_energy_reduce(int nstruc, const StructGeom* geom, const double* __restrict__ E_atom,
                                double* __restrict__ E_struct) {
  const int lane = threadIdx.x & 31;
  const int sidx = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (sidx >= nstruc) return;
  const StructGeom& g = geom[sidx];
  double s = 0.0, c = 0.0;
  for (int a = lane; a < g.natoms; a += 32) {
    double t, e;
    two_sum(s, E_atom[g.atom_off + a], t, e);
    s = t;
    c += e;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    double so = __shfl_xor_sync(0xffffffffu, s, d);
    double co = __shfl_xor_sync(0xffffffffu, c, d);
    double t, e;
    two_sum(s, so, t, e);
    s = t;
    c = c + co + e;
  }
  if (lane == 0) E_struct[sidx] = s + c;
}

// Structures that have no chunks (at most AE_ECHUNK atoms): a warp each.
// Pairwise order (a lane's run, then a tree over the lanes): the rounding error
// stays within (AE_ECHUNK/32 + 5) ulp of sum |E_i|
__device__ __forceinline__ void energy_warp(int sidx, const EnergySum& e) {
  const int lane = threadIdx.x & 31;
  if (sidx >= e.nstruc) return;
  const int n = e.geom[sidx].natoms;
  if (n > AE_ECHUNK) return;
  const double* E = e.E_atom + e.geom[sidx].atom_off;
  double s = 0.0;
  for (int a = lane; a < n; a += 256) {
    double v[8];   // eight loads in flight
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = a + 32 * q < n ? E[a + 32 * q] : 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (a + 32 * q < n) s += v[q];
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  if (lane == 0) {
    e.E_struct[sidx] = s;
    if (e.E_out) e.E_out[sidx] = s;
  }
}
__global__ void k_energy_warp(EnergySum e) {
  energy_warp((blockIdx.x * blockDim.x + threadIdx.x) >> 5, e);
}

// the others: a block of 256 threads per chunk of AE_ECHUNK atoms (eight atoms a thread,
// then a tree); of a structure with several chunks the last block to finish
// adds them in the same way: one launch, the same order every time.  (One warp
// per chunk and a second kernel took 13 us at 4,000 atoms, a chain of 64 loads
// and FP64 additions.  4,095 structures of 145 atoms and one of 4,096, the energy
// stage: 496 us with one last block that added the chunks of every structure,
// 39 with a block for each structure, 12 like this.)
__device__ __forceinline__ double block_sum256(double s, double* ws) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  s = ws[threadIdx.x & 7];
#pragma unroll
  for (int d = 4; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  return s;
}
__device__ __forceinline__ void energy_chunk(int c, const EnergySum& e) {
  __shared__ double ws[8];
  __shared__ bool s_last;
  const int sidx = e.chunk_struct[c];
  const StructGeom& g = e.geom[sidx];
  const int c0 = g.chunk_off, count = (g.natoms + AE_ECHUNK - 1) / AE_ECHUNK;
  const int a0 = (c - c0) * AE_ECHUNK, a1 = min(g.natoms, a0 + AE_ECHUNK);
  double s = 0.0;
#pragma unroll
  for (int q = 0; q < AE_ECHUNK / 256; ++q) {
    const int a = a0 + q * 256 + threadIdx.x;
    if (a < a1) s += e.E_atom[g.atom_off + a];
  }
  s = block_sum256(s, ws);
  if (count > 1) {
    if (threadIdx.x == 0) {
      e.part[c] = s;
      __threadfence();
      s_last = atomicAdd(e.ticket + sidx, 1u) == (unsigned)count - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const volatile double* vp = e.part + c0;
    s = 0.0;
    for (int k = threadIdx.x; k < count; k += 256) s += vp[k];
    s = block_sum256(s, ws);
    if (threadIdx.x == 0) e.ticket[sidx] = 0u;
  }
  if (threadIdx.x == 0) {
    e.E_struct[sidx] = s;
    if (e.E_out) e.E_out[sidx] = s;
  }
}
// block b of a launch of energy_blocks(e) blocks of 256 threads: the chunks
// first, as they take longest
__device__ __forceinline__ void energy_block(int b, const EnergySum& e) {
  if (b < e.nchunks) energy_chunk(b, e);
  else energy_warp(((b - e.nchunks) * 256 + threadIdx.x) >> 5, e);
}
__global__ void __launch_bounds__(256) k_energy_blocks(EnergySum e) { energy_block(blockIdx.x, e); }

template <typename T>
__global__ void k_forces_out(int natoms, const T* __restrict__ Facc, double* __restrict__ F,
                             double f) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= natoms) return;
  F[3 * i] = f * (double)Facc[4 * i];
  F[3 * i + 1] = f * (double)Facc[4 * i + 1];
  F[3 * i + 2] = f * (double)Facc[4 * i + 2];
}

// The results of a pass in one launch: the first `eblocks` blocks sum the
// energies (energy_block), the others write the forces and
// copy the atoms' energies.  The sums are a chain of loads and FP64 additions
// of a few blocks, as long as a launch of its own at any size; here it runs
// beside the forces (one pass of 256 Cu atoms 62 -> 53 us, with the grouping by
// species inside the search).
template <typename T>
__global__ void __launch_bounds__(256) k_results(int eblocks, EnergySum e, int natoms, const T* __restrict__ Facc,
                                                 double* __restrict__ F, double f,
                                                 double* __restrict__ E_atoms) {
  wait_for_previous();
  if ((int)blockIdx.x < eblocks) {
    energy_block(blockIdx.x, e);
    return;
  }
  const int i = (blockIdx.x - eblocks) * 256 + threadIdx.x;
  if (i >= natoms) return;
  if (F) {
    F[3 * i] = f * (double)Facc[4 * i];
    F[3 * i + 1] = f * (double)Facc[4 * i + 1];
    F[3 * i + 2] = f * (double)Facc[4 * i + 2];
  }
  if (E_atoms) E_atoms[i] = e.E_atom[i];
}

__global__ void k_types(int natoms, const int* __restrict__ t1, int* __restrict__ t0, int ntypes,
                        unsigned* status) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= natoms) return;
  int t = t1[i] - 1;
  if (t < 0 || t >= ntypes) {
    atomicOr(status, AE_ST_BAD_TYPE);
    t = 0;
  }
  t0[i] = t;
}

// FP32 FMA throughput probe: independent FMA chains per thread, enough
// blocks to fill every SM.  Used only to measure the denominator of the
// FP32 roofline of the descriptor kernels.
__global__ void k_fma_peak(float* out, int iters, float seed) {
  float a0 = seed + threadIdx.x, a1 = a0 + 1.f, a2 = a0 + 2.f, a3 = a0 + 3.f;
  float a4 = a0 + 4.f, a5 = a0 + 5.f, a6 = a0 + 6.f, a7 = a0 + 7.f;
  const float m = 0.999999f, c = 1e-7f;
  for (int k = 0; k < iters; ++k) {
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      a0 = fmaf(a0, m, c); a1 = fmaf(a1, m, c); a2 = fmaf(a2, m, c); a3 = fmaf(a3, m, c);
      a4 = fmaf(a4, m, c); a5 = fmaf(a5, m, c); a6 = fmaf(a6, m, c); a7 = fmaf(a7, m, c);
    }
  }
  float r = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (r == 12345.678f) out[blockIdx.x] = r;
}

}  // namespace

int ae_fma_peak(double* tflops, cudaStream_t s) {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  float* out = nullptr;
  if (cudaMalloc(&out, 4096 * sizeof(float)) != cudaSuccess) return 1;
  const int blocks = nsm * 8, threads = 256, iters = 4096;
  k_fma_peak<<<blocks, threads, 0, s>>>(out, 16, 1.f);   // warm-up
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  float best = 1e30f;
  for (int rep = 0; rep < 5; ++rep) {
    cudaEventRecord(e0, s);
    k_fma_peak<<<blocks, threads, 0, s>>>(out, iters, 1.f);
    cudaEventRecord(e1, s);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms < best) best = ms;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  double flops = 2.0 * 8 * 16 * (double)iters * blocks * threads;
  *tflops = flops / (best * 1e-3) / 1e12;
  return (int)cudaGetLastError();
}

int ae_launch_types(int natoms, const int* types1, int* types0, int ntypes, unsigned* status,
                    cudaStream_t s) {
  if (natoms <= 0) return 0;
  k_types<<<(natoms + 255) / 256, 256, 0, s>>>(natoms, types1, types0, ntypes, status);
  return (int)cudaGetLastError();
}

namespace {
constexpr size_t MLP_SMEM_MAX = 227 * 1024;   // (no static shared memory beside it)
template <typename T>
size_t mlp_smem(int wtotal) {
  return sizeof(T) * ((((size_t)wtotal + 1) & ~(size_t)1) + (size_t)MLP_WARPS * mlp_warp_elems());
}

template <typename T>
int launch_mlp(const PotDevice& pd, const DescBuffers& b, const T* W, int wtotal, int nsm,
               cudaStream_t s) {
  const size_t smem = mlp_smem<T>(wtotal);
  allow_smem(k_mlp<T>, smem, MLP_SMEM_MAX);
  const int blocks = min((b.natoms + MLP_WARPS - 1) / MLP_WARPS, nsm * 4);
  launch_next(k_mlp<T>, blocks, 32 * MLP_WARPS, smem, s, pd, b, W, wtotal);
  return (int)cudaGetLastError();
}

// Whether the FP64 networks go by tiles of atoms (k_mlp64): where their layers,
// of up to 32 nodes, leave a third of the lanes of a warp per atom idle, the
// weights leave room for several blocks on an SM, and the atoms fill the SMs
// (or, for one small network, are few).  The measure is the FP64 instructions
// of an atom's layers, a warp each and flattened, with tanh at 45 (the
// library's two branches) and 32.  A warp per atom and tiles (us): 26-20-20-1
// 2,304 atoms 31 and 33, 2,916 55 and 45, 32,000 348 and 252, 256 20 and 17, 864
// 21 and 23; 40-25-25-1 two species 2,916 74 and 55, 10,976 170 and 158; but
// 32-32-32-1 three species 8,255 125 and 165, 72,519 967 and 942; rutile's 9,000
// 170 and 207; 32-50-50-1 1.0 to 1.2 times as long by tiles; five species
// 57-20-20-1 (63 KB of weights) of 4,496 72 and 119, eight species 32-32-32-1 of
// 1,000 31 and 74.
bool networks_in_tiles(const PotDevice& pd, const DescBuffers& b, int wtotal, int nsm) {
  if (mlp_smem<double>(wtotal) > MLP_SMEM_MAX) return true;
  if (wtotal > 4096) return false;
  const bool many = b.natoms >= 16 * nsm;
  const bool few = b.natoms >= 32 && b.natoms <= 4 * nsm && wtotal <= 2048;
  if (!many && !few) return false;
  long long warp = 0, flat = 0;   // 32 lanes each
  int widest = 0;
  for (int t = 0; t < pd.ntypes; ++t) {
    const NetTable& net = pd.sp[t].net;
    for (int l = 0; l + 1 < net.nlayers - 1; ++l) {
      const int in = net.nnodes[l], out = net.nnodes[l + 1];
      widest = max(widest, out);
      warp += 32 * ((out + 31) / 32 * (in + 45) + (in + 31) / 32 * out);
      flat += out * (in + 32) + in * out;
    }
  }
  return widest <= 32 && 10 * warp >= 15 * flat;
}

int launch_mlp64(const PotDevice& pd, const DescBuffers& b, int wtotal, int nsm, cudaStream_t s) {
  Mlp64Shape sh{};
  int hidden = 0;
  for (int t = 0; t < pd.ntypes; ++t) {
    const NetTable& net = pd.sp[t].net;
    hidden = max(hidden, net.nlayers - 2);
    for (int l = 1; l < net.nlayers - 1; ++l) sh.hmax = max(sh.hmax, net.nnodes[l]);
  }
  sh.hmax |= 1;
  sh.in = pd.nsf_pad | 1;
  sh.per = (sh.in + 2 * hidden * sh.hmax) | 1;
  // eight atoms per warp where that leaves two warps per SM or more, fewer
  // for few atoms or long rows
  auto bytes = [&](int tile) {
    return sizeof(double) * ((size_t)wtotal + (size_t)MLP64_WARPS * tile * sh.per);
  };
  sh.tile = 8;
  while (sh.tile > 1 && (b.natoms < 2 * nsm * MLP64_WARPS * sh.tile || bytes(sh.tile) > 110 * 1024))
    sh.tile /= 2;
  const size_t need = bytes(sh.tile);
  allow_smem(k_mlp64, need, AE_SMEM_MAX);
  const int tiles = (b.natoms + sh.tile - 1) / sh.tile;
  const int blocks = min((tiles + MLP64_WARPS - 1) / MLP64_WARPS, nsm * 4);
  launch_next(k_mlp64, blocks, 32 * MLP64_WARPS, need, s, pd, b, wtotal, sh);
  return (int)cudaGetLastError();
}
}  // namespace

int ae_launch_mlp(const PotDevice& pd, const DescBuffers& b, int fp64, cudaStream_t s) {
  if (b.natoms <= 0) return 0;
  int wtotal = 0;
  for (int t = 0; t < pd.ntypes; ++t) wtotal = max(wtotal, pd.sp[t].net.wtotal);
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (!fp64) return launch_mlp<float>(pd, b, pd.w32, wtotal, nsm, s);
  return networks_in_tiles(pd, b, wtotal, nsm) ? launch_mlp64(pd, b, wtotal, nsm, s)
                                               : launch_mlp<double>(pd, b, pd.w64, wtotal, nsm, s);
}

namespace {
// (a single structure has chunks at any size)
int energy_blocks(const EnergySum& e) {
  return e.nchunks + (e.nstruc > 1 || e.nchunks == 0 ? (e.nstruc + 7) / 8 : 0);
}
}  // namespace

int ae_launch_energy_reduce_chunked(const EnergySum& e, cudaStream_t s) {
  if (e.nstruc <= 0) return 0;
  if (e.nchunks == 0)   // (two warps a block spread better)
    k_energy_warp<<<(e.nstruc + 1) / 2, 64, 0, s>>>(e);
  else
    k_energy_blocks<<<energy_blocks(e), 256, 0, s>>>(e);
  return (int)cudaGetLastError();
}

int ae_launch_results(const EnergySum& e, int natoms, const void* Facc, int fp64, double* F,
                      double sign, double* E_atoms, cudaStream_t s) {
  const int eblocks = e.nstruc > 0 ? energy_blocks(e) : 0;
  const int blocks = eblocks + (F || E_atoms ? (natoms + 255) / 256 : 0);
  if (blocks == 0) return 0;
  if (fp64)
    launch_next(k_results<double>, blocks, 256, 0, s, eblocks, e, natoms, (const double*)Facc, F,
                sign, E_atoms);
  else
    launch_next(k_results<float>, blocks, 256, 0, s, eblocks, e, natoms, (const float*)Facc, F, sign,
                E_atoms);
  return (int)cudaGetLastError();
}

int ae_launch_energy_reduce(int nstruc, const StructGeom* geom, const double* E_atom,
                            double* E_struct, cudaStream_t s) {
  if (nstruc <= 0) return 0;
  k_energy_reduce<<<(nstruc + 7) / 8, 256, 0, s>>>(nstruc, geom, E_atom, E_struct);
  return (int)cudaGetLastError();
}

int ae_launch_forces_out(int natoms, const void* Facc, int fp64, double* F, double sign,
                         cudaStream_t s) {
  if (natoms <= 0) return 0;
  if (fp64)
    k_forces_out<double><<<(natoms + 255) / 256, 256, 0, s>>>(natoms, (const double*)Facc, F, sign);
  else
    k_forces_out<float><<<(natoms + 255) / 256, 256, 0, s>>>(natoms, (const float*)Facc, F, sign);
  return (int)cudaGetLastError();
}
