// Stable partition of the atoms by species in one block of B threads, a tile of
// B atoms at a time: order (ascending index inside a species) and the species'
// offsets.
#pragma once

template <int B>
struct PartitionScratch {
  int cnt[AE_MAXT], tile[AE_MAXT];
  int wc[B / 32][AE_MAXT];
};

template <int B>
__device__ __forceinline__ void partition_block(int n, int ntypes, const int* types, int* order,
                                                int* spec_off, PartitionScratch<B>& s) {
  static_assert(B >= 32 && B <= 1024, "a lane per warp");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < AE_MAXT) s.cnt[threadIdx.x] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += B) atomicAdd(&s.cnt[types[i]], 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    int o = 0;
    for (int t = 0; t < ntypes; ++t) {
      const int c = s.cnt[t];
      spec_off[t] = o;
      s.cnt[t] = o;
      o += c;
    }
    spec_off[ntypes] = o;
  }
  for (int base = 0; base < n; base += B) {
    const int i = base + threadIdx.x;
    const int t = i < n ? types[i] : -1;
    unsigned mine = 0;
    __syncthreads();
    for (int q = 0; q < ntypes; ++q) {
      const unsigned m = __ballot_sync(0xffffffffu, t == q);
      if (q == t) mine = m;
      if (lane == 0) s.wc[warp][q] = __popc(m);
    }
    __syncthreads();
    // a warp per species scans the warps' counts
    for (int q = warp; q < ntypes; q += B / 32) {
      const int c = lane < B / 32 ? s.wc[lane][q] : 0;
      int x = c;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
      }
      if (lane < B / 32) s.wc[lane][q] = x - c;
      if (lane == 31) s.tile[q] = x;
    }
    __syncthreads();
    if (t >= 0) order[s.cnt[t] + s.wc[warp][t] + __popc(mine & ((1u << lane) - 1u))] = i;
    __syncthreads();
    if (threadIdx.x < ntypes) s.cnt[threadIdx.x] += s.tile[threadIdx.x];
  }
}
