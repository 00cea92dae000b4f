// Coloured Gauss-Seidel sweeps (sm_100a).
//
// A sweep visits the colours in order; the rows of one colour are
// independent, and each colour needs the results of the ones before it.  On
// the levels below the finest the rows couple to tens or hundreds of others,
// so there are 10 to 170 colours of 17 to 500 rows each: the work of a
// colour is under a microsecond, and a plain launch per colour (5.7 us each
// with its drain) was nearly the whole time of a solve.  What bounds a sweep
// is the chain from colour to colour.  Measured on the default configuration
// at 64^3 (458 colours on 7 levels, FP64 PCG, 14 iterations): 82.7 ms with
// plain launches, 40.4 ms with dependent launches that load a row's entries
// ahead, 16.0 ms with the cluster kernel on the levels it fits (14.9 ms with the
// later changes to the other kernels of the cycle).  Two kernels:
//
//   k_gs_cluster  every colour of every sweep in one launch of one
//       thread-block cluster.  Each block keeps the whole iterate in its
//       shared memory and gathers from there; a row's new value is stored
//       into the copies of all blocks (distributed shared memory) by
//       st.async, which also counts its bytes on the receiving block's
//       mbarrier of that colour.  A row waits for its own block's mbarriers
//       of all earlier colours, so nothing but the arrival of the values
//       separates one colour from the next.  A value is sent only after its
//       row's gathers, so no value of a later colour can overwrite one that
//       is still to be read.  Rows are dealt to the cluster's row groups in
//       colour order, one after another across colours, so a group's next
//       row is usually several colours away; its entries (up to 16 per lane)
//       are loaded into registers before the wait, its bounds one row
//       earlier still.  Per colour 0.55 us (rows of 100 entries) to 0.95 us
//       (250 entries, up to 600).  A hardware cluster barrier per colour in
//       place of the counted stores took 1.9 us per colour; loading the next
//       row before the current one is summed (8 entries per lane of both in
//       registers) 1.5 us on the 250-entry rows, whose remainder then had to
//       be loaded inside the colour.
//   k_gs_color    one colour per launch over the whole GPU, for levels whose
//       iterate does not fit in shared memory or whose colours hold many
//       rows; launched with programmatic stream serialization, the row's
//       bounds and first entries loaded before the wait for the previous
//       colour; 1 to 32 lanes per row by its length (gs_color_lanes).
//
// Row update: x_i += invd_i·(b_i - A_i x)          (src/smoothers.jl:203-217)
#pragma once

#include "dr_kernels.cuh"

namespace dr {
namespace kern {

constexpr int kGsThreads = 512;  // threads per block of the cluster kernel
constexpr int kGsBatch = 8;      // entries per lane loaded ahead (k_gs_color)
constexpr int kGsClusterBatch = 16;  // the same in k_gs_cluster

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_map(unsigned saddr, unsigned rank) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  return a;
}
// Store a value into a block's shared memory and count its bytes on that
// block's mbarrier.
__device__ __forceinline__ void cluster_send(unsigned addr, double v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr), "d"(v),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cluster_send(unsigned addr, float v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(addr), "f"(v),
               "r"(bar)
               : "memory");
}
// Bounded wait for the first phase of a mbarrier that blocks of the cluster
// count on.
__device__ __forceinline__ bool cluster_wait_bounded(uint64_t* bar, int limit) {
  for (int i = 0; i < limit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar))
        : "memory");
    if (ok) return true;
  }
  return false;
}

// A row (meta: row, first and last + 1 entry, colour) and the first B
// entries of each of its G lanes.  Slots past the row's end repeat its last
// entry; an empty row loads nothing.
template <int G, int B, typename T>
struct GsRow {
  int4 m = {0, 0, 0, 0};
  int c[B];
  T v[B];
  __device__ __forceinline__ void load(const int4& mm, int lane, const int* __restrict__ ci,
                                       const T* __restrict__ av) {
    m = mm;
#pragma unroll
    for (int h = 0; h < B; h += 8)
      if (m.y + h * G < m.z) {
#pragma unroll
        for (int j = h; j < h + 8; ++j) {
          const int k = min(m.y + lane + j * G, m.z - 1);
          c[j] = __ldg(ci + k);
          v[j] = __ldg(av + k);
        }
      }
  }
  // Σ a_ij x_j over this lane's entries, in four interleaved sums (with one
  // lane per row, a row's rounding errors are then those of a sum over four
  // lanes)
  __device__ __forceinline__ T dot(int lane, const int* __restrict__ ci, const T* __restrict__ av,
                                   const T* x) const {
    T s[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
    for (int h = 0; h < B; h += 8)
      if (m.y + h * G < m.z) {
        T xv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) xv[j] = x[c[h + j]];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (m.y + lane + (h + j) * G < m.z) s[j & 3] += v[h + j] * xv[j];
      }
    for (int k = m.y + lane + B * G; k < m.z; k += G) s[0] += __ldg(av + k) * x[__ldg(ci + k)];
    return (s[0] + s[1]) + (s[2] + s[3]);
  }
};

// The lanes of a row's group in the warp.
template <int G>
__device__ __forceinline__ unsigned group_mask() {
  return G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (threadIdx.x & 31 & ~(G - 1)));
}

// Dynamic shared memory of k_gs_cluster: the iterate, then one mbarrier per
// colour and sweep.
template <typename T>
__host__ __device__ constexpr size_t gs_cluster_smem(int n, long long colours) {
  return (((size_t)n * sizeof(T) + 15) & ~(size_t)15) + (size_t)colours * 8;
}

// Sweeps over all colours of one level in one cluster (gridDim.x = cluster
// size).  coff[0..ncolors]: first position of each colour in meta; x: the
// iterate in global memory, read at the start and written at the end.
// wait_limit: polls of a colour's mbarrier before a thread gives up and flags
// the error.
template <int G, typename T>
__global__ void __launch_bounds__(kGsThreads, 1)
k_gs_cluster(int n, int ncolors, const int* __restrict__ coff, const int4* __restrict__ meta,
             const int* __restrict__ ci, const T* __restrict__ av, const T* __restrict__ b,
             const T* __restrict__ invd, T* __restrict__ x, int steps, int* err, int wait_limit) {
  extern __shared__ __align__(16) unsigned char gs_smem[];
  T* const xs = reinterpret_cast<T*>(gs_smem);
  uint64_t* const bars = reinterpret_cast<uint64_t*>(gs_smem + gs_cluster_smem<T>(n, 0));
  const unsigned C = cluster_size(), rank = cluster_rank();
  const int lane = threadIdx.x & (G - 1);
  const unsigned gmask = group_mask<G>();
  // row groups numbered so that consecutive rows go to different blocks
  const int NG = (int)C * (kGsThreads / G);
  const int g0 = (threadIdx.x / G) * (int)C + (int)rank;
  const int mine = g0 < n ? (n - g0 + NG - 1) / NG : 0;  // this group's rows in a sweep
  const int total = mine * steps, nphase = ncolors * steps;
  auto at = [&](int t) { return g0 + (t < mine ? t : t % mine) * NG; };

  // the patterns and matrix values are never written by a kernel in flight
  GsRow<G, kGsClusterBatch, T> cur;
  int4 m1 = {0, 0, 0, 0};
  if (total > 0) cur.load(__ldg(meta + at(0)), lane, ci, av);
  if (total > 1) m1 = __ldg(meta + at(1));
  for (int k = threadIdx.x; k < nphase; k += kGsThreads) {
    const int c = k % ncolors;
    mbar_init(bars + k, 1);
    mbar_expect_tx(bars + k, (uint32_t)(__ldg(coff + c + 1) - __ldg(coff + c)) * (uint32_t)sizeof(T));
  }
  fence_mbar_init();
  pdl_trigger();
  pdl_wait();
  T cb = T(0), cd = T(0);
  if (total > 0) {
    cb = __ldg(b + cur.m.x);
    cd = __ldg(invd + cur.m.x);
  }
  for (int i = threadIdx.x; i < n; i += kGsThreads) xs[i] = x[i];
  __syncwarp();
  cluster_arrive();  // every block's copy and mbarriers are ready before any send
  cluster_wait();
  const unsigned xs_addr = smem_u32(xs), bars_addr = smem_u32(bars);
  int waited = 0;
  // A thread whose wait runs out reads no more of the iterate, but its rows
  // are still sent (the results are discarded), so that every mbarrier's bytes
  // arrive and no group is left short of a lane.
  bool ok = true;
  for (int t = 0; t < total; ++t) {
    const int phase = (t < mine ? 0 : t / mine * ncolors) + cur.m.w;
    while (waited < phase && ok) {
      ok = cluster_wait_bounded(bars + waited, wait_limit);
      waited += ok;
    }
    T sum = ok ? cur.dot(lane, ci, av, xs) : T(0);
#pragma unroll
    for (int o = G >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(gmask, sum, o);
    const T xn = xs[cur.m.x] + cd * (cb - sum);
    __syncwarp(gmask);  // every lane has read the old value
    const unsigned xa = xs_addr + (unsigned)cur.m.x * (unsigned)sizeof(T);
    const unsigned ba = bars_addr + (unsigned)phase * 8u;
    for (unsigned q = lane; q < C; q += G) cluster_send(cluster_map(xa, q), xn, cluster_map(ba, q));
    // the next row's entries, on their way while the colours in between finish
    if (t + 1 < total) {
      cur.load(m1, lane, ci, av);
      cb = __ldg(b + m1.x);
      cd = __ldg(invd + m1.x);
      if (t + 2 < total) m1 = __ldg(meta + at(t + 2));
    }
  }
  // Every value sent to this block has arrived before it writes its part of x
  // and leaves, also when a wait gave up on the way.
  bool landed = true;
  while (waited < nphase && landed) {
    landed = cluster_wait_bounded(bars + waited, kWaitLimit);
    waited += landed;
  }
  if (!ok || !landed) atomicExch(err, 1);
  __syncwarp();
  cluster_arrive();  // this block sends no more: the others may leave
  for (int i = (int)rank * kGsThreads + (int)threadIdx.x; i < n; i += (int)C * kGsThreads) x[i] = xs[i];
  __syncwarp();
  cluster_wait();
}

// Gauss-Seidel update of one colour: `cnt` rows from meta.
template <int G, typename T>
__global__ void __launch_bounds__(kBlock)
k_gs_color(int cnt, const int4* __restrict__ meta, const int* __restrict__ ci, const T* __restrict__ av,
           const T* __restrict__ b, const T* __restrict__ invd, T* x) {
  constexpr int GPB = kBlock / G;
  const int lane = threadIdx.x & (G - 1);
  const int stride = gridDim.x * GPB;
  int idx = blockIdx.x * GPB + threadIdx.x / G;
  const unsigned gmask = group_mask<G>();
  GsRow<G, kGsBatch, T> r;
  if (idx < cnt) r.load(__ldg(meta + idx), lane, ci, av);  // never written by a kernel in flight
  pdl_trigger();
  pdl_wait();
  while (idx < cnt) {
    // x of the same colour is never a neighbour, so plain loads are safe
    const int row = r.m.x;
    const T bi = __ldg(b + row), di = __ldg(invd + row), xi = x[row];
    T sum = r.dot(lane, ci, av, x);
    idx += stride;
    if (idx < cnt) r.load(__ldg(meta + idx), lane, ci, av);
#pragma unroll
    for (int o = G >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(gmask, sum, o);
    if (lane == 0) x[row] = xi + di * (bi - sum);
  }
}

}  // namespace kern
}  // namespace dr
