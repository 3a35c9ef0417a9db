// reduce.cuh -- single-launch grid reductions with a device-side finalize.
//
// Every block reduces its NRED per-thread doubles (warp shuffles, then one
// value per warp in shared memory) and writes them to its partial slot
// partials[(rhs * nslots + slot) * NRED + k].  The last block to arrive (an
// atomic ticket on `counter`) sums, for each right-hand side, its nslots
// partials in a fixed strided order followed by a fixed shuffle / shared-memory
// tree, so the result does not depend on which block finished last, and hands
// the totals to f.finalize(rhs, tot) on the device.  The ticket is reset for
// the next launch on the same stream.  A functor with a member
// finalize_warp(rhs, tot, lane) has it run by the 32 lanes of a warp instead
// (scalar updates over many entries, e.g. the shifts of a multi-shift solve or
// a Hessenberg column, then take one round of global-memory latency, not one
// per entry, and a few registers per lane).
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

namespace clg {

template <class F, class = void>
struct has_warp_finalize : std::false_type {};
template <class F>
struct has_warp_finalize<F, std::void_t<decltype(&F::finalize_warp)>> : std::true_type {};

// A reduction whose result the next kernel needs can leave the last step to it:
// the producer's blocks only write their partials (block_partials) and end, and
// every block of the consumer adds them up itself (block_total, the same order
// in every block) while its own loads are in flight.  The fence, the ticket,
// the last block's second pass and its scalar update, 4 to 6 us at the end of a
// launch during which nothing else runs, become about 1 us beside other work.
// For few partials (a launch of one right-hand side); with many right-hand
// sides a kernel of one block each does it (epi_final_kernel), which still
// spares every block of the producer its fence and ticket.
template <int NRED>
__device__ __forceinline__ void block_partials(const double (&acc)[NRED], double* partials, int64_t slot) {
  __shared__ double sm[NRED][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < NRED; ++k) {
    double v = acc[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) sm[k][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < NRED) {
    double v = 0.0;
    for (int w = 0; w < nw; ++w) v += sm[threadIdx.x][w];
    partials[slot * NRED + threadIdx.x] = v;
  }
}
// sum of n partials, the same in every thread of the block (at most 8 warps)
__device__ __forceinline__ double block_total(const double* partials, int n) {
  __shared__ double sm[8];
  constexpr int U = 4;
  double s = 0.0;
  for (int i0 = threadIdx.x; i0 < n; i0 += U * (int)blockDim.x) {
    double v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * (int)blockDim.x;
      v[u] = i < n ? __ldcg(partials + i) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) s += v[u];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) t += sm[w];
  return t;
}
// A site functor with PARTIALS = true leaves its partials to the next kernel; one
// with a member prologue(rhs, first block) has it run by every thread before the
// sites (it may hold barriers) and returns whether there is work.
template <class F, class = void>
struct partials_only : std::false_type {};
template <class F>
struct partials_only<F, std::void_t<decltype(F::PARTIALS)>> : std::bool_constant<F::PARTIALS> {};
template <class F, class = void>
struct has_prefetch : std::false_type {};
template <class F>
struct has_prefetch<F, std::void_t<decltype(&F::prefetch)>> : std::true_type {};
template <class F, class = void>
struct has_prologue : std::false_type {};
template <class F>
struct has_prologue<F, std::void_t<decltype(&F::prologue)>> : std::true_type {};
// One with ONE_LATTICE = true belongs to solvers that clg_solve_lattices does not
// run, and has no batch form (launch_sites).
template <class F, class = void>
struct one_lattice : std::false_type {};
template <class F>
struct one_lattice<F, std::void_t<decltype(F::ONE_LATTICE)>> : std::bool_constant<F::ONE_LATTICE> {};

// The last block's part: totals per right-hand side -> f.finalize.  Called by
// every thread of that block (at most 256 threads, 8 warps).
template <int NRED, class F>
__device__ __forceinline__ void grid_final_reduce(const F& f, unsigned nslots, int nrhs, const double* partials,
                                                  unsigned* counter) {
  __shared__ double sm[NRED][8];
  __shared__ double tot[NRED];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = (blockDim.x + 31) >> 5;
  // U independent partial loads in flight per thread and step (fixed order)
  constexpr int U = NRED >= 8 ? 1 : 8 / NRED;
  // several right-hand sides: warp w sums and finalises rhs w, w + nw, ...
  // (each finalize touches only its own rhs's state), so the finalize
  // latencies of up to nw right-hand sides overlap and no block barrier
  // separates them
  if (nrhs > 1) {
    for (int r = warp; r < nrhs; r += nw) {
      double s[NRED];
#pragma unroll
      for (int k = 0; k < NRED; ++k) s[k] = 0.0;
      const double* pr = partials + (int64_t)r * nslots * NRED;
      for (unsigned b0 = lane; b0 < nslots; b0 += U * 32) {
        double v[U][NRED];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const unsigned b = b0 + u * 32;
#pragma unroll
          for (int k = 0; k < NRED; ++k) v[u][k] = b < nslots ? __ldcg(pr + (int64_t)b * NRED + k) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int k = 0; k < NRED; ++k) s[k] += v[u][k];
      }
#pragma unroll
      for (int k = 0; k < NRED; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_down_sync(0xffffffffu, s[k], o);
      }
      if constexpr (has_warp_finalize<F>::value) {
#pragma unroll
        for (int k = 0; k < NRED; ++k) s[k] = __shfl_sync(0xffffffffu, s[k], 0);
        f.finalize_warp(r, s, lane);
      } else {
        if (lane == 0) f.finalize(r, s);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) *counter = 0u;
    return;
  }
  for (int r = 0; r < nrhs; ++r) {
    double s[NRED];
#pragma unroll
    for (int k = 0; k < NRED; ++k) s[k] = 0.0;
    const double* pr = partials + (int64_t)r * nslots * NRED;
    for (unsigned b0 = threadIdx.x; b0 < nslots; b0 += U * blockDim.x) {
      double v[U][NRED];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned b = b0 + u * blockDim.x;
#pragma unroll
        for (int k = 0; k < NRED; ++k) v[u][k] = b < nslots ? __ldcg(pr + (int64_t)b * NRED + k) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int k = 0; k < NRED; ++k) s[k] += v[u][k];
    }
#pragma unroll
    for (int k = 0; k < NRED; ++k) {
      double v = s[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) sm[k][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < NRED) {
      double v = 0.0;
      for (int w = 0; w < nw; ++w) v += sm[threadIdx.x][w];
      tot[threadIdx.x] = v;
    }
    __syncthreads();
    if constexpr (has_warp_finalize<F>::value) {
      if (threadIdx.x < 32) f.finalize_warp(r, tot, (int)threadIdx.x);
    } else {
      if (threadIdx.x == 0) f.finalize(r, tot);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *counter = 0u;
}

// Block partials + ticket + (last block) final reduction.  `contribute` must be
// uniform over the block: a block that does not contribute (its right-hand
// side is finished) writes no partial and only takes its ticket, so the caller's
// finalize must ignore the totals of such right-hand sides.
template <int NRED, class F>
__device__ __forceinline__ void grid_reduce_finalize(double (&acc)[NRED], const F& f, int rhs, unsigned slot,
                                                     unsigned nslots, int nrhs, double* partials, unsigned* counter,
                                                     bool contribute = true) {
  __shared__ double sm[NRED][8];
  __shared__ bool last;
  if (contribute) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < NRED; ++k) {
      double v = acc[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) sm[k][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < NRED) {
      double v = 0.0;
      for (int w = 0; w < nw; ++w) v += sm[threadIdx.x][w];
      partials[((int64_t)rhs * nslots + slot) * NRED + threadIdx.x] = v;
      // only the partials must be visible to the last block before the ticket
      __threadfence();
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const unsigned t = atomicAdd(counter, 1u);
    last = (t == nslots * (unsigned)nrhs - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  grid_final_reduce<NRED>(f, nslots, nrhs, partials, counter);
}

// Two-level form for grids with many blocks per right-hand side (the residual
// hops' epilogues: one block per 32-256 sites, thousands per right-hand side).
// `contribute` (uniform over the block) says whether the block writes a partial
// of right-hand side rhs.  The slots of each right-hand side are grouped by
// `group`; the block that completes a group (ticket counter[1 + rhs * ngroups +
// g]) sums the group's partials in slot order and writes the group total to
// gpart[(rhs * ngroups + g) * NRED + k]; the block that completes the last group
// of all (ticket counter[0]) runs grid_final_reduce over the group totals.  No
// block reads more than `group` partials, every sum has a fixed order
// (deterministic), and the tickets are reset for the next launch.
template <int NRED, class F>
__device__ __forceinline__ void grid_reduce_finalize2(double (&acc)[NRED], const F& f, int rhs, bool contribute,
                                                      unsigned slot, unsigned nslots, int nrhs, unsigned group,
                                                      double* partials, double* gpart, unsigned* counter) {
  __shared__ double sm[NRED][8];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = (blockDim.x + 31) >> 5;
  if (contribute) {
#pragma unroll
    for (int k = 0; k < NRED; ++k) {
      double v = acc[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) sm[k][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < NRED) {
      double v = 0.0;
      for (int w = 0; w < nw; ++w) v += sm[threadIdx.x][w];
      partials[((int64_t)rhs * nslots + slot) * NRED + threadIdx.x] = v;
      __threadfence();
    }
    __syncthreads();
  }
  const unsigned ngroups = (nslots + group - 1) / group;
  const unsigned g = slot / group;
  const unsigned g0 = g * group;
  const unsigned gs = min(group, nslots - g0);
  unsigned* gc = counter + 1 + (int64_t)rhs * ngroups + g;
  if (threadIdx.x == 0) last = atomicAdd(gc, 1u) == gs - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // this block completed group g of its right-hand side: the total, in slot order
  double s[NRED];
#pragma unroll
  for (int k = 0; k < NRED; ++k) s[k] = 0.0;
  const double* pg = partials + ((int64_t)rhs * nslots + g0) * NRED;
  for (unsigned b = threadIdx.x; b < gs; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < NRED; ++k) s[k] += __ldcg(pg + (int64_t)b * NRED + k);
#pragma unroll
  for (int k = 0; k < NRED; ++k) {
    double v = s[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) sm[k][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < NRED) {
    double v = 0.0;
    for (int w = 0; w < nw; ++w) v += sm[threadIdx.x][w];
    gpart[((int64_t)rhs * ngroups + g) * NRED + threadIdx.x] = v;
    __threadfence();
  }
  if (threadIdx.x == 0) *gc = 0u;
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == ngroups * (unsigned)nrhs - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  grid_final_reduce<NRED>(f, ngroups, nrhs, gpart, counter);
}

// The two-level reduction for blocks that each cover every right-hand side of
// one slot (the tile hops): each block has written partials[(rhs * nslots +
// blockIdx.x) * NRED + k] for the right-hand sides it computed (with a fence).
// The block that completes a group of `group` slots (ticket counter[1 + g])
// sums the group's partials per right-hand side in slot order (warp w takes
// rhs w, w + nwarps, ...) into gpart[(rhs * ngroups + g) * NRED + k]; the block
// that completes the last group runs grid_final_reduce over the group totals.
// Every block of the grid must call this (it has barriers).
template <int NRED, class F>
__device__ __forceinline__ void tile_reduce_finalize(const F& f, unsigned nslots, int nrhs, unsigned group,
                                                     const double* partials, double* gpart, unsigned* counter) {
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  const unsigned ngroups = (nslots + group - 1) / group;
  const unsigned g = blockIdx.x / group;
  const unsigned g0 = g * group;
  const unsigned gs = min(group, nslots - g0);
  unsigned* gc = counter + 1 + g;
  if (threadIdx.x == 0) last = atomicAdd(gc, 1u) == gs - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int r = warp; r < nrhs; r += nw) {
    double s[NRED];
#pragma unroll
    for (int k = 0; k < NRED; ++k) s[k] = 0.0;
    const double* pg = partials + ((int64_t)r * nslots + g0) * NRED;
    for (unsigned b = lane; b < gs; b += 32)
#pragma unroll
      for (int k = 0; k < NRED; ++k) s[k] += __ldcg(pg + (int64_t)b * NRED + k);
#pragma unroll
    for (int k = 0; k < NRED; ++k) {
      double v = s[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) gpart[((int64_t)r * ngroups + g) * NRED + k] = v;
    }
    if (lane == 0) __threadfence();
  }
  if (threadIdx.x == 0) *gc = 0u;
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == ngroups - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  grid_final_reduce<NRED>(f, ngroups, nrhs, gpart, counter);
}

}  // namespace clg
