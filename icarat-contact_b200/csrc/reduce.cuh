// reduce.cuh -- deterministic grid-wide reductions without a second launch.
//
// Every block reduces its values (warp shuffles, then shared memory) and
// writes them to red.partials[block]; the block that finishes last (atomic
// ticket) sums all partials in block order and hands the totals to a
// finisher functor run by its thread 0.  The summation order depends only on
// the launch shape, so results are bitwise reproducible run to run.
#pragma once
#include "icb_internal.hpp"

namespace icb
{

/// the ticket of the last-block pattern: an atomic add with acquire-release
/// semantics at GPU scope, which orders this thread's partial stores before
/// the ticket (release) and, for the last block, the other blocks' partials
/// before its reads (acquire) -- without a full sequentially consistent fence
__device__ __forceinline__ unsigned ticket_acq_rel(unsigned *counter, unsigned take = 1)
{
  unsigned t;
  asm volatile("atom.acq_rel.gpu.add.u32 %0, [%1], %2;"
               : "=r"(t)
               : "l"(counter), "r"(take)
               : "memory");
  return t;
}

__device__ __forceinline__ double warp_sum_d(double v)
{
#pragma unroll
  for(int o = 16; o > 0; o >>= 1)
    v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

/// w(0) .. w(NW - 1) added by halves: three additions deep for eight values instead of
/// eight
template <int NW, class W> __device__ __forceinline__ double sum_by_halves(const W &w)
{
  double v[NW];
#pragma unroll
  for(int q = 0; q < NW; q++)
    v[q] = w(q);
#pragma unroll
  for(int o = NW / 2; o > 0; o >>= 1)
#pragma unroll
    for(int q = 0; q < o; q++)
      v[q] += v[q + o];
  return v[0];
}

/// the last block's part of a grid-wide sum: the nb blocks' partials in a fixed
/// order (thread t takes t, t + blockDim, ...; then the warps in order), the
/// total handed to fin, the counter ready for the next launch
template <int NV, class Fin>
__device__ __forceinline__ void partials_finish(double (&sw)[32][NV], const RedScratch &red,
                                                const Fin &fin, int nb)
{
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nth = blockDim.x * blockDim.y * blockDim.z;
  const int nw = (nth + 31) >> 5;
  double s[NV];
#pragma unroll
  for(int k = 0; k < NV; k++)
    s[k] = 0.0;
  for(int b = tid; b < nb; b += nth)
#pragma unroll
    for(int k = 0; k < NV; k++)
      s[k] += __ldcg(red.partials + (long long)b * NV + k);
#pragma unroll
  for(int k = 0; k < NV; k++)
    s[k] = warp_sum_d(s[k]);
  __syncthreads();
  if((tid & 31) == 0)
#pragma unroll
    for(int k = 0; k < NV; k++)
      sw[tid >> 5][k] = s[k];
  __syncthreads();
  if(tid == 0)
  {
    double tot[NV];
#pragma unroll
    for(int k = 0; k < NV; k++)
    {
      tot[k] = 0.0;
      for(int w = 0; w < nw; w++)
        tot[k] += sw[w][k];
    }
    *red.counter = 0u;
    fin(tot);
  }
}

/// the same by the first warp alone, one value a block: lane l takes block l + 32 q
/// of every 32 N into sum q, adds the N sums by halves, then the lanes' are added
template <int N, class Fin>
__device__ __forceinline__ void partials_finish_warp(const RedScratch &red, const Fin &fin, int nb)
{
  const int lane = threadIdx.x;
  if(lane >= 32)
    return;
  double t[N];
#pragma unroll
  for(int q = 0; q < N; q++)
    t[q] = 0.0;
  for(int t0 = 0; t0 < nb; t0 += 32 * N)
  {
    double v[N];
#pragma unroll
    for(int q = 0; q < N; q++)
      v[q] = t0 + lane + 32 * q < nb ? __ldcg(red.partials + t0 + lane + 32 * q) : 0.0;
#pragma unroll
    for(int q = 0; q < N; q++)
      if(t0 + lane + 32 * q < nb)
        t[q] += v[q];
  }
  double s[1] = {warp_sum_d(sum_by_halves<N>([&](int q) { return t[q]; }))};
  if(lane == 0)
  {
    *red.counter = 0u;
    fin(s);
  }
}

/// the reduction of block `bid` of `nb` blocks: a batched launch that runs
/// several independent grids passes each block's index and count within its
/// own grid, so every grid reduces exactly as its own launch would
template <int NV, class Fin>
__device__ __forceinline__ void block_reduce_at(double (&v)[NV], const RedScratch &red, Fin fin,
                                                int bid, int nb)
{
  __shared__ double sw[32][NV];
  __shared__ int last;
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nth = blockDim.x * blockDim.y * blockDim.z;
  const int nw = (nth + 31) >> 5;
#pragma unroll
  for(int k = 0; k < NV; k++)
    v[k] = warp_sum_d(v[k]);
  if((tid & 31) == 0)
#pragma unroll
    for(int k = 0; k < NV; k++)
      sw[tid >> 5][k] = v[k];
  __syncthreads();
  if(tid == 0)
  {
#pragma unroll
    for(int k = 0; k < NV; k++)
    {
      double s = 0.0;
      for(int w = 0; w < nw; w++)
        s += sw[w][k];
      red.partials[(long long)bid * NV + k] = s;
    }
    const unsigned t = ticket_acq_rel(red.counter);
    last = (t == unsigned(nb - 1));
  }
  __syncthreads();
  if(!last)
    return;
  __threadfence();
  partials_finish<NV>(sw, red, fin, nb);
}

/// The finish of a sum whose partials sit at slots fixed by the work, not by
/// the block that computed them (so the launch may be cut into any number of
/// blocks): each block calls it once, after its threads stored their slots;
/// the last of the nb blocks to arrive sums slots [0, nslots) in a fixed order
/// (thread t takes t, t + blockDim, ...; then the warps in order) and hands
/// the total to fin.  `wrote`: this thread stored slots (it fences them).
template <class Fin>
__device__ __forceinline__ void slots_reduce_finish(const RedScratch &red, long long nslots,
                                                    int nb, bool wrote, Fin fin)
{
  __shared__ double sw[32];
  __shared__ int last;
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nth = blockDim.x * blockDim.y * blockDim.z;
  const int nw = (nth + 31) >> 5;
  if(wrote)
    __threadfence();
  __syncthreads();
  if(tid == 0)
    last = ticket_acq_rel(red.counter) == unsigned(nb - 1);
  __syncthreads();
  if(!last)
    return;
  __threadfence();
  // one block is left to sum them: its loads eight to a group, or the sum is
  // a chain of their latencies (640 x 320 elements, 7,704 slots on 128
  // threads)
  constexpr int G = 8;
  double s = 0.0;
  for(long long k = tid; k < nslots; k += (long long)G * nth)
  {
    double v[G];
#pragma unroll
    for(int g = 0; g < G; g++)
      v[g] = k + (long long)g * nth < nslots ? __ldcg(red.partials + k + (long long)g * nth) : 0.0;
#pragma unroll
    for(int g = 0; g < G; g++)
      if(k + (long long)g * nth < nslots)
        s += v[g];
  }
  s = warp_sum_d(s);
  if((tid & 31) == 0)
    sw[tid >> 5] = s;
  __syncthreads();
  if(tid == 0)
  {
    double tot = 0.0;
    for(int w = 0; w < nw; w++)
      tot += sw[w];
    *red.counter = 0u;
    fin(&tot);
  }
}

template <int NV, class Fin>
__device__ __forceinline__ void block_reduce(double (&v)[NV], const RedScratch &red,
                                             Fin fin)
{
  block_reduce_at<NV>(v, red, fin, blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z),
                      gridDim.x * gridDim.y * gridDim.z);
}

struct FinStore
{
  double *out;
  __device__ void operator()(const double *t) const { *out = t[0]; }
};

} // namespace icb
