// batchq.cuh -- the work queue of a batched launch: many problems' launches
// of one kernel run by one grid of persistent CTAs.
//
// A batched launch is a table of per-problem launch records and a map of
// items (record, block of that record's own grid) in record order.  The CTAs
// take chunks of items from an atomic counter (one item each while a launch
// fits in one wave); an item runs that
// block of that problem's launch.  A problem whose solve has stopped has
// nothing to do in any of its blocks, so the CTA that meets one of its items
// skips the rest of that record's items in its chunk at once and moves the
// counter past the record's last item: a converged problem costs a few
// counter steps, not a block launch (or a chunk) each.  The last CTA to
// leave resets the counters for the next launch on the stream.
#pragma once
#include <algorithm>

#include "icb_internal.hpp"
#include "reduce.cuh"

namespace icb
{
/// a block's coordinates and its grid's extent: blockIdx / gridDim of a
/// launch of its own, or the block's place in one grid of a batched launch
struct Blk
{
  unsigned x, y, z, gx, gy, gz;
};
__device__ __forceinline__ Blk this_block()
{
  return Blk{blockIdx.x, blockIdx.y, blockIdx.z, gridDim.x, gridDim.y, gridDim.z};
}

struct BatchQueue
{
  unsigned *next = nullptr; ///< items handed out
  unsigned *done = nullptr; ///< CTAs that have left
  int items = 0;
  int chunk = 1; ///< items a CTA takes at a time (queue_chunk)
};
/// items per chunk: 1 while every item gets a CTA of its own in one wave
/// (small launches stay fully parallel), more for launches many waves long,
/// so a converged problem's items are skipped several at a time
constexpr int kMaxChunk = 16;
inline int queue_chunk(int items, int capacity)
{
  return std::max(1, std::min(kMaxChunk, items / std::max(1, 2 * capacity)));
}

/// nb(rec): blocks of a record's own grid; skip(rec): the record's blocks
/// have nothing to do (read by one thread, the same for the whole record
/// while any of its blocks is pending); run(rec, b, n): blocks b .. b + n - 1
/// of the record, at most a chunk
template <class Rec, class Nb, class Skip, class Run>
__device__ __forceinline__ void batch_runs(const Rec *__restrict__ D, const int2 *__restrict__ map,
                                            const BatchQueue &q, Nb nb, Skip skip, Run run)
{
  __shared__ int base, jump;
  const bool lead = threadIdx.x == 0 && threadIdx.y == 0 && threadIdx.z == 0;
  for(;;)
  {
    if(lead)
      base = int(atomicAdd(q.next, unsigned(q.chunk)));
    __syncthreads();
    const int b0 = base;
    __syncthreads();
    if(b0 >= q.items)
      break;
    const int b1 = min(b0 + q.chunk, q.items);
    for(int it = b0; it < b1;)
    {
      const int2 m = map[it];
      const Rec &r = D[m.x];
      const int left = nb(r) - m.y;
      // a record found running stays so while any of its items is pending
      if(lead)
      {
        jump = skip(r) ? left : 0;
        // the record's items are contiguous in the map: move the queue
        // past its last one, so no CTA takes another chunk of it (chunks
        // already taken skip it here)
        if(jump > 0)
          atomicMax(q.next, unsigned(it + jump));
      }
      __syncthreads();
      const int j = jump;
      __syncthreads();
      if(j > 0)
      {
        it += j;
        continue;
      }
      const int n = min(b1 - it, left);
      run(r, m.y, n);
      __syncthreads(); // the bodies' shared memory is reused by the next run
      it += n;
    }
  }
  if(lead)
  {
    __threadfence();
    const unsigned g = gridDim.x * gridDim.y * gridDim.z;
    if(atomicAdd(q.done, 1u) == g - 1)
    {
      *q.next = 0u;
      *q.done = 0u;
    }
  }
}

/// the items one at a time: run(rec, b, fresh), block b of the record, fresh
/// when it is the first of its run (what a body stages per record in shared
/// memory survives from there)
template <class Rec, class Nb, class Skip, class Run>
__device__ __forceinline__ void batch_queue(const Rec *__restrict__ D, const int2 *__restrict__ map,
                                            const BatchQueue &q, Nb nb, Skip skip, Run run)
{
  batch_runs(D, map, q, nb, skip, [&](const Rec &r, int b, int n) {
    for(int t = 0; t < n; t++)
    {
      if(t)
        __syncthreads();
      run(r, b + t, t == 0);
    }
  });
}

/// Blocks b0 .. b0 + n - 1 of a launch with a grid-wide sum (T threads, gx
/// blocks): acc(B, v) does block B's work and adds to v.  The blocks' partials,
/// and so the total, are those of their own launch; but the run has one
/// barrier, one fence and one ticket, where a block at a time takes those after
/// its few entries a thread -- a chain of latencies that bounded these kernels
/// (32 designs of 6.1M DOFs, a block at a time and in runs: residual update 96
/// and 66 us, r.z 49 and 35, x and p 76 and 50).  HALVES: the warps' sums are added by
/// halves and the blocks' by the first warp, as the one-kernel OC update does
/// (oc_exchange).
template <int NV, int T, bool HALVES = false, class Acc, class Fin>
__device__ __forceinline__ void sum_runs(int b0, int n, unsigned gx, const RedScratch &red,
                                         const Acc &acc, const Fin &fin)
{
  static_assert(!HALVES || NV == 1, "one value a block");
  __shared__ double part[kMaxChunk][T / 32][NV], sw[32][NV];
  __shared__ int last;
  const int tid = threadIdx.x;
  for(int t = 0; t < n; t++)
  {
    double v[NV] = {};
    acc(Blk{unsigned(b0 + t), 0, 0, gx, 1, 1}, v);
#pragma unroll
    for(int k = 0; k < NV; k++)
      v[k] = warp_sum_d(v[k]);
    if((tid & 31) == 0)
#pragma unroll
      for(int k = 0; k < NV; k++)
        part[t][tid >> 5][k] = v[k];
  }
  __syncthreads();
  static_assert(kMaxChunk * NV <= T, "a partial a thread");
  if(tid < n * NV)
  {
    double s = 0.0;
    if constexpr(HALVES)
      s = sum_by_halves<T / 32>([&](int w) { return part[tid / NV][w][tid % NV]; });
    else
      for(int w = 0; w < T / 32; w++)
        s += part[tid / NV][w][tid % NV];
    red.partials[(long long)b0 * NV + tid] = s;
    __threadfence();
  }
  __syncthreads();
  if(tid == 0)
    last = ticket_acq_rel(red.counter, unsigned(n)) + unsigned(n) == gx;
  __syncthreads();
  if(!last)
    return;
  __threadfence();
  if constexpr(HALVES)
    partials_finish_warp<T / 32>(red, fin, int(gx));
  else
    partials_finish<NV>(sw, red, fin, int(gx));
}

/// CTAs of a persistent batched launch (the kernel's residency on every SM,
/// no more than the chunks there are); sets q.chunk
inline int queue_grid(const void *kern, int threads, int smem, BatchQueue &q)
{
  int per = 0;
  if(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem) != cudaSuccess ||
     per < 1)
  {
    (void)cudaGetLastError();
    per = 1;
  }
  const int cap = per * num_sms();
  q.chunk = queue_chunk(q.items, cap);
  const int chunks = (q.items + q.chunk - 1) / q.chunk;
  return std::max(1, std::min(cap, chunks));
}
} // namespace icb
