// exchange.cuh -- sums over all CTAs of a cooperative kernel, several times a
// launch (pcgtile.cu, the OC update of opt.cu).
//
// Every CTA puts its sum in a slot of its own and one of its warps polls all
// slots.  A slot holds a pattern that no sum takes until it is written, so the
// value is its own flag; each CTA adds the same values in the same order, so all
// get the same bits.  Slots are used in turns of several sets; the set to be used
// next but one is emptied on the way (what orders that: see the callers).
#pragma once
#include "icb_internal.hpp"

namespace icb
{
/// doubles of a CTA's slots in a set: a 128-byte line of its own.  Lines that
/// several CTAs write while all poll them move between the L2's halves with
/// every write: an exchange of 117 CTAs takes 4.4 us with packed slots, 2.4 us
/// with 32 bytes each and 1.6 us with a line each (1.1 us for 20 CTAs).
constexpr int kExSlot = 16;
constexpr int kExCtas = 256;           ///< parts (CTAs or more) of an exchange at most
/// polls of a wait before a CTA gives up (about two seconds on a GPU that runs
/// nothing else), unless the option exchange_spin_limit says otherwise
constexpr unsigned kExPolls = 1u << 22;
constexpr unsigned long long kExEmpty = ~0ull;

#ifdef __CUDACC__
__device__ __forceinline__ void slot_store(double *s, unsigned long long b)
{
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(s), "l"(b) : "memory");
}
__device__ __forceinline__ void slot_put(double *s, double v)
{
  // a NaN keeps being one, but not the empty pattern
  slot_store(s, v != v ? 0x7ff8000000000000ull : (unsigned long long)__double_as_longlong(v));
}
/// acquire-release fence at GPU scope (__threadfence is sequentially consistent)
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ unsigned long long slot_read(const double *s)
{
  unsigned long long b;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(b) : "l"(s) : "memory");
  return b;
}

/// the part of exchange() that one warp does: v, and whether a poll ran out, to sres
template <int NV>
__device__ __forceinline__ void exchange_poll(double (&v)[NV], int parts, int first, double *set,
                                              unsigned polls, double *sres)
{
  const int lane = threadIdx.x & 31;
  constexpr int PER = kExCtas / 32; // slots a lane polls
  unsigned long long b[PER][NV];
#pragma unroll
  for(int q = 0; q < PER; q++)
#pragma unroll
    for(int k = 0; k < NV; k++)
      b[q][k] = lane + 32 * q < parts ? kExEmpty : 0ull;
  bool more = true;
  for(unsigned n = 0; n < polls && more; n++)
  {
    more = false;
#pragma unroll
    for(int q = 0; q < PER; q++)
#pragma unroll
      for(int k = 0; k < NV; k++)
        if(b[q][k] == kExEmpty)
        {
          b[q][k] = slot_read(set + (lane + 32 * q) * kExSlot + first + k);
          more |= b[q][k] == kExEmpty;
        }
    more = __any_sync(0xffffffffu, more);
  }
#pragma unroll
  for(int k = 0; k < NV; k++)
  {
    double t[PER];
#pragma unroll
    for(int q = 0; q < PER; q++)
      t[q] = __longlong_as_double((long long)b[q][k]);
#pragma unroll
    for(int o = PER / 2; o > 0; o >>= 1)
#pragma unroll
      for(int q = 0; q < o; q++)
        t[q] += t[q + o];
    v[k] = t[0];
  }
#pragma unroll
  for(int o = 16; o > 0; o >>= 1)
#pragma unroll
    for(int k = 0; k < NV; k++)
      v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  if(lane == 0)
  {
#pragma unroll
    for(int k = 0; k < NV; k++)
      sres[k] = v[k];
    sres[2] = more ? 1.0 : 0.0;
  }
}

/// Replace v by its sum over all threads of all CTAs, values first .. first + NV
/// - 1 of slot set `set`.  `clear` (may be NULL): the set to empty.  With it,
/// a fence follows the CTA's own stores to the slots: whoever sees a later value
/// of this CTA and fences too sees all its stores before this exchange.  False
/// when a slot was still empty after `polls` polls (the same in all threads of
/// the CTA).
template <int NT, int NV>
__device__ __forceinline__ bool exchange(double (&v)[NV], int first, double *set, double *clear,
                                         unsigned polls, double (*sw)[2], double *sres)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int G = gridDim.x, cta = blockIdx.x;
#pragma unroll
  for(int o = 16; o > 0; o >>= 1)
#pragma unroll
    for(int k = 0; k < NV; k++)
      v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  if(lane == 0)
#pragma unroll
    for(int k = 0; k < NV; k++)
      sw[warp][k] = v[k];
  __syncthreads();
  if(warp == 0)
  {
    static_assert(NT / 32 <= 16, "the warps' sums are added by 16 lanes");
#pragma unroll
    for(int k = 0; k < NV; k++)
      v[k] = lane < NT / 32 ? sw[lane][k] : 0.0;
#pragma unroll
    for(int o = 8; o > 0; o >>= 1)
#pragma unroll
      for(int k = 0; k < NV; k++)
        v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if(lane == 0)
#pragma unroll
      for(int k = 0; k < NV; k++)
        slot_put(set + cta * kExSlot + first + k, v[k]);
    if(clear)
    {
      if(lane < 3)
        slot_store(clear + cta * kExSlot + lane, kExEmpty);
      fence_gpu();
    }
    exchange_poll(v, G, first, set, polls, sres);
  }
  __syncthreads();
#pragma unroll
  for(int k = 0; k < NV; k++)
    v[k] = sres[k];
  return sres[2] == 0.0;
}

/// The same when this CTA has parts blockIdx.x + gridDim.x b, b < nb, of `parts`: their
/// warps' sums in sw[b] (exchange_part), the total in v.  `clear` empties the slots of
/// all of them.
template <int NV> __device__ __forceinline__ void exchange_part(double (&v)[NV], double (&sw)[2])
{
#pragma unroll
  for(int o = 16; o > 0; o >>= 1)
#pragma unroll
    for(int k = 0; k < NV; k++)
      v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  if((threadIdx.x & 31) == 0)
#pragma unroll
    for(int k = 0; k < NV; k++)
      sw[k] = v[k];
}
template <int NT, int NV>
__device__ __forceinline__ bool exchange_parts(double (&v)[NV], int nb, int parts, int first,
                                               double *set, double *clear, unsigned polls,
                                               double (*sw)[NT / 32][2], double *sres)
{
  const int lane = threadIdx.x & 31;
  __syncthreads();
  if(threadIdx.x < 32)
  {
    static_assert(NT / 32 <= 16, "the warps' sums are added by 16 lanes");
    for(int b = 0; b < nb; b++)
    {
#pragma unroll
      for(int k = 0; k < NV; k++)
        v[k] = lane < NT / 32 ? sw[b][lane][k] : 0.0;
#pragma unroll
      for(int o = 8; o > 0; o >>= 1)
#pragma unroll
        for(int k = 0; k < NV; k++)
          v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
      const int at = (blockIdx.x + gridDim.x * b) * kExSlot;
      if(lane == 0)
#pragma unroll
        for(int k = 0; k < NV; k++)
          slot_put(set + at + first + k, v[k]);
      if(clear && lane < 3)
        slot_store(clear + at + lane, kExEmpty);
    }
    if(clear)
      fence_gpu();
    exchange_poll(v, parts, first, set, polls, sres);
  }
  __syncthreads();
#pragma unroll
  for(int k = 0; k < NV; k++)
    v[k] = sres[k];
  return sres[2] == 0.0;
}
#endif
} // namespace icb
