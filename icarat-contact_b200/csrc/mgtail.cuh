// mgtail.cuh -- the coarse levels of a multigrid V-cycle as one launch
// (mgtail.cu): arguments and launchers.
#pragma once
#include "icb_internal.hpp"

namespace icb
{
/// levels of a tail at most, and smoothing steps it takes
constexpr int kTailLevels = 12, kTailSmooth = 8;
/// shared memory of a tail
constexpr int kTailSmem = 200 << 10;
/// Whether a tail may begin at this level.  A phase on one SM grows with the rounds its
/// warps make, a launch over the whole GPU takes 3.7 to 5 us at any of these sizes.  In
/// 2D a warp takes 32 nodes of a row: two rounds of the FP32 tail's 32 warps pay, three
/// of the FP64 tail's 16.  Microseconds a PCG iteration with the tail beginning at the
/// level and one level below it: FP32, two rounds, 56x26 nodes 68.6 and 70.1, 51x26 82.4
/// and 84.1; three, 46x43 73.7 and 71.1; four, 51x49 80.1 and 75.6, 81x41 86.4 and 78.3;
/// FP64, two rounds, 51x16 71.6 and 74.7; three, 31x41 74.9 and 75.5, 61x21 72.4 and 72.5;
/// four, 34x32 61.9 and 59.1; five, 34x33 79.1 and 74.3.  In 3D a thread takes a node: 343
/// nodes FP32 77.2 and 78.6, FP64 85.2 and 86.1; 468 FP32 78.6 and 79.6; 512 81.8 and
/// 80.2, FP64 equal.
///
/// In a batch (2D) the tails of all designs are one launch, and a level above them costs
/// eight more for the few designs that have one of its size: up to 3400 (FP32) or 1400
/// (FP64) nodes there (8 designs 19.0 ms, with the rule above 20.0; 32 designs equal).
template <typename T> inline bool tail_level(const Dims &d, bool batch)
{
  if(d.dim == 3)
    return d.nnode <= 480;
  return (d.sx + 31LL) / 32 * d.sy <= (sizeof(T) == 4 ? 64 : 48) ||
         (batch && d.nnode <= (sizeof(T) == 4 ? 3400 : 1400));
}

/// the element matrix (2D, 64 entries) or its corner-mode form (3D, 45) of the
/// tail's last smoothed level: a kernel parameter, so that its entries are
/// constant operands of their multiply-adds.  The other levels' matrices are
/// powers of two times it (their elements' edges are doubled), a factor their
/// moduli carry exactly (TailLevel::es).
template <typename T> struct TailK
{
  T v[64];
};
template <typename T> struct TailLevel
{
  int nx, ny, nz, sx, sy, sz;
  int shx, shy, shz; ///< coarsening from the level before (MgPcg's Level::sh)
  T es;
  long long ld;
  const T *E, *dinv;
  int oX, oT, oB, oD, oE; ///< its vectors in shared memory (entries of T)
};
/// levels lv[0] .. lv[nlev - 1] (the last one solved by its dense inverse):
/// out <- V-cycle(b) on lv[0]
template <typename T> struct TailArgs
{
  int dim, nlev, nu, nc;
  int smem, oAcc, oSb; ///< bytes; offsets of the 3D scratch and the dense right-hand side
  T c1[kTailSmooth], c2[kTailSmooth];
  TailLevel<T> lv[kTailLevels];
  const T *b;
  T *out;
  const double *Ainv;
  const int *entry; ///< per coarsest unknown its entry in the padded vectors
  const KState *gate;
};
/// whether coarse levels run as one launch (option mg_tail, default on)
bool mg_tail_enabled();
void set_mg_tail(bool on);
/// entries of TailK
constexpr int tail_k(int dim) { return dim == 2 ? 64 : 45; }
/// lay the levels out in shared memory; false when they do not fit
template <typename T> bool tail_plan(TailArgs<T> &A);
/// entry of component c of node (i, j, k) in a level's padded vectors
template <typename T> int tail_entry(const TailLevel<T> &L, int dim, int c, int i, int j, int k);
/// one V-cycle tail on stream s
template <typename T>
void launch_mg_tail(const TailArgs<T> &A, const TailK<T> &K, cudaStream_t s);
/// n tails of 2D problems (device records of one element matrix) as one launch;
/// smem: the largest of the records
template <typename T>
void launch_mg_tail_batch(const TailArgs<T> *D, int n, int smem, const TailK<T> &K,
                          cudaStream_t s);
} // namespace icb
