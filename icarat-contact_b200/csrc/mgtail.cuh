// mgtail.cuh -- the coarse levels of a multigrid V-cycle as one launch
// (mgtail.cu): arguments and launchers.
#pragma once
#include "icb_internal.hpp"

namespace icb
{
/// levels of a tail at most, and smoothing steps it takes
constexpr int kTailLevels = 12, kTailSmooth = 8;
/// shared memory of a tail, and most nodes of its first level.  A phase of the
/// largest first levels takes about 2.1 us (2D FP64, 1281 nodes), 2.9 us (2D FP32,
/// 3321) or 1.6 us (3D FP32, 396) on its one SM, a launch over the whole GPU 3.7 to
/// 5 us at any of these sizes; the next finer level has four (2D) or eight (3D)
/// times the nodes and would be slower here.
constexpr int kTailSmem = 200 << 10;
template <typename T> constexpr long long tail_nodes(int dim)
{
  return dim == 2 ? (sizeof(T) == 4 ? 3400 : 1400) : 512;
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
/// n tails (device records of one dimension and element matrix) as one launch;
/// smem: the largest of the records
template <typename T>
void launch_mg_tail_batch(const TailArgs<T> *D, int n, int dim, int smem, const TailK<T> &K,
                          cudaStream_t s);
} // namespace icb
