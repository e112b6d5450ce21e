// hex8modal.cuh -- the corner-mode form of the Hex8 element product, shared by
// the operator (operator.cu) and the multigrid's coarse-level kernel (mgtail.cu).
//
// The 8 corners of a box element are the vertices of a unit cube, so the
// 8-point Hadamard transform  h_s = sum_a (-1)^(s.o_a) u_a  (s, o_a in {0,1}^3)
// takes a component's corner values to the element's corner modes: the mean,
// the three first differences, the three mixed second differences and the
// xyz twist.  For an isotropic material on a box (every Hex8 element of the
// structured grids) K0 is block-diagonal in that basis: the 24 x 24 matrix
// Kt = H K0 H / 64 (H = H8 (x) I3, DOF s*3+c) has 45 nonzeros in 11 dense
// blocks -- {e_xx, e_yy, e_zz}, the three shear pairs, four blocks of mixed
// second differences and the three twist modes; the rigid translations (s = 0)
// are its null rows.  So  K0 u = H (Kt (H u))  costs two butterflies and 45
// FMAs instead of 576.  The host builds Kt from K0 and checks that every entry
// outside the blocks vanishes (to rounding); an element matrix that fails the
// check runs on the dense kernel (operator.cu).
//
// The marching column shares the butterflies between layers: the x-y half of
// the transform is applied once per node plane (the top plane of element k is
// the bottom plane of element k+1), and the top-face result is carried up in
// x-y mode form, where the next element's bottom-face result is added to it
// before the one inverse x-y butterfly per plane.
#pragma once
#include "icb_internal.hpp"

namespace icb
{
/// local node index of the corner with offsets (a,b) in a plane (meshBox order)
__host__ __device__ constexpr int lnode(int a, int b) { return (a ^ b) + 2 * b; }

constexpr int kModalNnz = 45;
template <typename T> struct KModal
{
  T v[kModalNnz]; ///< Kt entries, block by block, row-major within a block
};
/// the 11 blocks of Kt (modal DOF s*3+c), listed by their modal DOFs
struct ModalBlocks
{
  int n[11];
  int dof[11][3];
};
__host__ __device__ constexpr ModalBlocks modal_blocks()
{
  return ModalBlocks{{3, 2, 2, 2, 2, 2, 3, 2, 1, 1, 1},
                     {{3, 7, 14},
                      {4, 6, 0},
                      {5, 12, 0},
                      {8, 13, 0},
                      {9, 20, 0},
                      {10, 17, 0},
                      {11, 16, 18},
                      {15, 19, 0},
                      {21, 0, 0},
                      {22, 0, 0},
                      {23, 0, 0}}};
}

/// yh = Kt uh, block B onwards (OFF: offset of block B in K.v); every index
/// is a compile-time constant, so uh and yh stay in registers
template <int B, int OFF, typename T>
__device__ __forceinline__ void modal_blocks_apply(const KModal<T> &K, const T (&uh)[24],
                                                   T (&yh)[24])
{
  if constexpr(B < 11)
  {
    constexpr ModalBlocks MB = modal_blocks();
    constexpr int n = MB.n[B];
    constexpr int a = MB.dof[B][0], b = MB.dof[B][1], c = MB.dof[B][2];
    if constexpr(n == 1)
      yh[a] = K.v[OFF] * uh[a];
    else if constexpr(n == 2)
    {
      yh[a] = fma(K.v[OFF + 1], uh[b], K.v[OFF] * uh[a]);
      yh[b] = fma(K.v[OFF + 3], uh[b], K.v[OFF + 2] * uh[a]);
    }
    else
    {
      yh[a] = fma(K.v[OFF + 2], uh[c], fma(K.v[OFF + 1], uh[b], K.v[OFF] * uh[a]));
      yh[b] = fma(K.v[OFF + 5], uh[c], fma(K.v[OFF + 4], uh[b], K.v[OFF + 3] * uh[a]));
      yh[c] = fma(K.v[OFF + 8], uh[c], fma(K.v[OFF + 7], uh[b], K.v[OFF + 6] * uh[a]));
    }
    modal_blocks_apply<B + 1, OFF + n * n>(K, uh, yh);
  }
}

/// x-y half of the transform on one plane, corners in lnode order
/// (q0 (0,0), q1 (1,0), q2 (1,1), q3 (0,1)) -> modes h[sx + 2 sy]
template <typename T> __device__ __forceinline__ void plane_modes(const T u[4], T h[4])
{
  const T a = u[0] + u[1], b = u[0] - u[1], c = u[3] + u[2], e = u[3] - u[2];
  h[0] = a + c;
  h[1] = b + e;
  h[2] = a - c;
  h[3] = b - e;
}
/// its inverse up to a factor 4 (the factors of both butterflies, 64 in all,
/// are folded into Kt): modes -> corners
template <typename T> __device__ __forceinline__ void plane_corners(const T h[4], T u[4])
{
  const T p = h[0] + h[2], m = h[0] - h[2], r = h[1] + h[3], n = h[1] - h[3];
  u[0] = p + r;
  u[1] = p - r;
  u[2] = m - n;
  u[3] = m + n;
}

/// Kt of K0 (operator.cu), cached per host thread; false when K0 has entries
/// outside the blocks above rounding (such a matrix runs on the dense kernel)
template <typename T> bool modal_form_cached(const T *K, KModal<T> &m);
} // namespace icb
