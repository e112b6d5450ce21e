// pcgtile.hpp -- the Jacobi-PCG of a small problem as one cooperative kernel
// (pcgtile.cu).
#pragma once
#include "exchange.cuh"

namespace icb
{
/// 1-D assembled mass and stiffness stencils of one axis: off-diagonals h/6
/// and -1/h, diagonal h/3 and 1/h per element beside the node
struct HelmAxis
{
  double mo, mh, so, sh;
};
/// the 3D Helmholtz operator as a tensor product of them (helm.cu)
struct HelmTensor
{
  HelmAxis a[3];
  double re2;
};
/// the grid's nodes cut into px x py x pz boxes of at most bx x by x bz nodes
struct PcgTiles
{
  int px = 0, py = 0, pz = 0, bx = 0, by = 0, bz = 0;
  int smem = 0; ///< bytes of a box
  int boxes() const { return px * py * pz; }
};
/// the cut for a grid (dim 1: a scalar field on it), or boxes() == 0 when the
/// problem is too large for it
PcgTiles pcg_tiles(const Dims &d);
/// doubles of the exchange slots of a cut: three sets
inline int pcg_tile_slots(const PcgTiles &t) { return 3 * kExSlot * t.boxes(); }
/// Iterate from the state k_pcg_init left (r, p, KState) until the solve
/// stops: x, r, and the final KState; p is overwritten.  z: scratch of the
/// vectors' length plus pcg_tile_slots() doubles.  jobs: solves of this form now on
/// the device, this one among them; with several a CTA takes several boxes, so that
/// they run side by side.  The results are bitwise the same for any number.
void launch_pcg_tiles(const PcgTiles &t, const Dims &d, const double *K, const double *E,
                      const double *invdiag, double *x, double *r, double *p, double *z,
                      KState *st, int jobs, cudaStream_t s);
/// the same for the 3D Helmholtz operator (d.dim = 1)
void launch_pcg_tiles(const PcgTiles &t, const Dims &d, const HelmTensor &C,
                      const double *invdiag, double *x, double *r, double *p, double *z,
                      KState *st, int jobs, cudaStream_t s);
} // namespace icb
