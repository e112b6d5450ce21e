// pcgtile.hpp -- the Jacobi-PCG of a small problem as one cooperative kernel
// (pcgtile.cu).
#pragma once
#include "exchange.cuh"

namespace icb
{
/// the grid's nodes cut into px x py x pz boxes of at most bx x by x bz nodes,
/// one CTA each
struct PcgTiles
{
  int px = 0, py = 0, pz = 0, bx = 0, by = 0, bz = 0;
  int smem = 0; ///< bytes of a CTA
  int ctas() const { return px * py * pz; }
};
/// the cut for a grid, or ctas() == 0 when the problem is too large for it
PcgTiles pcg_tiles(const Dims &d);
/// doubles of the exchange slots of a cut: three sets
inline int pcg_tile_slots(const PcgTiles &t) { return 3 * kExSlot * t.ctas(); }
/// Iterate from the state k_pcg_init left (r, p, KState) until the solve
/// stops: x, r, and the final KState; p is overwritten.  z: scratch of the
/// vectors' length plus pcg_tile_slots() doubles.
void launch_pcg_tiles(const PcgTiles &t, const Dims &d, const double *K, const double *E,
                      const double *invdiag, double *x, double *r, double *p, double *z,
                      KState *st, cudaStream_t s);
} // namespace icb
