// conetile.cuh -- the cone filter's stencil on shared-memory tiles: the 3D filter
// and the volume of the 2D OC update (opt.cu).
//
// The stencil {|offset * h| <= r} is a set of columns along the last axis (z; y in
// 2D): column (di, dj) holds the offsets |dk| <= hk(di, dj)
// with weights that depend on |di|, |dj| and |dk| only.  A thread sums R
// consecutive outputs of one column of elements: per group of columns
// (+-di, +-dj) it reads R + 2 hk tile values of each, adds the group's values
// at one z first and spends R (2 hk + 1) multiply-adds on the sums, so a value
// read from shared memory serves every output it contributes to and a weight
// is applied once per group (at r = 3 41 shared reads and 43 FP64
// operations per output instead of 123 of each).
#pragma once
#include "icb_internal.hpp"

namespace icb
{
constexpr int kConeMaxHz = 4;        ///< largest half height of a column (unrolled loops)
constexpr int kConeSmem = 100 << 10; ///< most shared memory of a tile (two CTAs per SM)
constexpr int kConeMaxHalo = 256;     ///< no tile's halo is wider (keeps its size in an int)

/// the stencil as columns, on the device
struct ConeCols
{
  /// (di, dj, hk, first weight), di, dj >= 0, per group of columns; 2D: dj = 0
  const int4 *col = nullptr;
  const double *w = nullptr; ///< per group hk + 1 weights, |dk| = 0 .. hk
  int ncol = 0;
  int hx = 0, hy = 0, hz = 0; ///< halo of the tile; 2D: hy = 0, hz along y
};

/// the tile of a 256-thread block: 32 x 8 x R outputs and its halo
template <int R> struct ConeTile
{
  __host__ __device__ static int wx(const ConeCols &C) { return 32 + 2 * C.hx; }
  __host__ __device__ static int wy(const ConeCols &C) { return 8 + 2 * C.hy; }
  __host__ __device__ static int cells(const ConeCols &C)
  {
    return wx(C) * wy(C) * (R + 2 * C.hz);
  }

  /// put f(element index) at every cell of the tile with corner (x0, y0, z0),
  /// 0 outside the grid (which adds exactly nothing to a sum).  The threads
  /// take the cells in order, 256 apart, their coordinates advanced instead of
  /// divided out, eight cells' loads in flight.
  template <class F>
  static __device__ __forceinline__ void stage(double *tile, const Dims &g, const ConeCols &C,
                                               int x0, int y0, int z0, F f)
  {
    const int W = wx(C), H = wy(C), n = cells(C);
    const int drow = 256 / W, dx = 256 - drow * W, dz = drow / H, dy = drow - dz * H;
    int row = threadIdx.x / W, tx = threadIdx.x - row * W, tz = row / H, ty = row - tz * H;
    constexpr int U = 8;
    for(int q0 = threadIdx.x; q0 < n; q0 += 256 * U)
    {
      double v[U];
#pragma unroll
      for(int m = 0; m < U; m++)
      {
        const int i = x0 - C.hx + tx, j = y0 - C.hy + ty, k = z0 - C.hz + tz;
        const bool in = q0 + 256 * m < n && unsigned(i) < unsigned(g.nx) &&
                        unsigned(j) < unsigned(g.ny) && unsigned(k) < unsigned(g.nz);
        v[m] = in ? f(i + (long long)g.nx * (j + (long long)g.ny * k)) : 0.0;
        tx += dx;
        ty += dy;
        tz += dz;
        if(tx >= W)
        {
          tx -= W;
          ty++;
        }
        if(ty >= H)
        {
          ty -= H;
          tz++;
        }
      }
#pragma unroll
      for(int m = 0; m < U; m++)
        if(q0 + 256 * m < n)
          tile[q0 + 256 * m] = v[m];
    }
  }

  /// add the columns (+-di, +-dj) of half height HK: their values at one z are
  /// added first (PX, PY: di, dj > 0), then weighted
  template <int HK, bool PX, bool PY>
  static __device__ __forceinline__ void column(const double *p, int di, int djW,
                                                const double *__restrict__ w, int zs,
                                                double (&acc)[R])
  {
    double wv[HK + 1];
#pragma unroll
    for(int q = 0; q <= HK; q++)
      wv[q] = __ldg(w + q);
    p -= HK * zs;
    const double *a = p + djW + di, *b = p + djW - di, *c = p - djW + di, *e = p - djW - di;
#pragma unroll
    for(int m = 0; m < R + 2 * HK; m++)
    {
      double v = a[m * zs];
      if(PX)
        v += b[m * zs];
      if(PY)
        v += PX ? c[m * zs] + e[m * zs] : c[m * zs];
#pragma unroll
      for(int r = 0; r < R; r++)
      {
        const int dk = m - HK - r;
        if(dk >= -HK && dk <= HK)
          acc[r] = fma(wv[dk < 0 ? -dk : dk], v, acc[r]);
      }
    }
  }
  template <int HK>
  static __device__ __forceinline__ void columns(const double *p, int di, int djW,
                                                 const double *__restrict__ w, int zs,
                                                 double (&acc)[R])
  {
    if(di && djW)
      column<HK, true, true>(p, di, djW, w, zs, acc);
    else if(di)
      column<HK, true, false>(p, di, djW, w, zs, acc);
    else if(djW)
      column<HK, false, true>(p, di, djW, w, zs, acc);
    else
      column<HK, false, false>(p, di, djW, w, zs, acc);
  }

  /// acc[r] += the stencil's sum around p + r zs in a tile of row width W
  static __device__ __forceinline__ void sum_columns(const double *p, int W, int zs,
                                                     const ConeCols &C, double (&acc)[R])
  {
    for(int c = 0; c < C.ncol; c++)
    {
      const int4 o = __ldg(C.col + c);
      const double *w = C.w + o.w;
      static_assert(kConeMaxHz == 4, "one case per half height");
      switch(o.z)
      {
      case 0: columns<0>(p, o.x, o.y * W, w, zs, acc); break;
      case 1: columns<1>(p, o.x, o.y * W, w, zs, acc); break;
      case 2: columns<2>(p, o.x, o.y * W, w, zs, acc); break;
      case 3: columns<3>(p, o.x, o.y * W, w, zs, acc); break;
      default: columns<4>(p, o.x, o.y * W, w, zs, acc); break;
      }
    }
  }
  /// acc[r] = sum over the stencil at outputs (lane, warp, z0 + r)
  static __device__ __forceinline__ void sums(const double *tile, const ConeCols &C,
                                              double (&acc)[R])
  {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int W = wx(C), zs = W * wy(C);
    const double *t0 = tile + C.hz * zs + (warp + C.hy) * W + lane + C.hx;
#pragma unroll
    for(int r = 0; r < R; r++)
      acc[r] = 0.0;
    sum_columns(t0, W, zs, C, acc);
  }

  /// f(r, element index) for this thread's outputs inside the grid
  template <class F>
  static __device__ __forceinline__ void outputs(const Dims &g, int x0, int y0, int z0, F f)
  {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = x0 + lane, j = y0 + warp;
    if(i >= g.nx || j >= g.ny)
      return;
#pragma unroll
    for(int r = 0; r < R; r++)
      if(z0 + r < g.nz)
        f(r, i + (long long)g.nx * (j + (long long)g.ny * (z0 + r)));
  }
};
} // namespace icb
