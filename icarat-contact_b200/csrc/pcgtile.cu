// pcgtile.cu -- the Jacobi-PCG of a small problem as one cooperative kernel.
//
// Three kernels an iteration are bound by their launches when the vectors fit
// on the chip: 14.8 us an iteration at 10k unknowns, 17.7 us at 81k.  Here every
// CTA owns a box of nodes for the whole solve, with its part of x, r and D^-1,
// the search direction on the box and a ring around it, and the moduli in shared
// memory.  An iteration is two exchanges between the CTAs:
//   q = K p on the box;                           exchange p.q
//   r -= alpha q, z = D^-1 r published;           exchange r.r, r.z
//   x += alpha p, p = z + beta p on the box and, from the neighbours' z, on
//   the ring
// An exchange is one store of the CTA's sum and one warp's poll of everybody's:
// the slots hold a pattern that no sum takes until they are written, so the
// value is its own flag, and each CTA adds the same values in the same order.
// The published z are their own flags too, so nobody waits for a fence: what
// orders the emptying of slots and of z against their next use is one fence an
// iteration, taken while the second exchange's sums are on their way (see the
// kernel).  What is left of an iteration is two round trips through L2, four
// chains of FP64 additions and the element work.  An iteration, three kernels
// against one: 120 x 40 (9,920 unknowns) 14.9 and 4.7 us, 60 x 20 x 20 (79,380) 17.9
// and 7.7, 540 x 540 (585,360) 33.0 and 10.1, 48 x 46 x 45 (318,000) 26.5 and 16.4.
//
// The 3D Helmholtz filter's solves (12 iterations or so) take the same form with a
// scalar a node and its separable stencil: a filter call at R = 2.2, host arrays in
// and out, takes 201 us instead of 363 on 40 x 20 x 20 elements, 518 instead of 699
// on 80 x 40 x 40 and 1,113 instead of 1,301 on 128 x 64 x 64, about the largest grid
// whose vectors fit; an MMA run on 80 x 40 x 40 17.2 -> 15.0 ms.
//
// Solves that run at the same time (host threads, the batch runner's workers, the
// server's slots) share the SMs: each then gives a CTA several boxes of its cut.  A
// box's arithmetic and its place in the sums are the same wherever it runs, so a
// solve's iterates do not depend on what else is in flight.
//
// The launch is cooperative (every CTA is resident), and every wait is bounded (an
// iteration's polls of the ring together): a CTA whose wait runs out marks the
// solve ICB_ERR_TIMEOUT and returns, and so do the others when theirs run out.
// The mark stays, whatever status CTA 0 ends with.
#include "pcgtile.hpp"

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <climits>

#include "hex8modal.cuh"

namespace icb
{
namespace
{
/// threads of a CTA: one a node in 2D; in 3D two, one for the four elements
/// below the node and one for the four above (168 registers a thread: 160 bytes spill)
template <int DIM> constexpr int kThreads = DIM == 3 ? 384 : 256;
template <int DIM> constexpr int kNodeThreads = DIM == 3 ? 192 : 256;
/// of the scalar form: one a node, as many as an exchange takes
constexpr int kScalarThreads = 512;
constexpr int kTileSmem = 200 << 10, kScalarSmem = 226 << 10;
/// boxes of a CTA at most, and their shared memory (their sums take some more).  With
/// more solves in flight than that some wait, which beats more boxes: eight solves on
/// 60x20x20 5.0 us an iteration and solve with up to four, 5.7 with up to eight
constexpr int kTileShare = 4, kShareSmem = 222 << 10;

template <int DIM> struct ElemK;
template <> struct ElemK<2>
{
  double k[64];
  __device__ __forceinline__ double operator()(int r, int c) const { return k[r * 8 + c]; }
};
/// upper triangle (the full 24 x 24 matrix exceeds the constant bank's
/// parameters)
template <> struct ElemK<3>
{
  double k[300];
  __device__ __forceinline__ double operator()(int r, int c) const
  {
    return r <= c ? k[r * 24 - r * (r - 1) / 2 + (c - r)]
                  : k[c * 24 - c * (c - 1) / 2 + (r - c)];
  }
};

/// a CTA's box and the layout of its shared memory
template <int DIM> struct Box
{
  int x0, y0, z0, nx, ny, nz, own; // its nodes
  int W, WH, pad;                  // padded box: row, plane, all
  __device__ __forceinline__ int at(int i, int j, int k) const
  {
    return i + 1 + (j + 1) * W + (DIM == 3 ? (k + 1) * WH : 0);
  }
};

/// q = (K p) at padded entry c0 of the box (2D): its four elements' products
__device__ __forceinline__ void node_product2(const ElemK<2> &K, const double *p, const double *E,
                                              const Box<2> &B, int c0, double (&q)[2])
{
  q[0] = q[1] = 0.0;
#pragma unroll
  for(int e = 0; e < 4; e++)
  {
    // element e: low corner at c0 - (ex, ey); the node is its corner (ex, ey)
    const int ex = e & 1, ey = e >> 1, l = lnode(ex, ey);
    const int base = c0 - ex - ey * B.W;
    const double Ee = E[base];
    double ue[8];
#pragma unroll
    for(int m = 0; m < 4; m++)
#pragma unroll
      for(int c = 0; c < 2; c++)
        ue[lnode(m & 1, m >> 1) * 2 + c] = p[c * B.pad + base + (m & 1) + (m >> 1) * B.W];
#pragma unroll
    for(int c = 0; c < 2; c++)
    {
      double s = 0.0;
#pragma unroll
      for(int j = 0; j < 8; j++)
        s = fma(K(l * 2 + c, j), ue[j], s);
      q[c] = fma(Ee, s, q[c]);
    }
  }
}

/// q = the share of the four elements below (EZ = 1) or above (EZ = 0) the node
/// at padded entry c0 in K p (3D), neighbour by neighbour: a neighbour's values
/// are read once for all elements that hold it.  They are taken relative to the
/// node's own (a rigid translation has no forces): the sums then do not cancel,
/// as in the operator's corner-mode form (without that a 33 x 2 x 2 beam needed
/// 794 iterations instead of 718), and the node's own columns drop out.
template <int EZ>
__device__ __forceinline__ void node_product3(const ElemK<3> &K, const double *p, const double *E,
                                              const Box<3> &B, int c0, double (&q)[3])
{
  double u0[3], s[4][3];
#pragma unroll
  for(int c = 0; c < 3; c++)
  {
    u0[c] = p[c * B.pad + c0];
#pragma unroll
    for(int e = 0; e < 4; e++)
      s[e][c] = 0.0;
  }
#pragma unroll
  for(int mz = 0; mz < 2; mz++)
#pragma unroll
    for(int dy = -1; dy <= 1; dy++)
#pragma unroll
      for(int dx = -1; dx <= 1; dx++)
      {
        const int dz = mz - EZ;
        if(dx == 0 && dy == 0 && dz == 0)
          continue;
        const int at = c0 + dx + dy * B.W + dz * B.WH;
        double u[3];
#pragma unroll
        for(int c = 0; c < 3; c++)
          u[c] = p[c * B.pad + at] - u0[c];
#pragma unroll
        for(int e = 0; e < 4; e++)
        {
          // element e: the node is its corner (ex, ey, EZ), the neighbour (mx, my, mz)
          const int ex = e & 1, ey = e >> 1, mx = dx + ex, my = dy + ey;
          if(mx < 0 || mx > 1 || my < 0 || my > 1)
            continue;
          const int l = lnode(ex, ey) + 4 * EZ, m = lnode(mx, my) + 4 * mz;
#pragma unroll
          for(int c = 0; c < 3; c++)
#pragma unroll
            for(int c2 = 0; c2 < 3; c2++)
              s[e][c] = fma(K(l * 3 + c, m * 3 + c2), u[c2], s[e][c]);
        }
      }
#pragma unroll
  for(int c = 0; c < 3; c++)
  {
    q[c] = 0.0;
#pragma unroll
    for(int e = 0; e < 4; e++)
      q[c] = fma(E[c0 - (e & 1) - (e >> 1) * B.W - EZ * B.WH], s[e][c], q[c]);
  }
}

/// the Helmholtz operator at padded entry c0 of the box: the separable sums of
/// k_helm_apply3 in its order (the same bits).  `at`: an own node's sown entry,
/// whose flags say where the grid ends beside it
constexpr int kAtBits = 16;       ///< of a sown entry: the padded entry
constexpr int kAtLow = 1 << 16;   ///< no node at -1 on axis a: kAtLow << 2 a
constexpr int kAtHigh = 2 << 16;  ///< none at +1: kAtHigh << 2 a
constexpr int kAtFace = 1 << 22;  ///< a neighbour CTA reads the node
__device__ __forceinline__ double node_helm(const HelmTensor &C, const double *p, const Box<3> &B,
                                            int at)
{
  const int c0 = at & ((1 << kAtBits) - 1);
  double md[3], sd[3];
#pragma unroll
  for(int a = 0; a < 3; a++)
  {
    const bool lo = !(at & (kAtLow << 2 * a)), hi = !(at & (kAtHigh << 2 * a));
    md[a] = (lo ? C.a[a].mh : 0.0) + (hi ? C.a[a].mh : 0.0);
    sd[a] = (lo ? C.a[a].sh : 0.0) + (hi ? C.a[a].sh : 0.0);
  }
  const HelmAxis &ax = C.a[0], &ay = C.a[1], &az = C.a[2];
  double G[3], H[3];
#pragma unroll
  for(int k = 0; k < 3; k++)
  {
    double mx[3], sx[3];
#pragma unroll
    for(int r = 0; r < 3; r++)
    {
      const double *q = p + c0 + (r - 1) * B.W + (k - 1) * B.WH;
      const double c = q[0], e = q[-1] + q[1];
      mx[r] = fma(md[0], c, ax.mo * e);
      sx[r] = fma(sd[0], c, ax.so * e);
    }
    G[k] = fma(md[1], mx[1], ay.mo * (mx[0] + mx[2]));
    H[k] = G[k] + C.re2 * (fma(md[1], sx[1], ay.mo * (sx[0] + sx[2])) +
                           fma(sd[1], mx[1], ay.so * (mx[0] + mx[2])));
  }
  return fma(md[2], H[1], az.mo * (H[0] + H[2])) + C.re2 * fma(sd[2], G[1], az.so * (G[0] + G[2]));
}

/// what the kernel is given as its operator and threads: NC = DIM the elastic
/// one, NC = 1 the 3D Helmholtz filter's
template <int DIM, int NC> struct TileOp
{
  using K = ElemK<DIM>;
  static constexpr int NT = kThreads<DIM>, kSmem = kTileSmem;
};
template <> struct TileOp<3, 1>
{
  using K = HelmTensor;
  static constexpr int NT = kScalarThreads, kSmem = kScalarSmem;
};

/// body(k, t, w) for the threads t of box k, in its warp w: the CTA's own threads when
/// it has one box, else a warp at a time, `wbox` of each of the nb boxes
template <bool MANY, int NT, class F>
__device__ __forceinline__ void each_thread(int nb, int wbox, const F &body)
{
  const int tid = threadIdx.x, warp = tid >> 5;
  if(!MANY)
  {
    body(0, tid, warp);
    return;
  }
  for(int t = warp; t < nb * wbox; t += NT / 32)
  {
    const int k = t / wbox, w = t - k * wbox;
    body(k, 32 * w + (tid & 31), w);
  }
}

/// One box a CTA; MANY: the boxes blockIdx.x + gridDim.x k (tile_share).  A box is in
/// shared memory with the direction and the moduli on the padded box, x, r, D^-1 and
/// products of its own nodes and their (padded entry, node); the (entry, node) of all
/// boxes' rings follow as one list.  With many boxes a warp takes 32 of a box's threads
/// at a time: each adds the nodes that thread would add, so the boxes' sums, and with
/// them all iterates, are bitwise those of one box a CTA.
template <int DIM, int NC, bool MANY>
__global__ void __launch_bounds__(TileOp<DIM, NC>::NT)
    k_pcg_tiles(const __grid_constant__ typename TileOp<DIM, NC>::K K, const Dims d, const PcgTiles T,
                const double *__restrict__ E, const double *__restrict__ dinv,
                double *__restrict__ x, double *__restrict__ r, double *p0, double *z, double *slots,
                const unsigned polls, KState *st)
{
  constexpr int NT = TileOp<DIM, NC>::NT, NB = MANY ? kTileShare : 1;
  constexpr bool kElastic = NC == DIM;
  extern __shared__ __align__(16) double pcg_dyn[];
  __shared__ double sw[NB][NT / 32][2], sres[3];
  __shared__ int nring, nown[NB];
  const int cta = blockIdx.x, tid = threadIdx.x, warp = tid >> 5;
  const int G = gridDim.x, boxes = T.px * T.py * T.pz;
  const int nb = MANY ? (boxes - cta + G - 1) / G : 1;
  // every CTA reads the state before any writes it (the last thing a solve does)
  if(st->stop)
    return;
  const double thr = st->thr;
  const int maxit = st->maxit;
  double rz = st->rz, rr = st->rr;
  const int cap = T.bx * T.by * T.bz;
  Box<DIM> B;
  B.W = T.bx + 2;
  B.WH = DIM == 3 ? B.W * (T.by + 2) : 0;
  B.pad = B.W * (T.by + 2) * (DIM == 3 ? T.bz + 2 : 1);
  // of box k: k stride further
  const int stride = MANY ? T.smem / 8 - (B.pad - cap) : 0;
  double *sp = pcg_dyn, *sE = sp + NC * B.pad, *sx = sE + (kElastic ? B.pad : 0),
         *sr = sx + NC * cap, *sd = sr + NC * cap, *sq = sd + NC * cap, *sz = sq + NC * cap;
  int2 *sown = reinterpret_cast<int2 *>(sq + (NC == 3 ? 2 : 1) * NC * cap);
  int2 *sring = MANY ? reinterpret_cast<int2 *>(pcg_dyn + nb * stride) : sown + cap;
  const int wbox = (min(cap, NT) + 31) / 32; // warps of a box with nodes
  if(tid == 0)
    nring = 0;
  if(MANY)
    for(int t = tid; t < NB * (NT / 32) * 2; t += NT)
      (&sw[0][0][0])[t] = 0.0; // the warps of a box without nodes
  __syncthreads();
  for(int k = 0; k < nb; k++)
  {
    const int box = cta + G * k, o = k * stride;
    const int cx = box % T.px, cy = box / T.px % T.py, cz = box / (T.px * T.py);
    B.x0 = cx * T.bx, B.y0 = cy * T.by, B.z0 = cz * T.bz;
    B.nx = min(T.bx, d.sx - B.x0), B.ny = min(T.by, d.sy - B.y0), B.nz = min(T.bz, d.sz - B.z0);
    B.own = B.nx * B.ny * B.nz;
    if(tid == 0)
      nown[k] = B.own;
    // the box and its ring: moduli and direction, 0 outside the grid
    for(int t = tid; t < B.pad; t += NT)
    {
      const int row = t / B.W, i = t - row * B.W - 1;
      const int kz = DIM == 3 ? row / (T.by + 2) - 1 : 0;
      const int j = row - (DIM == 3 ? (kz + 1) * (T.by + 2) : 0) - 1;
      const int gx = B.x0 + i, gy = B.y0 + j, gz = B.z0 + kz;
      [[maybe_unused]] const bool elem = unsigned(gx) < unsigned(d.nx) &&
                                         unsigned(gy) < unsigned(d.ny) &&
                                         (DIM == 2 || unsigned(gz) < unsigned(d.nz));
      if constexpr(kElastic)
        sE[o + t] = elem ? E[gx + (long long)d.nx * (gy + (long long)d.ny * gz)] : 0.0;
      const bool node = unsigned(gx) < unsigned(d.sx) && unsigned(gy) < unsigned(d.sy) &&
                        unsigned(gz) < unsigned(d.sz);
      const int g = gx + d.sx * (gy + d.sy * gz);
#pragma unroll
      for(int c = 0; c < NC; c++)
        sp[o + c * B.pad + t] = node ? __ldcg(p0 + c * d.ld + g) : 0.0;
      if(node && !(unsigned(i) < unsigned(B.nx) && unsigned(j) < unsigned(B.ny) &&
                   unsigned(kz) < unsigned(B.nz)))
        // any order: the entries are independent
        sring[atomicAdd(&nring, 1)] = make_int2(o + t, g);
    }
    for(int n = tid; n < B.own; n += NT)
    {
      const int row = n / B.nx, i = n - row * B.nx, kz = row / B.ny, j = row - kz * B.ny;
      const int g = B.x0 + i + d.sx * (B.y0 + j + d.sy * (B.z0 + kz));
      int at = B.at(i, j, kz);
      if constexpr(!kElastic)
      {
        const int l[3] = {i, j, kz}, lo[3] = {B.x0, B.y0, B.z0}, nn[3] = {B.nx, B.ny, B.nz},
                  last[3] = {d.sx - 1, d.sy - 1, d.sz - 1};
#pragma unroll
        for(int a = 0; a < 3; a++)
        {
          const int ga = lo[a] + l[a];
          at |= ga == 0 ? kAtLow << 2 * a : 0;
          at |= ga == last[a] ? kAtHigh << 2 * a : 0;
          at |= (l[a] == 0 && ga > 0) || (l[a] == nn[a] - 1 && ga < last[a]) ? kAtFace : 0;
        }
      }
      sown[o + n] = make_int2(at, g);
#pragma unroll
      for(int c = 0; c < NC; c++)
      {
        sx[o + c * cap + n] = 0.0;
        sr[o + c * cap + n] = r[c * d.ld + g];
        sd[o + c * cap + n] = dinv[c * d.ld + g];
      }
    }
  }
  __syncthreads();
  // nodes of box k
  auto own = [&](int k) { return MANY ? nown[k] : B.own; };
  // the state of the loop, the same in every thread of every CTA
  int iter = 0, matvecs = 0, status = ICB_OK, conv = 0;
  double alpha = 0.0, beta = 0.0, pq = 0.0;
  for(int it = 0;; it++)
  {
    // slots: three sets in turn; published z: the buffers z and p0 in turn (p0
    // was read by all before the first exchange).  Every CTA has read the last
    // iteration's slots and z before it arrives at this one's first exchange, so
    // both are emptied after that exchange and before the second one's fence.
    // The next value this CTA puts (first exchange of it + 1) is read by all
    // before their own fence (second exchange of it + 1), and only after that
    // fence do they read the emptied z (end of it + 1) or slots (it + 2) again.
    double *set = slots + (it % 3) * kExSlot * boxes;
    double *clear = slots + ((it + 2) % 3) * kExSlot * boxes;
    double *zcur = it & 1 ? p0 : z, *zold = it & 1 ? z : p0;
    // q = K p and p.q on the box (constrained rows of q are 0)
    if constexpr(NC == 3)
    {
      // threads for the elements below the nodes and others for those above
      double q[3];
      auto below = [&](int o, int n) {
        node_product3<1>(K, sp + o, sE + o, B, sown[o + n].x, q);
#pragma unroll
        for(int c = 0; c < 3; c++)
          sq[o + c * cap + n] = q[c];
      };
      auto above = [&](int o, int n) {
        node_product3<0>(K, sp + o, sE + o, B, sown[o + n].x, q);
#pragma unroll
        for(int c = 0; c < 3; c++)
          sz[o + c * cap + n] = q[c];
      };
      constexpr int NN = kNodeThreads<3>;
      if constexpr(MANY)
      {
        const int wn = (cap + 31) / 32;
        for(int t = warp; t < nb * 2 * wn; t += NT / 32)
        {
          const int k = t / (2 * wn), w = t - k * 2 * wn;
          const int n = 32 * (w < wn ? w : w - wn) + (tid & 31);
          if(n < own(k))
          {
            if(w < wn)
              above(k * stride, n);
            else
              below(k * stride, n);
          }
        }
      }
      else if(tid >= NN)
        for(int n = tid - NN; n < B.own; n += NN)
          below(0, n);
      else
        for(int n = tid; n < B.own; n += NN)
          above(0, n);
      __syncthreads();
    }
    double v[1] = {0.0};
    each_thread<MANY, NT>(nb, wbox, [&](int k, int t, int w) {
      const int o = k * stride, nk = own(k);
      if(MANY)
        v[0] = 0.0;
#pragma unroll 1
      for(int n = t; n < nk; n += NT)
      {
        const int at = sown[o + n].x, c0 = kElastic ? at : at & ((1 << kAtBits) - 1);
        double q[NC];
        if constexpr(!kElastic)
          q[0] = node_helm(K, sp + o, B, at);
        else if constexpr(DIM == 2)
          node_product2(K, sp + o, sE + o, B, c0, q);
#pragma unroll
        for(int c = 0; c < NC; c++)
        {
          const int e = o + c * cap + n;
          if constexpr(NC == 3)
            q[c] = sz[e] + sq[e];
          if(sd[e] == 0.0)
            q[c] = 0.0;
          sq[e] = q[c];
          v[0] += sp[o + c * B.pad + c0] * q[c];
        }
      }
      if(MANY)
        exchange_part<1>(v, sw[k][w]);
    });
    bool ok = MANY ? exchange_parts<NT, 1>(v, nb, boxes, 0, set, nullptr, polls, sw, sres)
                   : exchange<NT, 1>(v, 0, set, nullptr, polls, sw[0], sres);
    pq = v[0];
    if(!ok)
    {
      status = ICB_ERR_TIMEOUT;
      break;
    }
    matvecs++;
    alpha = rz / pq;
    if(!(pq > 0.0) || !isfinite(alpha))
    {
      status = ICB_ERR_BREAKDOWN;
      break;
    }
    // r -= alpha q; z = D^-1 r for the neighbours; r.r and r.z
    double w2[2] = {0.0, 0.0};
    each_thread<MANY, NT>(nb, wbox, [&](int k, int t, int w) {
      const int o = k * stride, nk = own(k);
      if(MANY)
        w2[0] = w2[1] = 0.0;
#pragma unroll 1
      for(int n = t; n < nk; n += NT)
      {
        const int2 to = sown[o + n];
#pragma unroll
        for(int c = 0; c < NC; c++)
        {
          const int e = o + c * cap + n;
          const double ri = sr[e] - alpha * sq[e];
          sr[e] = ri;
          const double zi = sd[e] * ri;
          // an elastic box is small: nearly all its nodes are on its faces
          if(kElastic || (to.x & kAtFace))
          {
            slot_put(zcur + c * d.ld + to.y, zi);
            slot_store(zold + c * d.ld + to.y, kExEmpty);
          }
          w2[0] += ri * ri;
          w2[1] += ri * zi;
        }
      }
      if(MANY)
        exchange_part<2>(w2, sw[k][w]);
    });
    ok = MANY ? exchange_parts<NT, 2>(w2, nb, boxes, 1, set, clear, polls, sw, sres)
              : exchange<NT, 2>(w2, 1, set, clear, polls, sw[0], sres);
    if(!ok)
    {
      status = ICB_ERR_TIMEOUT;
      break;
    }
    rr = w2[0];
    if(!isfinite(rr) || !isfinite(w2[1]))
    {
      status = ICB_ERR_NAN;
      break;
    }
    conv = rr < thr;
    if(!conv)
    {
      beta = w2[1] / rz;
      rz = w2[1];
    }
    // x += alpha p; p = z + beta p on the box, then on the ring
    each_thread<MANY, NT>(nb, wbox, [&](int k, int t, int) {
      const int o = k * stride, nk = own(k);
#pragma unroll 1
      for(int n = t; n < nk; n += NT)
      {
        const int at = sown[o + n].x, c0 = kElastic ? at : at & ((1 << kAtBits) - 1);
#pragma unroll
        for(int c = 0; c < NC; c++)
        {
          const int e = o + c * cap + n, a = o + c * B.pad + c0;
          const double pi = sp[a];
          sx[e] += alpha * pi;
          sp[a] = fma(beta, pi, sd[e] * sr[e]);
        }
      }
    });
    if(conv)
      break;
    iter++;
    if(iter >= maxit)
    {
      status = ICB_ERR_MAXITER;
      break;
    }
    bool late = false;
    unsigned left = polls;
    for(int t = tid; t < nring && !late; t += NT)
    {
      const int2 e = sring[t];
      unsigned long long b[NC];
      bool more = true;
#pragma unroll
      for(int c = 0; c < NC; c++)
        b[c] = kExEmpty;
      for(; left > 0 && more; left--)
      {
        more = false;
#pragma unroll
        for(int c = 0; c < NC; c++)
          if(b[c] == kExEmpty)
          {
            b[c] = slot_read(zcur + c * d.ld + e.y);
            more |= b[c] == kExEmpty;
          }
      }
      late = more;
#pragma unroll
      for(int c = 0; c < NC; c++)
        sp[c * B.pad + e.x] = fma(beta, sp[c * B.pad + e.x], __longlong_as_double((long long)b[c]));
    }
    if(__syncthreads_or(late))
    {
      status = ICB_ERR_TIMEOUT;
      break;
    }
  }
  each_thread<MANY, NT>(nb, wbox, [&](int k, int t, int) {
    const int o = k * stride, nk = own(k);
    for(int n = t; n < nk; n += NT)
    {
      const int g = sown[o + n].y;
#pragma unroll
      for(int c = 0; c < NC; c++)
      {
        x[c * d.ld + g] = sx[o + c * cap + n];
        r[c * d.ld + g] = sr[o + c * cap + n];
      }
    }
  });
  if(tid == 0 && status == ICB_ERR_TIMEOUT)
  {
    atomicExch(&st->status, ICB_ERR_TIMEOUT);
    st->stop = 1;
  }
  else if(cta == 0 && tid == 0)
  {
    st->pq = pq;
    st->alpha = alpha;
    st->beta = beta;
    st->rr = rr;
    st->rz = rz;
    st->iter = iter;
    st->matvecs = matvecs;
    st->conv = conv;
    // ICB_OK until now, unless another CTA's wait ran out; one that runs out
    // later stores over this
    atomicCAS(&st->status, ICB_OK, status);
    st->stop = 1;
  }
}
} // namespace

static std::atomic<unsigned> g_exchange_spin{kExPolls};
unsigned exchange_spin_limit() { return g_exchange_spin.load(); }
void set_exchange_spin_limit(unsigned polls) { g_exchange_spin = polls; }

PcgTiles pcg_tiles(const Dims &d)
{
  PcgTiles best;
  long long bestCost = LLONG_MAX;
  // dim 1: a scalar on the nodes of a grid (the Helmholtz filter's; 3D only, and
  // a box takes what shared memory holds)
  const bool scalar = d.dim == 1, solid = scalar ? d.sz > 1 : d.dim == 3;
  if(scalar && !solid)
    return best;
  const int G = num_sms(), nc = d.dim;
  // nodes a CTA takes at most: six (3D) or eight (2D) a thread; its shared memory
  // ends near there, and 3D is still 1.6 times the three kernels' speed
  const long long most = scalar       ? LLONG_MAX
                         : d.dim == 3 ? 6 * kNodeThreads<3>
                                      : 8 * kNodeThreads<2>;
  if(G > kExCtas || d.nnode >= (1LL << 30))
    return best;
  for(int px = 1; px <= std::min(G, d.sx); px++)
    for(int py = 1; px * py <= G && py <= d.sy; py++)
    {
      const int pzMost = solid ? std::min(G / (px * py), d.sz) : 1;
      for(int pz = 1; pz <= pzMost; pz++)
      {
        PcgTiles t;
        t.bx = (d.sx + px - 1) / px, t.by = (d.sy + py - 1) / py, t.bz = (d.sz + pz - 1) / pz;
        // boxes that end up empty are not launched
        t.px = (d.sx + t.bx - 1) / t.bx, t.py = (d.sy + t.by - 1) / t.by;
        t.pz = (d.sz + t.bz - 1) / t.bz;
        const long long own = (long long)t.bx * t.by * t.bz;
        if(own > most)
          continue;
        const long long pad =
            (long long)(t.bx + 2) * (t.by + 2) * (solid ? t.bz + 2 : 1);
        const long long bytes = 8 * (pad * (scalar ? 1 : nc + 1) + (d.dim == 3 ? 5 : 4) * nc * own) + 8 * pad;
        if(bytes > (scalar ? kScalarSmem : kTileSmem))
          continue;
        // cycles of an iteration that depend on the cut: the element work, the
        // ring, and the polls of two exchanges (measured slopes)
        const long long cost = own * (d.dim == 3 ? 20 : scalar ? 3 : 4) + (pad - own) * 3 + t.boxes() * 12;
        if(cost < bestCost)
        {
          bestCost = cost;
          best = t;
          best.smem = int(bytes);
        }
      }
    }
  return best;
}

/// boxes of a CTA when `jobs` solves are on the device: each then takes its part of the
/// SMs.  The cut for one solve fills the chip, so that a second one would wait for it.
/// Microseconds an iteration and solve, with 1, 2, 4 and 8 threads solving: one box a
/// CTA always, this rule, and three kernels an iteration
///   40x15x15   7.2 7.0 6.9 6.9    7.0  5.2  3.4  3.4   16.5  9.4  5.4  3.4
///   60x20x20   7.8 7.6 7.5 7.5    7.8  6.6  5.4  5.0   18.1 11.0  6.3  4.5
///   50x30x30  10.4 10.1 10.0 10.0 10.3  8.8  8.7  8.3  21.9 13.0  8.1  6.8
///   40x40x40  12.5 12.2 12.2 12.2 12.5 10.5 10.5 10.0  24.2 14.7 10.5 10.3
///   300x100    5.8 5.6 5.6 5.6    5.8  5.2  3.8  3.9   16.6  9.0  5.3  3.5
///   120x40     5.0 2.6 1.7 1.7    4.8  2.5  1.8  1.8   15.9  8.4  4.3  2.4
/// Boxes of more than half of kShareSmem (3D grids of more than 70k nodes or so, 2D ones
/// of more than 150k) stay alone on an SM: 48x46x45 16.4 with any number, three kernels
/// 27.3, 17.0, 12.6 and 13.0; 540x540 10.2, three kernels 32.2, 18.8, 15.1, 16.6.
static int tile_share(const PcgTiles &t, int jobs)
{
  const long long m = ((long long)t.boxes() * jobs + num_sms() - 1) / num_sms();
  return int(std::max(1LL, std::min<long long>({m, kTileShare, kShareSmem / t.smem})));
}

template <int DIM, int NC, bool MANY>
static void run_tiles_as(const PcgTiles &t, int share, const Dims &d,
                         typename TileOp<DIM, NC>::K K, const double *E, const double *invdiag,
                         double *x, double *r, double *p, double *z, KState *st, cudaStream_t s)
{
  const size_t nsoa = size_t(NC) * size_t(d.ld);
  // the shared-memory opt-in is a per-device attribute shared by every host
  // thread: always its largest value
  ICB_CUDA(cudaFuncSetAttribute(k_pcg_tiles<DIM, NC, MANY>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                MANY ? kShareSmem : TileOp<DIM, NC>::kSmem));
  double *slots = z + nsoa; // a multiple of 64 doubles past z: line-aligned
  ICB_CUDA(cudaMemsetAsync(z, 0xff, sizeof(double) * (nsoa + pcg_tile_slots(t)), s)); // kExEmpty
  Dims dd = d;
  PcgTiles tt = t;
  unsigned polls = exchange_spin_limit();
  void *args[] = {&K, &dd, &tt, &E, &invdiag, &x, &r, &p, &z, &slots, &polls, &st};
  ICB_CUDA(cudaLaunchCooperativeKernel((const void *)k_pcg_tiles<DIM, NC, MANY>,
                                       dim3(unsigned((t.boxes() + share - 1) / share)),
                                       dim3(TileOp<DIM, NC>::NT), args, size_t(t.smem) * share, s));
  count_launch();
}
template <int DIM, int NC>
static void run_tiles(const PcgTiles &t, const Dims &d, const typename TileOp<DIM, NC>::K &K,
                      const double *E, const double *invdiag, double *x, double *r, double *p,
                      double *z, KState *st, int jobs, cudaStream_t s)
{
  // a filter call is more copies and host time than solve: half of those in flight are
  // on the device at once (80x40x40, 2 threads: 250 us a call, 293 counting all)
  const int share = tile_share(t, NC == DIM ? jobs : jobs / 2);
  (share > 1 ? run_tiles_as<DIM, NC, true> : run_tiles_as<DIM, NC, false>)(
      t, share, d, K, E, invdiag, x, r, p, z, st, s);
}

void launch_pcg_tiles(const PcgTiles &t, const Dims &d, const double *K, const double *E,
                      const double *invdiag, double *x, double *r, double *p, double *z,
                      KState *st, int jobs, cudaStream_t s)
{
  if(d.dim == 2)
  {
    ElemK<2> k;
    std::copy(K, K + 64, k.k);
    run_tiles<2, 2>(t, d, k, E, invdiag, x, r, p, z, st, jobs, s);
  }
  else
  {
    ElemK<3> k;
    for(int i = 0, m = 0; i < 24; i++)
      for(int j = i; j < 24; j++)
        k.k[m++] = K[i * 24 + j];
    run_tiles<3, 3>(t, d, k, E, invdiag, x, r, p, z, st, jobs, s);
  }
}

void launch_pcg_tiles(const PcgTiles &t, const Dims &d, const HelmTensor &C,
                      const double *invdiag, double *x, double *r, double *p, double *z,
                      KState *st, int jobs, cudaStream_t s)
{
  run_tiles<3, 1>(t, d, C, nullptr, invdiag, x, r, p, z, st, jobs, s);
}
} // namespace icb
