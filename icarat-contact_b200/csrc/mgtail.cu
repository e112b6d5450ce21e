// mgtail.cu -- the coarse levels of a multigrid V-cycle as one launch.
//
// Below a few thousand nodes a level's eight kernels (first smoothing step,
// Chebyshev steps, residual, transfers) are bound by their launches: each runs
// 3 to 5 us for well under a microsecond of work.  Here one CTA takes all of
// them with every vector of every level in its shared memory; a phase is its
// arithmetic and one block barrier.  What bounds a phase is the length of a
// thread's instruction stream, so the vectors are padded by a ring of zeros (no
// bounds checks), a warp takes 32 nodes of a row (no index division), a node's
// components lie side by side (one vector load) and the element matrix is a
// kernel parameter (constant operands).
//
// Every node's value is computed by the operations of the kernels this replaces
// in their order -- the Q4 operator's two element columns per node, the Hex8
// corner-mode operator's four, the transfers, the dense product -- so a V-cycle
// is bitwise the one of separate launches.  (Padding adds zeros to sums that
// skip what lies outside the grid, and a constrained entry is one whose inverse
// diagonal is 0: neither changes a bit.)
//
// OC run on 120 x 40 elements (FP64, 10 steps) 25.7 -> 19.2 ms, on 640 x 320 (mixed,
// 5 steps) 16.4 -> 14.7 ms, MMA run on 80 x 40 x 40 21.1 -> 19.2 ms.
//
// A form that spread each level over a cluster of 16 CTAs, the vectors in
// global memory, took 2 us a phase: the store to L2, the barrier's release and
// acquire and the load back cost 1 us alone.
#include "mgtail.cuh"

#include <algorithm>
#include <atomic>

#include "hex8modal.cuh"
#include "reduce.cuh"

namespace icb
{
namespace
{
/// threads of the CTA: as many as 64 (FP32) or 128 (FP64) registers each allow.  (The 3D
/// FP64 form spills 268 bytes a thread at that.)
template <typename T> constexpr int kTailThreads = sizeof(T) == 4 ? 1024 : 512;

template <typename T, int DIM> struct TailVec;
template <> struct TailVec<float, 2>
{
  using V = float2;
};
template <> struct TailVec<double, 2>
{
  using V = double2;
};

/// a level as the CTA works on it.  Node (i, j, k) is entry at(i, j, k) of the
/// padded arrays: W entries a row, H rows a plane; 2D vectors hold a node's two
/// components side by side, 3D ones a plane of entries per component (stride
/// C).  Element (i, j, k) is entry at(i, j, k) of E.
template <typename T> struct TailView
{
  int nx, ny, nz, sx, sy, sz, W, WH, C;
  T *x, *t, *b, *d, *E;
  __device__ __forceinline__ int at(int i, int j, int k) const
  {
    return i + 1 + (j + 1) * W + (k + 1) * WH;
  }
};
template <typename T> __host__ __device__ inline int tail_row(const TailLevel<T> &L)
{
  return L.sx + 2;
}
/// padded rows: one below, two above (a restriction reaches one past the ring)
template <typename T> __host__ __device__ inline int tail_plane(const TailLevel<T> &L)
{
  return (L.sx + 2) * (L.sy + 3);
}
template <typename T> __host__ __device__ inline int tail_cells(const TailLevel<T> &L, int dim)
{
  return tail_plane(L) * (dim == 3 ? L.sz + 3 : 1) + 4;
}
template <typename T, int DIM>
__device__ __forceinline__ TailView<T> tail_view(const TailLevel<T> &L, T *sm)
{
  TailView<T> v;
  v.nx = L.nx, v.ny = L.ny, v.nz = L.nz;
  v.sx = L.sx, v.sy = L.sy, v.sz = L.sz;
  v.W = tail_row(L);
  v.WH = DIM == 3 ? tail_plane(L) : 0;
  v.C = tail_cells(L, DIM);
  v.x = sm + L.oX;
  v.t = sm + L.oT;
  v.b = sm + L.oB;
  v.d = sm + L.oD;
  v.E = sm + L.oE;
  return v;
}
/// f(i, j, k) for the nodes of an sx x sy x sz grid, a warp per 32 of a row
template <typename T, int DIM, class F>
__device__ __forceinline__ void tail_rows(int sx, int sy, int sz, F f)
{
  const int lane = threadIdx.x & 31, nxb = (sx + 31) >> 5;
  const int tasks = nxb * sy * (DIM == 3 ? sz : 1);
  for(int task = int(threadIdx.x >> 5); task < tasks; task += kTailThreads<T> / 32)
  {
    const int row = task / nxb, i = (task - row * nxb) * 32 + lane;
    const int k = DIM == 3 ? row / sy : 0, j = row - k * sy;
    if(i < sx)
      f(i, j, k);
  }
}
/// the same with the values load(i, j, k, v) reads from global memory handed to
/// store(i, j, k, v): four nodes' loads in flight a thread
template <typename T, int DIM, int N, class Ld, class St>
__device__ __forceinline__ void tail_rows_load(int sx, int sy, int sz, Ld load, St store)
{
  constexpr int U = 4, NW = kTailThreads<T> / 32;
  const int lane = threadIdx.x & 31, nxb = (sx + 31) >> 5;
  const int tasks = nxb * sy * (DIM == 3 ? sz : 1);
  for(int task0 = int(threadIdx.x >> 5); task0 < tasks; task0 += U * NW)
  {
    T v[U][N];
    int ii[U], jj[U], kk[U];
#pragma unroll
    for(int u = 0; u < U; u++)
    {
      const int task = task0 + u * NW, row = task / nxb;
      ii[u] = (task - row * nxb) * 32 + lane;
      kk[u] = DIM == 3 ? row / sy : 0;
      jj[u] = row - kk[u] * sy;
      if(task >= tasks || ii[u] >= sx)
        ii[u] = -1;
      else
        load(ii[u], jj[u], kk[u], v[u]);
    }
#pragma unroll
    for(int u = 0; u < U; u++)
      if(ii[u] >= 0)
        store(ii[u], jj[u], kk[u], v[u]);
  }
}
/// entry of component c at node entry p
template <typename T, int DIM>
__device__ __forceinline__ int tail_at(const TailView<T> &L, int c, int p)
{
  return DIM == 2 ? 2 * p + c : c * L.C + p;
}

/// the operator's fused output (OP_RESIDUAL, OP_CHEB of operator.cu)
template <bool CHEB, typename T>
__device__ __forceinline__ T tail_out(T Au, T us, T b, T dinv, T prev, T c1, T c2)
{
  const T r = b - Au;
  if(!CHEB)
    return dinv != T(0) ? r : b; // b is 0 on constrained entries
  T dn = c2 * dinv * r;
  if(c1 != T(0))
    dn += c1 * (us - prev);
  return us + dn;
}

/// one phase: y <- b - K u (CHEB = false) or the Chebyshev step on u with y
/// holding the iterate before it.  acc: scratch of the 3D form (12 values per
/// element column and node plane)
template <bool CHEB, typename T, int DIM>
__device__ __forceinline__ void tail_apply(const TailView<T> &L, const TailK<T> &K, T c1, T c2,
                                           const T *u, T *y, T *acc)
{
  if constexpr(DIM == 2)
  {
    using V = typename TailVec<T, 2>::V;
    const V *uv = reinterpret_cast<const V *>(u);
    V *yv = reinterpret_cast<V *>(y);
    const V *bv = reinterpret_cast<const V *>(L.b), *dv = reinterpret_cast<const V *>(L.d);
    tail_rows<T, 2>(L.sx, L.sy, 1, [&](int i, int j, int) {
      const int p = L.at(i, j, 0), W = L.W;
      V v[3][3];
#pragma unroll
      for(int b = 0; b < 3; b++)
#pragma unroll
        for(int a = 0; a < 3; a++)
          v[b][a] = uv[p + (b - 1) * W + a - 1];
      const T E[2][2] = {{L.E[p - W - 1], L.E[p - W]}, {L.E[p - 1], L.E[p]}};
      const V bb = bv[p], dd = dv[p];
      V pv;
      if(CHEB)
        pv = yv[p];
      T o[2];
#pragma unroll
      for(int c = 0; c < 2; c++)
      {
        T col[2];
#pragma unroll
        for(int a = 0; a < 2; a++) // the left and the right element column
        {
          T s[2];
#pragma unroll
          for(int b = 0; b < 2; b++) // the element below (node on its top), above
          {
            const int row = lnode(1 - a, 1 - b) * 2 + c;
            const T ue[8] = {v[b][a].x,         v[b][a].y,         v[b][a + 1].x,
                             v[b][a + 1].y,     v[b + 1][a + 1].x, v[b + 1][a + 1].y,
                             v[b + 1][a].x,     v[b + 1][a].y};
            s[b] = T(0);
#pragma unroll
            for(int q = 0; q < 8; q++)
              s[b] = fma(K.v[row * 8 + q], ue[q], s[b]);
          }
          const T carry = E[0][a] * s[0];
          col[a] = fma(E[1][a], s[1], carry);
        }
        o[c] = col[0] + col[1];
      }
      V w;
      w.x = tail_out<CHEB>(o[0], v[1][1].x, bb.x, dd.x, pv.x, c1, c2);
      w.y = tail_out<CHEB>(o[1], v[1][1].y, bb.y, dd.y, pv.y, c1, c2);
      yv[p] = w;
    });
  }
  else
  {
    // every element column (ei, ej) at every node plane k once -- the top face
    // of the element below plus the bottom face of the element above -- then
    // every node the sum of its four columns
    const KModal<T> &Km = reinterpret_cast<const KModal<T> &>(K);
    const int ncol = L.nx * L.ny, items = ncol * L.sz;
    for(int it = threadIdx.x; it < items; it += kTailThreads<T>)
    {
      const int k = it / ncol, col = it - k * ncol, ej = col / L.nx, ei = col - ej * L.nx;
      const int p = L.at(ei, ej, k);
      const int qoff[4] = {0, 1, L.W + 1, L.W};
      T h[3][3][4];
#pragma unroll
      for(int z = 0; z < 3; z++)
#pragma unroll
        for(int c = 0; c < 3; c++)
        {
          const T *q = u + c * L.C + p + (z - 1) * L.WH;
          T v[4];
#pragma unroll
          for(int r = 0; r < 4; r++)
            v[r] = q[qoff[r]];
          plane_modes(v, h[z][c]);
        }
      const T E0 = L.E[p - L.WH], E1 = L.E[p];
      T hb[3][4];
#pragma unroll
      for(int e = 0; e < 2; e++)
      {
        T uh[24], yh[24];
#pragma unroll
        for(int s = 0; s < 4; s++)
#pragma unroll
          for(int c = 0; c < 3; c++)
          {
            uh[s * 3 + c] = h[e][c][s] + h[e + 1][c][s];
            uh[(s + 4) * 3 + c] = h[e][c][s] - h[e + 1][c][s];
          }
        yh[0] = yh[1] = yh[2] = T(0);
        modal_blocks_apply<0, 0>(Km, uh, yh);
#pragma unroll
        for(int s = 0; s < 4; s++)
#pragma unroll
          for(int c = 0; c < 3; c++)
            hb[c][s] = e == 0 ? E0 * (yh[s * 3 + c] - yh[(s + 4) * 3 + c])
                              : fma(E1, yh[s * 3 + c] + yh[(s + 4) * 3 + c], hb[c][s]);
      }
#pragma unroll
      for(int c = 0; c < 3; c++)
      {
        T corner[4];
        plane_corners(hb[c], corner);
#pragma unroll
        for(int r = 0; r < 4; r++)
          acc[(c * 4 + r) * items + it] = corner[r];
      }
    }
    __syncthreads();
    const int nn = L.sx * L.sy * L.sz;
    for(int n = threadIdx.x; n < nn; n += kTailThreads<T>)
    {
      const int row = n / L.sx, i = n - row * L.sx, k = row / L.sy, j = row - k * L.sy;
      const int p = L.at(i, j, k);
      const T *a = acc + k * ncol + (j - 1) * L.nx + i - 1;
      const bool x0 = i > 0, x1 = i < L.nx, y0 = j > 0, y1 = j < L.ny;
#pragma unroll
      for(int c = 0; c < 3; c++)
      {
        const T *ac = a + c * 4 * items;
        const T q2 = x0 && y0 ? ac[lnode(1, 1) * items] : T(0);
        const T q3 = x1 && y0 ? ac[lnode(0, 1) * items + 1] : T(0);
        const T q1 = x0 && y1 ? ac[lnode(1, 0) * items + L.nx] : T(0);
        const T q0 = x1 && y1 ? ac[L.nx + 1] : T(0);
        const T o = (q2 + q3) + (q1 + q0);
        const int m = c * L.C + p;
        y[m] = tail_out<CHEB>(o, u[m], L.b[m], L.d[m], CHEB ? y[m] : T(0), c1, c2);
      }
    }
  }
}

/// b_c = R r_f (restrict_b of mg_impl.cuh); CONS: the level below smooths, its
/// constrained entries of b are 0 (the dense solve reads free entries only)
template <typename T, int DIM>
__device__ __forceinline__ void tail_restrict(const TailView<T> &F, const T *r,
                                              const TailLevel<T> &G, const TailView<T> &C,
                                              bool cons)
{
  const T h = T(0.5);
  const int shx = G.shx, shy = G.shy, shz = DIM == 3 ? G.shz : 0;
  tail_rows<T, DIM>(C.sx, C.sy, C.sz, [&](int I, int J, int Kz) {
    const int pc = C.at(I, J, Kz), pf = F.at(I << shx, J << shy, Kz << shz);
#pragma unroll
    for(int c = 0; c < DIM; c++)
    {
      T s = T(0);
      for(int dk = -shz; dk <= shz; dk++)
      {
        T sk = T(0);
        for(int dj = -shy; dj <= shy; dj++)
        {
          const int q = pf + dj * F.W + dk * F.WH;
          const T lo = shx ? r[tail_at<T, DIM>(F, c, q - 1)] : T(0);
          const T hi = shx ? r[tail_at<T, DIM>(F, c, q + 1)] : T(0);
          const T v = r[tail_at<T, DIM>(F, c, q)] + h * (lo + hi);
          sk = dj ? fma(h, v, sk) : sk + v;
        }
        s = dk ? fma(h, sk, s) : s + sk;
      }
      const int m = tail_at<T, DIM>(C, c, pc);
      C.b[m] = cons && C.d[m] == T(0) ? T(0) : s;
    }
  });
}

/// x_f += P x_c (prolong_rows_b of mg_impl.cuh)
template <typename T, int DIM>
__device__ __forceinline__ void tail_prolong(const TailView<T> &F, T *xf, const TailLevel<T> &G,
                                             const TailView<T> &C)
{
  const T h = T(0.5);
  const int shx = G.shx, shy = G.shy, shz = DIM == 3 ? G.shz : 0;
  tail_rows<T, DIM>(F.sx, F.sy, F.sz, [&](int i, int j, int k) {
    const int p = F.at(i, j, k);
    const int I0 = i >> shx, I1 = (i + shx) >> shx, J0 = j >> shy, J1 = (j + shy) >> shy;
    const int K0 = k >> shz, K1 = (k + shz) >> shz;
    const int r00 = C.at(0, J0, K0), r10 = C.at(0, J1, K0);
    const int r01 = C.at(0, J0, K1), r11 = C.at(0, J1, K1);
#pragma unroll
    for(int c = 0; c < DIM; c++)
    {
      const int m = tail_at<T, DIM>(F, c, p);
      auto x = [&](int q) { return C.x[tail_at<T, DIM>(C, c, q)]; };
      const T a = h * (x(r00 + I0) + x(r00 + I1)), b = h * (x(r10 + I0) + x(r10 + I1));
      T a2 = a, b2 = b;
      if(DIM == 3)
      {
        a2 = h * (x(r01 + I0) + x(r01 + I1));
        b2 = h * (x(r11 + I0) + x(r11 + I1));
      }
      if(F.d[m] != T(0))
        xf[m] = xf[m] + h * (h * (a + b) + h * (a2 + b2));
    }
  });
}

/// x_c = A^-1 b_c over the free coarse DOFs (A.entry: their entries in the
/// padded vectors), a warp per row, its lanes' sums in dense_apply_b's order.
/// Four rows' entries are loaded together while they fit five a lane (nc <= 160).
template <typename T>
__device__ __forceinline__ void tail_dense(const TailArgs<T> &A, const TailView<T> &C, double *sb)
{
  constexpr int NW = kTailThreads<T> / 32;
  const int lane = threadIdx.x & 31, warp = int(threadIdx.x >> 5), n = A.nc;
  constexpr int R = 4;
  double a[R][5];
  int row[R];
  auto load = [&](int i0) {
#pragma unroll
    for(int r = 0; r < R; r++)
    {
      row[r] = i0 + r < n ? __ldg(A.entry + i0 + r) : 0;
#pragma unroll
      for(int q = 0; q < 5; q++)
      {
        const int j = lane + 32 * q;
        a[r][q] = i0 + r < n && j < n ? __ldg(A.Ainv + (i0 + r) * n + j) : 0.0;
      }
    }
  };
  if(n <= 160)
    load(warp * R); // ahead of the right-hand side
  for(int j = threadIdx.x; j < n; j += kTailThreads<T>)
    sb[j] = double(C.b[__ldg(A.entry + j)]);
  __syncthreads();
  if(n <= 160)
  {
    for(int i0 = warp * R; i0 < n; i0 += NW * R)
    {
      if(i0 != warp * R)
        load(i0);
#pragma unroll
      for(int r = 0; r < R; r++)
      {
        double s = 0.0;
#pragma unroll
        for(int q = 0; q < 5; q++)
          if(lane + 32 * q < n)
            s += a[r][q] * sb[lane + 32 * q];
        s = warp_sum_d(s);
        if(lane == 0 && i0 + r < n)
          C.x[row[r]] = T(s);
      }
    }
  }
  else
    for(int i = warp; i < n; i += NW)
    {
      double s = 0.0;
      for(int j = lane; j < n; j += 32)
        s += __ldg(A.Ainv + (long long)i * n + j) * sb[j];
      s = warp_sum_d(s);
      if(lane == 0)
        C.x[__ldg(A.entry + i)] = T(s);
    }
}

template <typename T, int DIM>
__device__ __forceinline__ void tail_body(const TailArgs<T> &A, const TailK<T> &K)
{
  if(A.gate && (A.gate->stop || A.gate->conv))
    return;
  extern __shared__ __align__(16) unsigned char tail_dyn[];
  T *sm = reinterpret_cast<T *>(tail_dyn);
  T *acc = reinterpret_cast<T *>(tail_dyn + A.oAcc);
  double *sb = reinterpret_cast<double *>(tail_dyn + A.oSb);
  const int last = A.nlev - 1;
  // the padding and the coarsest x are 0; then the levels' moduli (with their
  // factor) and inverse diagonals, and the right-hand side
  for(int q = threadIdx.x; q < A.oAcc / 16; q += kTailThreads<T>)
    reinterpret_cast<uint4 *>(tail_dyn)[q] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  for(int l = 0; l < last; l++)
  {
    const TailLevel<T> &G = A.lv[l];
    const TailView<T> L = tail_view<T, DIM>(G, sm);
    tail_rows_load<T, DIM, 1 + 2 * DIM>(
        L.sx, L.sy, L.sz,
        [&](int i, int j, int k, T(&v)[1 + 2 * DIM]) {
          const long long n = i + (long long)G.sx * (j + (long long)G.sy * k);
          const bool el = i < L.nx && j < L.ny && (DIM == 2 || k < L.nz);
          v[0] = el ? __ldg(G.E + i + (long long)G.nx * (j + (long long)G.ny * k)) * G.es : T(0);
#pragma unroll
          for(int c = 0; c < DIM; c++)
          {
            v[1 + c] = __ldg(G.dinv + c * G.ld + n);
            v[1 + DIM + c] = l == 0 ? A.b[c * G.ld + n] : T(0);
          }
        },
        [&](int i, int j, int k, const T(&v)[1 + 2 * DIM]) {
          const int p = L.at(i, j, k);
          L.E[p] = v[0];
#pragma unroll
          for(int c = 0; c < DIM; c++)
          {
            L.d[tail_at<T, DIM>(L, c, p)] = v[1 + c];
            if(l == 0)
              L.b[tail_at<T, DIM>(L, c, p)] = v[1 + DIM + c];
          }
        });
  }
  __syncthreads();
  for(int l = 0; l < last; l++)
  {
    const TailView<T> L = tail_view<T, DIM>(A.lv[l], sm);
    if(l)
    {
      const TailView<T> F = tail_view<T, DIM>(A.lv[l - 1], sm);
      tail_restrict<T, DIM>(F, A.nu % 2 ? F.x : F.t, A.lv[l], L, true);
      __syncthreads();
    }
    // the iterates alternate between t and x, from the first step on zero (t);
    // the iterate before it is 0 (x)
    T *cur = L.t, *oth = L.x;
    tail_rows<T, DIM>(L.sx, L.sy, L.sz, [&](int i, int j, int k) {
      const int p = L.at(i, j, k);
#pragma unroll
      for(int c = 0; c < DIM; c++)
      {
        const int m = tail_at<T, DIM>(L, c, p);
        cur[m] = A.c2[0] * L.d[m] * L.b[m];
      }
    });
    __syncthreads();
    for(int s = 1; s < A.nu; s++)
    {
      tail_apply<true, T, DIM>(L, K, A.c1[s], A.c2[s], cur, oth, acc);
      T *w = cur;
      cur = oth;
      oth = w;
      __syncthreads();
    }
    tail_apply<false, T, DIM>(L, K, T(0), T(0), cur, oth, acc);
    __syncthreads();
  }
  const TailView<T> C = tail_view<T, DIM>(A.lv[last], sm);
  {
    const TailView<T> F = tail_view<T, DIM>(A.lv[last - 1], sm);
    tail_restrict<T, DIM>(F, A.nu % 2 ? F.x : F.t, A.lv[last], C, false);
  }
  __syncthreads();
  tail_dense<T>(A, C, sb);
  __syncthreads();
  for(int l = last - 1; l >= 0; l--)
  {
    const TailView<T> L = tail_view<T, DIM>(A.lv[l], sm);
    // nu steps end in t (nu odd) or x, 2 nu in x
    T *cur = A.nu % 2 ? L.t : L.x, *oth = A.nu % 2 ? L.x : L.t;
    tail_prolong<T, DIM>(L, cur, A.lv[l + 1], tail_view<T, DIM>(A.lv[l + 1], sm));
    __syncthreads();
    for(int s = 0; s < A.nu; s++)
    {
      tail_apply<true, T, DIM>(L, K, A.c1[s], A.c2[s], cur, oth, acc);
      T *w = cur;
      cur = oth;
      oth = w;
      __syncthreads();
    }
  }
  const TailLevel<T> &G = A.lv[0];
  const TailView<T> L = tail_view<T, DIM>(G, sm);
  tail_rows<T, DIM>(L.sx, L.sy, L.sz, [&](int i, int j, int k) {
    const int p = L.at(i, j, k);
    const long long n = i + (long long)G.sx * (j + (long long)G.sy * k);
#pragma unroll
    for(int c = 0; c < DIM; c++)
      A.out[c * G.ld + n] = L.x[tail_at<T, DIM>(L, c, p)];
  });
}

template <typename T, int DIM>
__global__ void __launch_bounds__(kTailThreads<T>)
    k_mg_tail(const __grid_constant__ TailArgs<T> A, const __grid_constant__ TailK<T> K)
{
  tail_body<T, DIM>(A, K);
}
template <typename T>
__global__ void __launch_bounds__(kTailThreads<T>)
    k_mg_tail_batch(const TailArgs<T> *__restrict__ D, const __grid_constant__ TailK<T> K)
{
  tail_body<T, 2>(D[blockIdx.x], K);
}

/// the shared-memory opt-in: a per-device function attribute shared by every
/// host thread, always its largest value
template <typename Kern> void tail_optin(Kern kern)
{
  ICB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmem));
}
} // namespace

static std::atomic<bool> g_mg_tail{true};
bool mg_tail_enabled() { return g_mg_tail; }
void set_mg_tail(bool on) { g_mg_tail = on; }

template <typename T> bool tail_plan(TailArgs<T> &A)
{
  const int last = A.nlev - 1;
  long long at = 0, acc = 0;
  auto take = [&](long long n) { // 16-byte aligned
    const long long o = at;
    at += (n * (long long)sizeof(T) + 15) / 16 * 16;
    return int(std::min<long long>(o / (long long)sizeof(T), 1 << 28));
  };
  for(int l = 0; l <= last; l++)
  {
    TailLevel<T> &L = A.lv[l];
    if((long long)L.sx * L.sy * L.sz > (1 << 20))
      return false;
    const long long n = tail_cells(L, A.dim);
    L.oX = take(A.dim * n);
    L.oB = take(A.dim * n);
    L.oT = L.oD = L.oE = 0;
    if(l < last)
    {
      L.oT = take(A.dim * n);
      L.oD = take(A.dim * n);
      L.oE = take(n);
      if(A.dim == 3)
        acc = std::max(acc, 12LL * L.nx * L.ny * L.sz * (long long)sizeof(T));
    }
  }
  A.oAcc = int(std::min<long long>(at, 1 << 28));
  at += (acc + 15) / 16 * 16;
  A.oSb = int(std::min<long long>(at, 1 << 28));
  at += 8LL * A.nc;
  A.smem = int(std::min<long long>(at, 1 << 28));
  return at <= kTailSmem;
}
template <typename T> int tail_entry(const TailLevel<T> &L, int dim, int c, int i, int j, int k)
{
  const int p = i + 1 + (j + 1) * tail_row(L) + (dim == 3 ? (k + 1) * tail_plane(L) : 0);
  return dim == 2 ? 2 * p + c : c * tail_cells(L, 3) + p;
}
template int tail_entry<float>(const TailLevel<float> &, int, int, int, int, int);
template int tail_entry<double>(const TailLevel<double> &, int, int, int, int, int);
template bool tail_plan<float>(TailArgs<float> &);
template bool tail_plan<double>(TailArgs<double> &);

template <typename T>
void launch_mg_tail(const TailArgs<T> &A, const TailK<T> &K, cudaStream_t s)
{
  auto run = [&](auto kern) {
    tail_optin(kern);
    kern<<<1, kTailThreads<T>, A.smem, s>>>(A, K);
  };
  A.dim == 2 ? run(k_mg_tail<T, 2>) : run(k_mg_tail<T, 3>);
  ICB_CUDA(cudaGetLastError());
  count_launch();
}
template void launch_mg_tail<float>(const TailArgs<float> &, const TailK<float> &, cudaStream_t);
template void launch_mg_tail<double>(const TailArgs<double> &, const TailK<double> &, cudaStream_t);

template <typename T>
void launch_mg_tail_batch(const TailArgs<T> *D, int n, int smem, const TailK<T> &K,
                          cudaStream_t s)
{
  tail_optin(k_mg_tail_batch<T>);
  k_mg_tail_batch<T><<<n, kTailThreads<T>, smem, s>>>(D, K);
  ICB_CUDA(cudaGetLastError());
  count_launch();
}
template void launch_mg_tail_batch<float>(const TailArgs<float> *, int, int,
                                          const TailK<float> &, cudaStream_t);
template void launch_mg_tail_batch<double>(const TailArgs<double> *, int, int,
                                           const TailK<double> &, cudaStream_t);
} // namespace icb
