// mg_tile.cuh -- one multigrid level's half of a V-cycle in one launch.
//
// Going down, a level does three dependent passes (colour 0 from x = 0, colour
// 1 against it, restriction of the colour-0 residual); coming up, three more
// (coarse correction of colour 0, colour 1, colour 0).  As separate launches
// each costs about 3 us of launch, load latency and tail on the small levels,
// however little work it does.  Here a block owns a tile of columns and runs
// the three passes on its own, re-solving the columns of the neighbouring
// tiles that its own depend on: a pass reaches one column further, so colour 0
// is taken up to two columns (in steps along i or j) outside the tile and
// colour 1 up to one.  The copies agree bit for bit with the owner's, since
// every block forms them from the same values in the same order -- the order
// of the passes in mg.cuh, so the result is theirs bit for bit.
//
// A region column of colour c is a slot q = lj * Wh + li / 2 of the tile's
// (TX + 4) x (TY + 4) region, Wh = (TX + 4) / 2; shared arrays are
// [level][slot], so lanes run along the slots without bank conflicts, and the
// neighbours of a slot in the other colour's array are at q + o - 1, q + o
// (o = (c + lj) & 1) in its row and q -+ Wh in the rows below and above.
// Columns outside the domain, and the levels below the bed and above the
// surface, hold zeros, so the couplings need no case distinctions.
#pragma once
#include "mg.cuh"

namespace nhw {

// Tiles are 4 x 4 columns, so a level's 32 slots fill one warp: the smallest
// tile, with the most blocks, because these launches serve the levels whose
// columns do not fill the GPU.  12 x 4 and larger tiles solve fewer columns
// twice but were no faster there.
struct TileS {
  static constexpr int TX = 4, TY = 4, Wh = (TX + 4) / 2, H = TY + 4, NS = Wh * H;
  static_assert(NS == 32, "a level's slots fill one warp");
};

// Line solve of one column, in place, of more than 20 levels and in the block
// cycle below, where line_solve_regs' code and registers cost more than its
// loads save (256 x 8 x 10 FP32+IR: 11.6 against 12.4 to 24 us a cycle, as a
// call, in one loop or written out).  Levels go through registers four at a
// time, the next four's shared loads issued before the current ones' stores (a
// store to x holds back every later load of it).  x, a, inv, c point at level
// 0; NS elements to the next.
template <int NS, class T>
__device__ __forceinline__ void line_solve_smem(T* __restrict__ x, const T* __restrict__ a, const T* __restrict__ inv,
                                                const T* __restrict__ c, int K) {
  T y = (T)0;
  int k = 0;
  if (K >= 4) {
    T r[4], f[4], d[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) { r[t] = x[t * NS]; f[t] = a[t * NS]; d[t] = inv[t * NS]; }
    for (; k + 8 <= K; k += 4) {
      T rn[4], fn[4], dn[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) { rn[t] = x[(4 + t) * NS]; fn[t] = a[(4 + t) * NS]; dn[t] = inv[(4 + t) * NS]; }
#pragma unroll
      for (int t = 0; t < 4; ++t) { y = (r[t] - f[t] * y) * d[t]; x[t * NS] = y; }
#pragma unroll
      for (int t = 0; t < 4; ++t) { r[t] = rn[t]; f[t] = fn[t]; d[t] = dn[t]; }
      x += 4 * NS;
      a += 4 * NS;
      inv += 4 * NS;
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) { y = (r[t] - f[t] * y) * d[t]; x[t * NS] = y; }
    x += 4 * NS;
    a += 4 * NS;
    inv += 4 * NS;
    k += 4;
  }
  for (; k < K; ++k, x += NS, a += NS, inv += NS) { y = (*x - *a * y) * *inv; *x = y; }
  // x now points at level K, y = x_{K-1}; levels K-2 .. 0
  x -= 2 * NS;
  c += (K - 2) * NS;
  k = K - 2;
  if (k >= 3) {
    T r[4], f[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) { r[t] = x[-t * NS]; f[t] = c[-t * NS]; }
    for (; k >= 7; k -= 4) {
      T rn[4], fn[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) { rn[t] = x[-(4 + t) * NS]; fn[t] = c[-(4 + t) * NS]; }
#pragma unroll
      for (int t = 0; t < 4; ++t) { y = r[t] - f[t] * y; x[-t * NS] = y; }
#pragma unroll
      for (int t = 0; t < 4; ++t) { r[t] = rn[t]; f[t] = fn[t]; }
      x -= 4 * NS;
      c -= 4 * NS;
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) { y = r[t] - f[t] * y; x[-t * NS] = y; }
    x -= 4 * NS;
    c -= 4 * NS;
    k -= 4;
  }
  for (; k >= 0; --k, x -= NS, c -= NS) { y = *x - *c * y; *x = y; }
}

// CH: levels fetched ahead (line_solve_regs); as many as the registers hold
template <class T>
constexpr int kAhead = sizeof(T) == 4 ? 5 : 2;
template <int NS, int CH, class T>
__device__ __forceinline__ void line_solve_tile(T* x, const T* __restrict__ a, const T* __restrict__ inv,
                                                const T* __restrict__ c, int K) {
  auto put = [&](int k, T z) { x[k * NS] = z; };
  if (K <= 10) line_solve_regs<NS, 10, CH>(x, a, inv, c, K, put);
  else if (K <= 20) line_solve_regs<NS, 20, CH>(x, a, inv, c, K, put);
  else line_solve_smem<NS>(x, a, inv, c, K);
}

// The operator of one level at a column of colour c: line factors, cross
// terms and in-level couplings.  Level 0 (kFine) reads the colour-split copy,
// coarse levels the natural layout.
template <class T, bool kFine>
struct TileOp {
  const T *a_, *inv_, *cp_, *x_;   // C13, 1/den, c/den, first cross term at level 0
  T cxx, cyy;
  int sk;
  size_t ss;                       // stride of a cross term
  __device__ __forceinline__ TileOp(const MGL<T>& L, int color, int ii, int jj) {
    if (kFine) {
      const int Mh = (L.M + 1) >> 1, nmh = Mh * L.N;
      const size_t cs = (size_t)nmh * L.K;
      a_ = L.sp + (size_t)color * cs + (Mh * jj + (ii >> 1));
      ss = 2 * cs;
      inv_ = a_ + ss; cp_ = inv_ + ss; x_ = cp_ + ss;
      sk = nmh;
    } else {
      const int c = ii + L.M * jj;
      ss = (size_t)L.n;
      a_ = L.coef + 2 * ss + c; x_ = a_ + ss;
      inv_ = L.linv + c; cp_ = L.lcp + c;
      sk = L.M * L.N;
    }
    cxx = cx_of(L, jj); cyy = cy_of(L, ii);
  }
  __device__ __forceinline__ T inv(int k) const { return inv_[sk * k]; }
  __device__ __forceinline__ T cp(int k) const { return cp_[sk * k]; }
  __device__ __forceinline__ T a(int k) const { return k > 0 ? a_[sk * k] : (T)0; }
  // couplings of level k: east, west, north, south, then the cross terms to
  // the same four columns a level up (minus them a level down)
  __device__ __forceinline__ void couplings(int k, T (&g)[8]) const {
    const T* f = x_ + sk * k;
    g[7] = f[0]; g[5] = f[ss]; g[4] = f[2 * ss]; g[6] = f[3 * ss];
    g[0] = g[1] = cxx;
    g[2] = g[3] = cyy;
  }
};
// Off-column part of A x at a slot from the couplings g and the other
// colour's values: p, u, d its row of slots at this level and a level up and
// down; w, e, s, n the neighbours' offsets.  Summed in the order of
// off_column_c, or column by column as off_column_pc (where a pass of mg.cuh
// corrects the neighbours as it reads them).
template <bool kByColumn, class T>
__device__ __forceinline__ T tile_off(const T (&g)[8], const T* __restrict__ p, const T* __restrict__ u,
                                      const T* __restrict__ d, int w, int e, int s, int n) {
  T v = (T)0;
  if (kByColumn) {
    v += g[0] * p[e]; v += g[4] * u[e]; v -= g[4] * d[e];
    v += g[1] * p[w]; v += g[5] * u[w]; v -= g[5] * d[w];
    v += g[2] * p[n]; v += g[6] * u[n]; v -= g[6] * d[n];
    v += g[3] * p[s]; v += g[7] * u[s]; v -= g[7] * d[s];
  } else {
    v += g[0] * p[e]; v += g[1] * p[w]; v += g[2] * p[n]; v += g[3] * p[s];
    v += g[4] * u[e]; v += g[5] * u[w]; v += g[6] * u[n]; v += g[7] * u[s];
    v -= g[4] * d[e]; v -= g[5] * d[w]; v -= g[6] * d[n]; v -= g[7] * d[s];
  }
  return v;
}

// One column of a thread: its place in the region and in the level, and how
// far outside the tile it is.
template <class G>
struct TileCol {
  int ii, jj, dist, o;
  bool in;
  __device__ __forceinline__ TileCol(int q, int color, int i0, int j0, int M, int N) {
    const int lj = q / G::Wh, pos = q - lj * G::Wh;
    o = (color + lj) & 1;
    const int li = 2 * pos + o;
    ii = i0 - 2 + li;
    jj = j0 - 2 + lj;
    const int dx = max(max(2 - li, li - (G::TX + 1)), 0), dy = max(max(2 - lj, lj - (G::TY + 1)), 0);
    dist = dx + dy;
    in = ii >= 0 && ii < M && jj >= 0 && jj < N;
  }
};

// shared memory of a tile: x of both colours with a zero level at either end,
// and the three line factors of each colour
template <class G, class T>
__host__ __device__ constexpr size_t tile_smem(int K) {
  return sizeof(T) * (size_t)G::NS * (2 * (K + 2) + 6 * K);
}

// Right-hand side forms of level 0: a call gives the value, put() stores it --
// by the block that owns the column.
template <class T>
struct TileB {
  const T* b;
  __device__ __forceinline__ TileB bind(const DevScal*) const { return *this; }
  __device__ __forceinline__ T operator()(int ic) const { return b[ic]; }
  __device__ __forceinline__ void put(int, T) const {}
};
// p = r + beta q, q = p - omega v of the last iteration (k_bicg_xr_sl): p itself
// cannot be both read by the neighbouring tiles and updated in place
template <class T>
struct TileInP {
  T* p;
  const T* r;
  const T* q;
  T beta = (T)0;
  __device__ __forceinline__ TileInP bind(const DevScal* sc) const {
    TileInP u = *this;
    u.beta = (T)sc->beta;
    return u;
  }
  __device__ __forceinline__ T operator()(int ic) const { return r[ic] + beta * q[ic]; }
  __device__ __forceinline__ void put(int ic, T val) const { p[ic] = val; }
};
// s = r - alpha v
template <class T>
struct TileInS {
  T* s;
  const T* r;
  const T* v;
  T alpha = (T)0;
  __device__ __forceinline__ TileInS bind(const DevScal* sc) const {
    TileInS u = *this;
    u.alpha = (T)sc->alpha;
    return u;
  }
  __device__ __forceinline__ T operator()(int ic) const { return r[ic] - alpha * v[ic]; }
  __device__ __forceinline__ void put(int ic, T val) const { s[ic] = val; }
};

// Down: colour 0 from x = 0, colour 1, then b_c = P0^T (b - A x).  The
// residual is zero on colour 1 (its lines are solved exactly against the
// values of colour 0) and minus the off-column part of A x on colour 0.
// Colour 0 of x goes to L.xp for the way up; colour 1 is not needed again.
//
// blockDim = (NS, ceil(K / LPT)); a thread has LPT levels of one slot of each
// colour.  Its loads do not depend on x and are all issued before the first
// use -- and before the test whether the solve has stopped -- so that their
// latency is paid once and not once a pass.  Bound by latency on these levels:
// one load round trip, two line solves' chains, five block barriers (GB300,
// 64 x 8 x 20 FP32: 9.3 us as three launches, 5.1 us; 256 x 8 x 10, with the
// line solves written out, 5.7 -> 4.0; 0.55 us is an empty launch).
template <class T, bool kFine, class G, int LPT, class In>
__global__ void __launch_bounds__(1024) k_mg_down(MGL<T> L, MGL<T> C, int ntile_x, const DevScal* sc, In in) {
  constexpr int NS = G::NS, Wh = G::Wh;
  extern __shared__ unsigned char smem_raw[];
  const int stopped = sc->conv;
  const In inb = in.bind(sc);
  const int K = L.K, M = L.M, N = L.N, MN = M * N;
  T* x0 = reinterpret_cast<T*>(smem_raw);
  T* x1 = x0 + (K + 2) * NS;
  T* l0 = x1 + (K + 2) * NS;
  T* l1 = l0 + 3 * K * NS;
  const int q = threadIdx.x, ty = threadIdx.y, by = blockDim.y;
  const int tj = blockIdx.x / ntile_x, i0 = (blockIdx.x - tj * ntile_x) * G::TX, j0 = tj * G::TY;
  const TileCol<G> c0(q, 0, i0, j0, M, N), c1(q, 1, i0, j0, M, N);
  const bool u0 = c0.in && c0.dist <= 2, u1 = c1.in && c1.dist <= 1, own0 = u0 && c0.dist == 0,
             own1 = u1 && c1.dist == 0;
  const TileOp<T, kFine> A0(L, 0, c0.ii, c0.jj), A1(L, 1, c1.ii, c1.jj);
  const int col0 = c0.ii + M * c0.jj, col1 = c1.ii + M * c1.jj;
  T g[LPT][8], b0[LPT], v0[LPT], a0[LPT], p0[LPT], b1[LPT], v1[LPT], a1[LPT], p1[LPT];
#pragma unroll
  for (int t = 0; t < LPT; ++t) {
    const int k = ty + t * by;
    b0[t] = v0[t] = a0[t] = p0[t] = b1[t] = v1[t] = a1[t] = p1[t] = (T)0;
#pragma unroll
    for (int m = 0; m < 8; ++m) g[t][m] = (T)0;
    if (u0 && k < K) {
      b0[t] = inb(col0 + MN * k);
      v0[t] = A0.inv(k);
      a0[t] = A0.a(k);
      p0[t] = A0.cp(k);
    }
    if (u1 && k < K) {
      b1[t] = inb(col1 + MN * k);
      v1[t] = A1.inv(k);
      a1[t] = A1.a(k);
      p1[t] = A1.cp(k);
      A1.couplings(k, g[t]);
    }
  }
  if (stopped) return;
#pragma unroll
  for (int t = 0; t < LPT; ++t) {
    const int k = ty + t * by;
    if (k < K) {
      x0[(k + 1) * NS + q] = b0[t];
      l0[k * NS + q] = a0[t]; l0[(K + k) * NS + q] = v0[t]; l0[(2 * K + k) * NS + q] = p0[t];
      l1[k * NS + q] = a1[t]; l1[(K + k) * NS + q] = v1[t]; l1[(2 * K + k) * NS + q] = p1[t];
      if (own0) inb.put(col0 + MN * k, b0[t]);
      if (own1) inb.put(col1 + MN * k, b1[t]);
    }
  }
  if (ty == 0) {
    x0[q] = (T)0; x0[(K + 1) * NS + q] = (T)0;
    x1[q] = (T)0; x1[(K + 1) * NS + q] = (T)0;
  }
  __syncthreads();
  if (ty == 0 && u0) line_solve_tile<NS, kAhead<T>>(x0 + NS + q, l0 + q, l0 + K * NS + q, l0 + 2 * K * NS + q, K);
  __syncthreads();
#pragma unroll
  for (int t = 0; t < LPT; ++t) {
    const int k = ty + t * by;
    if (u1 && k < K) {
      const T* x = x0 + (k + 1) * NS + q;
      b1[t] -= tile_off<false>(g[t], x, x + NS, x - NS, c1.o - 1, c1.o, -Wh, Wh);
    }
    if (own0 && k < K) A0.couplings(k, g[t]);
  }
#pragma unroll
  for (int t = 0; t < LPT; ++t) {
    const int k = ty + t * by;
    if (k < K) x1[(k + 1) * NS + q] = b1[t];
    if (own0 && k < K) L.xp[col0 + MN * k] = x0[(k + 1) * NS + q];
  }
  __syncthreads();
  if (ty == 0 && u1) line_solve_tile<NS, kAhead<T>>(x1 + NS + q, l1 + q, l1 + K * NS + q, l1 + 2 * K * NS + q, K);
  __syncthreads();
  // the off-column part at the tile's colour-0 cells, in place of x0, then its
  // sums over the aggregates
#pragma unroll
  for (int t = 0; t < LPT; ++t) {
    const int k = ty + t * by;
    if (own0 && k < K) {
      const T* x = x1 + (k + 1) * NS + q;
      x0[(k + 1) * NS + q] = tile_off<false>(g[t], x, x + NS, x - NS, c0.o - 1, c0.o, -Wh, Wh);
    }
  }
  __syncthreads();
  const int lx = L.rx >> 1, ly = L.ry >> 1;   // log2 of aggregates of 1, 2, 4
  const int ncx = G::TX >> lx, nc = ncx * (G::TY >> ly);
  if (q >= nc) return;
  const int cj = q / ncx, ci = q - cj * ncx;
  const int I = (i0 >> lx) + ci, J = (j0 >> ly) + cj;
  if (I >= C.M || J >= C.N) return;
  const int li0 = 2 + (ci << lx), lj0 = 2 + (cj << ly);
  for (int k = ty; k < K; k += by) {
    T acc = (T)0;
    for (int b = 0; b < L.ry; ++b) {
      const int lj = lj0 + b;
      for (int li = li0 + ((li0 + lj) & 1); li < li0 + L.rx; li += 2)   // colour 0: li + lj even (0 outside the domain)
        acc -= x0[(k + 1) * NS + lj * Wh + (li >> 1)];
    }
    C.b[I + C.M * (J + C.N * k)] = acc;
  }
}

// Up: colour 0 corrected by w P x_c, then colour 1, then colour 0.
template <class T, bool kFine, class G, int LPT>
__global__ void __launch_bounds__(1024) k_mg_up(MGL<T> L, Prolong<T> P, int ntile_x, const DevScal* sc) {
  constexpr int NS = G::NS, Wh = G::Wh;
  extern __shared__ unsigned char smem_raw[];
  const int stopped = sc->conv;
  const int K = L.K, M = L.M, N = L.N, MN = M * N;
  T* x0 = reinterpret_cast<T*>(smem_raw);
  T* x1 = x0 + (K + 2) * NS;
  T* l0 = x1 + (K + 2) * NS;
  T* l1 = l0 + 3 * K * NS;
  const int q = threadIdx.x, ty = threadIdx.y, by = blockDim.y;
  const int tj = blockIdx.x / ntile_x, i0 = (blockIdx.x - tj * ntile_x) * G::TX, j0 = tj * G::TY;
  const TileCol<G> c0(q, 0, i0, j0, M, N), c1(q, 1, i0, j0, M, N);
  const bool u0 = c0.in && c0.dist <= 2, u1 = c1.in && c1.dist <= 1, own0 = u0 && c0.dist == 0,
             own1 = u1 && c1.dist == 0;
  const TileOp<T, kFine> A0(L, 0, c0.ii, c0.jj), A1(L, 1, c1.ii, c1.jj);
  const int col0 = c0.ii + M * c0.jj, col1 = c1.ii + M * c1.jj;
  typename Prolong<T>::Stencil st{};
  if (u0) st = P.stencil(c0.ii, c0.jj);
  T g[LPT][8], x[LPT], b0[LPT], v0[LPT], a0[LPT], p0[LPT], b1[LPT], v1[LPT], a1[LPT], p1[LPT];
#pragma unroll
  for (int t = 0; t < LPT; ++t) {
    const int k = ty + t * by;
    x[t] = b0[t] = v0[t] = a0[t] = p0[t] = b1[t] = v1[t] = a1[t] = p1[t] = (T)0;
#pragma unroll
    for (int m = 0; m < 8; ++m) g[t][m] = (T)0;
    if (u1 && k < K) {
      b1[t] = L.b[col1 + MN * k];
      v1[t] = A1.inv(k);
      a1[t] = A1.a(k);
      p1[t] = A1.cp(k);
      A1.couplings(k, g[t]);
    }
    if (own0 && k < K) {
      v0[t] = A0.inv(k);
      b0[t] = L.b[col0 + MN * k];
      a0[t] = A0.a(k);
      p0[t] = A0.cp(k);
    }
    if (u0 && k < K) x[t] = P.at(L.xp, col0 + MN * k, st, k);
  }
  if (stopped) return;
#pragma unroll
  for (int t = 0; t < LPT; ++t) {
    const int k = ty + t * by;
    if (k < K) {
      x0[(k + 1) * NS + q] = x[t];
      l0[k * NS + q] = a0[t]; l0[(K + k) * NS + q] = v0[t]; l0[(2 * K + k) * NS + q] = p0[t];
      l1[k * NS + q] = a1[t]; l1[(K + k) * NS + q] = v1[t]; l1[(2 * K + k) * NS + q] = p1[t];
    }
  }
  if (ty == 0) {
    x0[q] = (T)0; x0[(K + 1) * NS + q] = (T)0;
    x1[q] = (T)0; x1[(K + 1) * NS + q] = (T)0;
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < LPT; ++t) {
    const int k = ty + t * by;
    if (u1 && k < K) {
      const T* y = x0 + (k + 1) * NS + q;
      b1[t] -= tile_off<true>(g[t], y, y + NS, y - NS, c1.o - 1, c1.o, -Wh, Wh);
    }
    if (own0 && k < K) A0.couplings(k, g[t]);
  }
#pragma unroll
  for (int t = 0; t < LPT; ++t) {
    const int k = ty + t * by;
    if (k < K) x1[(k + 1) * NS + q] = b1[t];
  }
  __syncthreads();
  if (ty == 0 && u1) line_solve_tile<NS, kAhead<T>>(x1 + NS + q, l1 + q, l1 + K * NS + q, l1 + 2 * K * NS + q, K);
  __syncthreads();
#pragma unroll
  for (int t = 0; t < LPT; ++t) {
    const int k = ty + t * by;
    if (own0 && k < K) {
      const T* y = x1 + (k + 1) * NS + q;
      x0[(k + 1) * NS + q] = b0[t] - tile_off<false>(g[t], y, y + NS, y - NS, c0.o - 1, c0.o, -Wh, Wh);
    }
    if (own1 && k < K) L.x[col1 + MN * k] = x1[(k + 1) * NS + q];
  }
  __syncthreads();
  if (ty == 0 && own0) line_solve_tile<NS, kAhead<T>>(x0 + NS + q, l0 + q, l0 + K * NS + q, l0 + 2 * K * NS + q, K);
  __syncthreads();
#pragma unroll
  for (int t = 0; t < LPT; ++t) {
    const int k = ty + t * by;
    if (own0 && k < K) L.x[col0 + MN * k] = x0[(k + 1) * NS + q];
  }
}

// The small levels at the end of the hierarchy (up to kCycleSlots slots a
// colour each) as one block's V-cycle: red-black sweeps and full residuals in
// the order of k_mg_cta_cycle, bit for bit its result.  x of the level being
// worked on and the coarse solution stay in shared memory; a level's operator
// is loaded into registers once a visit.  One block of the GPU: bound by its
// load latencies (three visits, one restriction through global memory) and by
// the chains of its nine line solves, 2 x 20 dependent levels each.
// Slots are numbered over the level's own columns, q = jj * Mh + ii / 2.
constexpr int kCycleSlots = 32;
constexpr int kCycleColumns = 2 * kCycleSlots;
template <class T>
__host__ __device__ inline int cycle_slots(const MGL<T>& L) { return ((L.M + 1) >> 1) * L.N; }
// x of both colours, three line factors, the coarse solution
template <class T>
__host__ __device__ constexpr size_t cycle_smem(int K) {
  return sizeof(T) * ((size_t)kCycleSlots * (2 * (K + 2) + 3 * K) + (size_t)kCycleColumns * K);
}

// A thread's cells of one level (LPT of each colour) with their operator.  The
// cells of a colour are dealt to the threads densely, cell = level * slots +
// slot: the coarsest level of 8 slots fills 3 warps of 20 levels, not 20, and
// an FP64 instruction holds the SM's pipe for 16 cycles whatever its lanes do.
template <class T, int LPT>
struct CycleLevel {
  T g[2][LPT][8], b[2][LPT], a[2][LPT], v[2][LPT], p[2][LPT];
  int w[2][LPT], e[2][LPT], s[2][LPT], n[2][LPT], ii[2][LPT], jj[LPT], col[2][LPT], q[LPT], k[LPT], ns;
  bool in[2][LPT];
  __device__ __forceinline__ void load(const MGL<T>& L, int tid, int nt) {
    const int K = L.K, M = L.M, N = L.N, MN = M * N, Mh = (M + 1) >> 1;
    const size_t n0 = (size_t)L.n;
    ns = Mh * N;
#pragma unroll
    for (int t = 0; t < LPT; ++t) {
      const int cell = tid + t * nt;
      k[t] = cell / ns;
      q[t] = cell - k[t] * ns;
      jj[t] = q[t] / Mh;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int o = (c + jj[t]) & 1;
        ii[c][t] = 2 * (q[t] - jj[t] * Mh) + o;
        in[c][t] = k[t] < K && ii[c][t] < M;
        col[c][t] = ii[c][t] + M * jj[t];
        // offsets of the neighbours' slots; 0, with a zero coupling, where there is none
        const bool im = ii[c][t] > 0, ip = ii[c][t] < M - 1, jm = jj[t] > 0, jp = jj[t] < N - 1;
        w[c][t] = in[c][t] && im ? o - 1 : 0;
        e[c][t] = in[c][t] && ip ? o : 0;
        s[c][t] = in[c][t] && jm ? -Mh : 0;
        n[c][t] = in[c][t] && jp ? Mh : 0;
        b[c][t] = a[c][t] = v[c][t] = p[c][t] = (T)0;
#pragma unroll
        for (int m = 0; m < 8; ++m) g[c][t][m] = (T)0;
        if (in[c][t]) {
          const int ic = col[c][t] + MN * k[t];
          const T* cf = L.coef + ic;
          b[c][t] = L.b[ic];
          a[c][t] = k[t] > 0 ? cf[2 * n0] : (T)0;
          v[c][t] = L.linv[ic];
          p[c][t] = L.lcp[ic];
          const T cx = cx_of(L, jj[t]), cy = cy_of(L, ii[c][t]);
          if (ip) { g[c][t][0] = cx; g[c][t][4] = cf[5 * n0]; }
          if (im) { g[c][t][1] = cx; g[c][t][5] = cf[4 * n0]; }
          if (jp) { g[c][t][2] = cy; g[c][t][6] = cf[6 * n0]; }
          if (jm) { g[c][t][3] = cy; g[c][t][7] = cf[3 * n0]; }
        }
      }
    }
  }
};

template <class T, int LPT>
struct CycleBlock {
  static constexpr int NS = kCycleSlots;
  T* x[2];    // [K + 2][NS] of each colour
  T* f;       // line factors of the colour being solved, [3][K][NS]
  T* xc;      // solution of the level below, [K][columns]
  int K, tid, nt;
  // one half-sweep; x of the other colour as it stands, or zero
  template <bool kByColumn>
  __device__ __forceinline__ void sweep(const CycleLevel<T, LPT>& V, const MGL<T>& L, int c, bool zero = false) {
#pragma unroll
    for (int t = 0; t < LPT; ++t)
      if (V.in[c][t]) {
        const int r = V.k[t] * NS + V.q[t];
        const T* y = x[1 - c] + r + NS;
        T off = (T)0;
        if (!zero) off = tile_off<kByColumn>(V.g[c][t], y, y + NS, y - NS, V.w[c][t], V.e[c][t], V.s[c][t], V.n[c][t]);
        x[c][r + NS] = V.b[c][t] - off;
        f[r] = V.a[c][t]; f[K * NS + r] = V.v[c][t]; f[2 * K * NS + r] = V.p[c][t];
      }
    __syncthreads();
    if (tid < V.ns) {   // a slot without a column (an odd row's end) solves zeros
      const int Mh = (L.M + 1) >> 1, jj = tid / Mh;
      if (2 * (tid - jj * Mh) + ((c + jj) & 1) < L.M)
        line_solve_smem<NS>(x[c] + NS + tid, f + tid, f + K * NS + tid, f + 2 * K * NS + tid, K);
    }
    __syncthreads();
  }
  // x = 0 at the slots of both colours
  __device__ __forceinline__ void clear() {
    for (int r = tid; r < (K + 2) * NS; r += nt) x[0][r] = x[1][r] = (T)0;
  }
  // x of the level, in the natural layout
  __device__ __forceinline__ void store(const CycleLevel<T, LPT>& V, T* out, int MN) const {
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int t = 0; t < LPT; ++t)
        if (V.in[c][t]) out[V.col[c][t] + MN * V.k[t]] = x[c][(V.k[t] + 1) * NS + V.q[t]];
  }
};

template <class T, int LPT>
__global__ void __launch_bounds__(640, 1) k_mg_cycle(MGSet<T> set, int nl, const DevScal* sc, T w, int coarse_sweeps) {
  constexpr int NS = kCycleSlots;
  extern __shared__ unsigned char smem_raw[];
  const int stopped = sc->conv;
  CycleBlock<T, LPT> B;
  const int K = B.K = set.L[0].K;
  const int tid = B.tid = threadIdx.x, nt = B.nt = blockDim.x;
  B.x[0] = reinterpret_cast<T*>(smem_raw);
  B.x[1] = B.x[0] + (K + 2) * NS;
  B.f = B.x[1] + (K + 2) * NS;
  B.xc = B.f + 3 * K * NS;
  CycleLevel<T, LPT> V;
  V.load(set.L[0], tid, nt);
  if (stopped) return;
  for (int l = 0; l < nl - 1; ++l) {
    const MGL<T>& F = set.L[l];
    if (l > 0) V.load(F, tid, nt);
    B.clear();
    __syncthreads();
    B.template sweep<false>(V, F, 0, true);
    B.template sweep<false>(V, F, 1);
    B.store(V, F.x, F.M * F.N);
    __syncthreads();
    cta_restrict(F, set.L[l + 1]);
  }
  if (nl > 1) V.load(set.L[nl - 1], tid, nt);
  B.clear();
  __syncthreads();
  for (int s = 0; s < coarse_sweeps; ++s) {
    B.template sweep<false>(V, set.L[nl - 1], 0, s == 0);
    B.template sweep<false>(V, set.L[nl - 1], 1);
  }
  for (int l = nl - 2;; --l) {
    // level l + 1 is done: its x to the level above, or out
    B.store(V, l < 0 ? set.L[0].x : B.xc, set.L[l + 1].M * set.L[l + 1].N);
    if (l < 0) break;
    const MGL<T>& F = set.L[l];
    V.load(F, tid, nt);
    __syncthreads();
    B.clear();
    __syncthreads();
    Prolong<T> P = prolong_from(F, set.L[l + 1], w);
    P.xc = B.xc;
#pragma unroll
    for (int t = 0; t < LPT; ++t)
      if (V.in[0][t])
        B.x[0][(V.k[t] + 1) * NS + V.q[t]] =
            P.at(F.x, V.col[0][t] + F.M * F.N * V.k[t], P.stencil(V.ii[0][t], V.jj[t]), V.k[t]);
    __syncthreads();
    B.template sweep<true>(V, F, 1);
    B.template sweep<false>(V, F, 0);
  }
}

}  // namespace nhw
