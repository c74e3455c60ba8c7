// Plain FP64 grouped block GEMM: the drop-in numerical path.
//
// Replaces the per-pair dgemm/zgemm of contractDATA_group (Source/
// QSpace_aux.cc:27-355 -> wbarray::contract Source/wbarray.cc:3389-3500 ->
// DZGEMM Source/wbarray_blas.cc:121-213) for the output blocks that the
// tensor-core launch leaves (small or shallow sums) and for the 16x16 cells of
// tiles that launch lists.  One CTA owns one 32x32 tile or one cell of one output block
// and sums all block pairs of that block in plan order, so the result is
// deterministic and needs no atomics.  The K loop stages 32xKC panels of
// op(A) and KCx32 panels of op(B) in shared memory (coalesced loads in either
// storage order), the next panel's loads in flight behind the current one's
// arithmetic; each thread accumulates a 2x2 sub-tile with FP64 FMAs.
//
// GB300's FP64 pipe (about 2 multiply-adds per clock and SM) bounds this
// kernel: a panel step of a full tile keeps it busy for 540 clocks, against
// 512 or 1024 bytes loaded, so a small tile costs no bandwidth.  32x32 tiles
// spread a list of small blocks over four times the SMs of 64x64 ones.
#include <algorithm>

#include "qs_internal.h"

namespace qs {

namespace {
constexpr int THREADS = 256;  // 16 x 16, two rows and two columns each

template <bool CPLX>
struct Elem;
template <>
struct Elem<false> {
  using T = double;
  static constexpr int KC = 16;
  __device__ static T zero() { return 0.0; }
  __device__ static T load(const double *p, int64_t i, bool /*conj*/, double f) { return p[i] * f; }
  __device__ static void fma(T &c, T a, T b) { c = ::fma(a, b, c); }
  __device__ static void store(double *p, int64_t i, T v) { p[i] = v; }
};
template <>
struct Elem<true> {
  using T = double2;
  static constexpr int KC = 8;
  __device__ static T zero() { return make_double2(0.0, 0.0); }
  __device__ static T load(const double *p, int64_t i, bool conj, double f) {
    double2 v = reinterpret_cast<const double2 *>(p)[i];
    return make_double2(v.x * f, (conj ? -v.y : v.y) * f);
  }
  __device__ static void fma(T &c, T a, T b) {
    c.x = ::fma(a.x, b.x, c.x);
    c.x = ::fma(-a.y, b.y, c.x);
    c.y = ::fma(a.x, b.y, c.y);
    c.y = ::fma(a.y, b.x, c.y);
  }
  __device__ static void store(double *p, int64_t i, T v) { reinterpret_cast<double2 *>(p)[i] = v; }
};

// One staged K panel into the accumulators, for the NI x NJ leading 16 x 16
// groups of the tile and the first kn of its KC steps (CTA-uniform bounds):
// padding would cost the FP64 pipe as much as real work.
template <class E, int NI, int NJ, class P, class Acc>
__device__ __forceinline__ void panel_fma(Acc &acc, const P &sm, int tx, int ty, int kn) {
  using T = typename E::T;
  constexpr int KC = P::KC;
#pragma unroll
  for (int kk = 0; kk < KC; ++kk) {
    if (kk < kn) {
      T a[NI], b[NJ];
#pragma unroll
      for (int i = 0; i < NI; ++i) a[i] = sm.a[kk][tx + 16 * i];
#pragma unroll
      for (int j = 0; j < NJ; ++j) b[j] = sm.b[kk][ty + 16 * j];
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) E::fma(acc[i][j], a[i], b[j]);
    }
  }
}

// Panels of a TS x TS tile: a cell's are twice as deep as a tile's, the same
// loads for every thread and half the barriers a step.
template <class E, int TS>
struct Panels {
  static constexpr int KC = E::KC * (F64_TILE / TS);
  typename E::T a[KC][TS + 1], b[KC][TS + 1];
};

template <bool CPLX, int TS>
__device__ __forceinline__ void tile_product(const TileDesc &t, const PairDesc *__restrict__ pairs,
                                             const double *__restrict__ A, const double *__restrict__ B,
                                             double *__restrict__ C, Panels<Elem<CPLX>, TS> &sm) {
  using E = Elem<CPLX>;
  using T = typename E::T;
  constexpr int KC = Panels<E, TS>::KC, TM = TS, TN = TS, G = TS / 16;
  constexpr int NL = TM * KC / THREADS;  // elements of each panel per thread
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const bool two_rows = G > 1 && t.M - t.m0 > 16, two_cols = G > 1 && t.N - t.n0 > 16;

  T acc[G][G];
#pragma unroll
  for (int i = 0; i < G; ++i)
#pragma unroll
    for (int j = 0; j < G; ++j) acc[i][j] = E::zero();

  // panel (p, k0) into registers; (mm, kk) / (nn, kk) of element e follow the
  // operand's fast index
  T va[NL], vb[NL];
  bool ta = false, tb = false;
  auto fetch = [&](int p, int k0) {
    const PairDesc pd = pairs[p];
    ta = pd.trans & 1;
    tb = pd.trans & 2;
#pragma unroll
    for (int u = 0; u < NL; ++u) {
      const int e = tid + u * THREADS;
      // op(A)(m,k): stored M x K (m fastest) or K x M (k fastest)
      const int ka = k0 + (ta ? e % KC : e / TM), m = t.m0 + (ta ? e / KC : e % TM);
      va[u] = E::zero();
      if (m < t.M && ka < pd.K)
        va[u] = E::load(A, pd.a_off + (ta ? (int64_t)ka + (int64_t)m * pd.lda : (int64_t)m + (int64_t)ka * pd.lda),
                        pd.trans & 4, pd.afac);
      // op(B)(k,n): stored K x N (k fastest) or N x K (n fastest)
      const int kb = k0 + (tb ? e / TN : e % KC), n = t.n0 + (tb ? e % TN : e / KC);
      vb[u] = E::zero();
      if (n < t.N && kb < pd.K)
        vb[u] = E::load(B, pd.b_off + (tb ? (int64_t)n + (int64_t)kb * pd.ldb : (int64_t)kb + (int64_t)n * pd.ldb),
                        pd.trans & 8, 1.0);
    }
    return pd.K;
  };

  int p = t.p0, k0 = 0, K = 0;
  while (p < t.p1 && (K = pairs[p].K) <= 0) ++p;
  if (p < t.p1) fetch(p, 0);
  while (p < t.p1) {
#pragma unroll
    for (int u = 0; u < NL; ++u) {
      const int e = tid + u * THREADS;
      sm.a[ta ? e % KC : e / TM][ta ? e / KC : e % TM] = va[u];
      sm.b[tb ? e / TN : e % KC][tb ? e % TN : e / KC] = vb[u];
    }
    const int kn = min(KC, K - k0);
    // the next panel: of this pair, or of the next one that has depth
    k0 += KC;
    if (k0 >= K) {
      k0 = 0;
      do ++p;
      while (p < t.p1 && (K = pairs[p].K) <= 0);
    }
    __syncthreads();
    if (p < t.p1) fetch(p, k0);
    if (two_rows) {
      if (two_cols) panel_fma<E, G, G>(acc, sm, tx, ty, kn);
      else panel_fma<E, G, 1>(acc, sm, tx, ty, kn);
    } else {
      if (two_cols) panel_fma<E, 1, G>(acc, sm, tx, ty, kn);
      else panel_fma<E, 1, 1>(acc, sm, tx, ty, kn);
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < G; ++j) {
    const int n = t.n0 + ty + 16 * j;
    if (n >= t.N) continue;
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int m = t.m0 + tx + 16 * i;
      if (m < t.M) E::store(C, t.c_off + (int64_t)m + (int64_t)n * t.ldc, acc[i][j]);
    }
  }
}

// CTAs 0 .. ntiles-1 compute the listed tiles.  The others take the tiles that
// the tensor-core launch listed (MissList) one after the other until none is
// left, in list order: about largest first, as that launch's tiles are.  Of a
// tile they compute the 16 x 16 cells that hold missed outputs: one missed
// output costs a quarter of the FP64 time (64 small blocks from a plan, a few
// cells missed: 67 -> 52 us).  Taken in order, tiles of different depths spread
// evenly (300 complex products of log-normal operands, every tile missed: 29.2 ->
// 25.0 ms; dealt out in turn, the last CTAs ran alone).  With none listed these
// CTAs take about 1 us.
template <bool CPLX>
__global__ void __launch_bounds__(THREADS)
gemm_f64_kernel(const PairDesc *__restrict__ pairs, const TileDesc *__restrict__ tiles, int ntiles,
                const TileDesc *__restrict__ checked, int nchecked, MissList miss,
                const double *__restrict__ A, const double *__restrict__ B, double *__restrict__ C) {
  __shared__ union {
    Panels<Elem<CPLX>, F64_TILE> tile;
    Panels<Elem<CPLX>, F64_CELL> cell;
  } sm;
  __shared__ int taken;
  if ((int)blockIdx.x < ntiles) {
    tile_product<CPLX, F64_TILE>(tiles[blockIdx.x], pairs, A, B, C, sm.tile);
    return;
  }
  const int n = miss.head[0];
  while (n > 0) {
    if (threadIdx.x == 0) taken = atomicAdd(miss.head + 1, 1);
    __syncthreads();
    const int k = taken;
    __syncthreads();  // `taken` is rewritten by the next round
    if (k >= n) return;
    const int tile = miss.list[k];
    int lo = 0, hi = nchecked - 1;  // the block: last one whose first tile is <= tile
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (checked[mid].first <= tile) lo = mid;
      else hi = mid - 1;
    }
    TileDesc t = checked[lo];
    const int rows = (t.M + F64_TILE - 1) / F64_TILE, i = tile - t.first;
    t.m0 = (i % rows) * F64_TILE;
    t.n0 = (i / rows) * F64_TILE;
    const bool one_row = t.M - t.m0 <= F64_CELL, one_col = t.N - t.n0 <= F64_CELL;
    const int all = (one_row ? 5 : 15) & (one_col ? 3 : 15), cells = miss.cells(tile);
    if (cells == all) {
      tile_product<CPLX, F64_TILE>(t, pairs, A, B, C, sm.tile);
      continue;
    }
    for (int c = 0; c < 4; ++c) {
      if (!((cells >> c) & 1)) continue;
      TileDesc u = t;
      u.m0 += (c & 1) * F64_CELL;
      u.n0 += (c >> 1) * F64_CELL;
      u.M = min(u.M, u.m0 + F64_CELL);
      u.N = min(u.N, u.n0 + F64_CELL);
      tile_product<CPLX, F64_CELL>(u, pairs, A, B, C, sm.cell);
    }
  }
}
}  // namespace

void launch_gemm_f64(Ctx *ctx, const PairDesc *d_pairs, const TileDesc *d_tiles, int64_t ntiles,
                     const TileDesc *d_checked, int64_t nchecked, const MissList &miss, const double *A,
                     const double *B, double *C, int is_complex) {
  const int64_t takers = nchecked > 0 ? std::min<int64_t>(miss.n, (int64_t)std::max(ctx->num_sms, 1) * 5) : 0;
  if (ntiles + takers <= 0) return;
  if (ntiles + takers > 0x7fffffff) fail(QS_ERR_SHAPE, "gemm_f64: too many tiles");
  if (!takers) {  // else the marks of the tensor-core launch before it stand
    ctx->mark(0);
    ctx->mark(1);
  }
  const unsigned grid = (unsigned)(ntiles + takers);
  if (is_complex)
    gemm_f64_kernel<true><<<grid, THREADS, 0, ctx->stream>>>(d_pairs, d_tiles, (int)ntiles, d_checked, (int)nchecked,
                                                             miss, A, B, C);
  else
    gemm_f64_kernel<false><<<grid, THREADS, 0, ctx->stream>>>(d_pairs, d_tiles, (int)ntiles, d_checked,
                                                              (int)nchecked, miss, A, B, C);
  QS_LAUNCHED(ctx);
  ctx->mark(2);
}

}  // namespace qs
