// Deep output blocks of a grouped product: cut along the summed depth into
// parts that run as output blocks of their own, then summed in part order.
//
// The reference computes such a block with one zgemm per pair into the
// output block (Source/QSpace_aux.cc:27-355), each call parallel inside BLAS.
// The grouped kernels here parallelise over output tiles instead, one CTA per
// tile for the block's whole depth; a block with a handful of tiles and a
// sum of millions (the reduced density matrix or the overlap of tensors with
// large bonds) would keep a few SMs busy for the whole launch.  Cutting the
// depth into parts gives every part its own tiles; the parts' sum is formed
// by one kernel in a fixed order, so the result does not depend on how the
// work was scheduled.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "qs_internal.h"

namespace qs {

namespace {

// Depth of a part (elements of K, complex or real) and the parallel work a
// block should reach: output tiles (64 x 32 outputs as the unit of the
// estimate) for the products, and strips of 16 lines (each slicing its lines
// over the whole depth) for the digit preparation of the split path.
constexpr int64_t KPART = 4096;
constexpr int64_t TARGET_TILES = 256;
constexpr int64_t TARGET_STRIPS = 1024;

int64_t parts_of(const std::vector<PairDesc> &pairs, int64_t p0, int64_t p1, int32_t M, int32_t N) {
  int64_t depth = 0;
  for (int64_t p = p0; p < p1; ++p) depth += std::max<int32_t>(pairs[p].K, 0);
  if (depth < 2 * KPART) return 1;
  const int64_t tiles = std::max<int64_t>(1, ((int64_t)M + 63) / 64 * (((int64_t)N + 31) / 32));
  const int64_t strips = std::max<int64_t>(1, ((int64_t)M + N + 7) / 8);
  const int64_t want = std::max(TARGET_TILES / tiles, TARGET_STRIPS / strips);
  return std::max<int64_t>(1, std::min<int64_t>(depth / KPART, want));
}

// Sums the parts of every deep block.  A block of few values and many parts
// (a site density matrix: one element, 256 parts) gives each value a warp, whose
// lanes sum every 32nd part and are then added by a fixed tree: 38 -> 4 us
// against one thread per value; others one thread per value in part order.
__global__ void reduce_parts_kernel(const DeepReduce *__restrict__ red, const double *__restrict__ T,
                                    double *__restrict__ C, int es) {
  const DeepReduce r = red[blockIdx.y];
  const int64_t n = (int64_t)r.M * r.N;
  const bool by_warp = r.nparts >= 16 && n * es <= 8192;
  const int lane = threadIdx.x & 31;
  const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, all = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = by_warp ? first >> 5 : first; e < n * es; e += by_warp ? all >> 5 : all) {
    const int64_t x = e / es, c = e % es;  // element, part of a complex value
    const int64_t i = x % r.M, j = x / r.M;
    const double *t = T + r.t_off * es + e;
    double s = 0.0;
    for (int q = by_warp ? lane : 0; q < r.nparts; q += by_warp ? 32 : 1) s += t[(int64_t)q * n * es];
    if (by_warp) {
#pragma unroll
      for (int w = 16; w > 0; w >>= 1) s += __shfl_down_sync(0xffffffffu, s, w);
    }
    if (!by_warp || lane == 0) C[(r.c_off + i + j * (int64_t)r.ldc) * es + c] = s;
  }
}

// Shallow blocks: C(i, j) = sum over the block's pairs, in order, of
// afac sum_k op(A)(i, k) op(B)(k, j), with at most SHALLOW_K terms in all.  A
// thread owns lines of one side (rows of op(A) with their unit-stride stores;
// columns of op(B) when there are few rows and more columns) and keeps the
// sums of up to NC lines of the other side in registers, so that it loads
// each element of its line once; the other side's terms sit in shared memory.
// The FP64 multiply-adds bound it (2 per clock and SM): a pair's factor scales
// the terms in shared memory, once per CTA (4 blocks of 900 x 900 x 8 with
// factors: 72 us when it scaled each thread's elements, 56 us here).  Applying an MPO tensor
// over a leg of dimension 3 (12 million outputs, up to 3 terms of 3): 190 us
// with one thread per output and a permuted copy, 144 us here (caches cold), 73 us
// of it the FP64 pipe's.
struct ShallowTask {
  int64_t c_off;
  int32_t p0, p1, M, N, ldc;
  int32_t swapped;          // lines are columns of C
  int32_t l0, l1;           // lines of this task
  int32_t o0;               // first line of the other side
  int32_t pad_;
};
constexpr int SHALLOW_THREADS = 128;
constexpr int SHALLOW_NC = 4;  // lines of the other side per CTA
// lines per thread: their loads are in flight together (one line at a time
// leaves the kernel at 2.3 TB/s)
template <bool CPLX>
constexpr int shallow_u() { return CPLX ? 2 : 4; }

// Offset of index l in a view's legs (first leg fastest).
__device__ __forceinline__ int64_t legs_offset(int n, const int32_t *dim, const int64_t *str, int32_t l) {
  int64_t off = 0;
  for (int i = 0; i + 1 < n; ++i) {
    const int32_t q = (int32_t)((uint32_t)l / (uint32_t)dim[i]);
    off += (l - q * dim[i]) * str[i];
    l = q;
  }
  return n > 0 ? off + l * str[n - 1] : off;
}

// Addresses of one operand in the role it plays: line l, depth k.
struct ShallowAddr {
  int64_t off, ls, ks;
  const OperandView *v;
  __device__ __forceinline__ int64_t line(int32_t l) const {
    return off + (v ? legs_offset(v->nl, v->ldim, v->lstr, l) : l * ls);
  }
  __device__ __forceinline__ int64_t depth(int32_t k) const {
    return v ? legs_offset(v->nk, v->kdim, v->kstr, k) : k * ks;
  }
};
__device__ __forceinline__ ShallowAddr shallow_addr(const PairDesc &P, bool b, const OperandView *views, int p) {
  const bool t = P.trans & (b ? 2 : 1);
  const int64_t ld = b ? P.ldb : P.lda;
  // A: line = row, depth = column; B: line = column, depth = row
  const bool unit_line = b == t;
  ShallowAddr a{b ? P.b_off : P.a_off, unit_line ? 1 : ld, unit_line ? ld : 1, nullptr};
  if (views && views[p].nl > 0) a.v = views + p;
  return a;
}

// Output (l, c) of a task with each pair's factor on its sum, f (x y), where
// f y is no normal number: x (f y) overflows, or loses bits that a large x
// brings back.
template <bool CPLX>
__device__ __noinline__ void shallow_scaled_sums(const ShallowTask *tg, const PairDesc *pairs, const OperandView *vx,
                                                 const OperandView *vy, const double *X, const double *Y, double *C,
                                                 int l, int c) {
  const ShallowTask t = *tg;
  double re = 0.0, im = 0.0;
  for (int p = t.p0; p < t.p1; ++p) {
    const PairDesc &P = pairs[p];
    if (P.K <= 0) continue;
    const ShallowAddr ax = shallow_addr(P, t.swapped, vx, p), ay = shallow_addr(P, !t.swapped, vy, p);
    const bool cx = P.trans & (t.swapped ? 8 : 4), cy = P.trans & (t.swapped ? 4 : 8);
    double sr = 0.0, si = 0.0;
    for (int k = 0; k < P.K; ++k) {
      const int64_t i = ax.line(l) + ax.depth(k), j = ay.line(t.o0 + c) + ay.depth(k);
      if (CPLX) {
        const double xr = X[2 * i], xi = cx ? -X[2 * i + 1] : X[2 * i + 1];
        const double yr = Y[2 * j], yi = cy ? -Y[2 * j + 1] : Y[2 * j + 1];
        sr = fma(xr, yr, fma(-xi, yi, sr));
        si = fma(xr, yi, fma(xi, yr, si));
      } else {
        sr = fma(X[i], Y[j], sr);
      }
    }
    re = fma(P.afac, sr, re);
    im = fma(P.afac, si, im);
  }
  const int64_t i = t.swapped ? t.o0 + c : l, j = t.swapped ? l : t.o0 + c;
  const int64_t o = t.c_off + i + j * (int64_t)t.ldc;
  if (CPLX) {
    C[2 * o] = re;
    C[2 * o + 1] = im;
  } else {
    C[o] = re;
  }
}

// The lines of this thread against NC lines of the other side (a count known
// at compile time: predicated multiply-adds would take the FP64 pipe as real
// ones do).
template <bool CPLX, int NC>
__device__ __forceinline__ void shallow_lines(const ShallowTask &t, const PairDesc *__restrict__ pairs,
                                              const OperandView *vx, const double *__restrict__ X, bool wide_x,
                                              const double2 (*yc)[SHALLOW_NC], double *__restrict__ C, bool wide_c) {
  constexpr int U = shallow_u<CPLX>();
  const int lb = t.l0 + threadIdx.x;
  if (lb >= t.l1) return;
  double re[U][NC], im[U][NC];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int c = 0; c < NC; ++c) re[u][c] = im[u][c] = 0.0;
  int term = 0;
  for (int p = t.p0; p < t.p1; ++p) {
    const PairDesc &P = pairs[p];
    const int K = P.K;
    if (K <= 0) continue;
    const ShallowAddr ax = shallow_addr(P, t.swapped, vx, p);
    const bool cx = P.trans & (t.swapped ? 8 : 4);
    int64_t lo[U];
#pragma unroll
    for (int u = 0; u < U; ++u) lo[u] = ax.line(min(lb + u * SHALLOW_THREADS, t.l1 - 1));
    for (int k = 0; k < K; ++k) {
      const int64_t kd = ax.depth(k);
      double xr[U], xi[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = lo[u] + kd;
        xi[u] = 0.0;
        if (CPLX) {
          const double2 x = wide_x ? reinterpret_cast<const double2 *>(X)[i] : make_double2(X[2 * i], X[2 * i + 1]);
          xr[u] = x.x;
          xi[u] = cx ? -x.y : x.y;
        } else {
          xr[u] = X[i];
        }
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const double2 y = yc[term + k][c];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          re[u][c] = fma(xr[u], y.x, re[u][c]);
          if (CPLX) {
            re[u][c] = fma(-xi[u], y.y, re[u][c]);
            im[u][c] = fma(xr[u], y.y, im[u][c]);
            im[u][c] = fma(xi[u], y.x, im[u][c]);
          }
        }
      }
    }
    term += K;
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t l = lb + u * SHALLOW_THREADS;
    if (l >= t.l1) break;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int64_t i = t.swapped ? t.o0 + c : l, j = t.swapped ? l : t.o0 + c;
      const int64_t o = t.c_off + i + j * (int64_t)t.ldc;
      if (!CPLX) {
        C[o] = re[u][c];
      } else if (wide_c) {
        reinterpret_cast<double2 *>(C)[o] = make_double2(re[u][c], im[u][c]);
      } else {
        C[2 * o] = re[u][c];
        C[2 * o + 1] = im[u][c];
      }
    }
  }
}

template <bool CPLX>
__global__ void __launch_bounds__(SHALLOW_THREADS)
shallow_kernel(const ShallowTask *__restrict__ tasks, const PairDesc *__restrict__ pairs,
               const OperandView *__restrict__ va, const OperandView *__restrict__ vb, const double *__restrict__ A,
               const double *__restrict__ B, double *__restrict__ C) {
  constexpr int NC = SHALLOW_NC;
  __shared__ double2 yc[SHALLOW_K][NC];  // the other side, with the factors: term (in pair, k order) x line
  __shared__ int off[NC];                // a scaled entry of the line is no normal number
  if (threadIdx.x < NC) off[threadIdx.x] = 0;
  __syncthreads();
  const ShallowTask t = tasks[blockIdx.x];
  const int other = t.swapped ? t.M : t.N;
  const int nc = min(NC, other - t.o0);
  const OperandView *vx = t.swapped ? vb : va, *vy = t.swapped ? va : vb;
  const double *__restrict__ X = t.swapped ? B : A;
  const double *__restrict__ Y = t.swapped ? A : B;
  // complex buffers may be aligned to 8 bytes only
  const bool wide_x = (reinterpret_cast<uintptr_t>(X) & 15) == 0, wide_c = (reinterpret_cast<uintptr_t>(C) & 15) == 0;
  int term = 0;
  for (int p = t.p0; p < t.p1; ++p) {
    const PairDesc P = pairs[p];
    const int K = max(P.K, 0);
    const ShallowAddr ay = shallow_addr(P, !t.swapped, vy, p);
    const bool cy = P.trans & (t.swapped ? 4 : 8);
    for (int e = threadIdx.x; e < K * NC; e += SHALLOW_THREADS) {
      const int k = e / NC, c = e % NC;
      double2 v = make_double2(0.0, 0.0);
      if (c < nc) {
        const int64_t i = ay.line(t.o0 + c) + ay.depth(k);
        if (CPLX) v = make_double2(Y[2 * i], cy ? -Y[2 * i + 1] : Y[2 * i + 1]);
        else v.x = Y[i];
      }
      auto scale = [&](double y) {
        const double z = y * P.afac;
        const int e = __double2hiint(z) >> 20 & 0x7ff;
        if ((e == 0 || e == 0x7ff) && y != 0.0 && P.afac != 0.0) off[c] = 1;
        return z;
      };
      if (P.afac != 1.0) v = make_double2(scale(v.x), scale(v.y));
      yc[term + k][c] = v;
    }
    term += K;
  }
  __syncthreads();
  switch (nc) {
    case 1: shallow_lines<CPLX, 1>(t, pairs, vx, X, wide_x, yc, C, wide_c); break;
    case 2: shallow_lines<CPLX, 2>(t, pairs, vx, X, wide_x, yc, C, wide_c); break;
    case 3: shallow_lines<CPLX, 3>(t, pairs, vx, X, wide_x, yc, C, wide_c); break;
    default: shallow_lines<CPLX, 4>(t, pairs, vx, X, wide_x, yc, C, wide_c); break;
  }
  for (int c = 0; c < nc; ++c)
    if (off[c])
      for (int l = t.l0 + threadIdx.x; l < t.l1; l += SHALLOW_THREADS)
        shallow_scaled_sums<CPLX>(tasks + blockIdx.x, pairs, vx, vy, X, Y, C, l, c);
}

// One CTA per output element of a small block: every thread sums its share
// of the block's (pair, k) terms in order, then a fixed tree reduces them.
struct DotTask {
  int64_t c_off;
  int32_t p0, p1, M, ldc, i, j;
};
constexpr int DOT_THREADS = 256;
constexpr int DOT_U = 4;
constexpr int DOT_SELF_U = 8;

template <bool CPLX>
__global__ void __launch_bounds__(DOT_THREADS, 4)
dot_kernel(const DotTask *__restrict__ tasks, const PairDesc *__restrict__ pairs, const double *__restrict__ A,
           const double *__restrict__ B, double *__restrict__ C) {
  __shared__ double red[2][DOT_THREADS];
  const DotTask t = tasks[blockIdx.x];
  double re = 0.0, im = 0.0;
  // complex buffers may be aligned to 8 bytes only
  const bool wide = ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) == 0;
  for (int p = t.p0; p < t.p1; ++p) {
    const PairDesc P = pairs[p];
    const bool ta = P.trans & 1, tb = P.trans & 2, ca = P.trans & 4, cb = P.trans & 8;
    const int64_t a0 = P.a_off + (ta ? t.i * (int64_t)P.lda : t.i), as = ta ? 1 : P.lda;
    const int64_t b0 = P.b_off + (tb ? t.j : t.j * (int64_t)P.ldb), bs = tb ? P.ldb : 1;
    // An operand against its own conjugate (a norm, a diagonal entry of a
    // density matrix): two multiply-adds per term and one load instead of four
    // and two; the imaginary part is zero.  The four bound the kernel (GB300's
    // FP64 pipe does two per clock and SM; a site density matrix of bond 8192,
    // 5 10^6 terms: 209 -> 171 us for the call).  Sums that leave the finite
    // numbers take the general form below.
    if (CPLX && A + 2 * a0 == B + 2 * b0 && as == bs && ca != cb) {
      double s[DOT_SELF_U];
#pragma unroll
      for (int u = 0; u < DOT_SELF_U; ++u) s[u] = 0.0;
      for (int64_t k = threadIdx.x; k < P.K; k += DOT_SELF_U * DOT_THREADS) {
        double2 a[DOT_SELF_U];
#pragma unroll
        for (int u = 0; u < DOT_SELF_U; ++u) {
          const int64_t kk = k + u * DOT_THREADS, ia = a0 + kk * as;
          a[u] = make_double2(0.0, 0.0);
          if (kk < P.K)
            a[u] = wide ? reinterpret_cast<const double2 *>(A)[ia] : make_double2(A[2 * ia], A[2 * ia + 1]);
        }
#pragma unroll
        for (int u = 0; u < DOT_SELF_U; ++u) s[u] = fma(a[u].x, a[u].x, fma(a[u].y, a[u].y, s[u]));
      }
#pragma unroll
      for (int u = 1; u < DOT_SELF_U; ++u) s[0] += s[u];
      if (isfinite(s[0])) {
        re += P.afac * s[0];
        continue;
      }
    }
    // DOT_U terms in flight per thread, each with its own running sum
    double sr[DOT_U], si[DOT_U];
#pragma unroll
    for (int u = 0; u < DOT_U; ++u) sr[u] = si[u] = 0.0;
    for (int64_t k = threadIdx.x; k < P.K; k += DOT_U * DOT_THREADS) {
      double2 a[DOT_U], b[DOT_U];
#pragma unroll
      for (int u = 0; u < DOT_U; ++u) {
        const int64_t kk = k + u * DOT_THREADS;
        a[u] = b[u] = make_double2(0.0, 0.0);
        if (kk < P.K) {
          const int64_t ia = a0 + kk * as, ib = b0 + kk * bs;
          if (CPLX) {
            a[u] = wide ? reinterpret_cast<const double2 *>(A)[ia] : make_double2(A[2 * ia], A[2 * ia + 1]);
            b[u] = wide ? reinterpret_cast<const double2 *>(B)[ib] : make_double2(B[2 * ib], B[2 * ib + 1]);
          } else {
            a[u].x = A[ia];
            b[u].x = B[ib];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < DOT_U; ++u) {
        if (k + u * DOT_THREADS >= P.K) break;
        if (CPLX) {
          const double ai = ca ? -a[u].y : a[u].y, bi = cb ? -b[u].y : b[u].y;
          sr[u] = fma(a[u].x, b[u].x, fma(-ai, bi, sr[u]));
          si[u] = fma(a[u].x, bi, fma(ai, b[u].x, si[u]));
        } else {
          sr[u] = fma(a[u].x, b[u].x, sr[u]);
        }
      }
    }
#pragma unroll
    for (int u = 1; u < DOT_U; ++u) {
      sr[0] += sr[u];
      si[0] += si[u];
    }
    re += P.afac * sr[0];
    im += P.afac * si[0];
  }
  red[0][threadIdx.x] = re;
  red[1][threadIdx.x] = im;
  __syncthreads();
  for (int w = DOT_THREADS / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      red[0][threadIdx.x] += red[0][threadIdx.x + w];
      red[1][threadIdx.x] += red[1][threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const int64_t o = t.c_off + t.i + t.j * (int64_t)t.ldc;
    if (CPLX) {
      C[2 * o] = red[0][0];
      C[2 * o + 1] = red[1][0];
    } else {
      C[o] = red[0][0];
    }
  }
}

}  // namespace

void run_dot(Ctx *ctx, const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
             const std::vector<int32_t> &bM, const std::vector<int32_t> &bN, const std::vector<int64_t> &coff,
             const std::vector<int32_t> *bldc, const std::vector<int64_t> &blocks, const double *A,
             const double *B, double *C, bool cplx) {
  std::vector<DotTask> tasks;
  for (int64_t b : blocks)
    for (int32_t j = 0; j < bN[b]; ++j)
      for (int32_t i = 0; i < bM[b]; ++i)
        tasks.push_back(DotTask{coff[b], (int32_t)grp[b], (int32_t)grp[b + 1], bM[b],
                                bldc ? (*bldc)[b] : std::max(bM[b], 1), i, j});
  if (tasks.empty()) return;
  if (tasks.size() > 0x7fffffff) fail(QS_ERR_SHAPE, "small-block products: too many outputs");
  DevLists L;
  const size_t st = L.add(tasks), sp = L.add(pairs);
  L.commit(ctx);
  const DotTask *dt = L.at<DotTask>(st);
  const PairDesc *dp = L.at<PairDesc>(sp);
  if (cplx) dot_kernel<true><<<(unsigned)tasks.size(), DOT_THREADS, 0, ctx->stream>>>(dt, dp, A, B, C);
  else dot_kernel<false><<<(unsigned)tasks.size(), DOT_THREADS, 0, ctx->stream>>>(dt, dp, A, B, C);
  QS_LAUNCHED(ctx);
}

bool is_shallow(const std::vector<PairDesc> &pairs, int64_t p0, int64_t p1) {
  int64_t depth = 0;
  for (int64_t p = p0; p < p1; ++p) depth += std::max<int32_t>(pairs[p].K, 0);
  return depth <= SHALLOW_K;
}

bool shallow_direct_wins(const std::vector<PairDesc> &pairs, int64_t p0, int64_t p1, int32_t M, int32_t N,
                         bool cplx) {
  int64_t depth = 0;
  for (int64_t p = p0; p < p1; ++p) depth += std::max<int32_t>(pairs[p].K, 0);
  const double m = M, n = N, cm = cplx ? 2.0 : 1.0;
  // direct: FP64 multiply-adds at ~1 TFLOP/s and the output written once
  const double direct = (cplx ? 8.0 : 2.0) * m * n * (double)depth / 1.0e12 + 8.0 * cm * m * n / 5.0e12;
  // tiled: 128 x 32 tiles of the real form, either orientation, ~3000 cycles
  // each (one k-block and the epilogue) spread over 152 SMs at 2 GHz
  auto tiles = [](double r, double c) { return std::ceil(r / 128.0) * std::ceil(c / 32.0); };
  const double t = std::min(tiles(cm * m, n), tiles(cm * n, m));
  const double tiled = t * 3000.0 / (152.0 * 2.0e9);
  return direct < tiled;
}

// Tasks over the listed blocks, whose pairs are numbered consecutively in
// list order (the compact pair list that goes with them).
static std::vector<ShallowTask> shallow_tasks(const std::vector<int64_t> &grp, const std::vector<int32_t> &bM,
                                              const std::vector<int32_t> &bN, const std::vector<int64_t> &coff,
                                              const std::vector<int32_t> *bldc, const std::vector<int64_t> &blocks,
                                              bool cplx) {
  const int NC = SHALLOW_NC, LINES = SHALLOW_THREADS * (cplx ? shallow_u<true>() : shallow_u<false>());
  std::vector<ShallowTask> tasks;
  int64_t p = 0;
  for (int64_t b : blocks) {
    ShallowTask t{};
    t.c_off = coff[b];
    t.p0 = (int32_t)p;
    p += grp[b + 1] - grp[b];
    t.p1 = (int32_t)p;
    t.M = bM[b];
    t.N = bN[b];
    t.ldc = bldc ? (*bldc)[b] : std::max(bM[b], 1);
    // rows as lines keep the stores coalesced; a block of fewer rows than a
    // warp has more parallelism along its columns
    t.swapped = t.M < 32 && t.N > t.M;
    const int32_t lines = t.swapped ? t.N : t.M, other = t.swapped ? t.M : t.N;
    for (int32_t o = 0; o < other; o += NC)
      for (int64_t l = 0; l < lines; l += LINES) {
        t.o0 = o;
        t.l0 = (int32_t)l;
        t.l1 = (int32_t)std::min<int64_t>(lines, l + LINES);
        tasks.push_back(t);
      }
  }
  if (tasks.size() > 0x7fffffff) fail(QS_ERR_SHAPE, "shallow products: too many tasks");
  return tasks;
}

template <class T>
static std::vector<T> pairs_of(const std::vector<T> &all, const std::vector<int64_t> &grp,
                               const std::vector<int64_t> &blocks) {
  std::vector<T> out;
  for (int64_t b : blocks) out.insert(out.end(), all.begin() + grp[b], all.begin() + grp[b + 1]);
  return out;
}

static void launch_shallow(Ctx *ctx, const ShallowTask *tasks, int64_t n, const PairDesc *pairs,
                           const OperandView *va, const OperandView *vb, const double *A, const double *B, double *C,
                           bool cplx) {
  if (cplx) shallow_kernel<true><<<(unsigned)n, SHALLOW_THREADS, 0, ctx->stream>>>(tasks, pairs, va, vb, A, B, C);
  else shallow_kernel<false><<<(unsigned)n, SHALLOW_THREADS, 0, ctx->stream>>>(tasks, pairs, va, vb, A, B, C);
  QS_LAUNCHED(ctx);
}

void run_shallow(Ctx *ctx, const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                 const std::vector<int32_t> &bM, const std::vector<int32_t> &bN, const std::vector<int64_t> &coff,
                 const std::vector<int32_t> *bldc, const std::vector<int64_t> &blocks, const double *A,
                 const double *B, double *C, bool cplx, const std::vector<OperandView> *va,
                 const std::vector<OperandView> *vb) {
  const std::vector<ShallowTask> tasks = shallow_tasks(grp, bM, bN, coff, bldc, blocks, cplx);
  if (tasks.empty()) return;
  const std::vector<PairDesc> pp = pairs_of(pairs, grp, blocks);
  const std::vector<OperandView> none;
  const std::vector<OperandView> wa = va ? pairs_of(*va, grp, blocks) : none;
  const std::vector<OperandView> wb = vb ? pairs_of(*vb, grp, blocks) : none;
  DevLists L;
  const size_t st = L.add(tasks), sp = L.add(pp), sa = L.add(wa), sb = L.add(wb);
  L.commit(ctx);
  launch_shallow(ctx, L.at<ShallowTask>(st), (int64_t)tasks.size(), L.at<PairDesc>(sp),
                 wa.empty() ? nullptr : L.at<OperandView>(sa), wb.empty() ? nullptr : L.at<OperandView>(sb), A, B, C,
                 cplx);
}

ShallowPlan shallow_prepare(Ctx *ctx, PlanLists &mem, const std::vector<PairDesc> &pairs,
                            const std::vector<int64_t> &grp, const std::vector<int32_t> &bM,
                            const std::vector<int32_t> &bN, const std::vector<int64_t> &coff,
                            const std::vector<int32_t> *bldc, const std::vector<int64_t> &blocks, bool cplx) {
  const std::vector<ShallowTask> tasks = shallow_tasks(grp, bM, bN, coff, bldc, blocks, cplx);
  const std::vector<PairDesc> pp = pairs_of(pairs, grp, blocks);
  ShallowPlan sp;
  sp.cplx = cplx;
  sp.ntasks = (int64_t)tasks.size();
  if (tasks.empty()) return sp;
  const size_t st = mem.add(tasks), so = mem.add(pp);
  mem.commit(ctx);
  sp.tasks = mem.at<ShallowTask>(st);
  sp.pairs = mem.at<PairDesc>(so);
  return sp;
}

void shallow_launch(Ctx *ctx, const ShallowPlan &sp, const double *A, const double *B, double *C) {
  if (!sp.ntasks) return;
  launch_shallow(ctx, static_cast<const ShallowTask *>(sp.tasks), sp.ntasks, static_cast<const PairDesc *>(sp.pairs),
                 nullptr, nullptr, A, B, C, sp.cplx);
}

BlockList select_blocks(const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                        const std::vector<int32_t> &bM, const std::vector<int32_t> &bN,
                        const std::vector<int64_t> &coff, const std::vector<int32_t> *bldc,
                        const std::vector<char> &sel) {
  BlockList L;
  L.grp.push_back(0);
  for (size_t b = 0; b < bM.size(); ++b) {
    if (!sel[b]) continue;
    for (int64_t p = grp[b]; p < grp[b + 1]; ++p) {
      L.pairs.push_back(pairs[p]);
      L.src.push_back((int32_t)p);
    }
    L.grp.push_back((int64_t)L.pairs.size());
    L.bM.push_back(bM[b]);
    L.bN.push_back(bN[b]);
    L.bldc.push_back(bldc ? (*bldc)[b] : std::max(bM[b], 1));
    L.coff.push_back(coff[b]);
  }
  return L;
}

bool has_deep_blocks(const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                     const std::vector<int32_t> &bM, const std::vector<int32_t> &bN) {
  for (size_t b = 0; b < bM.size(); ++b)
    if (parts_of(pairs, grp[b], grp[b + 1], bM[b], bN[b]) > 1) return true;
  return false;
}

bool split_deep(const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                const std::vector<int32_t> &bM, const std::vector<int32_t> &bN,
                const std::vector<int64_t> &coff, const std::vector<int32_t> *bldc, DeepSplit &out,
                const std::vector<char> *keep) {
  auto cut = [&](size_t b) -> int64_t {
    if (keep && (*keep)[b]) return 1;
    return parts_of(pairs, grp[b], grp[b + 1], bM[b], bN[b]);
  };
  bool any = false;
  for (size_t b = 0; b < bM.size() && !any; ++b) any = cut(b) > 1;
  if (!any) return false;
  DeepSplit d;
  d.grp.push_back(0);
  for (size_t b = 0; b < bM.size(); ++b) {
    const int64_t p0 = grp[b], p1 = grp[b + 1];
    const int32_t M = bM[b], N = bN[b];
    const int32_t ldc = bldc ? (*bldc)[b] : std::max(M, 1);
    const int64_t np = cut(b);
    if (np <= 1) {
      for (int64_t p = p0; p < p1; ++p) {
        d.pairs.push_back(pairs[p]);
        d.src.push_back((int32_t)p);
      }
      d.grp.push_back((int64_t)d.pairs.size());
      d.bM.push_back(M);
      d.bN.push_back(N);
      d.bldc.push_back(ldc);
      d.coff.push_back(coff[b]);
      d.part.push_back(0);
      continue;
    }
    int64_t depth = 0;
    for (int64_t p = p0; p < p1; ++p) depth += std::max<int32_t>(pairs[p].K, 0);
    const int64_t mn = (int64_t)M * N;
    DeepReduce r{coff[b], d.temp_elems, M, N, ldc, (int32_t)np};
    d.red.push_back(r);
    // part q covers the summed depth [q D / np, (q + 1) D / np): the pairs'
    // K ranges are cut where the parts meet
    int64_t p = p0, k = 0;  // position: pair p, depth k inside it
    for (int64_t q = 0; q < np; ++q) {
      const int64_t end = (q + 1 == np) ? depth : depth * (q + 1) / np;
      int64_t at = depth * q / np;
      while (at < end && p < p1) {
        const PairDesc &s = pairs[p];
        const int64_t K = std::max<int32_t>(s.K, 0);
        const int64_t take = std::min(K - k, end - at);
        if (take > 0) {
          PairDesc t = s;
          const int64_t lda = s.lda, ldb = s.ldb;
          // op(A) columns k .. k+take: A not transposed is M x K (column k at
          // k lda), transposed it is stored K x M (row k at k); op(B) rows
          // likewise
          t.a_off = s.a_off + ((s.trans & 1) ? k : k * lda);
          t.b_off = s.b_off + ((s.trans & 2) ? k * ldb : k);
          t.K = (int32_t)take;
          d.pairs.push_back(t);
          d.src.push_back((int32_t)p);
        }
        k += take;
        at += take;
        if (k >= K) {
          ++p;
          k = 0;
        }
      }
      // pairs without depth contribute nothing; a part left without pairs
      // still gets one of them so that its block is written (zeros)
      if ((int64_t)d.pairs.size() == d.grp.back()) {
        PairDesc t = pairs[p0];
        t.K = 0;
        d.pairs.push_back(t);
        d.src.push_back((int32_t)p0);
      }
      d.grp.push_back((int64_t)d.pairs.size());
      d.bM.push_back(M);
      d.bN.push_back(N);
      d.bldc.push_back(std::max(M, 1));
      d.coff.push_back(r.t_off + q * mn);
      d.part.push_back(1);
    }
    d.temp_elems += np * mn;
  }
  out = std::move(d);
  return true;
}

void launch_reduce_parts(Ctx *ctx, const DeepReduce *d_red, int64_t nred, const double *T, double *C, bool cplx) {
  if (nred <= 0) return;
  if (nred > 65535) fail(QS_ERR_SHAPE, "too many deep output blocks in one launch");
  const int gx = std::max(1, std::min(64, (int)(1024 / std::max<int64_t>(nred, 1)) + 1));
  reduce_parts_kernel<<<dim3(gx, (unsigned)nred), 256, 0, ctx->stream>>>(d_red, T, C, cplx ? 2 : 1);
  QS_LAUNCHED(ctx);
}

}  // namespace qs
