// Split-precision grouped block GEMM on the sm_103a tensor cores.
//
// Method (error-free digit slicing in the spirit of Ozaki, Ogita, Oishi and
// Rump, Numer. Algorithms 59 (2012), adapted to FP16 operands with exact FP32
// accumulation):
//
//  * Every output block gets one power-of-two scale per row of op(A) and per
//    column of op(B), taken over all block pairs that feed it
//    (E_i = max exponent of row i, F_j likewise).  Rows/columns are then
//    |x| < 2^E.
//  * Each scaled FP64 entry is rounded to the integer N = round(x 2^(bS-E))
//    and cut into S balanced signed digits of b bits,
//    N = sum_t d_t 2^(b(S-1-t)), |d_0| <= 2^b, |d_t| <= 2^(b-1).
//    The digits are small integers, exact in FP16.  The cut uses integer
//    operations on the FP64 bit pattern, and one FP64 multiply-add an entry
//    for 8-bit digits of at most 48 bits.
//  * The product of the two digit expansions is
//      sum_k x_ik y_kj = 2^(E_i+F_j-2b) sum_g 2^(-bg) acc_g,
//      acc_g = sum_k sum_{t+u=g} d_t(ik) d'_u(kj),   g = 0..S-1
//    (the triangular part; terms with t+u >= S are below the target).  b is
//    chosen so that |acc_g| < 2^24 for every partial sum: all tensor-core
//    accumulations in FP32 are then exact integer arithmetic.  When the summed
//    depth of a block exceeds that bound, the K loop is cut into chunks whose
//    accumulators are drained and added exactly (int64).
//  * The S digit tiles of B are laid side by side along N, so one
//    tcgen05.mma with A-digit t and N = (S-t)*32 produces all products
//    d_t * d'_u (u = 0..S-1-t) at once and drops each into the TMEM columns of
//    accumulator group g = t+u (column offset 32*g).  S(S+1)/2 digit
//    products therefore take about S + S/2 wide MMA instructions per K step.
//  * The CG factor of each pair is folded into A's digits with an exact
//    integer product (53 x 53 bits) before rounding, so pairs with different
//    factors share the accumulators.
//  * The epilogue reads the S accumulators from TMEM, combines them in int64
//    fixed point over all accumulator chunks of the block, and converts the
//    sum once (int64 to FP64, round to nearest even) with an integer exponent
//    add for the scale 2^(E_i+F_j-2b): GB300's FP64 pipe is narrow.  One CTA
//    owns one 128x32 output tile at a time and sums the block pairs in plan
//    order: the result is deterministic (atomics only list outputs that the
//    FP64-grade launch leaves to the FP64 kernel, not their values).
//
// Data movement: a slicing kernel writes the digits of every pair operand once
// into an HBM arena, pre-tiled in the tcgen05 K-major, no-swizzle core-matrix
// layout (8 rows x 16 bytes per core matrix); the GEMM kernel then moves
// whole digit tiles with 1-D TMA bulk copies (cp.async.bulk + mbarrier
// transaction counts) into a multi-stage shared-memory ring.  Warp roles:
// warp 0 = TMA producer, warp 1 = TMEM owner and MMA issuer, the other
// warps = epilogue (EPI_WARPS / 4 per TMEM lane quarter).  Every mbarrier wait is bounded; on
// timeout the kernel records an error code, stops issuing work, waits a
// bounded time for what is in flight, frees its TMEM and returns.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <memory>
#include <numeric>
#include <type_traits>

#include "qs_internal.h"
#include "qs_split.h"
#include "qs_xcache.h"

namespace qs {

namespace {

constexpr int TMS = 128;          // output tile rows (MMA M)
constexpr int TNS = 32;           // output tile cols (per digit group)
constexpr int TKS = 32;           // K block per pipeline stage (two MMA K steps)
constexpr int KCM = TKS / 8;      // core matrices along K in a digit tile
constexpr int A_DIGIT_BYTES = TMS * TKS * 2;  // 8 KB
constexpr int B_DIGIT_BYTES = TNS * TKS * 2;  // 2 KB
constexpr int MAX_STAGES = 8;
constexpr int EMPTY_EXP = -30000;
constexpr int NONFINITE_EXP = 20000;  // lines with an infinity or NaN (FP64-grade launches)
constexpr int SMEM_HDR = 2048;   // barriers, TMEM slot, abort flag; tile-descriptor slots at 1024
constexpr int SMEM_LIMIT = 227 * 1024;
constexpr uint32_t WAIT_LIMIT = 1u << 22;  // bounded mbarrier polls (seconds)
constexpr int EPI_WARPS = 16;     // epilogue warps (4 per TMEM lane quarter)
constexpr int GEMM_THREADS = 64 + 32 * EPI_WARPS;
constexpr int TILE_SLOTS = 1024;  // shared-memory offset of the epilogue warps' descriptor slots

struct SplitPair {
  int64_t a_off, b_off;    // element offsets of op(A)/op(B) storage
  int64_t as_off, bs_off;  // byte offsets of this pair's digit tiles
  int32_t M, N, K;         // logical (complex or real) sizes
  int32_t lda, ldb, trans;
  int32_t Mr, Kr;          // real rows of op(A~) and real depth
  int32_t MT, NT, KB;      // tile counts
  int32_t eoff, foff;      // exponent array offsets of the output block
  int32_t e_afac;          // exponent added by the CG factor (|afac| < 2^e)
  int32_t fe, fneg;        // CG factor folded into A's digits: fm 2^fe, sign
  uint64_t fm;             // (fm = 0: factor 1)
  double fac;              // the factor
  int32_t swap;            // block computed as C^T = op(B)^T op(A)^T: the A role reads the B arena
  // Real form of a complex block.  dupb = 0: A~ (2M x 2K) rows 2m, 2m+1 =
  // (Re, -Im), (Im, Re) of row m of op(A), B~ (2K x N) rows 2k, 2k+1 = (Re, Im)
  // of op(B), C~ (2M x N) rows = (Re, Im) of C.  dupb = 1: A' (M x 2K) columns
  // 2k, 2k+1 = (Re, Im) of op(A), B' (2K x 2N) columns 2n = (Re; -Im) and
  // 2n+1 = (Im; Re) of column n of op(B), C' (M x 2N) columns = (Re, Im) of C.
  int32_t dupb;
  int32_t Nr;              // real columns of op(B~)
  int32_t pad_;
};

struct SplitTile {
  int64_t c_off;           // double offset of the output block (first member: 8-byte aligned)
  int32_t p0, p1;
  int32_t mt, nt;
  int32_t Mr, N, ldc;
  int32_t eoff, foff;
  int32_t nchunk;          // drains of the accumulators
  int32_t rshift;          // bits dropped below the lowest group (int64 headroom)
  // output address of tile row r, column j (doubles from c_off):
  // (r >> rsplit) * rs + (r & rsplit) + (j >> csplit) * ldc + (j & csplit),
  // splits = rsplit | csplit << 1 | swapped << 2 | rdup << 3 | cdup << 4;
  // rsplit = 1 for a complex block computed transposed in the A-duplicated
  // form (its rows interleave Re/Im of C's columns), csplit = 1 for one in
  // the B-duplicated form, not transposed (its columns interleave Re/Im of
  // C's columns); swapped: the block is computed as C^T; rdup / cdup: two
  // tile rows / columns per row / column of the computed block
  int32_t rs, splits;
  int32_t fbase;           // FP64-grade launches: first FP64 tile of the block
};
constexpr int TILE_WORDS = (int)(sizeof(SplitTile) / 4);
static_assert(sizeof(SplitTile) % 8 == 0 && TILE_WORDS <= 16, "tile descriptor fits one 64-byte slot");

// ------------------------------------------------------------ bit helpers
// Largest magnitude of a line, as far as its exponent goes: the high words'
// maximum without the signs, and the low words' bits (a line of subnormals
// below 2^-1042 has zero high words).
struct LineMax {
  unsigned hi = 0, lo = 0;
  __device__ __forceinline__ void add(double x) {
    hi = max(hi, (unsigned)__double2hiint(x) & 0x7fffffffu);
    lo |= (unsigned)__double2loint(x);
  }
  // biased exponent of the maximum (at least 1), 0 for a line of zeros
  __device__ __forceinline__ int key() const { return (hi | lo) ? max((int)(hi >> 20), 1) : 0; }
};

// A factor f (CG coefficient) as an exact integer mantissa and exponent,
// f = fm * 2^fe, 2^52 <= fm < 2^53; fm = 0 means "no factor" (f = 1); fe = -100000
// means f = 0.
struct Factor {
  unsigned long long fm;
  int fe;
  bool neg;
  double f;  // the factor itself
};

__host__ __device__ inline Factor make_factor(double f) {
  Factor r{0ull, 0, false, f};
  if (f == 1.0) return r;
  unsigned long long bits;
  memcpy(&bits, &f, 8);
  int be = (int)((bits >> 52) & 0x7ff);
  unsigned long long m = bits & 0xFFFFFFFFFFFFFull;
  if (be != 0) {
    m |= 1ull << 52;
  } else if (m) {
    // a subnormal factor: normalised, since scaled_int keeps the upper bits of
    // the product of the two mantissas
    for (be = 1; !(m >> 52); --be) m <<= 1;
  }
  r.fm = m;
  r.fe = be - 1075;
  r.neg = (bits >> 63) != 0;
  if (!m) { r.fm = 0; r.fe = 0; r.neg = false; r.fe = -100000; }  // f == 0
  return r;
}

// N = round(x f 2^(b*S - E)); |x f| < 2^E is guaranteed by construction of
// E, so |N| <= 2^(bS) (b*S <= 62).  Integer operations only.
__device__ __forceinline__ long long scaled_int(double x, int E, int bS, const Factor &F) {
  const long long bits = __double_as_longlong(x);
  int be = (int)((bits >> 52) & 0x7ff);
  unsigned long long mant = bits & 0xFFFFFFFFFFFFFull;
  if (be == 0) be = 1; else mant |= (1ull << 52);
  long long N = 0;
  bool neg = bits < 0;
  if (mant != 0 && F.fe > -100000) {
    if (F.fm == 0) {
      // N = round(mant * 2^shift)
      const int shift = be - 1075 + bS - E;
      if (shift >= 0) N = (long long)(mant << min(shift, 62));
      else if (shift > -62) N = (long long)((mant + (1ull << (-shift - 1))) >> (-shift));
    } else {
      // product with the factor's mantissa: the upper 64 bits of
      // (mant 2^11) (fm 2^11), i.e. mant fm 2^-42 truncated (relative error
      // < 2^-63, far below the 2^-(bS) of the digits), then the rounding shift
      // (|x f| < 2^E holds by construction of E)
      const unsigned long long P = __umul64hi(mant << 11, F.fm << 11);
      const int shift = be - 1075 + F.fe + 42 + bS - E;
      if (shift >= 0) N = (long long)(P << min(shift, 62));
      else if (shift > -64) N = (long long)((P >> (-shift - 1)) + 1 >> 1);
      neg ^= F.neg;
    }
    if (neg) N = -N;
  }
  return N;
}

// Balanced base-2^B digits of N as floats (exact small integers):
//   N = sum_t d_t 2^(B(S-1-t)),  d_t in [-2^(B-1), 2^(B-1)) for t >= 1,
//   |d_0| <= 2^B.
// With H = sum_{t>=1} 2^(B-1) 2^(B(S-1-t)), the low B(S-1) bits of M = N + H
// are the base-2^B digits d_t + 2^(B-1), and d_0 = floor(M / 2^(B(S-1))).
// Each digit is a funnel shift, one logic op (mask | 2^23 exponent) and one
// FP32 subtraction; all values are exact in FP16 (at most 9 significant bits).
template <int S, int B>
__device__ __forceinline__ void digits_f(long long N, float (&d)[S]) {
  constexpr long long HALF = 1LL << (B - 1);
  constexpr unsigned MASK = (1u << B) - 1;
  long long H = 0;
#pragma unroll
  for (int t = 1; t < S; ++t) H = (H << B) + HALF;
  const long long M = N + H;
  const unsigned lo = (unsigned)M, hi = (unsigned)((unsigned long long)M >> 32);
#pragma unroll
  for (int t = 1; t < S; ++t) {
    const int sh = B * (S - 1 - t);
    const unsigned w = sh >= 32 ? (hi >> (sh - 32)) : (sh == 0 ? lo : __funnelshift_r(lo, hi, sh));
    d[t] = __int_as_float((int)((w & MASK) | 0x4B000000u)) - (8388608.0f + (float)HALF);
  }
  const int d0 = (int)(M >> (B * (S - 1)));
  d[0] = __int_as_float(0x4B400000 + d0) - 12582912.0f;
}

// ---- digits of two values as packed FP16 planes
// The digits are integers of at most 9 bits, exact in FP16.  For 8-bit digits
// a value is first brought into the fixed-point word
//   W = N + sum_{t>=1} 2^7 2^(8(S-1-t)) + 2^9 2^(8(S-1)),
// whose bytes are d_t + 128 and whose ten bits from 8(S-1) on are d_0 + 512
// (bits above are not looked at).  One byte permute takes the same digit of
// two values, one logic operation puts it behind the exponent of 1024 (an
// FP16 whose last place is one) and one packed subtraction removes the
// offset: 1.5 instructions per digit, against 3.5 with a shift, a mask, an
// FP32 subtraction and a conversion (the strips' ALU pipe was 60-70 % busy).
template <int S>
__host__ __device__ constexpr unsigned long long word_offset() {
  unsigned long long h = 0;
  for (int t = 1; t < S; ++t) h = (h << 8) + 128;
  return h + (512ull << (8 * (S - 1)));
}

// Words of at most six digits come from the FP64 pipe, idle otherwise: the low
// mantissa bits of x f + C are N = round(x f 2^(8S-E)) plus C's own, for C =
// 2^(E-8S) (2^52 + 2^51 + word_offset).  C is not a normal number for extreme
// E: those lines take the integer form.
template <int S>
struct LineScale {
  double c = 0.0;
  bool fast = false;
  __device__ __forceinline__ LineScale(int E) {
    const int be = E - 8 * S + 52 + 1023;
    fast = S <= 6 && be > 0 && be < 2046;
    if (fast) c = __longlong_as_double(((long long)be << 52) + (1ll << 51) + (long long)word_offset<S>());
  }
};

template <int S, int B>
__device__ __forceinline__ unsigned long long fixed_word(double x, int E, const LineScale<S> &ls, const Factor &F) {
  if constexpr (B == 8) {
    if (S <= 6 && ls.fast) return (unsigned long long)__double_as_longlong(fma(x, F.f, ls.c));
    return (unsigned long long)scaled_int(x, E, B * S, F) + word_offset<S>();
  } else {
    return (unsigned long long)scaled_int(x, E, B * S, F);
  }
}

// Plane t of the digits of two values: (first, second) as the halves of w[t].
template <int S, int B>
__device__ __forceinline__ void digit_planes(unsigned long long w0, unsigned long long w1, uint32_t (&w)[S]) {
  if constexpr (B == 8) {
    const uint32_t l0 = (uint32_t)w0, h0 = (uint32_t)(w0 >> 32), l1 = (uint32_t)w1, h1 = (uint32_t)(w1 >> 32);
    const __half2 off = __float2half2_rn(1152.0f), off0 = __float2half2_rn(1536.0f);
    auto sub = [](uint32_t v, __half2 o) {
      const __half2 d = __hsub2(*reinterpret_cast<const __half2 *>(&v), o);
      return *reinterpret_cast<const uint32_t *>(&d);
    };
#pragma unroll
    for (int t = 1; t < S; ++t) {
      const int by = S - 1 - t;
      const uint32_t k = by & 3, sel = k | ((4 + k) << 8);
      const uint32_t u = by < 4 ? __byte_perm(l0, l1, sel) : __byte_perm(h0, h1, sel);
      w[t] = sub((u & 0x00FF00FFu) | 0x64006400u, off);
    }
    constexpr int top = S - 1;  // first byte of the leading field
    uint32_t u;
    if constexpr (top == 3) u = __byte_perm(__funnelshift_r(l0, h0, 24), __funnelshift_r(l1, h1, 24), 0x5410);
    else if constexpr (top < 3) u = __byte_perm(l0, l1, top == 1 ? 0x6521 : 0x7632);
    else u = __byte_perm(h0, h1, top == 4 ? 0x5410 : top == 5 ? 0x6521 : 0x7632);
    w[0] = sub((u & 0x03FF03FFu) | 0x64006400u, off0);
  } else {
    float d0[S], d1[S];
    digits_f<S, B>((long long)w0, d0);
    digits_f<S, B>((long long)w1, d1);
#pragma unroll
    for (int t = 0; t < S; ++t) {
      const __half2 v = __floats2half2_rn(d0[t], d1[t]);
      w[t] = *reinterpret_cast<const uint32_t *>(&v);
    }
  }
}

// max(|d_0| - 1/2, 0) of two leading digits (exact in FP16): d_0 is rounded, so
// this, not |d_0|, stays below the entry's own magnitude (up to 0.4 %: the
// other digits reach 128/255 of a unit, not a half).
__device__ __forceinline__ uint32_t lower_magnitudes(uint32_t w) {
  const uint32_t a = w & 0x7FFF7FFFu;
  const __half2 m = __hmax2(__hsub2(*reinterpret_cast<const __half2 *>(&a), __float2half2_rn(0.5f)), __float2half2_rn(0.0f));
  return *reinterpret_cast<const uint32_t *>(&m);
}

// L2 eviction priorities of the strip kernels (createpolicy, PTX ISA 7.4+):
// the first read of an operand line is kept (evict_last) for the re-read of
// phase 2, which is its last use (evict_first), and the digit stores stream
// through (evict_first), so that they do not push the operand lines out.
__device__ __forceinline__ uint64_t l2_policy_keep() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_stream() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ double2 ld_pol(const double2 *a, uint64_t pol) {
  double2 v;
  asm volatile("ld.global.nc.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(v.x), "=d"(v.y) : "l"(a), "l"(pol));
  return v;
}
__device__ __forceinline__ double ld_pol(const double *a, uint64_t pol) {
  double v;
  asm volatile("ld.global.nc.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(a), "l"(pol));
  return v;
}
__device__ __forceinline__ void st_pol(uint8_t *a, uint4 v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.v4.b32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(a), "r"(v.x), "r"(v.y), "r"(v.z),
               "r"(v.w), "l"(pol)
               : "memory");
}

// Element (line, k) of a pair's operand in the role being sliced: plain
// (lda/ldb, trans) addressing, or the offset tables of the operand's strided
// view when the contraction reads a permuted operand in place.
struct OpAddr {
  int64_t ls, ks;             // plain: line * ls + k * ks
  const int64_t *lt, *kt;     // or the view's tables (nullptr: plain)
  bool kunit;                 // unit depth stride (neighbouring k adjacent)
  __device__ __forceinline__ int64_t line(int64_t m) const { return lt ? lt[m] : m * ls; }
  __device__ __forceinline__ int64_t depth(int64_t k) const { return kt ? kt[k] : k * ks; }
};
// A role: lines are rows of op(A) (contiguous along k when transposed); B
// role: lines are columns of op(B) (contiguous along k when not transposed).
__device__ __forceinline__ OpAddr view_addr(const OperandView *views, int p, int64_t ls, int64_t ks) {
  if (views && views[p].nl > 0) {
    const OperandView &v = views[p];
    return OpAddr{0, 0, v.ltab, v.ktab, v.nk > 0 && v.kstr[0] == 1};
  }
  return OpAddr{ls, ks, nullptr, nullptr, ks == 1};
}
__device__ __forceinline__ OpAddr addr_a(const SplitPair &P, const OperandView *views, int p) {
  const bool ta = P.trans & 1;
  return view_addr(views, p, ta ? (int64_t)P.lda : 1, ta ? 1 : (int64_t)P.lda);
}
__device__ __forceinline__ OpAddr addr_b(const SplitPair &P, const OperandView *views, int p) {
  const bool tb = P.trans & 2;
  return view_addr(views, p, tb ? 1 : (int64_t)P.ldb, tb ? (int64_t)P.ldb : 1);
}

// ---------------------------------------------- exponents and slicing, fused
// One CTA per strip of STRIP real lines of one output block: rows of op(A~)
// (A role) or columns of op(B~) (B role), over every pair of the block and
// its whole depth.
//  Phase 1: the exponent of each line of the strip -- the largest exponent
//    key over all pairs and all k (both parts of a complex element), plus the
//    pair's CG-factor exponent for the A role -- kept in shared memory and
//    written to E / F for the epilogue (every line belongs to one strip, so
//    plain stores).  A line of zeros keeps EMPTY_EXP.
//  Phase 2: the digits of the strip's lines for every pair and k-block,
//    written into the pre-tiled digit arena.  It re-reads what phase 1 has
//    just read: a strip holds at most STRIP lines of the block's depth, so
//    the re-read is mostly served from L2 and the FP64 operands cross HBM
//    once.
// A complex block in the A-duplicated form turns each row m of op(A) into
// the real rows 2m, 2m+1 of A~ (rows (Re, -Im) and (Im, Re) along k) and
// each column of op(B) into one column of B~ (rows 2k, 2k+1 = (Re, Im));
// in the B-duplicated form row m of op(A) is one row of A' ((Re, Im) along
// k) and column n of op(B) the columns 2n, 2n+1 of B' ((Re; -Im), (Im; Re)).
constexpr int STRIP = 16;          // real lines per strip (two core-matrix groups)
// 256 threads, five CTAs an SM: the last wave of deep strips is shorter than with
// 128 threads and ten CTAs (480 real products 176 -> 169 us, 300 complex FP64
// products 1150 -> 1138 us, the 2000-product batch the same); 512 threads leave
// too few strips in flight (4.54 -> 4.98 ms)
constexpr int STRIP_THREADS = 256;

// Phase 1 for the lines l0 .. l0+nl-1 of op(X) (X = A role: rows, line m at
// m + k*ld (contig: k + m*ld); X = B role: columns, line n at k + n*ld
// (contig) or n + k*ld), max over the pairs p0..p1-1 into smax[line].
template <bool CPLX, bool ROLE_B, bool HP>
__device__ __forceinline__ void strip_maxima(const SplitPair *__restrict__ pairs, const OperandView *views, int p0,
                                             int p1, int l0, int nl, const double *__restrict__ Aarena,
                                             const double *__restrict__ Barena, int *smax) {
  if (threadIdx.x < STRIP) smax[threadIdx.x] = EMPTY_EXP;
  __syncthreads();
  for (int p = p0; p < p1; ++p) {
    const SplitPair &P = pairs[p];
    // a swapped pair's roles read the other arena
    const double *__restrict__ X = (ROLE_B != (P.swap != 0)) ? Barena : Aarena;
    const int64_t off = ROLE_B ? P.b_off : P.a_off;
    const OpAddr ad = ROLE_B ? addr_b(P, views, p) : addr_a(P, views, p);
    // lines contiguous along k (unit depth stride): neighbouring lanes take
    // neighbouring k of one line; else neighbouring lines
    const bool contig = ad.kunit;
    constexpr int NPH = STRIP_THREADS / STRIP;
    const int line = contig ? threadIdx.x / NPH : threadIdx.x % STRIP;
    const int ph = contig ? threadIdx.x % NPH : threadIdx.x / STRIP;
    LineMax lm;
    if (line < nl) {
      const uint64_t keep = l2_policy_keep();
      const int64_t base = off + ad.line(l0 + line);
      int k = ph;
      for (; k + 3 * NPH < P.K; k += 4 * NPH) {
        const int64_t o0 = base + ad.depth(k), o1 = base + ad.depth(k + NPH), o2 = base + ad.depth(k + 2 * NPH),
                      o3 = base + ad.depth(k + 3 * NPH);
        if (CPLX) {
          const double2 *x = reinterpret_cast<const double2 *>(X);
          const double2 v[4] = {ld_pol(x + o0, keep), ld_pol(x + o1, keep), ld_pol(x + o2, keep), ld_pol(x + o3, keep)};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            lm.add(v[u].x);
            lm.add(v[u].y);
          }
        } else {
          const double v[4] = {ld_pol(X + o0, keep), ld_pol(X + o1, keep), ld_pol(X + o2, keep), ld_pol(X + o3, keep)};
#pragma unroll
          for (int u = 0; u < 4; ++u) lm.add(v[u]);
        }
      }
      for (; k < P.K; k += NPH) {
        const int64_t o = base + ad.depth(k);
        if (CPLX) {
          const double2 v = ld_pol(reinterpret_cast<const double2 *>(X) + o, keep);
          lm.add(v.x);
          lm.add(v.y);
        } else {
          lm.add(ld_pol(X + o, keep));
        }
      }
    }
    int key = lm.key();
    // an infinity or NaN: no scale; every tile that reads the line goes to the FP64 kernel
    if (HP && key == 0x7ff) key = NONFINITE_EXP + 1022 - (ROLE_B ? 0 : P.e_afac);
    if (key) atomicMax(&smax[line], key - 1022 + (ROLE_B ? 0 : P.e_afac));
  }
  __syncthreads();
}

// A role.  Task = (first pair, end pair, first real row r0 of the strip).
template <bool CPLX, int S, int B, bool HP>
__device__ __forceinline__ void strip_a(const SplitPair *__restrict__ pairs, const OperandView *views, int4 tk,
                                        const double *__restrict__ Aarena, const double *__restrict__ Barena,
                                        int *__restrict__ E, uint8_t *__restrict__ arena) {
  constexpr int NP = S + (HP ? 1 : 0);  // digit planes, and the magnitudes of the leading one
  __shared__ int smax[STRIP];
  const int p0 = tk.x, p1 = tk.y, r0 = tk.z;
  const SplitPair &Q = pairs[p0];
  const bool dup = CPLX && Q.dupb == 0;  // two real rows per row of op(A)
  const int l0 = dup ? r0 / 2 : r0;
  const int nl = min(dup ? STRIP / 2 : STRIP, Q.M - l0);
  strip_maxima<CPLX, false, HP>(pairs, views, p0, p1, l0, nl, Aarena, Barena, smax);
  if (threadIdx.x < nl) {
    const int e = smax[threadIdx.x];
    if (dup) {
      E[Q.eoff + 2 * (l0 + threadIdx.x)] = e;
      E[Q.eoff + 2 * (l0 + threadIdx.x) + 1] = e;
    } else {
      E[Q.eoff + l0 + threadIdx.x] = e;
    }
  }
  const int mt = r0 / TMS, rl = r0 % TMS;
  const uint64_t last = l2_policy_stream();  // last use of operand lines; digit stores
  for (int p = p0; p < p1; ++p) {
    const SplitPair &P = pairs[p];
    const double *__restrict__ A = P.swap ? Barena : Aarena;
    const bool ca = P.trans & 4;
    const OpAddr ad = addr_a(P, views, p);
    const Factor Fa{P.fm, P.fe, P.fneg != 0, P.fac};
    uint8_t *tiles = arena + P.as_off + (int64_t)mt * P.KB * NP * A_DIGIT_BYTES;
    if (dup) {
      // item = one row of op(A) (real rows 2m, 2m+1) x 4 complex k
      const int items = (STRIP / 2) * KCM * P.KB;
      for (int w = threadIdx.x; w < items; w += blockDim.x) {
        const int kb = w / ((STRIP / 2) * KCM), i = w % ((STRIP / 2) * KCM);
        const int ml = i % (STRIP / 2), q = i / (STRIP / 2);
        if (ml >= nl) continue;  // rows past the block feed discarded outputs only: not written
        const int64_t lo = P.a_off + ad.line(l0 + ml);
        const int Ei = smax[ml];
        double2 a[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int k = (kb * TKS + q * 8) / 2 + j;
          a[j] = make_double2(0.0, 0.0);
          if (k < P.K) a[j] = ld_pol(reinterpret_cast<const double2 *>(A) + lo + ad.depth(k), last);
        }
        // ( re, im ) per plane; the rows 2m and 2m+1 are formed from it at the
        // stores, which saves half of the digit registers (72 -> 54, two more
        // CTAs per SM; the strips of the 2000-product batch 1.98 -> 1.89 ms)
        uint32_t pw[NP][4];
        const LineScale<S> ls(Ei);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t w2[S];
          digit_planes<S, B>(fixed_word<S, B>(a[j].x, Ei, ls, Fa),
                             fixed_word<S, B>(ca ? -a[j].y : a[j].y, Ei, ls, Fa), w2);
#pragma unroll
          for (int t = 0; t < S; ++t) pw[t][j] = w2[t];
          if constexpr (HP) pw[S][j] = lower_magnitudes(w2[0]);
        }
        const int rr0 = rl + 2 * ml, rr1 = rr0 + 1;
        uint8_t *tile = tiles + (int64_t)kb * NP * A_DIGIT_BYTES;
        uint8_t *d0 = tile + ((rr0 >> 3) * KCM + q) * 128 + (rr0 & 7) * 16;
        uint8_t *d1 = tile + ((rr1 >> 3) * KCM + q) * 128 + (rr1 & 7) * 16;
#pragma unroll
        for (int t = 0; t < NP; ++t) {
          const uint32_t neg = t < S ? 0x80000000u : 0u;  // row 2m: ( re, -im )
          st_pol(d0 + t * A_DIGIT_BYTES,
                 make_uint4(pw[t][0] ^ neg, pw[t][1] ^ neg, pw[t][2] ^ neg, pw[t][3] ^ neg), last);
          // row 2m+1: ( im, re )
          st_pol(d1 + t * A_DIGIT_BYTES,
                 make_uint4(__byte_perm(pw[t][0], 0, 0x1032), __byte_perm(pw[t][1], 0, 0x1032),
                            __byte_perm(pw[t][2], 0, 0x1032), __byte_perm(pw[t][3], 0, 0x1032)),
                 last);
        }
      }
    } else {
      // item = one real row x 8 real k (4 complex k of the B-duplicated form)
      const int items = STRIP * KCM * P.KB;
      for (int w = threadIdx.x; w < items; w += blockDim.x) {
        const int kb = w / (STRIP * KCM), i = w % (STRIP * KCM);
        const int rloc = i % STRIP, q = i / STRIP;
        if (rloc >= nl) continue;
        const int64_t lo = P.a_off + ad.line(l0 + rloc);
        const int Ei = smax[rloc];
        uint32_t pk[NP][4];
        if constexpr (CPLX) {
          double2 a[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int k = (kb * TKS + q * 8) / 2 + j;
            a[j] = make_double2(0.0, 0.0);
            if (k < P.K) a[j] = ld_pol(reinterpret_cast<const double2 *>(A) + lo + ad.depth(k), last);
          }
          const LineScale<S> ls(Ei);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t w2[S];
            digit_planes<S, B>(fixed_word<S, B>(a[j].x, Ei, ls, Fa),
                               fixed_word<S, B>(ca ? -a[j].y : a[j].y, Ei, ls, Fa), w2);
#pragma unroll
            for (int t = 0; t < S; ++t) pk[t][j] = w2[t];
          }
        } else {
          double v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int kk = kb * TKS + q * 8 + e;
            v[e] = 0.0;
            if (kk < P.Kr) v[e] = ld_pol(A + lo + ad.depth(kk), last);
          }
          const LineScale<S> ls(Ei);
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            uint32_t w2[S];
            digit_planes<S, B>(fixed_word<S, B>(v[e], Ei, ls, Fa), fixed_word<S, B>(v[e + 1], Ei, ls, Fa), w2);
#pragma unroll
            for (int t = 0; t < S; ++t) pk[t][e >> 1] = w2[t];
          }
        }
        if constexpr (HP) {
#pragma unroll
          for (int j = 0; j < 4; ++j) pk[S][j] = lower_magnitudes(pk[0][j]);
        }
        const int rr = rl + rloc;
        uint8_t *dst = tiles + (int64_t)kb * NP * A_DIGIT_BYTES + ((rr >> 3) * KCM + q) * 128 + (rr & 7) * 16;
#pragma unroll
        for (int t = 0; t < NP; ++t)
          st_pol(dst + t * A_DIGIT_BYTES, make_uint4(pk[t][0], pk[t][1], pk[t][2], pk[t][3]), last);
      }
    }
  }
}

// B role.  Task = (first pair, end pair, first real column c0 of the strip).
template <bool CPLX, int S, int B, bool HP>
__device__ __forceinline__ void strip_b(const SplitPair *__restrict__ pairs, const OperandView *views, int4 tk,
                                        const double *__restrict__ Aarena, const double *__restrict__ Barena,
                                        int *__restrict__ F, uint8_t *__restrict__ arena) {
  constexpr int NP = S + (HP ? 1 : 0);
  __shared__ int smax[STRIP];
  const int p0 = tk.x, p1 = tk.y, c0 = tk.z;
  const SplitPair &Q = pairs[p0];
  const bool dup = CPLX && Q.dupb != 0;  // two real columns per column of op(B)
  const int l0 = dup ? c0 / 2 : c0;
  const int nl = min(dup ? STRIP / 2 : STRIP, Q.N - l0);
  strip_maxima<CPLX, true, HP>(pairs, views, p0, p1, l0, nl, Aarena, Barena, smax);
  if (threadIdx.x < nl) {
    const int e = smax[threadIdx.x];
    if (dup) {
      F[Q.foff + 2 * (l0 + threadIdx.x)] = e;
      F[Q.foff + 2 * (l0 + threadIdx.x) + 1] = e;
    } else {
      F[Q.foff + l0 + threadIdx.x] = e;
    }
  }
  const int nt = c0 / TNS, cl = c0 % TNS;
  const int ncols = dup ? 2 * nl : nl;  // real columns of this strip inside the block
  const Factor F1{0ull, 0, false, 1.0};
  const uint64_t last = l2_policy_stream();  // last use of operand lines; digit stores
  for (int p = p0; p < p1; ++p) {
    const SplitPair &P = pairs[p];
    const double *__restrict__ Bm = P.swap ? Aarena : Barena;
    const bool cb = P.trans & 8;
    const OpAddr ad = addr_b(P, views, p);
    uint8_t *tiles = arena + P.bs_off + (int64_t)nt * P.KB * NP * B_DIGIT_BYTES;
    // item = one real column x 8 real k
    const int items = STRIP * KCM * P.KB;
    for (int w = threadIdx.x; w < items; w += blockDim.x) {
      const int kb = w / (STRIP * KCM), i = w % (STRIP * KCM);
      const int cloc = i % STRIP, q = i / STRIP;
      if (cloc >= ncols) continue;  // columns past the block feed discarded outputs only
      const int c = cl + cloc;
      const int Fj = smax[dup ? cloc >> 1 : cloc];
      uint32_t pk[NP][4];
      if constexpr (CPLX) {
        const int64_t lo = P.b_off + ad.line(dup ? l0 + (cloc >> 1) : l0 + cloc);
        double2 x[4];
        // B~ (A-duplicated form): rows 2k, 2k+1 = (Re, Im) of element k; B'
        // (B-duplicated form): the same 4 complex k per 8 real rows
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int k = (kb * TKS + q * 8) / 2 + j;
          x[j] = make_double2(0.0, 0.0);
          if (k < P.K) x[j] = ld_pol(reinterpret_cast<const double2 *>(Bm) + lo + ad.depth(k), last);
        }
        // B-duplicated form: even columns ( re; -im ), odd ones ( im; re )
        const bool odd = dup && (cloc & 1);
        const uint32_t sel = odd ? 0x1032u : 0x3210u, neg = dup && !odd ? 0x80000000u : 0u;
        const LineScale<S> ls(Fj);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t w2[S];
          digit_planes<S, B>(fixed_word<S, B>(x[j].x, Fj, ls, F1),
                             fixed_word<S, B>(cb ? -x[j].y : x[j].y, Fj, ls, F1), w2);
#pragma unroll
          for (int t = 0; t < S; ++t) pk[t][j] = dup ? __byte_perm(w2[t], 0, sel) ^ neg : w2[t];
        }
      } else {
        const int64_t lo = P.b_off + ad.line(l0 + cloc);
        double v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int kk = kb * TKS + q * 8 + e;
          v[e] = 0.0;
          if (kk < P.Kr) v[e] = ld_pol(Bm + lo + ad.depth(kk), last);
        }
        const LineScale<S> ls(Fj);
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          uint32_t w2[S];
          digit_planes<S, B>(fixed_word<S, B>(v[e], Fj, ls, F1), fixed_word<S, B>(v[e + 1], Fj, ls, F1), w2);
#pragma unroll
          for (int t = 0; t < S; ++t) pk[t][e >> 1] = w2[t];
        }
      }
      if constexpr (HP) {
#pragma unroll
        for (int j = 0; j < 4; ++j) pk[S][j] = lower_magnitudes(pk[0][j]);
      }
      uint8_t *dst = tiles + (int64_t)kb * NP * B_DIGIT_BYTES + ((c >> 3) * KCM + q) * 128 + (c & 7) * 16;
#pragma unroll
      for (int t = 0; t < NP; ++t)
        st_pol(dst + t * B_DIGIT_BYTES, make_uint4(pk[t][0], pk[t][1], pk[t][2], pk[t][3]), last);
    }
  }
}

// VIEWS = false: no pair of the launch reads its operand through a view, and
// the view addressing is compiled out
template <bool CPLX, int S, bool VIEWS, bool HP>
__global__ void __launch_bounds__(STRIP_THREADS, 5)
strip_a_kernel(const SplitPair *__restrict__ pairs, const OperandView *__restrict__ views_in,
               const int4 *__restrict__ tasks, const double *__restrict__ A, const double *__restrict__ B,
               int *__restrict__ E, uint8_t *__restrict__ arena, int b) {
  const OperandView *views = VIEWS ? views_in : nullptr;
  const int4 tk = tasks[blockIdx.x];
  if constexpr (HP) {  // FP64-grade launches: always 8-bit digits
    strip_a<CPLX, S, 8, true>(pairs, views, tk, A, B, E, arena);
  } else {
    switch (b) {  // the host admits b = 5..8 only
      case 5: strip_a<CPLX, S, 5, false>(pairs, views, tk, A, B, E, arena); break;
      case 6: strip_a<CPLX, S, 6, false>(pairs, views, tk, A, B, E, arena); break;
      case 7: strip_a<CPLX, S, 7, false>(pairs, views, tk, A, B, E, arena); break;
      default: strip_a<CPLX, S, 8, false>(pairs, views, tk, A, B, E, arena); break;
    }
  }
}

// VIEWS = false: no pair of the launch reads its operand through a view, and
// the view addressing is compiled out
template <bool CPLX, int S, bool VIEWS, bool HP>
__global__ void __launch_bounds__(STRIP_THREADS, 5)
strip_b_kernel(const SplitPair *__restrict__ pairs, const OperandView *__restrict__ views_in,
               const int4 *__restrict__ tasks, const double *__restrict__ A, const double *__restrict__ B,
               int *__restrict__ F, uint8_t *__restrict__ arena, int b) {
  const OperandView *views = VIEWS ? views_in : nullptr;
  const int4 tk = tasks[blockIdx.x];
  if constexpr (HP) {  // FP64-grade launches: always 8-bit digits
    strip_b<CPLX, S, 8, true>(pairs, views, tk, A, B, F, arena);
  } else {
    switch (b) {  // the host admits b = 5..8 only
      case 5: strip_b<CPLX, S, 5, false>(pairs, views, tk, A, B, F, arena); break;
      case 6: strip_b<CPLX, S, 6, false>(pairs, views, tk, A, B, F, arena); break;
      case 7: strip_b<CPLX, S, 7, false>(pairs, views, tk, A, B, F, arena); break;
      default: strip_b<CPLX, S, 8, false>(pairs, views, tk, A, B, F, arena); break;
    }
  }
}

// ------------------------------------------------------- PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// One lane of a converged warp.  A branch on elect.sync tells the compiler that
// a single thread runs it: operands of tcgen05.mma, commits and bulk copies then
// reach the uniform registers directly (12 clocks an instruction; 46 behind a
// branch on the lane number, where they go through a loop over active lanes).
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: returns false (and raises the CTA abort flag and the global
// error word) when the barrier phase did not complete in time, or when
// another role already aborted.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag,
                                          int *err, int code) {
  for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  atomicExch(err, code);
  return false;
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// SWIZZLE_NONE K-major shared-memory matrix descriptor: start address, LBO =
// byte distance between core matrices adjacent in K, SBO = between core
// matrices adjacent in M/N, descriptor version 1 (bits 46-47).
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}
// kind::f16 instruction descriptor: D=F32, A=B=FP16, both K-major, N, M=128.
__host__ __device__ constexpr uint32_t make_idesc(int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TMS >> 4) << 24);
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Recombination.  The S accumulators hold exact
// integers (|acc_g| <= 2^24); their weighted sum
//   V = sum_g acc_g 2^(b(S-1-g) - r)
// is formed in 64-bit fixed point (r low bits of the smallest groups are
// rounded away so that V and the sum over accumulator chunks keep headroom),
// then turned into an FP64 value V * 2^scale (fixed_to_double).
// Wrapping 32 x 32 -> 64-bit multiply-add: acc + (int64)a * m (mod 2^64).
__device__ __forceinline__ unsigned long long mad_wide(int a, int m, unsigned long long acc) {
  unsigned long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(m), "l"(acc));
  return d;
}

// How accumulator group g enters the fixed-point sum V = sum_g acc_g 2^sh_g
// (sh_g = b(S-1-g) - r): sh >= 32 adds acc * 2^(sh-32) to the high 32-bit
// word, 0 <= sh <= 30 adds acc * 2^sh to the low 64-bit word, sh < 0 adds
// acc / 2^-sh rounded.  All words wrap; V itself fits in int64, so
// V = hi * 2^32 + lo (mod 2^64) is exact.

// V * 2^scale by one int64 -> FP64 conversion (round to nearest even) and an
// exponent add; `rare` is raised where that does not hold (the result is no
// normal number) and fixed_to_double_rare has to be taken.  No branch: a
// thread's eight outputs overlap (one after the other, each with its own
// branches and its own reads of the tile's descriptor, took 4400 clocks a tile).
__device__ __forceinline__ double fixed_to_double(long long V, int scale, bool &rare) {
  const double d = __ll2double_rn(V);
  const int hi = __double2hiint(d), e = (hi >> 20 & 0x7ff) + scale;
  rare |= V != 0 && (unsigned)(e - 1) >= 2046u;
  return __hiloint2double(V != 0 ? hi + (int)((unsigned)scale << 20) : 0, __double2loint(d));
}
__device__ __noinline__ double fixed_to_double_rare(long long V, int scale) { return ldexp(__ll2double_rn(V), scale); }
// Folds accumulator groups G0..G0+NG-1 of one set (this thread's TMEM lane,
// 8 columns from cbase) into the fixed-point words: group g enters with shift
// sh = b(S-1-g) - rsh, >= 32 into the high word Vh, 0..30 into the low word
// Vl (the host keeps sh off 31), < 0 rounded down by -sh bits; exactly one
// form applies to a group (uniform branch).
template <int S, int G0, int NG>
__device__ __forceinline__ void fold_groups(uint32_t set_base, int cbase, int b, int rsh,
                                            unsigned long long (&Vl)[8], unsigned int (&Vh)[8]) {
  float acc[NG][8];
#pragma unroll
  for (int g = 0; g < NG; ++g) tmem_ld8(set_base + (uint32_t)((G0 + g) * TNS + cbase), acc[g]);
  tmem_wait_ld();
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    const int sh = b * (S - 1 - (G0 + g)) - rsh;
    if (sh >= 32) {
      const unsigned m = 1u << (sh - 32);
#pragma unroll
      for (int c = 0; c < 8; ++c) Vh[c] += (unsigned int)__float2int_rn(acc[g][c]) * m;
    } else if (sh >= 0) {
#pragma unroll
      for (int c = 0; c < 8; ++c) Vl[c] = mad_wide(__float2int_rn(acc[g][c]), 1 << sh, Vl[c]);
    } else {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int a = __float2int_rn(acc[g][c]);
        Vl[c] = mad_wide((a + (1 << (-sh - 1))) >> -sh, 1, Vl[c]);
      }
    }
  }
}

// Smallest certificate of an output, sum_k m_ik m_kj in units of
// 2^(E_i+F_j-16) with m = max(|d_0| - 1/2, 0) (lower_magnitudes).  It is a lower
// bound of sum_k |a_ik b_kj| up to 0.8 % (m's 0.4 % twice; the FP32 sums add
// 2^-10 at most).  What a term loses: 2^-57 of full scale per entry's rounding
// and 6 2^-58 (a little more) for the digit products left out, together
// 10.02 2^-58 2^(E_i+F_j).  A sum of at least a third of full scale keeps K terms
// of that below 0.95 K u sum_k |a_ik b_kj|, u = 2^-53: the bound of an FP64 dot
// product, K u of the same sum.  (The rounded magnitudes |d_0| with a sixteenth
// of full scale had left 17 K u: |d_0| doubles an entry just above half a unit.)
// Against sequential FP64 sums, root mean square error over outputs that pass,
// in u sum |ab|: normal entries 0.16 to 0.47 at K = 32 and 0.03 to 0.48 at 1024;
// log-normal (sigma 2) 0.37 to 1.3 at 32, 1.1 to 8.8 at 1024 (with a sixteenth:
// 1.7 to 1.5 at 64, 16 to 9 at 4096); one dominant term 2.2 to 27 at 4096.
constexpr float CERT_MIN = 65536.0f / 3.0f;

// FP64-grade fold (S digits, two 64-bit words): the groups 0..HG-1 into Vh
// with weights 2^(b(HG-1-g)), the others into Vl with 2^(b(S-1-g)), so that
// V = Vh 2^(b(S-HG)) + Vl exactly (no bit of any group is dropped; the words
// hold 25 + b(HG-1) resp. 25 + b(S-HG-1) bits and the chunk count's).  The
// certificate group S (products of the leading digits' magnitudes) is summed
// in FP32: it is compared with a threshold only.
constexpr int HG = 4;
template <int S, int G0, int NG>
__device__ __forceinline__ void fold_groups_hp(uint32_t set_base, int cbase, int b, unsigned long long (&Vl)[8],
                                               unsigned long long (&Vh)[8], float (&cert)[8]) {
  float acc[NG][8];
#pragma unroll
  for (int g = 0; g < NG; ++g) tmem_ld8(set_base + (uint32_t)((G0 + g) * TNS + cbase), acc[g]);
  tmem_wait_ld();
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    const int gg = G0 + g;
    if (gg == S) {
#pragma unroll
      for (int c = 0; c < 8; ++c) cert[c] += acc[g][c];
    } else if (gg < HG) {
      const int m = 1 << (b * (HG - 1 - gg));
#pragma unroll
      for (int c = 0; c < 8; ++c) Vh[c] = mad_wide(__float2int_rn(acc[g][c]), m, Vh[c]);
    } else {
      const int m = 1 << (b * (S - 1 - gg));
#pragma unroll
      for (int c = 0; c < 8; ++c) Vl[c] = mad_wide(__float2int_rn(acc[g][c]), m, Vl[c]);
    }
  }
}

// (Vh 2^lb + Vl) 2^scale rounded once to FP64: the sum is normalised into 62
// bits with a sticky bit below (24 <= lb <= 31).
__device__ __forceinline__ double wide_to_double(long long Vh, long long Vl, int lb, int scale) {
  const long long T = Vh + (Vl >> lb);                       // floor of the sum / 2^lb
  const unsigned long long rem = (unsigned long long)Vl & ((1ull << lb) - 1);
  const int room = __clzll(T < 0 ? ~T : T) - 2;              // left shifts that keep a spare bit
  const int k = min(max(room, 0), lb);
  long long V = (long long)((unsigned long long)T << k) | (long long)(rem >> (lb - k));
  if (rem & ((1ull << (lb - k)) - 1)) V |= 1;                // sticky
  bool rare = false;
  const double d = fixed_to_double(V, scale + lb - k, rare);
  return rare ? fixed_to_double_rare(V, scale + lb - k) : d;
}

// Chunking rule shared by the host and the MMA issuer: a new chunk starts
// when adding the next K block would push the summed (real) depth of the
// current chunk above kchunk.
__device__ __forceinline__ int kblock_depth(int Kr, int kb) { return min(TKS, Kr - kb * TKS); }

// ------------------------------------------------------------ GEMM kernel
// Persistent: one CTA per SM walks tiles r*G + c (snake order over the
// depth-sorted tile list so every CTA gets a similar mix).  The three roles
// step through the same sequence; the TMA ring and the accumulator hand-off
// run continuously across tile boundaries.  TMEM holds two accumulator sets
// (S groups x 32 columns each): the epilogue drains one while the MMA issuer
// fills the other.
__device__ __forceinline__ int tile_of(int r, int c, int G) { return r * G + ((r & 1) ? (G - 1 - c) : c); }

//
// HP: the FP64-grade launch of the plain path (see f64_tensor_takes): S
// digits plus one plane of the leading digits' magnitudes (lower_magnitudes)
// per operand, whose product (accumulator group S) bounds sum_k |a_ik b_kj|
// from below.  An
// output whose bound is too small for the digits' truncation to stay at the
// level of an FP64 sum, or whose row or column holds an infinity or NaN,
// has its FP64 cell listed (MissList), which the FP64 kernel then computes.
template <int S, bool HP>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_split_kernel(const SplitTile *__restrict__ tiles, int ntiles, const SplitPair *__restrict__ pairs,
                  const uint8_t *__restrict__ arena, const int *__restrict__ E,
                  const int *__restrict__ F, double *__restrict__ C, int b, int nstages,
                  int kchunk, int *err, MissList miss) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t *full = reinterpret_cast<uint64_t *>(smem);       // [MAX_STAGES]
  uint64_t *empty = full + MAX_STAGES;                        // [MAX_STAGES]
  uint64_t *acc_full = full + 2 * MAX_STAGES;                 // [2]
  uint64_t *acc_empty = acc_full + 2;                         // [2]
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + 512);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + 516);
  uint8_t *stages = smem + SMEM_HDR;
  constexpr int NP = S + (HP ? 1 : 0);
  constexpr uint32_t A_BYTES = NP * A_DIGIT_BYTES, B_BYTES = NP * B_DIGIT_BYTES;
  constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr uint32_t SET_COLS = NP * TNS;  // columns of one accumulator set
  constexpr uint32_t NCOLS = (2 * SET_COLS <= 256) ? 256 : 512;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = gridDim.x, cta = blockIdx.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < nstages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], EPI_WARPS);  // one arrive per epilogue warp
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(NCOLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      // ------------------------------------------------ TMA producer
      int it = 0, st = 0;  // stage it % nstages, its phase bit ph
      uint32_t ph = 0;
      bool ok = true;
      for (int r = 0; ok; ++r) {
        const int ti = tile_of(r, cta, G);
        if (ti >= ntiles) break;
        const SplitTile &T = tiles[ti];
        for (int p = T.p0; p < T.p1 && ok; ++p) {
          const SplitPair &P = pairs[p];
          const int KB = P.KB;
          const uint8_t *a_src = arena + P.as_off + (int64_t)T.mt * KB * A_BYTES;
          const uint8_t *b_src = arena + P.bs_off + (int64_t)T.nt * KB * B_BYTES;
          for (int kb = 0; kb < KB; ++kb, ++it) {
            if (!mbar_wait(&empty[st], ph ^ 1u, abort_flag, err, 1)) { ok = false; break; }
            uint8_t *sa = stages + (size_t)st * STAGE_BYTES;
            mbar_expect_tx(&full[st], STAGE_BYTES);
            bulk_g2s(sa, a_src + (int64_t)kb * A_BYTES, A_BYTES, &full[st]);
            bulk_g2s(sa + A_BYTES, b_src + (int64_t)kb * B_BYTES, B_BYTES, &full[st]);
            if (++st == nstages) {
              st = 0;
              ph ^= 1u;
            }
          }
        }
      }
      // Wait (bounded) until every stage issued has landed, so that no bulk
      // copy is still writing shared memory when the CTA exits.
      const int issued = it;
      for (int j = max(0, issued - nstages); j < issued; ++j) {
        const int st = j % nstages;
        const uint32_t ph = (uint32_t)((j / nstages) & 1);
        for (uint32_t i = 0; i < WAIT_LIMIT && !mbar_try_wait(&full[st], ph); ++i) {
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // ------------------------------------------------ MMA issuer
      // one instruction per A digit t: N = (S - t) * 32 columns of B digits
      uint32_t idesc[S];
#pragma unroll
      for (int j = 0; j < S; ++j) idesc[j] = make_idesc(TNS * (j + 1));
      int it = 0, u = 0;  // u: accumulator uses (chunks) handed to the epilogue
      int st = 0;         // stage it % nstages, its phase bit ph
      uint32_t ph = 0;
      // shared-memory descriptors of stage 0; stage st adds st * STAGE_BYTES
      // to the start address field (addresses stay below 2^18, so the 14-bit
      // field never carries)
      const uint64_t desc0 = make_desc(smem_u32(stages), 128, KCM * 128);
      bool ok = true;
      // before filling set u & 1 for use u >= 2, wait until use u - 2 is read
      auto acquire = [&](int uu) -> bool {
        if (uu >= 2) {
          if (!mbar_wait(&acc_empty[uu & 1], (uint32_t)(((uu >> 1) - 1) & 1), abort_flag, err, 2)) return false;
          tc_fence_after();
        }
        return true;
      };
      for (int r = 0; ok; ++r) {
        const int ti = tile_of(r, cta, G);
        if (ti >= ntiles) break;
        const SplitTile &T = tiles[ti];
        int depth = 0;
        bool fresh = true;
        if (!acquire(u)) { ok = false; break; }
        // the sizes of the next pair are loaded one pair ahead, so that the
        // global-load latency stays off the issue path
        const int p1 = T.p1;
        int KBn = pairs[T.p0].KB, Krn = pairs[T.p0].Kr;
        for (int p = T.p0; p < p1 && ok; ++p) {
          const int KB = KBn, Kr = Krn;
          if (p + 1 < p1) {
            KBn = pairs[p + 1].KB;
            Krn = pairs[p + 1].Kr;
          }
          for (int kb = 0; kb < KB; ++kb, ++it) {
            const int dk = max(kblock_depth(Kr, kb), 0);
            if (!fresh && depth + dk > kchunk) {
              // this chunk is done: hand the set to the epilogue, go on in
              // the other set
              umma_commit(&acc_full[u & 1]);
              ++u;
              if (!acquire(u)) { ok = false; break; }
              fresh = true;
              depth = 0;
            }
            depth += dk;
            if (!mbar_wait(&full[st], ph, abort_flag, err, 3)) { ok = false; break; }
            tc_fence_after();
            const uint64_t dst0 = desc0 + (uint64_t)((st * STAGE_BYTES) >> 4);
            const uint32_t dset = tmem + (uint32_t)((u & 1) * SET_COLS);
            // digit t of K step ks: N = (S - t) * 32 columns
            auto digit = [&](int t, int ks) {
              const uint64_t ad = dst0 + (uint64_t)((t * A_DIGIT_BYTES + ks * 256) >> 4);
              const uint64_t bd = dst0 + (uint64_t)((A_BYTES + ks * 256) >> 4);
              umma_f16(dset + (uint32_t)(t * TNS), ad, bd, idesc[S - 1 - t], (fresh && ks == 0 && t == 0) ? 0u : 1u);
            };
            auto magnitude = [&](int ks) {
              const uint64_t ad = dst0 + (uint64_t)((S * A_DIGIT_BYTES + ks * 256) >> 4);
              const uint64_t bd = dst0 + (uint64_t)((A_BYTES + S * B_DIGIT_BYTES + ks * 256) >> 4);
              umma_f16(dset + (uint32_t)(S * TNS), ad, bd, idesc[0], (fresh && ks == 0) ? 0u : 1u);
            };
            // The tensor core takes four instructions ahead: with the long
            // products last they outlast the commit and the wait for the next
            // stage (a stage's products run in 0.91 of the time of t = 0..S-1
            // twice, at S = 6 with nothing else on the SM).
#pragma unroll
            for (int t = 0; t < S; ++t) digit(t, 0);
            if constexpr (HP) {
              magnitude(0);
              magnitude(1);
            }
#pragma unroll
            for (int t = S - 1; t >= 0; --t) digit(t, 1);
            fresh = false;
            umma_commit(&empty[st]);
            if (++st == nstages) {
              st = 0;
              ph ^= 1u;
            }
          }
        }
        if (!ok) break;
        umma_commit(&acc_full[u & 1]);
        ++u;
      }
      // every MMA must have completed before TMEM is released: wait until the
      // epilogue has read the last two uses
      if (ok) {
        for (int uu = max(0, u - 2); uu < u; ++uu)
          mbar_wait(&acc_empty[uu & 1], (uint32_t)((uu >> 1) & 1), abort_flag, err, 4);
      } else {
        umma_commit(&acc_full[u & 1]);
        for (uint32_t i = 0; i < WAIT_LIMIT && !mbar_try_wait(&acc_full[u & 1], (uint32_t)((u >> 1) & 1)); ++i) {
        }
      }
    }
  } else {
    // ------------------------------------------- epilogue (warps 2..)
    // warp w reads TMEM lane quarter w % 4; each run of four warps covers
    // all quarters for CW consecutive columns of the tile.
    const int q = warp & 3;
    constexpr int CW = TNS * 4 / EPI_WARPS;
    static_assert(CW == 8, "the drain reads 8 columns per thread and group");
    const int cbase = ((warp - 2) >> 2) * CW;
    const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
    const int scale_b = -b * (S + 1);
    int u = 0;
    bool ok = true;
    // The next tile's descriptor is fetched one tile ahead (one word per
    // lane) and handed over through this warp's shared-memory slot, so that
    // its global-load latency hides behind the current tile: short tiles are
    // bound by the epilogue.
    uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + TILE_SLOTS + (warp - 2) * 64);
    int ti = tile_of(0, cta, G);
    uint32_t tw = (ti < ntiles && lane < TILE_WORDS) ? reinterpret_cast<const uint32_t *>(tiles + ti)[lane] : 0u;
    for (int r = 0; ok; ++r) {
      if (ti >= ntiles) break;
      __syncwarp();  // every lane is done with the previous descriptor
      if (lane < TILE_WORDS) tslot[lane] = tw;
      __syncwarp();
      // fields are read from the slot where used (no registers held)
      const SplitTile &T = *reinterpret_cast<const SplitTile *>(tslot);
      ti = tile_of(r + 1, cta, G);
      tw = (ti < ntiles && lane < TILE_WORDS) ? reinterpret_cast<const uint32_t *>(tiles + ti)[lane] : 0u;
      const int i_glob = T.mt * TMS + q * 32 + lane;
      const bool rv = i_glob < T.Mr;
      // the row's exponent and, one per lane, those of the warp's columns are
      // fetched now, so that their latency hides behind the accumulation
      const int j0 = T.nt * TNS + cbase;
      const int Ei = rv ? E[T.eoff + i_glob] : 0;
      int Fl = 0;
      if constexpr (!HP) Fl = lane < CW && j0 + lane < T.N ? F[T.foff + j0 + lane] : 0;
      const int rsh = T.rshift;
      unsigned long long Vl[CW];
      std::conditional_t<HP, unsigned long long, unsigned int> Vh[CW];
      float cert[CW];
#pragma unroll
      for (int jj = 0; jj < CW; ++jj) {
        Vl[jj] = 0;
        Vh[jj] = 0;
        cert[jj] = 0.0f;
      }
      for (int ch = 0; ch < T.nchunk; ++ch, ++u) {
        // one lane polls; the warp proceeds together (tcgen05.ld is .aligned)
        int w = 1;
        if (lane == 0) w = mbar_wait(&acc_full[u & 1], (uint32_t)((u >> 1) & 1), abort_flag, err, 5) ? 1 : 0;
        w = __shfl_sync(0xffffffffu, w, 0);
        if (!w) { ok = false; break; }
        tc_fence_after();
        const uint32_t set_base = lane_base + (uint32_t)((u & 1) * SET_COLS);
        // the groups' columns are in flight together (one wait per batch of up
        // to six): the drain is bound by TMEM load latency otherwise
        if constexpr (HP) {
          fold_groups_hp<S, 0, 4>(set_base, cbase, b, Vl, Vh, cert);
          fold_groups_hp<S, 4, NP - 4>(set_base, cbase, b, Vl, Vh, cert);
        } else if constexpr (S <= 6) {
          fold_groups<S, 0, S>(set_base, cbase, b, rsh, Vl, Vh);
        } else {
          fold_groups<S, 0, 4>(set_base, cbase, b, rsh, Vl, Vh);
          fold_groups<S, 4, S - 4>(set_base, cbase, b, rsh, Vl, Vh);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[u & 1]);
      }
      if (!ok) break;
      if constexpr (HP) {
        bool out = false;  // an output misses the certificate
        if (rv) {
          const int rsplit = T.splits & 1, csplit = (T.splits >> 1) & 1;
          double *crow = C + T.c_off + (int64_t)(i_glob >> rsplit) * T.rs + (i_glob & rsplit);
#pragma unroll
          for (int jj = 0; jj < CW; ++jj) {
            const int j = j0 + jj;
            if (j >= T.N) continue;
            const int Fj = F[T.foff + j];
            crow[(int64_t)(j >> csplit) * T.ldc + (j & csplit)] =
                wide_to_double((long long)Vh[jj], (long long)Vl[jj], b * (S - HG), Ei + Fj + scale_b);
            // a row or column of zeros (EMPTY_EXP) is exact
            out |= max(Ei, Fj) >= NONFINITE_EXP || (min(Ei, Fj) > EMPTY_EXP && cert[jj] < CERT_MIN);
          }
        }
        if (__any_sync(0xffffffffu, out)) {
          // a thread's eight columns lie in one cell; one lane per cell lists it
          static_assert(F64_CELL % CW == 0, "columns of a thread in one cell");
          const int rdup = (T.splits >> 3) & 1, cdup = (T.splits >> 4) & 1;
          const bool sw = T.splits & 4;
          const int rows = sw ? T.N >> cdup : T.Mr >> rdup;  // of C
          const int r = sw ? j0 >> cdup : i_glob >> rdup, c = sw ? i_glob >> rdup : j0 >> cdup;
          const int tile = T.fbase + r / F64_TILE + c / F64_TILE * ((rows + F64_TILE - 1) / F64_TILE);
          const int cell = (r / F64_CELL & 1) | (c / F64_CELL & 1) << 1;
          const unsigned same = __match_any_sync(0xffffffffu, out ? tile * 4 + cell : -1);
          if (out && lane == __ffs(same) - 1) miss.add(tile, cell);
        }
      } else {
        // the eight outputs side by side, then their stores (1024 x 1024 blocks
        // of depth 128: 508 -> 422 us)
        double v[CW];
        bool rare = false;
        const int sc0 = Ei + scale_b + rsh;
#pragma unroll
        for (int jj = 0; jj < CW; ++jj) {
          const int Fj = __shfl_sync(0xffffffffu, Fl, jj);
          v[jj] = fixed_to_double((long long)(((unsigned long long)Vh[jj] << 32) + Vl[jj]), sc0 + Fj, rare);
        }
        const int splits = T.splits, rsplit = splits & 1, csplit = (splits >> 1) & 1, N = T.N;
        const int64_t ldc = T.ldc;
        double *crow = C + T.c_off + (int64_t)(i_glob >> rsplit) * T.rs + (i_glob & rsplit);
        if (rare) {
#pragma unroll
          for (int jj = 0; jj < CW; ++jj)
            v[jj] = fixed_to_double_rare((long long)(((unsigned long long)Vh[jj] << 32) + Vl[jj]),
                                         sc0 + F[T.foff + min(j0 + jj, N - 1)]);
        }
#pragma unroll
        for (int jj = 0; jj < CW; ++jj) {
          const int j = j0 + jj;
          if (rv && j < N) crow[(j >> csplit) * ldc + (j & csplit)] = v[jj];
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOLS) : "memory");
  }
}

template <int NP>
size_t smem_bytes(int nstages) {
  return SMEM_HDR + (size_t)nstages * NP * (A_DIGIT_BYTES + B_DIGIT_BYTES);
}

template <int NP>
int pick_stages() {
  const size_t per = (size_t)NP * (A_DIGIT_BYTES + B_DIGIT_BYTES);
  int n = (int)((SMEM_LIMIT - SMEM_HDR) / per);
  return std::max(1, std::min(n, MAX_STAGES));
}

template <int S, bool HP>
void launch_split_s(Ctx *ctx, bool cplx, const SplitPair *d_pairs, const OperandView *d_va, const OperandView *d_vb,
                    const int4 *d_sa, int nsa, const int4 *d_sb, int nsb, const SplitTile *d_tiles, int ntiles,
                    const double *A, const double *B, double *C, int *dE, int *dF, uint8_t *arena, int b,
                    int kchunk, int *err, bool may_fork, const MissList &miss, bool marks) {
  if (b < 5 || b > 8 || b * S > 62 || (HP && (b != 8 || d_va || d_vb))) fail(QS_ERR_INTERNAL, "split: unsupported digit plan b=%d S=%d", b, S);
  cudaStream_t st = ctx->stream;
  if (marks) ctx->mark(0);
  // the two roles' strips are independent: the B role runs on the
  // context's second stream beside the A role, so that neither launch's
  // last partial wave leaves SMs idle; the GEMM waits for both (not on the
  // allocation-free path, which creates no stream)
  const bool fork = may_fork && nsa && nsb;
  cudaStream_t sb = st;
  if (fork) {
    ctx->ensure_aux();
    QS_CUDA(cudaEventRecord(ctx->aux_fork, st));
    QS_CUDA(cudaStreamWaitEvent(ctx->aux, ctx->aux_fork, 0));
    sb = ctx->aux;
  }
  auto strips = [&](auto cx) {
    constexpr bool CX = decltype(cx)::value;
    if (nsb) {
      if (!HP && d_vb)
        strip_b_kernel<CX, S, !HP, HP><<<nsb, STRIP_THREADS, 0, sb>>>(d_pairs, d_vb, d_sb, A, B, dF, arena, b);
      else
        strip_b_kernel<CX, S, false, HP><<<nsb, STRIP_THREADS, 0, sb>>>(d_pairs, nullptr, d_sb, A, B, dF, arena, b);
      QS_LAUNCHED(ctx);
    }
    if (nsa) {
      if (!HP && d_va)
        strip_a_kernel<CX, S, !HP, HP><<<nsa, STRIP_THREADS, 0, st>>>(d_pairs, d_va, d_sa, A, B, dE, arena, b);
      else
        strip_a_kernel<CX, S, false, HP><<<nsa, STRIP_THREADS, 0, st>>>(d_pairs, nullptr, d_sa, A, B, dE, arena, b);
      QS_LAUNCHED(ctx);
    }
  };
  if (cplx) strips(std::true_type{});
  else strips(std::false_type{});
  if (fork) {
    QS_CUDA(cudaEventRecord(ctx->aux_join, ctx->aux));
    QS_CUDA(cudaStreamWaitEvent(st, ctx->aux_join, 0));
  }
  constexpr int NP = S + (HP ? 1 : 0);
  const int nst = pick_stages<NP>();
  const size_t sm = smem_bytes<NP>(nst);
  QS_CUDA(cudaFuncSetAttribute(gemm_split_kernel<S, HP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  if (marks) ctx->mark(1);
  const int grid = std::min(ntiles, std::max(ctx->num_sms, 1));
  gemm_split_kernel<S, HP><<<grid, GEMM_THREADS, sm, st>>>(d_tiles, ntiles, d_pairs, arena, dE, dF, C, b, nst, kchunk,
                                                           err, miss);
  QS_LAUNCHED(ctx);
  if (marks) ctx->mark(2);
}

}  // namespace


// ---------------------------------------------------------------- host side
// Largest summed (real) depth that keeps every accumulator group exact:
// |sum_{t+u=g} d_t d'_u| <= 2^(2b) (1 + max(0, g-1)/4) per term.
static int kchunk_of(int b, int S) {
  const double grow = std::max(1.0, 1.0 + (S - 2) / 4.0);
  const double kc = std::floor(16777216.0 / (std::ldexp(1.0, 2 * b) * grow));
  return (int)std::min(kc, 1.0e9);
}

// Accumulator drains of one output block: a new chunk starts when the next K
// block would push the chunk's summed depth above kchunk (the MMA issuer
// applies the same rule).
// (counted per pair, not per K block: a reduced density matrix over a large
// bond sums 10^5 blocks, which took 0.6 ms of a call)
static int chunks_of(const std::vector<PairDesc> &pairs, int64_t p0, int64_t p1, int cm, int kchunk) {
  const int64_t per = std::max(1, kchunk / TKS);  // whole K blocks of a chunk
  int64_t nchunk = 1, depth = 0;
  bool fresh = true;
  for (int64_t p = p0; p < p1; ++p) {
    const int64_t Kr = std::max<int64_t>((int64_t)pairs[p].K * cm, 0);
    int64_t whole = Kr / TKS;
    const int64_t tail = Kr % TKS;
    if (whole > 0) {
      const int64_t room = fresh ? per : std::max<int64_t>(0, (kchunk - depth) / TKS);
      if (whole <= room) {
        depth += whole * TKS;
      } else {
        whole -= room;
        nchunk += (whole + per - 1) / per;
        depth = ((whole - 1) % per + 1) * TKS;
      }
      fresh = false;
    }
    if (tail > 0 || Kr == 0) {
      if (!fresh && depth + tail > kchunk) {
        ++nchunk;
        depth = 0;
      }
      depth += tail;
      fresh = false;
    }
  }
  return (int)nchunk;
}

// Digit plan: the (bits, digits) pair that reaches the wanted precision at
// the lowest modelled cost over the actual tiles -- tensor work grows as
// S(S+1)/2 per K block, and each accumulator drain costs about as much as
// DRAIN_UNITS single-digit K blocks (small: with two accumulator sets the
// drain overlaps the next chunk's products).  QS_SPLIT_DRAIN_UNITS and
// QS_SPLIT_BITS override the model for tuning.
static double drain_units() {
  const char *e = std::getenv("QS_SPLIT_DRAIN_UNITS");
  return e ? std::atof(e) : 12.0;
}

DigitPlan choose_digits_for(const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                            const std::vector<int32_t> &blk_M, const std::vector<int32_t> &blk_N, int cm,
                            double tol, int forced_slices, int forced_bits) {
  if (!(tol > 0)) tol = 1e-12;
  // bits of precision wanted: the tolerance plus a margin for the growth of
  // the error with the summed depth relative to |C|.
  const int need = (int)std::ceil(-std::log2(tol)) + 8;
  DigitPlan best{0, 0, 0};
  double best_cost = 1e300;
  const int64_t nb = (int64_t)blk_M.size();
  const double DRAIN_UNITS = drain_units();
  const char *fb = std::getenv("QS_SPLIT_BITS");
  int bhi = fb ? std::atoi(fb) : 8, blo = fb ? std::atoi(fb) : 5;
  if (forced_bits > 0) bhi = blo = forced_bits;
  for (int b = bhi; b >= blo; --b) {
    int S = forced_slices > 0 ? forced_slices : (need - 1 + b - 1) / b;
    S = std::max(S, 2);
    if (S > 8 || b * S > 62) continue;
    const int kchunk = kchunk_of(b, S);
    if (kchunk < TKS) continue;
    double cost = 0;
    for (int64_t g = 0; g < nb; ++g) {
      const double tiles = double((blk_M[g] * cm + TMS - 1) / TMS) * double((blk_N[g] + TNS - 1) / TNS);
      double kbs = 0;
      for (int64_t p = grp[g]; p < grp[g + 1]; ++p) kbs += std::max(1, (pairs[p].K * cm + TKS - 1) / TKS);
      cost += tiles * (S * (S + 1) / 2.0 * kbs + DRAIN_UNITS * chunks_of(pairs, grp[g], grp[g + 1], cm, kchunk));
    }
    if (cost < best_cost) {
      best_cost = cost;
      best.bits = b;
      best.nslices = S;
      best.err_bound = (S + 2) * std::ldexp(1.0, -b * S);
    }
  }
  if (!best.nslices) fail(QS_ERR_NUMERIC, "no digit plan for tol=%g, slices=%d", tol, forced_slices);
  return best;
}

// Digits of the FP64-grade launches: 7 x 8 bits and the magnitude plane fill
// the two accumulator sets of TMEM (8 groups x 32 columns x 2).
constexpr int HP_BITS = 8, HP_DIGITS = 7;

// Host-side work lists of one planned split product.
struct SplitWork {
  int S = 0, b = 0, kchunk = 0;
  bool hp = false;  // FP64-grade: one more plane per operand, misses listed
  int64_t nE = 0, nF = 0, arena = 0;
  std::vector<SplitPair> sp;
  // strips of STRIP real lines: (first pair, end pair, first line, 0) of the
  // A role (rows of op(A~)) and of the B role (columns of op(B~))
  std::vector<int4> sa, sb;
  std::vector<SplitTile> tiles;
  // strided views of the A and B roles per pair (empty: none)
  std::vector<OperandView> va, vb;
};

// Their device copies, the exponent arrays and the digit arena.
struct SplitDev {
  SplitPair *pairs = nullptr;
  int4 *sa = nullptr, *sb = nullptr;
  SplitTile *tiles = nullptr;
  OperandView *va = nullptr, *vb = nullptr;
  int *E = nullptr, *F = nullptr;
  uint8_t *arena = nullptr;
  MissList miss;  // FP64-grade
};

// Host half of the split path: digit plan, per-pair digit geometry and arena
// offsets, and the device work lists (exponent lines, slicing tiles, output
// tiles in launch order).
// Layout of each output block: computed as C or as C^T = op(B)^T op(A)^T,
// and for complex blocks with the real form duplicating A (A~ is 2M x 2K) or
// B (B' is 2K x 2N; see SplitPair), whichever is estimated cheapest (a layout
// other than the plain one must be at least 3 % cheaper).  The estimate per
// k-block of the block's pairs, in bytes of slicing traffic: 26900 per
// 128 x 32 output tile (GEMM), plus the digit bytes the slicing writes for
// the A role (128-row tiles, 48 KB at six digits) and for the B role
// (32-column tiles, 12 KB, weighted 0.86) -- fitted to GB300 timings of the
// split GEMM (5.65 ns per tile and k-block) and of the slicing kernels (0.21
// and 0.18 ps per byte).  A swapped pair exchanges the roles and storage of
// its operands: A' = op(B)^T reads B's storage (transposed unless op(B) was),
// B' = op(A)^T reads A's, with the conjugation flags exchanged; the tiles
// store C^T transposed.  Returns per block bit 0 = swapped, bit 1 = B
// duplicated.
static std::vector<uint8_t> orient_blocks(const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                                          std::vector<int32_t> &bM, std::vector<int32_t> &bN, int cm,
                                          std::vector<PairDesc> &tp) {
  const int64_t nb = (int64_t)bM.size();
  std::vector<uint8_t> mode(nb, 0);
  bool any = false;
  // rows of the A role and columns of the B role, real form
  auto cost = [&](int64_t rows, int64_t cols) {
    const double mt = double((rows + TMS - 1) / TMS), nt = double((cols + TNS - 1) / TNS);
    return 26900.0 * mt * nt + 49152.0 * mt + 10530.0 * nt;
  };
  for (int64_t g = 0; g < nb; ++g) {
    const int64_t m = bM[g], n = bN[g];
    double c[4] = {cost(m * cm, n), cost(n * cm, m), 1e300, 1e300};
    if (cm == 2) {
      c[2] = cost(m, 2 * n);
      c[3] = cost(n, 2 * m);
    }
    int best = 0;
    for (int o = 1; o < 4; ++o)
      if (c[o] < c[best]) best = o;
    if (c[best] >= 0.97 * c[0]) best = 0;
    // bit 0: swapped (layouts 1 and 3), bit 1: B duplicated (layouts 2 and 3)
    mode[g] = (uint8_t)(((best & 1) ? 1 : 0) | (best >= 2 ? 2 : 0));
    if (mode[g] & 1) any = true;
  }
  if (!any) return mode;
  tp = pairs;
  for (int64_t g = 0; g < nb; ++g) {
    if (!(mode[g] & 1)) continue;
    std::swap(bM[g], bN[g]);
    for (int64_t p = grp[g]; p < grp[g + 1]; ++p) {
      PairDesc &d = tp[p];
      const int t = d.trans;
      std::swap(d.M, d.N);
      std::swap(d.a_off, d.b_off);
      std::swap(d.lda, d.ldb);
      d.trans = ((t & 2) ? 0 : 1) | ((t & 1) ? 0 : 2) | ((t & 8) ? 4 : 0) | ((t & 4) ? 8 : 0);
    }
  }
  return mode;
}

static SplitResult plan_split(const std::vector<PairDesc> &pairs_in, const std::vector<int64_t> &grp,
                              const std::vector<int32_t> &blk_M_in, const std::vector<int32_t> &blk_N_in,
                              const std::vector<int64_t> &c_off, bool cplx, int forced_slices, double tol,
                              const std::vector<int32_t> *blk_ldc, SplitWork &w, int forced_bits = 0,
                              const std::vector<OperandView> *va = nullptr,
                              const std::vector<OperandView> *vb = nullptr,
                              const std::vector<int32_t> *fbase = nullptr) {
  SplitResult res;
  const int64_t nb = (int64_t)blk_M_in.size();
  const int cm = cplx ? 2 : 1;
  std::vector<int32_t> blk_M = blk_M_in, blk_N = blk_N_in;
  std::vector<PairDesc> swapped_pairs;
  const std::vector<uint8_t> mode = orient_blocks(pairs_in, grp, blk_M, blk_N, cm, swapped_pairs);
  const std::vector<PairDesc> &pairs = swapped_pairs.empty() ? pairs_in : swapped_pairs;
  // strided operand views follow their operands into the roles: a block
  // computed as C^T reads op(B)^T in the A role and op(A)^T in the B role,
  // whose lines are B's columns resp. A's rows -- the same views, exchanged
  if ((va && !va->empty()) || (vb && !vb->empty())) {
    const OperandView none{};
    w.va.assign(pairs.size(), none);
    w.vb.assign(pairs.size(), none);
    for (int64_t g = 0; g < nb; ++g)
      for (int64_t p = grp[g]; p < grp[g + 1]; ++p) {
        const OperandView x = (va && !va->empty()) ? (*va)[p] : none, y = (vb && !vb->empty()) ? (*vb)[p] : none;
        if (mode[g] & 1) {
          w.va[p] = y;
          w.vb[p] = x;
        } else {
          w.va[p] = x;
          w.vb[p] = y;
        }
      }
    // a role without views runs the strips with the view code compiled out
    auto none_in = [](const std::vector<OperandView> &v) {
      return std::none_of(v.begin(), v.end(), [](const OperandView &x) { return x.nl > 0; });
    };
    if (none_in(w.va)) w.va.clear();
    if (none_in(w.vb)) w.vb.clear();
  }
  w.hp = fbase != nullptr;
  DigitPlan dp = w.hp ? DigitPlan{HP_BITS, HP_DIGITS, (HP_DIGITS + 2) * std::ldexp(1.0, -HP_BITS * HP_DIGITS)}
                      : choose_digits_for(pairs, grp, blk_M, blk_N, cm, tol, forced_slices, forced_bits);
  const int S = dp.nslices, b = dp.bits;
  const int NP = S + (w.hp ? 1 : 0);
  const int kchunk = kchunk_of(b, S);
  w.S = S;
  w.b = b;
  w.kchunk = kchunk;
  res.nslices = S;
  res.bits = b;
  res.err_bound = dp.err_bound;

  // per-pair digit geometry and arena offsets
  std::vector<SplitPair> &sp = w.sp;
  sp.resize(pairs.size());
  std::vector<int64_t> eoff(nb), foff(nb);
  int64_t &nE = w.nE, &nF = w.nF;
  nE = nF = 0;
  // real rows of the A role and real columns of the B role per block
  std::vector<int64_t> rows_r(nb), cols_r(nb);
  for (int64_t g = 0; g < nb; ++g) {
    const bool dupb = mode[g] & 2;
    rows_r[g] = (int64_t)blk_M[g] * (dupb ? 1 : cm);
    cols_r[g] = (int64_t)blk_N[g] * (dupb ? 2 : 1);
    eoff[g] = nE;
    foff[g] = nF;
    nE += rows_r[g];
    nF += cols_r[g];
  }
  if (nE > INT32_MAX || nF > INT32_MAX) fail(QS_ERR_SHAPE, "split: exponent arrays too large");
  int64_t &arena = w.arena;
  arena = 0;
  std::vector<int4> &sa = w.sa, &sb = w.sb;
  std::vector<SplitTile> &tiles = w.tiles;
  std::vector<SplitTile> of_block(nb, SplitTile{});  // a block's tiles, but for their place
  std::vector<int64_t> depth(nb, 0), order(nb);      // in K blocks
  int64_t ntiles = 0;
  for (int64_t g = 0; g < nb; ++g) {
    // every pair's CG factor is folded into its A digits (exact integer
    // product), so the pairs of a block share the accumulators
    for (int64_t p = grp[g]; p < grp[g + 1]; ++p) {
      const PairDesc &d = pairs[p];
      SplitPair &s = sp[p];
      s.a_off = d.a_off;
      s.b_off = d.b_off;
      s.M = d.M;
      s.N = d.N;
      s.K = d.K;
      s.lda = d.lda;
      s.ldb = d.ldb;
      s.trans = d.trans;
      s.dupb = (mode[g] & 2) ? 1 : 0;
      s.Mr = d.M * (s.dupb ? 1 : cm);
      s.Nr = d.N * (s.dupb ? 2 : 1);
      s.Kr = d.K * cm;
      s.MT = (s.Mr + TMS - 1) / TMS;
      s.NT = (s.Nr + TNS - 1) / TNS;
      s.KB = std::max(1, (s.Kr + TKS - 1) / TKS);
      s.eoff = (int32_t)eoff[g];
      s.foff = (int32_t)foff[g];
      const Factor f = make_factor(d.afac);
      s.fm = f.fm;
      s.fe = f.fe;
      s.fneg = f.neg ? 1 : 0;
      s.fac = d.afac;
      int e = 0;
      if (d.afac != 1.0 && d.afac != 0.0) std::frexp(d.afac, &e);
      s.e_afac = e;
      s.swap = mode[g] & 1;
      s.as_off = arena;
      arena += (int64_t)s.MT * s.KB * NP * A_DIGIT_BYTES;
      s.bs_off = arena;
      arena += (int64_t)s.NT * s.KB * NP * B_DIGIT_BYTES;
    }
    // exponent + slicing strips over all pairs of the block
    if (grp[g + 1] > grp[g]) {
      for (int64_t r0 = 0; r0 < rows_r[g]; r0 += STRIP)
        sa.push_back(make_int4((int)grp[g], (int)grp[g + 1], (int)r0, 0));
      for (int64_t c0 = 0; c0 < cols_r[g]; c0 += STRIP)
        sb.push_back(make_int4((int)grp[g], (int)grp[g + 1], (int)c0, 0));
    }
    const int nchunk = chunks_of(pairs, grp[g], grp[g + 1], cm, kchunk);
    // int64 headroom of the fixed-point sum over all chunks:
    // nchunk * 2^(24.2 + b(S-1) - r) < 2^63
    int lg = 0;
    while ((1 << lg) < nchunk) ++lg;
    int rshift = std::max(0, 25 + b * (S - 1) + lg - 63);
    // the epilogue adds each group with a shift of at most 30 into its low
    // 64-bit word or of at least 32 into its high 32-bit word: no group may
    // land exactly on bit 31
    for (int t = 0; t < S; ++t)
      if (b * (S - 1 - t) - rshift == 31) ++rshift;
    SplitTile &t = of_block[g];
    t.c_off = c_off[g] * cm;
    t.p0 = (int32_t)grp[g];
    t.p1 = (int32_t)grp[g + 1];
    t.Mr = (int32_t)rows_r[g];
    t.N = (int32_t)cols_r[g];
    // column stride of C in its elements, in the caller's orientation
    const int64_t ldc0 = blk_ldc ? (*blk_ldc)[g] : std::max(blk_M_in[g], 1);
    if (ldc0 * cm > INT32_MAX) fail(QS_ERR_SHAPE, "split: leading dimension %lld of a complex C", (long long)ldc0);
    const bool swp = mode[g] & 1, dupb = mode[g] & 2;
    if (!swp && !dupb) {
      t.ldc = (int32_t)(ldc0 * cm);
      t.rs = 1;
      t.splits = 0;
    } else if (!dupb && cm == 1) {
      t.ldc = 1;
      t.rs = (int32_t)ldc0;
      t.splits = 0;
    } else if (!dupb) {
      t.ldc = 2;
      t.rs = (int32_t)(2 * ldc0);
      t.splits = 1;
    } else if (!swp) {
      // C' = M x 2N: row m at 2m, column j at (j/2) of C's columns, part j%2
      t.rs = 2;
      t.ldc = (int32_t)(2 * ldc0);
      t.splits = 2;
    } else {
      // C'^T = N x 2M: row n at column n of C, column j = element j of the
      // interleaved (Re, Im) column
      t.rs = (int32_t)(2 * ldc0);
      t.ldc = 1;
      t.splits = 0;
    }
    if (swp) t.splits |= 4;
    if (cm == 2) t.splits |= dupb ? 16 : 8;
    t.fbase = fbase ? (*fbase)[g] : 0;
    t.eoff = (int32_t)eoff[g];
    t.foff = (int32_t)foff[g];
    t.nchunk = nchunk;
    t.rshift = rshift;
    for (int64_t p = grp[g]; p < grp[g + 1]; ++p) depth[g] += sp[p].KB;
    order[g] = g;
    ntiles += ((rows_r[g] + TMS - 1) / TMS) * ((cols_r[g] + TNS - 1) / TNS);
  }
  // Longest tiles first (by their blocks' summed depth, a stable order): the
  // tail of the launch is short.
  std::stable_sort(order.begin(), order.end(), [&](int64_t x, int64_t y) { return depth[x] > depth[y]; });
  tiles.reserve((size_t)ntiles);
  for (int64_t g : order) {
    const int MT = (int)((rows_r[g] + TMS - 1) / TMS), NT = (int)((cols_r[g] + TNS - 1) / TNS);
    SplitTile t = of_block[g];
    for (t.nt = 0; t.nt < NT; ++t.nt)
      for (t.mt = 0; t.mt < MT; ++t.mt) tiles.push_back(t);
  }
  if (tiles.empty()) return res;
  if (tiles.size() > 0x7fffffff || sa.size() > 0x7fffffff || sb.size() > 0x7fffffff)
    fail(QS_ERR_SHAPE, "split: launch too large");
  res.slice_bytes = arena;
  res.ntiles = (int64_t)tiles.size();

  return res;
}

// Device half: launches the exponent, slicing and GEMM kernels of a planned
// split product on the context's stream, with every work list, exponent
// array and the digit arena already on the device.
static void launch_split(Ctx *ctx, const SplitWork &w, bool cplx, const SplitDev &d, const double *A,
                         const double *B, double *C, int *err, bool may_fork = true, bool marks = true) {
  if (w.hp) {
    launch_split_s<HP_DIGITS, true>(ctx, cplx, d.pairs, nullptr, nullptr, d.sa, (int)w.sa.size(), d.sb,
                                    (int)w.sb.size(), d.tiles, (int)w.tiles.size(), A, B, C, d.E, d.F, d.arena, w.b,
                                    w.kchunk, err, may_fork, d.miss, marks);
    return;
  }
  switch (w.S) {
#define QS_CASE(SS)                                                                                      \
  case SS:                                                                                               \
    launch_split_s<SS, false>(ctx, cplx, d.pairs, d.va, d.vb, d.sa, (int)w.sa.size(), d.sb,               \
                              (int)w.sb.size(), d.tiles, (int)w.tiles.size(), A, B, C, d.E, d.F, d.arena, \
                              w.b, w.kchunk, err, may_fork, MissList{}, marks);                          \
    break;
    QS_CASE(2)
    QS_CASE(3)
    QS_CASE(4)
    QS_CASE(5)
    QS_CASE(6)
    QS_CASE(7)
    QS_CASE(8)
#undef QS_CASE
    default:
      fail(QS_ERR_INTERNAL, "split: unsupported digit count %d", w.S);
  }
}

static SplitResult run_split_lists(Ctx *ctx, const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                                   const std::vector<int32_t> &blk_M, const std::vector<int32_t> &blk_N,
                                   const std::vector<int64_t> &c_off, const double *A, const double *B, double *C,
                                   bool cplx, int forced_slices, double tol, const std::vector<int32_t> *blk_ldc,
                                   int forced_bits, const std::vector<OperandView> *va,
                                   const std::vector<OperandView> *vb);

// Sends a planned product's work lists (one staging copy; L keeps them until the
// launches are queued); the arena and the miss list are the caller's.
static SplitDev stage_split_work(Ctx *ctx, const SplitWork &w, DevLists &L) {
  SplitDev d;
  const size_t sp = L.add(w.sp), sa = L.add(w.sa), sb = L.add(w.sb), st = L.add(w.tiles);
  const size_t va = L.add(w.va), vb = L.add(w.vb);
  const size_t se = L.space((size_t)w.nE * sizeof(int)), sf = L.space((size_t)w.nF * sizeof(int));
  L.commit(ctx);
  d.pairs = L.at<SplitPair>(sp);
  d.sa = L.at<int4>(sa);
  d.sb = L.at<int4>(sb);
  d.tiles = L.at<SplitTile>(st);
  if (!w.va.empty()) d.va = L.at<OperandView>(va);
  if (!w.vb.empty()) d.vb = L.at<OperandView>(vb);
  d.E = L.at<int>(se);
  d.F = L.at<int>(sf);
  return d;
}

// Shallow output blocks (summed depth <= SHALLOW_K) are computed directly in
// FP64 (run_shallow); deep ones (few tiles, a very deep sum) are cut along
// their depth into parts computed as blocks of their own in a temporary
// buffer and summed in part order (split_deep).  Both decisions depend on the
// block alone, and the digit plan is the one of the list as given, so a
// block gives the same bits whatever else is in the launch.  Deeper blocks
// with a pair read through a view run as they are.
SplitResult run_split(Ctx *ctx, const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                      const std::vector<int32_t> &blk_M, const std::vector<int32_t> &blk_N,
                      const std::vector<int64_t> &c_off, const double *A, const double *B, double *C,
                      bool cplx, int forced_slices, double tol, const std::vector<int32_t> *blk_ldc,
                      int forced_bits, const std::vector<OperandView> *va,
                      const std::vector<OperandView> *vb) {
  const size_t nb = blk_M.size();
  const int64_t eb = cplx ? 16 : 8;
  // blocks with a pair read through a view are not cut along their depth
  std::vector<char> keep;
  if (va || vb) {
    keep.assign(nb, 0);
    for (size_t g = 0; g < nb; ++g)
      for (int64_t p = grp[g]; p < grp[g + 1]; ++p)
        if ((va && (*va)[p].nl > 0) || (vb && (*vb)[p].nl > 0)) keep[g] = 1;
  }
  std::vector<char> shallow(nb, 0), rest(nb, 1);
  std::vector<int64_t> shallow_ids;
  for (size_t g = 0; g < nb; ++g)
    if (is_shallow(pairs, grp[g], grp[g + 1]) &&
        shallow_direct_wins(pairs, grp[g], grp[g + 1], blk_M[g], blk_N[g], cplx)) {
      shallow[g] = 1;
      rest[g] = 0;
      shallow_ids.push_back((int64_t)g);
    }
  if (!shallow_ids.empty()) {
    const DigitPlan dp = choose_digits_for(pairs, grp, blk_M, blk_N, cplx ? 2 : 1, tol, forced_slices, forced_bits);
    SplitResult res;
    if (shallow_ids.size() < nb) {
      const BlockList R = select_blocks(pairs, grp, blk_M, blk_N, c_off, blk_ldc, rest);
      std::vector<OperandView> va2, vb2;
      for (int32_t q : R.src) {
        if (va) va2.push_back((*va)[q]);
        if (vb) vb2.push_back((*vb)[q]);
      }
      res = run_split(ctx, R.pairs, R.grp, R.bM, R.bN, R.coff, A, B, C, cplx, dp.nslices, tol, &R.bldc, dp.bits,
                      va ? &va2 : nullptr, vb ? &vb2 : nullptr);
    }
    run_shallow(ctx, pairs, grp, blk_M, blk_N, c_off, blk_ldc, shallow_ids, A, B, C, cplx, va, vb);
    if (!res.nslices) {
      res.nslices = dp.nslices;
      res.bits = dp.bits;
      res.err_bound = dp.err_bound;
    }
    return res;
  }
  DeepSplit ds;
  if (reinterpret_cast<uintptr_t>(C) % eb == 0 &&
      split_deep(pairs, grp, blk_M, blk_N, c_off, blk_ldc, ds, keep.empty() ? nullptr : &keep)) {
    const DigitPlan dp = choose_digits_for(pairs, grp, blk_M, blk_N, cplx ? 2 : 1, tol, forced_slices, forced_bits);
    double *T = dev_alloc<double>(ctx, (size_t)std::max<int64_t>(ds.temp_elems, 1) * (cplx ? 2 : 1));
    DeepReduce *d_red = nullptr;
    // the views follow their pairs (pairs of cut blocks have none)
    std::vector<OperandView> va2, vb2;
    for (int32_t q : ds.src) {
      if (va) va2.push_back((*va)[q]);
      if (vb) vb2.push_back((*vb)[q]);
    }
    try {
      ds.place((int64_t)(reinterpret_cast<intptr_t>(T) - reinterpret_cast<intptr_t>(C)) / eb);
      d_red = dev_upload(ctx, ds.red);
      // parts with a few outputs: one CTA per output element in FP64
      // (run_dot; a tile would compute 4096 outputs for each); the rest
      // through the split path
      std::vector<char> sel(ds.bM.size(), 1);
      std::vector<int64_t> small;
      for (size_t g = 0; g < ds.bM.size(); ++g)
        if (ds.part[g] && (int64_t)ds.bM[g] * ds.bN[g] <= DOT_OUTPUTS) {
          sel[g] = 0;
          small.push_back((int64_t)g);
        }
      if (small.size() < ds.bM.size()) require_whole_elements(A, B, nullptr, cplx);
      run_dot(ctx, ds.pairs, ds.grp, ds.bM, ds.bN, ds.coff, &ds.bldc, small, A, B, C, cplx);
      SplitResult res;
      res.nslices = dp.nslices;
      res.bits = dp.bits;
      res.err_bound = dp.err_bound;
      if (small.size() < ds.bM.size()) {
        const BlockList R = select_blocks(ds.pairs, ds.grp, ds.bM, ds.bN, ds.coff, &ds.bldc, sel);
        std::vector<OperandView> va3, vb3;
        for (int32_t q : R.src) {
          if (va) va3.push_back(va2[q]);
          if (vb) vb3.push_back(vb2[q]);
        }
        res = run_split_lists(ctx, R.pairs, R.grp, R.bM, R.bN, R.coff, A, B, C, cplx, dp.nslices, tol, &R.bldc,
                              dp.bits, va ? &va3 : nullptr, vb ? &vb3 : nullptr);
      }
      launch_reduce_parts(ctx, d_red, (int64_t)ds.red.size(), T, C, cplx);
      dev_free(ctx, d_red);
      dev_free(ctx, T);
      return res;
    } catch (...) {
      cudaStreamSynchronize(ctx->stream);
      if (d_red) dev_free(ctx, d_red);
      dev_free(ctx, T);
      throw;
    }
  }
  return run_split_lists(ctx, pairs, grp, blk_M, blk_N, c_off, A, B, C, cplx, forced_slices, tol, blk_ldc,
                         forced_bits, va, vb);
}

static SplitResult run_split_lists(Ctx *ctx, const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                                   const std::vector<int32_t> &blk_M, const std::vector<int32_t> &blk_N,
                                   const std::vector<int64_t> &c_off, const double *A, const double *B, double *C,
                                   bool cplx, int forced_slices, double tol, const std::vector<int32_t> *blk_ldc,
                                   int forced_bits, const std::vector<OperandView> *va,
                                   const std::vector<OperandView> *vb) {
  SplitWork w;
  SplitResult res = plan_split(pairs, grp, blk_M, blk_N, c_off, cplx, forced_slices, tol, blk_ldc, w, forced_bits,
                               va, vb);
  if (w.tiles.empty()) return res;
  require_whole_elements(A, B, nullptr, cplx);  // the products' stores are single doubles
  DevLists L;
  SplitDev d = stage_split_work(ctx, w, L);
  // the digit arena is pooled scratch
  d.arena = static_cast<uint8_t *>(ctx->ensure_scratch((size_t)std::max<int64_t>(w.arena, 256)));
  launch_split(ctx, w, cplx, d, A, B, C, ctx->d_err, true, true);
  return res;
}

SplitResult run_split_static(Ctx *ctx, const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                             const std::vector<int32_t> &blk_M, const std::vector<int32_t> &blk_N,
                             const std::vector<int64_t> &c_off, const double *A, const double *B, double *C,
                             bool cplx, int forced_slices, double tol, const std::vector<int32_t> *blk_ldc,
                             uint8_t *scratch, size_t cap, int *err) {
  SplitWork w;
  SplitResult res = plan_split(pairs, grp, blk_M, blk_N, c_off, cplx, forced_slices, tol, blk_ldc, w);
  if (w.tiles.empty()) return res;
  require_whole_elements(A, B, nullptr, cplx);
  size_t used = 0;
  auto take = [&](size_t bytes) {
    const size_t o = used;
    used += (std::max<size_t>(bytes, 1) + 255) / 256 * 256;
    return o;
  };
  const size_t o_pairs = take(w.sp.size() * sizeof(SplitPair));
  const size_t o_sa = take(w.sa.size() * sizeof(int4)), o_sb = take(w.sb.size() * sizeof(int4));
  const size_t o_tiles = take(w.tiles.size() * sizeof(SplitTile));
  const size_t o_E = take((size_t)w.nE * sizeof(int)), o_F = take((size_t)w.nF * sizeof(int));
  const size_t o_arena = take((size_t)w.arena);
  if (used > cap)
    fail(QS_ERR_OOM, "split (static scratch): this pair list needs %zu bytes of scratch (%lld of them "
         "FP16 digits), more than the %zu available", used, (long long)w.arena, cap);
  SplitDev d;
  d.pairs = reinterpret_cast<SplitPair *>(scratch + o_pairs);
  d.sa = reinterpret_cast<int4 *>(scratch + o_sa);
  d.sb = reinterpret_cast<int4 *>(scratch + o_sb);
  d.tiles = reinterpret_cast<SplitTile *>(scratch + o_tiles);
  d.E = reinterpret_cast<int *>(scratch + o_E);
  d.F = reinterpret_cast<int *>(scratch + o_F);
  d.arena = scratch + o_arena;
  auto put = [&](void *dst, const void *src, size_t bytes) {
    if (bytes) QS_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
  };
  put(d.pairs, w.sp.data(), w.sp.size() * sizeof(SplitPair));
  put(d.sa, w.sa.data(), w.sa.size() * sizeof(int4));
  put(d.sb, w.sb.data(), w.sb.size() * sizeof(int4));
  put(d.tiles, w.tiles.data(), w.tiles.size() * sizeof(SplitTile));
  launch_split(ctx, w, cplx, d, A, B, C, err, false);
  // the work lists are copied from pageable host memory, which the GPU may
  // read when the copies execute rather than when they are queued: keep them
  // alive until then
  QS_CUDA(cudaStreamSynchronize(ctx->stream));
  return res;
}

// Digit widths b whose plan meets `tol` (with `forced_slices` digits when
// that is set): the candidates an autotuner times.
std::vector<int> split_candidate_bits(double tol, int forced_slices) {
  if (!(tol > 0)) tol = 1e-12;
  const int need = (int)std::ceil(-std::log2(tol)) + 8;
  std::vector<int> out;
  for (int b = 8; b >= 5; --b) {
    int S = forced_slices > 0 ? forced_slices : (need - 1 + b - 1) / b;
    S = std::max(S, 2);
    if (S > 8 || b * S > 62 || kchunk_of(b, S) < TKS) continue;
    out.push_back(b);
  }
  return out;
}

// ------------------------------------------- FP64-grade tensor-core products
// Blocks the tensor-core launch takes: a summed real depth of at least
// F64T_DEPTH (below it nearly every tile of normally distributed operands holds
// an output that misses the certificate: 99 % of the 32 x 32 tiles at depth 12,
// 78 % at 16, 28 % at 20, 6 % at 24, 0.4 % at 32) and at least F64T_WORK real
// multiply-adds, which take the narrow FP64 pipe (about 2 multiply-adds per
// clock and SM) 9 us in one tile; the three launches take about 25 us in sum
// whatever the block.  Measured, FP64 tiles against this path: 300 complex
// products of 8..1024 per side 23.1 -> 1.25 ms (21.4 TFLOP/s of FP64 work;
// error against a 64-bit product 1.2e-15 -> 7.0e-16), 64 real blocks of
// 4..96 105 -> 53..60 us.
constexpr int64_t F64T_DEPTH = 16, F64T_MAX_DEPTH = 1 << 20;
constexpr double F64T_WORK = 32768.0;
// Digit bytes of one launch (blocks above it get a launch of their own), and
// of a block that still takes this path.
constexpr int64_t F64T_CHUNK_BYTES = int64_t(2) << 30, F64T_BLOCK_BYTES = int64_t(8) << 30;
// Digits that a call leaves as the context's scratch for the next one; more go
// back to the pool at its end (about 3 us a call), where every allocation of the
// library finds them.
constexpr int64_t F64T_KEEP_BYTES = int64_t(16) << 20;

// Whether the tensor-core launch takes a block; `bytes` its digits (at most).
static bool f64_tensor_takes(const std::vector<PairDesc> &pairs, int64_t p0, int64_t p1, int64_t M, int64_t N,
                             int64_t ldc, bool cplx, int64_t &bytes) {
  const int64_t cm = cplx ? 2 : 1;
  auto up = [](int64_t x, int64_t t) { return (x + t - 1) / t * t; };
  int64_t depth = 0, kpad = 0;
  for (int64_t p = p0; p < p1; ++p) {
    const int64_t K = std::max<int32_t>(pairs[p].K, 0);
    depth += K * cm;
    kpad += up(std::max<int64_t>(K * cm, 1), TKS);
    // a factor of 0 keeps the FP64 kernel's 0 * x (NaN for an infinite x)
    if (!std::isfinite(pairs[p].afac) || pairs[p].afac == 0.0) return false;
  }
  // (the tiles' strides are 32-bit counts of doubles)
  if (depth < F64T_DEPTH || depth > F64T_MAX_DEPTH || M > (1 << 24) || N > (1 << 24) || ldc * cm > INT32_MAX ||
      double(M) * double(N) * double(depth) * double(cm) < F64T_WORK)
    return false;
  // either operand's real form may be the duplicated one
  bytes = (up(M * cm, TMS) + up(N * cm, TMS)) * kpad * (HP_DIGITS + 1) * 2;
  return bytes <= F64T_BLOCK_BYTES;
}

F64TensorList plan_f64_tensor(const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                              const std::vector<int32_t> &bM, const std::vector<int32_t> &bN,
                              const std::vector<int64_t> &coff, const std::vector<int32_t> *bldc, bool cplx,
                              const std::vector<char> &skip, int64_t limit) {
  F64TensorList tl;
  const int64_t nb = (int64_t)bM.size();
  tl.on.assign(nb, 0);
  tl.fbase.assign(nb, 0);
  for (int64_t g = 0; g < nb; ++g) {
    const int64_t M = bM[g], N = bN[g], ldc = bldc ? (*bldc)[g] : std::max(bM[g], 1);
    int64_t bytes = 0;
    if ((!skip.empty() && skip[g]) || !f64_tensor_takes(pairs, grp[g], grp[g + 1], M, N, ldc, cplx, bytes) ||
        bytes > limit)
      continue;
    const int64_t tiles = ((M + F64_TILE - 1) / F64_TILE) * ((N + F64_TILE - 1) / F64_TILE);
    if (tl.ntiles + tiles > INT32_MAX / 4) continue;
    tl.on[g] = 1;
    tl.fbase[g] = (int32_t)tl.ntiles;
    TileDesc t{};
    t.c_off = coff[g];
    t.p0 = (int32_t)grp[g];
    t.p1 = (int32_t)grp[g + 1];
    t.M = bM[g];
    t.N = bN[g];
    t.ldc = (int32_t)ldc;
    t.cblk = (int32_t)g;
    t.first = tl.fbase[g];
    tl.checked.push_back(t);
    tl.ntiles += tiles;
    tl.bytes.push_back(bytes);
  }
  return tl;
}

// The block ranges of launches that hold at most `limit` bytes of digits each
// (a block above it gets a launch of its own).
static std::vector<std::pair<int64_t, int64_t>> f64_chunks(const F64TensorList &tl, int64_t limit) {
  std::vector<std::pair<int64_t, int64_t>> chunks;
  int64_t held = 0;
  for (size_t k = 0; k < tl.checked.size(); ++k) {
    const int64_t g = tl.checked[k].cblk;
    if (chunks.empty() || held + tl.bytes[k] > limit) {
      chunks.push_back({g, g});
      held = 0;
    }
    chunks.back().second = g + 1;
    held += tl.bytes[k];
  }
  return chunks;
}

// Work lists of the launch of one block range of a list.
static void plan_f64_chunk(const F64TensorList &tl, std::pair<int64_t, int64_t> range,
                           const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                           const std::vector<int32_t> &bM, const std::vector<int32_t> &bN,
                           const std::vector<int64_t> &coff, const std::vector<int32_t> *bldc, bool cplx,
                           SplitWork &w) {
  std::vector<char> sel(bM.size(), 0);
  std::vector<int32_t> fb;
  for (int64_t g = range.first; g < range.second; ++g)
    if (tl.on[g]) {
      sel[g] = 1;
      fb.push_back(tl.fbase[g]);
    }
  const BlockList L = select_blocks(pairs, grp, bM, bN, coff, bldc, sel);
  plan_split(L.pairs, L.grp, L.bM, L.bN, L.coff, cplx, 0, 0, &L.bldc, w, 0, nullptr, nullptr, &fb);
}

int64_t f64_digit_bytes(const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                        const std::vector<int32_t> &bM, const std::vector<int32_t> &bN,
                        const std::vector<int64_t> &coff, bool cplx) {
  // the blocks as run_f64 has them: no shallow ones, deep ones cut into parts,
  // of which those with a few outputs have no digits
  std::vector<char> rest(bM.size(), 1);
  for (size_t b = 0; b < bM.size(); ++b) rest[b] = !is_shallow(pairs, grp[b], grp[b + 1]);
  const BlockList R = select_blocks(pairs, grp, bM, bN, coff, nullptr, rest);
  DeepSplit ds;
  const bool deep = split_deep(R.pairs, R.grp, R.bM, R.bN, R.coff, &R.bldc, ds);
  std::vector<char> skip(deep ? ds.bM.size() : R.bM.size(), 0);
  if (deep)
    for (size_t b = 0; b < skip.size(); ++b) skip[b] = ds.part[b] && (int64_t)ds.bM[b] * ds.bN[b] <= DOT_OUTPUTS;
  const F64TensorList tl = deep ? plan_f64_tensor(ds.pairs, ds.grp, ds.bM, ds.bN, ds.coff, &ds.bldc, cplx, skip)
                                : plan_f64_tensor(R.pairs, R.grp, R.bM, R.bN, R.coff, &R.bldc, cplx, skip);
  int64_t sum = 0, most = 0;
  for (int64_t x : tl.bytes) {
    sum += x;
    most = std::max(most, x);
  }
  return std::min(sum, std::max(most, F64T_CHUNK_BYTES));
}

// Plans the launches of a list and hands them to `allocate`, with fewer digits
// (at first `most`) a launch where that finds no room; false when the launches of single blocks
// do not fit either.
template <class F>
static bool plan_f64_launches(const F64TensorList &tl, const std::vector<PairDesc> &pairs,
                              const std::vector<int64_t> &grp, const std::vector<int32_t> &bM,
                              const std::vector<int32_t> &bN, const std::vector<int64_t> &coff,
                              const std::vector<int32_t> *bldc, bool cplx, int64_t most,
                              std::vector<SplitWork> &ws, F allocate) {
  size_t tried = 0;
  for (int64_t limit = std::min(F64T_CHUNK_BYTES, most); tried < tl.checked.size(); limit /= 4) {
    const auto chunks = f64_chunks(tl, limit);
    if (chunks.size() == tried) continue;
    tried = chunks.size();
    ws.clear();
    ws.resize(tried);
    for (size_t k = 0; k < tried; ++k) plan_f64_chunk(tl, chunks[k], pairs, grp, bM, bN, coff, bldc, cplx, ws[k]);
    try {
      allocate();
      return true;
    } catch (const Error &e) {
      if (e.code != QS_ERR_OOM) throw;
      cudaGetLastError();
    }
  }
  return false;
}

bool run_f64_tensor(Ctx *ctx, const F64TensorList &tl, const std::vector<PairDesc> &pairs,
                    const std::vector<int64_t> &grp, const std::vector<int32_t> &bM, const std::vector<int32_t> &bN,
                    const std::vector<int64_t> &coff, const std::vector<int32_t> *bldc, const double *A,
                    const double *B, double *C, bool cplx, const MissList &miss) {
  std::vector<SplitWork> ws;
  std::vector<std::unique_ptr<DevLists>> lists;
  std::vector<SplitDev> ds;
  std::unique_ptr<DevLists> own;
  // every allocation before the first launch
  auto allocate = [&] {
    ds.clear();
    lists.clear();
    int64_t arena = 256;
    for (const SplitWork &w : ws) {
      lists.push_back(std::make_unique<DevLists>());
      ds.push_back(stage_split_work(ctx, w, *lists.back()));
      arena = std::max(arena, w.arena);
    }
    uint8_t *digits;
    if (arena <= F64T_KEEP_BYTES || (size_t)arena <= ctx->scratch_bytes) {
      digits = static_cast<uint8_t *>(ctx->ensure_scratch((size_t)arena));
    } else {
      own = std::make_unique<DevLists>();
      const size_t o = own->space((size_t)arena);
      own->commit(ctx);
      digits = own->at<uint8_t>(o);
    }
    for (SplitDev &d : ds) {
      d.arena = digits;
      d.miss = miss;
    }
  };
  if (!plan_f64_launches(tl, pairs, grp, bM, bN, coff, bldc, cplx, ctx->f64_digits, ws, allocate)) return false;
  for (size_t k = 0; k < ws.size(); ++k) launch_split(ctx, ws[k], cplx, ds[k], A, B, C, ctx->d_err, true, k == 0);
  return true;
}

// A planned split product that can be launched many times: its work lists,
// exponent arrays and digit arena are memory owned by the handle (PlanLists),
// so their addresses stay fixed (a CUDA graph can replay the launch).
// An FP64-grade plan may hold several launches, which share the arena.
struct SplitPlanHandle {
  std::vector<SplitWork> w;
  std::vector<SplitDev> d;
  bool cplx = false;
  MissList miss;  // FP64-grade; the head is cleared before the first launch
  std::unique_ptr<PlanLists> lists;
  // every launch's lists and exponent arrays, one arena, and the miss list of
  // `tiles` FP64 tiles
  void allocate(Ctx *ctx, int64_t tiles = 0) {
    lists.reset(new PlanLists);
    d.clear();
    PlanLists &mem = *lists;
    int64_t arena = 0;
    struct At {
      size_t pairs, sa, sb, tiles, E, F;
    };
    std::vector<At> at;
    for (const SplitWork &x : w) {
      arena = std::max(arena, x.arena);
      at.push_back({mem.add(x.sp), mem.add(x.sa), mem.add(x.sb), mem.add(x.tiles), mem.space((size_t)x.nE * sizeof(int)),
                    mem.space((size_t)x.nF * sizeof(int))});
    }
    miss.n = tiles;
    // digits behind the lists, at 256 bytes, made the 2000-product plan 0.9 % slower
    // (4540 -> 4581 us; 4547 at 64 KB or 2 MB)
    constexpr size_t ALIGN = 64 << 10;
    const size_t digits = mem.space((size_t)arena + ALIGN), head = mem.space(miss.head_bytes()),
                 list = mem.space(miss.list_bytes());
    mem.commit(ctx);
    if (tiles) {
      miss.head = mem.at<int>(head);
      miss.list = mem.at<int>(list);
    }
    for (const At &x : at) {
      SplitDev v;
      v.arena = mem.at<uint8_t>(digits);
      v.arena += (ALIGN - reinterpret_cast<uintptr_t>(v.arena) % ALIGN) % ALIGN;
      v.pairs = mem.at<SplitPair>(x.pairs);
      v.sa = mem.at<int4>(x.sa);
      v.sb = mem.at<int4>(x.sb);
      v.tiles = mem.at<SplitTile>(x.tiles);
      v.E = mem.at<int>(x.E);
      v.F = mem.at<int>(x.F);
      v.miss = miss;
      d.push_back(v);
    }
  }
};

SplitPlanHandle *split_plan_create(Ctx *ctx, const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                                   const std::vector<int32_t> &blk_M, const std::vector<int32_t> &blk_N,
                                   const std::vector<int64_t> &c_off, const std::vector<int32_t> &blk_ldc,
                                   bool cplx, int forced_slices, double tol, int bits, SplitResult *res) {
  std::unique_ptr<SplitPlanHandle> h(new SplitPlanHandle);
  h->cplx = cplx;
  h->w.resize(1);
  const SplitResult r =
      plan_split(pairs, grp, blk_M, blk_N, c_off, cplx, forced_slices, tol, &blk_ldc, h->w[0], bits);
  if (res) *res = r;
  if (h->w[0].tiles.empty())
    h->w.clear();
  else
    h->allocate(ctx);
  return h.release();
}

SplitPlanHandle *f64_tensor_plan_create(Ctx *ctx, const F64TensorList &tl, const std::vector<PairDesc> &pairs,
                                        const std::vector<int64_t> &grp, const std::vector<int32_t> &bM,
                                        const std::vector<int32_t> &bN, const std::vector<int64_t> &coff,
                                        const std::vector<int32_t> &bldc, bool cplx, MissList &miss) {
  std::unique_ptr<SplitPlanHandle> h(new SplitPlanHandle);
  h->cplx = cplx;
  if (!plan_f64_launches(tl, pairs, grp, bM, bN, coff, &bldc, cplx, ctx->f64_digits, h->w, [&] { h->allocate(ctx, tl.ntiles); }))
    return nullptr;
  miss = h->miss;
  return h.release();
}

void split_plan_launch(Ctx *ctx, SplitPlanHandle *h, const double *A, const double *B, double *C) {
  if (h->miss.n) QS_CUDA(cudaMemsetAsync(h->miss.head, 0, h->miss.head_bytes(), ctx->stream));
  for (size_t k = 0; k < h->w.size(); ++k)
    if (!h->w[k].tiles.empty()) launch_split(ctx, h->w[k], h->cplx, h->d[k], A, B, C, ctx->d_err, true, k == 0);
}

// The caller makes sure no launch of the handle is still running.
void split_plan_destroy(SplitPlanHandle *h) { delete h; }

}  // namespace qs
