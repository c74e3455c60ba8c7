// Split-precision grouped block GEMM (FP64 emulated with FP16 digits on the
// 5th-generation tensor cores).  See qs_gemm_split.cu for the method.
#pragma once

#include <cstdint>
#include <vector>

#include "qs_internal.h"

namespace qs {

struct SplitResult {
  int nslices = 0;
  int bits = 0;
  double err_bound = 0;
  int64_t slice_bytes = 0;
  int64_t ntiles = 0;
};

struct DigitPlan {
  int bits;    // bits per digit (the leading digit carries bits+1)
  int nslices; // digits per operand
  double err_bound;
};
// The digit plan the split path picks for a grouped product (cm = 2 for
// complex), optionally with the digit count and/or width forced.
DigitPlan choose_digits_for(const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                            const std::vector<int32_t> &blk_M, const std::vector<int32_t> &blk_N, int cm,
                            double tol, int forced_slices, int forced_bits = 0);

// With va / vb (one per pair; nl = 0 for none) the slicing reads op(A) /
// op(B) of a pair through its strided view instead of (lda, trans): a
// permuted operand needs no copy.
SplitResult run_split(Ctx *ctx, const std::vector<PairDesc> &pairs,
                      const std::vector<int64_t> &grp, const std::vector<int32_t> &blk_M,
                      const std::vector<int32_t> &blk_N, const std::vector<int64_t> &c_off,
                      const double *A, const double *B, double *C, bool cplx,
                      int forced_slices, double tol,
                      const std::vector<int32_t> *blk_ldc = nullptr, int forced_bits = 0,
                      const std::vector<OperandView> *va = nullptr,
                      const std::vector<OperandView> *vb = nullptr);

// The same product with every device buffer carved from caller-provided
// scratch (`cap` bytes, 256-byte aligned) instead of allocated; the bounded
// waits report to `err`.  A plan that does not fit is refused (QS_ERR_OOM)
// before anything is copied or launched.
SplitResult run_split_static(Ctx *ctx, const std::vector<PairDesc> &pairs,
                             const std::vector<int64_t> &grp, const std::vector<int32_t> &blk_M,
                             const std::vector<int32_t> &blk_N, const std::vector<int64_t> &c_off,
                             const double *A, const double *B, double *C, bool cplx,
                             int forced_slices, double tol, const std::vector<int32_t> *blk_ldc,
                             uint8_t *scratch, size_t cap, int *err);

// FP64-grade products on the tensor cores, for the plain FP64 path: digits of
// 56 bits per operand, summed without rounding, with a certificate per output
// that the truncation stays at the level of an FP64 sum.  Where it does not
// (and where a line holds an infinity or NaN) the launch lists the output's
// cell (MissList), and the FP64 kernel computes it.
struct F64TensorList {
  std::vector<char> on;         // per block: computed by the tensor-core launch
  std::vector<int32_t> fbase;   // per block: first FP64 tile
  std::vector<TileDesc> checked;  // the blocks as launch_gemm_f64 takes them
  std::vector<int64_t> bytes;     // their digits (at most)
  int64_t ntiles = 0;  // FP64 tiles of the checked blocks
};
// The blocks of a list that the tensor-core launch takes (a property of the
// block and of `limit`, the most digits a launch may hold), except those marked
// in `skip`.  The list holds no shallow blocks: the FP64 path computes all of
// them directly (run_shallow), which takes complex buffers aligned to 8 bytes.
F64TensorList plan_f64_tensor(const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                              const std::vector<int32_t> &bM, const std::vector<int32_t> &bN,
                              const std::vector<int64_t> &coff, const std::vector<int32_t> *bldc, bool cplx,
                              const std::vector<char> &skip, int64_t limit = INT64_MAX);
// Bytes of digits that the plain FP64 path holds at a time for a list (at
// most), alone or as part of a longer one.
int64_t f64_digit_bytes(const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                        const std::vector<int32_t> &bM, const std::vector<int32_t> &bN,
                        const std::vector<int64_t> &coff, bool cplx);
// Runs them (strips and products), in several launches where the digits are
// many or room is short; false when the device has no room for the digits of one
// block or for the lists (nothing ran: the caller computes every tile in FP64).
bool run_f64_tensor(Ctx *ctx, const F64TensorList &tl, const std::vector<PairDesc> &pairs,
                    const std::vector<int64_t> &grp, const std::vector<int32_t> &bM, const std::vector<int32_t> &bN,
                    const std::vector<int64_t> &coff, const std::vector<int32_t> *bldc, const double *A,
                    const double *B, double *C, bool cplx, const MissList &miss);

// Reusable split plans (stable device addresses, for CUDA graph replay).
struct SplitPlanHandle;
std::vector<int> split_candidate_bits(double tol, int forced_slices);
// bits = 0: the cost model picks the digit width
SplitPlanHandle *split_plan_create(Ctx *ctx, const std::vector<PairDesc> &pairs, const std::vector<int64_t> &grp,
                                   const std::vector<int32_t> &blk_M, const std::vector<int32_t> &blk_N,
                                   const std::vector<int64_t> &c_off, const std::vector<int32_t> &blk_ldc,
                                   bool cplx, int forced_slices, double tol, int bits, SplitResult *res);
// The FP64-grade form; nullptr when the device has no room for the digits.
SplitPlanHandle *f64_tensor_plan_create(Ctx *ctx, const F64TensorList &tl, const std::vector<PairDesc> &pairs,
                                        const std::vector<int64_t> &grp, const std::vector<int32_t> &bM,
                                        const std::vector<int32_t> &bN, const std::vector<int64_t> &coff,
                                        const std::vector<int32_t> &bldc, bool cplx, MissList &miss);
void split_plan_launch(Ctx *ctx, SplitPlanHandle *h, const double *A, const double *B, double *C);
void split_plan_destroy(SplitPlanHandle *h);

}  // namespace qs
