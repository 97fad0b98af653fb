// rc_tile.h -- the shared-memory tile kernels of 7- and 27-point operators (rc_tile.cu).
#pragma once
#include "rc_internal.h"

namespace rcb {

// Storage of a step's blocks: FP64, c128, or the correction filter's bfloat16 (pairs) with FP32 (c64) arithmetic.
enum TileType { TT_F64 = 0, TT_C128, TT_BF16, TT_BF16C };

// Whether the operator has the structure and the block (row length ld) the size for the tile kernels.
bool tile_supported(const rc_ctx* ctx, const rc_op* op, TileType type, int64_t ld, bool resid = false);
// y = alpha A x + beta x + gamma z (+ sig[c] src): rm_step_rows' step; z may be null, src goes with TT_BF16*.
// False (nothing launched) when a pointer is not 16-byte aligned or the driver refuses a tensor map.
bool tile_step(rc_ctx* ctx, rc_op* op, TileType type, int64_t ld, const void* x, const void* z, void* y, double alpha,
               double beta, double gamma, const void* src, const float* sig);
// The residual block of rc_resid.cu (FP64 / c128 Y): R (or null) and the partial column sums of squares of *parts CTAs
// into S_RPART.
bool tile_resid(rc_ctx* ctx, rc_op* op, const void* Y, int64_t ld, int64_t s, const double* lam, int64_t res_count,
                void* R, int64_t ldr, double** part, int64_t* parts, rc_status* st);
// One row of packed weights: the neighbours at -P, -L, -1, 0, 1, L, P, (unused).
template <class TC>
struct RowWeights {
    TC w[8];
};
// Whether a CSR operator's rows have the 7-point structure and their packed weights are there, or this context may lay
// them out; and the weights, for a step on a block of `bytes` (null: not laid out, the step takes the gather kernels).
bool tile_rows(const rc_ctx* ctx, const rc_op* op, bool fp32);
const void* tile_weights(rc_ctx* ctx, rc_op* op, bool fp32, int64_t bytes);
// Gives back the weights of this context's operators, which only save time (not those that another context or a
// captured graph reads): whether there were any. For an allocation that failed.
bool tile_weights_release(rc_ctx* ctx);
// op_step of a column-major FP64 block from tiles in shared memory (rc_cmstep.cu): *done is false (nothing launched)
// where the operator, the types or the size are not for it. res_count > 0: also the partial column sums of
// |y - lam x|^2 of *parts tiles, in S_RPART.
rc_status cm_step(rc_ctx* ctx, rc_op* op, const StepArgs& a, const double* lam, int64_t res_count, double** part,
                  int64_t* parts, bool* done);

}  // namespace rcb
