// rc_gemm.cu -- the dual tall-skinny product of the Rayleigh-Ritz step for callback operators, real blocks
// with s <= 96, on the FP64 tensor pipe (mma.sync m8n8k4 .f64).
//
//  xt2:   Y = X T (n x k times k x nc, k, nc <= 96) with W T beside it, persistent CTAs with T resident
//         in shared memory, 32-row tiles of X and W, 8-row warp slabs (callback operators; plain products
//         are in rc_xt.cu): W T is formed for the columns that need it, reducing
//         ||(W T)_c - lam_c (X T)_c||^2 for c < res_count; with R32 it writes the residual block
//         R = W T - (X T) diag(lam) in row-major FP32 (the source term of an FP32-storage
//         correction filter; native real operators take R from rc_resid.cu instead).
// These replace cublasDgemm(OP_T, OP_N) and cublasDgemm(OP_N, OP_N) plus the residual kernel
// of the reference (RayleighChebyshevLMCuda.h:2139-2161, :2200-2285).
//
// mma.m8n8k4 .f64 fragments (g = lane / 4, q = lane % 4): A (8x4, row) a = A[g][q];
// B (4x8, col) b = B[q][g]; C (8x8) {c0, c1} = C[g][2q], C[g][2q+1].
#include <algorithm>
#include "rc_common.cuh"
#include "rc_dmma.cuh"
#include "rc_internal.h"

namespace rcb {

// Copy rows [r0, r0 + RT) of columns [0, ncols) of a column-major block into a shared tile laid
// out column by column with `rp` doubles per column (rows past r_end read as zero).
template <int RT, bool V16>
__device__ __forceinline__ void load_cols_async(double* tile, int rp, const double* __restrict__ src, int64_t ld,
                                                int ncols, int64_t r0, int64_t r_end, int tid, int nthreads) {
    if (V16) {
        constexpr int H = RT / 2;
        for (int e = tid; e < ncols * H; e += nthreads) {
            const int c = e / H, rr = 2 * (e - c * H);
            const int64_t r = r0 + rr;
            const int64_t left = r_end - r;
            const int bytes = left >= 2 ? 16 : (left == 1 ? 8 : 0);
            const double* gp = bytes ? src + r + (int64_t)c * ld : src;
            cp_async16(tile + c * rp + rr, gp, bytes);
        }
    } else {
        for (int e = tid; e < ncols * RT; e += nthreads) {
            const int c = e / RT, rr = e - c * RT;
            const int64_t r = r0 + rr;
            const bool ok = r < r_end;
            cp_async8(tile + c * rp + rr, ok ? src + r + (int64_t)c * ld : src, ok ? 8 : 0);
        }
    }
}

// ---------------------------------------------------------------------------------------
// xt2
// ---------------------------------------------------------------------------------------
constexpr int XM_RT = 32;         // rows per tile
constexpr int XM_RP = XM_RT + 4;  // doubles per column of a shared X/W tile (= 4 mod 16)
constexpr int XM_CT = 6;          // 8-column mma tiles per warp (48 columns)

// Doubles per column of the shared T (>= k rounded up to 4, = 4 mod 16).
__host__ __device__ inline int xm_kpt(int k) {
    int k4 = (k + 3) / 4 * 4;
    while (k4 % 16 != 4) k4 += 4;
    return k4;
}

// Warps: 4 row slabs (8 rows each) x NH column halves (48 columns each).
template <int NH, bool V16>
__global__ void __launch_bounds__(128 * NH, 1)
xt_mma_kernel(int64_t n, int k, int nc, const double* __restrict__ X, int64_t ldx, const double* __restrict__ Tm,
              int64_t ldt, double* __restrict__ Y, int64_t ldy, const double* __restrict__ W, int64_t ldw,
              const double* __restrict__ lam, int dual_cols, int res_count, double* __restrict__ rpart,
              float* __restrict__ R32, int64_t ldr) {
    constexpr int NT = 128 * NH;
    constexpr int OPS = 2;
    const int kpt = xm_kpt(k);
    const int k4 = (k + 3) / 4 * 4;
    extern __shared__ __align__(16) double xms[];
    double* Ts = xms;                                  // [NH*48][kpt]
    double* tiles = Ts + (size_t)NH * 48 * kpt;        // [2][OPS][k4][XM_RP]
    const int stage = OPS * k4 * XM_RP;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int slab = warp & 3, half = warp >> 2;
    const int cbase = half * 48;
    for (int e = tid; e < NH * 48 * kpt; e += NT) {
        const int c = e / kpt, kk = e - c * kpt;
        Ts[e] = (c < nc && kk < k) ? Tm[kk + (int64_t)c * ldt] : 0.0;
    }
    // zero the padding columns k..k4 of every operand of both stages once
    {
        const int per = (k4 - k) * XM_RP;
        for (int e = tid; e < 2 * OPS * per; e += NT) {
            const int st = e / per, f = e - st * per;
            tiles[st * k4 * XM_RP + k * XM_RP + f] = 0.0;
        }
    }
    // mma tiles of this warp whose columns need W T (warp-uniform)
    const int dtiles = max(0, min(XM_CT, (dual_cols - cbase + 7) / 8));
    double lamc[XM_CT][2], rs[XM_CT][2];
#pragma unroll
    for (int j = 0; j < XM_CT; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = cbase + j * 8 + 2 * q + h;
            lamc[j][h] = c < dual_cols ? lam[c] : 0.0;
            rs[j][h] = 0.0;
        }
    const int64_t ntiles = (n + XM_RT - 1) / XM_RT;
    auto issue = [&](int64_t t, int b) {
        double* st = tiles + b * stage;
        const int64_t r0 = t * XM_RT;
        load_cols_async<XM_RT, V16>(st, XM_RP, X, ldx, k, r0, n, tid, NT);
        load_cols_async<XM_RT, V16>(st + k4 * XM_RP, XM_RP, W, ldw, k, r0, n, tid, NT);
    };
    // two stages, one barrier per tile
    int buf = 0;
    int64_t t = blockIdx.x;
    if (t < ntiles) issue(t, 0);
    cp_async_commit();
    for (; t < ntiles; t += gridDim.x) {
        cp_async_wait0();
        __syncthreads();
        const int64_t tn = t + gridDim.x;
        if (tn < ntiles) issue(tn, buf ^ 1);
        cp_async_commit();
        const double* xs = tiles + buf * stage + slab * 8 + g + q * XM_RP;
        const double* ws = xs + k4 * XM_RP;
        const double* ts = Ts + (cbase + g) * kpt + q;
        double acc[XM_CT][2], acc2[XM_CT][2];
#pragma unroll
        for (int j = 0; j < XM_CT; ++j) acc[j][0] = acc[j][1] = acc2[j][0] = acc2[j][1] = 0.0;
#pragma unroll 2
        for (int k0 = 0; k0 < k4; k0 += 4) {
            const double a = xs[k0 * XM_RP];
            double b[XM_CT];
#pragma unroll
            for (int j = 0; j < XM_CT; ++j) b[j] = ts[j * 8 * kpt + k0];
#pragma unroll
            for (int j = 0; j < XM_CT; ++j) dmma(acc[j][0], acc[j][1], a, b[j]);
            if (dtiles > 0) {
                const double w = ws[k0 * XM_RP];
#pragma unroll
                for (int j = 0; j < XM_CT; ++j)
                    if (j < dtiles) dmma(acc2[j][0], acc2[j][1], w, b[j]);
            }
        }
        const int64_t r = t * XM_RT + slab * 8 + g;
        if (r < n) {
#pragma unroll
            for (int j = 0; j < XM_CT; ++j) {
                const int c = cbase + j * 8 + 2 * q;
                if (c < nc) Y[r + (int64_t)c * ldy] = acc[j][0];
                if (c + 1 < nc) Y[r + (int64_t)(c + 1) * ldy] = acc[j][1];
                if (j < dtiles) {
                    const double d0 = acc2[j][0] - lamc[j][0] * acc[j][0];
                    const double d1 = acc2[j][1] - lamc[j][1] * acc[j][1];
                    if (c < res_count) rs[j][0] = fma(d0, d0, rs[j][0]);
                    if (c + 1 < res_count) rs[j][1] = fma(d1, d1, rs[j][1]);
                    if (R32) {
                        if (c + 1 < nc) {
                            *reinterpret_cast<float2*>(R32 + r * ldr + c) = make_float2((float)d0, (float)d1);
                        } else if (c < nc) {
                            R32[r * ldr + c] = (float)d0;
                        }
                    }
                }
            }
        }
        buf ^= 1;
    }
    if (res_count > 0) {
        __syncthreads();  // the last tile's reads are done before its stage is reused below
        // per column: sum over g (lanes with the same q), then over the four row slabs in order
        double* red = tiles;  // [4][NH*48]; the tiles are no longer read
#pragma unroll
        for (int j = 0; j < XM_CT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double v = rs[j][h];
                v += __shfl_xor_sync(0xffffffffu, v, 4);
                v += __shfl_xor_sync(0xffffffffu, v, 8);
                v += __shfl_xor_sync(0xffffffffu, v, 16);
                if (g == 0) red[slab * NH * 48 + cbase + j * 8 + 2 * q + h] = v;
            }
        __syncthreads();
        for (int c = tid; c < res_count; c += NT) {
            double v = 0.0;
#pragma unroll
            for (int sl = 0; sl < 4; ++sl) v += red[sl * NH * 48 + c];
            rpart[(size_t)blockIdx.x * res_count + c] = v;
        }
    }
}

__global__ void resid2_reduce_kernel(int64_t nblocks, int res_count, const double* __restrict__ rpart,
                                     double* __restrict__ res) {
    const int c = blockIdx.x;
    __shared__ double sc[32];
    double v = 0.0;
    for (int64_t b = threadIdx.x; b < nblocks; b += blockDim.x) v += rpart[(size_t)b * res_count + c];
    v = block_sum(v, sc);
    if (threadIdx.x == 0) res[c] = sqrt(v);
}

bool xt2_supported(int dtype, int64_t k, int64_t nc) {
    return dtype == RC_REAL64 && k >= 1 && k <= 96 && nc >= 1 && nc <= 96;
}

template <int NH, bool V16>
static rc_status xt_mma_launch(rc_ctx* ctx, unsigned grid, int64_t n, int64_t k, int64_t nc, const double* X,
                               int64_t ldx, const double* T, int64_t ldt, double* Y, int64_t ldy, const double* W,
                               int64_t ldw, const double* lam, int64_t dual_cols, int64_t res_count, double* rpart,
                               float* R32, int64_t ldr) {
    const int k4 = (int)((k + 3) / 4 * 4);
    const size_t smem =
        ((size_t)NH * 48 * xm_kpt((int)k) + (size_t)4 * k4 * XM_RP) * sizeof(double);
    RC_CU(ctx, allow_max_smem(ctx, xt_mma_kernel<NH, V16>));
    xt_mma_kernel<NH, V16><<<grid, 128 * NH, smem, ctx->stream>>>(
        n, (int)k, (int)nc, X, ldx, T, ldt, Y, ldy, W, ldw, lam, (int)dual_cols, (int)res_count, rpart, R32, ldr);
    return RC_OK;
}

// Y = X T; with W: residual norms ||(W T)_c - lam_c Y_c|| for c < res_count into res (device),
// and with R32 the residual block (all nc columns) in row-major FP32 with leading dimension ldr.
rc_status xt2(rc_ctx* ctx, int64_t n, int64_t k, int64_t nc, const double* X, int64_t ldx, const double* T,
              int64_t ldt, double* Y, int64_t ldy, const double* W, int64_t ldw, const double* lam, int64_t res_count,
              double* res, float* R32, int64_t ldr) {
    const bool dual = W != nullptr && lam != nullptr && (res_count > 0 || R32 != nullptr);
    const int64_t dual_cols = dual ? (R32 ? nc : std::min(res_count, nc)) : 0;
    if (R32 && (ldr % 2 != 0 || (uintptr_t)R32 % 8 != 0))
        return rc_fail(ctx, RC_ERR_INVALID, "xt2: the residual block needs an even leading dimension");
    const int nh = nc <= 48 ? 1 : 2;
    const int64_t ntiles = (n + XM_RT - 1) / XM_RT;
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ntiles, ctx->sm_count));
    double* rpart = nullptr;
    if (res_count > 0) {
        void* p = nullptr;
        RC_TRY(rc_slot(ctx, S_RPART, (size_t)grid * res_count * sizeof(double), &p));
        rpart = (double*)p;
    }
    const bool v16 =
        ((uintptr_t)X % 16 == 0) && (ldx % 2 == 0) && (!dual || (((uintptr_t)W % 16 == 0) && ldw % 2 == 0));
    if (!dual) return rc_fail(ctx, RC_ERR_INVALID, "xt2: the second block is required");
#define RC_XM(NHV)                                                                                                \
    (v16 ? xt_mma_launch<NHV, true>(ctx, grid, n, k, nc, X, ldx, T, ldt, Y, ldy, W, ldw, lam, dual_cols, res_count, \
                                    rpart, R32, ldr)                                                              \
         : xt_mma_launch<NHV, false>(ctx, grid, n, k, nc, X, ldx, T, ldt, Y, ldy, W, ldw, lam, dual_cols, res_count, \
                                     rpart, R32, ldr))
    rc_status st;
    st = nh == 1 ? RC_XM(1) : RC_XM(2);
#undef RC_XM
    RC_TRY(st);
    ctx->launches++;
    RC_CU(ctx, cudaGetLastError());
    if (res_count > 0) {
        resid2_reduce_kernel<<<(unsigned)res_count, 256, 0, ctx->stream>>>(grid, (int)res_count, rpart, res);
        ctx->launches++;
        RC_CU(ctx, cudaGetLastError());
    }
    return RC_OK;
}

}  // namespace rcb
