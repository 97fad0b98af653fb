// rc_xt.cu -- tall-skinny products Y = alpha X T + beta Y on the FP64 tensor pipe, real and complex,
// with Y = X allowed: the Ritz vectors V Q, CholeskyQR's V T, and the deflation X - E C. Replaces
// cublas{D,Z}gemm(OP_N, OP_N) of the reference (RayleighChebyshevLMCuda.h:2178-2200).
//
// A CTA takes row tiles of 16 RS rows and, per tile, accumulates up to 192 columns in registers: warp
// (slab, group) of RS x CG forms 16 rows x 8 CT columns (CT <= 6) of mma.m8n8k4 tiles. X streams through a
// ring of shared-memory stages in slabs of the inner dimension (32 real or 16 complex columns). T stays in
// shared memory for the whole kernel where that leaves room for two CTAs of 8 warps per SM (RES); else its
// slabs stream beside those of X, from a copy in the stages' layout (xt_pack_kernel, at most 0.6 MB, in L2),
// for one CTA of 16 warps. One more warp fills the ring, and the warps wait only for the stages they read: copies
// issued by the 16 product warps themselves (cp.async) and a CTA barrier per slab kept the tensor pipe at 24-26
// of 37 TFLOP/s (without the copies the same loop ran at 35). A slab of X is one TMA tile copy (two with an odd
// leading dimension: even and odd columns); as a bulk copy per column, 32 of 1 KB, the copies took as long as the
// products of a triangular T. A tile's rows of X are read completely before its rows of Y are stored, and no other
// CTA uses them, so Y may be X.
//
// Which rows and which inner indices a lane's fragments hold is free as long as X, T and Y agree. Chosen so
// that every shared-memory read and every store of Y moves 16 bytes (g = lane / 4, q = lane % 4):
//   real     a warp's two row tiles are the even and the odd rows of its 16, two consecutive mma take the
//            even and the odd inner indices: a lane reads rows 2g, 2g+1 of inner index 2q (and 2q+1), and
//            inner indices 2q, 2q+1 of a column of T. With an odd leading dimension (ODD) the odd columns
//            of X start 8 bytes off a 16-byte boundary: they are copied from the row before and read
//            one row later, with 8-byte reads.
//   complex  with T = Tr + i Ti the two row tiles are the real and the imaginary parts of 8 rows: a lane reads
//            one entry (re, im) of X and one of T, and adds re Tr - im Ti and im Tr + re Ti.
//
// TRI: T is upper triangular (CholeskyQR's R^-1): tiles of eight columns stop at their last row of T, half the products.
// Sums that leave out products with exact zeros are the same. 10^6 rows x 96 columns 440 us against 595,
// 2x10^6 x 48 339 against 413, 500,000 x 192 782 against 1160, complex 442,368 x 192 2.44 ms against 3.77.
//
// Bound: the FP64 tensor pipe (37 TFLOP/s measured for mma.m8n8k4 on 148 SMs), or HBM below about 48
// columns. Measured, with the kernels this one replaced (a resident-T mma kernel for at most 96 real
// columns, FP64 SIMT otherwise): 10^6 rows x 96 columns 31 TFLOP/s (24 before), with an odd leading
// dimension 31 (24), 2x10^6 rows x 48 columns 4.2 TB/s, 500,000 x 192 real 31 TFLOP/s, 442,368 x 192 complex
// 34.7 TFLOP/s (24 in SIMT); row-major, 216,611 x 36 with both outputs 47 us (65).
#include <algorithm>
#include <type_traits>
#include "rc_common.cuh"
#include "rc_dmma.cuh"
#include "rc_internal.h"

namespace rcb {

constexpr int XT_CT = 6;         // 8-column tiles per warp, at most
constexpr int XT_COLS = 192;     // columns per pass, at most
constexpr int XT_STAGES = 4;     // stages, at most

// Shared-memory geometry, in doubles. T: one column of a slab (RES: of all of T) per TP (xt_tpitch) doubles;
// X column-major: one column of a slab per (real rows + XPAD) doubles. With these pitches (T 8, X 2 mod 16)
// the 16-byte fragment reads have no bank conflicts. X row-major: whole rows as they are in memory.
template <bool CPLX>
struct XtGeo {
    static constexpr int KS = CPLX ? 16 : 32;     // inner indices per slab (32 doubles of a column of T)
    static constexpr int TP = 40;
    static constexpr int XPAD = 2;
};
__host__ __device__ inline int xt_tpitch(int kd) {  // RES: the kd doubles of a column of T
    int p = (kd + 7) / 8 * 8;
    return p % 16 == 8 ? p : p + 8;
}

// Column of a pass at place p of T in shared memory: a warp's 8-column tiles, every cg-th from its group on, lie one
// after the other.
__device__ __forceinline__ int xt_column(int p, int ct, int cg) {
    const int t = p >> 3, grp = t / ct;
    return (grp + cg * (t - grp * ct)) * 8 + (p & 7);
}

// T (k x nc, doubles per column kd = k or 2k) in the stages' layout: P[pass][slab][place][TP], zero-padded.
__global__ void xt_pack_kernel(int kd, int nc, int ct, int cg, int nk, int passes, const double* __restrict__ T, int64_t lt,
                               double* __restrict__ P) {
    constexpr int TP = XtGeo<false>::TP;
    const int ncp = 8 * ct * cg;
    const int64_t total = (int64_t)passes * nk * ncp * TP;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int j = (int)(e % TP);
        const int64_t f = e / TP;
        const int c = (int)(f % ncp);
        const int64_t h = f / ncp;
        const int ks = (int)(h % nk), pass = (int)(h / nk);
        const int cc = pass * ncp + xt_column(c, ct, cg), kk = ks * 32 + j;
        P[e] = j < 32 && kk < kd && cc < nc ? T[kk + (int64_t)cc * lt] : 0.0;
    }
}

// Column-major X (xv16): tiles of up to 128 rows (and two, the pitch) of a slab's columns; with an odd leading dimension
// the even columns, and the odd ones (of which the first has index 1) from the row before the block's first.
struct XtMaps {
    CUtensorMap x, odd;
};

template <bool CPLX, bool RM, bool ODD, int CT, bool RES, bool TRI>
__global__ void __launch_bounds__(RES && !RM ? 288 : 544, RES && !RM ? 2 : 1)
xt_dmma_kernel(const __grid_constant__ XtMaps maps, int64_t n, int k, int nc, const double* X, int64_t ldx, const double* __restrict__ Tm, int64_t ldt,
               double* Y, int64_t ldy, double* Yrm, int64_t ldyr, double alpha, double beta, int rs, int cg,
               int stages, bool xv16, int yal, int lost) {
    using G = XtGeo<CPLX>;
    constexpr int CW = CPLX ? 2 : 1;              // doubles per scalar
    extern __shared__ __align__(128) double xtsm[];
    __shared__ __align__(8) uint64_t bars[2 * XT_STAGES];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = rs * cg;
    const int g = lane >> 2, q = lane & 3;
    const int MT = 16 * rs;                       // real rows per tile, a power of two
    const int lmt = 31 - __clz(MT);
    const int64_t rows = CW * n, lx = CW * ldx, ly = CW * ldy, lt = CW * ldt;
    const int ncp = 8 * CT * cg;                  // columns of this pass, padded
    const int c0 = blockIdx.y * ncp;              // first column of this pass
    const int ncl = min(nc - c0, ncp);
    const int BR = min(MT, 128);                  // rows per copied tile
    const int xpitch = RM ? (int)ldx : BR + G::XPAD;
    const int tpitch = RES ? xt_tpitch(CW * k) : G::TP;
    const int half = G::KS * xpitch;              // a copied tile
    const int xsz = RM ? MT * xpitch : MT / BR * half;
    const int tsz = RES ? 0 : ncp * G::TP;
    const int stage = xsz + tsz;
    const int nk = RM ? 1 : (k + G::KS - 1) / G::KS;  // slabs per tile
    const int64_t ntiles = (rows + MT - 1) >> lmt;
    double* ring = xtsm + (RES ? ncp * tpitch : 0);
    const uint32_t full = smem_u32(bars), empty = full + 8 * XT_STAGES;
    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full + 8 * s, xv16 ? 1 : 33);
            mbar_init(empty + 8 * s, nw);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if constexpr (RES) {
        const double* T0 = Tm + (int64_t)c0 * lt;
        for (int e = tid; e < ncp * tpitch; e += blockDim.x) {
            const int p = e / tpitch, kk = e - p * tpitch, c = xt_column(p, CT, cg);
            xtsm[e] = c < ncl && kk < CW * k ? T0[kk + (int64_t)c * lt] : 0.0;
        }
    }
    __syncthreads();
    int b = 0;
    unsigned ph = 0;
    if (warp == nw) {  // the producer
        bool ok = true;
        int64_t used = 0;
        for (int64_t t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
            const int64_t r0 = t << lmt;
            const int valid = (int)min((int64_t)MT, rows - r0);
            for (int ks = 0; ks < nk; ++ks) {
                if (used >= stages && (lost || !mbar_wait(empty + 8 * b, ph ^ 1))) {
                    ok = false;
                    break;
                }
                const uint32_t bar = full + 8 * b;
                double* xd = ring + b * stage;
                const int k0 = ks * G::KS, kn = RM ? k : min(G::KS, k - k0);
                if (xv16) {
                    unsigned bytes = RES ? 0u : (unsigned)tsz * 8;
                    if constexpr (RM) {  // whole rows, one run
                        bytes += (unsigned)(valid * lx) * 8;
                        if (lane == 0) {
                            mbar_arrive_tx(bar, bytes);
                            bulk_copy(smem_u32(xd), X + r0 * lx, bytes, bar);
                        }
                    } else if (lane == 0) {
                        mbar_arrive_tx(bar, bytes + (unsigned)xsz * 8);
                        for (int h = 0; h < MT / BR; ++h) {
                            const uint32_t d = smem_u32(xd + h * half);
                            const int rr = (int)(r0 + h * BR);
                            if constexpr (ODD) {
                                tma_load_2d(d, &maps.x, rr, k0 / 2, bar);
                                tma_load_2d(d + half * 4, &maps.odd, rr, k0 / 2, bar);
                            } else {
                                tma_load_2d(d, &maps.x, rr, k0, bar);
                            }
                        }
                    }
                } else {
                    // 8-byte aligned columns
                    if (lane == 0) mbar_arrive_tx(bar, RES ? 0u : (unsigned)tsz * 8);
                    __syncwarp();
                    const double* src = X + r0 + k0 * lx;
                    for (int kk = 0; kk < kn; ++kk, src += lx)
                        for (int r = lane; r < valid; r += 32) cp_async8(xd + (r >> 7) * half + kk * xpitch + (r & 127), src + r, 8);
                    cp_async_arrive(bar);
                }
                if (!RES && lane == 0)
                    bulk_copy(smem_u32(xd + xsz), Tm + ((int64_t)blockIdx.y * nk + ks) * tsz, (unsigned)tsz * 8, bar);
                ++used;
                if (++b == stages) {
                    b = 0;
                    ph ^= 1;
                }
            }
        }
        // the last copies land before the CTA ends: wait for the stages still in flight
        for (int s = 0; s < stages && s < used; ++s) {
            if (--b < 0) {
                b = stages - 1;
                ph ^= 1;
            }
            if (!mbar_wait(full + 8 * b, ph)) break;
        }
        cp_async_wait0();
        return;
    }

    // a warp's 8-column tiles: every cg-th from its group on (TRI: the groups' work is nearly the same)
    const int slab = warp / cg, grp = warp - slab * cg;
    double acc[2][CT][2];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int j = 0; j < CT; ++j) acc[m][j][0] = acc[m][j][1] = 0.0;
    bool ok = !lost;
    for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        for (int ks = ok ? 0 : nk; ks < nk; ++ks) {
            if (!mbar_wait_warp(full + 8 * b, ph)) {
                ok = false;
                break;
            }
            const double* xs = ring + b * stage;
            const double* tp = (RES ? xtsm + ks * 32 : xs + xsz) + (grp * 8 * CT + g) * tpitch + 2 * q;
            const int kn = RM ? k : min(G::KS, k - ks * G::KS);
            int kk = 0;
            const int xr = (slab >> 3) * half + (slab & 7) * 16 + 2 * g;
            const double* xa = CPLX ? xs + q * xpitch + xr
                                    : (RM ? xs + (slab * 16 + 2 * g) * xpitch + 2 * q
                                          : xs + (ODD ? 1 : 2) * q * xpitch + xr);
            // the products with the warp's tiles from J on, up to the last inner index of tile J
            auto products = [&](auto first) {
                constexpr int J = decltype(first)::value;
                const int end = TRI ? min(kn, 8 * ((c0 >> 3) + grp + cg * J + 1) - ks * G::KS) : kn;
                if constexpr (CPLX) {
#pragma unroll 1
                    for (; kk < end; kk += 4, xa += 4 * xpitch, tp += 8) {
                        double2 v = *reinterpret_cast<const double2*>(xa);
                        double2 w[CT];
                        if constexpr (!TRI) {
#pragma unroll
                            for (int j = J; j < CT; ++j) w[j] = *reinterpret_cast<const double2*>(tp + j * 8 * tpitch);
                        }
                        if (kk + q >= kn) v = make_double2(0.0, 0.0);  // past the last inner index: stale
                        const double nim = -v.y;
                        if constexpr (TRI) {  // one tile of T at a time: fewer registers
#pragma unroll
                            for (int j = J; j < CT; ++j) {
                                const double2 u = *reinterpret_cast<const double2*>(tp + j * 8 * tpitch);
                                dmma(acc[0][j][0], acc[0][j][1], v.x, u.x);
                                dmma(acc[1][j][0], acc[1][j][1], v.y, u.x);
                                dmma(acc[0][j][0], acc[0][j][1], nim, u.y);
                                dmma(acc[1][j][0], acc[1][j][1], v.x, u.y);
                            }
                            continue;
                        }
#pragma unroll
                        for (int j = J; j < CT; ++j) {
                            dmma(acc[0][j][0], acc[0][j][1], v.x, w[j].x);
                            dmma(acc[1][j][0], acc[1][j][1], v.y, w[j].x);
                        }
#pragma unroll
                        for (int j = J; j < CT; ++j) {
                            dmma(acc[0][j][0], acc[0][j][1], nim, w[j].y);
                            dmma(acc[1][j][0], acc[1][j][1], v.x, w[j].y);
                        }
                    }
                } else {
#pragma unroll 1
                    for (; kk < end; kk += 8, xa += RM ? 8 : (ODD ? 4 : 8) * xpitch, tp += 8) {
                        // v: two rows of an inner index (column-major X), or two inner indices of a row
                        const double2 v0 = *reinterpret_cast<const double2*>(xa);
                        const double2 v1 = ODD ? make_double2(xa[half / 2 + 1], xa[half / 2 + 2])
                                               : *reinterpret_cast<const double2*>(xa + xpitch);
                        double2 w[CT];
                        if constexpr (!TRI) {
#pragma unroll
                            for (int j = J; j < CT; ++j) w[j] = *reinterpret_cast<const double2*>(tp + j * 8 * tpitch);
                        }
                        double a00 = v0.x, a10 = RM ? v1.x : v0.y, a01 = RM ? v0.y : v1.x, a11 = v1.y;
                        if (kk + 8 > kn) {  // past the last inner index: stale
                            if (kk + 2 * q >= kn) a00 = a10 = 0.0;
                            if (kk + 2 * q + 1 >= kn) a01 = a11 = 0.0;
                        }
                        if constexpr (TRI) {
#pragma unroll
                            for (int j = J; j < CT; ++j) {
                                const double2 u = *reinterpret_cast<const double2*>(tp + j * 8 * tpitch);
                                dmma(acc[0][j][0], acc[0][j][1], a00, u.x);
                                dmma(acc[1][j][0], acc[1][j][1], a10, u.x);
                                dmma(acc[0][j][0], acc[0][j][1], a01, u.y);
                                dmma(acc[1][j][0], acc[1][j][1], a11, u.y);
                            }
                            continue;
                        }
#pragma unroll
                        for (int j = J; j < CT; ++j) {
                            dmma(acc[0][j][0], acc[0][j][1], a00, w[j].x);
                            dmma(acc[1][j][0], acc[1][j][1], a10, w[j].x);
                        }
#pragma unroll
                        for (int j = J; j < CT; ++j) {
                            dmma(acc[0][j][0], acc[0][j][1], a01, w[j].y);
                            dmma(acc[1][j][0], acc[1][j][1], a11, w[j].y);
                        }
                    }
                }
            };
            products(std::integral_constant<int, 0>{});
            if constexpr (TRI) {
                if constexpr (CT > 1) products(std::integral_constant<int, 1>{});
                if constexpr (CT > 2) products(std::integral_constant<int, 2>{});
                if constexpr (CT > 3) products(std::integral_constant<int, 3>{});
                if constexpr (CT > 4) products(std::integral_constant<int, 4>{});
                if constexpr (CT > 5) products(std::integral_constant<int, 5>{});
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + 8 * b);
            if (++b == stages) {
                b = 0;
                ph ^= 1;
            }
        }
        // a stage that never landed: the warp's part of this tile and of all that follow is NaN
        if (!ok) {
#pragma unroll
            for (int j = 0; j < CT; ++j)
                acc[0][j][0] = acc[0][j][1] = acc[1][j][0] = acc[1][j][1] = __longlong_as_double(0x7ff8000000000000ll);
        }
        // the tile's rows of Y: a lane's rows r, r + 1 of columns c, c + 1 per 8-column tile
        const int64_t r = (t << lmt) + slab * 16 + 2 * g;
        const bool two = r + 1 < rows;
        double* yc = Y + r + (int64_t)(c0 + grp * 8 + 2 * q) * ly;
#pragma unroll
        for (int j = 0; j < CT; ++j) {
            const int c = (grp + cg * j) * 8 + 2 * q;
            double2 y[2] = {make_double2(acc[0][j][0], acc[1][j][0]), make_double2(acc[0][j][1], acc[1][j][1])};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double* yp = yc + h * ly;
                if (r < rows && c + h < ncl) {
                    if (alpha != 1.0) y[h] = make_double2(alpha * y[h].x, alpha * y[h].y);
                    if (beta != 0.0) {
                        y[h].x = fma(beta, yp[0], y[h].x);
                        if (two) y[h].y = fma(beta, yp[1], y[h].y);
                    }
                    if (two && yal > h) {
                        *reinterpret_cast<double2*>(yp) = y[h];
                    } else {
                        yp[0] = y[h].x;
                        if (two) yp[1] = y[h].y;
                    }
                }
            }
            if (!CPLX && Yrm && r < rows) {  // row-major copy (even leading dimension: 16-byte pairs)
                double* yr = Yrm + r * ldyr + c0 + c;
                if (c + 1 < ncl) {
                    *reinterpret_cast<double2*>(yr) = make_double2(y[0].x, y[1].x);
                    if (two) *reinterpret_cast<double2*>(yr + ldyr) = make_double2(y[0].y, y[1].y);
                } else if (c < ncl) {
                    yr[0] = y[0].x;
                    if (two) yr[ldyr] = y[0].y;
                }
            }
            yc += 8 * cg * ly;
            acc[0][j][0] = acc[0][j][1] = acc[1][j][0] = acc[1][j][1] = 0.0;
        }
    }
}

// Y may be X when the columns fit one pass.
bool xt_dmma_in_place(int64_t nc) { return nc <= XT_COLS; }

rc_status xt_dmma(rc_ctx* ctx, int dtype, int64_t n, int64_t k, int64_t nc, const void* X, int64_t ldx, bool x_rm,
                  const void* T, int64_t ldt, void* Y, int64_t ldy, double alpha, double beta, double* Yrm,
                  int64_t ldyr, bool tri) {
    const bool cplx = dtype == RC_COMPLEX128;
    if (n < 1 || nc < 1) return RC_OK;
    if (k < 0 || k > INT32_MAX / 8 || nc > INT32_MAX / 8) return rc_fail(ctx, RC_ERR_INVALID, "xt: bad sizes");
    if (X == Y && (!xt_dmma_in_place(nc) || ldx != ldy || k != nc))
        return rc_fail(ctx, RC_ERR_INVALID, "xt: in place needs a square T of at most 192 columns");
    if (x_rm && (cplx || (uintptr_t)X % 16 != 0 || ldx % 2 != 0 || ldx < k || ldx > 96 || nc > 96))
        return rc_fail(ctx, RC_ERR_INVALID,
                       "xt: row-major X is real, with an even leading dimension in [k, 96], 16-byte aligned");
    if (Yrm && (cplx || ldyr % 2 != 0 || (uintptr_t)Yrm % 16 != 0))
        return rc_fail(ctx, RC_ERR_INVALID, "xt: the row-major copy is real, with an even leading dimension, 16-byte aligned");
    if (cplx && ((uintptr_t)X % 16 != 0 || (uintptr_t)T % 16 != 0))
        return rc_fail(ctx, RC_ERR_INVALID, "xt: complex blocks are 16-byte aligned");
    // equal passes of at most 192 columns, whole 8-column tiles; 1, 2 or 4 column groups of warps
    const int passes = (int)((nc + XT_COLS - 1) / XT_COLS);
    const int tiles8 = (int)(((nc + passes - 1) / passes + 7) / 8);
    // row-major X: groups of 3 tiles, so that 16 warps need no more than 64 rows of 96 columns per stage
    const int ct_max = x_rm ? 3 : XT_CT;
    const int cg = tiles8 <= ct_max ? 1 : (tiles8 <= 2 * ct_max ? 2 : 4);
    const int ct = (tiles8 + cg - 1) / cg;
    const int64_t rows = cplx ? 2 * n : n;
    constexpr int tp = XtGeo<false>::TP, pad = XtGeo<false>::XPAD;
    const int ks = cplx ? XtGeo<true>::KS : XtGeo<false>::KS;
    auto xbytes = [&](int r) {
        return (x_rm ? (size_t)16 * r * ldx : (size_t)ks * (16 * r + (r > 8 ? r / 8 : 1) * pad)) * sizeof(double);
    };
    // T resident: two CTAs of 8 warps with three stages each in an SM's shared memory (with two, the 96-column
    // product ran at 27 TFLOP/s against 31 with T streamed), or one of 16 warps for row-major X
    const int cw = cplx ? 2 : 1;
    const size_t half = (ctx->smem_optin + 1024) / 2 - 1536;
    const size_t tres = (size_t)8 * ct * cg * xt_tpitch(cw * (int)std::min<int64_t>(k, 4096)) * sizeof(double);
    const bool res = x_rm || (cg <= 2 && k <= 4096 && tres + 3 * xbytes(8 / cg) <= half);
    // rows per tile: as many as the CTA's warps take, fewer (down to 32) while that leaves SMs without a tile
    int rs = (res && !x_rm ? 8 : 16) / cg;
    while (rs > 2 && (rows + 16 * rs - 1) / (16 * rs) * passes < ctx->sm_count) rs /= 2;
    const size_t stage = xbytes(rs) + (res ? 0 : (size_t)8 * ct * cg * tp * sizeof(double));
    const size_t fixed = res ? tres : 0, room = res && !x_rm ? half : ctx->smem_optin - 2048;
    const int stages = (int)std::max<size_t>(2, std::min<size_t>(XT_STAGES, (room - fixed) / stage));
    const size_t smem = fixed + stages * stage + 64;  // a row's last fragment may reach past its stage
    const int64_t ntiles = (rows + 16 * rs - 1) / (16 * rs);
    const int64_t per_sm = res && !x_rm ? 2 : 1;
    const dim3 grid((unsigned)std::min<int64_t>(ntiles, std::max<int64_t>(1, ctx->sm_count * per_sm / passes)),
                    (unsigned)passes);
    bool xv16 = (cplx || (uintptr_t)X % 16 == 0) && rows < INT32_MAX - 256;  // else 8-byte copies
    bool odd = !cplx && xv16 && ldx % 2 != 0;
    XtMaps maps = {};
    if (!x_rm && xv16 && k > 0) {
        const int br = std::min(16 * rs, 128) + pad;
        const double* Xd = (const double*)X;
        if (odd)
            xv16 = tma_map_2d(&maps.x, Xd, n, (k + 1) / 2, 2 * ldx, br, ks / 2) &&
                   (k == 1 ? tma_map_2d(&maps.odd, Xd, n, 1, 2 * ldx, br, ks / 2)
                           : tma_map_2d(&maps.odd, Xd + ldx - 1, n + 1, k / 2, 2 * ldx, br, ks / 2));
        else
            xv16 = tma_map_2d(&maps.x, Xd, rows, k, cw * ldx, br, ks);
        odd = odd && xv16;
    }
    const void* Tk = T;
    if (!res) {  // T in the layout of the stages
        const int nk = (int)((k + ks - 1) / ks), ncp = 8 * ct * cg;
        const size_t total = (size_t)passes * nk * ncp * tp;
        void* P = nullptr;
        RC_TRY(rc_slot(ctx, S_XTP, std::max<size_t>(1, total) * sizeof(double), &P));
        if (total > 0) {
            xt_pack_kernel<<<(unsigned)std::min<size_t>((total + 255) / 256, 8 * 148), 256, 0, ctx->stream>>>(
                cw * (int)k, (int)nc, ct, cg, nk, passes, (const double*)T, cw * ldt, (double*)P);
            ctx->launches++;
            RC_CU(ctx, cudaGetLastError());
        }
        Tk = P;
    }
    // columns whose row pairs are 16-byte aligned: all (2), the even ones (1) or none
    const int yal = cplx ? 2 : ((uintptr_t)Y % 16 != 0 ? 0 : (ldy % 2 == 0 ? 2 : 1));
    auto launch = [&](auto kern) -> rc_status {
        RC_CU(ctx, allow_max_smem(ctx, kern));
        kern<<<grid, 32 * (rs * cg + 1), smem, ctx->stream>>>(maps, n, (int)k, (int)nc, (const double*)X, ldx,
                                                             (const double*)Tk, ldt, (double*)Y, ldy, Yrm, ldyr, alpha,
                                                             beta, rs, cg, stages, xv16, yal, ctx->lost);
        ctx->launches++;
        RC_CU(ctx, cudaGetLastError());
        return RC_OK;
    };
    auto by_width = [&](auto c, auto r, auto o, auto t, auto u) -> rc_status {
        constexpr bool C = decltype(c)::value, R = decltype(r)::value, O = decltype(o)::value, S = decltype(t)::value,
                       U = decltype(u)::value;
        switch (ct) {
            case 1: return launch(xt_dmma_kernel<C, R, O, 1, S, U>);
            case 2: return launch(xt_dmma_kernel<C, R, O, 2, S, U>);
            case 3: return launch(xt_dmma_kernel<C, R, O, 3, S, U>);
            case 4: return launch(xt_dmma_kernel<C, R, O, 4, S, U>);
            case 5: return launch(xt_dmma_kernel<C, R, O, 5, S, U>);
            default: return launch(xt_dmma_kernel<C, R, O, 6, S, U>);
        }
    };
    const std::true_type yes{};
    const std::false_type no{};
    if (x_rm) return by_width(no, yes, no, yes, no);
    auto by_shape = [&](auto u) -> rc_status {
        if (cplx) return res ? by_width(yes, no, no, yes, u) : by_width(yes, no, no, no, u);
        if (odd) return res ? by_width(no, no, yes, yes, u) : by_width(no, no, yes, no, u);
        return res ? by_width(no, no, no, yes, u) : by_width(no, no, no, no, u);
    };
    return tri ? by_shape(yes) : by_shape(no);
}

}  // namespace rcb
