// rc_cmstep.cu -- y = scale (alpha A x + beta x + gamma z) for column-major FP64 blocks of 5- and 7-point operators.
//
// A CTA owns a tile of grid points (2048; 1024 for complex CSR rows) and goes through the columns: their rows' weights
// stay in registers, and each column's box of points (the tile and its faces' neighbours) comes into a ring of
// shared-memory slots, several columns ahead: one TMA copy, or, for lines that are not 16-byte aligned, cp.async (every
// thread's part of a box lies at fixed offsets from the column's start; points outside the grid stay zero). A thread
// owns NP points in a line along z and reads the line once.
//
// The gather kernels (rc_filter.cu) have one thread per row, 256 consecutive rows per CTA: their far neighbours all
// come from L2, about four times the block's bytes, and L2 is the bound. A box of 32 x 8 x 8 points brings 1.6 times.
// The sums are formed in the gather kernels' order (the same bits).
//
// Measured, with the gather kernels' time and the HBM floor, us: CSR 128^3, 96 columns 588 (1170, 512); 7-point stencil
// 573 (1700, 494), with an odd nx 750; complex 24 x 24 x 768, 192 columns 443 (874, 415); 5-point 2048 x 1024, 64
// columns 382 (1063, 330). By cp.async alone the first took 758: its copies were 23 of the 68 % of L1's data cycles.
//
// RES: the column sums of |y - lam x|^2 beside it (Rayleigh-Ritz residuals, which would read both blocks again),
// per tile, in a fixed order.
#include <algorithm>
#include "rc_common.cuh"
#include "rc_dmma.cuh"
#include "rc_internal.h"
#include "rc_tile.h"

namespace rcb {

namespace {

constexpr int CM_THREADS = 512;
constexpr int CM_COPIES = 8;                      // copies per thread and column, at most
constexpr int CM_MAX_BOX = CM_COPIES * CM_THREADS;
constexpr size_t CM_MAX_SMEM = 224 * 1024;
// Smallest block for the tiles. Smaller ones stay in L2, where the gather kernels read at ease and a tile's start shows:
// complex CSR 40^3 x 24 (23 MB) 18.9 -> 25.5 us, 5 points 333 x 400 x 24 (26 MB) 16.8 -> 23.1, stencil 40^3 x 53 (27 MB)
// 18.9 -> 21.1, complex 56 x 61 x 50 x 13 (36 MB) 23.0 -> 24.1; no measured block beyond was slower (48^3 x 53, 45 MB; 40^3 x 96, 49 MB; 100^3 x 16, 128 MB 149 -> 79).
// Fewer than 8 columns leave no ring to fill.
constexpr int64_t kCmMinBytes = 40ll << 20;

// Largest waste of a plan, points copied and formed over those of the grid alone (narrow grids leave most of a tile
// outside), for which the tiles are taken. Steps on 45 to 880 MB, gather -> tiles, us: CSR 130 x 70 x 90 x 24 (1.69) 130 -> 114,
// 400 x 5 x 400 x 24 (2.0) 129 -> 137, 8 x 8 x 13,001 x 96 (2.5) 365 -> 560, 2 x 2 x 200,000 x 96 (21) 360 -> 3439; complex CSR
// 6 x 6 x 25,000 x 56 (2.04) 744 -> 682, 3 x 5 x 50,000 x 24 (4.9) 292 -> 498; stencil 300 x 2 x 1300 x 8 (2.8) 77 -> 66,
// 5 x 400 x 400 x 24 (3.8) 188 -> 261, 2 x 2 x 200,000 x 96 659 -> 3526; complex stencil 10 x 12 x 7000 x 24 (2.55) 242 -> 242,
// 300 x 2 x 1300 x 24 (4.9) 228 -> 366; 5 points 17 x 50,001 x 8 (1.94) 78 -> 74, 2 x 600,000 x 96 (8.7) 942 -> 2220.
template <class T>
constexpr double cm_max_waste(bool csr) { return csr ? (sizeof(T) == 16 ? 2.5 : 1.9) : (sizeof(T) == 16 ? 2.6 : 3.0); }

enum { CK_STENCIL7 = 0, CK_CSR7 = 1, CK_STENCIL5 = 2 };  // 5 points: the grid's y is the kernel's z
template <class T>
constexpr int cm_slots() { return sizeof(T) == 16 ? 4 : 6; }
template <class T>
constexpr int cm_points(int kind) { return sizeof(T) == 16 && kind == CK_CSR7 ? 2 : 4; }  // 16 registers a row there
// Whether lines that are not 16-byte aligned are taken too, by cp.async. Not CSR rows: their weights leave too few
// registers (81 x 83 x 77, 48 columns: 176 us against the gather's 143; the stencil 61 x 53 x 67, 60 columns: 77 against
// 122).
template <class T>
constexpr bool cm_copies(int kind) { return sizeof(T) == 8 && kind != CK_CSR7; }

struct CmArgs {
    int nx, ny, nz;                // the kernel's roles
    int tx, ltx, ty, tz, ntx, nty;
    int hx;                        // the tile's first column in the box
    int px, py, box, slot;         // the box's pitches and size, and the ring's step, in points
    int s, cols;                   // columns, and columns per CTA
    int lost;                      // rc_ctx::lost
};

template <class T, int KIND, bool RES, bool TMA>
__global__ void __launch_bounds__(CM_THREADS, 1)
cm_step_kernel(CmArgs A, const __grid_constant__ CUtensorMap map, const T* __restrict__ x, int64_t ldx, const T* z, int64_t ldz, T* y, int64_t ldy, T alpha,
               T beta, T gamma, double scale, const RowWeights<T>* __restrict__ weights,
               const double* __restrict__ diag, double offd, double theta, const double* __restrict__ lam,
               int res_count, double* __restrict__ part) {
    constexpr int NP = cm_points<T>(KIND), S = cm_slots<T>(), HY = KIND == CK_STENCIL5 ? 0 : 1;
    constexpr bool CPLX = IsComplex<T>::value;
    extern __shared__ __align__(128) unsigned char cms[];
    __shared__ __align__(8) uint64_t full[S];
    __shared__ double red[2][CM_THREADS / 32];
    T* sm = reinterpret_cast<T*>(cms);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t = blockIdx.x, tq = t / A.ntx;
    const int x0 = (t - tq * A.ntx) << A.ltx, y0 = (tq % A.nty) * A.ty, z0 = (tq / A.nty) * A.tz;
    const int c0 = blockIdx.y * A.cols, c1 = min(A.s, c0 + A.cols);
    int off[TMA ? 1 : CM_COPIES];  // rows of this thread's points of a box
    if constexpr (TMA) {
        if (tid == 0) {
            for (int k = 0; k < S; ++k) mbar_init(smem_u32(full + k), 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    } else {
        for (int e = tid; e < S * A.slot; e += CM_THREADS) sm[e] = s_zero(T());
    }
#pragma unroll
    for (int k = 0; k < (TMA ? 0 : CM_COPIES); ++k) {
        const int e = tid + CM_THREADS * k, r = e / A.px;
        const int bx = e - r * A.px, bz = r / A.py, by = r - bz * A.py;
        const int gx = x0 + bx - 1, gy = y0 + by - HY, gz = z0 + bz - 1;
        const int faces = (bx == 0 || bx == A.px - 1) + (HY && (by == 0 || by == A.py - 1)) + (bz == 0 || bz == A.tz + 1);
        const bool in = e < A.box && faces <= 1 && gx >= 0 && gx < A.nx && gy >= 0 && gy < A.ny && gz >= 0 && gz < A.nz;
        off[k] = in ? gx + A.nx * (gy + A.ny * gz) : -1;
    }
    __syncthreads();
    auto issue = [&](int c, int slot) {
        if constexpr (TMA) {
            if (tid == 0 && c < c1) {
                const uint32_t bar = smem_u32(full + slot);
                mbar_arrive_tx(bar, (unsigned)(A.box * sizeof(T)));
                tma_load_4d(smem_u32(sm + slot * A.slot), &map, (x0 - A.hx) * (int)(sizeof(T) / 4), y0 - HY, z0 - 1, c, bar);
            }
        } else {
            if (c < c1) {
                const T* src = x + (int64_t)c * ldx;
                T* dst = sm + slot * A.slot + tid;
#pragma unroll
                for (int k = 0; k < CM_COPIES; ++k)
                    if (off[k] >= 0) {
                        if constexpr (sizeof(T) == 16) cp_async16(dst + CM_THREADS * k, src + off[k], 16);
                        else cp_async8(dst + CM_THREADS * k, src + off[k], 8);
                    }
            }
            cp_async_commit();
        }
    };
    for (int p = 0; p < S - 1; ++p) issue(c0 + p, p);
    // this thread's points
    const int lx = tid & (A.tx - 1), q = tid >> A.ltx, lz = (q / A.ty) * NP, ly = q % A.ty;
    const int gx = x0 + lx, gy = y0 + ly, gz = z0 + lz, plane = A.nx * A.ny;
    const int row = (int)((unsigned)gx + (unsigned)A.nx * ((unsigned)gy + (unsigned)A.ny * (unsigned)gz));
    const int pz = A.px * A.py, o = lx + A.hx + A.px * (ly + HY) + pz * lz;  // the point below the first
    const bool in = gx < A.nx && gy < A.ny;
    T w[NP][7];
    double d[NP];
    T ph = s_zero(T()), phc = s_zero(T());
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        const bool ok = in && gz + k < A.nz;
        if constexpr (KIND == CK_CSR7) {
            const T* wr = weights[ok ? row + k * plane : 0].w;
#pragma unroll
            for (int j = 0; j < 7; ++j) w[k][j] = ok ? wr[j] : s_zero(T());
        } else {
            d[k] = ok ? diag[row + k * plane] : 0.0;
        }
    }
    if constexpr (CPLX && KIND == CK_STENCIL7) {
        double sn, cs;
        sincos(theta * (double)gx, &sn, &cs);
        ph = make_double2(cs, sn);
        phc = make_double2(cs, -sn);
    }
    int slot = 0;
    unsigned phase = 0;
    bool ok = true;  // a wait that ran out: the rest of the block is not a number
    for (int c = c0; c < c1; ++c) {
        if constexpr (TMA) {
            if (ok && (A.lost || !mbar_wait(smem_u32(full + slot), phase))) {
                ok = false;
                if (tid == 0)  // the columns under way land before the CTA ends
                    for (int k = c - c0; k < min(c1 - c0, c - c0 + S - 1); ++k)
                        if (!mbar_wait(smem_u32(full + k % S), (k / S) & 1)) break;
            }
        }
        else cp_async_wait<S - 2>();
        __syncthreads();
        if (ok) issue(c + S - 1, slot == 0 ? S - 1 : slot - 1);  // into the slot of column c - 1
        if (RES && warp == 0 && c > c0 && c - 1 < res_count) {
            double v = lane < CM_THREADS / 32 ? red[(c - 1) & 1][lane] : 0.0;
#pragma unroll
            for (int m = 8; m > 0; m >>= 1) v += __shfl_xor_sync(~0u, v, m);
            if (lane == 0) part[(int64_t)t * res_count + c - 1] = v;
        }
        const T* b = sm + slot * A.slot + o;
        double sum = 0.0;
        const double lm = RES && c < res_count ? lam[c] : 0.0;
        T ln[NP + 2], out[NP];
#pragma unroll
        for (int k = 0; k < NP + 2; ++k) ln[k] = b[k * pz];
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const T* p = b + (k + 1) * pz;
            const T zm = ln[k], xi = ln[k + 1], zp = ln[k + 2];
            T v;
            if constexpr (KIND == CK_CSR7) {
                T acc = s_fma(w[k][0], zm, s_zero(T()));
                acc = s_fma(w[k][1], p[-A.px], acc);
                acc = s_fma(w[k][2], p[-1], acc);
                acc = s_fma(w[k][3], xi, acc);
                acc = s_fma(w[k][4], p[1], acc);
                acc = s_fma(w[k][5], p[A.px], acc);
                acc = s_fma(w[k][6], zp, acc);
                v = s_mul(alpha, acc);
            } else {
                T nsum = s_add(s_zero(T()), p[-1]);
                nsum = s_add(nsum, p[1]);
                if constexpr (HY) {
                    if constexpr (CPLX) {
                        nsum = s_fma(ph, p[-A.px], nsum);
                        nsum = s_fma(phc, p[A.px], nsum);
                    } else {
                        nsum = s_add(nsum, p[-A.px]);
                        nsum = s_add(nsum, p[A.px]);
                    }
                }
                nsum = s_add(nsum, zm);
                nsum = s_add(nsum, zp);
                v = s_mul(alpha, s_add(s_rscale(d[k], xi), s_rscale(offd, nsum)));
            }
            out[k] = s_fma(beta, xi, v);
        }
        const int64_t col = (int64_t)c * ldy;
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            T v = out[k];
            if (in && gz + k < A.nz) {
                const int64_t i = row + k * plane;
                if (z) v = s_fma(gamma, z[i + (int64_t)c * ldz], v);
                v = s_rscale(scale, v);
                if (TMA && !ok) v = s_rscale(__longlong_as_double(0x7ff8000000000000ll), v);
                y[i + col] = v;
                if (RES) sum += s_abs2(resid_sub(lm, ln[k + 1], v));
            }
        }
        if (RES && c < res_count) {
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(~0u, sum, m);
            if (lane == 0) red[c & 1][warp] = sum;
        }
        if (++slot == S) {
            slot = 0;
            phase ^= 1;
        }
    }
    if (RES && c1 > c0 && c1 - 1 < res_count) {
        __syncthreads();
        if (tid == 0) {
            double v = 0.0;
            for (int k = 0; k < CM_THREADS / 32; ++k) v += red[(c1 - 1) & 1][k];
            part[(int64_t)t * res_count + c1 - 1] = v;
        }
    }
}

// Tile shape and columns per CTA: the fewest (CTAs per SM) x (columns, and a start of about five columns' time) x
// (points copied, and twice the points formed).
template <class T>
bool cm_plan(const rc_ctx* ctx, int kind, int64_t nx, int64_t ny, int64_t nz, int64_t s, bool tma, CmArgs* out, dim3* grid) {
    const int np = cm_points<T>(kind), tile = CM_THREADS * np, hy = kind == CK_STENCIL5 ? 0 : 2;
    double best = 0.0;
    for (int ltx = sizeof(T) == 16 ? 3 : 4; ltx <= 6; ++ltx)  // narrower rows: bank conflicts
        for (int tz = np; (tile >> ltx) / tz >= 1; tz *= 2) {
            CmArgs A = {};
            A.nx = (int)nx; A.ny = (int)ny; A.nz = (int)nz;
            A.tx = 1 << ltx; A.ltx = ltx; A.ty = (tile >> ltx) / tz; A.tz = tz;
            if (kind == CK_STENCIL5 && A.ty != 1) continue;
            // a TMA copy starts on 16 bytes, and a box has at most 256 of the map's 4-byte words a line
            A.hx = tma && sizeof(T) == 8 ? 2 : 1;
            A.px = A.tx + 2 * A.hx; A.py = A.ty + hy; A.box = A.px * A.py * (tz + 2);
            A.slot = (A.box * (int)sizeof(T) + 127) / 128 * (128 / (int)sizeof(T));
            if (tma ? A.px * (int)sizeof(T) / 4 > 256 || A.py > 256 || tz + 2 > 256 : A.box > CM_MAX_BOX) continue;
            if ((size_t)cm_slots<T>() * A.slot * sizeof(T) > CM_MAX_SMEM) continue;
            A.ntx = (int)((nx + A.tx - 1) / A.tx);
            A.nty = (int)((ny + A.ty - 1) / A.ty);
            const int64_t tiles = (int64_t)A.ntx * A.nty * ((nz + tz - 1) / tz);
            if (tiles > 0x7fffffff) continue;
            A.s = (int)s;
            for (int k = 1; k <= 16 && (s + k - 1) / k >= std::min<int64_t>(s, 8); ++k) {
                A.cols = (int)((s + k - 1) / k);
                const int64_t parts = (s + A.cols - 1) / A.cols, turns = (tiles * parts + ctx->sm_count - 1) / ctx->sm_count;
                const double cost = (double)turns * (A.cols + 5) * (A.box + 2 * tile);
                if (best == 0.0 || cost < best) {
                    best = cost;
                    *out = A;
                    *grid = dim3((unsigned)tiles, (unsigned)parts);
                }
            }
        }
    if (best == 0.0) return false;
    const double waste = (double)grid->x * (out->box + 2.0 * tile) / (3.0 * (double)nx * ny * nz);
    return ctx->tile > 1 || waste <= cm_max_waste<T>(kind == CK_CSR7);
}

template <class T, int KIND>
rc_status cm_launch(rc_ctx* ctx, const rc_op* op, const StepArgs& a, T alpha, T beta, T gamma, const double* lam,
                    int64_t res_count, const CmArgs& A, dim3 grid, const CUtensorMap* map, double* part, const void* weights) {
    const size_t smem = (size_t)cm_slots<T>() * A.slot * sizeof(T);
    const CUtensorMap none = {};
    const double theta = 2.0 * 3.14159265358979323846 * op->flux;
    auto run = [&](auto kern) -> rc_status {
        RC_CU(ctx, allow_max_smem(ctx, kern));
        kern<<<grid, CM_THREADS, smem, ctx->stream>>>(A, map ? *map : none, (const T*)a.x, a.ldx, (const T*)a.z, a.ldz, (T*)a.y, a.ldy,
                                                      alpha, beta, gamma, a.scale, (const RowWeights<T>*)weights,
                                                      op->diag64, op->offdiag, theta, lam, (int)res_count, part);
        ctx->launches++;
        ctx->tile_launches++;
        RC_CU(ctx, cudaGetLastError());
        return RC_OK;
    };
    if (map) return res_count > 0 ? run(cm_step_kernel<T, KIND, true, true>) : run(cm_step_kernel<T, KIND, false, true>);
    if constexpr (cm_copies<T>(KIND))
        return res_count > 0 ? run(cm_step_kernel<T, KIND, true, false>) : run(cm_step_kernel<T, KIND, false, false>);
    return RC_OK;
}

template <class T>
rc_status cm_step_t(rc_ctx* ctx, rc_op* op, const StepArgs& a, const double* lam, int64_t res_count, double** part,
                    int64_t* parts, bool* done) {
    const int kind = op->kind == 0 ? CK_CSR7 : (op->skind == 7 ? CK_STENCIL7 : CK_STENCIL5);
    const int64_t nx = kind == CK_CSR7 ? op->gx : op->nx;
    const int64_t ny = kind == CK_CSR7 ? op->gy : (kind == CK_STENCIL5 ? 1 : op->ny);
    const int64_t nz = kind == CK_CSR7 ? op->gz : (kind == CK_STENCIL5 ? op->ny : op->nz);
    CmArgs A;
    dim3 grid;
    // lines of x that start on 16 bytes everywhere come by TMA
    const bool tma = nx * sizeof(T) % 16 == 0 && a.ldx * sizeof(T) % 16 == 0 && (uintptr_t)a.x % 16 == 0 &&
               (uint64_t)a.ldx * sizeof(T) < (1ull << 40) && tensor_map_encode() != nullptr;
    if (!tma && !cm_copies<T>(kind)) return RC_OK;
    if (!cm_plan<T>(ctx, kind, nx, ny, nz, a.s, tma, &A, &grid)) return RC_OK;
    CUtensorMap map;
    if (tma) {
        constexpr int64_t W = sizeof(T) / 4;
        const int64_t dims[4] = {nx * W, ny, nz, a.s};
        const int box[4] = {A.px * (int)W, A.py, A.tz + 2, 1};
        if (!tma_map_words_4d(&map, a.x, dims, box, a.ldx * W)) return RC_OK;
    }
    A.lost = ctx->lost;
    const CUtensorMap* mp = tma ? &map : nullptr;
    double* pt = nullptr;
    if (res_count > 0) {
        void* p = nullptr;
        RC_TRY(rc_slot(ctx, S_RPART, (size_t)grid.x * res_count * sizeof(double), &p));
        *part = pt = (double*)p;
        *parts = grid.x;
    }
    // (after the allocation, which may take them back when memory is short)
    const void* weights = kind == CK_CSR7 ? tile_weights(ctx, op, false, op->n * a.s * (int64_t)sizeof(T)) : nullptr;
    if (kind == CK_CSR7 && !weights) return RC_OK;
    *done = true;
    T alpha, beta, gamma;
    if constexpr (IsComplex<T>::value) {
        alpha = make_double2(a.alpha[0], a.alpha[1]);
        beta = make_double2(a.beta[0], a.beta[1]);
        gamma = make_double2(a.gamma[0], a.gamma[1]);
    } else {
        alpha = a.alpha[0];
        beta = a.beta[0];
        gamma = a.gamma[0];
        if (kind == CK_STENCIL5)
            return cm_launch<T, CK_STENCIL5>(ctx, op, a, alpha, beta, gamma, lam, res_count, A, grid, mp, pt, weights);
    }
    if (kind == CK_CSR7)
        return cm_launch<T, CK_CSR7>(ctx, op, a, alpha, beta, gamma, lam, res_count, A, grid, mp, pt, weights);
    return cm_launch<T, CK_STENCIL7>(ctx, op, a, alpha, beta, gamma, lam, res_count, A, grid, mp, pt, weights);
}

}  // namespace

rc_status cm_step(rc_ctx* ctx, rc_op* op, const StepArgs& a, const double* lam, int64_t res_count, double** part,
                  int64_t* parts, bool* done) {
    *done = false;
    const bool cplx = op->dtype == RC_COMPLEX128;
    if (!ctx->tile || a.cp != P64 || a.xp != P64 || a.yp != P64 || (a.z && a.zp != P64)) return RC_OK;
    if (op->kind == 0 ? !(tile_rows(ctx, op, false) && ctx->csr_variant == 0)
                      : !(op->kind == 1 && (op->skind == 7 || (op->skind == 5 && !cplx))))
        return RC_OK;
    if (op->n > 0x7fffffff || a.s > 0x7fffffff) return RC_OK;  // row numbers of 31 bits
    if (ctx->tile == 1 && (a.s < 8 || op->n * a.s * (cplx ? 16 : 8) < kCmMinBytes)) return RC_OK;
    return cplx ? cm_step_t<double2>(ctx, op, a, lam, res_count, part, parts, done)
                : cm_step_t<double>(ctx, op, a, lam, res_count, part, parts, done);
}

}  // namespace rcb
