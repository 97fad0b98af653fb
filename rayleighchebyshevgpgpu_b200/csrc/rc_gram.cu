// rc_gram.cu -- tall-skinny symmetric (Hermitian) products G = X^H X and H = X^H W on the FP64 tensor pipe:
// the Gram matrix of CholeskyQR and the projected operator of the Ritz step. Only 8x8 tiles on and above the
// diagonal are formed (the reference's CPU formVtAV also forms the upper triangle, RayleighChebyshevLM.h:1928-1969;
// cublas{D,Z}gemm(OP_T/OP_C, OP_N), RayleighChebyshevLMCuda.h:2139-2161).
//
// A CTA walks its chunk of rows in slabs that one producer warp brings into a ring of shared-memory stages, one
// TMA tile copy per operand (rc_dmma.cuh; one bulk copy per column, 256 bytes, kept the pipe at 13 TFLOP/s of
// useful work at 96 columns). With T8 tile rows, product warp w of a set takes tile rows w and T8 - 1 - w of the
// upper triangle: T8 + 1 tiles, the same for every w, in registers for the whole chunk. Sets of warps differ in
// the product (G or H), for complex blocks in the part (Re or Im), or in the rows of a slab they take (KG groups,
// combined in shared memory at the end); a CTA holds up to 12 warps of them. Per-chunk partials are summed by
// gram_sum_kernel in a fixed order (deterministic).
//
// Fragments (g = lane / 4, q = lane % 4; A = X^T and B are read the same way, from X[k][c]):
//   column-major   one 16-byte read gives inner indices 2q and 2q + 1 of column 8 j + g: two mma;
//   odd ld         even and odd columns are tiles of their own, the odd ones from the 16-byte boundary before
//                  them, so that both have strides of 16 bytes: two 8-byte reads, k = q, q + 4, and tile j's
//                  columns in the order 0, 2, 4, 6, 1, 3, 5, 7;
//   row-major      two 8-byte reads, k = q, q + 4;
//   complex        one 16-byte read gives (re, im) of row q: Re += re re + im im, Im += re im - im re, the
//                  second with X's pair turned into (-im, re).
// The tiles are a little longer than a slab, so that their pitch in shared memory has no bank conflicts; what lies
// past the block is zero (TMA).
//
// Bound: the FP64 tensor pipe (37 TFLOP/s measured), HBM below about 50 columns. Measured, X^T X, with the
// kernels this one replaced (32x32 super-blocks of both triangles' diagonal blocks, cp.async by the product
// warps; SIMT for wider real blocks): 10^6 x 96 314 us (596; with an odd leading dimension 307, 795 before),
// 2x10^6 x 48 179 us (522), 2x10^6 x 24 85 us (200), 216,000 x 36 19 us (60), 500,000 x 192 753 us (2041),
// complex 442,368 x 96 534 us (752), X^H W x 192 2.22 ms (2.99); the sum over chunks 7-11 us (22-76).
#include <algorithm>
#include "rc_common.cuh"
#include "rc_dmma.cuh"
#include "rc_internal.h"

namespace rcb {

namespace {

enum { GL_CM = 0, GL_ODD = 1, GL_RM = 2 };
constexpr int GR_STAGES = 4, GR_WARPS = 12;

// Geometry in doubles. Column-major: SD doubles of a column per slab (a wide block's slabs are half as long), CP
// per column in shared memory; row-major: 32 rows per slab, CP per row. The pitches (8 mod 16 for 16-byte reads,
// 4 mod 16 for 8-byte ones) leave the fragment reads without bank conflicts.
template <int T8, int LAY>
struct GrGeo {
    static constexpr int SD = LAY != GL_RM && T8 > 12 ? 16 : 32;
    static constexpr int CP = LAY == GL_CM ? SD + 8 : (LAY == GL_ODD ? SD + 4 : (8 * T8 + 11) / 16 * 16 + 4);
    static constexpr int OP = LAY == GL_RM ? SD * CP : 8 * T8 * CP;  // doubles of an operand per stage
    static constexpr int STEPS = SD / 8;
};

template <int T8, int LAY>
__device__ __forceinline__ double2 gr_frag(const double* op, int j, int step, int g, int q) {
    using G = GrGeo<T8, LAY>;
    if constexpr (LAY == GL_CM) {
        return *reinterpret_cast<const double2*>(op + (8 * j + g) * G::CP + 8 * step + 2 * q);
    } else if constexpr (LAY == GL_ODD) {
        const int o = g >> 2;  // even columns, then odd ones, a row later
        const double* p = op + (o * 4 * T8 + 4 * j + (g & 3)) * G::CP + 8 * step + q + o;
        return make_double2(p[0], p[4]);
    } else {
        const double* p = op + (8 * step + q) * G::CP + 8 * j + g;
        return make_double2(p[0], p[4 * G::CP]);
    }
}
// Column of tile entry e (0..7).
template <int LAY>
__device__ __forceinline__ int gr_col(int e) { return LAY == GL_ODD ? 2 * (e & 3) + (e >> 2) : e; }

struct GrArgs {
    int64_t rows;        // rows per chunk, a multiple of the slab
    int64_t n;           // rows (complex: complex rows)
    int m;               // columns
    const double* X;     // leading dimensions in doubles
    int64_t lx;
    const double* W;
    int64_t lw;
    double* part;        // [set][chunk][m * m]
    int ops;             // operands per stage: 1 (X) or 2 (X and W)
    int sets;            // sets of warps per CTA that differ in the product or part
    int set0;            // first set of CTA row blockIdx.y (sets per row)
    int kg;              // groups over the rows of a slab
    int cplx;            // sets are Re, Im of X^H W (ops 2) or X^H X; else sets are X^T X, X^T W
    int only_w;          // real, one set: X^T W
    int stages;
    int aligned;         // TMA; else 8-byte copies (column-major)
    int lost;            // rc_ctx::lost
};
// X and W; with an odd leading dimension their even columns, then their odd ones.
struct GrMaps {
    CUtensorMap map[4];
};

// The product warps' loop over the chunk, for tile rows W and T8 - 1 - W.
template <int T8, int LAY, int W>
__device__ __forceinline__ void gr_rows(const GrArgs& A, const double* ring, int64_t slabs, uint32_t full, uint32_t empty,
                                        int set, int kgi, bool useW, bool im, int lane, double* comb, int warps, int* lost) {
    using G = GrGeo<T8, LAY>;
    constexpr int R1 = T8 - 1 - W;
    constexpr bool TWO = R1 > W;
    constexpr int NT = T8 - W + (TWO ? W + 1 : 0);
    const int g = lane >> 2, q = lane & 3;
    double acc[NT][2];
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = 0.0;
    const int stage = A.ops * G::OP;
    int b = 0;
    unsigned ph = 0;
    bool ok = !A.lost;
    if (!ok) slabs = 0;
    for (int64_t s = 0; s < slabs; ++s) {
        ok = mbar_wait_warp(full + 8 * b, ph);
        if (!ok) break;
        const double* xs = ring + b * stage;
        const double* ys = xs + (useW ? G::OP : 0);
#pragma unroll 1
        for (int step = kgi; step < G::STEPS; step += A.kg) {
            double2 a0 = gr_frag<T8, LAY>(xs, W, step, g, q), a1 = make_double2(0.0, 0.0);
            if (TWO) a1 = gr_frag<T8, LAY>(xs, R1, step, g, q);
            if (im) {
                a0 = make_double2(-a0.y, a0.x);
                a1 = make_double2(-a1.y, a1.x);
            }
#pragma unroll
            for (int j = W; j < T8; ++j) {
                const double2 v = gr_frag<T8, LAY>(ys, j, step, g, q);
                dmma(acc[j - W][0], acc[j - W][1], a0.x, v.x);
                if (TWO && j >= R1) dmma(acc[T8 - W + j - R1][0], acc[T8 - W + j - R1][1], a1.x, v.x);
                dmma(acc[j - W][0], acc[j - W][1], a0.y, v.y);
                if (TWO && j >= R1) dmma(acc[T8 - W + j - R1][0], acc[T8 - W + j - R1][1], a1.y, v.y);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + 8 * b);
        if (++b == A.stages) {
            b = 0;
            ph ^= 1;
        }
    }
    if (A.kg > 1) {  // the groups' sums, in order, through the ring (every slab has been read)
        constexpr int NP = (T8 + 1) / 2;
        asm volatile("bar.sync 1, %0;" ::"r"(warps * 32) : "memory");
        if (!ok && lane == 0) *lost = 1;
        double2* cb = reinterpret_cast<double2*>(comb) + ((set * NP + W) * (T8 + 1)) * 32 + lane;
        const int cs = A.sets * NP * (T8 + 1) * 32;
        if (kgi > 0) {
#pragma unroll
            for (int t = 0; t < NT; ++t) cb[(kgi - 1) * cs + t * 32] = make_double2(acc[t][0], acc[t][1]);
        }
        asm volatile("bar.sync 1, %0;" ::"r"(warps * 32) : "memory");
        if (kgi > 0) return;
        ok = *lost == 0;  // (any group)
        for (int k = 1; k < A.kg; ++k) {
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const double2 v = cb[(k - 1) * cs + t * 32];
                acc[t][0] += v.x;
                acc[t][1] += v.y;
            }
        }
    }
    double* P = A.part + ((size_t)(A.set0 * blockIdx.y + set) * gridDim.x + blockIdx.x) * (size_t)A.m * A.m;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        const int i = t < T8 - W ? W : R1, j = t < T8 - W ? W + t : R1 + t - (T8 - W);
        const int row = 8 * i + gr_col<LAY>(g);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int col = 8 * j + gr_col<LAY>(2 * q + h);
            if (row < A.m && col < A.m) P[row + (int64_t)col * A.m] = acc[t][h];
        }
    }
    if (ok) return;
    // a slab that never landed: the warp's tiles are NaN (written over them: to set or select the sums cost up to
    // kilobytes of spills)
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    for (int k = 0; k <= (TWO ? 1 : 0); ++k) {
        const int i = k ? R1 : W, row = 8 * i + gr_col<LAY>(g);
        for (int col = 8 * i + q; col < A.m; col += 4)
            if (row < A.m) P[row + (int64_t)col * A.m] = nan;
    }
}

template <int T8, int LAY, int W = 0>
__device__ __forceinline__ void gr_dispatch(int w, const GrArgs& A, const double* ring, int64_t slabs, uint32_t full,
                                            uint32_t empty, int set, int kgi, bool useW, bool im, int lane,
                                            double* comb, int warps, int* lost) {
    if constexpr (W < (T8 + 1) / 2) {
        if (w == W) gr_rows<T8, LAY, W>(A, ring, slabs, full, empty, set, kgi, useW, im, lane, comb, warps, lost);
        else gr_dispatch<T8, LAY, W + 1>(w, A, ring, slabs, full, empty, set, kgi, useW, im, lane, comb, warps, lost);
    }
}

template <int T8, int LAY>
__global__ void __launch_bounds__(32 * (GR_WARPS + 1), T8 <= 6 ? 2 : 1) gram_dmma_kernel(GrArgs A, const __grid_constant__ GrMaps M) {
    using G = GrGeo<T8, LAY>;
    extern __shared__ __align__(128) double grsm[];
    __shared__ __align__(8) uint64_t bars[2 * GR_STAGES];
    __shared__ int lost;  // a group's wait ran out
    constexpr int NP = (T8 + 1) / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int warps = NP * A.sets * A.kg;
    const uint32_t full = smem_u32(bars), empty = full + 8 * GR_STAGES;
    if (threadIdx.x == 0) {
        lost = 0;
        for (int s = 0; s < A.stages; ++s) {
            mbar_init(full + 8 * s, A.aligned ? 1 : 33);
            mbar_init(empty + 8 * s, warps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // a slab: SD doubles of each column (row-major: SD rows); rows counted in doubles of a column
    const int64_t cw = A.cplx ? 2 : 1;
    const int64_t r_begin = (int64_t)blockIdx.x * A.rows * cw;
    const int64_t r_end = min(A.n, ((int64_t)blockIdx.x + 1) * A.rows) * cw;
    const int64_t slabs = r_end > r_begin ? (r_end - r_begin + G::SD - 1) / G::SD : 0;
    if (warp < warps) {
        const int w = warp % NP, h = warp / NP, set = h % A.sets, kgi = h / A.sets;
        const int gset = A.set0 * blockIdx.y + set;  // which product (real) or part (complex)
        const bool useW = A.cplx ? A.ops == 2 : (A.only_w || gset == 1);
        gr_dispatch<T8, LAY>(w, A, grsm, slabs, full, empty, set, kgi, useW, A.cplx && gset == 1, lane, grsm, warps, &lost);
        return;
    }
    // the producer
    const int stage = A.ops * G::OP;
    int b = 0;
    unsigned ph = 0;
    int64_t used = 0;
    for (int64_t s = 0; s < slabs; ++s) {
        if (used >= A.stages && (A.lost || !mbar_wait(empty + 8 * b, ph ^ 1))) break;
        const uint32_t bar = full + 8 * b;
        double* st = grsm + b * stage;
        const int64_t r0 = r_begin + s * G::SD;
        if (A.aligned) {
            if (lane == 0) {
                mbar_arrive_tx(bar, (unsigned)(A.ops * G::OP * sizeof(double)));
                for (int o = 0; o < A.ops; ++o) {
                    double* d = st + o * G::OP;
                    if constexpr (LAY == GL_RM) {
                        tma_load_2d(smem_u32(d), &M.map[o], 0, (int)r0, bar);
                    } else if constexpr (LAY == GL_ODD) {
                        tma_load_2d(smem_u32(d), &M.map[o], (int)r0, 0, bar);
                        tma_load_2d(smem_u32(d + G::OP / 2), &M.map[2 + o], (int)r0, 0, bar);
                    } else {
                        tma_load_2d(smem_u32(d), &M.map[o], (int)r0, 0, bar);
                    }
                }
            }
            __syncwarp();
        } else {
            const int valid = (int)min((int64_t)G::SD, r_end - r0);
            for (int o = 0; o < A.ops; ++o) {
                const double* src = o ? A.W : A.X;
                const int64_t ld = o ? A.lw : A.lx;
                for (int c = 0; c < A.m; ++c)
                    for (int r = lane; r < G::SD; r += 32)
                        cp_async8(st + o * G::OP + c * G::CP + r, r < valid ? src + r0 + r + c * ld : src, r < valid ? 8 : 0);
            }
            cp_async_arrive(bar);
            if (lane == 0) mbar_arrive(bar);
        }
        ++used;
        if (++b == A.stages) {
            b = 0;
            ph ^= 1;
        }
    }
    for (int s = 0; s < A.stages && s < used; ++s) {  // copies still in flight land before the CTA ends
        if (--b < 0) {
            b = A.stages - 1;
            ph ^= 1;
        }
        if (!mbar_wait(full + 8 * b, ph)) break;
    }
    cp_async_wait0();
}

// C[i,j] (i <= j) = the sum over chunks, mirrored to exact symmetry (complex: set 0 is the real part, set 1 the
// imaginary one, diagonal real). 8 threads share an entry's chunks and add up in a fixed order.
__global__ void __launch_bounds__(256) gram_sum_kernel(int m, int chunks, int ny, int cplx, const double* __restrict__ part,
                                                       double* __restrict__ C0, double* __restrict__ C1) {
    __shared__ double sh[8][33];
    const int64_t total = (int64_t)m * m;
    const int64_t e = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
    const int t = threadIdx.x >> 5, y = blockIdx.y;
    const int i = (int)(e % m), j = (int)(e / m);
    const bool on = e < total && i <= j;
    double s = 0.0;
    if (on) {
        const double* p = part + (size_t)y * chunks * total + e;
#pragma unroll 4
        for (int c = t; c < chunks; c += 8) s += p[(size_t)c * total];
    }
    sh[t][threadIdx.x & 31] = s;
    __syncthreads();
    if (t != 0 || !on) return;
    for (int k = 1; k < 8; ++k) s += sh[k][threadIdx.x & 31];
    if (cplx) {
        if (y == 1 && i == j) s = 0.0;
        C0[2 * e + y] = s;
        C0[2 * (j + (int64_t)i * m) + y] = y ? -s : s;
    } else {
        double* C = y == 0 ? C0 : C1;
        C[e] = s;
        C[j + (int64_t)i * m] = s;
    }
}

template <int T8, int LAY>
rc_status gr_launch(rc_ctx* ctx, GrArgs A, double* C0, double* C1) {
    using G = GrGeo<T8, LAY>;
    constexpr int NP = (T8 + 1) / 2;
    GrMaps M = {};
    if (A.aligned) {
        const int64_t rows = A.cplx ? 2 * A.n : A.n;
        for (int o = 0; o < A.ops; ++o) {
            const double* p = o ? A.W : A.X;
            const int64_t ld = o ? A.lw : A.lx;
            bool ok;
            if (LAY == GL_RM) {
                ok = tma_map_2d(&M.map[o], p, A.m, rows, ld, G::CP, G::SD);
            } else if (LAY == GL_ODD) {
                ok = tma_map_2d(&M.map[o], p, rows, (A.m + 1) / 2, 2 * ld, G::CP, 4 * T8);
                // column 1 on, from the 16-byte boundary before it (one column: nothing to read, any valid map)
                ok = ok && (A.m > 1 ? tma_map_2d(&M.map[2 + o], p + ld - 1, rows + 1, A.m / 2, 2 * ld, G::CP, 4 * T8)
                                    : tma_map_2d(&M.map[2 + o], p, rows, 1, 2 * ld, G::CP, 4 * T8));
            } else {
                ok = tma_map_2d(&M.map[o], p, rows, A.m, ld, G::CP, 8 * T8);
            }
            if (!ok) return rc_fail(ctx, RC_ERR_CUDA, "gram: cuTensorMapEncodeTiled failed");
        }
    }
    const int sets_all = A.sets;
    // sets per CTA: all of them where their warps fit, else one (complex blocks past 96 columns)
    if (NP * A.sets > GR_WARPS) A.sets = 1;
    A.set0 = A.sets;
    const int gy = sets_all / A.sets;
    A.kg = 1;
    while (2 * A.kg <= G::STEPS && 2 * A.kg * NP * A.sets <= GR_WARPS) A.kg *= 2;
    const int warps = NP * A.sets * A.kg;
    const size_t stage = (size_t)A.ops * G::OP * sizeof(double);
    const size_t comb = (size_t)(A.kg - 1) * A.sets * NP * (T8 + 1) * 32 * 16;
    // resident CTAs: by registers (T8 <= 6: two), and by three stages each in shared memory
    const size_t sm = ctx->smem_optin + 1024;
    int per_sm = T8 <= 6 ? 2 : 1;
    if (T8 <= 3) per_sm = std::max(2, 16 / (warps + 1));
    while (per_sm > 1 && (3 * stage + 1536) * per_sm > sm) --per_sm;
    const size_t room = sm / per_sm - 1536;
    A.stages = (int)std::max<size_t>(2, std::min<size_t>(GR_STAGES, room / stage));
    const size_t smem = std::max(A.stages * stage, comb);
    const int slab = G::SD / (A.cplx ? 2 : 1);
    int64_t chunks = std::max<int64_t>(1, (int64_t)ctx->sm_count * per_sm / gy);
    A.rows = ((A.n + chunks - 1) / chunks + slab - 1) / slab * slab;
    chunks = (A.n + A.rows - 1) / A.rows;
    void* part = nullptr;
    RC_TRY(rc_slot(ctx, S_PART, (size_t)sets_all * chunks * A.m * A.m * sizeof(double), &part));
    A.part = (double*)part;
    RC_CU(ctx, allow_max_smem(ctx, gram_dmma_kernel<T8, LAY>));
    gram_dmma_kernel<T8, LAY><<<dim3((unsigned)chunks, (unsigned)gy), 32 * (warps + 1), smem, ctx->stream>>>(A, M);
    ctx->launches++;
    RC_CU(ctx, cudaGetLastError());
    const dim3 grid((unsigned)(((int64_t)A.m * A.m + 31) / 32), (unsigned)sets_all);
    gram_sum_kernel<<<grid, 256, 0, ctx->stream>>>(A.m, (int)chunks, sets_all, A.cplx, A.part, C0, C1);
    ctx->launches++;
    RC_CU(ctx, cudaGetLastError());
    return RC_OK;
}

template <int LAY>
rc_status gr_width(rc_ctx* ctx, const GrArgs& A, double* C0, double* C1) {
    const int t = (A.m + 7) / 8;
    if (t <= 1) return gr_launch<1, LAY>(ctx, A, C0, C1);
    if (t <= 2) return gr_launch<2, LAY>(ctx, A, C0, C1);
    if (t <= 3) return gr_launch<3, LAY>(ctx, A, C0, C1);
    if (t <= 4) return gr_launch<4, LAY>(ctx, A, C0, C1);
    if (t <= 5) return gr_launch<5, LAY>(ctx, A, C0, C1);
    if (t <= 6) return gr_launch<6, LAY>(ctx, A, C0, C1);
    if (t <= 8) return gr_launch<8, LAY>(ctx, A, C0, C1);
    if (t <= 10) return gr_launch<10, LAY>(ctx, A, C0, C1);
    if (t <= 12) return gr_launch<12, LAY>(ctx, A, C0, C1);
    if constexpr (LAY != GL_RM) {
        if (t <= 16) return gr_launch<16, LAY>(ctx, A, C0, C1);
        if (t <= 20) return gr_launch<20, LAY>(ctx, A, C0, C1);
        if (t <= 24) return gr_launch<24, LAY>(ctx, A, C0, C1);
    }
    return rc_fail(ctx, RC_ERR_UNSUPPORTED, "gram: block too wide");
}

}  // namespace

bool gram_dmma_supported(int64_t m, bool rm) { return m >= 1 && m <= (rm ? 96 : 192); }

// Products of the n x m block X with itself and / or with W (complex: one of them): CX = X^H X, CW = X^H W.
rc_status gram_dmma(rc_ctx* ctx, int dtype, int64_t n, int64_t m, const void* X, int64_t ldx, void* CX, const void* W,
                    int64_t ldw, void* CW, bool rm) {
    const bool cplx = dtype == RC_COMPLEX128;
    if (!gram_dmma_supported(m, rm) || (cplx && rm)) return rc_fail(ctx, RC_ERR_UNSUPPORTED, "gram: block too wide");
    if (cplx && CX && CW) {
        RC_TRY(gram_dmma(ctx, dtype, n, m, X, ldx, CX, nullptr, 0, nullptr, false));
        return gram_dmma(ctx, dtype, n, m, X, ldx, nullptr, W, ldw, CW, false);
    }
    if (!W || W == X) {  // X^H X only
        if (W == X && CW && ldw == ldx) CX = CW;
        W = nullptr;
        CW = nullptr;
    }
    GrArgs A = {};
    A.n = n;
    A.m = (int)m;
    A.lost = ctx->lost;
    A.X = (const double*)X;
    A.lx = cplx ? 2 * ldx : ldx;
    A.W = (const double*)W;
    A.lw = cplx ? 2 * ldw : ldw;
    A.ops = CW ? 2 : 1;
    A.cplx = cplx;
    A.sets = cplx ? 2 : (CX && CW ? 2 : 1);
    A.only_w = !cplx && CW && !CX;
    double* C0 = (double*)(CX ? CX : CW);
    double* C1 = (double*)(CX && CW ? CW : nullptr);
    const bool base16 = (uintptr_t)X % 16 == 0 && (!CW || (uintptr_t)W % 16 == 0);
    if (rm) {
        if (!base16 || ldx % 2 || ldx < m || (CW && (ldw % 2 || ldw < m)))
            return rc_fail(ctx, RC_ERR_INVALID, "gram: row-major blocks need even leading dimensions >= m, 16-byte aligned");
        if (n + 64 >= INT32_MAX) return rc_fail(ctx, RC_ERR_UNSUPPORTED, "gram: too many rows");
        A.aligned = 1;
        return gr_width<GL_RM>(ctx, A, C0, C1);
    }
    const bool even = A.lx % 2 == 0 && (!CW || A.lw % 2 == 0);
    const bool odd = A.lx % 2 != 0 && (!CW || A.lw % 2 != 0);
    // tile coordinates and extents are 32-bit, strides below 2^40 bytes
    A.aligned = base16 && (even || odd) && 2 * n + 64 < INT32_MAX && std::max(A.lx, A.lw) < ((int64_t)1 << 35);
    return A.aligned && odd ? gr_width<GL_ODD>(ctx, A, C0, C1) : gr_width<GL_CM>(ctx, A, C0, C1);
}

}  // namespace rcb
