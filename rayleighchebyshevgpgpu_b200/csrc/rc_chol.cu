// rc_chol.cu -- T = D^-1 R^-1 of a Gram matrix G = D R^H R D (D from its diagonal, R upper triangular), so that V T has
// orthonormal columns: the small factor of CholeskyQR and of the fused Ritz step, up to 192 columns.
//
// One elimination forms both: with Gh = D^-1 G D^-1 = L P L^H (P the pivots), step k takes conj(M[k,i]) / p_k times row k
// from the rows i > k of M (its upper triangle) and of Y = L^-1 (starting from I), and R^-1 = Y^H P^-1/2. What M and Y
// need lies in one square, M above the diagonal and Y below; column k turns from the one into the other at step k (before
// it holds M's lower triangle, which nothing reads), so every row below k gets the same update in all columns. The square
// is kept in registers: warp ty of a CTA owns columns, lane
// tx rows tx, tx + 32, ... ; each step the owners of row k + 1 put it, and its pivot's reciprocal, into shared memory
// (double buffered), and one barrier follows. Up to 96 columns one CTA holds it; beyond, a cluster of four CTAs takes
// every fourth column each, and rows go to all four.
//
// Measured, with the kernel before (matrices in shared memory or L2, two loops of s steps, one for the inverse, 1024
// threads), us: real s = 24 9.1 (20), 36 16.5 (33), 48 21 (48), 72 38 (89), 96 51 (138), 192 152 (1250); complex 96 99
// (190), 192 239 (1530). With 32 warps of 3 x 3 entries s = 96 took 98: the warps' own reads and publishing were issued
// 32 times a step; with the pivot's reciprocal in a warp of its own 60.
//
// Bound: the steps' chain of a barrier, the row's reads, an update and a division, and the updates' instruction issue.
#include <algorithm>
#include <type_traits>
#include "rc_cluster.cuh"
#include "rc_common.cuh"
#include "rc_internal.h"

namespace rcb {

namespace {

constexpr int kCholOneCta = 96, kCholMax = 192, kCholCluster = 4;
constexpr int kCholWarps = 8;  // few: a warp's reads of the row and its share of a step's overhead serve more columns

__device__ __forceinline__ double lane_value(double v, int lane) { return __shfl_sync(~0u, v, lane); }
__device__ __forceinline__ double2 lane_value(double2 v, int lane) {
    return make_double2(__shfl_sync(~0u, v.x, lane), __shfl_sync(~0u, v.y, lane));
}

// NA: rows per lane, NB: columns per warp, C: CTAs of the cluster. flags, pivout: chol_factor (rc_internal.h).
template <class T, int NA, int NB, int C>
__global__ void __launch_bounds__(32 * kCholWarps, 1)
chol_kernel(int s, int64_t nrows, const T* __restrict__ G, T* __restrict__ Tout, int* flags, double* pivout) {
    __shared__ T row[2][32 * NA];
    __shared__ double inv[2], pv[2], rd[32 * NA], piv[32 * NA];  // rd: 1 / d
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    const int rank = C > 1 ? (int)cl_rank() : 0;
    for (int i = tid; i < s; i += blockDim.x) {
        const double gi = s_real(G[i + (int64_t)i * s]);
        double d = (gi > 0.0 && isfinite(gi)) ? sqrt(gi) : 0.0;
        if (d == 0.0) {
            if (rank == 0) atomicOr(flags + 2, 1);
            d = 1.0;
        }
        rd[i] = 1.0 / d;
    }
    for (int i = s + tid; i < 32 * NA; i += blockDim.x) row[0][i] = row[1][i] = s_zero(T());
    cl_sync<(C > 1)>();  // every CTA of the cluster runs from here on
    int jc[NB];          // this warp's columns
#pragma unroll
    for (int b = 0; b < NB; ++b) jc[b] = rank + C * (ty + kCholWarps * b);
    T e[NA][NB];
    const double eps = 2.220446049250313e-16;
    // Fukaya et al. shift 11 (m n + n (n+1)) u ||Gh||_2 with ||Gh||_2 <= trace(Gh) = s.
    const double sigma = 11.0 * ((double)nrows * s + (double)s * (s + 1)) * eps * (double)s;
    bool bad = false;
    for (int attempt = 0; attempt < 2; ++attempt) {
        const double shift = attempt == 0 ? 0.0 : sigma;
        bad = false;
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int a = 0; a < NA; ++a)  // all loads in flight together
                e[a][b] = G[min(tx + 32 * a, s - 1) + (int64_t)min(jc[b], s - 1) * s];
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int a = 0; a < NA; ++a) {
                const int i = tx + 32 * a, j = jc[b];
                T g = e[a][b];
                if (i > j || j >= s || !isfinite(s_real(g)) || !isfinite(s_imag(g))) g = s_zero(T());
                else g = s_rscale(rd[i] * rd[j], g);
                if (i == j) g = s_from<T>(s_real(g) + shift, 0.0);
                e[a][b] = g;
            }
        // row k, in the lanes' rows KA (a constant: e stays in registers)
        auto publish = [&](int k, auto ka) {
            constexpr int KA = decltype(ka)::value;
            // (columns past s go along: no branch in a lane's run of stores)
            if constexpr (C == 1) {
                if (tx == (k & 31)) {
#pragma unroll
                    for (int b = 0; b < NB; ++b) row[k & 1][jc[b]] = e[KA][b];
                }
            } else {  // lane C b + c stores the value of column b into CTA c
                T v = s_zero(T());
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    const T w = lane_value(e[KA][b], k & 31);
                    if (tx / C == b) v = jc[b] == k ? s_from<T>(1.0, 0.0) : w;
                }
                if (tx < C * NB) cl_store(cl_addr(&row[k & 1][rank + C * (ty + kCholWarps * (tx / C))], tx % C), v);
            }
            if (ty == (k / C) % kCholWarps && rank == k % C) {  // the pivot's owner: its place in the row holds 1
                double p = 0.0;
#pragma unroll
                for (int b = 0; b < NB; ++b)
                    if (jc[b] == k) p = s_real(e[KA][b]);
                if constexpr (C == 1) {
                    if (tx == (k & 31)) {
                        row[k & 1][k] = s_from<T>(1.0, 0.0);
                        pv[k & 1] = p;
                        inv[k & 1] = 1.0 / (p > 1e-300 ? p : 1e-300);
                    }
                } else {
                    p = lane_value(p, k & 31);
                    if (tx < C) {
                        cl_store(cl_addr(&pv[k & 1], tx), p);
                        cl_store(cl_addr(&inv[k & 1], tx), 1.0 / (p > 1e-300 ? p : 1e-300));
                    }
                }
            }
        };
        // the steps whose rows are the lanes' rows KA; false when the factor broke down
        auto steps = [&](auto ka) -> bool {
            constexpr int KA = decltype(ka)::value;
            const int end = min(s, 32 * KA + 32);
            for (int k = 32 * KA; k < end; ++k) {
                const T* rw = row[k & 1];
                const double p = pv[k & 1], pinv = inv[k & 1];
                T f[NA];
#pragma unroll
                for (int a = KA; a < NA; ++a) {
                    const int i = tx + 32 * a;
                    f[a] = i > k ? s_rscale(-pinv, s_conj(rw[i])) : s_zero(T());
                }
                if (ty == (k / C) % kCholWarps) {  // column k of Y starts from zero
#pragma unroll
                    for (int b = 0; b < NB; ++b)
                        if (jc[b] == k) {
#pragma unroll
                            for (int a = KA; a < NA; ++a) e[a][b] = s_zero(T());
                        }
                }
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    const T r = rw[jc[b]];
#pragma unroll
                    for (int a = KA; a < NA; ++a) e[a][b] = s_fma(f[a], r, e[a][b]);
                }
                if (k + 1 < end) publish(k + 1, ka);
                else if constexpr (KA + 1 < NA) {
                    if (k + 1 < s) publish(k + 1, std::integral_constant<int, KA + 1>{});
                }
                if (tid == 0) piv[k] = p;
                if (!(p > 1e-13)) bad = true;
                cl_sync<(C > 1)>();
                if (bad && attempt == 0) return false;
            }
            return true;
        };
        publish(0, std::integral_constant<int, 0>{});
        cl_sync<(C > 1)>();
        bool on = steps(std::integral_constant<int, 0>{});
        if constexpr (NA > 1) on = on && steps(std::integral_constant<int, 1>{});
        if constexpr (NA > 2) on = on && steps(std::integral_constant<int, 2>{});
        if constexpr (NA > 3) on = on && steps(std::integral_constant<int, 3>{});
        if constexpr (NA > 4) on = on && steps(std::integral_constant<int, 4>{});
        if constexpr (NA > 5) on = on && steps(std::integral_constant<int, 5>{});
        if (!bad) break;
        if (attempt == 0) {
            if (rank == 0 && tid == 0) flags[0] |= 1;
        } else if (rank == 0 && tid == 0) {
            flags[1] = 1;
        }
    }
    if (rank == 0 && ty == 0 && pivout) {
        double m = 1e300;
        for (int i = tx; i < s; i += 32) m = fmin(m, piv[i]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) m = fmin(m, __shfl_xor_sync(~0u, m, d));
        if (tx == 0) pivout[0] = m;
    }
    // T[j, i] = conj(Y[i, j]) / (d_j sqrt(p_i)) for j < i, zero below the diagonal
    double rp[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const double p = tx + 32 * a < s ? piv[tx + 32 * a] : 1.0;
        rp[a] = 1.0 / sqrt(p > 1e-300 ? p : 1e-300);
    }
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            const int i = tx + 32 * a, j = jc[b];
            if (i < s && j < s) {
                const double w = rd[j] * rp[a];
                Tout[j + (int64_t)i * s] =
                    i > j ? s_rscale(w, s_conj(e[a][b])) : (i == j ? s_from<T>(w, 0.0) : s_zero(T()));
            }
        }
}

template <class T>
rc_status chol_launch(rc_ctx* ctx, int64_t s, int64_t nrows, const void* G, void* Tout, int* flags, double* pivout) {
    const int c = s <= kCholOneCta ? 1 : kCholCluster;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c);
    cfg.blockDim = dim3((unsigned)(32 * kCholWarps));
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = c > 1 ? 1 : 0;
    auto run = [&](auto kern) -> rc_status {
        RC_CU(ctx, cudaLaunchKernelEx(&cfg, kern, (int)s, nrows, (const T*)G, (T*)Tout, flags, pivout));
        ctx->launches++;
        return RC_OK;
    };
    switch ((s + 31) / 32) {
        case 1: return run(chol_kernel<T, 1, 4, 1>);
        case 2: return run(chol_kernel<T, 2, 8, 1>);
        case 3: return run(chol_kernel<T, 3, 12, 1>);
        case 4: return run(chol_kernel<T, 4, 4, kCholCluster>);
        case 5: return run(chol_kernel<T, 5, 5, kCholCluster>);
        default: return run(chol_kernel<T, 6, 6, kCholCluster>);
    }
}

}  // namespace

bool chol_registers(rc_ctx* ctx, int dtype, int64_t s, int64_t nrows, const void* G, void* Tout, int* flags,
                    double* pivout, rc_status* st) {
    if (s < 1 || s > kCholMax) return false;
    *st = dtype == RC_COMPLEX128 ? chol_launch<double2>(ctx, s, nrows, G, Tout, flags, pivout)
                                 : chol_launch<double>(ctx, s, nrows, G, Tout, flags, pivout);
    return true;
}

}  // namespace rcb
