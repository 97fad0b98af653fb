// rc_jacobi.cu -- the small Hermitian eigensolve of the Rayleigh-Ritz step in the shared memory of one
// cluster: parallel cyclic Jacobi (Brent & Luk, round-robin ordering), replacing host DSYEV/ZHPEVX
// (RayleighChebyshevLMCuda.h:570-642) and JacobiDiagonalizer.
//
// A sweep is a tournament of M = sp - 1 rounds over sp (even) indices; in round r pair i meets the indices
// top(i) = (r + i) mod M and bottom(i) = (r - i) mod M, pair 0 meets r and sp - 1. From one round to the
// next the tops move down one pair and the bottoms up one pair. So CTA c of the cluster keeps the columns
// of A and of Q (A Q = Q Lambda) of the pairs c P .. c P + P - 1 in shared memory and, per round, passes one
// top column to CTA c - 1 and one bottom column to CTA c + 1 (at the ends of the cluster into the other
// row); the rest stays in place, the rows of slots being rings whose heads move. All updates then read
// local memory:
//   angles    every CTA finds the rotations of its own pairs from its own columns and writes them to every
//             CTA of the cluster; meanwhile its other warps apply the last round's rotations to its columns
//             of Q, which no angle depends on;
//   update    A <- G^H A G on its own columns: thread (row pair i, own pair j) forms the 2x2 block
//             A[{p_i,q_i},{p_j,q_j}] <- G_i^H A G_j.
// with a cluster barrier after each (a CTA barrier when the cluster is one CTA). A column that leaves is
// stored straight into the neighbour's free slot.
//
// The bound is latency (two barriers, one angle's chain and one block's per round) and, for wide complex
// matrices, instruction issue, which the cluster divides: 0.6 us per round at s = 24 (one CTA), 1.5 at s = 96,
// 2.5 at s = 192 complex. The kernels before it kept A and Q in one CTA's shared memory (1024 threads, half of
// A updated and mirrored: 1.4 us per round at s = 24, 3 us at s = 96), or, when they did not fit (complex
// s > 82, real s > 118), in L2 for 32 CTAs with a grid barrier (10 us per round at s = 192 complex); the latter
// still serves what sixteen SMs cannot hold (complex s > 320, real s > 470).
//
// Rotation of pair (p, q): with d = a_qq - a_pp, h = 2 |a_pq| and r = 1 / sqrt(d^2 + h^2), the inner angle
// has cos 2t = |d| r and sin 2t = h r; with w = 1 / sqrt(2 (1 + cos 2t)), cos t = (1 + cos 2t) w and
// sin t = sin 2t w (half-angle formulas; two reciprocal square roots, no division). The complex sine is
// sgn(d) 2 r w a_pq. For small angles that cosine is often one ulp low, which every later sweep would multiply into the
// columns, so its last bit is taken from c^2 + |sin t|^2 = 1 (jc_unit; no change in time). Mean error of the squared
// column norms and of the eigenvalues (to the norm), with and without it: s = 24 real 7e-17 and 2.2e-16, 1.2e-15 and
// 5.2e-16; 192 complex 2.5e-16 and 4.6e-16, 1.2e-14 and 3.1e-15 (the kernels before: 4e-17 and 2.6e-16; 2.6e-14 and
// 7.1e-15). The matrix is first scaled by a power of two to entries of at most 1 (exact), so that the
// squares neither overflow nor underflow.
#include <algorithm>
#include "rc_cluster.cuh"
#include "rc_common.cuh"
#include "rc_internal.h"

namespace rcb {

namespace {

// The cosine with which c^2 + |t|^2 is 1 to the last bit, for c that is off by rounding (first order: c >= 0.7).
__device__ __forceinline__ double jc_unit(double c, double t) {
    return fma(0.5, fma(-t, t, fma(-c, c, 1.0)), c);
}
__device__ __forceinline__ double jc_unit(double c, double2 t) {
    return fma(0.5, fma(-t.y, t.y, fma(-t.x, t.x, fma(-c, c, 1.0))), c);
}
// The same shared-memory location in CTA `rank` of the cluster, as a generic address.
template <class U>
__device__ __forceinline__ U* jc_at(U* p, unsigned rank) {
    unsigned long long a = (unsigned long long)p, o;
    asm("mapa.u64 %0, %1, %2;" : "=l"(o) : "l"(a), "r"(rank));
    return (U*)o;
}
// c x - conj(t) y and t x + c y
__device__ __forceinline__ double jc_lo(double c, double t, double x, double y) { return fma(c, x, -t * y); }
__device__ __forceinline__ double jc_hi(double c, double t, double x, double y) { return fma(c, y, t * x); }
__device__ __forceinline__ double2 jc_lo(double c, double2 t, double2 x, double2 y) {
    return make_double2(fma(c, x.x, fma(-t.x, y.x, -t.y * y.y)), fma(c, x.y, fma(-t.x, y.y, t.y * y.x)));
}
__device__ __forceinline__ double2 jc_hi(double c, double2 t, double2 x, double2 y) {
    return make_double2(fma(c, y.x, fma(t.x, x.x, -t.y * x.y)), fma(c, y.y, fma(t.x, x.y, t.y * x.x)));
}
__device__ __forceinline__ double jc_block_max(double v, double* sc) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sc[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = sc[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) t = fmax(t, sc[w]);
    return t;
}
__device__ __forceinline__ double jc_maxabs(double v) { return fabs(v); }
__device__ __forceinline__ double jc_maxabs(double2 v) { return fmax(fabs(v.x), fabs(v.y)); }

// Whether a pair rotates: |a_pq| above the absolute threshold (squared) and the relative one.
__device__ __forceinline__ bool jc_rotates(double m2, double app, double aqq, double abs2) {
    constexpr double rel2 = 1e-15 * 1e-15;
    return m2 > abs2 && m2 > rel2 * fabs(app * aqq);
}

constexpr int kJcThreadsMax = 512;  // 128 registers; 672 and 768 threads were no faster

__device__ __forceinline__ bool jc_nonzero(double v) { return (__double2hiint(v) | __double2loint(v)) != 0; }
__device__ __forceinline__ bool jc_nonzero(double2 v) {
    return (__double2hiint(v.x) | __double2loint(v.x) | __double2hiint(v.y) | __double2loint(v.y)) != 0;
}

template <class T>
constexpr size_t jc_col_bytes(int sp) { return 2 * (size_t)sp * sizeof(T); }
// tops and bottoms with a free slot each, the fixed column; rotations, diagonal, exchange words
template <class T>
size_t jc_smem(int P, int C) {
    const int sp = 2 * P * C;
    return (2 * (size_t)(P + 1) + 1) * jc_col_bytes<T>(sp) + (size_t)sp * (sizeof(T) + 8) + (size_t)sp * 8 + 16 * 8 + 64;
}

// CL: a cluster of more than one CTA.
template <class T, bool CL>
__global__ void __launch_bounds__(kJcThreadsMax, 1)
jacobi_cluster_kernel(int s, int P, int C, const T* __restrict__ Ain, T* __restrict__ Qout, double* __restrict__ evals,
                      int* info, int max_sweeps) {
    extern __shared__ __align__(16) unsigned char jcs[];
    __shared__ double sc[32];
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const int rank = CL ? (int)cl_rank() : 0;
    const int np = P * C, sp = 2 * np, M = sp - 1, S = P + 1;
    const int csz = 2 * sp;                  // a column: sp rows of A, then sp rows of Q
    T* tops = (T*)jcs;
    T* bots = tops + S * csz;
    T* fixed = bots + S * csz;               // index sp - 1, in CTA 0
    T* rs2 = fixed + csz;                    // rotation of each pair, of this round and the last: complex sine,
    double* rc2 = (double*)(rs2 + 2 * np);   // cosine
    double* diag = rc2 + 2 * np;             // diagonal by index (at sweep starts and at the end)
    double* ex = diag + sp;                  // one word per CTA, exchanged
    const int i0 = rank * P;                 // first own pair

    auto top_index = [&](int r, int i) { const int x = r + i; return x >= M ? x - M : x; };
    auto bot_index = [&](int r, int i) { const int x = r - i; return i == 0 ? sp - 1 : (x < 0 ? x + M : x); };
    int th = 0, bh = 0;                      // heads of the rings of slots
    auto top_at = [&](int t0, int j) { const int x = t0 + j; return tops + (x >= S ? x - S : x) * csz; };
    auto bot_at = [&](int b0, int j) {
        const int x = b0 + j;
        return rank == 0 && j == 0 ? fixed : bots + (x >= S ? x - S : x) * csz;
    };
    // own column f of the first round's arrangement: its index and its place
    auto own_index = [&](int f) { return f < P ? top_index(0, i0 + f) : bot_index(0, i0 + f - P); };
    auto own_col = [&](int f) { return f < P ? top_at(th, f) : bot_at(bh, f - P); };
    // a value of this CTA to every CTA's ex[rank]
    auto share = [&](double v) {
        cl_sync<CL>();
        if (tid < C) (CL ? jc_at(ex, tid) : ex)[rank] = v;
        cl_sync<CL>();
    };
    auto share_diag = [&]() {
        for (int e = tid; e < 2 * P * C; e += nt) {
            const int k = e / (2 * P), f = e - k * 2 * P, x = own_index(f);
            (CL ? jc_at(diag, k) : diag)[x] = s_real(own_col(f)[x]);
        }
        cl_sync<CL>();
    };

    // the columns of round 0, a warp per column
    double mx = 0.0;
    for (int f = warp; f < 2 * P; f += nw) {
        const int x = own_index(f);
        T* col = own_col(f);
#pragma unroll 4
        for (int e = lane; e < sp; e += 32) {
            const T v = e < s && x < s ? Ain[e + (int64_t)x * s] : s_zero(T());
            col[e] = v;
            col[sp + e] = s_from<T>(e == x ? 1.0 : 0.0, 0.0);
            mx = fmax(mx, jc_maxabs(v));
        }
    }
    mx = jc_block_max(mx, sc);
    share(mx);
    for (int k = 0; k < C; ++k) mx = fmax(mx, ex[k]);
    int shift = 0;  // entries times 2^-shift
    if (mx > 0.0 && isfinite(mx)) frexp(mx, &shift);
    const double up = ldexp(1.0, -shift / 2), up2 = ldexp(1.0, -shift - (-shift / 2));  // 2^-shift in two factors
    double f2 = 0.0;
    for (int f = warp; f < 2 * P; f += nw) {
        T* col = own_col(f);
        for (int e = lane; e < sp; e += 32) {
            const T v = s_rscale(up2, s_rscale(up, col[e]));
            col[e] = v;
            f2 += s_abs2(v);
        }
    }
    f2 = block_sum(f2, sc);
    share(f2);
    f2 = 0.0;
    for (int k = 0; k < C; ++k) f2 += ex[k];
    const double abs2 = 1e-34 * f2;

    // The first warps find the angles; the others have Q. A thread keeps its row pair of A and its row of Q and
    // walks over own pairs.
    const int na = (np + 31) & ~31, nq = nt - na, tq = tid - na;
    const int a_dj = nt / np, a_i = tid % np, a_j = tid < a_dj * np ? tid / np : P;
    const int q_dj = nq >= s ? nq / s : 1, q_dr = nq >= s ? s : nq;
    const int q_r = tq >= 0 ? (nq >= s ? tq % s : tq) : s, q_j = tq >= 0 && nq >= s ? tq / s : 0;
    const bool q_on = tq >= 0 && q_j < q_dj;
    // slot after (d = 1) or before (d = -1) x in the rings
    auto step = [&](int x, int d) { return d > 0 ? (x + 1 == S ? 0 : x + 1) : (x == 0 ? S - 1 : x - 1); };
    // where the columns that leave go, with the heads at t0 and b0: the free slots of the neighbours (at the
    // ends of the cluster, of the own other row)
    auto leave_top = [&](int t0, int b0) {
        return rank == 0 ? cl_addr(bots + b0 * csz, 0) : cl_addr(tops + (t0 + P >= S ? t0 + P - S : t0 + P) * csz, rank - 1);
    };
    auto leave_bot = [&](int t0, int b0) {
        return rank == C - 1 ? cl_addr(tops + (t0 + P >= S ? t0 + P - S : t0 + P) * csz, rank)
                             : cl_addr(bots + step(b0, -1) * csz, rank + 1);
    };
    const bool moves = M > 1;
    // Q <- Q G with the rotations of table half h, the heads at t0 and b0
    auto update_q = [&](int h, int t0, int b0) {
        if (!q_on) return;
        const T* rs = rs2 + h * np + i0;
        const double* rc = rc2 + h * np + i0;
        const uint32_t otop = leave_top(t0, b0) + sp * sizeof(T), obot = leave_bot(t0, b0) + sp * sizeof(T);
        for (int row = q_r; row < s; row += q_dr) {
#pragma unroll 2
            for (int j = q_j; j < P; j += q_dj) {
                T* cp = top_at(t0, j) + sp + row;
                T* cq = bot_at(b0, j) + sp + row;
                const T sj = rs[j];
                const double cj = rc[j];
                const bool lt = moves && j == 0, lb = moves && j == P - 1;
                if (jc_nonzero(sj) || lt || lb) {
                    const T qp = *cp, qq = *cq;
                    const T n_p = jc_lo(cj, sj, qp, qq), n_q = jc_hi(cj, sj, qp, qq);
                    if (lt) cl_store(otop + row * sizeof(T), n_p);
                    else *cp = n_p;
                    if (lb) cl_store(obot + row * sizeof(T), n_q);
                    else *cq = n_q;
                }
            }
        }
    };
    int sweep = 0;
    for (; sweep < max_sweeps; ++sweep) {
        // a sweep in which no pair rotates changes nothing: stop before it
        share_diag();
        bool any = false;
        for (int f = warp; f < 2 * P; f += nw) {
            const int x = own_index(f);
            if (x >= s) continue;
            const T* col = own_col(f);
            const double dx = diag[x];
#pragma unroll 2
            for (int e = lane; e < x; e += 32) any |= jc_rotates(s_abs2(col[e]), diag[e], dx, abs2);
        }
        share(__syncthreads_or(any) ? 1.0 : 0.0);
        any = false;
        for (int k = 0; k < C; ++k) any |= ex[k] != 0.0;
        if (!any) break;

        double mysn = 0.0;  // largest squared sine of this thread's angles
        for (int r = 0; r < M; ++r) {
            T* rs = rs2 + (r & 1) * np;
            double* rc = rc2 + (r & 1) * np;
            // angles: thread (k, j) finds the rotation of own pair j and writes it to CTA k
            if (tid < np) {
                const int k = tid / P, j = tid - k * P;
                const int p = top_index(r, i0 + j), q = bot_index(r, i0 + j);
                double c = 1.0;
                T sn = s_zero(T());
                if (p < s && q < s) {
                    const T* cp = top_at(th, j);
                    const T* cq = bot_at(bh, j);
                    const T apq = cq[p];
                    const double app = s_real(cp[p]), aqq = s_real(cq[q]);
                    const double m2 = s_abs2(apq);
                    if (jc_rotates(m2, app, aqq, abs2)) {
                        const double d = aqq - app;
                        const double rr = rsqrt(fma(d, d, 4.0 * m2));
                        const double c1 = fma(fabs(d), rr, 1.0);  // 1 + cos 2t
                        const double w = rsqrt(2.0 * c1);
                        c = c1 * w;
                        sn = s_rscale(copysign(2.0 * rr * w, d), apq);
                        mysn = fmax(mysn, s_abs2(sn));
                        c = jc_unit(c, sn);
                    }
                }
                if constexpr (CL) {
                    cl_store(cl_addr(rc + i0 + j, k), c);
                    cl_store(cl_addr(rs + i0 + j, k), sn);
                } else {
                    rc[j] = c;
                    rs[j] = sn;
                }
            }
            if (r > 0) update_q((r - 1) & 1, step(th, -1), step(bh, 1));
            cl_sync<CL>();
            if (a_j < P) {
                const int p = top_index(r, a_i), q = bot_index(r, a_i);
                const double ci = rc[a_i];
                const T si = rs[a_i];
                const bool ri = jc_nonzero(si);
                const uint32_t otop = leave_top(th, bh), obot = leave_bot(th, bh);
#pragma unroll 2
                for (int j = a_j; j < P; j += a_dj) {
                    T* cp = top_at(th, j);
                    T* cq = bot_at(bh, j);
                    const double cj = rc[i0 + j];
                    const T sj = rs[i0 + j];
                    const bool lt = moves && j == 0, lb = moves && j == P - 1;
                    if (ri || jc_nonzero(sj) || lt || lb) {
                        T a_pp = cp[p], a_qp = cp[q], a_pq = cq[p], a_qq = cq[q];
                        const T b_pp = jc_lo(cj, sj, a_pp, a_pq), b_pq = jc_hi(cj, sj, a_pp, a_pq);
                        const T b_qp = jc_lo(cj, sj, a_qp, a_qq), b_qq = jc_hi(cj, sj, a_qp, a_qq);
                        // rows: conj(si) and si change places
                        a_pp = jc_lo(ci, s_conj(si), b_pp, b_qp);
                        a_qp = jc_hi(ci, s_conj(si), b_pp, b_qp);
                        a_pq = jc_lo(ci, s_conj(si), b_pq, b_qq);
                        a_qq = jc_hi(ci, s_conj(si), b_pq, b_qq);
                        if (a_i == i0 + j && ri) {  // the rotated pair itself: exact zeros, real diagonal
                            a_qp = s_zero(T());
                            a_pq = s_zero(T());
                            a_pp = s_from<T>(s_real(a_pp), 0.0);
                            a_qq = s_from<T>(s_real(a_qq), 0.0);
                        }
                        if (lt) {
                            cl_store(otop + p * sizeof(T), a_pp);
                            cl_store(otop + q * sizeof(T), a_qp);
                        } else {
                            cp[p] = a_pp;
                            cp[q] = a_qp;
                        }
                        if (lb) {
                            cl_store(obot + p * sizeof(T), a_pq);
                            cl_store(obot + q * sizeof(T), a_qq);
                        } else {
                            cq[p] = a_pq;
                            cq[q] = a_qq;
                        }
                    }
                }
            }
            cl_sync<CL>();
            if (moves) {
                th = step(th, 1);
                bh = step(bh, -1);
            }
        }
        update_q((M - 1) & 1, moves ? step(th, -1) : th, moves ? step(bh, 1) : bh);
        double ms = jc_block_max(mysn, sc);
        share(ms);
        for (int k = 0; k < C; ++k) ms = fmax(ms, ex[k]);
        // no rotation, or only rotations so small (|sin| < 1e-9) that the off-diagonal entries
        // they leave (of order sin^2) are below the rotation threshold of another sweep
        if (ms < 1e-18) {
            if (ms > 0.0) ++sweep;
            break;
        }
    }
    // ascending order (rank sort, ties by index); every CTA writes its own columns, a warp per column
    share_diag();
    for (int f = warp; f < 2 * P; f += nw) {
        const int x = own_index(f);
        if (x >= s) continue;
        const T* col = own_col(f) + sp;
        const double lx = diag[x];
        int c = 0;
        for (int e = lane; e < s; e += 32) c += diag[e] < lx || (diag[e] == lx && e < x);
        const int rk = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) evals[rk] = ldexp(lx, shift);
#pragma unroll 4
        for (int row = lane; row < s; row += 32) Qout[row + (int64_t)rk * s] = col[row];
    }
    if (rank == 0 && tid == 0 && info) info[0] = sweep;
    cl_sync<CL>();  // no CTA leaves while another may still write to it
}

template <class T>
rc_status jc_launch(rc_ctx* ctx, int s, int C, const void* A, void* Q, double* evals, int* info, int max_sweeps) {
    const int P = std::max((s + 2 * C - 1) / (2 * C), C > 1 ? 2 : 1);
    const size_t smem = jc_smem<T>(P, C);
    // Threads: the fewest with which a round's blocks of A (all threads) and entries of Q (those past the
    // angles' warps) take the fewest passes.
    const int np = P * C, na = (np + 31) / 32 * 32;
    int nt = na + 64;
    if (ctx->jacobi_threads > 0) {
        nt = std::max(nt, std::min(ctx->jacobi_threads, kJcThreadsMax));
    } else {
        int best = 1 << 30;
        for (int t = nt; t <= kJcThreadsMax; t += 32) {
            const int aj = std::max(1, t / np), qj = std::max(1, (t - na) / s);
            const int qr = std::max(1, (s + t - na - 1) / (t - na));  // rows per thread when nq < s
            const int cost = 3 * ((P + aj - 1) / aj) + (P + qj - 1) / qj * (t - na >= s ? 1 : qr);
            if (cost < best) {
                best = cost;
                nt = t;
            }
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)C);
    cfg.blockDim = dim3((unsigned)nt);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = C > 1 ? 1 : 0;
    if (C > 1) {
        RC_CU(ctx, allow_max_smem(ctx, jacobi_cluster_kernel<T, true>));
        RC_CU(ctx, cudaLaunchKernelEx(&cfg, jacobi_cluster_kernel<T, true>, s, P, C, (const T*)A, (T*)Q, evals, info,
                                      max_sweeps));
    } else {
        RC_CU(ctx, allow_max_smem(ctx, jacobi_cluster_kernel<T, false>));
        RC_CU(ctx, cudaLaunchKernelEx(&cfg, jacobi_cluster_kernel<T, false>, s, P, C, (const T*)A, (T*)Q, evals, info,
                                      max_sweeps));
    }
    ctx->launches++;
    return RC_OK;
}

}  // namespace

// Whether the device can run a cluster of 16 CTAs, more than the portable 8, with the shared memory they need
// (asked once per context).
template <class T>
static bool jc_sixteen(rc_ctx* ctx) {
    int& known = IsComplex<T>::value ? ctx->jacobi16_c : ctx->jacobi16_r;
    if (known < 0) {
        known = 0;
        auto kern = jacobi_cluster_kernel<T, true>;
        if (allow_max_smem(ctx, kern) == cudaSuccess &&
            cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(16);
            cfg.blockDim = dim3(kJcThreadsMax);
            cfg.dynamicSmemBytes = ctx->smem_optin - 1024;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = 16;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0) known = 1;
        }
        cudaGetLastError();
    }
    return known == 1;
}

// CTAs of the cluster for an s x s matrix, 0 when not even the largest holds it. More CTAs divide the updates but
// a barrier of a cluster costs 350-450 cycles against 15-45 of one CTA's; rc_small_eigh, off-diagonal 1e-2
// (us per call):
//   s = 36 real      1: 231   4: 311   8: 372    |  s = 96 real      1: 1650  4: 1100  8: 918   16: 1005
//   s = 48 real      1: 386   4: 374   8: 385    |  s = 192 real     4: 4580  8: 3110  16: 2717
//   s = 72 real      1: 876   4: 686   8: 772    |  s = 192 complex  8: 4316  16: 3336
// (the kernels before: 24 real 0.20 ms, 96 real 2.0, 192 complex 8.5 ms).
int jacobi_cluster_ctas(rc_ctx* ctx, int dtype, int64_t s) {
    if (s > 1024) return 0;
    const bool cplx = dtype == RC_COMPLEX128;
    const bool big = s > 128 && (cplx ? jc_sixteen<double2>(ctx) : jc_sixteen<double>(ctx));
    const int most = ctx->jacobi_ctas > 0 ? std::min(ctx->jacobi_ctas, 8) : (big ? 16 : 8);
    const int want = ctx->jacobi_ctas > 0 ? most : (s <= 40 ? 1 : (s <= 80 ? 4 : (s < 144 ? 8 : most)));
    int C = 1;
    while (2 * C <= want) C *= 2;
    for (; C <= most; C *= 2) {
        const int P = std::max(((int)s + 2 * C - 1) / (2 * C), C > 1 ? 2 : 1);
        const size_t smem = cplx ? jc_smem<double2>(P, C) : jc_smem<double>(P, C);
        if (smem + 1024 <= ctx->smem_optin && P * C + 96 <= kJcThreadsMax) return C;
    }
    return 0;
}

rc_status jacobi_cluster(rc_ctx* ctx, int dtype, int64_t s, int ctas, const void* A, void* Q, double* evals, int* info,
                         int max_sweeps) {
    return dtype == RC_COMPLEX128 ? jc_launch<double2>(ctx, (int)s, ctas, A, Q, evals, info, max_sweeps)
                                  : jc_launch<double>(ctx, (int)s, ctas, A, Q, evals, info, max_sweeps);
}

}  // namespace rcb
