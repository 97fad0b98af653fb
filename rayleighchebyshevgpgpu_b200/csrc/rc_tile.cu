// rc_tile.cu -- degree steps and residual blocks of 7- and 27-point operators on large row-major blocks, from
// tiles in shared memory.
//
// Rows are the points of a grid, i = x + nx (y + ny z); a matrix in CSR form takes part when its rows hold exactly
// the in-grid neighbours of such a grid (op->gx, found when the operator is created). A CTA takes tiles of tx x ty
// points and a panel of up to 12 16-byte slices of their columns, and marches along z. One producer warp brings
// the planes of x (with a halo of one point: what lies outside the grid reads as zero), of x_{k-2} and the source
// block, and of the rows' weights into rings of shared-memory slots, one TMA tile copy each; the other warps
// wait for the slots they read (rc_dmma.cuh). A thread owns one slice of four points in a line along y: it reads
// the line's six points once for the y neighbours of all four, two x neighbours each and the point above, and
// keeps the point below in registers. 27 points: the sums over three points along x of the six lines give the
// 3x3 sums of all four rows, which are kept for the planes above and below.
//
// The gather kernels (rc_filter_rm.cu, rc_resid.cu) read every neighbour through L1 for each thread: at 128^3 with
// 96 bfloat16 columns their loads and fills take 78 % of the L1 data cycles and 68 % of the issue slots, and a CSR
// row's index loads add to both; DRAM then runs at 0.7 of its rate. Here a row's neighbours cost 4.5 shared-memory
// reads instead of 8 (27 points: 4.5 instead of 9), no address or bounds arithmetic per neighbour, and nothing
// waits on DRAM but the producer. The sums are formed in the gather kernels' order (5- and 7-point: the same bits).
//
// Measured, against the gather kernels (time per step; its bytes at the measured copy rate, 6.55 TB/s): CSR 128^3, 96
// columns, bfloat16 347 -> 242 us (256: 7 % of the bytes are still in L2 from the step before), FP64 1146 -> 758 (758);
// 27 points 192^3, 48 columns, bfloat16 992 -> 467 (419), FP64 residual block 2204 -> 1016;
// complex stencil, 884,736 rows x 192 columns, bfloat16 pairs 570 -> 482 (415), bound by instruction issue.
//
// Units (a panel of a tile over ml planes) are taken in turn by one CTA per SM, panels fastest, then x, y, z: the
// tiles in flight are neighbours, so a halo's rows are read from DRAM once. ml is chosen so that the last turn is
// nearly full (tile_plan).
#include <algorithm>
#include <type_traits>
#include "rc_common.cuh"
#include "rc_dmma.cuh"
#include "rc_internal.h"
#include "rc_rmstep.cuh"
#include "rc_tile.h"
#include "rc_tileplan.h"

namespace rcb {

namespace {

// Smallest block (bytes) for which the tile kernels are taken for 7 points. Below, a step is a launch's latency either
// way, or the panels and units of a small grid leave SMs without work; the lines are where no measured grid (12 x 23 x 54
// to 61 x 53 x 67; 8, 24, 53 and 96 columns) was slower beyond them. Filters of 10 steps, gather -> tiles, us:
//   FP64      CSR 40^3 x 24 (12 MB) 177 -> 117; stencil 40^3 x 53 (26 MB) 207 -> 281, 48^3 x 53 (45 MB) 394 -> 319
//   c128      CSR 20^3 x 53 (6 MB) 121 -> 155, 12 x 48 x 64 x 53 (30 MB) 351 -> 373, 48^3 x 24 (40 MB) 474 -> 291;
//             stencil 16 x 40 x 40 x 8 (3 MB) 93 -> 102, 32^3 x 53 (26 MB) 256 -> 203
//   bfloat16  CSR 32^3 x 24 (1.5 MB) 131 -> 182, 48^3 x 53 (11 MB) 246 -> 189; stencil 48^3 x 24 (5 MB) 177 -> 156
//   pairs     CSR 40^3 x 96 (23 MB) 412 -> 452; stencil 94 MB of c128 376 -> 396
// 27 points: any block (8^3, 24 columns: 303 -> 69), where the plan pays (tile27_pays).
constexpr int64_t tile_min_bytes(TileType t, bool csr, bool resid) {
    switch (t) {
        case TT_F64: return csr || resid ? 4ll << 20 : 32ll << 20;
        case TT_C128: return csr ? 32ll << 20 : 16ll << 20;
        case TT_BF16: return csr ? 6ll << 20 : 4ll << 20;
        default: return 32ll << 20;
    }
}

enum { TK_STENCIL7 = 0, TK_CSR7 = 1, TK_STENCIL27 = 2 };
// Points along y per thread. 27 points: the sums of three planes of four points spill at 128 registers.
constexpr int tl_rows(int kind) { return kind == TK_STENCIL27 ? 2 : 4; }
constexpr int TL_MAX_SLOTS = 4;
constexpr int TL_MAX_SEG = 12;      // slices per panel, at most
constexpr int TL_MAX_SEG27 = 6;     // 27 points
constexpr int TL_THREADS = 384;     // product threads, at most

// What a kernel needs beside the maps. Sizes in bytes; slots are multiples of 128.
struct TileArgs {
    int nx, ny, nz, tx, ty, ltx;    // ltx: log2 of tx
    int ntx, nty, ml, nml;          // tiles along x and y, planes per unit, units along z
    int panels, nseg, slices;       // slices per panel and per row
    int units;
    int64_t ld;                     // elements per row
    int xslots, zslots, xbytes, zbytes, cbytes;
    int zops;                       // planes per z slot: x_{k-2} and / or the source block
    int has_z;
    int lost;                       // rc_ctx::lost
    double off;                     // stencils: every neighbour's weight, the diagonal and (complex) the phases
    const void* diag;
    const void* phase;
};

template <class TM, class TC>
struct TileStep {
    TM* y;
    const float* sig;
    TC alpha, beta, gamma;
};
struct TileResid {
    const double* lam;
    double* part;                   // [CTA][res_count]
    void* R;                        // row-major bfloat16 (rc_corr_t / rc_corr2_t), or null
    int64_t ldr;
    int res_count;
    int64_t s;
};
struct TileMaps {
    CUtensorMap x, z, src, co;
};

// A 16-byte shared-memory read, as one instruction (as two 8-byte ones, FP64 slices had two-way bank conflicts).
__device__ __forceinline__ uint4 lds16(uint32_t a) {
    uint4 u;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "r"(a));
    return u;
}

struct Unit {
    int panel, x0, y0, m0, m1;
};
__device__ __forceinline__ Unit tile_unit(const TileArgs& A, int u) {
    Unit U;
    U.panel = u % A.panels;
    int t = u / A.panels;
    U.x0 = (t % A.ntx) * A.tx;
    t /= A.ntx;
    U.y0 = (t % A.nty) * A.ty;
    U.m0 = (t / A.nty) * A.ml;
    U.m1 = min(A.nz, U.m0 + A.ml);
    return U;
}

// The ring positions of one side (producer or product warp).
struct Ring {
    int slot = 0;
    unsigned ph = 0;
    __device__ __forceinline__ void next(int slots) {
        if (++slot == slots) {
            slot = 0;
            ph ^= 1;
        }
    }
};

template <class TS, class TC, class TM>
struct TileVec {
    static constexpr int V = Slice<TS, TM>::V;
    // a += c x in the gather kernels' rounding (packed FP32 pairs for bfloat16 blocks and c64)
    __device__ static __forceinline__ void add(TC (&a)[V], TC c, const uint4& u) {
        const Slice<TS, TM> p = slice_from<TS, TM>(u);
        if constexpr (sizeof(TM) == 2) {
#pragma unroll
            for (int v = 0; v < V; v += 2) ffma2(c, c, p.v[v], p.v[v + 1], a[v], a[v + 1]);
        } else if constexpr (std::is_same<TC, float2>::value) {
#pragma unroll
            for (int v = 0; v < V; ++v) {
                ffma2(-c.y, c.y, p.v[v].y, p.v[v].x, a[v].x, a[v].y);
                ffma2(c.x, c.x, p.v[v].x, p.v[v].y, a[v].x, a[v].y);
            }
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v) a[v] = s_fma(c, s_cvt<TC>(p.v[v]), a[v]);
        }
    }
    // the same for a real c: the products with its zero imaginary part left out
    __device__ static __forceinline__ void addr(TC (&a)[V], real_t<TC> c, const uint4& u) {
        if constexpr (IsComplex<TC>::value) {
            const Slice<TS, TM> p = slice_from<TS, TM>(u);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                if constexpr (sizeof(c) == 4) ffma2(c, c, p.v[v].x, p.v[v].y, a[v].x, a[v].y);
                else a[v] = make_double2(fma(c, p.v[v].x, a[v].x), fma(c, p.v[v].y, a[v].y));
            }
        } else {
            add(a, c, u);
        }
    }
};

// What a CTA's product threads form, in every unit, set to NaN (after a plane that never landed). 27 points: called, not
// inlined, for its registers would be taken from the loops (192^3, 48 columns, a correction of 9 steps: 7.78 ms inlined,
// 7.70 called), and with its arguments by value: a reference to the kernel's parameters has every thread copy them to
// local memory at its start (7-point filter 100 x 90 x 60 x 24, 14 steps: 931 us inlined, 959 so).
template <int KIND, class TS, class TC, class TM, bool RESID>
__device__ __forceinline__ void tile_poison(const TileArgs& A, TM* y, const TileResid& Q) {
    constexpr int V = Slice<TS, TM>::V, TL_ROWS = tl_rows(KIND);
    constexpr bool CPLX = IsComplex<TC>::value;
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    unsigned id;  // (read again: places kept for these loops would cost the others registers)
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(id));
    const int r = (int)id / A.nseg, sg = (int)id - r * A.nseg;
    for (int u = blockIdx.x; u < A.units; u += gridDim.x) {
        const Unit U = tile_unit(A, u);
        const int gx = U.x0 + (r & (A.tx - 1)), gy = U.y0 + (r >> A.ltx) * TL_ROWS, slice = U.panel * A.nseg + sg;
        const int nrow = slice < A.slices && gx < A.nx ? max(0, min(TL_ROWS, A.ny - gy)) : 0;
        for (int m = U.m0; m < U.m1; ++m)
            for (int k = 0; k < nrow; ++k) {
                const int64_t i = gx + (int64_t)A.nx * (gy + k + (int64_t)A.ny * m), col = (int64_t)slice * V;
                if constexpr (RESID) {
                    if (!Q.R) continue;
                    using TR = typename std::conditional<CPLX, rc_corr2_t, rc_corr_t>::type;
                    void* R = (TR*)Q.R + i * Q.ldr + col;
                    if constexpr (sizeof(rc_corr_t) == 2) *(__nv_bfloat162*)R = __floats2bfloat162_rn((float)nan, (float)nan);
                    else *(float2*)R = make_float2((float)nan, (float)nan);
                } else {
                    Slice<TS, TM> bad;
#pragma unroll
                    for (int v = 0; v < V; ++v) bad.v[v] = s_from<TS>(nan, nan);
                    stv<TS, TM>(y + i * A.ld + col, bad);
                }
            }
    }
}

template <int KIND, class TS, class TC, class TM, bool RESID>
__device__ __noinline__ void tile_poison_call(TileArgs A, TM* y, TileResid Q) {
    tile_poison<KIND, TS, TC, TM, RESID>(A, y, Q);
}

template <int KIND, class TS, class TC, class TM, bool SRC, bool RESID>
__global__ void __launch_bounds__(TL_THREADS + 32, 1)
tile_kernel(TileArgs A, const __grid_constant__ TileMaps M, TileStep<TM, TC> S, TileResid Q) {
    constexpr int V = Slice<TS, TM>::V, TL_ROWS = tl_rows(KIND);
    constexpr bool CPLX = IsComplex<TC>::value;
    using TD = real_t<TC>;
    using Vec = TileVec<TS, TC, TM>;
    extern __shared__ __align__(128) unsigned char tls[];
    __shared__ __align__(8) uint64_t bars[4 * TL_MAX_SLOTS];
    const int tid = threadIdx.x, lane = tid & 31, nt = blockDim.x - 32;
    const uint32_t xfull = smem_u32(bars), xempty = xfull + 8 * TL_MAX_SLOTS, zfull = xempty + 8 * TL_MAX_SLOTS,
                   zempty = zfull + 8 * TL_MAX_SLOTS;
    const bool zring = A.zops > 0 || KIND == TK_CSR7;
    const int zslot = A.zops * A.zbytes + A.cbytes;
    unsigned char* xs0 = tls;
    unsigned char* zs0 = tls + A.xslots * A.xbytes;
    __shared__ int lost;
    if (tid == 0) {
        lost = 0;
        for (int s = 0; s < A.xslots; ++s) {
            mbar_init(xfull + 8 * s, 1);
            mbar_init(xempty + 8 * s, nt / 32);
        }
        for (int s = 0; s < A.zslots; ++s) {
            mbar_init(zfull + 8 * s, 1);
            mbar_init(zempty + 8 * s, nt / 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    Ring rx, rz;
    if (tid >= nt) {  // the producer: planes m0 - 1, m0, then m + 1 of x with the rest of plane m
        if (lane != 0) return;
        const int cw = A.nseg * 4;  // 32-bit words of a panel's row
        const unsigned xtx = (unsigned)(A.nseg * 16 * (A.tx + 2) * (A.ty + 2));
        const unsigned ztx = (unsigned)(A.zops * A.nseg * 16 * A.tx * A.ty) +
                             (KIND == TK_CSR7 ? (unsigned)(sizeof(RowWeights<TC>) * A.tx * A.ty) : 0u);
        int64_t nxl = 0, nzl = 0;
        bool ok = true;
        auto load_x = [&](const Unit& U, int m) {
            if (nxl >= A.xslots && (A.lost || !mbar_wait(xempty + 8 * rx.slot, rx.ph ^ 1))) return false;
            const uint32_t bar = xfull + 8 * rx.slot;
            mbar_arrive_tx(bar, xtx);
            tma_load_4d(smem_u32(xs0 + rx.slot * A.xbytes), &M.x, U.panel * cw, U.x0 - 1, U.y0 - 1, m, bar);
            rx.next(A.xslots);
            ++nxl;
            return true;
        };
        auto load_z = [&](const Unit& U, int m) {
            if (nzl >= A.zslots && (A.lost || !mbar_wait(zempty + 8 * rz.slot, rz.ph ^ 1))) return false;
            const uint32_t bar = zfull + 8 * rz.slot;
            unsigned char* d = zs0 + rz.slot * zslot;
            mbar_arrive_tx(bar, ztx);
            if (A.has_z) tma_load_4d(smem_u32(d), &M.z, U.panel * cw, U.x0, U.y0, m, bar);
            if (SRC) tma_load_4d(smem_u32(d + (A.zops - 1) * A.zbytes), &M.src, U.panel * cw, U.x0, U.y0, m, bar);
            if (KIND == TK_CSR7) tma_load_4d(smem_u32(d + A.zops * A.zbytes), &M.co, 0, U.x0, U.y0, m, bar);
            rz.next(A.zslots);
            ++nzl;
            return true;
        };
        for (int u = blockIdx.x; u < A.units && ok; u += gridDim.x) {
            const Unit U = tile_unit(A, u);
            ok = load_x(U, U.m0 - 1) && load_x(U, U.m0);
            for (int m = U.m0; m < U.m1 && ok; ++m) ok = load_x(U, m + 1) && (!zring || load_z(U, m));
        }
        // copies still in flight land before the CTA ends
        for (int s = 0; s < A.xslots && s < nxl; ++s) {
            if (--rx.slot < 0) {
                rx.slot = A.xslots - 1;
                rx.ph ^= 1;
            }
            if (!mbar_wait(xfull + 8 * rx.slot, rx.ph)) break;
        }
        for (int s = 0; s < A.zslots && s < nzl; ++s) {
            if (--rz.slot < 0) {
                rz.slot = A.zslots - 1;
                rz.ph ^= 1;
            }
            if (!mbar_wait(zfull + 8 * rz.slot, rz.ph)) break;
        }
        return;
    }

    const int row = tid / A.nseg, seg = tid - row * A.nseg;
    const int lx = row & (A.tx - 1), ly = (row >> A.ltx) * TL_ROWS;
    const int cb = A.nseg * 16, xp = (A.tx + 2) * cb;          // bytes of a point and of a line of the x tile
    const int xo = ly * xp + (lx + 1) * cb + seg * 16;         // line ly - 1 (halo) of this thread's column
    const int zo = (ly * A.tx + lx) * cb + seg * 16, zp = A.tx * cb;
    const TD* diag = (const TD*)A.diag;
    double sq[RESID ? V : 1];
#pragma unroll
    for (int v = 0; v < (RESID ? V : 1); ++v) sq[v] = 0.0;
    bool ok = !A.lost;
    for (int u = blockIdx.x; u < A.units && ok; u += gridDim.x) {
        const Unit U = tile_unit(A, u);
        const int gx = U.x0 + lx, gy = U.y0 + ly;
        const int slice = U.panel * A.nseg + seg;
        const bool col_on = slice < A.slices && gx < A.nx;
        const int nrow = col_on ? max(0, min(TL_ROWS, A.ny - gy)) : 0;
        const int64_t col = (int64_t)slice * V;
        const int64_t i0 = gx + (int64_t)A.nx * gy, plane = (int64_t)A.nx * A.ny;
        float sg[SRC ? V : 1];
        if (SRC) {
#pragma unroll
            for (int v = 0; v < V; ++v) sg[v] = col_on ? __ldg(S.sig + col + v) : 0.0f;
        }
        double lam[RESID ? V : 1];
        if (RESID) {
#pragma unroll
            for (int v = 0; v < V; ++v) lam[v] = col + v < Q.s ? Q.lam[col + v] : 0.0;
        }
        const TC off = s_from<TC>(A.off, 0.0);
        TC wm = off, wp = off;
        if constexpr (CPLX && KIND == TK_STENCIL7) {
            const TC p = col_on ? ((const TC*)A.phase)[gx] : off;
            wm = s_mul(off, p);
            wp = s_mul(off, s_conj(p));
        }
        // stencils: the diagonal of the next plane's points, fetched a plane ahead
        TD dn[TL_ROWS];
        auto fetch_diag = [&](int m) {
            if constexpr (KIND != TK_CSR7) {
#pragma unroll
                for (int k = 0; k < TL_ROWS; ++k)
                    dn[k] = k < nrow && m < U.m1 ? __ldg(diag + i0 + (int64_t)k * A.nx + (int64_t)m * plane) : TD(0);
            }
        };
        fetch_diag(U.m0);
        // the finished sums a (A x, or the box sum) of point k of plane m, whose own value is xi
        auto finish = [&](int m, int k, const TC (&a)[V], const uint4& xr, uint32_t zb) {
            const Slice<TS, TM> xi = slice_from<TS, TM>(xr);
            const int64_t i = i0 + (int64_t)k * A.nx + (int64_t)m * plane;
            if constexpr (RESID) {
                if (k >= nrow) return;
                float rv[2] = {0.0f, 0.0f};
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    if constexpr (CPLX) {
                        double2 d = make_double2(fma(-lam[v], xi.v[v].x, a[v].x), fma(-lam[v], xi.v[v].y, a[v].y));
                        if (col + v >= Q.s) d = make_double2(0.0, 0.0);
                        sq[v] = fma(d.y, d.y, fma(d.x, d.x, sq[v]));
                        rv[0] = (float)d.x;
                        rv[1] = (float)d.y;
                    } else {
                        const double d = col + v < Q.s ? fma(-lam[v], xi.v[v], a[v]) : 0.0;
                        sq[v] = fma(d, d, sq[v]);
                        rv[v] = (float)d;
                    }
                }
                if (Q.R) {
                    using TR = typename std::conditional<CPLX, rc_corr2_t, rc_corr_t>::type;
                    void* R = (TR*)Q.R + i * Q.ldr + col;
                    if constexpr (sizeof(rc_corr_t) == 2) *(__nv_bfloat162*)R = __floats2bfloat162_rn(rv[0], rv[1]);
                    else *(float2*)R = make_float2(rv[0], rv[1]);
                }
            } else {
                Slice<TS, TM> zi{}, si{}, out;
                if (A.has_z) zi = slice_from<TS, TM>(lds16(zb + zo + k * zp));
                if (SRC) si = slice_from<TS, TM>(lds16(zb + (A.zops - 1) * A.zbytes + zo + k * zp));
                if constexpr (sizeof(TM) == 2) {
#pragma unroll
                    for (int v = 0; v < V; v += 2) {
                        float r0, r1;
                        fmul2(S.alpha, S.alpha, a[v], a[v + 1], r0, r1);
                        ffma2(S.beta, S.beta, xi.v[v], xi.v[v + 1], r0, r1);
                        if (A.has_z) ffma2(S.gamma, S.gamma, zi.v[v], zi.v[v + 1], r0, r1);
                        if (SRC) ffma2(sg[v], sg[v + 1], si.v[v], si.v[v + 1], r0, r1);
                        out.v[v] = r0;
                        out.v[v + 1] = r1;
                    }
                } else if constexpr (SRC && CPLX) {
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        float r0, r1;
                        fmul2(S.alpha.x, S.alpha.x, a[v].x, a[v].y, r0, r1);
                        ffma2(S.beta.x, S.beta.x, xi.v[v].x, xi.v[v].y, r0, r1);
                        if (A.has_z) ffma2(S.gamma.x, S.gamma.x, zi.v[v].x, zi.v[v].y, r0, r1);
                        ffma2(sg[v], sg[v], si.v[v].x, si.v[v].y, r0, r1);
                        out.v[v] = make_float2(r0, r1);
                    }
                } else {
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        TC r = s_mul(S.alpha, a[v]);
                        r = s_fma(S.beta, s_cvt<TC>(xi.v[v]), r);
                        if (A.has_z) r = s_fma(S.gamma, s_cvt<TC>(zi.v[v]), r);
                        out.v[v] = s_cvt<TS>(r);
                    }
                }
                if (k < nrow) stv_once<TS, TM>(S.y + i * A.ld + col, out);
            }
        };
        auto wait_x = [&]() {
            ok = ok && mbar_wait(xfull + 8 * rx.slot, rx.ph);
            return smem_u32(xs0) + rx.slot * A.xbytes + xo;
        };
        // (all lanes come here whether their waits ran out or not, and go on together)
        auto free_x = [&](int slot) {
            ok = __all_sync(~0u, ok);
            __syncwarp();
            if (lane == 0) mbar_arrive(xempty + 8 * slot);
        };
        uint32_t zb = 0;
        auto wait_z = [&]() {
            if (!zring) return;
            ok = ok && mbar_wait(zfull + 8 * rz.slot, rz.ph);
            zb = smem_u32(zs0) + rz.slot * zslot;
        };
        auto free_z = [&]() {
            if (!zring) return;
            if constexpr (KIND == TK_STENCIL27) ok = __all_sync(~0u, ok);  // (7 points: with free_x after it)
            __syncwarp();
            if (lane == 0) mbar_arrive(zempty + 8 * rz.slot);
            rz.next(A.zslots);
        };
        if constexpr (KIND == TK_STENCIL27) {
            // 3x3 sums of the four points in one plane, and their own values
            auto plane_sums = [&](uint32_t p, TC (&b)[TL_ROWS][V], uint4 (&own)[TL_ROWS]) {
#pragma unroll
                for (int l = 0; l < TL_ROWS + 2; ++l) {
                    const uint4 c = lds16(p + l * xp);
                    const Slice<TS, TM> cl = slice_from<TS, TM>(lds16(p + l * xp - cb)), cc = slice_from<TS, TM>(c),
                                        cr = slice_from<TS, TM>(lds16(p + l * xp + cb));
                    if (l >= 1 && l <= TL_ROWS) own[l - 1] = c;
                    TC t[V];
#pragma unroll
                    for (int v = 0; v < V; ++v) t[v] = s_add(s_add(s_cvt<TC>(cl.v[v]), s_cvt<TC>(cc.v[v])), s_cvt<TC>(cr.v[v]));
#pragma unroll
                    for (int k = l - 2; k <= l; ++k) {
                        if (k < 0 || k >= TL_ROWS) continue;
#pragma unroll
                        for (int v = 0; v < V; ++v) b[k][v] = k == l ? t[v] : s_add(b[k][v], t[v]);
                    }
                }
            };
            TC s2[TL_ROWS][V], p0[TL_ROWS][V];  // sums of the planes below and here; of this plane
            uint4 own[TL_ROWS];
            {
                plane_sums(wait_x(), s2, own);
                free_x(rx.slot);
                rx.next(A.xslots);
                plane_sums(wait_x(), p0, own);
                free_x(rx.slot);
                rx.next(A.xslots);
#pragma unroll
                for (int k = 0; k < TL_ROWS; ++k)
#pragma unroll
                    for (int v = 0; v < V; ++v) s2[k][v] = s_add(s2[k][v], p0[k][v]);
            }
            for (int m = U.m0; m < U.m1 && ok; ++m) {
                TD d[TL_ROWS];
#pragma unroll
                for (int k = 0; k < TL_ROWS; ++k) d[k] = dn[k];
                fetch_diag(m + 1);
                TC p1[TL_ROWS][V];
                uint4 own1[TL_ROWS];
                plane_sums(wait_x(), p1, own1);
                free_x(rx.slot);
                rx.next(A.xslots);
                wait_z();
#pragma unroll
                for (int k = 0; k < TL_ROWS; ++k) {
                    const TC dm = s_sub(s_from<TC>((double)d[k], 0.0), off);
                    const Slice<TS, TM> xi = slice_from<TS, TM>(own[k]);
                    TC a[V];
#pragma unroll
                    for (int v = 0; v < V; ++v)
                        a[v] = s_fma(off, s_add(s2[k][v], p1[k][v]), s_mul(dm, s_cvt<TC>(xi.v[v])));
                    finish(m, k, a, own[k], zb);
                    own[k] = own1[k];
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        s2[k][v] = s_add(p0[k][v], p1[k][v]);
                        p0[k][v] = p1[k][v];
                    }
                }
                free_z();
            }
        } else {
            uint4 um[TL_ROWS];  // the points below
            {
                const uint32_t p = wait_x();
#pragma unroll
                for (int k = 0; k < TL_ROWS; ++k) um[k] = lds16(p + (k + 1) * xp);
                free_x(rx.slot);
                rx.next(A.xslots);
            }
            uint32_t pc = wait_x();
            ok = __all_sync(~0u, ok);
            int sc = rx.slot;
            rx.next(A.xslots);
            for (int m = U.m0; m < U.m1 && ok; ++m) {
                TD d[TL_ROWS];
                if constexpr (KIND == TK_STENCIL7) {
#pragma unroll
                    for (int k = 0; k < TL_ROWS; ++k) d[k] = dn[k];
                    fetch_diag(m + 1);
                }
                const uint32_t pn = wait_x();
                wait_z();
                uint4 c0 = lds16(pc), c1 = lds16(pc + xp);
#pragma unroll
                for (int k = 0; k < TL_ROWS; ++k) {
                    const uint4 c2 = lds16(pc + (k + 2) * xp);
                    const uint4 cl = lds16(pc + (k + 1) * xp - cb), cr = lds16(pc + (k + 1) * xp + cb);
                    const uint4 cn = lds16(pn + (k + 1) * xp);
                    TC a[V];
#pragma unroll
                    for (int v = 0; v < V; ++v) a[v] = s_zero(TC());
                    if constexpr (KIND == TK_STENCIL7) {
                        const TD w = (TD)A.off;
                        Vec::addr(a, d[k], c1);
                        Vec::addr(a, w, um[k]);
                        Vec::add(a, wm, c0);
                        Vec::addr(a, w, cl);
                        Vec::addr(a, w, cr);
                        Vec::add(a, wp, c2);
                        Vec::addr(a, w, cn);
                    } else {
                        RowWeights<TC> w;
                        {
                            uint4 r[sizeof(RowWeights<TC>) / 16];
                            const uint32_t wa = zb + A.zops * A.zbytes + ((ly + k) * A.tx + lx) * (int)sizeof(RowWeights<TC>);
#pragma unroll
                            for (int e = 0; e < (int)(sizeof(r) / 16); ++e) r[e] = lds16(wa + 16 * e);
                            memcpy(&w, r, sizeof(w));
                        }
                        Vec::add(a, w.w[0], um[k]);
                        Vec::add(a, w.w[1], c0);
                        Vec::add(a, w.w[2], cl);
                        Vec::add(a, w.w[3], c1);
                        Vec::add(a, w.w[4], cr);
                        Vec::add(a, w.w[5], c2);
                        Vec::add(a, w.w[6], cn);
                    }
                    finish(m, k, a, c1, zb);
                    um[k] = c1;
                    c0 = c1;
                    c1 = c2;
                }
                free_x(sc);
                free_z();
                pc = pn;
                sc = rx.slot;
                rx.next(A.xslots);
            }
            free_x(sc);
        }
    }
    if (!ok) {  // a plane that never landed
        if constexpr (KIND != TK_STENCIL27) tile_poison<KIND, TS, TC, TM, RESID>(A, S.y, Q);
        else tile_poison_call<KIND, TS, TC, TM, RESID>(A, S.y, Q);
    }
    if constexpr (RESID) {
        if (Q.res_count < 1) return;
        // column sums over the CTA's points, rows in order (the panel is the same in all its units)
        if (!ok) lost = 1;
        asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
        double* red = reinterpret_cast<double*>(tls);  // every slot has been read (or the sums are NaN)
        const int pw = A.nseg * V, rows = nt / A.nseg;
#pragma unroll
        for (int v = 0; v < V; ++v) red[row * pw + seg * V + v] = sq[v];
        asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
        const int c0 = (blockIdx.x % A.panels) * pw;
        for (int c = tid; c < Q.res_count; c += nt) {
            double t = 0.0;
            if (c >= c0 && c < c0 + pw)
                for (int r = 0; r < rows; ++r) t += red[r * pw + c - c0];
            if (lost && c >= c0 && c < c0 + pw) t = __longlong_as_double(0x7ff8000000000000ll);
            Q.part[(int64_t)blockIdx.x * Q.res_count + c] = t;
        }
    }
}

// Rows of the 7-point CSR structure: weights by neighbour, zeros where there is none.
template <class T>
__global__ void tile_pack_kernel(int64_t n, int nx, int ny, int nz, const int32_t* __restrict__ rowptr,
                                 const T* __restrict__ vals, RowWeights<T>* __restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t l = i / nx;
        const int x = (int)(i - l * nx), z = (int)(l / ny), y = (int)(l - (int64_t)z * ny);
        int k = rowptr[i];
        RowWeights<T> w;
        w.w[0] = z > 0 ? vals[k++] : s_zero(T());
        w.w[1] = y > 0 ? vals[k++] : s_zero(T());
        w.w[2] = x > 0 ? vals[k++] : s_zero(T());
        w.w[3] = vals[k++];
        w.w[4] = x + 1 < nx ? vals[k++] : s_zero(T());
        w.w[5] = y + 1 < ny ? vals[k++] : s_zero(T());
        w.w[6] = z + 1 < nz ? vals[k++] : s_zero(T());
        w.w[7] = s_zero(T());
        out[i] = w;
    }
}

// A CSR operator's weights are laid out once its steps have moved this many bytes of blocks through the gather kernels.
// A step loses 0.22 to 0.36 us per MB of its block (FP64 128^3 x 96, 1.6 GB: 1146 against 758 us; bfloat16, 0.4 GB: 347
// against 242; FP64 48^3 x 96, 85 MB: 68 against 50), and laying the weights out takes 0.45 ms: cudaMalloc 0.4 at every
// size from 1 MB on, the packing 0.05 per 134 MB. That is 1.2 to 2 GB of blocks; the line lies lower because most operators
// see hundreds of steps, but above what a single call on a small one moves. Eight new operators of 8,000 to 216,000 rows:
// their first batch of corrections 4.7 ms with weights for every grid from its creation on (and 2.9 ms more to create
// them), 3.2 ms now; 48^3 rows x 24 columns 0.9 and 0.6 ms.
constexpr int64_t kPackPerByte = 2, kPackBase = 256ll << 20;

struct Structure {
    int kind = -1;
    int64_t nx = 0, ny = 0, nz = 0;
};
Structure structure(const rc_ctx* ctx, const rc_op* op, bool fp32) {
    Structure S;
    if (op->kind == 1 && (op->skind == 7 || op->skind == 27)) {
        S.kind = op->skind == 7 ? TK_STENCIL7 : TK_STENCIL27;
        S.nx = op->nx;
        S.ny = op->ny;
        S.nz = op->nz;
    } else if (tile_rows(ctx, op, fp32)) {
        S.kind = TK_CSR7;
        S.nx = op->gx;
        S.ny = op->gy;
        S.nz = op->gz;
    }
    return S;
}
constexpr int tile_elem(TileType t) { return t == TT_BF16 ? 2 : (t == TT_BF16C ? 4 : (t == TT_F64 ? 8 : 16)); }

// Whether the plan is better than the gather kernels' form for 7 points: the waste of the grid's edges and halos (traffic
// against that of the points alone) and the threads of a CTA, of which there is one per SM. Filters of 10 steps on
// narrow and ragged grids, 3 to 40 columns, gather -> tiles, us: FP64 CSR 18 x 11 x 4000 x 12 (waste 2.0, 96 threads)
// 924 -> 1092, 37 x 70 x 200 x 40 (1.36, 160) 1596 -> 1229, the stencil 1117 -> 1269, 61 x 53 x 250 x 24 (1.25, 384)
// 1076 -> 854; bfloat16 CSR 24 x 24 x 1000 x 24 (1.39, 288) 504 -> 453, the stencil 417 -> 444; 37 x 70 x 200 x 24 (1.36,
// 96) 466 -> 511; pairs 18 x 11 x 4000 x 12 (2.03, 288) 701 -> 952. One slice a row of bfloat16 is too little for a TMA
// box's lines (100 x 90 x 60 x 8: 213 -> 290).
// Grids of few planes, and those whose units leave the last turn nearly empty, waste more than their edges: `total` is the
// waste with the planes that the turns read. FP64 stencil 300 x 130 x 1 x 130 (total 2.7) 331 -> 464, x 2 x 53 (2.04)
// 252 -> 274, x 4 x 53 (1.65) 533 -> 543; complex 300 x 130 x 1 x 53 (2.8) 297 -> 397, 300 x 2 x 130 x 53 (2.0) gains a
// tenth; bfloat16 100 x 90 x 5 x 130 (2.9, 12 MB) 258 -> 293, the CSR rows 256 -> 281, smaller blocks (x 53, 5 MB) 181 -> 157.
// (Not for steps without a second block, a filter's first and the residual, which were not measured there.)
bool tile_pays(TileType type, bool csr, int zops, double waste, double total, double mbytes, int threads, int nseg) {
    const bool bf16 = type == TT_BF16 || type == TT_BF16C;
    if (bf16 && nseg < 2) return false;
    if (waste > (csr && type != TT_BF16C ? 1.45 : 1.3)) return false;
    if (zops > 0 &&
        (type == TT_BF16 ? total > (csr ? 2.4 : 2.1) && mbytes > 10.0 : !csr && !bf16 && total > (type == TT_F64 ? 2.0 : 2.4)))
        return false;
    return threads >= (csr && !bf16 ? 160 : (type == TT_C128 ? 256 : 192));
}

// Tiles, slots and units for blocks of `slices` 16-byte slices a row; zops planes beside x, wbytes of weights a row.
bool tile_plan(const rc_ctx* ctx, const Structure& S, TileType type, int slices, int zops, int wbytes, TileArgs* out,
               unsigned* grid, size_t* smem) {
    TileArgs A = {};
    A.nx = (int)S.nx;
    A.ny = (int)S.ny;
    A.nz = (int)S.nz;
    A.slices = slices;
    A.lost = ctx->lost;
    const int seg_max = S.kind == TK_STENCIL27 ? TL_MAX_SEG27 : TL_MAX_SEG, R = tl_rows(S.kind);
    A.panels = (slices + seg_max - 1) / seg_max;
    A.nseg = (slices + A.panels - 1) / A.panels;
    A.zops = zops;
    auto up = [](int b) { return (b + 127) / 128 * 128; };
    const int room = (int)ctx->smem_optin - 2048;
    // The tile: whole warps of at most TL_THREADS, three slots of x; the least memory traffic over the grid, points of
    // the tiles past its edges included. A halo point costs half (it is in L2), a plane about 24 points by itself.
    double least = 1e300;
    for (int ltx = 2; ltx <= 5; ++ltx)
        for (int ty = R; ty <= 32; ty += R) {
            const int tx = 1 << ltx, nt = tx * ty / R * A.nseg;
            if (nt > TL_THREADS || nt % 32) continue;
            const int xb = up(A.nseg * 16 * (tx + 2) * (ty + 2)), zb = zops * up(A.nseg * 16 * tx * ty) + up(wbytes * tx * ty);
            if (3 * xb + (zb ? 2 : 0) * zb > room) continue;
            const double tiles = (double)((A.nx + tx - 1) / tx) * ((A.ny + ty - 1) / ty);
            const double cost = tiles * (tx * ty * (2.0 + zops) + 0.5 * ((tx + 2) * (ty + 2) - tx * ty) + 24.0);
            if (cost < least) {
                least = cost;
                A.tx = tx;
                A.ltx = ltx;
                A.ty = ty;
            }
        }
    if (!A.tx) return false;
    A.xbytes = up(A.nseg * 16 * (A.tx + 2) * (A.ty + 2));
    A.zbytes = up(A.nseg * 16 * A.tx * A.ty);
    A.cbytes = up(wbytes * A.tx * A.ty);
    const int zslot = zops * A.zbytes + A.cbytes;
    A.zslots = zslot ? 2 : 1;
    A.xslots = std::min(TL_MAX_SLOTS, (room - A.zslots * zslot) / A.xbytes);
    if (zslot && A.xslots == TL_MAX_SLOTS && 3 * zslot + A.xslots * A.xbytes <= room) A.zslots = 3;
    A.ntx = (A.nx + A.tx - 1) / A.tx;
    A.nty = (A.ny + A.ty - 1) / A.ty;
    const int64_t columns = (int64_t)A.panels * A.ntx * A.nty;
    const int64_t ctas = std::max<int64_t>(1, ctx->sm_count / A.panels) * A.panels;
    if (columns * A.nz > INT32_MAX) return false;
    double planes = 0.0;
    A.ml = tile_planes(A.nz, columns, ctas, &planes);
    if (ctx->tile == 1) {
        const double bytes = 16.0 * slices * A.nx * A.ny * A.nz, waste = least / ((double)A.nx * A.ny * (2.0 + zops));
        if (!(S.kind == TK_STENCIL27 ? tile27_pays(type == TT_BF16, planes, bytes)
                                     : tile_pays(type, S.kind == TK_CSR7, zops, waste,
                                                 waste * planes * ctas / ((double)columns * A.nz), bytes / 1048576.0,
                                                 A.tx * A.ty / R * A.nseg, A.nseg)))
            return false;
    }
    A.nml = (A.nz + A.ml - 1) / A.ml;
    A.units = (int)(columns * A.nml);
    *grid = (unsigned)std::min<int64_t>(ctas, A.units);
    // a CTA keeps its panel: whole turns of the panels
    *grid = *grid / A.panels * A.panels;
    const int red = A.tx * A.ty / R * A.nseg * 2 * 8;  // the residual's column sums
    *smem = (size_t)std::max(A.xslots * A.xbytes + A.zslots * zslot, red);
    *out = A;
    return true;
}

bool tile_map(CUtensorMap* map, const void* p, const Structure& S, int64_t words, int bw, int bx, int by) {
    const int64_t dims[4] = {words, S.nx, S.ny, S.nz};
    const int box[4] = {bw, bx, by, 1};
    return tma_map_words_4d(map, p, dims, box);
}

template <int KIND, class TS, class TC, class TM, bool SRC, bool RESID>
bool tile_launch(rc_ctx* ctx, const TileArgs& A, const TileMaps& M, const TileStep<TM, TC>& S, const TileResid& Q,
                 unsigned grid, size_t smem) {
    auto kern = tile_kernel<KIND, TS, TC, TM, SRC, RESID>;
    if (allow_max_smem(ctx, kern) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const int nt = A.tx * A.ty / tl_rows(KIND) * A.nseg;
    kern<<<grid, nt + 32, smem, ctx->stream>>>(A, M, S, Q);
    ctx->launches++;
    ctx->tile_launches++;
    return true;
}

}  // namespace

bool tile_supported(const rc_ctx* ctx, const rc_op* op, TileType type, int64_t ld, bool resid) {
    if (!ctx->tile) return false;
    const Structure S = structure(ctx, op, type == TT_BF16 || type == TT_BF16C);
    if (S.kind < 0 || (op->dtype == RC_COMPLEX128) != (type == TT_C128 || type == TT_BF16C)) return false;
    if (S.kind == TK_STENCIL27 && op->dtype == RC_COMPLEX128) return false;
    return ctx->tile > 1 || S.kind == TK_STENCIL27 ||
           op->n * ld * tile_elem(type) >= tile_min_bytes(type, S.kind == TK_CSR7, resid);
}

template <class TS, class TC, class TM, bool SRC>
static bool tile_step_t(rc_ctx* ctx, rc_op* op, TileType type, int64_t ld, const void* x, const void* z, void* y,
                        double alpha, double beta, double gamma, const void* src, const float* sig) {
    const bool fp32 = sizeof(real_t<TC>) == 4;
    const Structure st = structure(ctx, op, fp32);
    TileArgs A;
    unsigned grid;
    size_t smem;
    const int zops = (z ? 1 : 0) + (SRC ? 1 : 0);
    const int wb = st.kind == TK_CSR7 ? (int)sizeof(RowWeights<TC>) : 0;
    const int64_t words = ld * (int64_t)sizeof(TM) / 4;
    if (!tile_plan(ctx, st, type, (int)(words / 4), zops, wb, &A, &grid, &smem)) return false;
    const void* weights = wb ? tile_weights(ctx, op, fp32, op->n * ld * (int64_t)sizeof(TM)) : nullptr;
    if (wb && !weights) return false;
    A.ld = ld;
    A.has_z = z != nullptr;
    A.off = op->offdiag;
    A.diag = fp32 ? (const void*)op->diag32 : (const void*)op->diag64;
    A.phase = fp32 ? op->phase32 : op->phase64;
    TileMaps M = {};
    bool ok = tile_map(&M.x, x, st, words, A.nseg * 4, A.tx + 2, A.ty + 2);
    if (z) ok = ok && tile_map(&M.z, z, st, words, A.nseg * 4, A.tx, A.ty);
    if (SRC) ok = ok && tile_map(&M.src, src, st, words, A.nseg * 4, A.tx, A.ty);
    if (wb) ok = ok && tile_map(&M.co, weights, st, wb / 4, wb / 4, A.tx, A.ty);
    if (!ok) return false;
    TileStep<TM, TC> S;
    S.y = (TM*)y;
    S.sig = sig;
    S.alpha = s_from<TC>(alpha, 0.0);
    S.beta = s_from<TC>(beta, 0.0);
    S.gamma = s_from<TC>(gamma, 0.0);
    const TileResid Q = {};
    if (st.kind == TK_CSR7) return tile_launch<TK_CSR7, TS, TC, TM, SRC, false>(ctx, A, M, S, Q, grid, smem);
    if constexpr (!IsComplex<TC>::value)
        if (st.kind == TK_STENCIL27) return tile_launch<TK_STENCIL27, TS, TC, TM, SRC, false>(ctx, A, M, S, Q, grid, smem);
    return tile_launch<TK_STENCIL7, TS, TC, TM, SRC, false>(ctx, A, M, S, Q, grid, smem);
}

bool tile_step(rc_ctx* ctx, rc_op* op, TileType type, int64_t ld, const void* x, const void* z, void* y, double alpha,
               double beta, double gamma, const void* src, const float* sig) {
    if (((uintptr_t)x | (uintptr_t)z | (uintptr_t)y | (uintptr_t)src) % 16) return false;
    switch (type) {
        case TT_F64:
            return tile_step_t<double, double, double, false>(ctx, op, type, ld, x, z, y, alpha, beta, gamma, src, sig);
        case TT_C128:
            return tile_step_t<double2, double2, double2, false>(ctx, op, type, ld, x, z, y, alpha, beta, gamma, src, sig);
        case TT_BF16:
            return tile_step_t<float, float, __nv_bfloat16, true>(ctx, op, type, ld, x, z, y, alpha, beta, gamma, src, sig);
        case TT_BF16C:
            return tile_step_t<float2, float2, __nv_bfloat162, true>(ctx, op, type, ld, x, z, y, alpha, beta, gamma, src,
                                                                     sig);
    }
    return false;
}

template <class T>
static bool tile_resid_t(rc_ctx* ctx, rc_op* op, const void* Y, int64_t ld, TileResid Q, int64_t res_count,
                         double** part, int64_t* parts, rc_status* status) {
    const Structure st = structure(ctx, op, false);
    TileArgs A;
    unsigned grid;
    size_t smem;
    const int wb = st.kind == TK_CSR7 ? (int)sizeof(RowWeights<T>) : 0;
    const int64_t words = ld * (int64_t)sizeof(T) / 4;
    if (!tile_plan(ctx, st, IsComplex<T>::value ? TT_C128 : TT_F64, (int)(words / 4), 0, wb, &A, &grid, &smem)) return false;
    if (res_count > 0) {  // (before the weights: an allocation that fails may take them back)
        void* p = nullptr;
        *status = rc_slot(ctx, S_RPART, (size_t)grid * res_count * sizeof(double), &p);
        if (*status != RC_OK) return true;
        Q.part = *part = (double*)p;
        *parts = grid;
    }
    const void* weights = wb ? tile_weights(ctx, op, false, op->n * ld * (int64_t)sizeof(T)) : nullptr;
    if (wb && !weights) return false;
    A.ld = ld;
    A.off = op->offdiag;
    A.diag = op->diag64;
    A.phase = op->phase64;
    TileMaps M = {};
    bool ok = tile_map(&M.x, Y, st, words, A.nseg * 4, A.tx + 2, A.ty + 2);
    if (wb) ok = ok && tile_map(&M.co, weights, st, wb / 4, wb / 4, A.tx, A.ty);
    if (!ok) return false;
    const TileStep<T, T> S = {};
    if (st.kind == TK_CSR7) return tile_launch<TK_CSR7, T, T, T, false, true>(ctx, A, M, S, Q, grid, smem);
    if constexpr (!IsComplex<T>::value)
        if (st.kind == TK_STENCIL27) return tile_launch<TK_STENCIL27, T, T, T, false, true>(ctx, A, M, S, Q, grid, smem);
    return tile_launch<TK_STENCIL7, T, T, T, false, true>(ctx, A, M, S, Q, grid, smem);
}

bool tile_resid(rc_ctx* ctx, rc_op* op, const void* Y, int64_t ld, int64_t s, const double* lam, int64_t res_count,
                void* R, int64_t ldr, double** part, int64_t* parts, rc_status* st) {
    *st = RC_OK;
    if ((uintptr_t)Y % 16 || (uintptr_t)R % 4) return false;
    TileResid Q = {};
    Q.lam = lam;
    Q.R = R;
    Q.ldr = ldr;
    Q.res_count = (int)res_count;
    Q.s = s;
    return op->dtype == RC_COMPLEX128 ? tile_resid_t<double2>(ctx, op, Y, ld, Q, res_count, part, parts, st)
                                      : tile_resid_t<double>(ctx, op, Y, ld, Q, res_count, part, parts, st);
}

bool tile_rows(const rc_ctx* ctx, const rc_op* op, bool fp32) {
    if (op->kind != 0 || op->gx <= 0) return false;
    // only the operator's own context lays them out (a context belongs to one thread at a time), outside the server
    return op->pack[fp32].load() || (ctx == op->ctx && !ctx->serve && !op->pack_refused);
}

static bool capturing(const rc_ctx* ctx) {
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &s) == cudaSuccess) return s != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return true;
}

const void* tile_weights(rc_ctx* ctx, rc_op* op, bool fp32, int64_t bytes) {
    if (!tile_rows(ctx, op, fp32)) return nullptr;
    if (ctx != op->ctx) op->pack_shared.store(true);  // before the pointer is read: tile_weights_release
    if (const void* p = op->pack[fp32].load()) {
        if (ctx == op->ctx && !op->pack_shared.load() && capturing(ctx)) op->pack_shared.store(true);  // a graph keeps it
        return p;
    }
    if (ctx != op->ctx) return nullptr;
    const bool cplx = op->dtype == RC_COMPLEX128;
    const int64_t size = op->n * 8 * (int64_t)elem_bytes(op->dtype, fp32 ? P32 : P64);
    op->pack_moved[fp32] += bytes;
    if (ctx->tile == 1 && op->pack_moved[fp32] < kPackPerByte * size + kPackBase) return nullptr;
    if (capturing(ctx)) return nullptr;
    void* out = nullptr;
    if (cudaMalloc(&out, (size_t)size) != cudaSuccess) {
        cudaGetLastError();
        op->pack_refused = true;
        return nullptr;
    }
    const unsigned g = (unsigned)std::min<int64_t>((op->n + 255) / 256, 16 * kB200Sms);
    auto pack = [&](auto v) {
        using T = decltype(v);
        tile_pack_kernel<T><<<g, 256, 0, ctx->stream>>>(op->n, (int)op->gx, (int)op->gy, (int)op->gz, op->rowptr,
                                                        (const T*)(fp32 ? op->vals32 : op->vals64), (RowWeights<T>*)out);
    };
    if (fp32) cplx ? pack(float2()) : pack(float());
    else cplx ? pack(double2()) : pack(double());
    ctx->launches++;
    // complete before anyone sees them: the server's contexts read them on streams of their own
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
        cudaFree(out);
        return nullptr;
    }
    op->pack_bytes += size;
    ctx->op_bytes += size;
    op->pack[fp32].store(out);
    return out;
}

bool tile_weights_release(rc_ctx* ctx) {
    bool any = false;
    for (rc_op* op : ctx->ops)
        for (int k = 0; k < 2; ++k) {
            void* p = op->pack[k].exchange(nullptr);
            if (!p) continue;
            if (op->pack_shared.load()) {  // another context's stream, or a captured graph, may be reading them
                op->pack[k].store(p);
                continue;
            }
            cudaStreamSynchronize(ctx->stream);
            cudaFree(p);
            const int64_t size = op->n * 8 * (int64_t)elem_bytes(op->dtype, k ? P32 : P64);
            op->pack_bytes -= size;
            ctx->op_bytes -= size;
            op->pack_refused = any = true;
        }
    return any;
}

}  // namespace rcb
