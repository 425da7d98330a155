// Device-side building blocks of the M_N dual solve shared by the closure engines
// (closure_fp64.cu: persistent kernels; closure_rounds.cu: work-list rounds):
// warp utilities, the FP64 DMMA, mbarrier/bulk-copy helpers, the per-warp Cholesky,
// condition estimate and substitutions, and the per-cell Newton state machine of
// src/opt/optBatch.cpp:143-344 / src/opt/opt.cpp:139-355 (see closure_fp64.cu).
#pragma once
#include <type_traits>
#include "c3d_common.cuh"

#include <cfloat>

#ifndef M_PI
#define M_PI 3.14159265358979323846
#endif

namespace c3d {
namespace {

constexpr int STAGES = 3;
constexpr int GSTAGES = 2; // stages of the (larger) Gaunt chunks
constexpr int CST = 12;    // row stride of the coefficient tile (bank-conflict-free B fragments)
constexpr double EPS_HALF = DBL_EPSILON / 2;

enum Need : int { NEED_NONE = 0, NEED_H = 1, NEED_TRIAL = 2, NEED_PROBE = 3 };

// Phase clocks of the per-cell Newton logic (profiling builds only).
#ifdef C3D_NEWTON_CLOCKS
#define C3D_NCLK_DECL long long nclk_ = clock64();
#define C3D_NCLK(stats, slot, lane)                                                                \
    do {                                                                                           \
        long long t_ = clock64();                                                                  \
        if ((lane) == 0 && (stats))                                                                \
            atomicAdd(&(stats)[STAT_CLK_NEWTON + (slot)], (unsigned long long)(t_ - nclk_));       \
        nclk_ = t_;                                                                                \
    } while (0)
#else
#define C3D_NCLK_DECL
#define C3D_NCLK(stats, slot, lane)
#endif

struct SlotScalars {
    long long cell;
    long long passes;
    double u0, alphaScale, rtol, f, t, maxFactor, gd, fquad, r, gamma, err;
    int need, iter, totalIter, iterGamma, regIndex, maxIter, status, exhausted;
    // mixed precision: condition estimate of the last Hessian (-1: none yet; +inf: the
    // factorisation failed), FP64 moments forced for the rest of the closure, and the binary
    // exponent of the largest w_q e^{alpha.m_q} of the last reduced-precision pass (the
    // per-cell shift of the next one)
    double cnd;
    int fp64, cshift;
    int hprec; // precision of the last Hessian: 0 FP64, 1 BF16, 2 3xTF32
};

// Largest moment count (N+1)^2 whose padding to 8 gives NT tiles.
__host__ __device__ constexpr int max_nm_for(int nt)
{
    return nt == 1 ? 4 : nt == 2 ? 16 : nt == 4 ? 25 : nt == 5 ? 36 : nt == 7 ? 49 : 8 * nt;
}

template <int NT> struct Cfg {
    static constexpr int NMP = 8 * NT;
    static constexpr int NML = max_nm_for(NT);
    static constexpr int NPK = NML * (NML + 1) / 2;
    static constexpr int ROWS = NMP + 1; // basis rows + weight row
    static constexpr int CHUNK = ROWS * QCP;
    static constexpr int NTILE = NT * (NT + 1) / 2;
};

__host__ __device__ constexpr int pidx(int i, int j) { return (i * (i + 1)) / 2 + j; }

// Tile (ib, jb), ib >= jb, of the lower triangle of 8x8 tiles, in row order.
__host__ __device__ constexpr int tix(int ib, int jb) { return ib * (ib + 1) / 2 + jb; }

// Offset of element (r, c) inside a tile: row-major by pairs of columns, the pair index of
// row r XOR-ed with (r / 2) & 3. A pair (r, 2q), (r, 2q + 1) stays 16-byte aligned (the
// Cholesky and DMMA accumulator accesses), and the 8 elements of a column land in 8
// distinct 8-byte bank groups (the substitutions and row norms read columns).
__host__ __device__ constexpr int toff(int r, int c)
{
    return 8 * r + 2 * ((c >> 1) ^ ((r >> 1) & 3)) + (c & 1);
}
// Offset of the pair lane l holds in the m8n8 accumulator layout (row l / 4, pair l % 4).
__host__ __device__ constexpr int tpair(int l) { return toff(l >> 2, 2 * (l & 3)); }

// Per-warp state of one cell. The lower triangle of H (then of its Cholesky factor L) is
// either packed row by row (TILED = false) or stored as the lower triangle of 8x8 tiles of
// the matrix padded to 8 NT rows (TILED = true): tile (ib, jb) at 64 tix(ib, jb), inside the
// tile element (r, c) at toff(r, c); lane l of the m8n8k4 DMMA accumulator layout holds the
// pair at tpair(l). Padding rows are those of the identity. 16-byte alignment keeps
// L of every slot in an array aligned for the double2 tile accesses.
//
// W lanes of a warp work on a cell: the fewest (8, 16 or 32) that cover its padded rows twice, so
// that a warp carries 4, 2 or 1 cells and the serial parts (pivots, substitutions, sums in the
// reference's order) are issued once for all of them. The persistent engine keeps whole warps.
__host__ __device__ constexpr int cell_lanes(int nt) { return nt <= 2 ? 8 : nt <= 4 ? 16 : 32; }

template <int NT, bool TILED = false> struct alignas(16) Slot {
    static constexpr int NMP = Cfg<NT>::NMP;
    static constexpr int W = TILED ? cell_lanes(NT) : 32;
    static constexpr int NTILES = NT * (NT + 1) / 2;
    static constexpr int LSIZE = TILED ? 64 * NTILES : Cfg<NT>::NPK;
    static constexpr bool tiled = TILED;
    static constexpr int nt = NT;
    // alpha0 and uOrig are read by a new regularisation level only. Small orders (several cells
    // per warp) leave them in the cell's global state: two of the six vectors a visit would
    // load and store, and for N = 4 a fourth CTA per SM (54.7 KB each; Newton kernel of M_4
    // 64^3 9.75 -> 7.98 ms, of M_3 visits 2.5% faster). From N = 5 on neither limits, and the slot
    // keeps them (visits were 2% slower without).
    static constexpr bool KEEP = !TILED || W == 32;
    using Kept = typename std::conditional<KEEP, double[NMP], double *>::type;
    // A tiled slot is 48 bytes more than a multiple of 128: the assembly of H gathers moments at
    // 32-byte places of four slots, and a multiple of 32 left it half the banks, with the shared
    // data pipe 75% busy (M_5 visits 4% faster).
    static constexpr int PAD = TILED && KEEP ? 2 : 0;
    double u[NMP], alpha[NMP], g[NMP], d[NMP], alphaOld[NMP], rinv[NMP];
    double L[LSIZE + PAD];
    Kept alpha0, uOrig;
    SlotScalars s;
    // g, d, alphaOld and rinv as one array of 4 NMP doubles (scratch between Hessian visits),
    // addressed through the slot object so that it may span the four vectors
    __device__ __forceinline__ double *scratch()
    {
        return reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(this) +
                                          2 * NMP * sizeof(double));
    }
    // offset of element (i, j), i >= j
    __device__ static __forceinline__ int lx(int i, int j)
    {
        if (TILED)
            return 64 * tix(i >> 3, j >> 3) + toff(i & 7, j & 7);
        return pidx(i, j);
    }
};

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(FULL_MASK, v, o);
    return v;
}

__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = fmax(v, __shfl_xor_sync(FULL_MASK, v, o));
    return v;
}

// The lanes of a cell: mask, synchronisation and exchanges among them (lane arguments of the
// functions below count from the cell's first lane).
template <class S> __device__ __forceinline__ unsigned cell_mask()
{
    return S::W == 32 ? FULL_MASK : ((1u << (S::W & 31)) - 1u) << (threadIdx.x & 31 & ~(S::W - 1));
}
template <class S> __device__ __forceinline__ void cell_sync() { __syncwarp(cell_mask<S>()); }
template <class S, class V> __device__ __forceinline__ V cell_shfl(V v, int src)
{
    return __shfl_sync(cell_mask<S>(), v, src, S::W);
}
template <class S> __device__ __forceinline__ bool cell_any(bool v)
{
    return __any_sync(cell_mask<S>(), v);
}
template <class S> __device__ __forceinline__ double cell_sum(double v)
{
#pragma unroll
    for (int o = S::W / 2; o > 0; o >>= 1)
        v += __shfl_xor_sync(cell_mask<S>(), v, o);
    return v;
}
template <class S> __device__ __forceinline__ double cell_max(double v)
{
#pragma unroll
    for (int o = S::W / 2; o > 0; o >>= 1)
        v = fmax(v, __shfl_xor_sync(cell_mask<S>(), v, o));
    return v;
}

// First index of the largest |x| (LAPACK idamax semantics).
template <class S>
__device__ __forceinline__ int cell_iamax(double a0, double a1, int lane, int n)
{
    double best = (lane < n) ? fabs(a0) : -1.0;
    int bi = lane;
    if (lane + S::W < n) {
        double b = fabs(a1);
        if (b > best) {
            best = b;
            bi = lane + S::W;
        }
    }
#pragma unroll
    for (int o = S::W / 2; o > 0; o >>= 1) {
        double ob = __shfl_xor_sync(cell_mask<S>(), best, o);
        int oi = __shfl_xor_sync(cell_mask<S>(), bi, o);
        if (ob > best || (ob == best && oi < bi)) {
            best = ob;
            bi = oi;
        }
    }
    return bi;
}

__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// ---------------------------------------------------------------- mbarrier / bulk copy

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

// Returns false if the phase did not complete within the iteration limit.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int limit = 1 << 26)
{
    uint32_t addr = smem_u32(bar);
    for (int it = 0; it < limit; ++it) {
        uint32_t done;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(done)
                     : "r"(addr), "r"(parity)
                     : "memory");
        if (done)
            return true;
    }
    return false;
}

__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// After a wait that gave up at chunk k of n: one thread waits, again with a limit, for the copies
// in flight in the ring of ST stages (chunk j in stage (seq + j) % ST), which must not land in
// shared memory that the CTA has given back.
template <int ST> __device__ __noinline__ void ring_drain(uint64_t *full, uint32_t seq, int k, int n)
{
    for (int j = k; j < k + ST && j < n; ++j)
        mbar_wait(&full[(seq + j) % ST], ((seq + j) / ST) & 1u, 1 << 20);
}

// ---------------------------------------------------------------- per-warp linear algebra

// In-place right-looking Cholesky of the packed lower triangle; returns LAPACK info.
template <class S>
__device__ int warp_cholesky_packed(S &sl, int n, int lane)
{
    double *P = sl.L;
    for (int j = 0; j < n; ++j) {
        double ajj = P[pidx(j, j)];
        if (!(ajj > 0.0))
            return j + 1;
        double ljj = sqrt(ajj);
        double r = 1.0 / ljj;
        __syncwarp();
        if (lane == 0)
            P[pidx(j, j)] = ljj;
        for (int i = j + 1 + lane; i < n; i += 32)
            P[pidx(i, j)] *= r;
        __syncwarp();
        // trailing update P(i,k) -= L(i,j) L(k,j), j < k <= i < n, flattened over the warp
        int m = n - j - 1;
        int total = m * (m + 1) / 2;
        int ii = 0, kk = lane;
        while (kk > ii) { // locate element number `lane` in row-major triangle order
            kk -= ii + 1;
            ++ii;
        }
        for (int e = lane; e < total; e += 32) {
            int i = j + 1 + ii, k = j + 1 + kk;
            P[pidx(i, k)] = fma(-P[pidx(i, j)], P[pidx(k, j)], P[pidx(i, k)]);
            kk += 32;
            while (kk > ii) {
                kk -= ii + 1;
                ++ii;
            }
        }
        __syncwarp();
    }
    return 0;
}

// Blocked Cholesky of the tiled lower triangle (Slot<NT, true>); returns LAPACK info.
// Per tile column kb: lane l holds row l % 8 of the diagonal tile (the four octets repeat each
// other) and the 8 columns are factored with shuffles inside the tile; then each lane solves
// rows of the panel below against that tile, one row of 8 elements at a time, and the trailing
// tiles (ib, jb), kb < jb <= ib, receive -L(ib,kb) L(jb,kb)^T as two m8n8k4 DMMAs each (lane l
// holds L[l/4][4s + l%4] for k-step s, which is the A fragment of L(ib,kb) and the B fragment
// of L(jb,kb)^T). Every element sees the operations of the column-by-column form in its order.
// Nothing reads the factor's diagonal: the solves take the reciprocal pivots 1 / L_jj (sl.rinv),
// and the diagonal's places keep the pivots L_jj^2. The chain of pivots (reciprocal square roots)
// bounds it; the loop over tile columns stays rolled so that the code fits the instruction cache.
template <class S>
__device__ int warp_cholesky_tiled(S &sl, int n, int lane)
{
    constexpr int T = S::nt;
    static_assert(sizeof(S) % 16 == 0 && (8 * 8 * S::NMP) % 16 == 0,
                  "tiles must be 16-byte aligned in every slot");
    double *A = sl.L;
    int info = 0;
#pragma unroll 1
    for (int kb = 0; kb < T; ++kb) {
        double *D = A + 64 * tix(kb, kb);
        const int row = lane & 7;
        double v[8], rj[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double2 x = *reinterpret_cast<const double2 *>(&D[toff(row, 2 * q)]);
            v[2 * q] = x.x;
            v[2 * q + 1] = x.y;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            rj[j] = 1.0;
            // padding columns (identity rows, zero couplings, last tile only) stay as they are
            if (8 * kb + j < n) {
                const double ajj = cell_shfl<S>(v[j], j);
                if (!(ajj > 0.0) && info == 0)
                    info = 8 * kb + j + 1;
                rj[j] = rsqrt(ajj);
                if (row > j)
                    v[j] *= rj[j];
#pragma unroll
                for (int c = j + 1; c < 8; ++c) {
                    const double lc = cell_shfl<S>(v[j], c);
                    if (row >= c)
                        v[c] = fma(-v[j], lc, v[c]);
                }
            }
        }
        cell_sync<S>();
        if (lane < 8) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                *reinterpret_cast<double2 *>(&D[toff(row, 2 * q)]) =
                    make_double2(v[2 * q], v[2 * q + 1]);
        }
        if (lane == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                *reinterpret_cast<double2 *>(&sl.rinv[8 * kb + 2 * q]) =
                    make_double2(rj[2 * q], rj[2 * q + 1]);
        }
        cell_sync<S>();
#pragma unroll 1
        for (int i = lane; i < 8 * (T - 1 - kb); i += S::W) {
            double *P = A + 64 * tix(kb + 1 + (i >> 3), kb);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double2 x = *reinterpret_cast<const double2 *>(&P[toff(i & 7, 2 * q)]);
                v[2 * q] = x.x;
                v[2 * q + 1] = x.y;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[j] *= rj[j];
#pragma unroll
                for (int c = j + 1; c < 8; ++c)
                    v[c] = fma(-v[j], D[toff(c, j)], v[c]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
                *reinterpret_cast<double2 *>(&P[toff(i & 7, 2 * q)]) =
                    make_double2(v[2 * q], v[2 * q + 1]);
        }
        cell_sync<S>();
        if constexpr (S::W == 32) {
            const int f0 = toff(lane >> 2, lane & 3), f1 = toff(lane >> 2, 4 + (lane & 3));
#pragma unroll 1
            for (int jb = kb + 1; jb < T; ++jb) {
                const double *Bt = A + 64 * tix(jb, kb);
                const double b0 = Bt[f0], b1 = Bt[f1];
                // (four tiles at a time with loads first took 126 registers instead of 96 and was
                // 4% slower on the standalone orders, whose warps per SM it lowers)
#pragma unroll 2
                for (int ib = jb; ib < T; ++ib) {
                    const double *At = A + 64 * tix(ib, kb);
                    double2 *cp = reinterpret_cast<double2 *>(&A[64 * tix(ib, jb) + tpair(lane)]);
                    double2 c = *cp;
                    dmma(c.x, c.y, -At[f0], b0);
                    dmma(c.x, c.y, -At[f1], b1);
                    *cp = c;
                }
            }
        } else {
            // part of a warp per cell: row i's 8 columns of each trailing tile by FMAs
#pragma unroll 1
            for (int i = lane; i < 8 * (T - 1 - kb); i += S::W) {
                const int ib = kb + 1 + (i >> 3), r = i & 7;
                const double *P = A + 64 * tix(ib, kb);
                double p[8];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const double2 x = *reinterpret_cast<const double2 *>(&P[toff(r, 2 * q)]);
                    p[2 * q] = x.x;
                    p[2 * q + 1] = x.y;
                }
#pragma unroll 1
                for (int jb = kb + 1; jb <= ib; ++jb) {
                    const double *B = A + 64 * tix(jb, kb);
                    double *C = A + 64 * tix(ib, jb);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        double2 *cp = reinterpret_cast<double2 *>(&C[toff(r, 2 * q)]);
                        double2 c = *cp;
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const double2 x = *reinterpret_cast<const double2 *>(&B[toff(2 * q, 2 * k)]);
                            const double2 y = *reinterpret_cast<const double2 *>(&B[toff(2 * q + 1, 2 * k)]);
                            c.x = fma(-p[2 * k], x.x, c.x);
                            c.x = fma(-p[2 * k + 1], x.y, c.x);
                            c.y = fma(-p[2 * k], y.x, c.y);
                            c.y = fma(-p[2 * k + 1], y.y, c.y);
                        }
                        *cp = c;
                    }
                }
            }
        }
        cell_sync<S>();
    }
    return info;
}

template <class S>
__device__ __forceinline__ int warp_cholesky(S &sl, int n, int lane)
{
    if constexpr (S::tiled)
        return warp_cholesky_tiled(sl, n, lane);
    else
        return warp_cholesky_packed(sl, n, lane);
}

// x <- (L L^T)^{-1} x, x distributed as x0 = x[lane], x1 = x[lane+32]; column-oriented
// substitution (the order of the reference BLAS dtrsv and of src/utils.cpp:71-86).
// exactDiv selects division by L_kk (as the reference's own dpotrs) instead of the
// precomputed reciprocal.
template <class S>
__device__ __forceinline__ void warp_apply_inverse_tiled(const S &sl, int lane, double &x0,
                                                         double &x1);

template <class S>
__device__ void warp_apply_inverse(const S &sl, int n, int lane, double &x0, double &x1,
                                   bool exactDiv)
{
    if constexpr (S::tiled) {
        // the reciprocals serve both the estimate and the direction here: the blocked
        // factor already rounds differently from the reference's unblocked one
        (void)n;
        (void)exactDiv;
        warp_apply_inverse_tiled(sl, lane, x0, x1);
        return;
    }
    const double *P = sl.L;
    for (int k = 0; k < n; ++k) {
        double v = (k < S::W) ? x0 : x1;
        double xk = cell_shfl<S>(v, k & (S::W - 1));
        xk = exactDiv ? xk / P[S::lx(k, k)] : xk * sl.rinv[k];
        if (lane == (k & (S::W - 1))) {
            if (k < S::W)
                x0 = xk;
            else
                x1 = xk;
        }
        if (lane > k && lane < n)
            x0 = fma(-P[S::lx(lane, k)], xk, x0);
        if (lane + S::W > k && lane + S::W < n)
            x1 = fma(-P[S::lx(lane + S::W, k)], xk, x1);
    }
    for (int k = n - 1; k >= 0; --k) {
        double v = (k < S::W) ? x0 : x1;
        double xk = cell_shfl<S>(v, k & (S::W - 1));
        xk = exactDiv ? xk / P[S::lx(k, k)] : xk * sl.rinv[k];
        if (lane == (k & (S::W - 1))) {
            if (k < S::W)
                x0 = xk;
            else
                x1 = xk;
        }
        if (lane < k && lane < n)
            x0 = fma(-P[S::lx(k, lane)], xk, x0);
        if (lane + S::W < k && lane + S::W < n)
            x1 = fma(-P[S::lx(k, lane + S::W)], xk, x1);
    }
}

// x <- (L L^T)^{-1} x on the tiled factor: tile-blocked substitution. Every lane solves the
// diagonal tile's 8 rows (gathered by shuffles) in its own registers with the reciprocal
// pivots sl.rinv, in the order of the column-oriented form; the tiles off the diagonal act as
// 8-column mat-vec updates of the rows below (forward) or above (backward). Padding rows (L = I
// there, reciprocal 1) keep finite values and never feed the real rows. (One shuffle per row
// instead: 18.3k clocks per solve at n = 64.)
template <class S>
__device__ __forceinline__ void warp_apply_inverse_tiled(const S &sl, int lane, double &x0,
                                                         double &x1)
{
    constexpr int T = S::nt;
    constexpr int NMP = S::NMP;
    const double *A = sl.L;
    const int own = lane & 7;
    // the block's values and reciprocals; the lane's own row takes its value back
    auto gather = [&](int kb, double (&y)[8], double (&r)[8]) {
        const double v = kb < S::W / 8 ? x0 : x1;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            y[i] = cell_shfl<S>(v, (8 * kb + i) & (S::W - 1));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double2 t = *reinterpret_cast<const double2 *>(&sl.rinv[8 * kb + 2 * q]);
            r[2 * q] = t.x;
            r[2 * q + 1] = t.y;
        }
    };
    auto scatter = [&](int kb, const double (&y)[8]) {
        double v = y[0];
#pragma unroll
        for (int i = 1; i < 8; ++i)
            v = own == i ? y[i] : v;
        if ((lane >> 3) == (kb & (S::W / 8 - 1))) {
            if (kb < S::W / 8)
                x0 = v;
            else
                x1 = v;
        }
    };
#pragma unroll 1
    for (int kb = 0; kb < T; ++kb) {
        const double *D = A + 64 * tix(kb, kb);
        double y[8], r[8];
        gather(kb, y, r);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
#pragma unroll
            for (int q = 0; 2 * q < k; ++q) {
                const double2 l = *reinterpret_cast<const double2 *>(&D[toff(k, 2 * q)]);
                y[k] = fma(-l.x, y[2 * q], y[k]);
                if (2 * q + 1 < k)
                    y[k] = fma(-l.y, y[2 * q + 1], y[k]);
            }
            y[k] *= r[k];
        }
        scatter(kb, y);
        if (kb + 1 < T) {
            if (lane >= 8 * kb + 8 && lane < NMP) {
                const double *Lt = A + 64 * tix(lane >> 3, kb);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const double2 l = *reinterpret_cast<const double2 *>(&Lt[toff(own, 2 * q)]);
                    x0 = fma(-l.x, y[2 * q], x0);
                    x0 = fma(-l.y, y[2 * q + 1], x0);
                }
            }
            if (NMP > S::W && lane + S::W >= 8 * kb + 8 && lane + S::W < NMP) {
                const double *Lt = A + 64 * tix((lane + S::W) >> 3, kb);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const double2 l = *reinterpret_cast<const double2 *>(&Lt[toff(own, 2 * q)]);
                    x1 = fma(-l.x, y[2 * q], x1);
                    x1 = fma(-l.y, y[2 * q + 1], x1);
                }
            }
        }
    }
#pragma unroll 1
    for (int kb = T - 1; kb >= 0; --kb) {
        const double *D = A + 64 * tix(kb, kb);
        double y[8], r[8];
        gather(kb, y, r);
#pragma unroll
        for (int i = 7; i >= 0; --i) {
            y[i] *= r[i];
#pragma unroll
            for (int k = 0; k < i; ++k)
                y[k] = fma(-D[toff(i, k)], y[i], y[k]);
        }
        scatter(kb, y);
        if (lane < 8 * kb) {
            const double *Lt = A + 64 * tix(kb, lane >> 3);
#pragma unroll
            for (int c = 0; c < 8; ++c)
                x0 = fma(-Lt[toff(c, own)], y[c], x0);
        }
        if (NMP > S::W && lane + S::W < 8 * kb) {
            const double *Lt = A + 64 * tix(kb, (lane + S::W) >> 3);
#pragma unroll
            for (int c = 0; c < 8; ++c)
                x1 = fma(-Lt[toff(c, own)], y[c], x1);
        }
    }
}

template <class S>
__device__ __forceinline__ double vsum_abs(double x0, double x1, int lane, int n)
{
    double s = (lane < n ? fabs(x0) : 0.0) + (lane + S::W < n ? fabs(x1) : 0.0);
    return cell_sum<S>(s);
}

// Hager/Higham 1-norm estimate of (L L^T)^{-1} (N. J. Higham, ACM TOMS 14 (1988)
// 381-396, Alg. 4.1 -- the algorithm of LAPACK's dlacn2 as driven by dpocon).
// Returns 1/rcond with rcond = (1/est)/anorm.
template <class S>
__device__ double warp_condest(const S &sl, int n, int lane, double anorm)
{
    if (anorm == 0.0)
        return 1.0 / 0.0;
    double x0 = 1.0 / (double)n, x1 = 1.0 / (double)n;
    warp_apply_inverse(sl, n, lane, x0, x1, false);
    double est;
    if (n == 1) {
        est = fabs(cell_shfl<S>(x0, 0));
    } else {
        est = vsum_abs<S>(x0, x1, lane, n);
        int s0 = x0 >= 0.0 ? 1 : -1, s1 = x1 >= 0.0 ? 1 : -1;
        x0 = (double)s0;
        x1 = (double)s1;
        warp_apply_inverse(sl, n, lane, x0, x1, false);
        int j = cell_iamax<S>(x0, x1, lane, n);
        int iter = 2;
        for (;;) {
            x0 = (lane == j) ? 1.0 : 0.0;
            x1 = (lane + S::W == j) ? 1.0 : 0.0;
            warp_apply_inverse(sl, n, lane, x0, x1, false);
            double estold = est;
            est = vsum_abs<S>(x0, x1, lane, n);
            bool diff = (lane < n && (x0 >= 0.0 ? 1 : -1) != s0) ||
                        (lane + S::W < n && (x1 >= 0.0 ? 1 : -1) != s1);
            bool same = !cell_any<S>(diff);
            if (same || est <= estold)
                break;
            s0 = x0 >= 0.0 ? 1 : -1;
            s1 = x1 >= 0.0 ? 1 : -1;
            x0 = (double)s0;
            x1 = (double)s1;
            warp_apply_inverse(sl, n, lane, x0, x1, false);
            int jlast = j;
            j = cell_iamax<S>(x0, x1, lane, n);
            double xjl = cell_shfl<S>(jlast < S::W ? x0 : x1, jlast & (S::W - 1));
            double xj = fabs(cell_shfl<S>(j < S::W ? x0 : x1, j & (S::W - 1)));
            if (xjl != xj && iter < 5) {
                ++iter;
                continue;
            }
            break;
        }
        x0 = ((lane & 1) ? -1.0 : 1.0) * (1.0 + (double)lane / (double)(n - 1));
        x1 = (((lane + S::W) & 1) ? -1.0 : 1.0) * (1.0 + (double)(lane + S::W) / (double)(n - 1));
        warp_apply_inverse(sl, n, lane, x0, x1, false);
        double temp = 2.0 * (vsum_abs<S>(x0, x1, lane, n) / (double)(3 * n));
        if (temp > est)
            est = temp;
    }
    if (est == 0.0)
        return 1.0 / 0.0;
    double rcond = (1.0 / est) / anorm;
    return 1.0 / rcond;
}

template <class S>
__device__ __forceinline__ double cell_nrm2(const double *v, int n, int lane)
{
    double s = 0.0;
    if (lane < n)
        s = v[lane] * v[lane];
    if (lane + S::W < n)
        s = fma(v[lane + S::W], v[lane + S::W], s);
    return sqrt(cell_sum<S>(s));
}

// ---------------------------------------------------------------- Newton state machine

struct Outputs {
    double *u, *alpha;
    int *iters, *iterGamma, *regIdx, *status;
    unsigned long long *failCount; // cells finishing with a non-zero status
    unsigned long long *stats;     // running counters, layout STAT_* (may be null)
    double *gamma, *normG;         // final gamma and |g| per cell (may be null)
    float *cond;                   // condition estimate of the last Hessian per cell, read at
                                   // set-up as the mixed closure's first precision hint (may be null)
};

template <class S>
__device__ void finalize(S &sl, const ClosureParams &P, const Outputs &O, int lane)
{
    const int nm = P.nm;
    long long c = sl.s.cell;
    cell_sync<S>();
    if (sl.s.status != CELL_NONPOSITIVE_U0) {
        // postProcess: rescale (src/opt/optBatch.cpp:334-344, src/opt/opt.cpp:352-354)
        for (int i = lane; i < nm; i += S::W) {
            O.u[c * nm + i] = sl.u[i] * sl.s.u0;
            double a = sl.alpha[i];
            if (i == 0)
                a = a + sl.s.alphaScale;
            O.alpha[c * nm + i] = a;
        }
    }
    if (lane == 0) {
        if (O.iters) O.iters[c] = sl.s.totalIter;
        if (O.iterGamma) O.iterGamma[c] = sl.s.iterGamma < 0 ? 0 : sl.s.iterGamma;
        if (O.regIdx) O.regIdx[c] = sl.s.regIndex;
        if (O.status) O.status[c] = sl.s.status;
        if (O.gamma) O.gamma[c] = sl.s.gamma;
        if (O.normG) O.normG[c] = sl.s.err;
        if (O.cond) O.cond[c] = (float)sl.s.cnd;
        if (sl.s.status != CELL_OK && O.failCount)
            atomicAdd(O.failCount, 1ull);
        if (O.stats) {
            unsigned long long it = (unsigned long long)sl.s.totalIter;
            unsigned long long ig = (unsigned long long)(sl.s.iterGamma < 0 ? 0 : sl.s.iterGamma);
            atomicAdd(&O.stats[STAT_CELLS], 1ull);
            atomicAdd(&O.stats[STAT_ITERS], it);
            atomicAdd(&O.stats[STAT_ITER_GAMMA], ig);
            atomicMax(&O.stats[STAT_MAX_ITER], it);
            atomicMax(&O.stats[STAT_MAX_ITER_GAMMA], ig);
            if (sl.s.status != CELL_OK)
                atomicAdd(&O.stats[STAT_FAILED], 1ull);
            atomicAdd(&O.stats[STAT_REG_HIST + (sl.s.regIndex & 15)], 1ull);
            atomicAdd(&O.stats[STAT_ITER_HIST + (it < 63 ? it : 63)], 1ull);
        }
        sl.s.need = NEED_NONE;
        sl.s.cell = -1;
    }
    cell_sync<S>();
}

// Regularise (src/opt/opt.cpp:251-279). Returns false if the ladder is exhausted.
template <class S>
__device__ bool regularize(S &sl, const ClosureParams &P, int lane)
{
    const int nm = P.nm;
    cell_sync<S>();
    if (sl.s.regIndex >= P.nreg - 1)
        return false;
    int ri = sl.s.regIndex + 1;
    double r = P.reg[ri];
    for (int i = lane; i < nm; i += S::W)
        sl.u[i] = (i == 0) ? 1.0 : sl.uOrig[i] * (1.0 - r);
    cell_sync<S>();
    double rt = P.batched ? P.tol : cell_nrm2<S>(sl.u, nm, lane) * P.tol;
    for (int i = lane; i < nm; i += S::W)
        sl.alpha[i] = sl.alpha0[i];
    cell_sync<S>();
    if (lane == 0) {
        sl.s.regIndex = ri;
        sl.s.r = r;
        sl.s.rtol = rt;
        sl.s.iterGamma = 0;
        sl.s.iter = 0;
        sl.s.t = 1.0;
        if (!P.batched && ri == P.nreg - 1)
            sl.s.maxIter = 10 * sl.s.maxIter;
    }
    cell_sync<S>();
    return true;
}

// Starts the next Newton iteration. When the iteration is bound to regularise
// whatever H turns out to be (t == 0 after a failed line search, or the
// iteration cap reached), the regularisation is applied here without the H pass.
template <class S>
__device__ void begin_iteration(S &sl, const ClosureParams &P, const Outputs &O, int lane)
{
    for (;;) {
        cell_sync<S>();
        int maxIterEff = sl.s.maxIter;
        if (P.batched && sl.s.regIndex == P.nreg - 1)
            maxIterEff = 10 * P.maxIter;
        int iter = sl.s.iter + 1, total = sl.s.totalIter + 1;
        long long passes = sl.s.passes + 1;
        cell_sync<S>();
        if (lane == 0) {
            sl.s.iter = iter;
            sl.s.totalIter = total;
            sl.s.passes = passes;
        }
        cell_sync<S>();
        if (passes > P.passBudget) {
            if (lane == 0)
                sl.s.status = CELL_PASS_BUDGET;
            finalize(sl, P, O, lane);
            return;
        }
        if (total > 1 && (sl.s.t == 0.0 || iter >= maxIterEff)) {
            if (!regularize(sl, P, lane)) {
                if (lane == 0)
                    sl.s.status = CELL_LADDER_EXHAUSTED;
                finalize(sl, P, O, lane);
                return;
            }
            continue;
        }
        if (lane == 0)
            sl.s.need = (P.probe && total == 1) ? NEED_PROBE : NEED_H;
        cell_sync<S>();
        return;
    }
}

template <class S>
__device__ void load_cell(S &sl, const ClosureParams &P, const Outputs &O, long long c,
                          int lane)
{
    const int nm = P.nm;
    constexpr int NMP = S::NMP;
    double u0 = O.u[c * nm];
    double alphaScale = log(u0) * 2.0 * sqrt(M_PI);
    for (int i = lane; i < NMP; i += S::W) {
        double ui = 0.0, ai = 0.0;
        if (i < nm) {
            ui = O.u[c * nm + i] / u0;
            ai = O.alpha[c * nm + i];
            if (i == 0)
                ai = ai - alphaScale;
        }
        sl.u[i] = ui;
        sl.uOrig[i] = ui;
        sl.alpha[i] = ai;
        sl.alpha0[i] = ai;
        sl.g[i] = 0.0;
        sl.d[i] = 0.0;
    }
    cell_sync<S>();
    double rt = P.batched ? P.tol : cell_nrm2<S>(sl.u, nm, lane) * P.tol;
    if (lane == 0) {
        sl.s.cell = c;
        sl.s.passes = 0;
        sl.s.u0 = u0;
        sl.s.alphaScale = alphaScale;
        sl.s.rtol = rt;
        sl.s.t = 1.0;
        sl.s.r = 0.0;
        sl.s.gamma = 0.0;
        sl.s.err = 0.0;
        sl.s.iter = 0;
        sl.s.totalIter = 0;
        sl.s.iterGamma = 0;
        sl.s.regIndex = 0;
        sl.s.maxIter = P.maxIter;
        sl.s.status = CELL_OK;
        sl.s.cnd = O.cond ? (double)O.cond[c] : -1.0;
        sl.s.fp64 = 0;
        sl.s.cshift = 0;
        sl.s.hprec = 0;
    }
    cell_sync<S>();
    if (u0 <= 0) {
        if (lane == 0)
            sl.s.status = CELL_NONPOSITIVE_U0;
        finalize(sl, P, O, lane);
        return;
    }
    begin_iteration(sl, P, O, lane);
}

// Sets alpha = alphaOld + t d and requests a trial pass, or gives up with t = 0.
template <class S>
__device__ void next_trial(S &sl, const ClosureParams &P, const Outputs &O, int lane);

template <class S>
__device__ void next_trial(S &sl, const ClosureParams &P, const Outputs &O, int lane)
{
    const int nm = P.nm;
    double t = sl.s.t;
    cell_sync<S>();
    if (t * sl.s.maxFactor > EPS_HALF) {
        for (int i = lane; i < nm; i += S::W)
            sl.alpha[i] = __dadd_rn(sl.alphaOld[i], __dmul_rn(t, sl.d[i]));
        cell_sync<S>();
        if (lane == 0) {
            sl.s.need = NEED_TRIAL;
            if (O.stats)
                atomicAdd(&O.stats[STAT_TRIALS], 1ull);
        }
        cell_sync<S>();
    } else {
        // backtracked all the way (src/opt/linesearch.cpp:76-78)
        for (int i = lane; i < nm; i += S::W)
            sl.alpha[i] = sl.alphaOld[i];
        cell_sync<S>();
        // mixed precision: a direction from a reduced-precision Hessian is not the reference's
        // Newton direction; the iteration is redone from alphaOld with FP64 moments instead of
        // regularising
        const bool redo = P.mixed && sl.s.hprec != 0;
        if (lane == 0) {
            sl.s.t = redo ? 1.0 : 0.0;
            if (redo) {
                sl.s.fp64 = 1;
                if (O.stats)
                    atomicAdd(&O.stats[STAT_ESCALATED], 1ull);
            }
        }
        cell_sync<S>();
        begin_iteration(sl, P, O, lane);
    }
}

// A reduced-precision Hessian visit is redone with FP64 moments (same iteration); the cell
// keeps FP64 moments for the rest of the closure.
template <class S>
__device__ void escalate_fp64(S &sl, const Outputs &O, int lane)
{
    cell_sync<S>();
    if (lane == 0) {
        sl.s.fp64 = 1;
        sl.s.passes += 1;
        sl.s.need = NEED_H;
        if (O.stats)
            atomicAdd(&O.stats[STAT_ESCALATED], 1ull);
    }
    cell_sync<S>();
}

// f0 - sum_i a_i b_i (SUB) or f0 + sum_i a_i b_i over i < n in ascending order, unfused as the
// reference's loops: the products by the cell's lanes, through rinv (free outside
// the substitutions), the sum by its first lane. Returned to all lanes.
template <bool SUB, class S>
__device__ __forceinline__ double serial_dot(S &sl, double f0, const double *a, const double *b,
                                             int n, int lane)
{
    for (int i = lane; i < n; i += S::W)
        sl.rinv[i] = __dmul_rn(a[i], b[i]);
    cell_sync<S>();
    if (lane == 0)
#pragma unroll 4
        for (int i = 0; i < n; ++i)
            f0 = SUB ? __dsub_rn(f0, sl.rinv[i]) : __dadd_rn(f0, sl.rinv[i]);
    f0 = cell_shfl<S>(f0, 0);
    cell_sync<S>();
    return f0;
}

// gext (mixed precision): the FP64 moments <m_i e^{alpha.m}> and fqext = <e^{alpha.m}> of
// the pass, from which g and f are formed instead of from row 0 of the reduced-precision H.
// emin, emax: bounds of e^{alpha.m} over the quadrature (0: none).
template <class S>
__device__ void after_hessian(S &sl, const ClosureParams &P, const Outputs &O, int lane,
                              double m0, const double *gext = nullptr, double fqext = 0.0,
                              double emin = 0.0, double emax = 0.0)
{
    const int nm = P.nm;
    C3D_NCLK_DECL
    // g_i = H_i0 / m_0 - u_i ; f = H_00 / m_0^2 - alpha.u  (src/opt/fobj.cpp:121-129)
    for (int i = lane; i < nm; i += S::W)
        sl.g[i] = gext ? __dsub_rn(gext[i], sl.u[i]) : sl.L[S::lx(i, 0)] / m0 - sl.u[i];
    cell_sync<S>();
    if (gext && P.mixPolish > 0.0) {
        const double e0 = cell_nrm2<S>(sl.g, nm, lane);
        if (e0 > sl.s.rtol && e0 <= P.mixPolish * sl.s.rtol) {
            escalate_fp64(sl, O, lane);
            return;
        }
    }
    const double f = serial_dot<true>(sl, gext ? fqext : sl.L[0] / (m0 * m0), sl.alpha, sl.u, nm, lane);
    // emin G <= H <= emax G bounds the 1-norm condition number by nm kappa_2 (after_probe); when
    // that settles the test `condest > condHMax` -- with room for rounding -- neither norms nor
    // estimate are needed. The mixed closure routes by the record, so it takes the estimate.
    double norm1 = 0.0, record = nm * (emax * P.gramHi) / (0.5 * emin * P.gramLo);
    bool condSure = !P.mixed && emin > 0.0 && P.gramLo > 0.0 && record <= 1e12 &&
                    record <= 0.25 * P.condHMax;
    if (!condSure) {
        // 1-norm: max row sum of |H| (src/utils.cpp:35-49)
        double rs = 0.0, gmin = 1.0 / 0.0;
        for (int i = lane; i < nm; i += S::W) {
            double s = 0.0;
            if constexpr (S::tiled) {
                // row i = the row segments of tiles (ib, jb <= ib) and the column segments of
                // tiles (ib' > ib, ib); padding entries are 0
                const int ib = i >> 3, r = i & 7;
                for (int jb = 0; jb < ib; ++jb) {
                    const double *Lt = sl.L + 64 * tix(ib, jb);
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        s += fabs(Lt[toff(r, c)]);
                }
                const double *D = sl.L + 64 * tix(ib, ib);
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    s += fabs(c <= r ? D[toff(r, c)] : D[toff(c, r)]);
                for (int ib2 = ib + 1; ib2 < S::nt; ++ib2) {
                    const double *Lt = sl.L + 64 * tix(ib2, ib);
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        s += fabs(Lt[toff(c, r)]);
                }
            } else {
                for (int j = 0; j < nm; ++j)
                    s += fabs(j <= i ? sl.L[S::lx(i, j)] : sl.L[S::lx(j, i)]);
            }
            rs = fmax(rs, s);
            gmin = fmin(gmin, 2.0 * sl.L[S::lx(i, i)] - s); // Gershgorin: H_ii - sum_{j!=i} |H_ij|
        }
        norm1 = cell_max<S>(rs);
        gmin = -cell_max<S>(-gmin);
        // All eigenvalues of H are >= gmin, so when gmin > 0, ||H^-1||_1 <= sqrt(n)/gmin and the
        // 1-norm condition number is at most norm1 sqrt(n)/gmin. The Hager estimate can only be
        // smaller, so if this bound is below condHMax/2 the reference's test is false whatever the
        // estimate; the estimate is then skipped.
        record = norm1 * sqrt((double)nm) / gmin;
        condSure = gmin > 0.0 && record <= 0.5 * P.condHMax;
    }
    if (lane == 0) // the condition record: the bound, or the estimate below
        sl.s.cnd = condSure ? record : 0.0;
    cell_sync<S>();
    C3D_NCLK(O.stats, 1, lane);
    int info = warp_cholesky(sl, nm, lane);
    C3D_NCLK(O.stats, 2, lane);
    double cond = 0.0;
    if (info == 0) {
        // reciprocal pivots (the tiled factorisation leaves them in rinv)
        if constexpr (!S::tiled)
            for (int i = lane; i < nm; i += S::W)
                sl.rinv[i] = 1.0 / sl.L[S::lx(i, i)];
        cell_sync<S>();
        if (!condSure)
            cond = warp_condest(sl, nm, lane, norm1);
    }
    cell_sync<S>();
    C3D_NCLK(O.stats, 3, lane);

    if (lane == 0 && (info != 0 || !condSure))
        sl.s.cnd = info != 0 ? 1.0 / 0.0 : cond;
    bool bad = (info != 0) || (cond > P.condHMax);
    if (gext && bad) {
        escalate_fp64(sl, O, lane);
        return;
    }
    if (sl.s.totalIter == 1 && bad) {
        // isotropic restart (src/opt/opt.cpp:236-247)
        double rt = P.batched ? P.tol : cell_nrm2<S>(sl.u, nm, lane) * P.tol;
        for (int i = lane; i < nm; i += S::W) {
            double a = (i == 0) ? 2.0 * sqrt(M_PI) * log(0.5 / sqrt(M_PI)) : 0.0;
            sl.alpha0[i] = a;
            sl.alpha[i] = a;
        }
        cell_sync<S>();
        if (lane == 0) {
            sl.s.rtol = rt;
            sl.s.iter = 0;
            sl.s.iterGamma = 0;
            sl.s.t = 1.0;
        }
        cell_sync<S>();
        begin_iteration(sl, P, O, lane);
        return;
    }
    int maxIterEff = sl.s.maxIter;
    if (P.batched && sl.s.regIndex == P.nreg - 1)
        maxIterEff = 10 * P.maxIter;
    if (sl.s.iter >= maxIterEff || bad || sl.s.t == 0.0) {
        if (!regularize(sl, P, lane)) {
            if (lane == 0)
                sl.s.status = CELL_LADDER_EXHAUSTED;
            finalize(sl, P, O, lane);
            return;
        }
        begin_iteration(sl, P, O, lane);
        return;
    }
    // d = -H^{-1} g
    double x0 = lane < nm ? sl.g[lane] : 0.0;
    double x1 = lane + S::W < nm ? sl.g[lane + S::W] : 0.0;
    warp_apply_inverse(sl, nm, lane, x0, x1, true);
    if (lane < nm)
        sl.d[lane] = -x0;
    if (lane + S::W < nm)
        sl.d[lane + S::W] = -x1;
    cell_sync<S>();
    C3D_NCLK(O.stats, 4, lane);
    double err = cell_nrm2<S>(sl.g, nm, lane);
    double d1 = vsum_abs<S>(x0, x1, lane, nm);
    int pnOrder = (int)floor(sqrt((double)nm)) + 1;
    double minf = sqrt((2 * pnOrder + 1) / (2 * M_PI));
    double gamma = exp(2.0 * d1 * minf);
    double tolEff = sl.s.rtol;
    if (lane == 0) {
        sl.s.err = err;
        sl.s.gamma = gamma;
    }
    cell_sync<S>();
    if (err <= tolEff && gamma <= P.tolGamma) {
        finalize(sl, P, O, lane);
        return;
    }
    // line search set-up (src/opt/linesearch.cpp:41-54)
    double mf = 0.0;
    for (int i = lane; i < nm; i += S::W) {
        sl.alphaOld[i] = sl.alpha[i];
        mf = fmax(mf, fabs(sl.d[i]) / (fabs(sl.alpha[i]) + 1e-100));
    }
    mf = cell_max<S>(mf);
    cell_sync<S>();
    const double gd = serial_dot<false>(sl, 0.0, sl.g, sl.d, nm, lane);
    if (lane == 0) {
        if (err <= tolEff)
            sl.s.iterGamma += 1;
        sl.s.f = f;
        sl.s.maxFactor = mf;
        sl.s.gd = gd;
        sl.s.t = 1.0;
    }
    cell_sync<S>();
    next_trial(sl, P, O, lane);
}

// First visit of a cell after the probe pass. pm: the probe's entry -- the first-order
// moments mom_i (i < NMP, rows of M2 = the basis), then f's sum, e_min and e_max of
// e^{alpha.m_q}. g is formed as the full visit would form it: FP64 closure, from the Gaunt
// terms of the Hessian's column 0 (g0: g0n terms per row in the reference's CSR order, col
// -2 padding; H_i0 = sum_t v_t mom_col_t, g_i = H_i0 / m_0 - u_i, src/opt/fobj.cpp:121-129);
// mixed closure (g0 null), g_i = mom_i - u_i. The full visit ends the cell converged
// (src/opt/optBatch.cpp:185-250) when info = 0, cond <= condHMax, |g| <= rtol and
// gamma = exp(2 minf |d|_1) <= tolGamma. With lambda_min(H) >= e_min gramLo and
// lambda_max(H) <= e_max gramHi (exact arithmetic; halved for rounding): the 1-norm condition
// estimate is at most nm kappa_2 <= nm e_max gramHi / (e_min gramLo), kept below condHMax / 4
// (Cholesky of such an H succeeds); |d|_1 <= sqrt(nm) |g|_2 / lambda_min, and the gamma
// exponent is kept below half of log(tolGamma). A cell meeting these is finalized with the
// same multipliers, moments and counts as the full visit would give (its gamma record is the
// bound); any other goes on to the Hessian pass of the same iteration.
template <class S>
__device__ void after_probe(S &sl, const ClosureParams &P, const Outputs &O, int lane, double m0,
                            const double *pm, const GauntTerm *g0, int g0n)
{
    const int nm = P.nm;
    constexpr int NMP = S::NMP;
    for (int i = lane; i < nm; i += S::W) {
        double gi;
        if (g0) {
            double h = 0.0;
            for (int t = 0; t < g0n; ++t) {
                const GauntTerm e = g0[i * g0n + t];
                if (e.col >= 0)
                    h = __dadd_rn(h, __dmul_rn(pm[e.col], e.v));
            }
            gi = h / m0 - sl.u[i];
        } else {
            gi = __dsub_rn(pm[i], sl.u[i]);
        }
        sl.g[i] = gi;
    }
    cell_sync<S>();
    const double err = cell_nrm2<S>(sl.g, nm, lane);
    const double emin = pm[NMP + 1], emax = pm[NMP + 2];
    int maxIterEff = sl.s.maxIter;
    if (P.batched && sl.s.regIndex == P.nreg - 1)
        maxIterEff = 10 * P.maxIter;
    // (symmetric passes: the full visit's sums may round otherwise, within certSlack; a cell that
    // close to the tolerance is left to the full visit)
    bool ok = err + (P.sym ? P.certSlack : 0.0) <= sl.s.rtol && sl.s.iter < maxIterEff && sl.s.t != 0.0 && P.tolGamma > 1.0 &&
              emin > 0.0 && emax < 1.0 / 0.0 && P.gramLo > 0.0;
    double k1 = 0.0, gexp = 0.0;
    if (ok) {
        const double lam = 0.5 * emin * P.gramLo;
        k1 = nm * (emax * P.gramHi) / lam;
        const int pnOrder = (int)floor(sqrt((double)nm)) + 1;
        const double minf = sqrt((2 * pnOrder + 1) / (2 * M_PI));
        gexp = 2.0 * minf * sqrt((double)nm) * err / lam;
        ok = k1 <= 0.25 * P.condHMax && gexp <= 0.5 * log(P.tolGamma);
    }
    cell_sync<S>();
    if (ok) {
        if (lane == 0) {
            sl.s.err = err;
            sl.s.gamma = exp(gexp);
            sl.s.cnd = k1;
            if (O.stats)
                atomicAdd(&O.stats[STAT_CERTIFIED], 1ull);
        }
        cell_sync<S>();
        finalize(sl, P, O, lane);
        return;
    }
    if (lane == 0) {
        sl.s.passes += 1;
        sl.s.need = NEED_H;
        // mixed precision: a gradient already within the polish range would make the
        // reduced-precision Hessian visit of this iteration escalate (after_hessian); the cell
        // goes to the FP64 visit directly, with the same permanent FP64 routing
        if (P.mixed && P.mixPolish > 0.0 && err > sl.s.rtol && err <= P.mixPolish * sl.s.rtol)
            sl.s.fp64 = 1;
    }
    cell_sync<S>();
}

// Returns whether the trial was accepted: the iteration that then begins (unless it regularises)
// is at the trial's multipliers. A rejected last trial may begin one too, at the old ones.
template <class S>
__device__ bool after_trial(S &sl, const ClosureParams &P, const Outputs &O, int lane,
                            double fquad)
{
    const int nm = P.nm;
    const double fnew = serial_dot<true>(sl, fquad, sl.alpha, sl.u, nm, lane);
    double t = sl.s.t;
    bool accept = fnew <= __dadd_rn(sl.s.f, __dmul_rn(__dmul_rn(1e-3, t), sl.s.gd));
    cell_sync<S>();
    if (accept) {
        begin_iteration(sl, P, O, lane);
        return true;
    }
    if (lane == 0)
        sl.s.t = 0.5 * t;
    cell_sync<S>();
    next_trial(sl, P, O, lane);
    return false;
}

} // namespace

} // namespace c3d
