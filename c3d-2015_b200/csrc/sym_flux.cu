// The kinetic flux over an octant-symmetric quadrature (sym.cuh): the ansatz of the grid cells
// and the limited upwind stencil with its projection (src/flux_kinetic.cpp:20-198). Both forms
// of psi's producer (this file's ansatz kernel and the closure's probe) and its consumer use
// octant order, row 8 o + s.
#include "sym.cuh"

namespace c3d {

namespace {

__device__ __forceinline__ uint32_t saddr(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Asynchronous global -> shared copy of BYTES (8 or 16).
template <int BYTES> __device__ __forceinline__ void copy_async(uint32_t dst, const double *src)
{
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

} // namespace

// ---------------------------------------------------------------- ansatz

// psi[(row - r0) nall + c] = exp(alpha_c . m_row) (M_N) or alpha_c . m_row (P_N) for the rows
// r0 <= row < r1 and either all cells (list null) or the marked cells of the *count groups of 8
// consecutive cells in list (psi_groups_kernel), those whose multipliers a closure changed after
// its probe had written their psi. A warp holds 8 cells'
// multipliers as A fragments in shared memory and forms 64 exponents of each per block
// (sym_expand). Work items are (8 cells, a share of the blocks): a short list splits the
// blocks over the grid's warps.
// Bound by the FP64 pipe (16 DMMAs and 16 exponentials per lane and block for M_6).
template <int DEG>
__global__ void __launch_bounds__(128)
    sym_ansatz_kernel(SymTables T, int nm, long long nall, const double *__restrict__ alpha,
                      const long long *__restrict__ list, const unsigned int *__restrict__ count, int r0,
                      int r1, int isPn, double *__restrict__ psi)
{
    using C = SymCls<DEG>;
    __shared__ double sA[4][C::STEPS * 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *aF = sA[warp];
    const int b0 = r0 / (8 * SYM_BLK), b1 = (r1 + 8 * SYM_BLK - 1) / (8 * SYM_BLK);
    const long long groups = list ? (long long)*count : (nall + 7) / 8, warps = (long long)gridDim.x * 4;
    long long split = groups > 0 ? warps / groups : 1;
    split = split < 1 ? 1 : split > b1 - b0 ? b1 - b0 : split;
    const int per = (int)((b1 - b0 + split - 1) / split);
    for (long long w = (long long)blockIdx.x * 4 + warp; w < groups * split; w += warps) {
        const long long entry = list ? list[w / split] : (w / split) << 8 | 0xff;
        long long c = (entry >> 8) * 8 + (lane >> 2);
        if (!((entry >> (lane >> 2)) & 1) || c >= nall)
            c = -1;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < C::STEPS; ++k) {
            const int m = T.stepIdx[4 * k + (lane & 3)];
            aF[k * 32 + lane] = c >= 0 && m >= 0 ? alpha[c * nm + m] : 0.0;
        }
        __syncwarp();
        const int lo = b0 + (int)(w % split) * per, hi = min(b1, lo + per);
        for (int b = lo; b < hi; ++b) {
            double z[2][8];
            sym_expand<DEG>(aF, T.expo + (size_t)b * C::STEPS * 32, lane, z);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int row = 8 * (SYM_BLK * b + 2 * (lane & 3) + e);
                if (c >= 0 && row >= r0 && row < r1) {
                    double *p = psi + (long long)(row - r0) * nall + c;
#pragma unroll
                    for (int s = 0; s < 8; ++s)
                        p[(long long)s * nall] = isPn ? z[e][s] : exp(z[e][s]);
                }
            }
        }
    }
}

// ---------------------------------------------------------------- stencil and projection

// Slope of the limited reconstruction at a value with differences dm (to its upwind neighbour),
// dp (to its downwind one) and dc across both, times 4: minmod(th dp, dc / 2, th dm)
// (src/flux_kinetic.cpp:45-61) scaled by 2, th2 = 2 th >= 0, for dm and dp of one sign (sym_same;
// dc then has it too, and min(th |dm|, th |dp|) = th min(|dm|, |dp|)); otherwise it is 0.
__device__ __forceinline__ double sym_slope(double th2, double dm, double dp, double dc)
{
    const double m = th2 * (fabs(dm) < fabs(dp) ? dm : dp);
    return fabs(dc) < fabs(m) ? dc : m;
}
__device__ __forceinline__ bool sym_same(double a, double b)
{
    return (__double2hiint(a) ^ __double2hiint(b)) >= 0;
}

// Limited upwind difference along one axis in upwind coordinates, v2, v1 the upwind
// neighbours, v0 the cell, w1 the downwind neighbour:
//   f = (v0 + s(v1, v0, w1) / 2) - (v1 + s(v2, v1, v0) / 2),
// summed from the difference v0 - v1, which the slopes need too, so that a zero slope is a
// predicated-off FMA instead of a select.
// A direction of the opposite sign gives the mirror image with f and the cosine both negated,
// so f |cosine| serves every octant.
__device__ __forceinline__ double sym_axis(double th2, double v2, double v1, double v0, double w1)
{
    const double d2 = v1 - v2, d1 = v0 - v1, d0 = w1 - v0;
    const double s1 = sym_slope(th2, d1, d0, w1 - v1), s2 = sym_slope(th2, d2, d1, v0 - v2);
    double f = d1;
    if (sym_same(d1, d0))
        f = fma(0.25, s1, f);
    if (sym_same(d2, d1))
        f = fma(-0.25, s2, f);
    return f;
}

// Tile of a CTA: TX x 4 lines of 8 cells along z, one warp per line, staged with its halo per
// direction as [TX + 3][7][12] doubles: x planes and y rows in upwind order (mirrored for the
// reflections that flip the axis), z ascending from k0 - 2. The direction stride is 4 or 12
// mod 16 doubles, so the 4 directions x 4 cells that half a warp reads at once fall into
// distinct banks.
template <int TX> struct FluxTile {
    static constexpr int TY = 4, TZ = 8, RY = TY + 3, RZ = TZ + 4, PX = RY * RZ;
    static constexpr int DIR = (TX + 3) * PX;
    static constexpr int THREADS = 32 * TX * TY;
    static constexpr int PAIR = 8 * DIR; // a stage: 4 octant directions x the two x flips
    static constexpr int STAGES = 4;
    static_assert(DIR % 16 == 4 || DIR % 16 == 12, "bank pattern");
};

// flux(c) (+)= sum_q m_q (c_x fx + c_y fy + c_z fz) on the interior cells, c = cosine x weight /
// spacing, over the rows r0 <= row < r1 of psi (whole groups of 4 octant directions unless r1
// is the last row). Lane l of a warp owns cell l / 4 of the warp's line and, in group g, octant
// direction 4 g + l % 4: it forms the stencil of the 8 reflections one after another (a stage
// holds two, signs known at compile time), transforms the 8 values (sym_wht) and contracts
// them per class on the FP64 tensor pipe, A fragments straight from registers. Stages are filled
// by cp.async two pairs ahead, one barrier per pair. VEC: doubles per copy (2 when nz is even,
// so that rows are 16-byte aligned).
// wrapFlag (null: no): when it reads 0 the face ghosts' psi is not in place; their values are
// read at the periodic images.
template <int DEG, int TX, int VEC>
__global__ void __launch_bounds__(FluxTile<TX>::THREADS, TX == 4 ? 1 : 2)
    sym_flux_kernel(GridDims g, const double *__restrict__ psi, const double *__restrict__ tab,
                    const int *__restrict__ idx, int r0, int r1, double th2, int accumulate,
                    double *__restrict__ flux, const int *wrapFlag)
{
    using C = SymCls<DEG>;
    using F = FluxTile<TX>;
    constexpr int TAB = C::TILES * 32 + 16; // a group's fragments and weights
    constexpr int TABC = TAB / 2;           // 16-byte chunks
    // copies per direction: the tile's planes (4 full rows, 3 halo rows), then the x halo planes
    constexpr int FULL = F::RZ / VEC, INNER = F::TZ / VEC;
    constexpr int PLANE = F::TY * FULL + 3 * INNER;
    constexpr int PERDIR = TX * PLANE + 3 * F::TY * INNER;
    constexpr int COPIES = (8 * PERDIR + F::THREADS - 1) / F::THREADS;
    extern __shared__ __align__(128) double smem[]; // STAGES x PAIR, 2 x TAB
    double *sTab = smem + F::STAGES * F::PAIR;
    const int nm = g.nm, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long nall = g.nall();
    // tiles in blocks of 4 x 4 along x and y with z inside, so that CTAs running together read
    // each other's halos from L2
    const int ntx = (g.nx + TX - 1) / TX, nty = (g.ny + F::TY - 1) / F::TY,
              ntz = (g.nz + F::TZ - 1) / F::TZ;
    int i0, j0, k0;
    {
        constexpr int B = 4;
        int r = blockIdx.x;
        const int bx = r / (B * nty * ntz);
        r %= B * nty * ntz;
        const int hx = min(B, ntx - bx * B);
        const int by = r / (hx * B * ntz);
        r %= hx * B * ntz;
        const int hy = min(B, nty - by * B);
        i0 = 2 + (bx * B + r / (hy * ntz)) * TX;
        r %= hy * ntz;
        j0 = 2 + (by * B + r / ntz) * F::TY;
        k0 = 2 + (r % ntz) * F::TZ;
    }
    const bool wrap = wrapFlag && *wrapFlag == 0;
    // this thread's copies of a stage: destination (-1: none) and source offset from the
    // stage's first row for either y flip, in doubles. Positions outside the grid read a cell
    // inside it: only cells outside the grid use them.
    int dst[COPIES];
    uint32_t off[COPIES][2];
#pragma unroll
    for (int n = 0; n < COPIES; ++n) {
        const int e = tid + n * F::THREADS;
        const int dir = e / PERDIR; // bit 2: the x flip, bits 0-1: direction of the group
        int f = e % PERDIR, X, Y, kc;
        if (f < TX * PLANE) {
            X = 2 + f / PLANE;
            f %= PLANE;
            if (f < F::TY * FULL) {
                Y = 2 + f / FULL;
                kc = (f % FULL) * VEC;
            } else {
                f -= F::TY * FULL;
                Y = f / INNER;
                Y = Y < 2 ? Y : F::TY + 2;
                kc = 2 + (f % INNER) * VEC;
            }
        } else {
            f -= TX * PLANE;
            X = f / (F::TY * INNER);
            X = X < 2 ? X : TX + 2;
            f %= F::TY * INNER;
            Y = 2 + f / INNER;
            kc = 2 + (f % INNER) * VEC;
        }
        dst[n] = e < 8 * PERDIR ? (((dir * (TX + 3) + X) * F::RY + Y) * F::RZ + kc) * 8 : -1;
        auto image = [&](int a, int m) { return !wrap ? a : a < 2 ? a + m : a >= m + 2 && a < m + 4 ? a - m : a; };
        const int i = min(image(dir & 4 ? i0 + TX + 1 - X : i0 + X - 2, g.nx), g.nxg() - 1);
        const int k = min(image(k0 - 2 + kc, g.nz), g.nzg() - VEC);
#pragma unroll
        for (int sy = 0; sy < 2; ++sy) {
            const int j = min(image(sy ? j0 + F::TY + 1 - Y : j0 + Y - 2, g.ny), g.nyg() - 1);
            off[n][sy] = (uint32_t)((8 * (dir & 3) + ((dir >> 2) & 1)) * nall + g.cell(i, j, k));
        }
    }
    const int g0 = r0 / 32, ng = (r1 + 31) / 32 - g0;
    const uint32_t sBase = saddr(smem);
    // stage of group g0 + gi, reflections with y and z flips p, into ring slot p. The last
    // group's directions past r1 read row r1 - 1's octant direction: their weights are 0.
    auto issue = [&](int gi, int p) {
        if (gi < ng) {
            const int row = 32 * gi + 2 * p; // relative to r0
            const double *src = psi + (long long)row * nall;
            const uint32_t sb = sBase + (uint32_t)(p * F::PAIR) * 8;
            const bool last = row + 26 > r1 - r0;
#pragma unroll
            for (int n = 0; n < COPIES; ++n) {
                if (8 * PERDIR % F::THREADS != 0 && dst[n] < 0)
                    continue;
                uint32_t o = p & 1 ? off[n][1] : off[n][0];
                if (last) {
                    const int dir = (tid + n * F::THREADS) / PERDIR & 3;
                    const int past = 4 * gi + dir - ((r1 - r0) / 8 - 1);
                    if (past > 0)
                        o -= (uint32_t)(8 * past * nall);
                }
                copy_async<8 * VEC>(sb + (uint32_t)dst[n], src + o);
            }
            if (p == 0)
                for (int e = tid; e < TABC; e += F::THREADS)
                    copy_async<16>(saddr(sTab + (gi & 1) * TAB + 2 * e),
                                   tab + (size_t)(g0 + gi) * TAB + 2 * e);
        }
        copy_commit();
    };
    static_assert(F::STAGES == 4, "a ring slot per pair of the group");
#pragma unroll
    for (int p = 0; p < F::STAGES - 1; ++p)
        issue(0, p);
    const int wx = warp / F::TY, wy = warp % F::TY, z = lane >> 2, d = lane & 3;
    const int i = i0 + wx, j = j0 + wy, k = k0 + z;
    const long long myc =
        i < g.nx + 2 && j < g.ny + 2 && k < g.nz + 2 ? g.cell(i, j, k) : -1;
    double acc[C::TILES][2];
#pragma unroll
    for (int t = 0; t < C::TILES; ++t)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int m = idx[8 * t + 2 * d + e];
            acc[t][e] = accumulate && myc >= 0 && m >= 0 ? flux[myc * nm + m] : 0.0;
        }
    // offsets of the lane's cell in a direction's stage for either x and y flip
    int cellAt[2][2];
#pragma unroll
    for (int sx = 0; sx < 2; ++sx)
#pragma unroll
        for (int sy = 0; sy < 2; ++sy)
            cellAt[sx][sy] = (4 * sx + d) * F::DIR + ((sx ? TX - 1 - wx : wx) + 2) * F::PX +
                             ((sy ? F::TY - 1 - wy : wy) + 2) * F::RZ + z + 2;
    for (int gi = 0; gi < ng; ++gi) {
        double S[8], cx = 0.0, cy = 0.0, cz = 0.0;
        const double *tb = sTab + (gi & 1) * TAB;
        sym_for<4>([&](auto pp) {
            constexpr int p = pp.value, sy = p & 1, sz = p >> 1;
            constexpr int dz = sz ? -1 : 1;
            copy_wait<F::STAGES - 2>(); // this thread's copies of the stage have landed
            __syncthreads();            // everyone's, and stage (t - 1)'s readers are done
            issue(p == 0 ? gi : gi + 1, (p + 3) & 3);
            const double *st = smem + p * F::PAIR;
            if (p == 0) {
                cx = tb[C::TILES * 32 + d];
                cy = tb[C::TILES * 32 + 4 + d];
                cz = tb[C::TILES * 32 + 8 + d];
            }
#pragma unroll
            for (int sx = 0; sx < 2; ++sx) {
                const double *q = st + cellAt[sx][sy];
                const double v0 = q[0];
                const double fx = sym_axis(th2, q[-2 * F::PX], q[-F::PX], v0, q[F::PX]);
                const double fy = sym_axis(th2, q[-2 * F::RZ], q[-F::RZ], v0, q[F::RZ]);
                const double fz = sym_axis(th2, q[-2 * dz], q[-dz], v0, q[dz]);
                S[sx + 2 * p] = fma(fx, cx, fma(fy, cy, fz * cz));
            }
        });
        sym_wht(S);
        sym_contract<DEG>(S, tb, lane, acc);
    }
    copy_wait<0>();
    if (myc < 0)
        return;
#pragma unroll
    for (int t = 0; t < C::TILES; ++t)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int m = idx[8 * t + 2 * d + e];
            if (m >= 0)
                flux[myc * nm + m] = acc[t][e];
        }
}

// ---------------------------------------------------------------- launchers

template <int DEG>
static cudaError_t ansatz_t(const SymTables &T, int nm, long long nall, const double *alpha,
                            const long long *list, const unsigned int *count, int r0, int r1, int isPn,
                            double *psi, int numSMs, cudaStream_t st)
{
    const long long warps = (nall + 7) / 8;
    const long long cap = (long long)numSMs * 6;
    const unsigned grid = (unsigned)(list ? cap : (warps + 3) / 4 < 4 * cap ? (warps + 3) / 4 : 4 * cap);
    sym_ansatz_kernel<DEG><<<grid, 128, 0, st>>>(T, nm, nall, alpha, list, count, r0, r1, isPn, psi);
    return cudaGetLastError();
}

#define C3D_SYM_DEG(CALL)                                                                          \
    switch (deg) {                                                                                 \
    case 0: return CALL(0);                                                                        \
    case 1: return CALL(1);                                                                        \
    case 2: return CALL(2);                                                                        \
    case 3: return CALL(3);                                                                        \
    case 4: return CALL(4);                                                                        \
    case 5: return CALL(5);                                                                        \
    case 6: return CALL(6);                                                                        \
    case 7: return CALL(7);                                                                        \
    default: return cudaErrorInvalidValue;                                                         \
    }

cudaError_t launch_sym_ansatz(const SymTables &T, int deg, long long nall, const double *alpha,
                              const long long *list, const unsigned int *count, int r0, int r1, int isPn,
                              double *psi, int numSMs, cudaStream_t st)
{
#define CALL(D)                                                                                    \
    ansatz_t<D>(T, (D + 1) * (D + 1), nall, alpha, list, count, r0, r1, isPn, psi, numSMs, st)
    C3D_SYM_DEG(CALL)
#undef CALL
}

template <int DEG, int TX, int VEC>
static cudaError_t flux_v(const GridDims &g, const double *psi, const double *tab, const int *idx,
                          int r0, int r1, double th2, double *flux, const int *wrapFlag,
                          cudaStream_t st)
{
    using F = FluxTile<TX>;
    const int smem = (F::STAGES * F::PAIR + 2 * (SymCls<DEG>::TILES * 32 + 16)) * 8;
    auto kern = sym_flux_kernel<DEG, TX, VEC>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess)
        return e;
    const long long tiles = (long long)((g.nx + TX - 1) / TX) * ((g.ny + F::TY - 1) / F::TY) *
                            ((g.nz + F::TZ - 1) / F::TZ);
    kern<<<(unsigned)tiles, F::THREADS, smem, st>>>(g, psi, tab, idx, r0, r1, th2, r0 > 0 ? 1 : 0,
                                                    flux, wrapFlag);
    return cudaGetLastError();
}

template <int DEG>
static cudaError_t flux_t(const GridDims &g, const double *psi, const double *tab, const int *idx,
                          int r0, int r1, double th2, double *flux, const int *wrapFlag, int numSMs,
                          cudaStream_t st)
{
    const long long lines = (long long)((g.ny + 3) / 4) * ((g.nz + 7) / 8);
    const bool wide = lines * ((g.nx + 3) / 4) >= 2 * numSMs;
    if (g.nz % 2 == 0)
        return wide ? flux_v<DEG, 4, 2>(g, psi, tab, idx, r0, r1, th2, flux, wrapFlag, st)
                    : flux_v<DEG, 2, 2>(g, psi, tab, idx, r0, r1, th2, flux, wrapFlag, st);
    return wide ? flux_v<DEG, 4, 1>(g, psi, tab, idx, r0, r1, th2, flux, wrapFlag, st)
                : flux_v<DEG, 2, 1>(g, psi, tab, idx, r0, r1, th2, flux, wrapFlag, st);
}

// The stencil over psi's rows r0 <= row < r1 (psi points at row r0); accumulates when r0 > 0.
cudaError_t launch_sym_flux(const GridDims &g, int deg, const double *psi, const double *tab,
                            const int *idx, int r0, int r1, double theta, double *flux,
                            const int *wrapFlag, int numSMs, cudaStream_t st)
{
    const double th2 = theta > 0.0 ? 2.0 * theta : 0.0;
#define CALL(D) flux_t<D>(g, psi, tab, idx, r0, r1, th2, flux, wrapFlag, numSMs, st)
    C3D_SYM_DEG(CALL)
#undef CALL
}

} // namespace c3d
