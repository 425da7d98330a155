// The kinetic flux over an octant-symmetric quadrature (sym.cuh): the ansatz of the grid cells
// and the limited upwind stencil with its projection (src/flux_kinetic.cpp:20-198).
#include "sym.cuh"

namespace c3d {

namespace {

__device__ __forceinline__ uint32_t saddr(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void bar_init(uint64_t *b, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(saddr(b)), "r"(count));
}
__device__ __forceinline__ void bar_arrive(uint64_t *b)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(saddr(b)) : "memory");
}
// false if the phase did not complete within the iteration limit
__device__ __forceinline__ bool bar_wait(uint64_t *b, uint32_t parity)
{
    for (int it = 0; it < (1 << 26); ++it) {
        uint32_t done;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(done)
                     : "r"(saddr(b)), "r"(parity)
                     : "memory");
        if (done)
            return true;
    }
    return false;
}
// 16 bytes global -> shared, asynchronous
__device__ __forceinline__ void copy16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
// arrives on b once the thread's copies so far have landed (the arrival is in b's count)
__device__ __forceinline__ void copy_arrive(uint64_t *b)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(saddr(b)) : "memory");
}

} // namespace

// ---------------------------------------------------------------- ansatz

// psi (rows r0 <= row < r1, whole groups of 32 from r0 on; layout sym.cuh) = exp(alpha_c . m)
// (M_N) or alpha_c . m (P_N) for either all cells (list null) or the marked cells of the *count groups of 8
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
                const int row = 32 * (2 * b + e); // first row of the group
                if (c >= 0 && row >= r0 && row < r1) {
                    double *p = psi + ((long long)((row - r0) / 4) * nall + c) * 4 + (lane & 3);
#pragma unroll
                    for (int s = 0; s < 8; ++s)
                        p[(long long)(4 * s) * nall] = isPn ? z[e][s] : exp(z[e][s]);
                }
            }
        }
    }
}

// ---------------------------------------------------------------- stencil and projection

// Slope of the limited reconstruction at a value with differences dm (to its upwind neighbour),
// dp (to its downwind one) and dc across both, times 2: 2 minmod(th dp, dc / 2, th dm) =
// minmod(th2 dp, dc, th2 dm) (src/flux_kinetic.cpp:45-61), th2 = 2 th >= 0, for dm and dp of one sign (dc then
// has it too, and min(th |dm|, th |dp|) = th min(|dm|, |dp|)); otherwise it is 0. (The selects as
// predicated FP64 operations: 24 instructions fewer per cell and direction, 7% slower, since 12
// more go to the FP64 pipe.)
__device__ __forceinline__ double sym_slope(double th2, double dm, double dp, double dc)
{
    const double m = th2 * (fabs(dm) < fabs(dp) ? dm : dp);
    return fabs(dc) < fabs(m) ? dc : m;
}
// f += q s if a and b have one sign (a predicated FMA; as C++ it became an FMA and two selects)
__device__ __forceinline__ void sym_add_same(double &f, double q, double s, double a, double b)
{
    asm("{\n .reg .pred p;\n setp.ge.s32 p, %3, 0;\n @p fma.rn.f64 %0, %1, %2, %0;\n}\n"
        : "+d"(f)
        : "d"(q), "d"(s), "r"(__double2hiint(a) ^ __double2hiint(b)));
}

// Limited upwind difference along one axis in upwind coordinates, v2, v1 the upwind
// neighbours, v0 the cell, w1 the downwind neighbour:
//   f = (v0 + s(v1, v0, w1) / 2) - (v1 + s(v2, v1, v0) / 2)  (s / 2 = sym_slope / 4),
// summed from the difference v0 - v1, which the slopes need too, so that a zero slope is a
// predicated-off FMA instead of a select.
// A direction of the opposite sign gives the mirror image with f and the cosine both negated,
// so f |cosine| serves every octant.
__device__ __forceinline__ double sym_axis(double th2, double v2, double v1, double v0, double w1)
{
    const double d2 = v1 - v2, d1 = v0 - v1, d0 = w1 - v0;
    const double s1 = sym_slope(th2, d1, d0, w1 - v1), s2 = sym_slope(th2, d2, d1, v0 - v2);
    double f = d1;
    sym_add_same(f, 0.25, s1, d1, d0);
    sym_add_same(f, -0.25, s2, d2, d1);
    return f;
}

// Tile of a CTA: TX x 4 lines of 8 cells along z, one warp per line, staged with its halo per
// reflection and group of 4 octant directions as [TX + 3][7][12][4] doubles: x planes and y rows
// in upwind order (mirrored for the reflections that flip the axis), z ascending from k0 - 2,
// directions innermost (a warp reads 8 cells x 4 directions as 256 consecutive bytes).
template <int TX> struct FluxTile {
    static constexpr int TY = 4, TZ = 8, RY = TY + 3, RZ = TZ + 4;
    static constexpr int PZ = 4, PY = RZ * PZ, PX = RY * PY; // strides of a cell along z, y, x
    static constexpr int SLOT = (TX + 3) * PX;
    static constexpr int WARPS = TX * TY;           // stencil warps; then TX copy warps
    static constexpr int COPIERS = 32 * TX, THREADS = 32 * WARPS + COPIERS;
    // 16-byte copies of a slot: the tile's planes (4 full lines, 3 halo lines), the x halo planes
    static constexpr int FULL = 2 * RZ, INNER = 2 * TZ, PLANE = TY * FULL + 3 * INNER;
    static constexpr int COPIES = TX * PLANE + 3 * TY * INNER;
    static constexpr int PER = (COPIES + COPIERS - 1) / COPIERS;
};

// flux(c) (+)= sum_q m_q (c_x fx + c_y fy + c_z fz) on the interior cells, c = cosine x weight /
// spacing, over the rows r0 <= row < r1 of psi (whole groups of 4 octant directions). Lane l of
// a warp owns cell l / 4 of the warp's line and, in group g, octant direction 4 g + l % 4: it
// forms the stencil of the 8 reflections one after another (signs known at compile time),
// transforms the 8 values (sym_wht) and contracts them per class on the FP64 tensor pipe, A
// fragments straight from registers. A reflection's stage has its own ring slot, filled by
// copy warps that run up to 8 stages ahead; warps drift against each other inside the ring (full
// and empty barriers, no CTA barrier).
// Bound by the FP64 pipe's latency and issue: 137 warp instructions per 32 (cell, direction)
// pairs, 44 of them FP64; 0.6 instructions per clock and scheduler, FP64 pipe 39%, ALU 51%, DRAM
// 30%. M_6 64^3: 2.61 ms per call, 128^3: 20.6 ms (5.2 and 40.2 ms with all directions as one run
// each and no symmetry); M_4 64^3 1.31 ms, M_3 37 x 45 x 51 0.31 ms.
// (Bulk copies, one per line of cells, took 76 clocks each: 2.6 times slower as a whole. One
// barrier per pair of reflections spilled: N <= 5 1 to 6% slower, N = 6 1% faster.)
// wrapFlag (null: no): when it reads 0 the face ghosts' psi is not in place; their values are
// read at the periodic images.
template <int DEG, int TX>
__global__ void __launch_bounds__(FluxTile<TX>::THREADS, TX == 4 ? 1 : 2)
    sym_flux_kernel(GridDims g, const double *__restrict__ psi, const double *__restrict__ tab,
                    const int *__restrict__ idx, int r0, int r1, double th2, int accumulate,
                    double *__restrict__ flux, int *errorFlag, const int *wrapFlag)
{
    using C = SymCls<DEG>;
    using F = FluxTile<TX>;
    constexpr int TAB = C::TILES * 32 + 16; // a group's fragments and weights
    extern __shared__ __align__(128) double smem[]; // 8 x SLOT, 2 x TAB
    double *sTab = smem + 8 * F::SLOT;
    __shared__ uint64_t full[8], empty[8];
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
    if (tid == 0) {
        for (int s = 0; s < 8; ++s) {
            bar_init(&full[s], F::COPIERS);
            bar_init(&empty[s], F::WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    const int g0 = r0 / 32, ng = (r1 - r0 + 31) / 32;
    if (warp >= F::WARPS) {
        // Copy warps. A thread's copies have fixed places in a slot; their sources are the cells of
        // the lines from k0 - 2 (halo lines: the tile's 8 cells) in upwind order for either x and
        // y flip, at the periodic image of a wrapped ghost. Positions outside the grid read a
        // cell inside it: only cells outside the grid use them.
        const bool wrap = wrapFlag && *wrapFlag == 0;
        auto image = [&](int a, int m) { return !wrap ? a : a < 2 ? a + m : a >= m + 2 && a < m + 4 ? a - m : a; };
        uint32_t dst[F::PER], off[F::PER][2][2]; // bytes; 16-byte units from the rows' start
        const int ct = tid - 32 * F::WARPS;
#pragma unroll
        for (int n = 0; n < F::PER; ++n) {
            int f = min(ct + n * F::COPIERS, F::COPIES - 1), X, Y, h;
            if (f < TX * F::PLANE) {
                X = 2 + f / F::PLANE;
                f %= F::PLANE;
                if (f < F::TY * F::FULL) {
                    Y = 2 + f / F::FULL;
                    h = f % F::FULL;
                } else {
                    f -= F::TY * F::FULL;
                    Y = f / F::INNER;
                    Y = Y < 2 ? Y : F::TY + 2;
                    h = 4 + f % F::INNER;
                }
            } else {
                f -= TX * F::PLANE;
                X = f / (F::TY * F::INNER);
                X = X < 2 ? X : TX + 2;
                f %= F::TY * F::INNER;
                Y = 2 + f / F::INNER;
                h = 4 + f % F::INNER;
            }
            dst[n] = saddr(smem) + (uint32_t)(X * F::PX + Y * F::PY + h * 2) * 8;
            const int k = min(image(k0 - 2 + h / 2, g.nz), g.nzg() - 1);
#pragma unroll
            for (int sx = 0; sx < 2; ++sx)
#pragma unroll
                for (int sy = 0; sy < 2; ++sy) {
                    const int i = min(image(sx ? i0 + TX + 1 - X : i0 + X - 2, g.nx), g.nxg() - 1);
                    const int j = min(image(sy ? j0 + F::TY + 1 - Y : j0 + Y - 2, g.ny), g.nyg() - 1);
                    off[n][sx][sy] = (uint32_t)(2 * g.cell(i, j, k) + (h & 1));
                }
        }
        for (int gi = 0; gi < ng; ++gi) {
            bool ok = true;
            sym_for<8>([&](auto ss) {
                constexpr int s = ss.value;
                if (gi > 0 && !bar_wait(&empty[s], (gi - 1) & 1))
                    ok = false;
                const double *rows = psi + (long long)(8 * gi + s) * nall * 4;
#pragma unroll
                for (int n = 0; n < F::PER; ++n)
                    if (F::COPIES % F::COPIERS == 0 || ct + n * F::COPIERS < F::COPIES)
                        copy16(dst[n] + s * F::SLOT * 8, rows + 2ull * off[n][s & 1][(s >> 1) & 1]);
                if (s == 0)
                    for (int e = ct; e < TAB / 2; e += F::COPIERS)
                        copy16(saddr(sTab + (gi & 1) * TAB + 2 * e), tab + (size_t)(g0 + gi) * TAB + 2 * e);
                copy_arrive(&full[s]);
            });
            if (!ok) {
                atomicExch(errorFlag, 1);
                break;
            }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        return;
    }
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
    // the lane's cell in a slot for either x and y flip
    const double *cellAt[2][2];
#pragma unroll
    for (int sx = 0; sx < 2; ++sx)
#pragma unroll
        for (int sy = 0; sy < 2; ++sy)
            cellAt[sx][sy] = smem + ((sx ? TX - 1 - wx : wx) + 2) * F::PX +
                             ((sy ? F::TY - 1 - wy : wy) + 2) * F::PY + (z + 2) * F::PZ + d;
    bool ok = true;
    for (int gi = 0; gi < ng && ok; ++gi) {
        double S[8], cx = 0.0, cy = 0.0, cz = 0.0;
        const double *tb = sTab + (gi & 1) * TAB;
        sym_for<8>([&](auto ss) {
            constexpr int s = ss.value, dz = (s & 4) ? -F::PZ : F::PZ;
            if (!bar_wait(&full[s], gi & 1))
                ok = false;
            if (s == 0) {
                cx = tb[C::TILES * 32 + d];
                cy = tb[C::TILES * 32 + 4 + d];
                cz = tb[C::TILES * 32 + 8 + d];
            }
            const double *q = cellAt[s & 1][(s >> 1) & 1] + s * F::SLOT;
            const double v0 = q[0];
            const double fx = sym_axis(th2, q[-2 * F::PX], q[-F::PX], v0, q[F::PX]);
            const double fy = sym_axis(th2, q[-2 * F::PY], q[-F::PY], v0, q[F::PY]);
            const double fz = sym_axis(th2, q[-2 * dz], q[-dz], v0, q[dz]);
            S[s] = fma(fx, cx, fma(fy, cy, fz * cz));
            __syncwarp();
            if (lane == 0)
                bar_arrive(&empty[s]);
        });
        sym_wht(S);
        sym_contract<DEG>(S, tb, lane, acc);
    }
    if (!ok) {
        if (lane == 0)
            atomicExch(errorFlag, 1);
        return;
    }
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

template <int DEG, int TX>
static cudaError_t flux_v(const GridDims &g, const double *psi, const double *tab, const int *idx,
                          int r0, int r1, double th2, double *flux, int *errorFlag,
                          const int *wrapFlag, cudaStream_t st)
{
    using F = FluxTile<TX>;
    const int smem = (8 * F::SLOT + 2 * (SymCls<DEG>::TILES * 32 + 16)) * 8;
    auto kern = sym_flux_kernel<DEG, TX>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess)
        return e;
    const long long tiles = (long long)((g.nx + TX - 1) / TX) * ((g.ny + F::TY - 1) / F::TY) *
                            ((g.nz + F::TZ - 1) / F::TZ);
    kern<<<(unsigned)tiles, F::THREADS, smem, st>>>(g, psi, tab, idx, r0, r1, th2, r0 > 0 ? 1 : 0,
                                                    flux, errorFlag, wrapFlag);
    return cudaGetLastError();
}

template <int DEG>
static cudaError_t flux_t(const GridDims &g, const double *psi, const double *tab, const int *idx,
                          int r0, int r1, double th2, double *flux, int *errorFlag,
                          const int *wrapFlag, int numSMs, cudaStream_t st)
{
    // Tiles of 4 x planes: one CTA of 640 threads per SM, so whole waves of numSMs tiles. Tiles of
    // 2: two CTAs per SM, more halo (5 / 2 of psi against 7 / 4), measured in waves of the former
    // as 0.75 for up to a tile per SM, then 0.54 per tile and SM and a tail of 0.3, 1.06 at least.
    // M_6, 20 x 20 directions, 4 against 2 planes: 16^3 98 and 73 us, 24^3 99 and 106, 28^3 197
    // and 172, 32^3 198 and 210, 40^3 389 and 370, 64^3 1358 and 1443 (M_2, M_4 in proportion).
    const long long lines = (long long)((g.ny + 3) / 4) * ((g.nz + 7) / 8);
    const double x = (double)(lines * ((g.nx + 1) / 2)) / numSMs;
    const double two = x <= 1.0 ? 0.75 : fmax(1.06, 0.54 * x + 0.3);
    const long long four = (lines * ((g.nx + 3) / 4) + numSMs - 1) / numSMs;
    return four <= two
               ? flux_v<DEG, 4>(g, psi, tab, idx, r0, r1, th2, flux, errorFlag, wrapFlag, st)
               : flux_v<DEG, 2>(g, psi, tab, idx, r0, r1, th2, flux, errorFlag, wrapFlag, st);
}

// The stencil over psi's rows r0 <= row < r1 (psi points at row r0, a multiple of 32); accumulates
// when r0 > 0.
cudaError_t launch_sym_flux(const GridDims &g, int deg, const double *psi, const double *tab,
                            const int *idx, int r0, int r1, double theta, double *flux,
                            int *errorFlag, const int *wrapFlag, int numSMs, cudaStream_t st)
{
    const double th2 = theta > 0.0 ? 2.0 * theta : 0.0;
#define CALL(D) flux_t<D>(g, psi, tab, idx, r0, r1, th2, flux, errorFlag, wrapFlag, numSMs, st)
    C3D_SYM_DEG(CALL)
#undef CALL
}

} // namespace c3d
