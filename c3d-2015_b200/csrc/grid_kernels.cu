// Grid kernels of the M_N / P_N time step:
//   ghost fill        src/comm.cpp:281-323 (serial periodic communicateBoundaries)
//   kinetic flux      src/flux_kinetic.cpp:20-198
//   P_N moment flux   src/flux_moment.cpp:15-104
//   Euler stage       src/update.cpp:21-37
//   RK copy / average src/update.cpp:206-212, :268-274
//
// Layout: the reference's, cell-major with the moment index fastest, cells
// (i,j,k) with k fastest and two ghost layers per face; arrays cover all
// (nx+4)(ny+4)(nz+4) cells.
//
// Elementwise stages (ghost fill, Euler, average) reproduce the reference's
// arithmetic bit for bit (unfused operations in its order). The kinetic flux runs its
// two contractions (exponents alpha.m_q, projection onto the moments) on the FP64 tensor
// pipe, so its sums are reordered against the reference's (agreement to ~1e-15 relative).
#include "c3d_common.cuh"

#ifndef M_PI
#define M_PI 3.14159265358979323846
#endif

namespace c3d {


// ---------------------------------------------------------------- ghost fill

// For the ghost cell f of an axis of one cell, where a layer's image may be a ghost itself: the
// faces per layer, and the layer (0, 1 low outer and inner, 2, 3 high inner and outer). 0 else.
__device__ __forceinline__ long long one_cell_axis(const GridDims &g, long long f, int &layer)
{
    const long long px = (long long)g.ny * g.nz, py = (long long)g.nx * g.nz, pz = (long long)g.nx * g.ny;
    const long long per = f < 4 * px ? px : f < 4 * (px + py) ? py : pz;
    const int n = f < 4 * px ? g.nx : f < 4 * (px + py) ? g.ny : g.nz;
    if (n > 1)
        return 0;
    f -= f < 4 * px ? 0 : f < 4 * (px + py) ? 4 * px : 4 * (px + py);
    layer = (int)(f / per);
    return per;
}

// Two periodic ghost layers per face over interior ranges of the other two axes
// (no edges or corners). The three face groups read only interior cells (but for an axis of one
// cell, whose layers one warp copies in order), so they run as one launch. f0 > 0 skips the first f0 faces: f0 = 4 ny nz leaves the x faces to
// the caller (x-slab decomposition, whose x ghosts come from the neighbouring slabs). One warp
// per ghost cell: the cell indices cost several 64-bit divisions.
__global__ void ghost_fill_kernel(GridDims g, double *__restrict__ u, long long f0)
{
    const int lane = threadIdx.x & 31, nm = g.nm;
    const long long total = ghost_faces(g), warps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long f = f0 + (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5); f < total;
         f += warps) {
        long long dst, src;
        ghost_pair(g, f, dst, src);
        int layer;
        const long long per = one_cell_axis(g, f, layer);
        if (per == 0) {
            for (int m = lane; m < nm; m += 32)
                u[dst * nm + m] = u[src * nm + m];
        } else if (layer == 0) {
            // low layers, in the reference's order: the outer one takes the inner one's old values
            long long dst1, src1;
            ghost_pair(g, f + per, dst1, src1);
            for (int m = lane; m < nm; m += 32) {
                u[dst * nm + m] = u[src * nm + m];
                u[dst1 * nm + m] = u[src1 * nm + m];
            }
        } else if (layer >= 2) {
            // high layers: both end with the cell's values
            long long near;
            if (layer == 3)
                ghost_pair(g, f - per, near, src);
            for (int m = lane; m < nm; m += 32)
                u[dst * nm + m] = u[src * nm + m];
        }
    }
}

// What a mirrored closure copies from the periodic images to the face ghosts.
struct MirrorCopy {
    double *u, *alpha;
    int *iters, *iterGamma, *regIdx, *status;
    double *gamma, *normG;
    unsigned long long *stats;
};

// The face ghosts of a mirrored closure, one warp per ghost cell: multipliers, moments and
// records of the image, and the closure statistics a solve of the ghost would have added
// (finalize, closure_core.cuh), so that the totals equal those of solving every cell. The CTA's
// counters are 32-bit in shared memory (native atomics) and go to the context's once per CTA.
__global__ void ghost_mirror_copy_kernel(GridDims g, MirrorCopy C)
{
    __shared__ unsigned int sStat[STAT_COUNT];
    __shared__ unsigned long long sIters, sIterGamma;
    for (int q = threadIdx.x; q < STAT_COUNT; q += blockDim.x)
        sStat[q] = 0;
    if (threadIdx.x == 0)
        sIters = sIterGamma = 0;
    __syncthreads();
    unsigned long long iters = 0, iterGamma = 0;
    const int lane = threadIdx.x & 31, nm = g.nm;
    const long long total = ghost_faces(g), warps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long f = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; f < total; f += warps) {
        long long dst, src;
        ghost_pair(g, f, dst, src);
        for (int m = lane; m < nm; m += 32) {
            C.alpha[dst * nm + m] = C.alpha[src * nm + m];
            C.u[dst * nm + m] = C.u[src * nm + m];
        }
        if (lane == 0) {
            const int it = C.iters[src], ig = C.iterGamma[src], rg = C.regIdx[src], st = C.status[src];
            C.iters[dst] = it;
            C.iterGamma[dst] = ig;
            C.regIdx[dst] = rg;
            C.status[dst] = st;
            C.gamma[dst] = C.gamma[src];
            C.normG[dst] = C.normG[src];
            atomicAdd(&sStat[STAT_CELLS], 1u);
            iters += (unsigned long long)it;
            iterGamma += (unsigned long long)ig;
            atomicMax(&sStat[STAT_MAX_ITER], (unsigned int)it);
            atomicMax(&sStat[STAT_MAX_ITER_GAMMA], (unsigned int)ig);
            if (st != CELL_OK)
                atomicAdd(&sStat[STAT_FAILED], 1u);
            atomicAdd(&sStat[STAT_REG_HIST + (rg & 15)], 1u);
            atomicAdd(&sStat[STAT_ITER_HIST + (it < 63 ? it : 63)], 1u);
        }
    }
    if (iters) {
        atomicAdd(&sIters, iters);
        atomicAdd(&sIterGamma, iterGamma);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < STAT_COUNT; q += blockDim.x) {
        const unsigned long long v =
            q == STAT_ITERS ? sIters : q == STAT_ITER_GAMMA ? sIterGamma : sStat[q];
        if (v == 0)
            continue;
        if (q == STAT_MAX_ITER || q == STAT_MAX_ITER_GAMMA)
            atomicMax(&C.stats[q], v);
        else
            atomicAdd(&C.stats[q], v);
    }
}

// One closure's records along the x-line (i, (ny+3)/2, (nz+3)/2) of interior cells:
// {r, iter, iterGamma, gamma, normG} per cell (src/update.cpp:66-75 unbatched,
// :147-155 batched, where the stored gamma is the gamma-iteration count).
__global__ void line_log_kernel(GridDims g, ClosureParams P, const int *__restrict__ iters,
                                const int *__restrict__ iterGamma, const int *__restrict__ regIdx,
                                const double *__restrict__ gamma, const double *__restrict__ normG,
                                double *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.nx)
        return;
    const long long c = g.cell(2 + i, (g.ny + 3) / 2, (g.nz + 3) / 2);
    double *o = out + (size_t)i * 5;
    o[0] = P.reg[regIdx[c] & 15];
    o[1] = (double)iters[c];
    o[2] = (double)iterGamma[c];
    o[3] = P.batched ? (double)iterGamma[c] : gamma[c];
    o[4] = normG[c];
}

// *flag = 1 if any face ghost of a differs (bitwise) from its periodic image.
__global__ void ghost_mirror_check_kernel(GridDims g, const double *__restrict__ a, int *flag)
{
    const int lane = threadIdx.x & 31, nm = g.nm;
    const long long total = ghost_faces(g), warps = ((long long)gridDim.x * blockDim.x) >> 5;
    const unsigned long long *b = reinterpret_cast<const unsigned long long *>(a);
    bool diff = false;
    for (long long f = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; f < total; f += warps) {
        long long dst, src;
        ghost_pair(g, f, dst, src);
        for (int m = lane; m < nm; m += 32)
            diff |= b[dst * nm + m] != b[src * nm + m];
    }
    if (__syncthreads_or(diff) && threadIdx.x == 0)
        atomicExch(flag, 1);
}

// ---------------------------------------------------------------- ansatz hand-off from the closure

// psi of every face ghost and direction from its periodic image: the closure copied the face
// ghosts' multipliers from their images, so their ansatz values are the images' too (the probe
// pass wrote the solved cells' values). psi is rows x nall x T, T one direction of a cell (the
// general layout) or the 32 bytes of 4 directions (sym.cuh). Grid x: one thread per face ghost,
// consecutive threads on consecutive cells of a z line for the x and y faces; grid y: blocks of
// rPer rows.
struct alignas(32) Psi4 { double v[4]; };
template <class T>
__global__ void psi_face_copy_kernel(GridDims g, int rows, int rPer, T *__restrict__ psi)
{
    const long long nall = g.nall(), total = ghost_faces(g);
    const int r0 = blockIdx.y * rPer, r1 = min(rows, r0 + rPer);
    for (long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x; f < total;
         f += (long long)gridDim.x * blockDim.x) {
        long long dst, src;
        ghost_pair(g, f, dst, src);
#pragma unroll 4
        for (int r = r0; r < r1; ++r)
            psi[r * nall + dst] = psi[r * nall + src];
    }
}

// The groups of 8 consecutive cells with a marked cell, as entries (group << 8) | mask in any
// order, *count of them (zero before); the marks are cleared for the next closure.
__global__ void psi_groups_kernel(unsigned long long *mark, long long groups, long long *list,
                                  unsigned int *count)
{
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < groups;
         g += (long long)gridDim.x * blockDim.x) {
        const unsigned long long m = mark[g];
        if (m == 0)
            continue;
        mark[g] = 0;
        int mask = 0;
#pragma unroll
        for (int r = 0; r < 8; ++r)
            mask |= ((m >> (8 * r)) & 0xff) ? 1 << r : 0;
        list[atomicAdd(count, 1u)] = g << 8 | mask;
    }
}

// psi[q nall + c] = exp(alpha_c . m_q) for the marked cells c of the *count groups of list (one
// warp per group, directions over the lanes; exponent summed in the reference's order, unfused):
// the cells whose multipliers the closure changed after its probe pass had written their psi.
__global__ void psi_refresh_kernel(GridDims g, int nq, const double *__restrict__ M,
                                   const double *__restrict__ alpha,
                                   const long long *__restrict__ list,
                                   const unsigned int *__restrict__ count, double *__restrict__ psi)
{
    const int nm = g.nm;
    const long long nall = g.nall();
    const long long n = 8LL * *count;
    const int lane = threadIdx.x & 31;
    const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long i = w0; i < n; i += nw) {
        const long long e = list[i >> 3];
        if (!((e >> (i & 7)) & 1))
            continue;
        const long long c = (e >> 8) * 8 + (i & 7);
        const double *a = alpha + c * nm;
        for (int q = lane; q < nq; q += 32) {
            const double *m = M + (size_t)q * nm;
            double z = 0.0;
            for (int k = 0; k < nm; ++k)
                z = __dadd_rn(z, __dmul_rn(a[k], m[k]));
            psi[(long long)q * nall + c] = exp(z);
        }
    }
}

// ---------------------------------------------------------------- Euler / RK

// The interior cells of a z line are nz nm consecutive doubles, so the elementwise stages walk
// lines (blockIdx.y strided) with 32-bit indices inside one.
// Calls f(x, c, m) for every element x of moment m of interior cell c.
template <class F> __device__ __forceinline__ void for_interior(const GridDims &g, F &&f)
{
    const int nm = g.nm, len = g.nz * nm, lines = g.nx * g.ny;
    for (int l = blockIdx.y; l < lines; l += gridDim.y) {
        const long long c0 = g.cell(2 + l / g.ny, 2 + l % g.ny, 2);
        for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < len; t += gridDim.x * blockDim.x)
            f(c0 * nm + t, c0 + t / nm, t % nm);
    }
}

// Euler stage. MODE 0: u <- E(u); 1: uOld <- u, then u <- E(u) (the save of the first RK stage,
// where nothing changes u in between); 2: u <- 0.5 (E(u) + uOld) (the last RK stage). E rounds
// as the reference's expressions, unfused.
template <int MODE>
__global__ void euler_kernel(GridDims g, double *__restrict__ u, const double *__restrict__ flux,
                             const double *__restrict__ sigT, const double *__restrict__ sigS,
                             double dt, double *__restrict__ uOld)
{
    for_interior(g, [&](long long x, long long c, int m) {
        const double st = sigT[c], u0 = u[x];
        double v;
        if (m == 0) {
            double fac = __dsub_rn(__dadd_rn(1.0, __dmul_rn(dt, sigS[c])), __dmul_rn(dt, st));
            v = __dsub_rn(__dmul_rn(u0, fac), __dmul_rn(dt, flux[x]));
        } else {
            v = __dsub_rn(__dmul_rn(u0, __dsub_rn(1.0, __dmul_rn(dt, st))), __dmul_rn(dt, flux[x]));
        }
        if (MODE == 1)
            uOld[x] = u0;
        u[x] = MODE == 2 ? __dmul_rn(0.5, __dadd_rn(v, uOld[x])) : v;
    });
}

// uOld <- u (interior cells only)
__global__ void rk_save_kernel(GridDims g, const double *__restrict__ u, double *__restrict__ uOld)
{
    for_interior(g, [&](long long x, long long, int) { uOld[x] = u[x]; });
}

// ---------------------------------------------------------------- kinetic flux on the tensor pipe
//
// Directions come in tiles of 32. Per tile the host prepares (c3d_create) two copies of the
// basis in m8n8k4 fragment order, so that a warp reads each fragment as 32 consecutive
// doubles and a CTA stages a tile with one bulk copy:
//   ansatz     [j 0..3][k-step 0..2NT-1][lane]  M[32t + 8j + lane/4][4k + lane%4]   (B of Z = A M^T)
//   projection [k-step 0..7][j 0..NT-1][lane]   M[32t + 4k + lane%4][8j + lane/4]   (B of F += S M)
//              followed by c_x = (xi w)/dx, c_y = (eta w)/dy, c_z = (mu w)/dz and w of the
//              tile's 32 directions (a direction's limited differences along each axis are
//              weighted by c, whose sign is the cosine's).
// Directions past nq and moments past nm are zero.

constexpr int FLUX_STAGES = 2;

__device__ __forceinline__ void dmma_g(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ uint32_t smem_addr(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void fbar_init(uint64_t *bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_addr(bar)));
}
__device__ __forceinline__ void fbar_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
// Two bulk copies completing one phase of a barrier initialised for one arrival: a single
// arrive.expect_tx with the combined byte count, then both copies.
__device__ __forceinline__ void fbar_load2(void *dst0, const void *src0, uint32_t bytes0, void *dst1,
                                           const void *src1, uint32_t bytes1, uint64_t *bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)),
                 "r"(bytes0 + bytes1)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_addr(dst0)),
                 "l"(src0), "r"(bytes0), "r"(smem_addr(bar))
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_addr(dst1)),
                 "l"(src1), "r"(bytes1), "r"(smem_addr(bar))
                 : "memory");
}
// false if the phase did not complete within the iteration limit
__device__ __forceinline__ bool fbar_wait(uint64_t *bar, uint32_t parity, int limit = 1 << 26)
{
    for (int it = 0; it < limit; ++it) {
        uint32_t done;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(done)
                     : "r"(smem_addr(bar)), "r"(parity)
                     : "memory");
        if (done)
            return true;
    }
    return false;
}

// After a wait that gave up at tile k of n: one thread waits, again with a limit, for the copies in
// flight in the FLUX_STAGES stages (as ring_drain, closure_core.cuh).
__device__ __noinline__ void fbar_drain(uint64_t *bar, int k, int n)
{
    for (int j = k; j < k + FLUX_STAGES && j < n; ++j)
        fbar_wait(&bar[j % FLUX_STAGES], (j / FLUX_STAGES) & 1, 1 << 20);
}

// psi[(q - q0) nall + c] = exp(alpha_c . m_q) (M_N) or alpha_c . m_q (P_N) for the directions
// q0 <= q < q0 + nqc, q0 a multiple of 32. A CTA owns 64 cells (warp w: 8w..8w+7), keeps
// their multipliers as A fragments in registers and walks the direction tiles of the chunk
// (double-buffered bulk copies of the ansatz fragments): 8 NT DMMAs per 8 x 8 block.
template <int NT>
__global__ void __launch_bounds__(256)
    ansatz_dmma_kernel(GridDims g, const double *__restrict__ alpha, const double *__restrict__ mfA,
                       int q0, int nqc, int isPn, double *__restrict__ psi, int *errorFlag)
{
    constexpr int KS = 2 * NT;
    constexpr int TILE = 4 * KS * 32;
    __shared__ __align__(128) double sB[FLUX_STAGES][TILE];
    __shared__ uint64_t bar[FLUX_STAGES];
    __shared__ int sAbort;
    const int nm = g.nm;
    const long long nall = g.nall();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long c = (long long)blockIdx.x * 64 + 8 * warp + (lane >> 2);
    const int t0 = q0 >> 5, nt = (nqc + 31) >> 5;
    if (tid == 0) {
        sAbort = 0;
        for (int s = 0; s < FLUX_STAGES; ++s)
            fbar_init(&bar[s]);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        for (int s = 0; s < FLUX_STAGES && s < nt; ++s)
            fbar_load(sB[s], mfA + (size_t)(t0 + s) * TILE, TILE * 8, &bar[s]);
    }
    double a[KS];
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
        int k = 4 * kk + (lane & 3);
        a[kk] = (c < nall && k < nm) ? alpha[c * nm + k] : 0.0;
    }
    __syncthreads();
    for (int t = 0; t < nt; ++t) {
        const int s = t % FLUX_STAGES;
        if (!fbar_wait(&bar[s], (t / FLUX_STAGES) & 1))
            sAbort = 1;
        if (__syncthreads_or(sAbort)) {
            if (tid == 0) {
                atomicExch(errorFlag, 1);
                fbar_drain(bar, t, nt);
            }
            return;
        }
        const double *B = sB[s];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            double z0 = 0.0, z1 = 0.0;
#pragma unroll
            for (int kk = 0; kk < KS; ++kk)
                dmma_g(z0, z1, a[kk], B[(j * KS + kk) * 32 + lane]);
            const int ql = 32 * t + 8 * j + 2 * (lane & 3); // direction within the chunk
            if (c < nall) {
                if (ql < nqc)
                    psi[(long long)ql * nall + c] = isPn ? z0 : exp(z0);
                if (ql + 1 < nqc)
                    psi[(long long)(ql + 1) * nall + c] = isPn ? z1 : exp(z1);
            }
        }
        refill_fence();
        __syncthreads();
        if (tid == 0 && t + FLUX_STAGES < nt)
            fbar_load(sB[s], mfA + (size_t)(t0 + t + FLUX_STAGES) * TILE, TILE * 8, &bar[s]);
    }
}

// minmod of src/flux_kinetic.cpp:45-50 as a select: the same value (x when |x| < |y|, else
// y, for operands of one sign; 0 otherwise), except possibly for the sign of a zero and for
// operands whose product underflows.
__device__ __forceinline__ double minmod_sel(double x, double y)
{
    return (x * y > 0.0) ? (fabs(x) < fabs(y) ? x : y) : 0.0;
}

// Limited upwind difference along one axis for either sign of the direction weight c (the
// cosine's sign), src/flux_kinetic.cpp:130-189. With h = +1/2 (c > 0: values k1..k4 at offsets
// -2..1) or h = -1/2 (c <= 0: offsets -1..2),
//   f = ((k3 + h s(k2,k3,k4)) - k2) - h s(k1,k2,k3),  s(l,c,r) = slopefit (src/flux_kinetic.cpp:56-61)
//     = minmod(th (r - c), minmod((r - l) / 2, th (c - l))).
// Here s' = 2 s = minmod(2th (r - c), minmod(r - l, 2th (c - l))) and h s = (h/2) s': scaling by
// powers of two commutes with rounding and with the minmod's comparisons, so f rounds as the
// reference's expression with two multiplications fewer per axis (th2 = 2 th).
__device__ __forceinline__ double axis_flux_bf(double c, double th2, const double *pc,
                                               long long st)
{
    const bool pos = c > 0;
    const double *b = pos ? pc - 2 * st : pc - st;
    const double k1 = b[0], k2 = b[st], k3 = b[2 * st], k4 = b[3 * st];
    const double q = pos ? 0.25 : -0.25; // h / 2
    const double t32 = th2 * (k3 - k2);
    const double s1 = minmod_sel(th2 * (k4 - k3), minmod_sel(k4 - k2, t32));
    const double s2 = minmod_sel(t32, minmod_sel(k3 - k1, th2 * (k2 - k1)));
    return fma(-q, s2, fma(q, s1, k3) - k2);
}

// flux(c) (+)= sum_q m_q (c_x fx + c_y fy + c_z fz) (c = cosine x weight / spacing of the
// direction, fx.. the limited differences) for 64 interior cells per CTA (consecutive
// in the interior numbering). Per direction tile: the limited upwind differences S[q][cell]
// of the CTA (each thread 8 (cell, direction) pairs, loads issued two pairs at a time) go to
// shared memory, then F += S^T M on the FP64 tensor pipe (warp w: cells 8w..8w+7, all moment
// tiles), with the projection fragments and direction cosines staged by bulk copies.
template <int NT>
__global__ void __launch_bounds__(256)
    kinetic_dmma_kernel(GridDims g, const double *__restrict__ psi, const double *__restrict__ mfP,
                        int q0, int nqc, double theta, int accumulate, double *__restrict__ flux,
                        int *errorFlag)
{
    constexpr int TILE = 8 * NT * 32 + 128;
    constexpr int CS = 68; // S tile row stride (cells)
    const double th2 = 2.0 * theta;
    extern __shared__ __align__(128) double kinSmem[]; // sB[FLUX_STAGES][TILE], sS[32 * CS]
    double(*sB)[TILE] = reinterpret_cast<double(*)[TILE]>(kinSmem);
    double *sS = kinSmem + FLUX_STAGES * TILE;
    __shared__ long long sCell[64];
    __shared__ uint64_t bar[FLUX_STAGES];
    __shared__ int sAbort;
    const int nm = g.nm;
    const long long nall = g.nall(), nint = g.ninterior();
    const long long n0 = (long long)blockIdx.x * 64;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long sx = (long long)g.nyg() * g.nzg(), sy = g.nzg(), sz = 1;
    const int t0 = q0 >> 5, nt = (nqc + 31) >> 5;
    if (tid == 0) {
        sAbort = 0;
        for (int s = 0; s < FLUX_STAGES; ++s)
            fbar_init(&bar[s]);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        for (int s = 0; s < FLUX_STAGES && s < nt; ++s)
            fbar_load(sB[s], mfP + (size_t)(t0 + s) * TILE, TILE * 8, &bar[s]);
    }
    if (tid < 64)
        sCell[tid] = (n0 + tid < nint) ? interior_cell(g, n0 + tid) : -1;
    __syncthreads();
    const long long myc = sCell[8 * warp + (lane >> 2)];
    double acc[NT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e2 = 0; e2 < 2; ++e2) {
            int m = 8 * j + 2 * (lane & 3) + e2;
            acc[j][e2] = (accumulate && myc >= 0 && m < nm) ? flux[myc * nm + m] : 0.0;
        }
    const int cl = tid & 63;
    const long long c = sCell[cl];
    for (int t = 0; t < nt; ++t) {
        const int s = t % FLUX_STAGES;
        if (!fbar_wait(&bar[s], (t / FLUX_STAGES) & 1))
            sAbort = 1;
        if (__syncthreads_or(sAbort)) {
            if (tid == 0) {
                atomicExch(errorFlag, 1);
                fbar_drain(bar, t, nt);
            }
            return;
        }
        const double *dirs = sB[s] + 8 * NT * 32; // c_x, c_y, c_z, w per direction
#pragma unroll 2
        for (int i = 0; i < 8; ++i) {
            const int qq = (tid >> 6) + 4 * i;
            const int ql = 32 * t + qq;
            double sv = 0.0;
            if (c >= 0 && ql < nqc) {
                const double *pc = psi + (long long)ql * nall + c;
                const double cx = dirs[qq], cy = dirs[qq + 32], cz = dirs[qq + 64];
                const double fx = axis_flux_bf(cx, th2, pc, sx);
                const double fy = axis_flux_bf(cy, th2, pc, sy);
                const double fz = axis_flux_bf(cz, th2, pc, sz);
                sv = fx * cx + fy * cy + fz * cz;
            }
            sS[qq * CS + cl] = sv;
        }
        __syncthreads();
        const double *B = sB[s];
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const double a = sS[(4 * kk + (lane & 3)) * CS + 8 * warp + (lane >> 2)];
#pragma unroll
            for (int j = 0; j < NT; ++j)
                dmma_g(acc[j][0], acc[j][1], a, B[(kk * NT + j) * 32 + lane]);
        }
        refill_fence();
        __syncthreads();
        if (tid == 0 && t + FLUX_STAGES < nt)
            fbar_load(sB[s], mfP + (size_t)(t0 + t + FLUX_STAGES) * TILE, TILE * 8, &bar[s]);
    }
    if (myc < 0)
        return;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e2 = 0; e2 < 2; ++e2) {
            int m = 8 * j + 2 * (lane & 3) + e2;
            if (m < nm)
                flux[myc * nm + m] = acc[j][e2];
        }
}

// minmod(p, minmod(q, s)) of src/flux_kinetic.cpp:45-61 is symmetric in its three operands:
// sign * min(|p|, |q|, |s|) when all three have one sign, else 0 (the reference's nested form
// gives exactly that: its MIN/MAX select operands without rounding). Here the operand of
// smallest magnitude is chosen by two FP64 compares of absolute values and kept when the sign
// bits of the three high words agree: the same value as the nested form, except possibly for
// the sign of a zero. (On sm_100a this beat the nested selects by 10% in the staged flux, and
// an integer-pipe form and an fmin/fmax form by 8% and 30%.)
__device__ __forceinline__ double minmod3(double p, double q, double s)
{
    double m = fabs(q) < fabs(p) ? q : p;
    m = fabs(s) < fabs(m) ? s : m;
    const bool same =
        ((__double2hiint(p) ^ __double2hiint(q)) | (__double2hiint(q) ^ __double2hiint(s))) >= 0;
    return same ? m : 0.0;
}

// The limited upwind difference along one axis of src/flux_kinetic.cpp:130-189 from the four
// stencil values k1..k4 (offsets -2..1 with h = 1/2 for a positive cosine, -1..2 with h = -1/2
// otherwise): f = ((k3 + h s(k2,k3,k4)) - k2) - h s(k1,k2,k3), s = slopefit
// (src/flux_kinetic.cpp:56-61), evaluated as in axis_flux_bf: s' = 2 s from 2 th (th2) and
// unscaled centred differences, q = h / 2, so f rounds as the reference's expression.
__device__ __forceinline__ double axis_flux_m3(double q, double th2, double k1, double k2,
                                               double k3, double k4)
{
    const double t32 = th2 * (k3 - k2);
    const double s1 = minmod3(th2 * (k4 - k3), k4 - k2, t32);
    const double s2 = minmod3(t32, k3 - k1, th2 * (k2 - k1));
    return fma(-q, s2, fma(q, s1, k3) - k2);
}

// The kinetic flux of kinetic_dmma_kernel with psi staged in shared memory. A CTA owns one
// run of L consecutive interior cells along z (i, j, k0 .. k0 + L - 1; L = min(64, nz), L
// even, nz a multiple of L) and walks its direction chunk in sub-stages of KDS = 8
// directions, two in flight. Per direction a sub-stage holds seven contiguous runs of psi,
// brought in by 1-D bulk copies: the cell run with two halo cells on either side (L + 4
// values) and the three x- and three y-neighbour lines the upwind stencil of that direction
// reads (offsets -2, -1, +1 for a positive cosine, -1, +1, +2 otherwise; L values each), and
// the sub-stage's two projection k-steps and its directions' cosines and weights; warp d
// copies direction d (warp 0 also the projection data), each warp arriving on the stage's
// mbarrier with its bytes. Each thread forms the limited differences of the two (cell,
// direction) pairs whose values it holds in the DMMA A fragments of the sub-stage's two
// k-steps (cell 8 warp + lane / 4, direction 4 k + lane % 4), from shared memory and
// branch-free (the staged slots put the stencil values of either sign of the cosine at fixed
// places; the limiter is the three-operand minmod), then projects them onto the moments with
// DMMAs straight from its registers (k-steps 2v, 2v + 1 of the 32-direction fragment tile, in
// order), so the flux has the same values as kinetic_dmma_kernel's. One barrier per sub-stage,
// before its buffers are refilled.
static_assert(FLUX_STAGES == 2, "kinetic_staged_kernel rings two sub-stages");
constexpr int KDS = 8;                      // directions per sub-stage
constexpr int KRUN = 64;                    // longest cell run per CTA
// doubles staged per direction: the runs back to back (KPER = 4 mod 16, so the four directions
// a warp reads at once, one DMMA k-step, start a quarter of the banks apart; a padding to
// 8 mod 16 measured 2% slower)
constexpr int KPER = (KRUN + 4) + 6 * KRUN;
template <int NT> struct KinStage {
    static constexpr int FRAG = 2 * NT * 32;                    // two projection k-steps
    static constexpr int DOUBLES = KDS * KPER + FRAG + 4 * KDS; // + c_x, c_y, c_z, w of KDS dirs
};
template <int NT>
__global__ void __launch_bounds__(256, 3)
    kinetic_staged_kernel(GridDims g, const double *__restrict__ psi, const double *__restrict__ mfP,
                          const double *__restrict__ xiAll, const double *__restrict__ etaAll,
                          int q0, int nqc, int L, double theta, int accumulate,
                          double *__restrict__ flux, int *errorFlag, const int *wrapFlag)
{
    constexpr int TILE = 8 * NT * 32 + 128; // one 32-direction tile of mfP
    constexpr int SD = KinStage<NT>::DOUBLES, FRAG = KinStage<NT>::FRAG;
    static_assert((SD * 8) % 16 == 0 && (KPER * 8) % 16 == 0, "stage alignment");
    static_assert(KDS * 32 == 256, "one warp per direction of a sub-stage");
    extern __shared__ __align__(128) double kinSmem[];
    __shared__ uint64_t pbar[2];
    __shared__ long long sRun[9];
    const double th2 = 2.0 * theta;
    const int nm = g.nm;
    const long long nall = g.nall();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // block order: z run index slowest; the (i, j) lines in tiles of 16 x 16 (row-major,
    // partial tiles at the edges), so that CTAs running at the same time stage each other's
    // neighbour lines from L2
    int i, j, kb;
    {
        constexpr int TI = 16, TJ = 16;
        const long long lines = (long long)g.nx * g.ny;
        kb = (int)(blockIdx.x / lines);
        const long long r = blockIdx.x % lines, rowBlock = (long long)TI * g.ny;
        const int ti = (int)(r / rowBlock);
        const long long r2 = r % rowBlock;
        const int hi = min(TI, g.nx - ti * TI);
        const int tj = (int)(r2 / ((long long)hi * TJ));
        const int r3 = (int)(r2 % ((long long)hi * TJ));
        const int wj = min(TJ, g.ny - tj * TJ);
        i = 2 + ti * TI + r3 / wj;
        j = 2 + tj * TJ + r3 % wj;
    }
    const int k0 = 2 + kb * L;
    const int t0 = q0 >> 5, nu = (nqc + KDS - 1) / KDS;
    // start cell of run r: 0 the cell run with its z halo, 1-4 x offsets -2, -1, +1, +2,
    // 5-8 y offsets -2, -1, +1, +2
    // wrap (the closure copied the face ghosts from their periodic images and their psi was
    // not copied): stencil values of face ghosts are read at the images instead -- the x and
    // y neighbour lines of the periodic grid, and the z halo pairs of runs at either end
    const bool wrap = wrapFlag && *wrapFlag == 0;
    const bool lowB = wrap && k0 == 2, highB = wrap && k0 + L == g.nz + 2;
    if (tid < 9) {
        const int r = tid, o = (r - 1) & 3, d = o < 2 ? o - 2 : o - 1;
        auto per = [&](int a, int n) { return !wrap ? a : a < 2 ? a + n : a >= n + 2 ? a - n : a; };
        sRun[r] = r == 0    ? g.cell(i, j, k0 - 2)
                  : r <= 4 ? g.cell(per(i + d, g.nx), j, k0)
                           : g.cell(i, per(j + d, g.ny), k0);
    }
    const uint32_t perDir = (uint32_t)((L + 4) + 6 * L) * 8;
    // a direction's stage: the cell run, then x slots 0-2, then y slots 0-2 (offsets -2, -1,
    // +1 for a positive cosine, -1, +1, +2 otherwise)
    auto issue = [&](int u) {
        const int nd = min(KDS, nqc - KDS * u), d = warp;
        double *st = kinSmem + (u & 1) * SD;
        uint64_t *b = &pbar[u & 1];
        uint32_t bytes = d < nd ? perDir : 0u;
        if (d == 0)
            bytes += (FRAG + 4 * KDS) * 8;
        if (lane == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(
                             smem_addr(b)),
                         "r"(bytes)
                         : "memory");
        __syncwarp();
        const double *src = nullptr;
        double *dst = nullptr;
        uint32_t nb = 0;
        if (d < nd && lane < 7) {
            const int ql = KDS * u + d;
            int r = 0, off = 0;
            if (lane >= 1 && lane <= 3) {
                const int sl = lane - 1;
                r = (xiAll[q0 + ql] > 0 ? 1 : 2) + sl; // runs 1-4: offsets -2, -1, +1, +2
                off = (L + 4) + sl * L;
            } else if (lane >= 4) {
                const int sl = lane - 4;
                r = (etaAll[q0 + ql] > 0 ? 5 : 6) + sl;
                off = (L + 4) + (3 + sl) * L;
            }
            src = psi + (long long)ql * nall + sRun[r];
            dst = st + d * KPER + off;
            nb = (uint32_t)(r == 0 ? L + 4 : L) * 8;
            if (r == 0 && (lowB || highB)) {
                // the run without the halo pairs that lanes 12 and 13 bring from the images
                src += lowB ? 2 : 0;
                dst += lowB ? 2 : 0;
                nb -= (uint32_t)(2 * lowB + 2 * highB) * 8;
            }
        } else if (d < nd && ((lane == 12 && lowB) || (lane == 13 && highB))) {
            // z halo pair of a run at the low end (ghosts k = 0, 1 = images nz, nz + 1) or the
            // high end (k = nz + 2, nz + 3 = images 2, 3); 16-byte aligned: nz and L are even
            const int ql = KDS * u + d;
            src = psi + (long long)ql * nall + g.cell(i, j, lane == 12 ? g.nz : 2);
            dst = st + d * KPER + (lane == 12 ? 0 : L + 2);
            nb = 16;
        } else if (d == 0 && lane >= 7 && lane <= 11) {
            const int ql = KDS * u;
            const double *tile = mfP + (size_t)(t0 + (ql >> 5)) * TILE;
            const int v = (ql & 31) / KDS;
            if (lane == 7) {
                src = tile + v * FRAG;
                dst = st + KDS * KPER;
                nb = FRAG * 8;
            } else {
                src = tile + 8 * NT * 32 + 32 * (lane - 8) + KDS * v; // c_x, c_y, c_z, w
                dst = st + KDS * KPER + FRAG + KDS * (lane - 8);
                nb = KDS * 8;
            }
        }
        if (nb)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                             smem_addr(dst)),
                         "l"(src), "r"(nb), "r"(smem_addr(b))
                         : "memory");
    };
    if (tid == 0) {
        for (int s = 0; s < 2; ++s)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(&pbar[s])),
                         "r"(KDS));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    for (int u = 0; u < 2 && u < nu; ++u)
        issue(u);
    const int cw = 8 * warp + (lane >> 2); // the warp's projection cells
    const long long myc = cw < L ? g.cell(i, j, k0 + cw) : -1;
    double acc[NT][2];
#pragma unroll
    for (int jj = 0; jj < NT; ++jj)
#pragma unroll
        for (int e2 = 0; e2 < 2; ++e2) {
            int m = 8 * jj + 2 * (lane & 3) + e2;
            acc[jj][e2] = (accumulate && myc >= 0 && m < nm) ? flux[myc * nm + m] : 0.0;
        }
    for (int u = 0; u < nu; ++u) {
        const double *st = kinSmem + (u & 1) * SD;
        // a timed-out wait is agreed on at the barrier after the stencil (the data of that
        // sub-stage are then not used)
        const bool ok = fbar_wait(&pbar[u & 1], (u >> 1) & 1);
        const double *dirs = st + KDS * KPER + FRAG; // c_x[KDS], c_y[KDS], c_z[KDS], w[KDS]
        double afr[2]; // the thread's own A fragments of the sub-stage's two k-steps
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            // cell 8 warp + lane / 4, direction 4 r + lane % 4: the element of the DMMA A
            // fragment (k-step r) the thread holds
            const int cl = cw, d = 4 * r + (lane & 3);
            const int ql = KDS * u + d;
            double sv = 0.0;
            if (cl < L && ql < nqc) {
                const double *P = st + d * KPER;
                const double *xr = P + (L + 4), *yr = xr + 3 * L;
                const double c0 = P[cl + 2];
                // the direction's weights c = cosine x w / spacing per axis
                const double ox = dirs[d], oy = dirs[KDS + d], oz = dirs[2 * KDS + d];
                // branch-free: the staged x and y slots hold offsets (-2, -1, +1) for a positive
                // cosine and (-1, +1, +2) otherwise, so k1 and k4 always come from slots 0 and 2
                // and the cell's own value is k3 or k2; the z run holds offsets -2 .. +2
                const bool px = ox > 0, py = oy > 0, pz = oz > 0;
                const double ax = xr[L + cl], ay = yr[L + cl];
                const double fx = axis_flux_m3(px ? 0.25 : -0.25, th2, xr[cl], px ? ax : c0,
                                               px ? c0 : ax, xr[2 * L + cl]);
                const double fy = axis_flux_m3(py ? 0.25 : -0.25, th2, yr[cl], py ? ay : c0,
                                               py ? c0 : ay, yr[2 * L + cl]);
                const double *zb = P + cl + (pz ? 0 : 1);
                const double fz = axis_flux_m3(pz ? 0.25 : -0.25, th2, zb[0], zb[1], zb[2], zb[3]);
                sv = fx * ox + fy * oy + fz * oz;
            }
            afr[r] = sv;
        }
        // projection straight from the registers; one barrier per sub-stage (before its stage
        // is refilled), where a timed-out wait is agreed on
        const double *B = st + KDS * KPER;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int jj = 0; jj < NT; ++jj)
                dmma_g(acc[jj][0], acc[jj][1], afr[h], B[(h * NT + jj) * 32 + lane]);
        refill_fence();
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicExch(errorFlag, 1);
                fbar_drain(pbar, u, nu);
            }
            return;
        }
        if (u + 2 < nu)
            issue(u + 2);
    }
    if (myc < 0)
        return;
#pragma unroll
    for (int jj = 0; jj < NT; ++jj)
#pragma unroll
        for (int e2 = 0; e2 < 2; ++e2) {
            int m = 8 * jj + 2 * (lane & 3) + e2;
            if (m < nm)
                flux[myc * nm + m] = acc[jj][e2];
        }
}

// ---------------------------------------------------------------- P_N moment flux

// flux(c) = sum over the axes of (A+ tp + A- tm) / h, tp and tm the upwind differences of the
// moments for either sign of the cosine (src/flux_moment.cpp:57-101), for interior cells.
// The six nm x nm operators sit in shared memory as DMMA B fragments for the CTA's lifetime; a
// warp takes 8 MT interior cells at a time, its lanes form the A fragments of tp and tm
// (cell lane / 4, moment 4 k + lane % 4) from five neighbours, and per axis a sum over k-steps
// of both halves is divided by the spacing and added to the flux. Bound by the FP64 tensor
// pipe: 12 nm^2 FMA per cell padded to tiles of 8 x 4. P_5 on 64^3: 344 us per call, 2387 us
// with scalar unfused sums, one operator row per thread.
template <int NT, int MT>
__global__ void __launch_bounds__(256, NT <= 5 ? 2 : 1)
    moment_flux_kernel(GridDims g, const double *__restrict__ u, const double *__restrict__ ops,
                       double dx, double dy, double dz, double *__restrict__ flux)
{
    constexpr int KS = 2 * NT, FRAGS = KS * NT * 32;
    extern __shared__ __align__(128) double sOps[]; // [operator][k-step][tile][lane]
    const int nm = g.nm, ks = (nm + 3) / 4;
    for (int e = threadIdx.x; e < 6 * FRAGS; e += 256) {
        const int l = e & 31, t = (e >> 5) % NT, k = (e / (32 * NT)) % KS, op = e / FRAGS;
        const int row = 8 * t + l / 4, col = 4 * k + l % 4;
        sOps[e] = row < nm && col < nm ? ops[((size_t)op * nm + row) * nm + col] : 0.0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long nint = g.ninterior(), step = (long long)gridDim.x * 8 * 8 * MT;
    const long long st[3] = {(long long)g.nyg() * g.nzg(), g.nzg(), 1};
    for (long long n0 = ((long long)blockIdx.x * 8 + warp) * 8 * MT; n0 < nint; n0 += step) {
        long long c[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const long long n = n0 + 8 * m + (lane >> 2);
            c[m] = n < nint ? interior_cell(g, n) : -1;
        }
        double total[MT][NT][2];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            double acc[MT][NT][2];
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int t = 0; t < NT; ++t)
                    acc[m][t][0] = acc[m][t][1] = 0.0;
            const double *bp = sOps + (2 * ax) * FRAGS + lane, *bm = bp + FRAGS;
            const long long s = st[ax] * nm;
#pragma unroll 2
            for (int k = 0; k < ks; ++k) {
                const int col = 4 * k + (lane & 3);
                double tp[MT], tm[MT];
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    tp[m] = tm[m] = 0.0;
                    if (c[m] >= 0 && col < nm) {
                        const double *v = u + c[m] * nm + col;
                        const double v0 = v[0], p1 = v[s], p2 = v[2 * s], m1 = v[-s], m2 = v[-2 * s];
                        tp[m] = 0.25 * p1 + 0.75 * v0 - 1.25 * m1 + 0.25 * m2;
                        tm[m] = -0.25 * p2 + 1.25 * p1 - 0.75 * v0 - 0.25 * m1;
                    }
                }
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const double b = bp[(k * NT + t) * 32];
#pragma unroll
                    for (int m = 0; m < MT; ++m)
                        dmma_g(acc[m][t][0], acc[m][t][1], tp[m], b);
                }
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const double b = bm[(k * NT + t) * 32];
#pragma unroll
                    for (int m = 0; m < MT; ++m)
                        dmma_g(acc[m][t][0], acc[m][t][1], tm[m], b);
                }
            }
            const double h = ax == 0 ? dx : ax == 1 ? dy : dz;
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int t = 0; t < NT; ++t)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const double f = acc[m][t][e] / h;
                        total[m][t][e] = ax == 0 ? f : total[m][t][e] + f;
                    }
        }
#pragma unroll
        for (int m = 0; m < MT; ++m)
            if (c[m] >= 0)
#pragma unroll
                for (int t = 0; t < NT; ++t)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int row = 8 * t + 2 * (lane & 3) + e;
                        if (row < nm)
                            flux[c[m] * nm + row] = total[m][t][e];
                    }
    }
}

// ---------------------------------------------------------------- launchers

static int grid_for(long long n, int threads, int numSMs)
{
    long long b = (n + threads - 1) / threads;
    long long cap = (long long)numSMs * 16;
    if (b > cap)
        b = cap;
    return b < 1 ? 1 : (int)b;
}

cudaError_t launch_ghost_fill(const GridDims &g, double *u, int numSMs, cudaStream_t st,
                              bool skipX)
{
    const long long f0 = skipX ? 4LL * g.ny * g.nz : 0;
    ghost_fill_kernel<<<grid_for((ghost_faces(g) - f0) * 32, 256, numSMs), 256, 0, st>>>(g, u, f0);
    return cudaGetLastError();
}

cudaError_t launch_line_log(const GridDims &g, const ClosureParams &P, const int *iters,
                            const int *iterGamma, const int *regIdx, const double *gamma,
                            const double *normG, double *out, cudaStream_t st)
{
    line_log_kernel<<<(g.nx + 127) / 128, 128, 0, st>>>(g, P, iters, iterGamma, regIdx, gamma,
                                                         normG, out);
    return cudaGetLastError();
}

cudaError_t launch_ghost_mirror_copy(const GridDims &g, double *u, double *alpha, int *iters,
                                     int *iterGamma, int *regIdx, int *status, double *gamma,
                                     double *normG, unsigned long long *stats, int numSMs,
                                     cudaStream_t st)
{
    ghost_mirror_copy_kernel<<<grid_for(ghost_faces(g) * 32, 256, numSMs), 256, 0, st>>>(
        g, MirrorCopy{u, alpha, iters, iterGamma, regIdx, status, gamma, normG, stats});
    return cudaGetLastError();
}

cudaError_t launch_ghost_mirror_check(const GridDims &g, const double *a, int *flag, int numSMs,
                                      cudaStream_t st)
{
    ghost_mirror_check_kernel<<<grid_for(ghost_faces(g) * 32, 256, numSMs), 256, 0, st>>>(g, a, flag);
    return cudaGetLastError();
}

cudaError_t launch_psi_groups(const GridDims &g, unsigned char *mark, long long *list,
                              unsigned int *count, int numSMs, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(count, 0, sizeof(unsigned int), st);
    if (e != cudaSuccess)
        return e;
    const long long groups = (g.nall() + 7) / 8;
    psi_groups_kernel<<<grid_for(groups, 256, numSMs), 256, 0, st>>>(
        reinterpret_cast<unsigned long long *>(mark), groups, list, count);
    return cudaGetLastError();
}

cudaError_t launch_psi_refresh(const GridDims &g, int nq, const double *M, const double *alpha,
                               const long long *list, const unsigned int *count, double *psi,
                               int numSMs, cudaStream_t st)
{
    psi_refresh_kernel<<<2 * numSMs, 256, 0, st>>>(g, nq, M, alpha, list, count, psi);
    return cudaGetLastError();
}

// comp: doubles per cell and row (1 or 4)
cudaError_t launch_psi_face_copy(const GridDims &g, int rows, int comp, double *psi, cudaStream_t st)
{
    constexpr int RPER = 64;
    const dim3 grid((unsigned)((ghost_faces(g) + 255) / 256), (unsigned)ceil_div(rows, RPER));
    if (comp == 4)
        psi_face_copy_kernel<<<grid, 256, 0, st>>>(g, rows, RPER, reinterpret_cast<Psi4 *>(psi));
    else
        psi_face_copy_kernel<<<grid, 256, 0, st>>>(g, rows, RPER, psi);
    return cudaGetLastError();
}

static dim3 interior_grid(const GridDims &g)
{
    const long long lines = (long long)g.nx * g.ny;
    return dim3((unsigned)(((long long)g.nz * g.nm + 255) / 256), (unsigned)(lines < 65535 ? lines : 65535));
}

// mode as euler_kernel's (uOld may be null in mode 0)
cudaError_t launch_euler(const GridDims &g, double *u, const double *flux, const double *sigT,
                         const double *sigS, double dt, double *uOld, int mode, cudaStream_t st)
{
    const dim3 grid = interior_grid(g);
    if (mode == 0)
        euler_kernel<0><<<grid, 256, 0, st>>>(g, u, flux, sigT, sigS, dt, uOld);
    else if (mode == 1)
        euler_kernel<1><<<grid, 256, 0, st>>>(g, u, flux, sigT, sigS, dt, uOld);
    else
        euler_kernel<2><<<grid, 256, 0, st>>>(g, u, flux, sigT, sigS, dt, uOld);
    return cudaGetLastError();
}

cudaError_t launch_rk_save(const GridDims &g, const double *u, double *uOld, cudaStream_t st)
{
    rk_save_kernel<<<interior_grid(g), 256, 0, st>>>(g, u, uOld);
    return cudaGetLastError();
}

// Robustness re-projection after the closure (the note in the reference's readme.txt:
// "one should calculate a new u^n so that u^n = <m exp(m^T alpha^n)> exactly ... and scale
// u^n and alpha^n so that u_0^n does not change"): per cell u' = sum_q w_q m_q e^{alpha.m_q};
// with s = u_0 / u'_0, u <- (u_0, s u'_1, ..., s u'_{nm-1}) and alpha_0 <- alpha_0 + log(s)/m_0
// (m_0 = 1/(2 sqrt(pi)); e^{alpha.m} s = e^{alpha'.m}). A CTA owns 64 cells: per direction
// tile the exponents (DMMA, multipliers as A fragments), c = w e^{z} into shared memory, then
// the moments (DMMA with the projection fragments) -- the ansatz and projection layouts of
// the kinetic flux.
template <int NT>
__global__ void __launch_bounds__(256)
    reproject_kernel(GridDims g, double *__restrict__ u, double *__restrict__ alpha,
                     const double *__restrict__ mfA, const double *__restrict__ mfP, int nq,
                     int *errorFlag)
{
    constexpr int KS = 2 * NT;
    constexpr int TA = 4 * KS * 32, TP = 8 * NT * 32 + 128;
    constexpr int CS = 68;
    extern __shared__ __align__(128) double rpSmem[]; // sA[2][TA], sP[2][TP], sC[32][CS]
    double(*sA)[TA] = reinterpret_cast<double(*)[TA]>(rpSmem);
    double(*sP)[TP] = reinterpret_cast<double(*)[TP]>(rpSmem + FLUX_STAGES * TA);
    double *sC = rpSmem + FLUX_STAGES * (TA + TP);
    __shared__ uint64_t bar[FLUX_STAGES];
    __shared__ int sAbort;
    const int nm = g.nm;
    const long long nall = g.nall();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long c = (long long)blockIdx.x * 64 + 8 * warp + (lane >> 2);
    const int nt = (nq + 31) >> 5;
    if (tid == 0) {
        sAbort = 0;
        for (int st = 0; st < FLUX_STAGES; ++st)
            fbar_init(&bar[st]);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        for (int st = 0; st < FLUX_STAGES && st < nt; ++st)
            fbar_load2(sA[st], mfA + (size_t)st * TA, TA * 8, sP[st], mfP + (size_t)st * TP,
                       TP * 8, &bar[st]);
    }
    double a[KS];
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
        int k = 4 * kk + (lane & 3);
        a[kk] = (c < nall && k < nm) ? alpha[c * nm + k] : 0.0;
    }
    double acc[NT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j)
        acc[j][0] = acc[j][1] = 0.0;
    __syncthreads();
    for (int t = 0; t < nt; ++t) {
        const int st = t % FLUX_STAGES;
        if (!fbar_wait(&bar[st], (t / FLUX_STAGES) & 1))
            sAbort = 1;
        if (__syncthreads_or(sAbort)) {
            if (tid == 0) {
                atomicExch(errorFlag, 1);
                fbar_drain(bar, t, nt);
            }
            return;
        }
        const double *w = sP[st] + 8 * NT * 32 + 96;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            double z0 = 0.0, z1 = 0.0;
#pragma unroll
            for (int kk = 0; kk < KS; ++kk)
                dmma_g(z0, z1, a[kk], sA[st][(j * KS + kk) * 32 + lane]);
            const int qq = 8 * j + 2 * (lane & 3);
            sC[qq * CS + 8 * warp + (lane >> 2)] = w[qq] * exp(z0);
            sC[(qq + 1) * CS + 8 * warp + (lane >> 2)] = w[qq + 1] * exp(z1);
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const double av = sC[(4 * kk + (lane & 3)) * CS + 8 * warp + (lane >> 2)];
#pragma unroll
            for (int j = 0; j < NT; ++j)
                dmma_g(acc[j][0], acc[j][1], av, sP[st][(kk * NT + j) * 32 + lane]);
        }
        refill_fence();
        __syncthreads();
        if (tid == 0 && t + FLUX_STAGES < nt)
            fbar_load2(sA[st], mfA + (size_t)(t + FLUX_STAGES) * TA, TA * 8, sP[st],
                       mfP + (size_t)(t + FLUX_STAGES) * TP, TP * 8, &bar[st]);
    }
    // lane 4r holds moment 0 of cell r of the warp's tile
    const double un0 = __shfl_sync(0xffffffffu, acc[0][0], lane & ~3);
    if (c >= nall)
        return;
    const double u0 = u[c * nm];
    const double sc = u0 / un0;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e2 = 0; e2 < 2; ++e2) {
            int m = 8 * j + 2 * (lane & 3) + e2;
            if (m > 0 && m < nm)
                u[c * nm + m] = sc * acc[j][e2];
        }
    if ((lane & 3) == 0)
        alpha[c * nm] += 2.0 * sqrt(M_PI) * log(sc);
}

template <int NT>
static cudaError_t reproject_t(const GridDims &g, double *u, double *alpha, const double *mfA,
                               const double *mfP, int nq, int *errorFlag, cudaStream_t st)
{
    constexpr int KS = 2 * NT;
    const size_t smem =
        (size_t)(FLUX_STAGES * (4 * KS * 32 + 8 * NT * 32 + 128) + 32 * 68) * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(reproject_kernel<NT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess)
        return e;
    reproject_kernel<NT><<<(unsigned)((g.nall() + 63) / 64), 256, smem, st>>>(g, u, alpha, mfA,
                                                                             mfP, nq, errorFlag);
    return cudaGetLastError();
}

cudaError_t launch_reproject(const GridDims &g, double *u, double *alpha, const double *mfA,
                             const double *mfP, int nq, int *errorFlag, cudaStream_t st)
{
    switch ((g.nm + 7) / 8) {
    case 1: return reproject_t<1>(g, u, alpha, mfA, mfP, nq, errorFlag, st);
    case 2: return reproject_t<2>(g, u, alpha, mfA, mfP, nq, errorFlag, st);
    case 3: return reproject_t<3>(g, u, alpha, mfA, mfP, nq, errorFlag, st);
    case 4: return reproject_t<4>(g, u, alpha, mfA, mfP, nq, errorFlag, st);
    case 5: return reproject_t<5>(g, u, alpha, mfA, mfP, nq, errorFlag, st);
    case 6: return reproject_t<6>(g, u, alpha, mfA, mfP, nq, errorFlag, st);
    case 7: return reproject_t<7>(g, u, alpha, mfA, mfP, nq, errorFlag, st);
    case 8: return reproject_t<8>(g, u, alpha, mfA, mfP, nq, errorFlag, st);
    default: return cudaErrorInvalidValue;
    }
}

// Fragment-order copies of the basis for the flux kernels (layouts above); nt = ceil(nq/32)
// tiles each.
size_t flux_frag_doubles(int nm, int nq, int which)
{
    const int NT = (nm + 7) / 8, nt = (nq + 31) / 32;
    return (size_t)nt * (which == 0 ? 4 * 2 * NT * 32 : 8 * NT * 32 + 128);
}

void flux_frags(int nm, int nq, const double *M, const double *w, const double *xi,
                const double *eta, const double *mu, double rdx, double rdy, double rdz,
                double *mfA, double *mfP)
{
    const int NT = (nm + 7) / 8, KS = 2 * NT, nt = (nq + 31) / 32;
    auto m = [&](int q, int k) { return (q < nq && k < nm) ? M[(size_t)q * nm + k] : 0.0; };
    for (int t = 0; t < nt; ++t) {
        double *A = mfA + (size_t)t * 4 * KS * 32;
        for (int j = 0; j < 4; ++j)
            for (int kk = 0; kk < KS; ++kk)
                for (int l = 0; l < 32; ++l)
                    A[(j * KS + kk) * 32 + l] = m(32 * t + 8 * j + l / 4, 4 * kk + l % 4);
        double *P = mfP + (size_t)t * (8 * NT * 32 + 128);
        for (int kk = 0; kk < 8; ++kk)
            for (int j = 0; j < NT; ++j)
                for (int l = 0; l < 32; ++l)
                    P[(kk * NT + j) * 32 + l] = m(32 * t + 4 * kk + l % 4, 8 * j + l / 4);
        double *D = P + 8 * NT * 32;
        for (int qq = 0; qq < 32; ++qq) {
            int q = 32 * t + qq;
            D[qq] = q < nq ? (xi[q] * w[q]) * rdx : 0.0;
            D[32 + qq] = q < nq ? (eta[q] * w[q]) * rdy : 0.0;
            D[64 + qq] = q < nq ? (mu[q] * w[q]) * rdz : 0.0;
            D[96 + qq] = q < nq ? w[q] : 0.0;
        }
    }
}

template <int NT>
static cudaError_t kinetic_t(const GridDims &g, const double *alpha, const double *mfA,
                             const double *mfP, const double *xi, const double *eta, int nq,
                             int qChunk, int runLen, double theta, int isPn, double *psi,
                             bool psiReady, double *flux, int *errorFlag, const int *wrapFlag,
                             cudaStream_t st)
{
    if (psiReady)
        qChunk = nq; // psi of every direction is in place: the stencil alone, in one pass
    for (int q0 = 0; q0 < nq; q0 += qChunk) {
        int nqc = nq - q0 < qChunk ? nq - q0 : qChunk;
        if (!psiReady)
            ansatz_dmma_kernel<NT><<<(unsigned)((g.nall() + 63) / 64), 256, 0, st>>>(
                g, alpha, mfA, q0, nqc, isPn, psi, errorFlag);
        // staged psi when the z lines split into even runs of at most 64 cells (runLen: the
        // run length chosen by the autotuner, 0 for min(64, nz))
        const int L = runLen > 0 ? runLen : (g.nz < KRUN ? g.nz : KRUN);
        if (L % 2 == 0 && L <= KRUN && g.nz % L == 0) {
            const size_t smem = (size_t)(2 * KinStage<NT>::DOUBLES) * 8;
            auto kern = kinetic_staged_kernel<NT>;
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)smem);
            if (e != cudaSuccess)
                return e;
            kern<<<(unsigned)((long long)g.nx * g.ny * (g.nz / L)), 256, smem, st>>>(
                    g, psi, mfP, xi, eta, q0, nqc, L, theta, q0 > 0 ? 1 : 0, flux, errorFlag,
                    wrapFlag);
            e = cudaGetLastError();
            if (e != cudaSuccess)
                return e;
            continue;
        }
        if (wrapFlag) // the global-load form reads the face ghosts themselves
            return cudaErrorInvalidValue;
        const size_t kinSmem = (size_t)(FLUX_STAGES * (8 * NT * 32 + 128) + 32 * 68) * 8;
        // opt in above the 48 KB default for the dynamic part plus the ~1.3 KB static part
        if (kinSmem > 46 * 1024) {
            cudaError_t e = cudaFuncSetAttribute(kinetic_dmma_kernel<NT>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)kinSmem);
            if (e != cudaSuccess)
                return e;
        }
        kinetic_dmma_kernel<NT><<<(unsigned)((g.ninterior() + 63) / 64), 256, kinSmem, st>>>(
            g, psi, mfP, q0, nqc, theta, q0 > 0 ? 1 : 0, flux, errorFlag);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

// qChunk: a multiple of 32 unless it covers all of nq.
// psiReady: psi[q nall + c] already holds the ansatz of every direction (handed off by the
// closure), so only the stencil and projection run.
// wrapFlag (staged stencil only, else null): a device flag; when it reads 0 the face ghosts'
// psi is not in place and their stencil values are read at their periodic images.
bool kinetic_staged_used(const GridDims &g, int runLen)
{
    const int L = runLen > 0 ? runLen : (g.nz < KRUN ? g.nz : KRUN);
    return L % 2 == 0 && L <= KRUN && g.nz % L == 0;
}

cudaError_t launch_kinetic_flux(const GridDims &g, const double *alpha, const double *mfA,
                                const double *mfP, const double *xi, const double *eta, int nq,
                                int qChunk, int runLen, double theta, int isPn, double *psi,
                                bool psiReady, double *flux, int *errorFlag, const int *wrapFlag,
                                cudaStream_t st)
{
    if (qChunk < nq && (qChunk & 31))
        return cudaErrorInvalidValue;
#define C3D_NT_CASE(NT)                                                                            \
    case NT:                                                                                       \
        return kinetic_t<NT>(g, alpha, mfA, mfP, xi, eta, nq, qChunk, runLen, theta, isPn, psi,  \
                             psiReady, flux, errorFlag, wrapFlag, st);
    switch ((g.nm + 7) / 8) {
        C3D_NT_CASE(1)
        C3D_NT_CASE(2)
        C3D_NT_CASE(3)
        C3D_NT_CASE(4)
        C3D_NT_CASE(5)
        C3D_NT_CASE(6)
        C3D_NT_CASE(7)
        C3D_NT_CASE(8)
    default:
        return cudaErrorInvalidValue;
    }
#undef C3D_NT_CASE
}

template <int NT, int MT>
static cudaError_t moment_flux_t(const GridDims &g, const double *u, const double *ops, double dx,
                                 double dy, double dz, double *flux, int numSMs, cudaStream_t st)
{
    const int smem = 6 * 2 * NT * NT * 32 * 8;
    cudaError_t e = cudaFuncSetAttribute(moment_flux_kernel<NT, MT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess)
        return e;
    const long long blocks = (g.ninterior() + 64 * MT - 1) / (64 * MT);
    const long long cap = (long long)numSMs * (NT <= 5 ? 2 : 1);
    moment_flux_kernel<NT, MT><<<(unsigned)(blocks < cap ? blocks : cap), 256, smem, st>>>(
        g, u, ops, dx, dy, dz, flux);
    return cudaGetLastError();
}

// Two tiles of 8 cells per warp share each operator fragment's load; small grids take one so
// that more SMs get cells.
cudaError_t launch_moment_flux(const GridDims &g, const double *u, const double *ops, double dx,
                               double dy, double dz, double *flux, int numSMs, cudaStream_t st)
{
    const bool wide = g.ninterior() >= 256LL * numSMs;
#define C3D_NT_CASE(NT)                                                                            \
    case NT:                                                                                       \
        return wide ? moment_flux_t<NT, 2>(g, u, ops, dx, dy, dz, flux, numSMs, st)                \
                    : moment_flux_t<NT, 1>(g, u, ops, dx, dy, dz, flux, numSMs, st);
    switch ((g.nm + 7) / 8) {
        C3D_NT_CASE(1)
        C3D_NT_CASE(2)
        C3D_NT_CASE(3)
        C3D_NT_CASE(4)
        C3D_NT_CASE(5)
        C3D_NT_CASE(6)
        C3D_NT_CASE(7)
        C3D_NT_CASE(8)
    default:
        return cudaErrorInvalidValue;
    }
#undef C3D_NT_CASE
}

} // namespace c3d
