// Work-list form of the FP64 M_N closure: the reference's batched structure
// (Optimization::opt with its stacks, src/opt/optBatch.cpp:350-472) on the device.
//
// A closure runs in rounds over a device work list of cells that need a quadrature
// pass (a Hessian evaluation or a line-search trial):
//   init kernel    per cell: scale u and alpha (preProcess, src/opt/optBatch.cpp:312-331),
//                  start the first Newton iteration, append the cell to the work list;
//   pass kernel    per listed cell: exponents alpha.m_q and either the extended moments
//                  of the Gaunt form (DMMA, 8 cells per warp over the staged octant tables, or 16
//                  per CTA over staged M2^T chunks) or the direct Hessian tiles, or the trial's f;
//   Newton kernel  8, 16 or 32 lanes per listed cell: assemble H, Cholesky, condition estimate,
//                  direction, stop tests, Armijo (solveTheRest, src/opt/optBatch.cpp:143-283)
//                  with the state machine shared with the persistent kernels; cells that
//                  need another pass are appended to the next round's list.
// Separating the passes (tensor-pipe work, small shared memory) from the per-cell logic
// (latency-bound, serial chains per cell) lets each run at its own occupancy; a cell that
// needs many iterations only ever occupies the short lists of later rounds.
#include "closure_core.cuh"

#include <mutex>
#include <vector>
#include "rounds_launch.h"
#include "sym.cuh"
#include "umma.cuh"

#include <cuda_bf16.h>
#include <cstdio>
#include <type_traits>

namespace c3d {

// Per-cell Newton state between rounds: the slot without the factor, the reciprocal
// pivots and the gradient (recomputed from H on every Hessian visit, unused by trials).
template <int NT> struct CellState {
    static constexpr int NMP = Cfg<NT>::NMP;
    double u[NMP], alpha[NMP], alpha0[NMP], uOrig[NMP], d[NMP], alphaOld[NMP];
    SlotScalars s;
};

namespace {

template <int W>
__device__ __forceinline__ void copy_scalars(SlotScalars &dst, const SlotScalars &src, int lane)
{
    static_assert(sizeof(SlotScalars) % 8 == 0, "whole words");
#pragma unroll
    for (int i = lane; i < (int)sizeof(SlotScalars) / 8; i += W)
        reinterpret_cast<unsigned long long *>(&dst)[i] =
            reinterpret_cast<const unsigned long long *>(&src)[i];
}

// Whether a slot leaves alpha0 and uOrig in the cell's state.
template <class S> constexpr bool keeps_in_state = std::is_pointer<decltype(S::alpha0)>::value;

// lineSearch = false skips d and alphaOld, which a probe visit recomputes before use.
template <int NT, class S>
__device__ void state_to_slot(CellState<NT> &st, S &sl, int lane, bool lineSearch = true)
{
    constexpr int NMP = Cfg<NT>::NMP;
    if constexpr (keeps_in_state<S>) {
        if (lane == 0) {
            sl.alpha0 = st.alpha0;
            sl.uOrig = st.uOrig;
        }
    }
    for (int i = lane; i < NMP; i += S::W) {
        sl.u[i] = st.u[i];
        sl.alpha[i] = st.alpha[i];
        if constexpr (!keeps_in_state<S>) {
            sl.alpha0[i] = st.alpha0[i];
            sl.uOrig[i] = st.uOrig[i];
        }
        if (lineSearch) {
            sl.d[i] = st.d[i];
            sl.alphaOld[i] = st.alphaOld[i];
        }
    }
    copy_scalars<S::W>(sl.s, st.s, lane);
    cell_sync<S>();
}

template <int NT, class S>
__device__ void slot_to_state(const S &sl, CellState<NT> &st, int lane)
{
    constexpr int NMP = Cfg<NT>::NMP;
    cell_sync<S>();
    for (int i = lane; i < NMP; i += S::W) {
        st.u[i] = sl.u[i];
        st.alpha[i] = sl.alpha[i];
        if constexpr (!keeps_in_state<S>) {
            st.alpha0[i] = sl.alpha0[i];
            st.uOrig[i] = sl.uOrig[i];
        }
        st.d[i] = sl.d[i];
        st.alphaOld[i] = sl.alphaOld[i];
    }
    copy_scalars<S::W>(st.s, sl.s, lane);
}

// The work lists of one round: 0 trials and FP64 Hessian passes, 1 BF16 Hessian passes,
// 2 3xTF32 Hessian passes (lists 1 and 2: mixed-precision closure only), 3 first visits
// through the probe pass (convergence certificate) or, with an octant-symmetric quadrature (whose
// probe visits never enter a list), trials and FP64 Hessian passes in the reference's order.
constexpr int NLISTS = 4;

// 2-norm of a cell's multipliers beyond alpha_0 from which the passes of a symmetric quadrature
// keep the reference's order over the full basis. Such cells sit at the realizability boundary
// (exponents to -1600, condition numbers to 1e9, steps of 1e-3 along directions of 1e6, a few
// directions carrying the moments), where the rounding of the basis and of the sums decides at
// which multipliers inside the stopping tolerance the iteration ends: over three steps of M_6
// pulses on 20^3, 24^3, 26^3 and 28^3 the farthest cell ended 9.4e-8, 1.0e-8, 8.9e-9 and 7.2e-8
// from the oracle's with the symmetric passes, 1.6e-9, 1.1e-9, 4.3e-9 and 1.7e-8 in its order; on
// 32^3, where no norm passes 25, 1.0e-10 and 3.7e-11. Standalone vectors with components of unit
// variance reach 8 (N = 7).
constexpr double REF_NORM = 32.0;
struct Lists {
    int *list[NLISTS];
    unsigned int *count[NLISTS];
};

// The list of a cell's next pass. Mixed precision: the Hessian's moments in BF16 when the
// last condition estimate is <= condBf16, in 3xTF32 up to condMixMax or when there is no
// estimate yet, else (and after mixIterMax iterations at one regularisation level, or once a
// reduced-precision factorisation failed) in FP64; far: the multipliers exceed REF_NORM.
template <class S> __device__ int route_list(const S &sl, const ClosureParams &P, bool far)
{
    if (sl.s.need == NEED_PROBE)
        return 3;
    if (sl.s.need != NEED_H || !P.mixed || sl.s.fp64 || sl.s.iter > P.mixIterMax)
        return far ? 3 : 0;
    const double c = sl.s.cnd;
    if (c < 0.0)
        return 2;
    if (c <= P.condBf16)
        return 1;
    if (c <= P.condMixMax)
        return 2;
    return far ? 3 : 0;
}

// Appends cell c to its list when it still needs a pass.
template <class S>
__device__ void append_if_needed(const S &sl, const ClosureParams &P, long long c, int lane,
                                 const Lists &out)
{
    bool far = false;
    if (P.sym) {
        cell_sync<S>();
        double a2 = 0.0;
        for (int i = lane; i < P.nm; i += S::W)
            a2 = i > 0 ? fma(sl.alpha[i], sl.alpha[i], a2) : a2;
        far = !(cell_sum<S>(a2) <= REF_NORM * REF_NORM);
    }
    if (lane == 0 && sl.s.need != NEED_NONE) {
        // selects, not an indexed parameter array (which would be copied to local memory)
        const int l = route_list(sl, P, far);
        unsigned int *cnt = l == 0   ? out.count[0]
                            : l == 1 ? out.count[1]
                            : l == 2 ? out.count[2]
                                     : out.count[3];
        int *lst = l == 0 ? out.list[0] : l == 1 ? out.list[1] : l == 2 ? out.list[2] : out.list[3];
        unsigned int pos = atomicAdd(cnt, 1u);
        lst[pos] = (int)c;
    }
}

} // namespace

constexpr int RW = 8;  // warps (cells) per CTA of the init and pass kernels
// cells per CTA of the Newton kernel (NEWTON_THREADS threads, cell_lanes of them per cell)
__host__ __device__ constexpr int newton_cells(int nt) { return NEWTON_THREADS / cell_lanes(nt); }

// Entries a round kernel works on: n, or with nDev (the list's device counter, as the
// graph-resident round loop launches them) the smaller of n and *nDev.
__device__ __forceinline__ int round_entries(int n, const unsigned int *nDev)
{
    return nDev ? (int)min((unsigned int)n, *nDev) : n;
}

template <int NT> using TSlot = Slot<NT, true>;

// Per-warp state of a first visit after the probe pass: the vectors and scalars of Slot
// without the factor (the probe's Newton kernel forms no Hessian).
template <int NT> struct alignas(16) ProbeSlot {
    static constexpr int NMP = Cfg<NT>::NMP, W = cell_lanes(NT);
    double u[NMP], alpha[NMP], alpha0[NMP], uOrig[NMP], g[NMP], d[NMP], alphaOld[NMP];
    double pm[NMP + 8]; // the cell's probe entry, loaded before the cell's state
    SlotScalars s;
};
template <int NT, int MODE>
using NewtonSlot = typename std::conditional<MODE == 2, ProbeSlot<NT>, TSlot<NT>>::type;

template <int NT>
__global__ void __launch_bounds__(RW * 32)
    rounds_init_kernel(ClosureParams P, long long ncells, const int *__restrict__ cellMap,
                       Outputs O, CellState<NT> *state, Lists out)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Slot<NT> *slots = reinterpret_cast<Slot<NT> *>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long c = (long long)blockIdx.x * RW + warp;
    if (c >= ncells)
        return;
    Slot<NT> &sl = slots[warp];
    // the state and work lists use the closure's own numbering c; outputs the grid cell's
    load_cell(sl, P, O, cellMap ? (long long)cellMap[c] : c, lane);
    if (sl.s.need != NEED_NONE)
        slot_to_state(sl, state[c], lane);
    append_if_needed(sl, P, c, lane, out);
}

// Pass of the Gaunt form over RWP = 16 listed cells per CTA (warp w: cells 2w, 2w + 1):
// per staged chunk of QC directions, each lane forms the exponents alpha.m_q of both cells
// for its direction (the reference's order: moment index ascending, unfused,
// src/opt/fobj.cpp:64-79) and c_q = w_q e^{alpha.m_q}; then either the extended moments
// mom_k = sum_q M2[k][q] c_q of the cells that need H, as a DMMA GEMM [nm2 x QC] x [QC x 16]
// (each A fragment of M2 serves both 8-cell tiles), or the trial objective's quadrature sum.
// Chunk layout (c3d_set_gaunt): nm2 rows of M2 then the weight row, row stride QCP.
constexpr int RWP = 16;
constexpr int CST2 = 20; // row stride (cells) of the coefficient tile: conflict-free B fragments

template <int NT, int NT2>
__global__ void __launch_bounds__(RW * 32, 2)
    rounds_pass_gaunt_kernel(ClosureParams P, const double *__restrict__ chunks, int nm2,
                             const int *__restrict__ list, int n, const unsigned int *nDev,
                             CellState<NT> *state, double *__restrict__ momBuf, int *errorFlag)
{
    n = round_entries(n, nDev);
    if (blockIdx.x * RWP >= n)
        return;
    constexpr int NM2P = 8 * NT2;
    constexpr int RT = (NT2 + RW - 1) / RW;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int nm = P.nm, nchunks = P.nchunks;
    const int CH = (nm2 + 1) * QCP; // doubles per chunk (multiple of 4: 16-byte copies)
    double *stage = reinterpret_cast<double *>(smem_raw);
    double *cbuf = stage + GSTAGES * CH; // QC x CST2
    // multipliers of warp w's two cells interleaved, (cell 2w, cell 2w + 1) per moment: one
    // 16-byte broadcast load feeds both cells' exponents
    double2 *alph = reinterpret_cast<double2 *>(cbuf + QC * CST2); // RW x nm
    uint64_t *full = reinterpret_cast<uint64_t *>(alph + RW * nm);
    __shared__ int s_abort;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t chunkBytes = CH * sizeof(double);
    int need[2];
    long long cell[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int pos = blockIdx.x * RWP + 2 * warp + e;
        need[e] = NEED_NONE;
        cell[e] = -1;
        if (pos < n) {
            cell[e] = list[pos];
            need[e] = state[cell[e]].s.need;
        }
        for (int i = lane; i < nm; i += 32) {
            const double a = cell[e] >= 0 ? state[cell[e]].alpha[i] : 0.0;
            if (e == 0)
                alph[warp * nm + i].x = a;
            else
                alph[warp * nm + i].y = a;
        }
    }
    if (tid == 0) {
        for (int s = 0; s < GSTAGES; ++s)
            mbar_init(&full[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        s_abort = 0;
        for (int k = 0; k < GSTAGES && k < nchunks; ++k) {
            mbar_expect_tx(&full[k], chunkBytes);
            bulk_g2s(stage + k * CH, chunks + (size_t)k * CH, chunkBytes, &full[k]);
        }
    }
    __syncthreads();
    const bool anyH = __syncthreads_or(need[0] == NEED_H || need[1] == NEED_H);
    const double2 *aw = alph + warp * nm;
    double acc[RT][2][2];
#pragma unroll
    for (int r = 0; r < RT; ++r)
        acc[r][0][0] = acc[r][0][1] = acc[r][1][0] = acc[r][1][1] = 0.0;
    double fpart0 = 0.0, fpart1 = 0.0;
    const bool any = need[0] != NEED_NONE || need[1] != NEED_NONE;
    for (int k = 0; k < nchunks; ++k) {
        uint32_t s = k % GSTAGES, parity = (k / GSTAGES) & 1u;
        if (!mbar_wait(&full[s], parity))
            s_abort = 1;
        if (__syncthreads_or(s_abort)) {
            if (tid == 0) {
                atomicExch(errorFlag, 1);
                ring_drain<GSTAGES>(full, 0, k, nchunks);
            }
            return;
        }
        const double *ch = stage + s * CH;
        double c0 = 0.0, c1 = 0.0;
        if (any) {
            double z0 = 0.0, z1 = 0.0;
            for (int i = 0; i < nm; ++i) {
                const double m = ch[i * QCP + lane];
                const double2 a = aw[i];
                z0 = __dadd_rn(z0, __dmul_rn(a.x, m));
                z1 = __dadd_rn(z1, __dmul_rn(a.y, m));
            }
            const double wq = ch[nm2 * QCP + lane];
            if (need[0] != NEED_NONE) {
                c0 = __dmul_rn(wq, exp(z0));
                if (need[0] == NEED_TRIAL)
                    fpart0 = __dadd_rn(fpart0, c0);
            }
            if (need[1] != NEED_NONE) {
                c1 = __dmul_rn(wq, exp(z1));
                if (need[1] == NEED_TRIAL)
                    fpart1 = __dadd_rn(fpart1, c1);
            }
        }
        cbuf[lane * CST2 + 2 * warp] = (need[0] == NEED_H) ? c0 : 0.0;
        cbuf[lane * CST2 + 2 * warp + 1] = (need[1] == NEED_H) ? c1 : 0.0;
        __syncthreads();
        if (anyH) {
#pragma unroll
            for (int g = 0; g < QC / 4; ++g) {
                const double b0 = cbuf[(4 * g + (lane & 3)) * CST2 + (lane >> 2)];
                const double b1 = cbuf[(4 * g + (lane & 3)) * CST2 + 8 + (lane >> 2)];
#pragma unroll
                for (int r = 0; r < RT; ++r) {
                    const int rt = warp + r * RW;
                    const int row = 8 * rt + (lane >> 2);
                    if (rt < NT2) {
                        const double a = row < nm2 ? ch[row * QCP + 4 * g + (lane & 3)] : 0.0;
                        dmma(acc[r][0][0], acc[r][0][1], a, b0);
                        dmma(acc[r][1][0], acc[r][1][1], a, b1);
                    }
                }
            }
        }
        refill_fence();
        __syncthreads();
        if (tid == 0 && k + GSTAGES < nchunks) {
            mbar_expect_tx(&full[s], chunkBytes);
            bulk_g2s(stage + s * CH, chunks + (size_t)(k + GSTAGES) * CH, chunkBytes, &full[s]);
        }
    }
    if (anyH) {
        const int base = blockIdx.x * RWP;
#pragma unroll
        for (int r = 0; r < RT; ++r) {
            const int rt = warp + r * RW;
            if (rt < NT2) {
                const int kk = 8 * rt + (lane >> 2);
#pragma unroll
                for (int t = 0; t < 2; ++t)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int p = base + 8 * t + 2 * (lane & 3) + e;
                        if (p < n)
                            momBuf[(size_t)p * NM2P + kk] = acc[r][t][e];
                    }
            }
        }
    }
    const double fq0 = warp_sum(fpart0), fq1 = warp_sum(fpart1);
    if (lane == 0) {
        if (need[0] == NEED_TRIAL)
            state[cell[0]].s.fquad = fq0;
        if (need[1] == NEED_TRIAL)
            state[cell[1]].s.fquad = fq1;
    }
}

// Pass of the direct form: per listed cell, the lower-triangle DMMA tiles of H (packed
// into hBuf[pos]) or the trial's quadrature sum.
template <int NT>
__global__ void __launch_bounds__(RW * 32, 1)
    rounds_pass_direct_kernel(ClosureParams P, const double *__restrict__ chunks,
                              const int *__restrict__ list, int n, const unsigned int *nDev,
                              CellState<NT> *state, double *__restrict__ hBuf, int *errorFlag)
{
    n = round_entries(n, nDev);
    if (blockIdx.x * RW >= n)
        return;
    constexpr int NMP = Cfg<NT>::NMP;
    constexpr int CH = Cfg<NT>::CHUNK;
    constexpr int ST = 3;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    double *stage = reinterpret_cast<double *>(smem_raw);
    double *alph = stage + ST * CH;
    uint64_t *full = reinterpret_cast<uint64_t *>(alph + RW * NMP);
    __shared__ int s_abort;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nm = P.nm, nchunks = P.nchunks;
    const uint32_t chunkBytes = CH * sizeof(double);
    const int pos = blockIdx.x * RW + warp;
    int need = NEED_NONE;
    long long cell = -1;
    if (pos < n) {
        cell = list[pos];
        need = state[cell].s.need;
    }
    for (int i = lane; i < NMP; i += 32)
        alph[warp * NMP + i] = (cell >= 0 && i < nm) ? state[cell].alpha[i] : 0.0;
    if (tid == 0) {
        for (int s = 0; s < ST; ++s)
            mbar_init(&full[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        s_abort = 0;
        for (int k = 0; k < ST && k < nchunks; ++k) {
            mbar_expect_tx(&full[k], chunkBytes);
            bulk_g2s(stage + k * CH, chunks + (size_t)k * CH, chunkBytes, &full[k]);
        }
    }
    __syncthreads();
    const double *al = alph + warp * NMP;
    double acc[Cfg<NT>::NTILE][2];
#pragma unroll
    for (int t = 0; t < Cfg<NT>::NTILE; ++t)
        acc[t][0] = acc[t][1] = 0.0;
    double fpart = 0.0;
    for (int k = 0; k < nchunks; ++k) {
        uint32_t s = k % ST, parity = (k / ST) & 1u;
        if (!mbar_wait(&full[s], parity))
            s_abort = 1;
        if (__syncthreads_or(s_abort)) {
            if (tid == 0) {
                atomicExch(errorFlag, 1);
                ring_drain<ST>(full, 0, k, nchunks);
            }
            return;
        }
        const double *ch = stage + s * CH;
        if (need != NEED_NONE) {
            double z = 0.0;
            for (int i = 0; i < nm; ++i)
                z = __dadd_rn(z, __dmul_rn(al[i], ch[i * QCP + lane]));
            double c = __dmul_rn(ch[NMP * QCP + lane], exp(z));
            if (need == NEED_TRIAL) {
                fpart = __dadd_rn(fpart, c);
            } else {
#pragma unroll
                for (int g = 0; g < QC / 4; ++g) {
                    double cq = __shfl_sync(FULL_MASK, c, 4 * g + (lane & 3));
                    double m[NT], a[NT];
#pragma unroll
                    for (int I = 0; I < NT; ++I) {
                        m[I] = ch[(8 * I + (lane >> 2)) * QCP + 4 * g + (lane & 3)];
                        a[I] = cq * m[I];
                    }
#pragma unroll
                    for (int I = 0; I < NT; ++I)
#pragma unroll
                        for (int J = 0; J <= I; ++J)
                            dmma(acc[I * (I + 1) / 2 + J][0], acc[I * (I + 1) / 2 + J][1], a[I],
                                 m[J]);
                }
            }
        }
        refill_fence();
        __syncthreads();
        if (tid == 0 && k + ST < nchunks) {
            mbar_expect_tx(&full[s], chunkBytes);
            bulk_g2s(stage + s * CH, chunks + (size_t)(k + ST) * CH, chunkBytes, &full[s]);
        }
    }
    if (need == NEED_H) {
        // tiles of the padded H, identity in the padding rows
        double *H = hBuf + (size_t)pos * TSlot<NT>::LSIZE;
#pragma unroll
        for (int I = 0; I < NT; ++I)
#pragma unroll
            for (int J = 0; J <= I; ++J) {
                const int t = I * (I + 1) / 2 + J;
                int row = 8 * I + (lane >> 2), col = 8 * J + 2 * (lane & 3);
                double v0 = acc[t][0], v1 = acc[t][1];
                if (row >= nm || col >= nm)
                    v0 = (row == col) ? 1.0 : 0.0;
                if (row >= nm || col + 1 >= nm)
                    v1 = (row == col + 1) ? 1.0 : 0.0;
                *reinterpret_cast<double2 *>(&H[64 * t + tpair(lane)]) = make_double2(v0, v1);
            }
    } else if (need == NEED_TRIAL) {
        double fq = warp_sum(fpart);
        if (lane == 0)
            state[cell].s.fquad = fq;
    }
}

// ---------------------------------------------------------------- mixed-precision pass
// Pass of the mixed-precision closure over MXC = 16 listed cells per CTA that need a Hessian
// (warp w: cells 2w, 2w + 1; lane: direction of the staged 32-direction chunk):
//   FP64   exponents alpha.m_q (moment index ascending, unfused), c_q = w_q e^{alpha.m_q},
//          f's sum over q, and the first-order moments <m_i e^{alpha.m}> (i < nm) as a DMMA
//          GEMM [nm x QC] x [QC x 16] -- the gradient and objective of the FP64 stopping test
//          and line search;
//   tcgen05 the extended moments mom_k = sum_q M2[k][q] c_q of the Gaunt Hessian as
//          D[128 x 16] += A[128 x K] B[16 x K]^T per M = 128 row tile (A: the staged M2 rows
//          in BF16, or hi and lo TF32 parts; B: the cells' c_q scaled by 2^-shift, the
//          cell's largest c of its previous pass, in the same format), FP32 accumulators in
//          tensor memory. 3xTF32: A_hi B_hi + A_hi B_lo + A_lo B_hi.
// One thread issues the MMAs of a chunk once the CTA has written its B tile; their commit
// releases the chunk's stage and B buffer. Staged chunk: the nm rows of M2 of degree <= N
// and the weight row (FP64, row stride QCP), then the A operand (c3d_set_gaunt).
// Output entry (stride NM2P + NMP + 8 doubles): the nm2 moments, the nm FP64 moments, f's sum.
template <int KIND> struct MixKind;
template <> struct MixKind<0> { // BF16
    static constexpr int ES = 2, NP = 1, KI = 16;
    static constexpr uint32_t FMT = 1;
};
template <> struct MixKind<1> { // 3xTF32
    static constexpr int ES = 4, NP = 2, KI = 8;
    static constexpr uint32_t FMT = 2;
};
template <> struct MixKind<2> { // probe: the FP64 part alone
    static constexpr int ES = 8, NP = 0, KI = 8;
    static constexpr uint32_t FMT = 0;
};
constexpr int MXC = 16;

template <int NT2> struct MixRows {
    static constexpr int NM2P = 8 * NT2;
    static constexpr int NA = NM2P < 128 ? 128 : NM2P; // staged A rows (zero beyond nm2)
    static constexpr int MT = NM2P <= 128 ? 1 : 2;     // M = 128 row tiles
    static constexpr int ROW1 = NM2P - 128;            // first row of tile 1 (overlaps tile 0)
    static_assert(NM2P <= 256, "two row tiles");
};

__host__ __device__ constexpr int mix_entry_doubles(int nmp, int nm2p) { return nm2p + nmp + 8; }
// Probe entry (KIND 2): the NMP first-order moments, f's sum, e_min, e_max.
__host__ __device__ constexpr int probe_entry_doubles(int nmp) { return nmp + 8; }

// KIND 2 is the probe pass of a cell's first visit (the convergence certificate): the FP64
// part alone, with the extreme values of e^{alpha.m_q} over the chunk's directions.
// ZD (the mixed closure's passes): the exponents of the chunk as a DMMA GEMM
// Z[32 x 16] = M_chunk^T [32 x nm] alpha [nm x 16] (warp w: directions 8 (w % 4) .., cells
// 8 (w / 4) ..) staged through shared memory, instead of the reference's unfused order.
[[maybe_unused]] constexpr int ZS = 18; // row stride (cells) of the exponent tile: 16-byte pairs, 8-lane phases
                       // conflict-free

// The first round of a closure with the convergence certificate: no list and no set-up
// kernel; list position p is closure cell off + p, its grid cell cellMap[off + p] (or the
// same index), and the probe pass reads the grid's moments and multipliers directly (the
// scaling of load_cell, src/opt/optBatch.cpp:312-331), the probe's Newton kernel sets the cell
// up with load_cell.
struct FirstRound {
    long long off;
    const int *cellMap;
    const double *u, *alpha;
    // ansatz hand-off to the kinetic flux (grid closures with the certificate): the probe pass
    // writes psi[q nall + c] = exp(alpha_c . m_q) of every cell it solves, and the probe's
    // Newton kernel marks the cells whose multipliers may still change (their psi is
    // rewritten after the closure). Null psi: no hand-off.
    double *psi;
    long long nall;
    unsigned char *mark;
    // nonzero: psi already holds the ansatz of every cell but the face ghosts for the closure's
    // starting multipliers (the previous closure's final ones), so the probe writes only the
    // face ghosts' (gnx, gny, gnz: the interior sizes that tell them)
    const int *psiValid;
    int gnx, gny, gnz;
    // symmetric quadrature: the probe pass finishes certified cells itself and lists the others'
    // positions here for the Newton kernel (null: every cell)
    int *todo;
    unsigned int *todoCount;
};
[[maybe_unused]] constexpr int PSTR = 17; // row stride (cells) of the probe's psi tile
[[maybe_unused]] constexpr int PRS = 3;   // stages of the mixed probe's psi read ring (chunks k .. k + 2)

// 8-byte asynchronous global -> shared copy (zero fill when !valid; src is not read then)
__device__ __forceinline__ void cp_async8(double *dst, const double *src, bool valid)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src),
                 "r"(valid ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

template <int NT, int NT2, int KIND, bool ZD>
__global__ void __launch_bounds__(RW * 32, KIND == 1 ? 1 : KIND == 2 ? 3 : 2)
    rounds_pass_mixed_kernel(ClosureParams P, const double *__restrict__ f64c,
                             const unsigned char *__restrict__ ac, const int *__restrict__ list,
                             int n, const unsigned int *nDev, CellState<NT> *state,
                             double *__restrict__ out, int *errorFlag, FirstRound first)
{
    n = round_entries(n, nDev);
    if (blockIdx.x * MXC >= n)
        return;
    using K = MixKind<KIND>;
    using R = MixRows<NT2>;
    constexpr int NMP = 8 * NT;
    constexpr int KG = QC * K::ES / 16, SBO = KG * 128;
    constexpr uint32_t APB = R::NA * QC * K::ES, BPB = MXC * QC * K::ES;
    constexpr bool TC = KIND < 2; // tensor-core moments
    constexpr int ESTR = TC ? mix_entry_doubles(NMP, R::NM2P) : probe_entry_doubles(NMP);
    constexpr uint32_t IDESC = umma_idesc(K::FMT, 128, MXC);
    static_assert(NT <= RW, "one FP64 row tile per warp");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int nm = P.nm, nchunks = P.nchunks;
    const uint32_t f64Bytes = (uint32_t)(nm + 1) * QCP * 8;
    const uint32_t f64Pad = (f64Bytes + 127u) & ~127u;
    const uint32_t stg = f64Pad + K::NP * APB;
    unsigned char *bbuf = smem_raw + GSTAGES * stg; // GSTAGES x NP x BPB
    double *cbuf = reinterpret_cast<double *>(bbuf + GSTAGES * K::NP * BPB); // QC x CST2
    double2 *alph = reinterpret_cast<double2 *>(cbuf + QC * CST2);          // RW x nm
    double *zbuf = reinterpret_cast<double *>(alph + RW * nm);              // ZD: QC x ZS
    double *psiT = zbuf + (ZD ? QC * ZS : 0);                               // probe: QC x PSTR
    double *psiR = psiT + (KIND == 2 ? QC * PSTR : 0); // mixed probe: PRS x QC x PSTR
    long long *psiCell =
        reinterpret_cast<long long *>(psiR + (KIND == 2 && ZD ? PRS * QC * PSTR : 0));
    uint64_t *full = reinterpret_cast<uint64_t *>(psiCell + (KIND == 2 ? MXC : 0));
    uint64_t *mmab = full + GSTAGES;
    uint64_t *fin = mmab + GSTAGES;
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    __shared__ int s_shift[MXC];
    __shared__ long long s_gc[MXC];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int base = blockIdx.x * MXC;
    // first round of a grid closure: hand the ansatz of every direction to the kinetic flux,
    // psi = u_0 e^{alpha_scaled . m_q} (the scaling shifts alpha_0 by log(u_0) 2 sqrt(pi), and
    // m_0 = 1 / (2 sqrt(pi)))
    const bool emit = KIND == 2 && !list && first.psi != nullptr;
    const bool valid = emit && first.psiValid && *first.psiValid != 0;
    long long cell[2];
    double scale[2], u0e[2] = {0.0, 0.0};
    int needMine = 0; // lane 0: one of the warp's cells has its psi written by this pass
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int pos = base + 2 * warp + e;
        cell[e] = pos < n ? (list ? list[pos] : first.off + pos) : -1;
        long long gc = -1;
        double ascale = 0.0;
        if (!list && cell[e] >= 0) {
            gc = first.cellMap ? first.cellMap[cell[e]] : cell[e];
            u0e[e] = first.u[gc * nm];
            ascale = log(u0e[e]) * 2.0 * sqrt(M_PI);
        }
        if constexpr (KIND == 2)
            if (lane == 0) {
                bool need = emit;
                if (valid && gc >= 0) {
                    // only a face ghost's psi may be missing (its image's was read instead)
                    const int gz = first.gnz + 4, gy = first.gny + 4;
                    const int k = (int)(gc % gz), j = (int)((gc / gz) % gy), i = (int)(gc / gz / gy);
                    const int in = (i >= 2 && i < first.gnx + 2) + (j >= 2 && j < first.gny + 2) +
                                   (k >= 2 && k < first.gnz + 2);
                    need = in == 2;
                }
                psiCell[2 * warp + e] = need ? gc : -1;
                s_gc[2 * warp + e] = gc;
                needMine |= need && gc >= 0;
            }
        for (int i = lane; i < nm; i += 32) {
            double a = 0.0;
            if (cell[e] >= 0) {
                if (list) {
                    a = state[cell[e]].alpha[i];
                } else {
                    a = first.alpha[gc * nm + i];
                    if (i == 0)
                        a = a - ascale;
                }
            }
            if (e == 0)
                alph[warp * nm + i].x = a;
            else
                alph[warp * nm + i].y = a;
        }
        const int sh = (cell[e] >= 0 && list) ? state[cell[e]].s.cshift : 0;
        if (lane == 0)
            s_shift[2 * warp + e] = sh;
        scale[e] = ldexp(1.0, -sh);
    }
    if (tid == 0) {
        for (int s = 0; s < GSTAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&mmab[s], 1);
        }
        mbar_init(fin, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        s_abort = 0;
        for (int k = 0; k < GSTAGES && k < nchunks; ++k) {
            unsigned char *st = smem_raw + k * stg;
            mbar_expect_tx(&full[k], f64Bytes + K::NP * APB);
            bulk_g2s(st, f64c + (size_t)k * (nm + 1) * QCP, f64Bytes, &full[k]);
            if constexpr (TC)
                bulk_g2s(st + f64Pad, ac + (size_t)k * K::NP * APB, K::NP * APB, &full[k]);
        }
    }
    if constexpr (TC)
        if (warp == 0)
            tmem_alloc(&s_tmem, 32);
    tc_fence_before();
    const int anyNeed = __syncthreads_or(needMine);
    tc_fence_after();
    const uint32_t tmem = TC ? s_tmem : 0u;
    // mixed probe with psi valid and no cell of the CTA needing its psi written: psi already
    // holds u_0 e^{alpha_scaled . m_q} of every cell, so the pass reads e^{alpha_scaled . m_q}
    // back (psi / u_0) instead of forming the exponent tile and the exponentials; the reads
    // run two chunks ahead through a ring of asynchronous copies
    const bool rd = ZD && valid && !anyNeed;
    auto psi_fetch = [&](int kc) {
        double *dst = psiR + (kc % PRS) * QC * PSTR;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int row = 4 * warp + 2 * i + (lane >> 4), j = lane & 15;
            const int q = kc * QC + row;
            const long long gc = s_gc[j];
            const bool ok = kc < nchunks && gc >= 0 && q < P.nq;
            cp_async8(dst + row * PSTR + j, ok ? first.psi + (long long)q * first.nall + gc : first.psi,
                      ok);
        }
        cp_async_commit();
    };
    if constexpr (KIND == 2 && ZD) {
        if (rd) {
            // u0e holds 1 / u_0 from here on: the read path writes no psi
            u0e[0] = 1.0 / u0e[0];
            u0e[1] = 1.0 / u0e[1];
            psi_fetch(0);
            psi_fetch(1);
        }
    }
    const double2 *aw = alph + warp * nm;
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    double fpart0 = 0.0, fpart1 = 0.0, cmax0 = 0.0, cmax1 = 0.0;
    double emin0 = 1.0 / 0.0, emin1 = 1.0 / 0.0, emax0 = 0.0, emax1 = 0.0;
    for (int k = 0; k < nchunks; ++k) {
        const uint32_t s = k % GSTAGES, parity = (k / GSTAGES) & 1u;
        if (!mbar_wait(&full[s], parity))
            s_abort = 1;
        if constexpr (KIND == 2 && ZD)
            if (rd)
                cp_async_wait<1>(); // this thread's copies of chunk k have landed
        if (__syncthreads_or(s_abort)) {
            if (tid == 0)
                ring_drain<GSTAGES>(full, 0, k, nchunks);
            break;
        }
        const unsigned char *stb = smem_raw + s * stg;
        const double *ch = reinterpret_cast<const double *>(stb);
        double z0 = 0.0, z1 = 0.0, ez0 = 0.0, ez1 = 0.0;
        if (KIND == 2 && ZD && rd) {
            // stage (k + 2) % PRS was last read in chunk k - 1, before the barrier above
            psi_fetch(k + 2);
            const double *pr = psiR + (k % PRS) * QC * PSTR + lane * PSTR + 2 * warp;
            const bool qv = k * QC + lane < P.nq; // padded directions: exponent 0
            ez0 = cell[0] >= 0 && qv ? pr[0] * u0e[0] : 1.0;
            ez1 = cell[1] >= 0 && qv ? pr[1] * u0e[1] : 1.0;
        } else if constexpr (ZD) {
            // A[dir r][k] = M2[k][8 dt + r], B[k][cell n] = alpha_n[k] (zero for k >= nm)
            const int dt = warp & 3, ct = warp >> 2, r = lane >> 2, kq = lane & 3;
            const int nb = 8 * ct + r;
            const double2 *ab = alph + (nb >> 1) * nm;
            double d0 = 0.0, d1 = 0.0;
            for (int ks = 0; ks < (nm + 3) / 4; ++ks) {
                const int k = 4 * ks + kq;
                double a = 0.0, b = 0.0;
                if (k < nm) {
                    a = ch[k * QCP + 8 * dt + r];
                    const double2 v = ab[k];
                    b = (nb & 1) ? v.y : v.x;
                }
                dmma(d0, d1, a, b);
            }
            *reinterpret_cast<double2 *>(&zbuf[(8 * dt + r) * ZS + 8 * ct + 2 * kq]) =
                make_double2(d0, d1);
            __syncthreads();
            const double2 zz = *reinterpret_cast<const double2 *>(&zbuf[lane * ZS + 2 * warp]);
            z0 = zz.x;
            z1 = zz.y;
        } else {
            for (int i = 0; i < nm; ++i) {
                const double m = ch[i * QCP + lane];
                const double2 a = aw[i];
                z0 = __dadd_rn(z0, __dmul_rn(a.x, m));
                z1 = __dadd_rn(z1, __dmul_rn(a.y, m));
            }
        }
        const double wq = ch[nm * QCP + lane];
        if (!(KIND == 2 && ZD && rd)) {
            ez0 = exp(z0);
            ez1 = exp(z1);
        }
        if constexpr (KIND == 2) {
            if (emit && !rd) {
                psiT[lane * PSTR + 2 * warp] = u0e[0] * ez0;
                psiT[lane * PSTR + 2 * warp + 1] = u0e[1] * ez1;
            }
        }
        const double c0 = cell[0] >= 0 ? __dmul_rn(wq, ez0) : 0.0;
        const double c1 = cell[1] >= 0 ? __dmul_rn(wq, ez1) : 0.0;
        fpart0 = __dadd_rn(fpart0, c0);
        fpart1 = __dadd_rn(fpart1, c1);
        if constexpr (TC) {
            cmax0 = fmax(cmax0, c0);
            cmax1 = fmax(cmax1, c1);
        } else {
            emin0 = fmin(emin0, ez0);
            emin1 = fmin(emin1, ez1);
            emax0 = fmax(emax0, ez0);
            emax1 = fmax(emax1, ez1);
        }
        cbuf[lane * CST2 + 2 * warp] = c0;
        cbuf[lane * CST2 + 2 * warp + 1] = c1;
        // B tile: cell row nn, direction column lane
        unsigned char *bt = bbuf + s * K::NP * BPB;
#pragma unroll
        for (int e = 0; e < (TC ? 2 : 0); ++e) {
            const int nn = 2 * warp + e;
            const double v = (e == 0 ? c0 : c1) * scale[e];
            const uint32_t off = (nn >> 3) * SBO + ((lane * K::ES) >> 4) * 128 + (nn & 7) * 16 +
                                 ((lane * K::ES) & 15);
            if constexpr (KIND == 0) {
                *reinterpret_cast<__nv_bfloat16 *>(bt + off) = __float2bfloat16_rn((float)v);
            } else {
                const uint32_t hi = to_tf32((float)v);
                const float lo = (float)(v - (double)__uint_as_float(hi));
                *reinterpret_cast<uint32_t *>(bt + off) = hi;
                *reinterpret_cast<uint32_t *>(bt + BPB + off) = to_tf32(lo);
            }
        }
        if constexpr (TC)
            fence_async_smem();
        __syncthreads();
        if (TC && tid == 0) {
            tc_fence_after();
            const uint32_t aAddr = umma_smem_u32(stb + f64Pad), bAddr = umma_smem_u32(bt);
#pragma unroll
            for (int j = 0; j < QC / K::KI; ++j)
#pragma unroll
                for (int t = 0; t < R::MT; ++t) {
                    const uint32_t d = tmem + 16 * t;
                    const uint32_t a0 = aAddr + (t == 0 ? 0 : (R::ROW1 / 8) * SBO) + 256 * j;
                    const uint32_t b0 = bAddr + 256 * j;
                    umma_issue<KIND == 1>(d, umma_desc(a0, SBO), umma_desc(b0, SBO), IDESC,
                                          (k > 0 || j > 0) ? 1u : 0u);
                    if constexpr (KIND == 1) {
                        umma_issue<true>(d, umma_desc(a0, SBO), umma_desc(b0 + BPB, SBO), IDESC, 1u);
                        umma_issue<true>(d, umma_desc(a0 + APB, SBO), umma_desc(b0, SBO), IDESC, 1u);
                    }
                }
            umma_commit(&mmab[s]);
        }
        if constexpr (KIND == 2) {
            // the chunk's psi rows: warp w stores directions 4w .. 4w + 3, 16 cells each
            if (emit && !rd) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int row = 4 * warp + 2 * i + (lane >> 4), j = lane & 15;
                    const long long gc = psiCell[j];
                    const int q = k * QC + row;
                    if (gc >= 0 && q < P.nq)
                        first.psi[(long long)q * first.nall + gc] = psiT[row * PSTR + j];
                }
            }
        }
        // FP64 first-order moments: warp w, rows 8w .. 8w + 7
        if (warp < NT) {
            const int row = 8 * warp + (lane >> 2);
#pragma unroll
            for (int g = 0; g < QC / 4; ++g) {
                const double b0 = cbuf[(4 * g + (lane & 3)) * CST2 + (lane >> 2)];
                const double b1 = cbuf[(4 * g + (lane & 3)) * CST2 + 8 + (lane >> 2)];
                const double a = row < nm ? ch[row * QCP + 4 * g + (lane & 3)] : 0.0;
                dmma(acc[0][0], acc[0][1], a, b0);
                dmma(acc[1][0], acc[1][1], a, b1);
            }
        }
        refill_fence();
        __syncthreads();
        if (tid == 0 && k + GSTAGES < nchunks) {
            // the MMAs of chunk k have read stage s and B buffer s
            if (TC && !mbar_wait(&mmab[s], parity)) {
                s_abort = 1;
            } else {
                unsigned char *st = smem_raw + s * stg;
                const int kn = k + GSTAGES;
                mbar_expect_tx(&full[s], f64Bytes + K::NP * APB);
                bulk_g2s(st, f64c + (size_t)kn * (nm + 1) * QCP, f64Bytes, &full[s]);
                if constexpr (TC)
                    bulk_g2s(st + f64Pad, ac + (size_t)kn * K::NP * APB, K::NP * APB, &full[s]);
            }
        }
    }
    if constexpr (KIND == 2 && ZD)
        if (rd)
            cp_async_wait<0>(); // no copy outstanding past the loop (an abort leaves it early)
    // every MMA complete before the accumulators are read and the columns freed
    if (TC && tid == 0) {
        umma_commit(fin);
        if (!mbar_wait(fin, 0))
            s_abort = 1;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const bool ok = s_abort == 0;
    if (!ok && tid == 0)
        atomicExch(errorFlag, 1);
    if (ok) {
        const int qw = warp & 3, t = warp >> 2;
        if (TC && t < R::MT) {
            uint32_t r[16];
            tmem_ld16(tmem + ((uint32_t)(32 * qw) << 16) + 16 * t, r);
            const int row = (t == 0 ? 0 : R::ROW1) + 32 * qw + lane;
            if (row < R::NM2P && (t == 0 || row >= 128)) {
#pragma unroll
                for (int j = 0; j < MXC; ++j)
                    if (base + j < n)
                        out[(size_t)(base + j) * ESTR + row] =
                            ldexp((double)__uint_as_float(r[j]), s_shift[j]);
            }
        }
        if (warp < NT) {
            const int kk = 8 * warp + (lane >> 2);
#pragma unroll
            for (int tt = 0; tt < 2; ++tt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int p = base + 8 * tt + 2 * (lane & 3) + e;
                    if (p < n)
                        out[(size_t)p * ESTR + (TC ? R::NM2P : 0) + kk] = acc[tt][e];
                }
        }
        const double fq0 = warp_sum(fpart0), fq1 = warp_sum(fpart1);
        double x0, x1, y0 = 0.0, y1 = 0.0;
        if constexpr (TC) {
            x0 = warp_max(cmax0);
            x1 = warp_max(cmax1);
        } else {
            x0 = -warp_max(-emin0);
            x1 = -warp_max(-emin1);
            y0 = warp_max(emax0);
            y1 = warp_max(emax1);
        }
        if (lane == 0) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int p = base + 2 * warp + e;
                if (p < n) {
                    double *o = out + (size_t)p * ESTR + (TC ? R::NM2P : 0) + NMP;
                    o[0] = e == 0 ? fq0 : fq1;
                    if constexpr (TC) {
                        const double cm = e == 0 ? x0 : x1;
                        int sh = (cm > 0.0 && cm < 1.0 / 0.0) ? ilogb(cm) : 0;
                        state[cell[e]].s.cshift = sh < -120 ? -120 : sh > 120 ? 120 : sh;
                    } else {
                        o[1] = e == 0 ? x0 : x1;
                        o[2] = e == 0 ? y0 : y1;
                    }
                }
            }
        }
    }
    if constexpr (TC) {
        tc_fence_before();
        __syncthreads();
        if (warp == 0) {
            tc_fence_after();
            tmem_dealloc(tmem, 32);
        }
    }
}

// ---------------------------------------------------------------- octant-symmetric passes
// The passes of a context whose quadrature has the octant symmetry (sym.cuh). A warp owns 8
// cells; per block of 8 octant directions a lane forms the 16 exponents of cell lane / 4 at 2
// octant directions x 8 reflections (sym_expand, one DMMA per 4 multipliers of a parity
// class), their exponentials and the class sums of w e^{alpha.m} (sym_wht), which the DMMAs of
// sym_contract project onto the class members straight from registers. The tables of a block
// are staged by bulk copies, SYM_STAGES deep, one barrier per block.

constexpr int SYM_STAGES = 3;
[[maybe_unused]] constexpr int SYM_PASS_WARPS = 4;
[[maybe_unused]] constexpr int SYM_PROBE_WARPS = 4; // (8 and 2 CTAs per SM: 2 to 5% slower for N <= 6)
[[maybe_unused]] constexpr unsigned PROBE_GRID = 148 * 16; // CTAs that walk a probe's list

// Degree of the basis of rounds_t<NT, NT2, true>.
__host__ __device__ constexpr int sym_order(int nt2)
{
    return nt2 == 1 ? 0 : nt2 == 2 ? 1 : nt2 == 4 ? 2 : nt2 == 7 ? 3 : nt2 == 11 ? 4 : nt2 == 16 ? 5
         : nt2 == 22 ? 6 : 7;
}

// Doubles of a staged block: expansion fragments of degree DEG, projection fragments of degree PD.
template <int DEG, int PD> struct SymStage {
    static constexpr int EXPO = SymCls<DEG>::STEPS * 32;
    static constexpr int PROJ = 2 * SymCls<PD>::TILES * 32;
    static constexpr int DOUBLES = EXPO + PROJ;
};
template <int DEG, int PD, int WARPS> constexpr size_t sym_smem()
{
    return (size_t)(SYM_STAGES * SymStage<DEG, PD>::DOUBLES + WARPS * SymCls<DEG>::STEPS * 32) * 8;
}

// Loads block b of the tables into stage b % SYM_STAGES (one thread).
template <int DEG, int PD>
__device__ __forceinline__ void sym_stage_load(const SymTables &T, int b, double *stage, uint64_t *full)
{
    using G = SymStage<DEG, PD>;
    const int s = b % SYM_STAGES;
    double *st = stage + s * G::DOUBLES;
    mbar_expect_tx(&full[s], G::DOUBLES * 8);
    bulk_g2s(st, T.expo + (size_t)b * G::EXPO, G::EXPO * 8, &full[s]);
    bulk_g2s(st + G::EXPO, T.proj + (size_t)b * G::PROJ, G::PROJ * 8, &full[s]);
}

// What a trial pass computes besides f: with fused trials the moments at the trial point, which
// the Newton kernel uses when it accepts the trial (the next iteration's Hessian visit then
// needs no pass of its own). Not fused when that visit belongs to a reduced-precision list.
__device__ __forceinline__ bool trial_fused(const ClosureParams &P, int fp64, int iter, double cnd)
{
    return !P.mixed || fp64 || iter + 1 > P.mixIterMax || cnd > P.condMixMax;
}

// Hessian and trial pass over the listed cells (the FP64 list): the nm2 extended moments of
// cells that need them into momBuf (stride 8 NT2), followed by bounds of e^{alpha.m} (the extreme
// high words, rounded outwards), and f's sum of trial cells into their state. FP64 pipe bound: 24
// class tiles over nq / 8 directions for the 169 moments of M_6 against 22 over nq. M_4 64^3:
// 2.7 ms per two steps (17.4 with all directions), M_5 visits 1.1 ns each. 8 warps per CTA: 1 to 15%
// slower; one CTA more per SM (fewer registers) 3 to 30%.
template <int NT, int NT2>
__global__ void __launch_bounds__(SYM_PASS_WARPS * 32, NT2 > 16 ? 2 : 4)
    sym_pass_kernel(ClosureParams P, SymTables T, const int *__restrict__ list, int n,
                    const unsigned int *nDev, CellState<NT> *state, double *__restrict__ momBuf,
                    int *errorFlag)
{
    n = round_entries(n, nDev);
    constexpr int WARPS = SYM_PASS_WARPS, DEG = sym_order(NT2), PD = 2 * DEG;
    if (blockIdx.x * (8 * WARPS) >= n)
        return;
    using C = SymCls<DEG>;
    using E = SymCls<PD>;
    using G = SymStage<DEG, PD>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    double *stage = reinterpret_cast<double *>(smem_raw);
    __shared__ uint64_t full[SYM_STAGES];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *aF = stage + SYM_STAGES * G::DOUBLES + warp * C::STEPS * 32;
    if (tid == 0) {
        for (int s = 0; s < SYM_STAGES; ++s)
            mbar_init(&full[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        for (int b = 0; b < SYM_STAGES && b < T.nb; ++b)
            sym_stage_load<DEG, PD>(T, b, stage, full);
    }
    const int pos = (blockIdx.x * WARPS + warp) * 8 + (lane >> 2);
    long long cell = -1;
    bool trial = false, wantH = false;
    if (pos < n) {
        cell = list[pos];
        const SlotScalars &sc = state[cell].s;
        trial = sc.need == NEED_TRIAL;
        wantH = sc.need == NEED_H || (trial && trial_fused(P, sc.fp64, sc.iter, sc.cnd));
    }
#pragma unroll
    for (int k = 0; k < C::STEPS; ++k) {
        const int m = T.stepIdx[4 * k + (lane & 3)];
        aF[k * 32 + lane] = cell >= 0 && m >= 0 ? state[cell].alpha[m] : 0.0;
    }
    const bool any = __any_sync(FULL_MASK, cell >= 0), anyH = __any_sync(FULL_MASK, wantH);
    double acc[E::TILES][2];
#pragma unroll
    for (int t = 0; t < E::TILES; ++t)
        acc[t][0] = acc[t][1] = 0.0;
    double f = 0.0;
    int lo = 0x7fffffff, hi = 0;
    __syncthreads();
    for (int b = 0; b < T.nb; ++b) {
        const double *st = stage + (b % SYM_STAGES) * G::DOUBLES;
        const bool ok = mbar_wait(&full[b % SYM_STAGES], (b / SYM_STAGES) & 1);
        if (any) {
            double v[2][8];
            sym_expand<DEG>(aF, st, lane, v);
            const double2 w = *reinterpret_cast<const double2 *>(T.w + SYM_BLK * b + 2 * (lane & 3));
#pragma unroll
            for (int e = 0; e < 2; ++e) {
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const double ez = exp(v[e][s]);
                    // (directions past the last have exponent 0: they only widen the bounds)
                    lo = min(lo, __double2hiint(ez));
                    hi = max(hi, __double2hiint(ez));
                    v[e][s] = (e == 0 ? w.x : w.y) * ez;
                }
                sym_wht(v[e]);
                f += v[e][0];
                if (anyH)
                    sym_contract<PD>(v[e], st + G::EXPO + e * (E::TILES * 32), lane, acc);
            }
        }
        refill_fence();
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicExch(errorFlag, 1);
                ring_drain<SYM_STAGES>(full, 0, b, T.nb);
            }
            return;
        }
        if (tid == 0 && b + SYM_STAGES < T.nb)
            sym_stage_load<DEG, PD>(T, b + SYM_STAGES, stage, full);
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        lo = min(lo, __shfl_xor_sync(FULL_MASK, lo, o));
        hi = max(hi, __shfl_xor_sync(FULL_MASK, hi, o));
    }
    if (wantH) {
        double *o = momBuf + (size_t)pos * (8 * NT2);
        static_assert((PD + 1) * (PD + 1) + 2 <= 8 * NT2, "room for the bounds");
        if ((lane & 3) == 0) {
            o[(PD + 1) * (PD + 1)] = __hiloint2double(lo, 0);
            o[(PD + 1) * (PD + 1) + 1] = __hiloint2double(hi, -1);
        }
#pragma unroll
        for (int t = 0; t < E::TILES; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int m = T.idx[8 * t + 2 * (lane & 3) + e];
                if (m >= 0)
                    o[m] = acc[t][e];
            }
    }
    f += __shfl_xor_sync(FULL_MASK, f, 1);
    f += __shfl_xor_sync(FULL_MASK, f, 2);
    if (trial && (lane & 3) == 0)
        state[cell].s.fquad = f;
}

// Probe pass of a closure's first round (FirstRound; see rounds_pass_mixed_kernel for the
// hand-off's psi and the certificate's entry): first-order moments, f's sum and bounds of
// e^{alpha.m} per cell. It always forms e^{alpha.m}: reading psi / u_0 back instead was no faster
// (11.9 against 10.8 ms per M_6 128^3 closure). A lane holds the gradient of a quarter of its
// cell's moments at the end, so the certificate is decided here (as after_probe decides it)
// and a certified cell finished -- no probe entry, no Newton visit (3.2 of 13.6 ms per closure
// there); the rest is listed for the Newton kernel. e_min and e_max come from the high words of
// the values (rounded outwards by 2^-20: the certificate keeps factors of 2 and 4 in hand).
// Bound by the FP64 pipe (vector 39% + DMMA 28% busy) and the latency of its chains. M_6 64^3:
// 1.44 ms per closure (6.8 with all directions), M_4 0.73.
template <int NT, int NT2>
__global__ void __launch_bounds__(SYM_PROBE_WARPS * 32, 4)
    sym_probe_kernel(ClosureParams P, SymTables T, int n, double *__restrict__ out, int *errorFlag,
                     Outputs O, FirstRound first)
{
    constexpr int WARPS = SYM_PROBE_WARPS, DEG = sym_order(NT2), NMP = 8 * NT;
    using C = SymCls<DEG>;
    using G = SymStage<DEG, DEG>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    double *stage = reinterpret_cast<double *>(smem_raw);
    __shared__ uint64_t full[SYM_STAGES];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nm = P.nm;
    double *aF = stage + SYM_STAGES * G::DOUBLES + warp * C::STEPS * 32;
    if (tid == 0) {
        for (int s = 0; s < SYM_STAGES; ++s)
            mbar_init(&full[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        for (int b = 0; b < SYM_STAGES && b < T.nb; ++b)
            sym_stage_load<DEG, DEG>(T, b, stage, full);
    }
    const int pos = (blockIdx.x * WARPS + warp) * 8 + (lane >> 2);
    const bool emit = first.psi != nullptr;
    const bool valid = emit && first.psiValid && *first.psiValid != 0;
    long long gc = -1;
    double u0 = 1.0, ascale = 0.0;
    bool write = false;
    if (pos < n) {
        const long long c = first.off + pos;
        gc = first.cellMap ? first.cellMap[c] : c;
        u0 = first.u[gc * nm];
        ascale = log(u0) * 2.0 * sqrt(M_PI);
        write = emit;
        if (valid) {
            // only a face ghost's psi may be missing (its image's was read instead)
            const int gz = first.gnz + 4, gy = first.gny + 4;
            const int k = (int)(gc % gz), j = (int)((gc / gz) % gy), i = (int)(gc / gz / gy);
            write = (i >= 2 && i < first.gnx + 2) + (j >= 2 && j < first.gny + 2) +
                        (k >= 2 && k < first.gnz + 2) == 2;
        }
    }
    const bool any = __any_sync(FULL_MASK, gc >= 0);
    // the moments are read at the end: their lines come to L2 meanwhile
    if (gc >= 0)
        for (int i = 16 * (lane & 3); i < nm; i += 64)
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(first.u + gc * nm + i));
#pragma unroll
    for (int k = 0; k < C::STEPS; ++k) {
        const int m = T.stepIdx[4 * k + (lane & 3)];
        double a = gc >= 0 && m >= 0 ? first.alpha[gc * nm + m] : 0.0;
        if (m == 0)
            a -= ascale;
        aF[k * 32 + lane] = a;
    }
    double acc[C::TILES][2];
#pragma unroll
    for (int t = 0; t < C::TILES; ++t)
        acc[t][0] = acc[t][1] = 0.0;
    double f = 0.0;
    int lo = 0x7fffffff, hi = 0;
    __syncthreads();
    for (int b = 0; b < T.nb; ++b) {
        const double *st = stage + (b % SYM_STAGES) * G::DOUBLES;
        const bool ok = mbar_wait(&full[b % SYM_STAGES], (b / SYM_STAGES) & 1);
        if (any) {
            double v[2][8];
            sym_expand<DEG>(aF, st, lane, v);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                double *p = first.psi + ((long long)(8 * (2 * b + e)) * first.nall + gc) * 4 + (lane & 3);
                const bool w = write && 4 * (2 * b + e) < T.no; // a whole group past the end: no rows
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    v[e][s] = exp(v[e][s]);
                    if (w)
                        p[(long long)(4 * s) * first.nall] = u0 * v[e][s];
                }
            }
            const double2 w = *reinterpret_cast<const double2 *>(T.w + SYM_BLK * b + 2 * (lane & 3));
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (SYM_BLK * b + 4 * e + (lane & 3) < T.no)
#pragma unroll
                    for (int s = 0; s < 8; ++s) {
                        lo = min(lo, __double2hiint(v[e][s]));
                        hi = max(hi, __double2hiint(v[e][s]));
                    }
#pragma unroll
                for (int s = 0; s < 8; ++s)
                    v[e][s] *= e == 0 ? w.x : w.y;
                sym_wht(v[e]);
                f += v[e][0];
                sym_contract<DEG>(v[e], st + G::EXPO + e * (C::TILES * 32), lane, acc);
            }
        }
        refill_fence();
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicExch(errorFlag, 1);
                ring_drain<SYM_STAGES>(full, 0, b, T.nb);
            }
            return;
        }
        if (tid == 0 && b + SYM_STAGES < T.nb)
            sym_stage_load<DEG, DEG>(T, b + SYM_STAGES, stage, full);
    }
    f += __shfl_xor_sync(FULL_MASK, f, 1);
    f += __shfl_xor_sync(FULL_MASK, f, 2);
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        lo = min(lo, __shfl_xor_sync(FULL_MASK, lo, o));
        hi = max(hi, __shfl_xor_sync(FULL_MASK, hi, o));
    }
    // gradient of the scaled cell (H_i0 / m_0 - u_i = <m_i e^{alpha.m}> - u_i) and its stopping test,
    // short of the tolerance by what the roundings of the full visit's form may differ by
    __shared__ unsigned int sCertified;
    if (tid == 0)
        sCertified = 0;
    __syncthreads();
    double g2 = 0.0, u2 = 0.0, us[C::TILES][2];
    const double inv = 1.0 / u0;
#pragma unroll
    for (int t = 0; t < C::TILES; ++t)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int m = T.idx[8 * t + 2 * (lane & 3) + e];
            us[t][e] = gc >= 0 && m >= 0 ? first.u[gc * nm + m] : 0.0;
        }
#pragma unroll
    for (int t = 0; t < C::TILES; ++t)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            // (padding: 0 - 0, its projection fragments are 0)
            const double ui = us[t][e] * inv, gi = acc[t][e] - ui;
            g2 = fma(gi, gi, g2);
            u2 = fma(ui, ui, u2);
        }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        g2 += __shfl_xor_sync(FULL_MASK, g2, o);
        u2 += __shfl_xor_sync(FULL_MASK, u2, o);
    }
    const double err = sqrt(g2), emin = __hiloint2double(lo, 0), emax = __hiloint2double(hi, -1);
    const double rtol = P.batched ? P.tol : sqrt(u2) * P.tol;
    const int maxIter = P.batched && P.nreg == 1 ? 10 * P.maxIter : P.maxIter;
    const double lam = 0.5 * emin * P.gramLo, k1 = nm * (emax * P.gramHi) / lam;
    const double minf = sqrt((2 * (DEG + 2) + 1) / (2 * M_PI));
    const double gexp = 2.0 * minf * (DEG + 1) * err / lam;
    const bool done = gc >= 0 && u0 > 0.0 && err + P.certSlack <= rtol && maxIter > 1 && P.passBudget >= 1 &&
                      P.tolGamma > 1.0 && emin > 0.0 && emax < 1.0 / 0.0 && P.gramLo > 0.0 &&
                      k1 <= 0.25 * P.condHMax && gexp <= 0.5 * log(P.tolGamma);
    // one list position per cell that goes on, claimed per warp
    const unsigned goes = __ballot_sync(FULL_MASK, gc >= 0 && !done && (lane & 3) == 0);
    unsigned at = 0;
    if (lane == 0 && goes)
        at = atomicAdd(first.todoCount, (unsigned)__popc(goes));
    at = __shfl_sync(FULL_MASK, at, 0) + __popc(goes & ((1u << lane) - 1u));
    if (done) {
        // finalize (closure_core.cuh) of a cell converged in its first iteration
#pragma unroll
        for (int t = 0; t < C::TILES; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int m = T.idx[8 * t + 2 * (lane & 3) + e];
                if (m >= 0)
                    O.u[gc * nm + m] = us[t][e] / u0 * u0;
            }
        if ((lane & 3) == 0) {
            O.alpha[gc * nm] = first.alpha[gc * nm] - ascale + ascale;
            if (O.iters) O.iters[gc] = 1;
            if (O.iterGamma) O.iterGamma[gc] = 0;
            if (O.regIdx) O.regIdx[gc] = 0;
            if (O.status) O.status[gc] = CELL_OK;
            if (O.gamma) O.gamma[gc] = exp(gexp);
            if (O.normG) O.normG[gc] = err;
            if (O.cond) O.cond[gc] = (float)k1;
            atomicAdd(&sCertified, 1u);
        }
    } else if (gc >= 0) {
        double *o = out + (size_t)pos * probe_entry_doubles(NMP);
#pragma unroll
        for (int t = 0; t < C::TILES; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int m = T.idx[8 * t + 2 * (lane & 3) + e];
                if (m >= 0)
                    o[m] = acc[t][e];
            }
        if ((lane & 3) == 0) {
            o[NMP] = f;
            o[NMP + 1] = emin;
            o[NMP + 2] = emax;
            first.todo[at] = pos;
        }
    }
    __syncthreads();
    if (tid == 0 && O.stats && sCertified) {
        const unsigned long long c = sCertified;
        atomicAdd(&O.stats[STAT_CELLS], c);
        atomicAdd(&O.stats[STAT_ITERS], c);
        atomicMax(&O.stats[STAT_MAX_ITER], 1ull);
        atomicAdd(&O.stats[STAT_REG_HIST], c);
        atomicAdd(&O.stats[STAT_ITER_HIST + 1], c);
        atomicAdd(&O.stats[STAT_CERTIFIED], c);
    }
}

// Newton logic for the listed cells: cell_lanes(NT) lanes per cell, state staged
// in shared memory with H in the tiled layout (TSlot).
// MODE 0: FP64 Hessians and trials. MODE 1: the list of a mixed-precision pass (entries of
// mix_entry_doubles): H from the reduced-precision moments, g and f from the pass's FP64
// moments; a visit whose moments are not all finite is redone in FP64. MODE 2: first visits
// after the probe pass (entries of probe_entry_doubles; g0: the Gaunt terms of H's column 0,
// g0n per row, null in the mixed closure), no Hessian. level: the list (0 FP64 and trials,
// 1 BF16, 2 3xTF32, 3 probe).
// GAUNT: the CTA assembles H_ij = sum_k beta_ijk mom_k (i >= j, the CSR terms of beta in
// the order of src/opt/fobj.cpp:81-99, laid out per tile slot by c3d_set_gaunt) for its
// cells that need a Hessian in one sweep over the tile slots per four cells. The cells' moments
// sit in the slots' g..rinv vectors, which a Hessian visit recomputes afterwards. Otherwise the pass
// wrote H in tiles to hBuf. fused: the symmetric passes' list 0 (moments at trial points, bounds of
// e^{alpha.m} behind the moments).
template <int NT, int NT2, bool GAUNT, int MODE>
__global__ void __launch_bounds__(NEWTON_THREADS)
    rounds_newton_kernel(ClosureParams P, double m0, const int *__restrict__ list, int n,
                         const unsigned int *nDev, CellState<NT> *state,
                         const double *__restrict__ buf,
                         const GauntTerm *__restrict__ stream, int streamLen,
                         Outputs Og, Lists out, int level, const GauntTerm *__restrict__ g0,
                         int g0n, FirstRound first, bool fused)
{
    constexpr int W = cell_lanes(NT), CELLS = newton_cells(NT);
    n = round_entries(n, MODE == 2 && first.todo ? first.todoCount : nDev);
    if (blockIdx.x * CELLS >= n)
        return;
    constexpr bool MIX = MODE == 1;
    constexpr int NM2P = 8 * NT2;
    constexpr int NMP = Cfg<NT>::NMP;
    constexpr int BSTR = MODE == 1 ? mix_entry_doubles(NMP, NM2P)
                                   : MODE == 2 ? probe_entry_doubles(NMP) : NM2P;
    constexpr int LS = TSlot<NT>::LSIZE;
    static_assert(!GAUNT || NM2P <= 4 * NMP, "moments must fit in g, d, alphaOld, rinv");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    using SlotT = NewtonSlot<NT, MODE>;
    SlotT *slots = reinterpret_cast<SlotT *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & (W - 1), ci = tid / W; // ci: the CTA's cell
    // the CTA's closure counters, added to the context's once at the end (one global atomic
    // per counter and CTA instead of several per finished cell)
    __shared__ unsigned long long sStat[STAT_COUNT];
    for (int q = tid; q < STAT_COUNT; q += NEWTON_THREADS)
        sStat[q] = 0;
    __syncthreads();
    Outputs O = Og;
    if (Og.stats)
        O.stats = sStat;
    // (a probe's list is walked by a grid smaller than the worst case)
    int blk = blockIdx.x;
    do {
    const bool active = blk * CELLS + ci < n;
    const int pos = MODE == 2 && active && first.todo ? first.todo[blk * CELLS + ci] : blk * CELLS + ci;
    const long long cell = active ? (list ? list[pos] : first.off + pos) : -1;
    bool needH = false;
    SlotT &sl = slots[ci];
    // probe visits: the probe entry's loads go out before the cell's state is read, so the
    // two global round trips overlap
    constexpr int PMR = (BSTR + W - 1) / W;
    double pmr[PMR];
    // Hessian and trial visits: the moments' loads go out first too, beside the list's and the
    // state's, whether or not the visit will want them (Newton kernel of M_4 64^3 7.99 -> 7.47 ms, of
    // M_3 and M_5 cells 3 to 7% faster, of order 7 2.95 -> 2.75 ms)
    constexpr int MMR = GAUNT && MODE != 2 ? (NM2P + W - 1) / W : 0;
    double mmr[MMR > 0 ? MMR : 1];
#pragma unroll
    for (int r = 0; r < MMR; ++r)
        mmr[r] = active && lane + W * r < NM2P ? buf[(size_t)pos * BSTR + lane + W * r] : 0.0;
    if constexpr (MODE == 2)
        if (active)
#pragma unroll
            for (int r = 0; r < PMR; ++r)
                pmr[r] = lane + W * r < BSTR ? buf[(size_t)pos * BSTR + lane + W * r] : 0.0;
    C3D_NCLK_DECL
    long long gcell = -1; // probe visits: the grid cell, for the ansatz hand-off's marks
    if (MODE == 2 && active && first.mark)
        gcell = !list ? (first.cellMap ? (long long)first.cellMap[cell] : cell) : state[cell].s.cell;
    if (active) {
        if (MODE == 2 && !list)
            load_cell(sl, P, O, first.cellMap ? (long long)first.cellMap[cell] : cell, lane);
        else
            state_to_slot(state[cell], sl, lane, MODE != 2);
        needH = MODE != 2 && sl.s.need == NEED_H;
    } else if (lane == 0) {
        sl.s.need = NEED_NONE;
    }
    bool nonFinite = false;
    // Trials come first. Fused: the pass also formed the moments at the trial point, so an
    // accepted trial goes on to the next iteration's Hessian visit here (unless that iteration
    // regularised, which moves the multipliers).
    bool tried = false;
    if constexpr (MODE == 0 && GAUNT) {
        if (active && !needH && sl.s.need == NEED_TRIAL) {
            tried = true;
            const bool moments = fused && trial_fused(P, sl.s.fp64, sl.s.iter, sl.s.cnd);
            const int reg = sl.s.regIndex;
            const bool accepted = after_trial(sl, P, O, lane, sl.s.fquad);
            needH = accepted && moments && sl.s.need == NEED_H && sl.s.regIndex == reg;
            if (!needH) {
                // on to another pass (or finished): stored before the assembly takes the scratch
                if (sl.s.need != NEED_NONE)
                    slot_to_state(sl, state[cell], lane);
                append_if_needed(sl, P, cell, lane, out);
            }
        }
    }
    if constexpr (MODE == 2) {
    } else if (GAUNT) {
        if (__syncthreads_or(needH)) {
            // The moments of each four cells, cells innermost, so that a term's loads for them are
            // two 16-byte accesses: moment k of cell w of the four at offset 4 (k / 4) + w of slot
            // k % 4's scratch (g, d, alphaOld, rinv: NM2P <= 4 NMP doubles). Slots whose cell
            // needs no Hessian hold nothing in theirs any more.
            static_assert(CELLS % 4 == 0, "moment layout");
            bool nf = false;
#pragma unroll
            for (int r = 0; r < MMR; ++r) {
                const int k = lane + W * r;
                const double v = needH ? mmr[r] : 0.0;
                nf |= MIX && !isfinite(v);
                if (k < NM2P)
                    slots[(ci & ~3) + (k & 3)].scratch()[(k & ~3) + (ci & 3)] = v;
            }
            nonFinite = cell_any<SlotT>(nf);
            // identity padding: the last tile row's rows past nm
            if (needH) {
                constexpr int T = NT;
                for (int e = lane; e < 32 * T; e += W)
                    *reinterpret_cast<double2 *>(&sl.L[64 * tix(T - 1, 0) + 2 * e]) =
                        make_double2(0.0, 0.0);
                cell_sync<SlotT>();
                if (lane < 8 && 8 * (T - 1) + lane >= P.nm)
                    sl.L[64 * tix(T - 1, T - 1) + toff(lane, lane)] = 1.0;
            }
            __shared__ int sNeedH[CELLS];
            if (lane == 0)
                sNeedH[ci] = needH;
            __syncthreads();
#pragma unroll 1
            for (int c4 = 0; c4 < CELLS; c4 += 4) {
                bool hw[4], any = false;
#pragma unroll
                for (int w = 0; w < 4; ++w)
                    any |= hw[w] = sNeedH[c4 + w] != 0;
                if (!any)
                    continue;
                double h[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
                for (int k = 0; k < streamLen; ++k) {
                    const GauntTerm gt = stream[k * NEWTON_THREADS + tid];
                    const double *m = slots[c4 + (gt.col & 3)].scratch() + (gt.col & ~3);
                    const double2 m01 = *reinterpret_cast<const double2 *>(m);
                    const double2 m23 = *reinterpret_cast<const double2 *>(m + 2);
                    h[0] = __dadd_rn(h[0], __dmul_rn(m01.x, gt.v));
                    h[1] = __dadd_rn(h[1], __dmul_rn(m01.y, gt.v));
                    h[2] = __dadd_rn(h[2], __dmul_rn(m23.x, gt.v));
                    h[3] = __dadd_rn(h[3], __dmul_rn(m23.y, gt.v));
                    if (gt.slot >= 0) {
#pragma unroll
                        for (int w = 0; w < 4; ++w) {
                            if (hw[w])
                                slots[c4 + w].L[gt.slot] = h[w];
                            h[w] = 0.0;
                        }
                    }
                }
            }
        }
        __syncthreads();
    } else if (needH) {
        const double2 *H = reinterpret_cast<const double2 *>(buf + (size_t)pos * LS);
        double2 *L = reinterpret_cast<double2 *>(sl.L);
        for (int e = lane; e < LS / 2; e += W)
            L[e] = H[e];
        cell_sync<SlotT>();
    }
    // (not fused, symmetric closure: the list of cells far out)
    if (MODE == 0 && GAUNT && P.sym && !fused && active && lane == 0 && O.stats)
        atomicAdd(&O.stats[STAT_FULL_ORDER], 1ull);
    if (active && !(tried && !needH)) {
    C3D_NCLK(O.stats, 0, lane);
    if constexpr (MODE == 2) {
        if (sl.s.need == NEED_PROBE) {
#pragma unroll
            for (int r = 0; r < PMR; ++r)
                if (lane + W * r < BSTR)
                    sl.pm[lane + W * r] = pmr[r];
            cell_sync<SlotT>();
            after_probe(sl, P, O, lane, m0, sl.pm, g0, g0n);
        }
    } else if (needH) {
        if (lane == 0) {
            sl.s.hprec = MIX ? level : 0;
            if (P.mixed && O.stats)
                atomicAdd(&O.stats[level == 1   ? STAT_H_BF16
                                   : level == 2 ? STAT_H_TF32X3
                                                : STAT_H_FP64],
                          1ull);
        }
        if constexpr (MIX) {
            if (nonFinite) {
                escalate_fp64(sl, O, lane);
            } else {
                const double *e = buf + (size_t)pos * BSTR + NM2P;
                after_hessian(sl, P, O, lane, m0, e, e[NMP]);
            }
        } else {
            double emin = 0.0, emax = 0.0;
            if constexpr (GAUNT)
                if (fused) { // the symmetric pass left its bounds behind the moments
                    const double *e = buf + (size_t)pos * BSTR +
                                      (2 * sym_order(NT2) + 1) * (2 * sym_order(NT2) + 1);
                    emin = e[0];
                    emax = e[1];
                }
            after_hessian(sl, P, O, lane, m0, nullptr, 0.0, emin, emax);
        }
        C3D_NCLK(O.stats, 5, lane);
    } else if (sl.s.need == NEED_TRIAL) {
        after_trial(sl, P, O, lane, sl.s.fquad);
        C3D_NCLK(O.stats, 7, lane);
    }
    if constexpr (MODE == 2) {
        // a cell that goes on past its probe visit (or failed there) may end with other
        // multipliers than the probe's: its psi is rewritten after the closure
        if (gcell >= 0 && lane == 0 && (sl.s.need != NEED_NONE || sl.s.status != CELL_OK))
            first.mark[gcell] = 1;
    }
    // a finished cell's state is not read again
    if (sl.s.need != NEED_NONE)
        slot_to_state(sl, state[cell], lane);
    append_if_needed(sl, P, cell, lane, out);
    C3D_NCLK(O.stats, 6, lane);
    }
    __syncthreads();
    } while (MODE == 2 && (blk += gridDim.x) * CELLS < n);
    if (Og.stats)
        for (int q = tid; q < STAT_COUNT; q += NEWTON_THREADS) {
            const unsigned long long v = sStat[q];
            if (v == 0)
                continue;
            if (q == STAT_MAX_ITER || q == STAT_MAX_ITER_GAMMA)
                atomicMax(&Og.stats[q], v);
            else
                atomicAdd(&Og.stats[q], v);
        }
}

// ---------------------------------------------------------------- host side
//
// The file is compiled once per C3D_ROUNDS_PART (Makefile): part 0 holds the shared host code and
// the dispatch, the other parts each instantiate rounds_t for a few orders, so that the
// orders compile in parallel.

#if C3D_ROUNDS_PART == 0
template <int NT> static size_t state_bytes_t() { return sizeof(CellState<NT>); }

size_t rounds_state_bytes(int nm)
{
    switch ((nm + 7) / 8) {
    case 1: return state_bytes_t<1>();
    case 2: return state_bytes_t<2>();
    case 3: return state_bytes_t<3>();
    case 4: return state_bytes_t<4>();
    case 5: return state_bytes_t<5>();
    case 6: return state_bytes_t<6>();
    case 7: return state_bytes_t<7>();
    default: return state_bytes_t<8>();
    }
}

// Doubles per list entry of the pass output buffer.
size_t rounds_buf_doubles(int nm, int nm2, bool gaunt, bool mixed)
{
    const int nt = (nm + 7) / 8;
    if (gaunt) {
        const int nm2p = 8 * ((nm2 + 7) / 8);
        const size_t e = (size_t)(mixed ? mix_entry_doubles(8 * nt, nm2p) : nm2p);
        const size_t pr = (size_t)probe_entry_doubles(8 * nt);
        return e > pr ? e : pr;
    }
    return (size_t)64 * nt * (nt + 1) / 2; // the tiled lower triangle
}

// Bytes of one staged chunk of the mixed pass's A operand (format 0 BF16, 1 TF32 hi + lo).
size_t mixed_a_chunk_bytes(int nm2, int fmt)
{
    const int nm2p = 8 * ((nm2 + 7) / 8);
    const int na = nm2p < 128 ? 128 : nm2p;
    return (size_t)na * QC * (fmt == 0 ? 2 : 8);
}
#endif

template <int NT, int KIND, bool ZD> static size_t mixed_pass_smem(const ClosureParams &P, int nm2)
{
    using K = MixKind<KIND>;
    const size_t f64Pad = ((size_t)(P.nm + 1) * QCP * 8 + 127) & ~(size_t)127;
    const size_t stg = f64Pad + (KIND < 2 ? mixed_a_chunk_bytes(nm2, KIND) : 0);
    return GSTAGES * stg + GSTAGES * (size_t)K::NP * MXC * QC * K::ES + (size_t)QC * CST2 * 8 +
           (size_t)RW * P.nm * 16 + (ZD ? (size_t)QC * ZS * 8 : 0) +
           (KIND == 2 ? (size_t)QC * PSTR * 8 + MXC * 8 : 0) +
           (KIND == 2 && ZD ? (size_t)PRS * QC * PSTR * 8 : 0) + (2 * GSTAGES + 1) * 8;
}

// ---------------------------------------------------------------- graph-resident round loop
//
// A closure is one CUDA graph: round 0 (set-up, or the certificate's probe round) then a
// conditional WHILE node whose body runs two rounds (lists A -> B, then B -> A) and sets the
// loop condition on the device, so no round waits for the host. Within a round, each list's
// pass and Newton kernels sit in a SWITCH node whose branch -- one of up to four launch sizes
// (up to 512, 8192, 65536 and `cap` entries) or none for an empty list -- a control kernel
// picks from the list's device counter; entries past `cap` are carried to the next round's
// list. The kernels read their entry count from the counter (round_entries).

// A list whose launches are all below a size has no branch above it (a graph's build takes
// about 25 us per kernel node, most of a new state's first step: M_2 16^3, 8000 cells, has 2
// branches per list), and the rare list of cells in the reference's order has 8192 and cap only.
constexpr int NTIER = 4;
__host__ __device__ inline long long tier_entries(int t, long long cap, bool rare)
{
    const long long t0 = rare ? (t == 0 ? 8192 : cap) : t == 0 ? 512 : t == 1 ? 8192 : 65536;
    return t < 3 && t0 < cap ? t0 : cap;
}
__host__ __device__ inline int tier_count(long long cap, bool rare)
{
    int n = 1;
    while (tier_entries(n - 1, cap, rare) < cap)
        ++n;
    return n;
}

struct TierHandles {
    cudaGraphConditionalHandle h[NLISTS];
};

#if C3D_ROUNDS_PART != 0
// Picks each used list's launch size (SWITCH branch; NTIER = none) from its counter (bit l of
// mask marks list l as used, of rare as a rare one) and clears the counters of the lists the
// round fills.
static __global__ void rounds_tier_kernel(const Lists in, Lists out, TierHandles th, unsigned int mask,
                                   unsigned int rare, long long cap, unsigned long long *launches)
{
    if (threadIdx.x != 0)
        return;
    for (int l = 0; l < NLISTS; ++l)
        *out.count[l] = 0;
    unsigned long long l2 = 1;
    for (int l = 0; l < NLISTS; ++l) {
        if (!((mask >> l) & 1u))
            continue;
        const long long c = (long long)*in.count[l];
        const bool ra = (rare >> l) & 1u;
        const int last = tier_count(cap, ra) - 1;
        int t = NTIER;
        for (int k = last; k >= 0; --k)
            if (c > 0 && c <= tier_entries(k, cap, ra))
                t = k;
        if (c > cap)
            t = last;
        cudaGraphSetConditional(th.h[l], (unsigned int)t);
        l2 += t < NTIER ? 2 : 0;
    }
    if (launches)
        atomicAdd(launches, l2);
}

// Entries past cap stay for the next round: appended to that round's list.
static __global__ void rounds_carry_kernel(const Lists in, Lists out, unsigned int mask, long long cap)
{
    __shared__ unsigned int base[NLISTS];
    for (int l = 0; l < NLISTS; ++l) {
        if (!((mask >> l) & 1u))
            continue;
        const long long c = (long long)*in.count[l];
        if (c <= cap)
            continue; // uniform over the block
        if (threadIdx.x == 0)
            base[l] = atomicAdd(out.count[l], (unsigned int)(c - cap));
        __syncthreads();
        for (long long i = cap + threadIdx.x; i < c; i += blockDim.x)
            out.list[l][base[l] + (i - cap)] = in.list[l][i];
        __syncthreads();
    }
}

// Loop condition after the body's two rounds: more work and the round limit not reached;
// past the limit the closure stops with errorFlag 2 (c3d_sync: C3D_ERR_TIMEOUT).
static __global__ void rounds_cond_kernel(const Lists in, unsigned int mask, unsigned int *rounds,
                                   long long maxRounds, int *errorFlag,
                                   cudaGraphConditionalHandle loop, unsigned long long *launches)
{
    if (threadIdx.x != 0)
        return;
    unsigned long long total = 0;
    for (int l = 0; l < NLISTS; ++l)
        if ((mask >> l) & 1u)
            total += *in.count[l];
    const unsigned int r = *rounds + 2;
    *rounds = r;
    bool more = total > 0;
    if (more && (long long)r >= maxRounds) {
        atomicExch(errorFlag, 2);
        more = false;
    }
    cudaGraphSetConditional(loop, more ? 1u : 0u);
    if (launches)
        atomicAdd(launches, 1ull);
}
#else
// Appends a conditional node after the current dependencies of the graph being captured on st.
cudaError_t capture_conditional(cudaStream_t st, cudaGraphConditionalHandle h,
                                       cudaGraphConditionalNodeType type, unsigned int size,
                                       cudaGraph_t **bodies)
{
    cudaStreamCaptureStatus status;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t *deps = nullptr;
    size_t ndeps = 0;
    cudaError_t e = cudaStreamGetCaptureInfo(st, &status, nullptr, &g, &deps, &ndeps);
    if (e != cudaSuccess)
        return e;
    if (status != cudaStreamCaptureStatusActive)
        return cudaErrorStreamCaptureInvalidated;
    cudaGraphNodeParams p = {};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = type;
    p.conditional.size = size;
    cudaGraphNode_t node;
    e = cudaGraphAddNode(&node, g, deps, ndeps, &p);
    if (e != cudaSuccess)
        return e;
    e = cudaStreamUpdateCaptureDependencies(st, &node, 1, cudaStreamSetCaptureDependencies);
    *bodies = p.conditional.phGraph_out;
    return e;
}

// Graph capture and instantiation run one thread at a time in the process (contexts driven
// from several host threads, as the serving loop does, build their graphs in turn; launches of
// built graphs do not wait).
std::mutex &graph_build_mutex()
{
    static std::mutex m;
    return m;
}
#endif

// The instantiated closure graphs of the last few configurations (a configuration is every
// launch parameter; switching, e.g., between precisions reuses its graph), with the streams
// their capture uses.
struct RoundsGraph {
    static constexpr int SLOTS = 6;
    struct Slot {
        std::vector<unsigned char> key;
        cudaGraphExec_t exec = nullptr;
        unsigned long long used = 0;
    } slot[SLOTS];
    unsigned long long tick = 0;
    cudaStream_t cs[3] = {nullptr, nullptr, nullptr};
    ~RoundsGraph()
    {
        for (Slot &s : slot)
            if (s.exec)
                cudaGraphExecDestroy(s.exec);
        for (cudaStream_t s : cs)
            if (s)
                cudaStreamDestroy(s);
    }
};

template <class T> static void key_add(std::vector<unsigned char> &k, const T &v)
{
    const unsigned char *b = reinterpret_cast<const unsigned char *>(&v);
    k.insert(k.end(), b, b + sizeof(T));
}

#if C3D_ROUNDS_PART == 0
std::vector<unsigned char> rounds_graph_key(const RoundsLaunch &R, bool gaunt)
{
    std::vector<unsigned char> k;
    key_add(k, *R.P);
    const void *ptrs[] = {R.chunks, R.gstream, R.cellMap, R.u, R.alpha, R.iters, R.iterGamma,
                          R.regIdx, R.status, R.failCount, R.stats, R.gamma, R.normG, R.cond,
                          R.state, R.listA, R.listB, R.counts, R.buf, R.mixF64, R.mixA[0],
                          R.mixA[1], R.g0, R.errorFlag, R.psi, R.mark, R.launchDev,
                          R.symN.expo, R.sym2.expo};
    for (const void *p : ptrs)
        key_add(k, p);
    key_add(k, R.nm2);
    key_add(k, R.streamLen);
    key_add(k, R.m0);
    key_add(k, R.ncells);
    key_add(k, R.batch);
    key_add(k, R.g0n);
    key_add(k, R.psiNall);
    key_add(k, R.maxRounds);
    key_add(k, gaunt);
    return k;
}
#endif

#if C3D_ROUNDS_PART != 0
template <int NT, int NT2, bool GAUNT> cudaError_t rounds_t(const RoundsLaunch &R)
{
    const ClosureParams &P = *R.P;
    CellState<NT> *state = reinterpret_cast<CellState<NT> *>(R.state);
    cudaStream_t st = R.stream;
    const bool mixed = GAUNT && P.mixed;
    cudaError_t e;
    size_t slotSmem = RW * sizeof(Slot<NT>);
    e = cudaFuncSetAttribute(rounds_init_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)slotSmem);
    if (e != cudaSuccess)
        return e;
    size_t newtonSmem = newton_cells(NT) * sizeof(TSlot<NT>);
    e = cudaFuncSetAttribute(rounds_newton_kernel<NT, NT2, GAUNT, 0>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)newtonSmem);
    if (e != cudaSuccess)
        return e;
    const bool probe = GAUNT && P.probe;
    const size_t probeSmem = newton_cells(NT) * sizeof(ProbeSlot<NT>);
    size_t passSmem, mixSmem[3] = {0, 0, 0};
    // octant-symmetric quadrature: the passes of sym.cuh
    const bool sym = GAUNT && P.sym;
    constexpr int DEG = sym_order(NT2);
    constexpr size_t symPassSmem = sym_smem<DEG, 2 * DEG, SYM_PASS_WARPS>(),
                     symProbeSmem = sym_smem<DEG, DEG, SYM_PROBE_WARPS>();
    if constexpr (GAUNT) {
        if (sym) {
            e = cudaFuncSetAttribute(sym_pass_kernel<NT, NT2>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)symPassSmem);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(sym_probe_kernel<NT, NT2>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)symProbeSmem);
            if (e != cudaSuccess)
                return e;
        }
        passSmem = GSTAGES * (size_t)(R.nm2 + 1) * QCP * 8 + (size_t)QC * CST2 * 8 +
                   (size_t)(RWP * P.nm + 1) * 8 + GSTAGES * 8;
        e = cudaFuncSetAttribute(rounds_pass_gaunt_kernel<NT, NT2>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)passSmem);
        if (e == cudaSuccess && probe) {
            e = cudaFuncSetAttribute(rounds_newton_kernel<NT, NT2, GAUNT, 2>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)probeSmem);
            mixSmem[2] = mixed ? mixed_pass_smem<NT, 2, true>(P, R.nm2)
                               : mixed_pass_smem<NT, 2, false>(P, R.nm2);
            if (e == cudaSuccess)
                e = mixed ? cudaFuncSetAttribute(rounds_pass_mixed_kernel<NT, NT2, 2, true>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)mixSmem[2])
                          : cudaFuncSetAttribute(rounds_pass_mixed_kernel<NT, NT2, 2, false>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)mixSmem[2]);
        }
        if (e == cudaSuccess && mixed) {
            e = cudaFuncSetAttribute(rounds_newton_kernel<NT, NT2, GAUNT, 1>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)newtonSmem);
            mixSmem[0] = mixed_pass_smem<NT, 0, true>(P, R.nm2);
            mixSmem[1] = mixed_pass_smem<NT, 1, true>(P, R.nm2);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(rounds_pass_mixed_kernel<NT, NT2, 0, true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)mixSmem[0]);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(rounds_pass_mixed_kernel<NT, NT2, 1, true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)mixSmem[1]);
        }
    } else {
        passSmem = 3 * (size_t)Cfg<NT>::CHUNK * 8 + (size_t)RW * Cfg<NT>::NMP * 8 + 3 * 8;
        e = cudaFuncSetAttribute(rounds_pass_direct_kernel<NT>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)passSmem);
    }
    if (e != cudaSuccess)
        return e;
    const double m0 = R.m0;
    const Outputs O{R.u,      R.alpha,     R.iters, R.iterGamma, R.regIdx,
                    R.status, R.failCount, R.stats, R.gamma,     R.normG, R.cond};

    Lists A, B;
    for (int l = 0; l < NLISTS; ++l) {
        A.list[l] = R.listA + (size_t)l * R.ncells;
        B.list[l] = R.listB + (size_t)l * R.ncells;
        A.count[l] = R.counts + l;
        B.count[l] = R.counts + NLISTS + l;
    }
    // the lists the graph's rounds can fill: FP64 Hessian passes and, when the mixed closure
    // routes any visit to reduced precision, its BF16 and 3xTF32 ones (probe passes happen in
    // round 0 only: no later visit is a first visit)
    const unsigned int usedLists = 1u | (mixed && P.mixIterMax > 0 ? 6u : 0u) | (sym ? 8u : 0u);
    const unsigned int rareLists = sym ? 8u : 0u;

    // pass + Newton kernels of list l: entries la[0 .. nb) (with nDev, at most *nDev of them),
    // the cells still in need appended to out
    auto launch_list = [&](int l, const int *la, int nb, const unsigned int *nDev, const Lists &out,
                           cudaStream_t s) {
        if (l == 3 && sym) {
            // the reference's order for cells far out
            if constexpr (GAUNT) {
                rounds_pass_gaunt_kernel<NT, NT2>
                    <<<(unsigned)((nb + RWP - 1) / RWP), RW * 32, passSmem, s>>>(
                        P, R.chunks, R.nm2, la, nb, nDev, state, R.buf, R.errorFlag);
                rounds_newton_kernel<NT, NT2, GAUNT, 0>
                    <<<(unsigned)((nb + newton_cells(NT) - 1) / newton_cells(NT)), NEWTON_THREADS,
                       newtonSmem, s>>>(P, m0, la, nb, nDev, state, R.buf, R.gstream, R.streamLen, O,
                                        out, 0, nullptr, 0, FirstRound{}, false);
            }
        } else if (l == 3) {
            // probe passes of first visits (Gaunt form only)
            if constexpr (GAUNT) {
                const unsigned grid = (unsigned)((nb + MXC - 1) / MXC);
                if (mixed)
                    rounds_pass_mixed_kernel<NT, NT2, 2, true><<<grid, RW * 32, mixSmem[2], s>>>(
                        P, R.mixF64, nullptr, la, nb, nDev, state, R.buf, R.errorFlag,
                        FirstRound{});
                else
                    rounds_pass_mixed_kernel<NT, NT2, 2, false><<<grid, RW * 32, mixSmem[2], s>>>(
                        P, R.mixF64, nullptr, la, nb, nDev, state, R.buf, R.errorFlag,
                        FirstRound{});
                rounds_newton_kernel<NT, NT2, GAUNT, 2>
                    <<<(unsigned)((nb + newton_cells(NT) - 1) / newton_cells(NT)), NEWTON_THREADS, probeSmem, s>>>(
                        P, m0, la, nb, nDev, state, R.buf, R.gstream, R.streamLen, O, out, l,
                        mixed ? nullptr : R.g0, R.g0n, FirstRound{}, false);
            }
        } else if (l > 0) {
            // mixed-precision Hessian passes (Gaunt form only)
            if constexpr (GAUNT) {
                const unsigned grid = (unsigned)((nb + MXC - 1) / MXC);
                if (l == 1)
                    rounds_pass_mixed_kernel<NT, NT2, 0, true><<<grid, RW * 32, mixSmem[0], s>>>(
                        P, R.mixF64, R.mixA[0], la, nb, nDev, state, R.buf, R.errorFlag,
                        FirstRound{});
                else
                    rounds_pass_mixed_kernel<NT, NT2, 1, true><<<grid, RW * 32, mixSmem[1], s>>>(
                        P, R.mixF64, R.mixA[1], la, nb, nDev, state, R.buf, R.errorFlag,
                        FirstRound{});
                rounds_newton_kernel<NT, NT2, GAUNT, 1>
                    <<<(unsigned)((nb + newton_cells(NT) - 1) / newton_cells(NT)), NEWTON_THREADS, newtonSmem, s>>>(
                        P, m0, la, nb, nDev, state, R.buf, R.gstream, R.streamLen, O, out, l,
                        nullptr, 0, FirstRound{}, false);
            }
        } else {
            if constexpr (GAUNT) {
                constexpr int per = 8 * SYM_PASS_WARPS;
                if (sym)
                    sym_pass_kernel<NT, NT2>
                        <<<(unsigned)((nb + per - 1) / per), SYM_PASS_WARPS * 32, symPassSmem, s>>>(
                            P, R.sym2, la, nb, nDev, state, R.buf, R.errorFlag);
                else
                    rounds_pass_gaunt_kernel<NT, NT2>
                        <<<(unsigned)((nb + RWP - 1) / RWP), RW * 32, passSmem, s>>>(
                            P, R.chunks, R.nm2, la, nb, nDev, state, R.buf, R.errorFlag);
            } else
                rounds_pass_direct_kernel<NT>
                    <<<(unsigned)((nb + RW - 1) / RW), RW * 32, passSmem, s>>>(
                        P, R.chunks, la, nb, nDev, state, R.buf, R.errorFlag);
            rounds_newton_kernel<NT, NT2, GAUNT, 0>
                <<<(unsigned)((nb + newton_cells(NT) - 1) / newton_cells(NT)), NEWTON_THREADS, newtonSmem, s>>>(
                    P, m0, la, nb, nDev, state, R.buf, R.gstream, R.streamLen, O, out, 0, nullptr,
                    0, FirstRound{}, sym);
        }
        return cudaGetLastError();
    };

    // round 0: set-up of every cell (with the certificate: set-up and probe pass in one round)
    auto round0 = [&](cudaStream_t s) -> cudaError_t {
        // the lists' counters, the round counter and the probe's list
        cudaError_t e0 = cudaMemsetAsync(R.counts, 0, (2 * NLISTS + 2) * sizeof(unsigned int), s);
        if (e0 != cudaSuccess)
            return e0;
        if (probe) {
            if constexpr (GAUNT) {
                for (long long off = 0; off < R.ncells; off += R.batch) {
                    const int nb = (int)((R.ncells - off) < R.batch ? (R.ncells - off) : R.batch);
                    const FirstRound fr{off,       R.cellMap,      R.u,      R.alpha,
                                        R.psi,     R.psiNall,      R.mark,
                                        R.psiValid, R.gnx,         R.gny,    R.gnz,
                                        sym ? B.list[3] : nullptr, sym ? R.counts + 2 * NLISTS + 1 : nullptr};
                    const unsigned grid = (unsigned)((nb + MXC - 1) / MXC);
                    constexpr int per = 8 * SYM_PROBE_WARPS;
                    const unsigned gridS = (unsigned)((nb + per - 1) / per);
                    if (sym && off > 0 && (e0 = cudaMemsetAsync(fr.todoCount, 0, sizeof(unsigned int), s)) != cudaSuccess)
                        return e0;
                    if (sym)
                        sym_probe_kernel<NT, NT2><<<gridS, SYM_PROBE_WARPS * 32, symProbeSmem, s>>>(
                            P, R.symN, nb, R.buf, R.errorFlag, O, fr);
                    else if (mixed)
                        rounds_pass_mixed_kernel<NT, NT2, 2, true><<<grid, RW * 32, mixSmem[2], s>>>(
                            P, R.mixF64, nullptr, nullptr, nb, nullptr, state, R.buf, R.errorFlag,
                            fr);
                    else
                        rounds_pass_mixed_kernel<NT, NT2, 2, false><<<grid, RW * 32, mixSmem[2], s>>>(
                            P, R.mixF64, nullptr, nullptr, nb, nullptr, state, R.buf, R.errorFlag,
                            fr);
                    const unsigned gridN = (unsigned)((nb + newton_cells(NT) - 1) / newton_cells(NT));
                    rounds_newton_kernel<NT, NT2, GAUNT, 2>
                        <<<sym && gridN > PROBE_GRID ? PROBE_GRID : gridN, NEWTON_THREADS, probeSmem, s>>>(
                            P, m0, nullptr, nb, nullptr, state, R.buf, R.gstream, R.streamLen, O,
                            A, 3, mixed ? nullptr : R.g0, R.g0n, fr, false);
                    *R.launches += 2;
                }
            }
        } else {
            rounds_init_kernel<NT><<<(unsigned)((R.ncells + RW - 1) / RW), RW * 32, slotSmem, s>>>(
                P, R.ncells, R.cellMap, O, state, A);
            *R.launches += 1;
        }
        return cudaGetLastError();
    };

    // Appends the closure to the graph being captured on cs[0] (top: that capture's top-level
    // graph, which owns the conditional handles); cs[1], cs[2] capture the loop and switch
    // bodies.
    auto capture_into = [&](cudaGraph_t top, cudaStream_t const *cs) -> cudaError_t {
        const long long cap = R.batch;
        cudaGraphConditionalHandle hLoop;
        TierHandles th[2];
        cudaError_t ec = cudaGraphConditionalHandleCreate(&hLoop, top, 1, cudaGraphCondAssignDefault);
        // one handle per SWITCH node the graph has (a handle without its node makes the
        // graph invalid)
        for (int hr = 0; hr < 2 && ec == cudaSuccess; ++hr)
            for (int l = 0; l < NLISTS && ec == cudaSuccess; ++l)
                if ((usedLists >> l) & 1u)
                    ec = cudaGraphConditionalHandleCreate(&th[hr].h[l], top, NTIER,
                                                          cudaGraphCondAssignDefault);
        const long long launches0 = *R.launches;
        if (ec == cudaSuccess)
            ec = round0(cs[0]);
        *R.launches = launches0;
        cudaGraph_t *loopBody = nullptr;
        if (ec == cudaSuccess)
            ec = capture_conditional(cs[0], hLoop, cudaGraphCondTypeWhile, 1, &loopBody);
        if (ec == cudaSuccess)
            ec = cudaStreamBeginCaptureToGraph(cs[1], loopBody[0], nullptr, nullptr, 0,
                                               cudaStreamCaptureModeRelaxed);
        if (ec != cudaSuccess)
            return ec;
        for (int hr = 0; hr < 2 && ec == cudaSuccess; ++hr) {
            const Lists &X = hr == 0 ? A : B, &Y = hr == 0 ? B : A;
            rounds_tier_kernel<<<1, 32, 0, cs[1]>>>(X, Y, th[hr], usedLists, rareLists, cap,
                                                  R.launchDev);
            ec = cudaGetLastError();
            for (int l = 0; l < NLISTS && ec == cudaSuccess; ++l) {
                if (!((usedLists >> l) & 1u))
                    continue;
                const bool rare = (rareLists >> l) & 1u;
                const int nt = tier_count(cap, rare);
                cudaGraph_t *tiers = nullptr;
                ec = capture_conditional(cs[1], th[hr].h[l], cudaGraphCondTypeSwitch, nt, &tiers);
                for (int t = 0; t < nt && ec == cudaSuccess; ++t) {
                    ec = cudaStreamBeginCaptureToGraph(cs[2], tiers[t], nullptr, nullptr, 0,
                                                       cudaStreamCaptureModeRelaxed);
                    if (ec == cudaSuccess) {
                        cudaError_t el = launch_list(l, X.list[l], (int)tier_entries(t, cap, rare),
                                                     X.count[l], Y, cs[2]);
                        cudaGraph_t body = nullptr;
                        ec = cudaStreamEndCapture(cs[2], &body);
                        if (ec == cudaSuccess)
                            ec = el;
                    }
                }
            }
            if (ec == cudaSuccess && cap < R.ncells) { // no list can outgrow cap otherwise
                rounds_carry_kernel<<<1, 1024, 0, cs[1]>>>(X, Y, usedLists, cap);
                ec = cudaGetLastError();
            }
        }
        if (ec == cudaSuccess) {
            rounds_cond_kernel<<<1, 32, 0, cs[1]>>>(A, usedLists, R.counts + 2 * NLISTS,
                                                    R.maxRounds, R.errorFlag, hLoop, R.launchDev);
            ec = cudaGetLastError();
        }
        cudaGraph_t body = nullptr;
        cudaError_t eb = cudaStreamEndCapture(cs[1], &body);
        return ec == cudaSuccess ? eb : ec;
    };

    const long long round0Launches = probe ? 2 * ((R.ncells + R.batch - 1) / R.batch) : 1;
    if (R.captureTop) {
        // inside the capture of a whole RK stage
        e = capture_into(R.captureTop, R.captureStreams);
        if (e == cudaSuccess)
            *R.launches += round0Launches + 1;
        return e;
    }
    if (R.graphs) {
        RoundsGraph *RG = reinterpret_cast<RoundsGraph *>(R.graphs);
        std::vector<unsigned char> key = rounds_graph_key(R, GAUNT);
        RoundsGraph::Slot *G = nullptr;
        for (RoundsGraph::Slot &s : RG->slot)
            if (s.exec && s.key == key)
                G = &s;
        if (!G) {
            std::lock_guard<std::mutex> lk(graph_build_mutex());
            // the least recently used slot; a graph in it may still run on the stream and is
            // destroyed once the stream is idle
            G = &RG->slot[0];
            for (RoundsGraph::Slot &s : RG->slot)
                if (s.used < G->used)
                    G = &s;
            if (G->exec) {
                if ((e = cudaStreamSynchronize(st)) != cudaSuccess)
                    return e;
                cudaGraphExecDestroy(G->exec);
                G->exec = nullptr;
            }
            for (int i = 0; i < 3; ++i)
                if (!RG->cs[i] && (e = cudaStreamCreateWithFlags(&RG->cs[i], cudaStreamNonBlocking)) !=
                                      cudaSuccess)
                    return e;
            cudaGraph_t top = nullptr;
            if ((e = cudaGraphCreate(&top, 0)) != cudaSuccess)
                return e;
            e = cudaStreamBeginCaptureToGraph(RG->cs[0], top, nullptr, nullptr, 0,
                                              cudaStreamCaptureModeRelaxed);
            if (e == cudaSuccess) {
                const cudaError_t ec = capture_into(top, RG->cs);
                cudaGraph_t topOut = nullptr;
                e = cudaStreamEndCapture(RG->cs[0], &topOut);
                if (e == cudaSuccess)
                    e = ec;
            }
            if (e == cudaSuccess)
                e = cudaGraphInstantiate(&G->exec, top, 0);
            cudaGraphDestroy(top);
            if (e != cudaSuccess) {
                // a failed capture may leave its streams unusable: start over with new ones
                G->exec = nullptr;
                for (cudaStream_t &cs : RG->cs) {
                    if (cs)
                        cudaStreamDestroy(cs);
                    cs = nullptr;
                }
                cudaGetLastError();
                return e;
            }
            G->key = key;
        }
        G->used = ++RG->tick;
        *R.launches += round0Launches + 1;
        return cudaGraphLaunch(G->exec, st);
    }

    // host-driven rounds: the host reads the list counts after each round
    if ((e = round0(st)) != cudaSuccess)
        return e;
    *R.launches += 1;
    long long rounds = 0;
    for (;;) {
        e = cudaMemcpyAsync(R.hostCount, A.count[0], NLISTS * sizeof(unsigned int),
                            cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(st);
        if (e != cudaSuccess)
            return e;
        if (R.hostSyncs)
            ++*R.hostSyncs;
        long long cnt[NLISTS], total = 0;
        for (int l = 0; l < NLISTS; ++l)
            total += (cnt[l] = R.hostCount[l]);
        if (total == 0)
            break;
        if (++rounds > R.maxRounds)
            return cudaErrorLaunchTimeout;
        e = cudaMemsetAsync(B.count[0], 0, NLISTS * sizeof(unsigned int), st);
        if (e != cudaSuccess)
            return e;
        *R.launches += 1;
        for (int l = 0; l < NLISTS; ++l) {
            for (long long off = 0; off < cnt[l]; off += R.batch) {
                int nb = (int)((cnt[l] - off) < R.batch ? (cnt[l] - off) : R.batch);
                if ((e = launch_list(l, A.list[l] + off, nb, nullptr, B, st)) != cudaSuccess)
                    return e;
                *R.launches += 2;
            }
        }
        Lists t = A;
        A = B;
        B = t;
    }
    return cudaSuccess;
}

#endif // C3D_ROUNDS_PART != 0

#if C3D_ROUNDS_PART == 0
template <int NT, int NT2, bool GAUNT> cudaError_t rounds_t(const RoundsLaunch &R);
#define C3D_ROUNDS extern template
#else
#define C3D_ROUNDS template
#endif
#define C3D_ROUNDS_T(NT, NT2, G) C3D_ROUNDS cudaError_t rounds_t<NT, NT2, G>(const RoundsLaunch &);
#if C3D_ROUNDS_PART == 0 || C3D_ROUNDS_PART == 1
C3D_ROUNDS_T(1, 1, true)
C3D_ROUNDS_T(1, 2, true)
C3D_ROUNDS_T(2, 4, true)
C3D_ROUNDS_T(2, 7, true)
#endif
#if C3D_ROUNDS_PART == 0 || C3D_ROUNDS_PART == 2
C3D_ROUNDS_T(4, 11, true)
C3D_ROUNDS_T(1, 1, false)
C3D_ROUNDS_T(2, 1, false)
C3D_ROUNDS_T(3, 1, false)
#endif
#if C3D_ROUNDS_PART == 0 || C3D_ROUNDS_PART == 3
C3D_ROUNDS_T(5, 16, true)
C3D_ROUNDS_T(4, 1, false)
#endif
#if C3D_ROUNDS_PART == 0 || C3D_ROUNDS_PART == 4
C3D_ROUNDS_T(7, 22, true)
#endif
#if C3D_ROUNDS_PART == 0 || C3D_ROUNDS_PART == 5
C3D_ROUNDS_T(8, 29, true)
#endif
#if C3D_ROUNDS_PART == 0 || C3D_ROUNDS_PART == 6
C3D_ROUNDS_T(5, 1, false)
C3D_ROUNDS_T(6, 1, false)
#endif
#if C3D_ROUNDS_PART == 0 || C3D_ROUNDS_PART == 7
C3D_ROUNDS_T(7, 1, false)
#endif
#if C3D_ROUNDS_PART == 0 || C3D_ROUNDS_PART == 8
C3D_ROUNDS_T(8, 1, false)
#endif

#if C3D_ROUNDS_PART == 0
void *rounds_graph_new() { return new RoundsGraph(); }
void rounds_graph_free(void *g) { delete reinterpret_cast<RoundsGraph *>(g); }

// Moment counts with a work-list Gaunt form (N <= 7).
bool rounds_gaunt_supported(int nm)
{
    return nm == 1 || nm == 4 || nm == 9 || nm == 16 || nm == 25 || nm == 36 || nm == 49 ||
           nm == 64;
}

cudaError_t launch_closure_rounds(const RoundsLaunch &R, bool gaunt)
{
    const int nm = R.P->nm;
    if (gaunt) {
        switch (nm) {
        case 1: return rounds_t<1, 1, true>(R);
        case 4: return rounds_t<1, 2, true>(R);
        case 9: return rounds_t<2, 4, true>(R);
        case 16: return rounds_t<2, 7, true>(R);
        case 25: return rounds_t<4, 11, true>(R);
        case 36: return rounds_t<5, 16, true>(R);
        case 49: return rounds_t<7, 22, true>(R);
        case 64: return rounds_t<8, 29, true>(R);
        default: return cudaErrorInvalidValue;
        }
    }
    switch ((nm + 7) / 8) {
    case 1: return rounds_t<1, 1, false>(R);
    case 2: return rounds_t<2, 1, false>(R);
    case 3: return rounds_t<3, 1, false>(R);
    case 4: return rounds_t<4, 1, false>(R);
    case 5: return rounds_t<5, 1, false>(R);
    case 6: return rounds_t<6, 1, false>(R);
    case 7: return rounds_t<7, 1, false>(R);
    case 8: return rounds_t<8, 1, false>(R);
    default: return cudaErrorInvalidValue;
    }
}
#endif // C3D_ROUNDS_PART == 0

} // namespace c3d
