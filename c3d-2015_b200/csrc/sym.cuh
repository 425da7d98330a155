// Octant symmetry of the angular quadrature.
//
// The tensor quadrature (src/init.cpp:509-548, Q even) maps onto itself under the reflections
// x -> -x, y -> -y, z -> -z, and each real spherical harmonic is even or odd under each of
// them. So the nq directions are no = nq / 8 directions o of the positive octant times the 8
// reflections s (bit 0 flips x, bit 1 y, bit 2 z), the harmonics fall into 8 parity classes c
// (same bits: odd under that flip), and
//     m(q_{o,s}) = (-1)^{popcount(c & s)} m(q_{o,0})          for m of class c.
// A contraction over directions, F_m = sum_q v_q m(q), is then a Walsh-Hadamard transform of
// the 8 reflected values of each o (24 additions), V_c[o] = sum_s (-1)^{popcount(c & s)} v_{o,s},
// and one contraction per class over the no octant directions, F_m = sum_o V_c[o] m(q_{o,0}); an
// expansion z_q = sum_m a_m m(q) is the transpose. The FP64 tensor pipe (64 FMA per SM and
// clock, shared with the vector FP64 instructions) bounds these kernels: for M_6 the projection
// takes 9 n-tiles of 8 class members over nq / 8 directions instead of 7 n-tiles over nq, 6.2
// times fewer DMMAs; the 169 extended moments of the Gaunt form 24 instead of 22 * 8.
//
// Directions come in blocks of 8 octant directions, position n of block b holding direction
// 8 b + 4 (n % 2) + n / 2, so that the two columns a lane owns in a DMMA result belong to the
// two groups of 4 consecutive directions of the block. psi of a symmetric context is
// [group of 4 directions][reflection][cell][4 directions]: a warp's 8 cells x 4 directions are
// 256 consecutive bytes, and a cell's 4 directions one sector, whatever the alignment of its row.
#pragma once
#include "c3d_common.cuh"

#include <utility>
#include <vector>

namespace c3d {

// Parity class of the real harmonic (l, m) (c3d_real_sh): odd under x, y, z flips.
__host__ __device__ constexpr int sym_class(int l, int m)
{
    const int a = m < 0 ? -m : m;
    return ((m >= 0 ? a : a + 1) & 1) | (m < 0 ? 2 : 0) | (((l + a) & 1) ? 4 : 0);
}
__host__ __device__ constexpr int sym_count(int deg, int c)
{
    int n = 0;
    for (int l = 0; l <= deg; ++l)
        for (int m = -l; m <= l; ++m)
            n += sym_class(l, m) == c ? 1 : 0;
    return n;
}

// Layout of the classes of the harmonics of degree <= DEG: class members in column order,
// padded to tiles of 8 columns (contraction outputs) or steps of 4 (expansion inputs).
template <int DEG> struct SymCls {
    __host__ __device__ static constexpr int tiles(int c) { return (sym_count(DEG, c) + 7) / 8; }
    __host__ __device__ static constexpr int steps(int c) { return (sym_count(DEG, c) + 3) / 4; }
    __host__ __device__ static constexpr int tile0(int c)
    {
        int n = 0;
        for (int i = 0; i < c; ++i)
            n += tiles(i);
        return n;
    }
    __host__ __device__ static constexpr int step0(int c)
    {
        int n = 0;
        for (int i = 0; i < c; ++i)
            n += steps(i);
        return n;
    }
    static constexpr int TILES = tile0(8);
    static constexpr int STEPS = step0(8);
};

constexpr int SYM_BLK = 8; // octant directions per block
__host__ __device__ constexpr int sym_at(int b, int n) { return 8 * b + 4 * (n & 1) + (n >> 1); }
// psi rows (directions, padded to whole groups) for nq directions
__host__ __device__ constexpr int sym_rows(int nq) { return (nq + 31) / 32 * 32; }

// Octant direction o (mu, xi, eta > 0) in the order of the tensor quadrature with Q nodes.
__host__ __device__ inline int sym_direction(int Q, int o)
{
    return (Q / 2 + o / (Q / 2)) * 2 * Q + o % (Q / 2);
}

// Device tables of a symmetric quadrature (built by sym_build, owned by the context).
//   expo  [block][step][lane]        B fragment of Z = A M^T: member 4 step + lane % 4 of its
//                                    class at position lane / 4 of the block
//   proj  [block][half][tile][lane]  B fragment of F += V M: direction 8 block + 4 half +
//                                    lane % 4, member 8 tile + lane / 4 of its class
//   flux  [group of 4 directions][tile][lane], then |xi| w / dx, |eta| w / dy, |mu| w / dz and
//                                    4 zeros of the group's directions (the kinetic flux)
//   w     [block][position]          weights of the octant directions (0 past the last)
//   idx   [tile][8]                  column of each class member, -1 padding
// Degrees: expo and stepIdx the basis' N; proj and idx N (the flux, the probe) or 2N (the Hessian
// passes of the Gaunt form).
struct SymTables {
    int no, nb; // octant directions, blocks
    const double *expo, *proj, *w;
    const int *stepIdx; // [step][4] column of each expansion input, -1 padding
    const int *idx;
};

// Host tables; empty when the quadrature or the basis lacks the symmetry.
struct SymHost {
    int no = 0, nb = 0;
    std::vector<double> expo, proj, flux, w;
    std::vector<int> stepIdx, idx;
};
// M[nq * nm], nm = (deg + 1)^2, with weights and cosines (null cosines: implied by the order of
// the tensor quadrature, as for a degree-2N basis over directions already checked). expoDeg:
// degree of the expansion tables.
bool sym_build(int deg, int expoDeg, int nq, const double *M, const double *w, const double *xi,
               const double *eta, const double *mu, double rdx, double rdy, double rdz, SymHost &T);

#ifdef __CUDACC__

// Calls f(std::integral_constant<int, 0>) .. f(<N - 1>): loops whose index is a constant.
template <class F, int... I>
__device__ __forceinline__ void sym_unroll(F &&f, std::integer_sequence<int, I...>)
{
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F> __device__ __forceinline__ void sym_for(F &&f)
{
    sym_unroll(f, std::make_integer_sequence<int, N>{});
}

__device__ __forceinline__ void sym_dmma(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// v_c <- sum_s (-1)^{popcount(c & s)} v_s
__device__ __forceinline__ void sym_wht(double (&v)[8])
{
#pragma unroll
    for (int b = 1; b < 8; b <<= 1)
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (!(i & b)) {
                const double x = v[i], y = v[i | b];
                v[i] = x + y;
                v[i | b] = x - y;
            }
}

// Exponents of a block for the warp's 8 cells: lane l gets z[e][s] of cell l / 4 and octant
// direction 4 e + l % 4 of the block. aF: the cells' multipliers as A fragments
// [step][lane]; bE: the block's expansion fragments.
template <int DEG>
__device__ __forceinline__ void sym_expand(const double *aF, const double *bE, int lane,
                                           double (&z)[2][8])
{
    using C = SymCls<DEG>;
    sym_for<8>([&](auto cc) {
        constexpr int c = cc.value;
        double d0 = 0.0, d1 = 0.0;
        sym_for<C::steps(c)>([&](auto kk) {
            constexpr int k = C::step0(c) + kk.value;
            sym_dmma(d0, d1, aF[k * 32 + lane], bE[k * 32 + lane]);
        });
        z[0][c] = d0;
        z[1][c] = d1;
    });
    sym_wht(z[0]);
    sym_wht(z[1]);
}

// Contracts the transformed values of one half block (v: class values of the lane's cell and
// direction) onto the class members: acc[tile] of cell l / 4, members 2 (l % 4), + 1.
template <int DEG>
__device__ __forceinline__ void sym_contract(const double (&v)[8], const double *bP, int lane,
                                             double (&acc)[SymCls<DEG>::TILES][2])
{
    using C = SymCls<DEG>;
    sym_for<8>([&](auto cc) {
        constexpr int c = cc.value;
        sym_for<C::tiles(c)>([&](auto tt) {
            constexpr int t = C::tile0(c) + tt.value;
            sym_dmma(acc[t][0], acc[t][1], v[c], bP[t * 32 + lane]);
        });
    });
}

#endif // __CUDACC__

} // namespace c3d
