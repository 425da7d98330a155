// Host tables of the octant-symmetric kernels (sym.cuh).
#include "sym.cuh"

#include <algorithm>
#include <cmath>

namespace c3d {

// The classes' members by column, padded with -1 to whole tiles or steps, as SymCls lays them out.
static void layout(int deg, int unit, std::vector<int> &slots)
{
    slots.clear();
    for (int c = 0; c < 8; ++c) {
        int n = 0, k = 0;
        for (int l = 0; l <= deg; ++l)
            for (int m = -l; m <= l; ++m, ++k)
                if (sym_class(l, m) == c) {
                    slots.push_back(k);
                    ++n;
                }
        for (; n % unit; ++n)
            slots.push_back(-1);
    }
}

bool sym_build(int deg, int expoDeg, int nq, const double *M, const double *w, const double *xi,
               const double *eta, const double *mu, double rdx, double rdy, double rdz, SymHost &T)
{
    const int nm = (deg + 1) * (deg + 1);
    const int Q = (int)std::lround(std::sqrt(nq / 2.0));
    if (2 * Q * Q != nq || Q % 2)
        return false;
    // reflections of direction (q1, q2) of the tensor quadrature
    auto flip = [&](int q, int s) {
        int q1 = q / (2 * Q), q2 = q % (2 * Q);
        if (s & 1)
            q2 = (3 * Q - 1 - q2) % (2 * Q);
        if (s & 2)
            q2 = 2 * Q - 1 - q2;
        if (s & 4)
            q1 = Q - 1 - q1;
        return q1 * 2 * Q + q2;
    };
    const double parity[8] = {1, -1, -1, 1, -1, 1, 1, -1}; // (-1)^popcount
    std::vector<int> cls(nm);
    for (int l = 0, k = 0; l <= deg; ++l)
        for (int m = -l; m <= l; ++m, ++k)
            cls[k] = sym_class(l, m);
    // The tables hold the positive octant's values, whose angles are the smallest and so carry the
    // least rounding (on near-singular M_6 cells the multipliers moved by 2e-9 relative against
    // the full table, by 5e-9 with the mean over the reflections; a last-bit change of the
    // moments moves them by 1e-9). A basis that differs from its reflections by more than the
    // rounding of its own sines and cosines is not symmetric.
    const double tol = 1e-13;
    T = SymHost{};
    T.no = nq / 8;
    T.nb = (T.no + SYM_BLK - 1) / SYM_BLK;
    const int np = T.nb * SYM_BLK;
    std::vector<double> B((size_t)np * nm, 0.0), cx(np, 0.0), cy(np, 0.0), cz(np, 0.0);
    T.w.assign(np, 0.0);
    for (int o = 0; o < T.no; ++o) {
        const int q0 = sym_direction(Q, o);
        const double *m0 = M + (size_t)q0 * nm;
        if (xi && !(xi[q0] > 0.0 && eta[q0] > 0.0 && mu[q0] > 0.0))
            return false;
        for (int s = 0; s < 8; ++s) {
            const int q = flip(q0, s);
            const double *ms = M + (size_t)q * nm;
            bool same = std::fabs(w[q] - w[q0]) <= tol * w[q0];
            for (int k = 0; k < nm; ++k) {
                const double v = parity[cls[k] & s] * ms[k];
                same = same && std::fabs(v - m0[k]) <= tol * (1.0 + std::fabs(m0[k]));
            }
            if (xi)
                same = same && std::fabs((s & 1 ? -xi[q] : xi[q]) - xi[q0]) <= tol &&
                       std::fabs((s & 2 ? -eta[q] : eta[q]) - eta[q0]) <= tol &&
                       std::fabs((s & 4 ? -mu[q] : mu[q]) - mu[q0]) <= tol;
            if (!same)
                return false;
        }
        std::copy(m0, m0 + nm, &B[(size_t)o * nm]);
        T.w[o / 8 * 8 + 2 * (o % 4) + o / 4 % 2] = w[q0]; // position of direction o
        if (xi) {
            cx[o] = (xi[q0] * w[q0]) * rdx;
            cy[o] = (eta[q0] * w[q0]) * rdy;
            cz[o] = (mu[q0] * w[q0]) * rdz;
        }
    }
    layout(deg, 8, T.idx);
    layout(expoDeg, 4, T.stepIdx);
    const int tiles = (int)T.idx.size() / 8, steps = (int)T.stepIdx.size() / 4;
    auto at = [&](int o, int k) { return k < 0 ? 0.0 : B[(size_t)o * nm + k]; };
    T.expo.resize((size_t)T.nb * steps * 32);
    T.proj.resize((size_t)T.nb * 2 * tiles * 32);
    for (int b = 0; b < T.nb; ++b)
        for (int l = 0; l < 32; ++l) {
            for (int k = 0; k < steps; ++k)
                T.expo[((size_t)b * steps + k) * 32 + l] = at(sym_at(b, l / 4), T.stepIdx[4 * k + l % 4]);
            for (int h = 0; h < 2; ++h)
                for (int t = 0; t < tiles; ++t)
                    T.proj[(((size_t)b * 2 + h) * tiles + t) * 32 + l] =
                        at(8 * b + 4 * h + l % 4, T.idx[8 * t + l / 4]);
        }
    if (xi) {
        const int ng = 2 * T.nb;
        const size_t per = (size_t)tiles * 32 + 16;
        T.flux.assign(per * ng, 0.0);
        for (int g = 0; g < ng; ++g) {
            double *f = T.flux.data() + per * g;
            for (int t = 0; t < tiles; ++t)
                for (int l = 0; l < 32; ++l)
                    f[t * 32 + l] = at(4 * g + l % 4, T.idx[8 * t + l / 4]);
            for (int d = 0; d < 4; ++d) {
                f[tiles * 32 + d] = cx[4 * g + d];
                f[tiles * 32 + 4 + d] = cy[4 * g + d];
                f[tiles * 32 + 8 + d] = cz[4 * g + d];
            }
        }
    }
    return true;
}

} // namespace c3d
