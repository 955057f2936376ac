// polish.h -- the correction of approximate eigenvectors some of whose eigenvalues lie so close that their
// vectors are mixed by more than a first-order correction mends.  Plain C++, so that CPU tests compile and
// check this code itself.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

namespace opsec {

// A correction to first order, its norms to second, leaves out a third of the cube of a coupling (relative to
// the distance of its two eigenvalues) and half the product of two couplings of one vector.  It holds up to
constexpr double kCloseCoupling = 1e-5;
constexpr double kCloseProduct = 2e-13;  // 1e-13: the rounding of FP64 sums over some hundred cells
// Beyond, eigenvalues with couplings from here on are gathered and diagonalised (left out then: 5e-15)
constexpr double kGroupCoupling = 1e-7;
// A coupling that is rounding, at most this times the largest eigenvalue, is left alone.
constexpr double kCouplingRounding = 8.0 * 2.220446049250313e-16;

namespace polish {

// Eigenvectors (columns of V) and eigenvalues w, largest first, of a symmetric c x c matrix by Jacobi rotations
inline void jacobi(int c, std::vector<double>& A, std::vector<double>& V, std::vector<double>& w) {
    V.assign((size_t)c * c, 0.0);
    for (int i = 0; i < c; i++) V[(size_t)i * c + i] = 1.0;
    auto a = [&](int i, int j) -> double& { return A[(size_t)j * c + i]; };
    for (int sweep = 0; sweep < 30; sweep++) {
        double off = 0.0;
        for (int j = 1; j < c; j++)
            for (int i = 0; i < j; i++) off = std::max(off, std::fabs(a(i, j)));
        if (!(off > 0.0)) break;
        for (int j = 1; j < c; j++)
            for (int i = 0; i < j; i++) {
                if (a(i, j) == 0.0) continue;
                const double z = (a(j, j) - a(i, i)) / (2.0 * a(i, j));
                const double t = (z >= 0 ? 1.0 : -1.0) / (std::fabs(z) + std::hypot(1.0, z));
                const double cs = 1.0 / std::hypot(1.0, t), sn = t * cs, aij = a(i, j);
                a(i, i) -= t * aij;
                a(j, j) += t * aij;
                a(i, j) = a(j, i) = 0.0;
                for (int k = 0; k < c; k++) {
                    if (k != i && k != j) {
                        const double x = a(k, i), y = a(k, j);
                        a(k, i) = a(i, k) = cs * x - sn * y;
                        a(k, j) = a(j, k) = sn * x + cs * y;
                    }
                    const double x = V[(size_t)i * c + k], y = V[(size_t)j * c + k];
                    V[(size_t)i * c + k] = cs * x - sn * y;
                    V[(size_t)j * c + k] = sn * x + cs * y;
                }
            }
    }
    std::vector<int> o(c);
    for (int i = 0; i < c; i++) o[i] = i;
    std::stable_sort(o.begin(), o.end(), [&](int x, int y) { return a(x, x) > a(y, y); });
    std::vector<double> U((size_t)c * c);
    w.resize(c);
    for (int i = 0; i < c; i++) {
        w[i] = a(o[i], o[i]);
        std::copy_n(V.begin() + (size_t)o[i] * c, c, U.begin() + (size_t)i * c);
    }
    V.swap(U);
}

}  // namespace polish

// k approximate eigenvectors X, largest eigenvalue first, nearly orthonormal: from G = X^T X and H = X^T S X
// (k x k, lower triangles, column-major) the k x m matrix E of the refined first m vectors X (I + E) and their
// Rayleigh quotients.  Eigenvalues coupled by more than kGroupCoupling of their distance are gathered in groups,
// whose parts of H, made orthonormal to first order, are diagonalised; then every coupling left is corrected to
// first order and the norms to second (the map of the device's kernel).  False when a group outgrows `most`,
// rotations bring up ever more of them, or values are not finite.
inline bool polish_close(int k, int m, const double* Glow, const double* Hlow, double* E, double* lam, int most = 128) {
    const size_t kk = (size_t)k * k;
    std::vector<double> G(kk), H(kk), l(k);
    for (int j = 0; j < k; j++)
        for (int i = j; i < k; i++) {
            const size_t o = (size_t)j * k + i, p = (size_t)i * k + j;
            if (!std::isfinite(Glow[o]) || !std::isfinite(Hlow[o])) return false;
            G[o] = G[p] = Glow[o];
            H[o] = H[p] = Hlow[o];
        }
    // H as orthonormal vectors would have it, off the diagonal; of one triangle, so that rounding over a
    // small distance of eigenvalues cancels between the two vectors' corrections
    auto low = [&](int i, int j) { return (size_t)std::min(i, j) * k + std::max(i, j); };
    auto coupling = [&](int i, int j) { return H[low(i, j)] - 0.5 * (l[i] + l[j]) * G[low(i, j)]; };
    auto above = [&](int i, int j) { return !(std::fabs(coupling(i, j)) <= kGroupCoupling * std::fabs(l[j] - l[i])); };
    auto strong = [&](int i, int j) { return above(i, j) && !(std::fabs(coupling(i, j)) <= kCouplingRounding * std::fabs(l[0])); };
    struct Group {
        std::vector<int> at;
        std::vector<double> Q;
    };
    std::vector<Group> done;
    // X Q for the columns of a group, row by row of M^T (both triangles are kept)
    auto rotate = [&](std::vector<double>& M, const Group& g) {
        const int c = (int)g.at.size();
        std::vector<double> t(c);
        for (int side = 0; side < 2; side++)
            for (int r = 0; r < k; r++) {
                auto e = [&](int col) -> double& { return side ? M[(size_t)r * k + col] : M[(size_t)col * k + r]; };
                for (int q = 0; q < c; q++) {
                    t[q] = 0.0;
                    for (int p = 0; p < c; p++) t[q] += e(g.at[p]) * g.Q[(size_t)q * c + p];
                }
                for (int q = 0; q < c; q++) e(g.at[q]) = t[q];
            }
    };
    for (int round = 0;; round++) {  // a rotation can bring a coupling closer to a third eigenvalue
        for (int i = 0; i < k; i++) l[i] = H[(size_t)i * k + i] / G[(size_t)i * k + i];
        std::vector<int> root(k);
        for (int i = 0; i < k; i++) root[i] = i;
        auto find = [&](int i) {
            while (root[i] != i) i = root[i] = root[root[i]];
            return i;
        };
        bool any = false;
        for (int j = 0; j < m; j++)  // two vectors past the first m need not be told apart
            for (int i = j + 1; i < k; i++)
                if (strong(i, j)) {
                    root[find(i)] = find(j);
                    any = true;
                }
        if (!any) break;
        if (round == 4) return false;
        std::vector<std::vector<int>> groups(k);
        for (int i = 0; i < k; i++) groups[find(i)].push_back(i);
        for (auto& at : groups) {
            const int c = (int)at.size();
            if (c < 2) continue;
            if (c > most) return false;
            Group g{at, {}};
            std::vector<double> A((size_t)c * c), w;
            for (int q = 0; q < c; q++)
                for (int p = 0; p < c; p++) A[(size_t)q * c + p] = p == q ? l[at[q]] : coupling(at[p], at[q]);
            polish::jacobi(c, A, g.Q, w);
            rotate(H, g);
            rotate(G, g);
            done.push_back(g);
        }
    }
    for (int j = 0; j < m; j++) {
        double* e = E + (size_t)j * k;
        double s2 = 0.0;
        for (int i = 0; i < k; i++) {
            if (i == j) continue;
            const double kij = above(i, j) || l[j] == l[i] ? 0.0 : coupling(i, j) / (l[j] - l[i]);
            e[i] = kij - 0.5 * G[low(i, j)];
            s2 += kij * kij;
        }
        e[j] = 1.0 + 0.5 * (1.0 - G[(size_t)j * k + j] - s2);
        for (auto g = done.rbegin(); g != done.rend(); ++g) {
            const int c = (int)g->at.size();
            std::vector<double> t(c, 0.0);
            for (int q = 0; q < c; q++)
                for (int p = 0; p < c; p++) t[p] += g->Q[(size_t)q * c + p] * e[g->at[q]];
            for (int p = 0; p < c; p++) e[g->at[p]] = t[p];
        }
        e[j] -= 1.0;
        lam[j] = l[j];
    }
    return true;
}

}  // namespace opsec
