// symmetry.h -- whether a survey's geometry makes eigenvalues of its signal matrix coincide exactly.
// Plain C++, so that CPU tests compile and check this code itself.
#pragma once

#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

#include "../../include/opsec_gpu.h"

namespace opsec {

// S depends on the cells' separations and Nbar alone, so a motion of the grid that maps the survey onto
// itself commutes with S.  One of order three or more forces pairs of equal eigenvalues (S is real: the
// eigenspaces of a complex eigenvalue of the motion and of its conjugate have the same spectrum); motions of
// order two force none.  Looked for: quarter turns about an axis (with or without its reflection) and thirds
// of a turn about a diagonal of a Cartesian grid, translations by a part of a periodic one, turns in phi by
// a part of a full circle.  Also true for the plain exchange of two Cartesian axes, which most often
// comes with a reflection and so with a quarter turn.
// `cells` may be any subset of the grid, in any order; Nbar equal to 1e-9 counts as equal.
class Symmetry {
  public:
    // coordsys 1 Cartesian (L > 0: periodic), 2 spherical; b: Min1, Max1, ...; n: cells an axis
    Symmetry(int coordsys, const double* b, const int* n, double L, bool full_phi, int ncells, const opsec_cell* cells)
        : coordsys_(coordsys), L_(L), full_phi_(full_phi), cells_(cells), ncells_(ncells) {
        for (int p = 0; p < 3; p++) {
            n_[p] = n[p];
            h_[p] = (b[2 * p + 1] - b[2 * p]) / n[p];
        }
    }

    bool forces_degeneracy() {
        if (coordsys_ == 2) return full_phi_ && shifted(2);
        for (int p = 0; p < 3; p++) {
            const int q = (p + 1) % 3, r = (p + 2) % 3;
            if (L_ > 0 && close(n_[p] * h_[p], L_) && shifted(p)) return true;
            if (!alike(p, q)) continue;
            const auto exchange = [=](int* d) { std::swap(d[p], d[q]); };
            if (maps_onto_itself(exchange)) return true;
            for (int f = 0; f < 2; f++) {
                const auto quarter = [=](int* d) {
                    const int t = d[p];
                    d[p] = d[q];
                    d[q] = n_[p] - 1 - t;
                    if (f) d[r] = n_[r] - 1 - d[r];
                };
                if (turns(quarter)) return true;
            }
        }
        if (alike(0, 1) && alike(1, 2))
            for (int f = 0; f < 4; f++) {
                const auto third = [=](int* d) {  // (y, z, x), two of them reflected or none
                    const int t = d[0];
                    d[0] = f == 1 || f == 2 ? n_[0] - 1 - d[1] : d[1];
                    d[1] = f == 1 || f == 3 ? n_[0] - 1 - d[2] : d[2];
                    d[2] = f == 2 || f == 3 ? n_[0] - 1 - t : t;
                };
                if (turns(third)) return true;
            }
        return false;
    }

  private:
    int coordsys_, n_[3];
    double h_[3], L_;
    bool full_phi_;
    const opsec_cell* cells_;
    int ncells_;
    std::vector<std::pair<long long, double>> at_;  // (grid cell, Nbar), sorted; filled for the first motion

    static bool close(double x, double y) { return std::fabs(x - y) <= 1e-9 * std::max(std::fabs(x), std::fabs(y)); }
    bool alike(int p, int q) const { return n_[p] == n_[q] && close(h_[p], h_[q]); }
    long long id(int d1, int d2, int d3) const { return ((long long)d1 * n_[1] + d2) * n_[2] + d3; }

    template <class Motion>
    bool maps_onto_itself(Motion g) {
        if (at_.empty()) {
            at_.reserve(ncells_);
            for (int a = 0; a < ncells_; a++) at_.emplace_back(id(cells_[a].d1, cells_[a].d2, cells_[a].d3), cells_[a].Nbar);
            if (!std::is_sorted(at_.begin(), at_.end())) std::sort(at_.begin(), at_.end());
        }
        for (int a = 0; a < ncells_; a++) {
            const opsec_cell& c = cells_[a];
            int d[3] = {c.d1, c.d2, c.d3};
            g(d);
            const std::pair<long long, double> key(id(d[0], d[1], d[2]), -HUGE_VAL);
            const auto it = std::lower_bound(at_.begin(), at_.end(), key);
            if (it == at_.end() || it->first != key.first || !close(it->second, c.Nbar)) return false;
        }
        return true;
    }
    // ... and is of order three or more on its cells
    template <class Motion>
    bool turns(Motion g) {
        if (!maps_onto_itself(g)) return false;
        for (int a = 0; a < ncells_; a++) {
            const opsec_cell& c = cells_[a];
            int d[3] = {c.d1, c.d2, c.d3};
            g(d);
            g(d);
            if (d[0] != c.d1 || d[1] != c.d2 || d[2] != c.d3) return true;
        }
        return false;
    }
    // invariant under a cyclic shift of axis p by n/4 or by n over an odd number (every cyclic group of
    // order above two holds one of these)
    bool shifted(int p) {
        const int n = n_[p];
        for (int k = 3; k <= n; k++)
            if (n % k == 0 && (k == 4 || k % 2) && turns([=](int* d) { d[p] = (d[p] + n / k) % n; })) return true;
        return false;
    }
};

}  // namespace opsec
