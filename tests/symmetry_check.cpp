// C entry point over opsec_gpu/csrc/symmetry.h for tests/test_symmetry_host.py (compiled there with g++;
// no CUDA).
#include "../opsec_gpu/csrc/symmetry.h"

extern "C" int chk_forces_degeneracy(int coordsys, const double* b, const int* n, double L, int full_phi, int ncells,
                                     const opsec_cell* cells) {
    return opsec::Symmetry(coordsys, b, n, L, full_phi != 0, ncells, cells).forces_degeneracy();
}
