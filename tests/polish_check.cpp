// C entry point over opsec_gpu/csrc/polish.h for tests/test_polish_host.py (compiled there with g++; no
// CUDA).
#include "../opsec_gpu/csrc/polish.h"

extern "C" int chk_polish(int k, int m, const double* G, const double* H, double* E, double* lam) {
    return opsec::polish_close(k, m, G, H, E, lam);
}
