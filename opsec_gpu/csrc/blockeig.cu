// Batched symmetric eigensolver for the azimuthal blocks of a full-sky signal matrix.
//
// The KL step (klt.cpp:173-248) needs the top-M eigenpairs of S; the reference gets them from
// ARPACK's implicitly restarted Lanczos on the whole S (ParpackSolver.cpp:111-123).  On a
// full-sky grid S is block diagonal in the azimuthal order m (and the mu parity), so the engine
// solves the blocks: every eigenvalue of every block (the global top-M cut needs them all), but
// eigenvectors only for the block eigenvalues that can survive the cut.
//
//   1. tridiag.cu: Householder reduction A = Q T Q^T of every block, in double-FP32 (df64.h).
//   2. spectrum_kernel: every eigenvalue of every T by bisection on FP32 Sturm counts of the
//      power-of-two-scaled T (to ~1e-6 of the block norm): enough to decide which block
//      eigenvalues can reach the global cut.
//   3. (host) the candidates: per block, the eigenvalues within a safe margin of the cut.
//   4. vectors_kernel: each candidate's eigenvalue from its FP32 bracket (confirmed by two Sturm
//      counts, narrowed until it holds this eigenvalue alone) by Rayleigh-quotient iteration on
//      twisted factorisations (the solutions of (T - s I) x = 0 from the top and from the bottom
//      meet at the row where the residual is smallest), in double-FP32 and at the end in FP64,
//      then its eigenvector of T from the last one.
//   5. cluster_kernel: Gram-Schmidt (twice) inside clusters of candidates closer than 1e-6 of the
//      block norm, where separately computed vectors need not be orthogonal.
//   6. backtransform_kernel: x = Q z by the stored reflectors, four at a time (double-FP32), written
//      as the block's eigenvector column (ascending eigenvalue order, the layout of LAPACK's syevd):
//      34 blocks of 512^2 1.85 -> 0.92 ms, 10 of 555^2 1.40 -> 0.53 against
//      one reflector at a time by CTAs of 16 vectors.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>

#include "df64.h"
#include "engine.h"
#include "packed.h"
#include "polish.h"

namespace opsec {
namespace {

constexpr int kMaxN = 1024;     // largest block of the batched form
constexpr int kMaxRows = 4096;  // largest matrix

// Deterministic CTA-wide sum: the same inputs give the same bits in every CTA of the cluster.
__device__ double cta_sum(double x, double* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp] = x;
    __syncthreads();
    if (warp == 0) {
        double y = lane < (int)(blockDim.x >> 5) ? red[lane] : 0.0;
#pragma unroll
        for (int o = 16; o; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
        if (lane == 0) red[32] = y;
    }
    __syncthreads();
    const double r = red[32];
    __syncthreads();
    return r;
}

// ---------------------------------------------------------------- the three-term recurrence
// Everything below follows the solutions of (T' - s I) x = 0 row by row, T' the block's T with its
// off-diagonals made -|e_i| (a similarity by signs):
//   x_{i+1} = ((d_i - s) x_i - |e_{i-1}| x_{i-1}) / |e_i|
// x_i is the leading i x i minor of T - s I over prod |e|, so its sign changes count the eigenvalues
// below s (Sturm), and the two solutions from the top and from the bottom are the two halves of a
// twisted factorisation's eigenvector.  With a_i = (d_i - s) / |e_i| and the ratio |e_{i-1}| / |e_i|
// tabulated per block a row is three instructions and one FMA of latency; the pivots' form of the
// same recurrence, q_{i+1} = d - s - e^2 / q_i, waits for a division in every row (FP32 some 60
// cycles, FP64 several hundred at this part's 1/64 rate).  Solutions grow and decay far beyond the
// exponent range, so they are rescaled by powers of two every few rows.  |e_i| is held at or above
// eps/4 of the block's scale, below the rounding of the reduction, which bounds the growth per row.
constexpr int kGrp32 = 4, kGrp64 = 8;  // rows between rescalings: 27 and 62 bits of growth a row

__device__ __forceinline__ int round_up(int n, int g) { return (n + g - 1) / g * g; }

// ---------------------------------------------------------------- spectrum (FP32 bisection)
// row: (d / |e|, 1 / |e|, -|e_{i-1}| / |e|), n a multiple of kGrp32 (rows past the end keep x)
__device__ __forceinline__ int sturm32(int n, const float4* row, float s) {
    float x = 1.f, xp = 0.f;
    unsigned cnt = 0;
    for (int i = 0; i < n; i += kGrp32) {
#pragma unroll
        for (int k = 0; k < kGrp32; k++) {
            const float4 t = row[i + k];
            const float y = fmaf(fmaf(-s, t.y, t.x), x, t.z * xp);
            cnt += (__float_as_uint(y) ^ __float_as_uint(x)) >> 31;
            xp = x;
            x = y;
        }
        const unsigned e = __float_as_uint(fmaxf(fabsf(x), fabsf(xp))) & 0x7f800000u;
        const float sc = __uint_as_float(0x7f000000u - e);  // 2^-exponent
        x *= sc;
        xp *= sc;
    }
    return (int)cnt;
}

// Power-of-two scale of a block (>= its Gershgorin bound), so that scaling is exact.
__device__ double block_scale(int n, const double* d, const double* e, double* red) {
    double m = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double r = fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0);
        m = fmax(m, r);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    double g = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) g = fmax(g, red[w]);
    __syncthreads();
    if (!(g > 0.0)) return 1.0;
    int ex;
    frexp(g, &ex);
    return ldexp(1.0, ex);  // 2^ex > g
}

// Every eigenvalue j (ascending) of block b to ~1e-6 of its scale; grid (nblk, ceil(n SECT / 256)).
// SECT lanes an eigenvalue, SECT - 1 of which count below one shift each: the bracket shrinks SECT-fold a
// count.  With two (bisection, one lane) the chip idles behind each count's chain of n rows.
template <int SECT>
__global__ void __launch_bounds__(256) spectrum_kernel(int n, const double* __restrict__ dg,
                                                       const double* __restrict__ eg, double* __restrict__ w,
                                                       double* __restrict__ scale_out) {
    extern __shared__ float4 rows32[];
    __shared__ double red[32];
    const int b = blockIdx.x, np = round_up(n, kGrp32);
    const double* db = dg + (size_t)b * n;
    const double* ebk = eg + (size_t)b * n;
    const double sc = block_scale(n, db, ebk, red);
    const double inv = 1.0 / sc;
    constexpr float kMinE = 1.4901161193847656e-8f;  // 2^-26
    for (int i = threadIdx.x; i < np; i += blockDim.x) {
        float4 t = make_float4(1.f, 0.f, 0.f, 0.f);
        if (i < n) {
            const float e = i + 1 < n ? fmaxf(fabsf((float)(ebk[i] * inv)), kMinE) : 1.f;
            const float ep = i > 0 ? fmaxf(fabsf((float)(ebk[i - 1] * inv)), kMinE) : 0.f;
            t = make_float4((float)(db[i] * inv) / e, 1.f / e, -ep / e, 0.f);
        }
        rows32[i] = t;
    }
    __syncthreads();
    if (blockIdx.y == 0 && threadIdx.x == 0) scale_out[b] = sc;
    constexpr int kLanes = SECT > 2 ? SECT : 1;
    const int t = blockIdx.y * blockDim.x + threadIdx.x, j = t / kLanes, q = t % kLanes;
    float lo = -1.0f, hi = 1.0f;  // the scaled spectrum lies in (-1, 1)
    if constexpr (SECT > 2) {
        const int base = threadIdx.x & 31 & ~(SECT - 1);
        for (int it = 0; it < 40 && hi - lo > 2.5e-7f; it++) {  // the same steps for every eigenvalue
            const float d = (hi - lo) * (1.f / SECT);
            const bool above = q + 1 == SECT || sturm32(np, rows32, fmaf((float)(q + 1), d, lo)) > j;
            const int h = __ffs((int)((__ballot_sync(0xffffffffu, above) >> base) & ((1u << SECT) - 1)));  // 1 .. SECT
            const float l = fmaf((float)(h - 1), d, lo);
            if (h < SECT) hi = fmaf((float)h, d, lo);
            lo = l;
        }
        if (j >= n || q) return;
    } else {
        if (j >= n) return;
        for (int it = 0; it < 40 && hi - lo > 2.5e-7f; it++) {
            const float mid = 0.5f * (lo + hi);
            if (sturm32(np, rows32, mid) > j) hi = mid;
            else lo = mid;
        }
    }
    w[(size_t)b * n + j] = 0.5 * ((double)lo + (double)hi) * sc;
}

// ---------------------------------------------------------------- candidate eigenpairs (FP64)
struct VecArgs {
    int n, nblk, ktot;
    const int* kc;       // [nblk] candidates per block (the top kc[b] eigenvalues)
    const int* koff;     // [nblk] their first column in the [row][ktot] arrays
    const double* dg;    // [nblk][n]
    const double* eg;
    const double* scale; // [nblk] power-of-two scale of each block
    double* w;           // [nblk][n] ascending: approximate in, candidates refined out
    double* Z;           // [n][ktot] eigenvectors of T, then of the block
    int* KX;             // scratch: exponents of groups of rows of X, then of Y ([ceil(n/2)][ktot] each)
    double* X;           // [n][ktot] scratch: the solution from the top
    double* Y;           // [n][ktot] scratch: the solution from the bottom
    bool polished;       // a correction of the vectors follows
    int* status;         // [nblk]: 0, or 1 when a bracket could not be confirmed, 2 when a cluster degenerated
};

// Per block, in shared memory: the rows of both recurrences (np = n rounded up to kGrp64).
struct Rows64 {
    const double *ff, *fi, *fb;  // from the top: d/|e_i|, 1/|e_i|, -|e_{i-1}|/|e_i|
    const double *bf, *bb;       // from the bottom: d/|e_{i-1}|, -|e_i|/|e_{i-1}| (1/|e_{i-1}| is fi[i-1])
};

// 2^-e for the exponent e of x (x normal), and e
__device__ __forceinline__ double exp_scale(double x, int* e) {
    const int h = (__double2hiint(x) >> 20) & 0x7ff;
    *e = h - 1023;
    return __hiloint2double((2046 - h) << 20, 0);
}
__device__ __forceinline__ unsigned hi_xor(double a, double b) { return (unsigned)(__double2hiint(a) ^ __double2hiint(b)); }

// The lanes that share a candidate: 2 to 32 neighbouring ones, which take the same decisions.
struct Team {
    unsigned mask;
    int size, sub, base;  // lanes, this lane's place among them, the first one
    template <class X>
    __device__ __forceinline__ X from(X v, int q) const {
        return __shfl_sync(mask, v, base + q);
    }
    __device__ __forceinline__ double sum(double v) const {
        for (int o = size / 2; o; o >>= 1) v += __shfl_xor_sync(mask, v, o);
        return v;
    }
    // the largest v's smallest r
    __device__ __forceinline__ void best(int* v, int* r) const {
        for (int o = size / 2; o; o >>= 1) {
            const int vo = __shfl_xor_sync(mask, *v, o), ro = __shfl_xor_sync(mask, *r, o);
            if (vo > *v || (vo == *v && ro < *r)) {
                *v = vo;
                *r = ro;
            }
        }
    }
};

// eigenvalues below the shift
__device__ int sturm64(int np, const Rows64& t, double s) {
    double x = 1.0, xp = 0.0;
    unsigned c = 0;
    for (int i = 0; i < np; i += kGrp64) {
#pragma unroll
        for (int k = 0; k < kGrp64; k++) {
            const double y = fma(fma(-s, t.fi[i + k], t.ff[i + k]), x, t.fb[i + k] * xp);
            c += hi_xor(y, x) >> 31;
            xp = x;
            x = y;
        }
        int e;
        const double sc = exp_scale(fmax(fabs(x), fabs(xp)), &e);
        x *= sc;
        xp *= sc;
    }
    return (int)c;
}

// The same counts in double-FP32 (47 bits; rescaled every row, FP32's exponent range being short):
// FP64 instructions take 64 cycles a warp on one scheduler's pipe, three of them a row.
struct RowsDf {
    const float2 *f, *g, *b;  // d/|e_i|, 1/|e_i|, -|e_{i-1}|/|e_i| as (hi, lo) pairs
};
__device__ int sturm_df(int np, const RowsDf& t, double s) {
    df x{1.f, 0.f}, xp{0.f, 0.f};
    const df ms = df_from(-s);
    unsigned c = 0;
#pragma unroll 4
    for (int i = 0; i < np; i++) {
        const df f = df_unpack(t.f[i]), g = df_unpack(t.g[i]), b = df_unpack(t.b[i]);
        const df y = df_fma(df_mul(b, xp), df_fma(f, ms, g), x);
        c += (__float_as_uint(y.h) ^ __float_as_uint(x.h)) >> 31;
        const unsigned e = __float_as_uint(fmaxf(fabsf(y.h), fabsf(x.h))) & 0x7f800000u;
        const float sc = __uint_as_float(0x7f000000u - e);  // 2^-exponent
        xp = df{x.h * sc, x.l * sc};
        x = df{y.h * sc, y.l * sc};
    }
    return (int)c;
}

// One step of the search for eigenvalue j in (lo, hi), which hold clo and chi eigenvalues below
// them: the bracket's interior shifts, evenly spaced, one a lane of the team (two where more no longer
// separate).  False when two do not.
template <class Count>
__device__ bool narrow(const Team& tm, Count count, int j, double* lo, double* hi, int* clo, int* chi) {
    for (int ns = tm.size;; ns = 2) {
        auto shift = [&](int q) { return q < 0 ? *lo : q >= ns ? *hi : *lo + (*hi - *lo) * ((q + 1) / (double)(ns + 1)); };
        const int q = min(tm.sub, ns - 1);
        const double s = shift(q);
        if (__all_sync(tm.mask, s > shift(q - 1) && s < shift(q + 1))) {
            const int c = count(s);
            const unsigned above = (__ballot_sync(tm.mask, c > j) >> tm.base) & (ns == 32 ? ~0u : (1u << ns) - 1);
            const int h = above ? __ffs((int)above) - 1 : ns;  // the first shift above eigenvalue j
            const double l = shift(h - 1), u = shift(h);
            const int cl = tm.from(c, max(h - 1, 0)), cu = tm.from(c, min(h, ns - 1));
            if (h > 0) *clo = cl;
            if (h < ns) *chi = cu;
            *lo = l;
            *hi = u;
            return true;
        }
        if (ns == 2) return false;
    }
}

// 2^k, zero far below the smallest normal
__device__ __forceinline__ double pow2i(int k) { return k < -1000 ? 0.0 : __hiloint2double((min(k, 1000) + 1023) << 20, 0); }

// Twisted factorisation at s: the solutions from the top (X) and from the bottom (Y), meeting at
// the row r where |x_r y_r| is largest: (T - s I)^{-1}_{rr} is x_r y_r over their (constant)
// Wronskian, so that is where the residual gamma_r of z = (x_i / x_r above, 1, y_i / y_r below) is
// least.  Entries carry the exponent of their group of kGrp64 rows.  Returns the
// Rayleigh-quotient correction gamma_r / |z|^2; |z|^2 in *nz_out.
// Even lanes of the team take the solution from the top, odd ones that from the bottom; the scans are dealt
// over all of them.
__device__ double rq_step(const Team& tm, int n, const Rows64& t, const double* __restrict__ d,
                          const double* __restrict__ e, double inv, double s, const VecArgs& a, int col, int* r_out,
                          double* nz_out) {
    const size_t K = (size_t)a.ktot;
    double* X = a.X + col;
    double* Y = a.Y + col;
    const int ngrp = (n + kGrp64 - 1) / kGrp64;
    int* KX = a.KX + col;
    int* KY = KX + (size_t)ngrp * K;
    __syncwarp(tm.mask);  // the last step's solutions have been read
    {
        const bool up = tm.sub & 1, own = tm.sub < 2;
        const double *pf = up ? t.bf : t.ff, *pb = up ? t.bb : t.fb;
        double* P = up ? Y : X;
        int* KP = up ? KY : KX;
        double x = 1.0, xp = 0.0;
        int kx = 0;
        for (int g = 0; g < ngrp; g++) {
            // rows of group g from the top, of group ngrp-1-g from the bottom (rows past n keep x)
            const int gi = up ? ngrp - 1 - g : g;
            if (own) KP[gi * K] = kx;
#pragma unroll
            for (int k = 0; k < kGrp64; k++) {
                const int i = gi * kGrp64 + (up ? kGrp64 - 1 - k : k);
                if (own && i < n) P[i * K] = x;
                const double xn = fma(fma(-s, t.fi[up ? max(i - 1, 0) : i], pf[i]), x, pb[i] * xp);
                xp = x;
                x = i < n ? xn : x;
            }
            int ex;
            const double sx = exp_scale(fmax(fabs(x), fabs(xp)), &ex);
            x *= sx;
            xp *= sx;
            kx += ex;
        }
    }
    __syncwarp(tm.mask);
    // the twist: log2 |x_r y_r| to 0.1 from the high words; kB groups' loads at a time, without branches
    constexpr int kB = 4;
    int r = 0, best = INT_MIN;
    for (int g0 = tm.sub; g0 < ngrp; g0 += kB * tm.size) {
        int l[kB * kGrp64], kg[kB];
#pragma unroll
        for (int u = 0; u < kB; u++) {
            const int g = min(g0 + u * tm.size, ngrp - 1);
            kg[u] = (KX[g * K] + KY[g * K]) << 10;
        }
#pragma unroll
        for (int k = 0; k < kB * kGrp64; k++) {
            const size_t o = (size_t)min((g0 + k / kGrp64 * tm.size) * kGrp64 + k % kGrp64, n - 1) * K;
            l[k] = ((__double2hiint(X[o]) & 0x7fffffff) >> 10) + ((__double2hiint(Y[o]) & 0x7fffffff) >> 10);
        }
#pragma unroll
        for (int k = 0; k < kB * kGrp64; k++) {
            const int v = l[k] + kg[k / kGrp64], i = (g0 + k / kGrp64 * tm.size) * kGrp64 + k % kGrp64;
            if (i < n && v > best) {
                best = v;
                r = i;
            }
        }
    }
    tm.best(&best, &r);
    // entries above and below r relative to it
    const double xr = 1.0 / X[r * K], yr = 1.0 / Y[r * K];
    const int kxr = KX[(r / kGrp64) * K], kyr = KY[(r / kGrp64) * K];
    double gamma = d[r] * inv - s;
    if (r > 0) gamma -= fabs(e[r - 1]) * inv * (X[(r - 1) * K] * xr * pow2i(KX[((r - 1) / kGrp64) * K] - kxr));
    if (r + 1 < n) gamma -= fabs(e[r]) * inv * (Y[(r + 1) * K] * yr * pow2i(KY[((r + 1) / kGrp64) * K] - kyr));
    double nz = 0.0;
    for (int g0 = tm.sub; g0 < ngrp; g0 += kB * tm.size) {
        double v[kB * kGrp64], fx[kB], fy[kB];
#pragma unroll
        for (int u = 0; u < kB; u++) {
            const int g = min(g0 + u * tm.size, ngrp - 1);
            fx[u] = pow2i(KX[g * K] - kxr);
            fy[u] = pow2i(KY[g * K] - kyr);
        }
#pragma unroll
        for (int k = 0; k < kB * kGrp64; k++) {
            const int i = min((g0 + k / kGrp64 * tm.size) * kGrp64 + k % kGrp64, n - 1);
            v[k] = (i < r ? X : Y)[(size_t)i * K];
        }
#pragma unroll
        for (int u = 0; u < kB; u++) {
            fx[u] *= xr;
            fy[u] *= yr;
        }
#pragma unroll
        for (int k = 0; k < kB * kGrp64; k++) {
            const int i = (g0 + k / kGrp64 * tm.size) * kGrp64 + k % kGrp64;
            const double zi = v[k] * (i < r ? fx[k / kGrp64] : fy[k / kGrp64]);
            nz = fma(zi, i < n && i != r ? zi : 0.0, nz);
        }
    }
    nz = 1.0 + tm.sum(nz);
    *r_out = r;
    *nz_out = nz;
    return gamma / nz;
}

// The first step of the iteration in double-FP32: the same solutions from both ends (exponents per
// kGrpDf rows), the twist row r, |z|^2 there in FP32 (it only scales the correction) and the
// correction.  tb: the rows of the recurrence from the bottom.
constexpr int kGrpDf = 2;
struct RowsDfB {
    const float2 *f, *b;  // d/|e_{i-1}|, -|e_i|/|e_{i-1}| (1/|e_{i-1}| is RowsDf::g[i-1])
};
__device__ __forceinline__ df rescaled(df v, float sc) { return df{v.h * sc, v.l * sc}; }
__device__ __forceinline__ float exp_scale(df a, df b, int* e) {
    const unsigned h = __float_as_uint(fmaxf(fabsf(a.h), fabsf(b.h))) & 0x7f800000u;
    *e = (int)(h >> 23) - 127;
    return __uint_as_float(0x7f000000u - h);
}
// d_r - s - |e_{r-1}| x_{r-1}/x_r - |e_r| y_{r+1}/y_r, the ratios given
__device__ __forceinline__ double gamma_of(int n, const double* d, const double* e, double inv, double s, int r, double tx,
                                           double ty) {
    double g = d[r] * inv - s;
    if (r > 0) g -= fabs(e[r - 1]) * inv * tx;
    if (r + 1 < n) g -= fabs(e[r]) * inv * ty;
    return g;
}
__device__ double rq_first(const Team& tm, int n, const RowsDf& t, const RowsDfB& tb, const double* __restrict__ d,
                           const double* __restrict__ e, double inv, double s, const VecArgs& a, int col, int* r_out,
                           double* nz_out) {
    const size_t K = (size_t)a.ktot;
    float2* X = reinterpret_cast<float2*>(a.X) + col;
    float2* Y = reinterpret_cast<float2*>(a.Y) + col;
    const int ngrp = (n + kGrpDf - 1) / kGrpDf;
    int* KX = a.KX + col;
    int* KY = KX + (size_t)ngrp * K;
    {
        const bool up = tm.sub & 1, own = tm.sub < 2;
        const float2 *pf = up ? tb.f : t.f, *pb = up ? tb.b : t.b;
        float2* P = up ? Y : X;
        int* KP = up ? KY : KX;
        const df ms = df_from(-s);
        df x{1.f, 0.f}, xp{0.f, 0.f};
        int kx = 0;
#pragma unroll 2
        for (int g = 0; g < ngrp; g++) {
            const int gi = up ? ngrp - 1 - g : g;
            if (own) KP[gi * K] = kx;
#pragma unroll
            for (int k = 0; k < kGrpDf; k++) {
                const int i = gi * kGrpDf + (up ? kGrpDf - 1 - k : k);
                if (own && i < n) P[i * K] = df_pack(x);
                const df xn = df_fma(df_mul(df_unpack(pb[i]), xp),
                                     df_fma(df_unpack(pf[i]), ms, df_unpack(t.g[up ? max(i - 1, 0) : i])), x);
                xp = x;
                if (i < n) x = xn;
            }
            int ex;
            const float sx = exp_scale(x, xp, &ex);
            x = rescaled(x, sx);
            xp = rescaled(xp, sx);
            kx += ex;
        }
    }
    __syncwarp(tm.mask);
    constexpr int kB = 32;  // rows' loads at a time, without branches
    int r = 0, best = INT_MIN;
    for (int i0 = tm.sub; i0 < n; i0 += kB * tm.size) {
        int l[kB];
#pragma unroll
        for (int k = 0; k < kB; k++) {
            const int i = min(i0 + k * tm.size, n - 1);
            const size_t o = (size_t)i * K, og = (size_t)(i / kGrpDf) * K;
            l[k] = ((KX[og] + KY[og]) << 10) + ((__float_as_int(X[o].x) & 0x7fffffff) >> 13) +
                   ((__float_as_int(Y[o].x) & 0x7fffffff) >> 13);
        }
#pragma unroll
        for (int k = 0; k < kB; k++)
            if (i0 + k * tm.size < n && l[k] > best) {
                best = l[k];
                r = i0 + k * tm.size;
            }
    }
    tm.best(&best, &r);
    auto pow2f = [](int k) { return k < -126 ? 0.f : __int_as_float((min(k, 126) + 127) << 23); };
    const int kxr = KX[(r / kGrpDf) * K], kyr = KY[(r / kGrpDf) * K];
    const float xr = 1.0f / X[r * K].x, yr = 1.0f / Y[r * K].x;
    float nz = 0.f;
    for (int i0 = tm.sub; i0 < n; i0 += kB * tm.size) {
        float v[kB], f[kB];
#pragma unroll
        for (int k = 0; k < kB; k++) {
            const int i = min(i0 + k * tm.size, n - 1);
            const bool top = i < r;
            v[k] = (top ? X : Y)[(size_t)i * K].x;
            f[k] = pow2f((top ? KX : KY)[(size_t)(i / kGrpDf) * K] - (top ? kxr : kyr));
        }
#pragma unroll
        for (int k = 0; k < kB; k++) {
            const int i = i0 + k * tm.size;
            const float zi = v[k] * (i < r ? xr : yr) * f[k];
            if (i < n && i != r) nz = fmaf(zi, zi, nz);
        }
    }
    const double nzs = 1.0 + tm.sum((double)nz);
    double tx = 0.0, ty = 0.0;
    if (r > 0)
        tx = df_to(df_unpack(X[(r - 1) * K])) / df_to(df_unpack(X[r * K])) * pow2i(KX[((r - 1) / kGrpDf) * K] - kxr);
    if (r + 1 < n)
        ty = df_to(df_unpack(Y[(r + 1) * K])) / df_to(df_unpack(Y[r * K])) * pow2i(KY[((r + 1) / kGrpDf) * K] - kyr);
    *r_out = r;
    *nz_out = nzs;
    return gamma_of(n, d, e, inv, s, r, tx, ty) / nzs;
}

// gamma_r at s for a given twist row: even lanes the solution from the top down to r, odd lanes the
// one from the bottom up to r, in double-FP32; nothing is stored.
__device__ double gamma_df(const Team& tm, int n, const RowsDf& t, const RowsDfB& tb, const double* __restrict__ d,
                           const double* __restrict__ e, double inv, double s, int r) {
    const bool up = tm.sub & 1;
    const float2 *pf = up ? tb.f : t.f, *pb = up ? tb.b : t.b, *pg = up ? t.g - 1 : t.g;
    const int i0 = up ? n - 1 : 0, di = up ? -1 : 1, steps = up ? n - 1 - r : r;
    const df ms = df_from(-s);
    df x{1.f, 0.f}, xp{0.f, 0.f};
#pragma unroll 4
    for (int q = 0; q < steps; q++) {
        const int i = i0 + di * q;
        const df y = df_fma(df_mul(df_unpack(pb[i]), xp), df_fma(df_unpack(pf[i]), ms, df_unpack(pg[i])), x);
        int ex;
        const float sc = exp_scale(y, x, &ex);
        xp = rescaled(x, sc);
        x = rescaled(y, sc);
    }
    __syncwarp(tm.mask);
    const double ratio = steps > 0 ? df_to(xp) / df_to(x) : 0.0;
    return gamma_of(n, d, e, inv, s, r, tm.from(ratio, 0), tm.from(ratio, 1));
}

// The rows of the recurrences of every block, five FP64 arrays and their double-FP32 pairs, each of
// np = n rounded up to kGrp64 entries: Rows64's ff, fi, fb, bf, bb, then RowsDf's and RowsDfB's f, g,
// b, f, b; last, the distance of each approximate eigenvalue to its nearer neighbour.
constexpr int kRowArrays = 11;
__global__ void rows_kernel(int n, int nblk, const double* __restrict__ dg, const double* __restrict__ eg,
                            const double* __restrict__ scale, const double* __restrict__ w, double* __restrict__ R) {
    const int np = round_up(n, kGrp64);
    constexpr double kMinE = 8.673617379884035e-19;  // 2^-60
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < np * nblk; t += gridDim.x * blockDim.x) {
        const int b = t / np, i = t % np;
        const double inv = 1.0 / scale[b];
        const double* dgb = dg + (size_t)b * n;
        const double* egb = eg + (size_t)b * n;
        double* r = R + (size_t)b * kRowArrays * np;
        double v[5] = {1.0, 0.0, 0.0, 0.0, 0.0};  // rows past the end keep x
        if (i < n) {
            const double d = dgb[i] * inv;
            const double e = i + 1 < n ? fmax(fabs(egb[i] * inv), kMinE) : 1.0;
            const double ep = i > 0 ? fmax(fabs(egb[i - 1] * inv), kMinE) : 1.0;
            v[1] = 1.0 / e;
            v[0] = d * v[1];
            v[2] = i > 0 ? -ep * v[1] : 0.0;
            v[3] = d / ep;
            v[4] = i + 1 < n ? -e / ep : 0.0;
        }
        if (i < n) {
            const double* wb = w + (size_t)b * n;
            const double down = i > 0 ? fabs(wb[i] - wb[i - 1]) : HUGE_VAL, up = i + 1 < n ? fabs(wb[i + 1] - wb[i]) : HUGE_VAL;
            r[10 * np + i] = fmin(down, up) * inv;
        }
        float2* f = reinterpret_cast<float2*>(r + 5 * np);
        for (int q = 0; q < 5; q++) r[q * np + i] = v[q];
        f[i] = df_pack(df_from(v[0]));
        f[np + i] = df_pack(df_from(v[1]));
        f[2 * np + i] = df_pack(df_from(v[2]));
        f[3 * np + i] = df_pack(df_from(v[3]));
        f[4 * np + i] = df_pack(df_from(v[4]));
    }
}

// grid (nblk, parts of kc), 4 warps of `per` candidates each, a team of lanes per candidate: candidate c
// (0 = largest) of block b.  An FP64 instruction takes a warp 64 cycles of its scheduler's pipe however
// many of its lanes work, so the candidates are dealt over all schedulers of the chip, and the lanes left
// over share a candidate: two directions of a solution, a shift of a Sturm count each, rows of the scans.
// The FP32 estimate's bracket is confirmed by double-FP32 Sturm counts.  An eigenvalue alone in
// its bracket is refined by Rayleigh-quotient iteration on twisted factorisations (cubic
// convergence; the iterate must stay in the bracket); an eigenvalue sharing its bracket is
// narrowed down first.  The last twisted factorisation gives the vector.
// Bound by the FP64 pipe (64 cycles an instruction, measured, with nothing to overlap) and by loads of the stored solutions (32 rows at a time: row by row their latency was half the kernel).
// Candidates of 34 blocks of 512^2 (4,351): 4.51 -> 1.15 ms against FP64 pivots with a division in
// every row; 34 of 1024^2 25.5 -> 3.77, 10 of 555^2 12.5 -> 2.01, 18 of 64^2 0.406 -> 0.092; with the lanes in teams
// 34 of 512^2 0.90 -> 0.46, 10 of 555^2 0.98 -> 0.46, one of 1728^2 5.11 -> 1.70, of 3150^2 6.05 -> 2.66.
// LOCAL: the block's rows in shared memory; otherwise (orders whose rows do not fit) read through L1.
template <bool LOCAL>
__global__ void __launch_bounds__(128) vectors_kernel(VecArgs a, const double* __restrict__ R, int per, int team) {
    extern __shared__ double rows64[];
    __shared__ unsigned flips[kMaxRows / 32];           // row i: whether entries i and i + 1 change sign by T's e_i
    __shared__ unsigned char before[kMaxRows / 32];  // parity of the words before
    const int b = blockIdx.x, n = a.n, np = round_up(n, kGrp64);
    const int kc = a.kc[b];
    if ((int)blockIdx.y * 4 * per >= kc) return;
    const double sc = a.scale[b], inv = 1.0 / sc;
    const double* dgb = a.dg + (size_t)b * n;
    const double* egb = a.eg + (size_t)b * n;
    const double* rows = R + (size_t)b * kRowArrays * np;
    const double* gaps = rows + 10 * np;
    if (LOCAL) {
        for (int i = threadIdx.x; i < 10 * np; i += 128) rows64[i] = rows[i];
        rows = rows64;
        __syncthreads();
    }
    const Rows64 t{rows, rows + np, rows + 2 * np, rows + 3 * np, rows + 4 * np};
    const float2* rowsf = reinterpret_cast<const float2*>(rows + 5 * np);
    const RowsDf tf{rowsf, rowsf + np, rowsf + 2 * np};
    const RowsDfB tfb{rowsf + 3 * np, rowsf + 4 * np};
    const int lane = threadIdx.x & 31;
    for (int w = threadIdx.x >> 5; 32 * w < n; w += 4) {
        const int i = 32 * w + lane;
        const unsigned m = __ballot_sync(0xffffffffu, i + 1 < n && !(egb[i] < 0.0));
        if (lane == 0) flips[w] = m;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 0, p = 0; 32 * w < n; w++) {
            before[w] = (unsigned char)p;
            p ^= __popc(flips[w]) & 1;
        }
    __syncthreads();
    const int c = (blockIdx.y * 4 + (threadIdx.x >> 5)) * per + lane / team;
    if (lane / team >= per || c >= kc) return;
    const int tb0 = lane / team * team;
    const Team tm{(team == 32 ? ~0u : (1u << team) - 1) << tb0, team, lane - tb0, tb0};
    const int j = n - 1 - c;  // ascending index
    const int col = a.koff[b] + c;
    const size_t K = (size_t)a.ktot;
    const double x = a.w[(size_t)b * n + j] * inv;
    auto count_df = [&](double sh) { return sturm_df(np, tf, sh); };
    auto count64 = [&](double sh) { return sturm64(np, t, sh); };
    // the FP32 estimate's bracket, confirmed
    double del = 8.0 * FLT_EPSILON, lo = -1.0, hi = 1.0;  // the scaled spectrum lies inside (-1, 1)
    int clo = 0, chi = n;
    for (int k = 0; k < 8 && (lo == -1.0 || hi == 1.0); k++, del *= 8.0) {
        const double sh[2] = {x - del, x + del};
        const int own = count_df(sh[tm.sub & 1]), cn[2] = {tm.from(own, 0), tm.from(own, 1)};
        if (cn[0] <= j && sh[0] > lo) {
            lo = sh[0];
            clo = cn[0];
        }
        if (cn[1] > j && sh[1] < hi) {
            hi = sh[1];
            chi = cn[1];
        }
    }
    if (lo == -1.0 || hi == 1.0) atomicMax(&a.status[b], 1);
    double lam = x, nz = 1.0;
    int r = n - 1;
    bool done = false;
    // a bracket holding several eigenvalues is narrowed until it holds this one alone: in double-FP32
    // down to well above its rounding, then in FP64
    for (int it = 0; it < 40 && chi - clo > 1 && hi - lo > 1e-12; it++)
        if (!narrow(tm, count_df, j, &lo, &hi, &clo, &chi)) break;
    if (chi - clo > 1) {
        lo -= 1e-13;  // a double-FP32 count may be off this close to an eigenvalue
        hi += 1e-13;
        const int own = count64(tm.sub & 1 ? hi : lo);
        clo = tm.from(own, 0);
        chi = tm.from(own, 1);
        for (int it = 0; it < 40 && chi - clo > 1 && hi - lo > 4.0 * DBL_EPSILON; it++)
            if (!narrow(tm, count64, j, &lo, &hi, &clo, &chi)) break;
    }
    if (chi - clo == 1) {
        // Converged when the correction is below 1e-14 of the block scale (T is scaled to norm < 1) and
        // 1e-10 of the distance to the next eigenvalue: the vector is that of the shift before the
        // correction, off by their quotient (left to the polish where there is one: 0.12 ms at 1,728
        // rows); or when it stops shrinking at the rounding of gamma.  One that stops shrinking above
        // that, between eigenvalues some 1e-10 apart, is bracketed by Sturm counts instead.
        const double tol = a.polished ? 1e-14 : fmin(1e-14, fmax(0.5 * DBL_EPSILON, 1e-10 * gaps[j]));
        double s = fmin(fmax(x, lo), hi), prev = 1.0;
        {
            // most of the way in double-FP32, at one twist row: an FP64 step costs four times as much
            double s1 = s, dl = rq_first(tm, n, tf, tfb, dgb, egb, inv, s, a, col, &r, &nz), pl = 1.0;
            for (int it = 0;; it++) {
                s1 += dl;
                if (!(s1 > lo && s1 < hi) || it == 4 || !(fabs(dl) < pl)) break;
                s = s1;
                if (fabs(dl) <= 1e-13) break;
                pl = fabs(dl);
                dl = gamma_df(tm, n, tf, tfb, dgb, egb, inv, s, r) / nz;
            }
        }
        // FP64 from there; an iterate that left the bracket starts again from the bracket narrowed to
        // double-FP32's resolution
        for (int att = 0; att < 2 && !done; att++) {
            if (att) {
                for (int it = 0; it < 40 && hi - lo > 1e-12; it++)
                    if (!narrow(tm, count_df, j, &lo, &hi, &clo, &chi)) break;
                lo -= 1e-13;
                hi += 1e-13;
                s = 0.5 * (lo + hi);
                prev = 1.0;
            }
            for (int it = 0; it < 8; it++) {
                const double dl = rq_step(tm, n, t, dgb, egb, inv, s, a, col, &r, &nz);
                const double s1 = s + dl;
                if (!(s1 > lo && s1 < hi)) break;  // left the bracket
                if (fabs(dl) <= tol || (fabs(dl) <= 16.0 * DBL_EPSILON && fabs(dl) > 0.25 * prev)) {
                    lam = s1;
                    done = true;  // the stored solutions belong to s
                    break;
                }
                prev = fabs(dl);
                s = s1;
            }
        }
    }
    if (!done) {
        for (int it = 0; it < 48 && hi - lo > 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + 1e-300; it++)
            if (!narrow(tm, count64, j, &lo, &hi, &clo, &chi)) break;
        lam = 0.5 * (lo + hi);
        rq_step(tm, n, t, dgb, egb, inv, lam, a, col, &r, &nz);
    }
    if (tm.sub == 0) a.w[(size_t)b * n + j] = lam * sc;
    const double s = 1.0 / sqrt(nz);
    if (!isfinite(s) || !(s > 0.0)) atomicMax(&a.status[b], 3);
    // the vector, normalised, with the signs of T's own off-diagonals (entry r positive)
    const int ngrp = (n + kGrp64 - 1) / kGrp64;
    const int* KX = a.KX + col;
    const int* KY = KX + (size_t)ngrp * K;
    const double* X = a.X + col;
    const double* Y = a.Y + col;
    const double xr = s / X[r * K], yr = s / Y[r * K];
    const int kxr = KX[(r / kGrp64) * K], kyr = KY[(r / kGrp64) * K];
    // parity of the sign flips above row i
    auto parity = [&](int i) { return before[i >> 5] ^ (__popc(flips[i >> 5] & ((1u << (i & 31)) - 1)) & 1); };
    const int pr = parity(r);
    constexpr int kU = 4;  // groups loaded at a time
    for (int g0 = tm.sub; g0 < ngrp; g0 += kU * team) {
        double v[kU * kGrp64], fx[kU], fy[kU];
#pragma unroll
        for (int u = 0; u < kU; u++) {
            const int g = min(g0 + u * team, ngrp - 1);
            fx[u] = xr * pow2i(KX[g * K] - kxr);
            fy[u] = yr * pow2i(KY[g * K] - kyr);
        }
#pragma unroll
        for (int k = 0; k < kU * kGrp64; k++) {
            const int i = (g0 + k / kGrp64 * team) * kGrp64 + k % kGrp64;
            v[k] = i < n ? (i < r ? X : Y)[i * K] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < kU * kGrp64; k++) {
            const int i = (g0 + k / kGrp64 * team) * kGrp64 + k % kGrp64;
            if (i < n) {
                const double zi = v[k] * (i < r ? fx[k / kGrp64] : fy[k / kGrp64]);
                a.Z[i * K + col] = parity(i) != pr ? -zi : zi;
            }
        }
    }
}

// Gram-Schmidt, twice, inside clusters of close candidates: grid (nblk, kmax), the CTA of a
// cluster's first candidate takes the cluster.
__global__ void __launch_bounds__(256) cluster_kernel(VecArgs a, double tol) {
    __shared__ double red[40];
    const int b = blockIdx.x, n = a.n, kc = a.kc[b], start = blockIdx.y;
    const size_t K = (size_t)a.ktot;
    const double* wb = a.w + (size_t)b * n;
    const double sc = a.scale[b];
    const int c0 = a.koff[b];
    // wb is ascending: candidate c has index n-1-c
    auto close = [&](int c) { return wb[n - c] - wb[n - 1 - c] < tol * sc; };  // candidates c-1 and c
    if (start + 1 >= kc || !close(start + 1) || (start > 0 && close(start))) return;
    for (int c = start + 1; c < kc && close(c); c++) {
        for (int pass = 0; pass < 2; pass++) {
            for (int k = start; k < c; k++) {
                double s = 0.0;
                for (int i = threadIdx.x; i < n; i += blockDim.x) s += a.Z[i * K + c0 + k] * a.Z[i * K + c0 + c];
                const double dot = cta_sum(s, red);
                for (int i = threadIdx.x; i < n; i += blockDim.x) a.Z[i * K + c0 + c] -= dot * a.Z[i * K + c0 + k];
                __syncthreads();
            }
            double s = 0.0;
            for (int i = threadIdx.x; i < n; i += blockDim.x) s += a.Z[i * K + c0 + c] * a.Z[i * K + c0 + c];
            const double nrm = sqrt(cta_sum(s, red));
            if (pass == 0 && nrm < 1e-2 && threadIdx.x == 0) atomicMax(&a.status[b], 2);
            const double inv = nrm > 0.0 ? 1.0 / nrm : 0.0;
            for (int i = threadIdx.x; i < n; i += blockDim.x) a.Z[i * K + c0 + c] *= inv;
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------- back-transformation
// x = H_0 H_1 ... H_{n-3} z.  Reflectors are applied kR at a time, H_c .. H_{c+kR-1} = I - V T V^T
// (the compact form of Schreiber and Van Loan, SIAM J. Sci. Stat. Comput. 10 (1989) 53): one pass
// over the rows forms V^T z, a kR x kR product and one pass subtracts V (T V^T z).
constexpr int kR = 4;
constexpr int kT = kR * (kR + 1) / 2;  // T's upper triangle, column by column

__device__ __forceinline__ df shfl_df(df x, int src) {
    return df{__shfl_sync(0xffffffffu, x.h, src), __shfl_sync(0xffffffffu, x.l, src)};
}
__device__ __forceinline__ df shfl_xor_df(df x, int o) {
    return df{__shfl_xor_sync(0xffffffffu, x.h, o), __shfl_xor_sync(0xffffffffu, x.l, o)};
}
// acc + x y, the low parts only added up (renormalised where the sum is used)
__device__ __forceinline__ df df_mac(df acc, df x, df y) {
    const float p = __fmul_rn(x.h, y.h);
    float e = fmaf(x.h, y.h, -p);
    e = fmaf(x.h, y.l, e);
    e = fmaf(x.l, y.h, e);
    float t;
    const float s = two_sum(acc.h, p, t);
    return df{s, acc.l + (t + e)};
}

// T of every group of kR reflectors: one warp each.  Reflectors past the last (n - 3) become zero
// rows (the last group of a block may end at row n).  V row c: zero from its group's first row to c and
// past n - 1 (tridiag.cu), then v.
__global__ void __launch_bounds__(128) compact_kernel(int n, int nblk, float4* __restrict__ Vall,
                                                      const double* __restrict__ tau, float2* __restrict__ T) {
    const int ngrp = (n - 2 + kR - 1) / kR, lane = threadIdx.x & 31;
    const int w = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (w >= ngrp * nblk) return;
    const int b = w / ngrp, c0 = (w % ngrp) * kR;
    const int vs = (n + 1) / 2;
    float4* V = Vall + (size_t)b * ((n + 3) & ~3) * vs;
    df tv[kR], g[kR][kR];
#pragma unroll
    for (int q = 0; q < kR; q++) {
        tv[q] = c0 + q <= n - 3 ? df_from(tau[(size_t)b * n + c0 + q]) : df{0.f, 0.f};
#pragma unroll
        for (int p = 0; p < kR; p++) g[p][q] = df{0.f, 0.f};
    }
    for (int i = c0 / 2 + lane; i < vs; i += 32) {
        df v[kR][2];
#pragma unroll
        for (int q = 0; q < kR; q++) {
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c0 + q <= n - 3)
                x = V[(size_t)(c0 + q) * vs + i];
            else
                V[(size_t)(c0 + q) * vs + i] = x;
            v[q][0] = df{x.x, x.z};
            v[q][1] = df{x.y, x.w};
        }
#pragma unroll
        for (int q = 1; q < kR; q++)
#pragma unroll
            for (int p = 0; p < q; p++) g[p][q] = df_mac(df_mac(g[p][q], v[p][0], v[q][0]), v[p][1], v[q][1]);
    }
#pragma unroll
    for (int q = 1; q < kR; q++)
#pragma unroll
        for (int p = 0; p < q; p++)
#pragma unroll
            for (int o = 16; o; o >>= 1) g[p][q] = df_add(g[p][q], shfl_xor_df(g[p][q], o));
    // T_qq = tau_q, T_pq = -tau_q sum_{p <= k < q} T_pk g_kq
    df t[kR][kR];
#pragma unroll
    for (int q = 0; q < kR; q++) {
        t[q][q] = tv[q];
#pragma unroll
        for (int p = 0; p < q; p++) {
            df s{0.f, 0.f};
#pragma unroll
            for (int k = p; k < q; k++) s = df_fma(s, t[p][k], g[k][q]);
            t[p][q] = df_mul(df{-tv[q].h, -tv[q].l}, s);
        }
    }
    if (lane == 0) {
        float2* o = T + (size_t)w * kT;
#pragma unroll
        for (int q = 0; q < kR; q++)
#pragma unroll
            for (int p = 0; p <= q; p++) o[q * (q + 1) / 2 + p] = df_pack(t[p][q]);
    }
}

// NV candidates of block b per warp, their rows in the warp's shared memory; warps work alone (no
// barriers).  The reflectors come from L2 twice per group, as one stream of asynchronous copies
// kPipe steps ahead (each lane copies what it will read), which runs on over the ends of passes and
// groups: with plain loads every step of 32 rows waited for L2.  More vectors a warp read the
// reflectors less often, fewer keep more warps in flight (launch_blockeig_vectors); the CTAs of a
// block are neighbours, so that its reflectors stay in L2.  Writes candidate c in FP64: as column
// n-1-c of the block (ascending order, column-major), or, with rows set, as row c of out while c <
// rows.
constexpr int kPipe = 4;
constexpr int kRing = kPipe * kR * 32;  // 16-byte pairs per warp
template <int NV>
__global__ void __launch_bounds__(128) backtransform_kernel(VecArgs a, const float4* __restrict__ Vall,
                                                            const float2* __restrict__ Tall, double* __restrict__ out,
                                                            int rows) {
    extern __shared__ float4 zsm[];
    const int b = blockIdx.y, n = a.n, kc = a.kc[b], vs = (n + 1) / 2;
    const int W = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = (blockIdx.x * W + warp) * NV;
    if (c0 >= kc) return;
    float4* ring = zsm + (size_t)warp * (kRing + NV * vs) + lane;  // [kPipe][kR][32], this lane's slots
    float4* z = zsm + (size_t)warp * (kRing + NV * vs) + kRing;    // [NV][vs], (hi, hi, lo, lo) of two rows
    const size_t K = (size_t)a.ktot;
    const int nv = min(NV, kc - c0);
    for (int i = lane; i < vs; i += 32) {
        const double* src = a.Z + (size_t)2 * i * K + a.koff[b] + c0;
#pragma unroll
        for (int v = 0; v < NV; v++) {
            const df x = df_from(v < nv ? src[v] : 0.0), y = df_from(v < nv && 2 * i + 1 < n ? src[K + v] : 0.0);
            z[v * vs + i] = make_float4(x.h, y.h, x.l, y.l);
        }
    }
    __syncwarp();
    const float4* V = Vall + (size_t)b * ((n + 3) & ~3) * vs;
    const int ngrp = (n - 2 + kR - 1) / kR;
    constexpr int NS = NV * kR;  // sums a group: (vector, reflector)
    // the stream: groups downwards, each twice, row pairs r0 / 2 + lane, + 32, ...
    int sg = ngrp - 1, sp = 0, si = 0, slot = 0;  // next step to issue: group, pass, offset
    auto issue = [&]() {
        if (sg >= 0) {
            const int i = sg * (kR / 2) + si + lane;
            if (i < vs) {
                const float4* src = V + (size_t)(sg * kR) * vs + i;
#pragma unroll
                for (int q = 0; q < kR; q++) {
                    const unsigned dst = (unsigned)__cvta_generic_to_shared(ring + (slot * kR + q) * 32);
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + (size_t)q * vs) : "memory");
                }
            }
            si += 32;
            if (sg * (kR / 2) + si >= vs) {
                si = 0;
                sg -= sp;
                sp ^= 1;
            }
        }
        slot = slot + 1 == kPipe ? 0 : slot + 1;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int k = 0; k < kPipe - 1; k++) issue();
    int rd = 0;
    auto load = [](const float4* p) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(p);
        return df2{t.x, t.y};
    };
    auto step = [&](df2 (&v)[kR]) {  // the next step's reflector entries
        asm volatile("cp.async.wait_group %0;" ::"n"(kPipe - 2) : "memory");
#pragma unroll
        for (int q = 0; q < kR; q++) v[q] = load(ring + (rd * kR + q) * 32);
        rd = rd + 1 == kPipe ? 0 : rd + 1;
        issue();
    };
    const f2 minus = pk(-1.f, -1.f);
    for (int g = ngrp - 1; g >= 0; g--) {
        const int r0 = g * (kR / 2);
        df2 ac2[NS];
#pragma unroll
        for (int k = 0; k < NS; k++) ac2[k] = df2{0, 0};
        for (int i0 = r0; i0 < vs; i0 += 32) {
            const int i = i0 + lane;
            df2 v[kR];
            step(v);
            if (i < vs) {
#pragma unroll
                for (int u = 0; u < NV; u++) {
                    const df2 x = load(z + u * vs + i);
                    const f2 nx = mul2(x.h, minus);
#pragma unroll
                    for (int q = 0; q < kR; q++) ac2[u * kR + q] = df2_mac(ac2[u * kR + q], v[q], x.h, x.l, nx);
                }
            }
        }
        df acc[NS];
#pragma unroll
        for (int k = 0; k < NS; k++) {
            df x, y;
            upk(ac2[k].h, &x.h, &y.h);
            upk(ac2[k].l, &x.l, &y.l);
            acc[k] = df_add(x, y);
        }
        // sum over the lanes, halving the sums held: lane l ends with sum l / (32 / NS)
        int o = 16;
#pragma unroll
        for (int h = NS / 2; h >= 1; h /= 2, o /= 2) {
            const bool up = lane & o;
#pragma unroll
            for (int k = 0; k < h; k++) {
                const df keep = up ? acc[k + h] : acc[k], give = up ? acc[k] : acc[k + h];
                acc[k] = df_add(keep, shfl_xor_df(give, o));
            }
        }
#pragma unroll
        for (int e = 16 / NS; e; e >>= 1) acc[0] = df_add(acc[0], shfl_xor_df(acc[0], e));
        // f = T d: this lane's row p of its vector u
        constexpr int kL = 32 / NS;  // lanes per sum
        const int mine = lane / kL, u0 = mine / kR, p0 = mine % kR;
        const float2* Tg = Tall + ((size_t)b * ngrp + g) * kT;
        df f{0.f, 0.f};
#pragma unroll
        for (int q = 0; q < kR; q++) {
            const df d = shfl_df(acc[0], (u0 * kR + q) * kL);
            if (q >= p0) f = df_fma(f, df_unpack(__ldg(Tg + q * (q + 1) / 2 + p0)), d);
        }
        f2 fh[NS], fl[NS], nfh[NS];  // -f, and its high part's negative
#pragma unroll
        for (int k = 0; k < NS; k++) {
            const df t = shfl_df(f, k * kL);
            fh[k] = pk(-t.h, -t.h);
            fl[k] = pk(-t.l, -t.l);
            nfh[k] = pk(t.h, t.h);
        }
        for (int i0 = r0; i0 < vs; i0 += 32) {
            const int i = i0 + lane;
            df2 v[kR];
            step(v);
            if (i < vs) {
#pragma unroll
                for (int u = 0; u < NV; u++) {
                    df2 x = load(z + u * vs + i);
#pragma unroll
                    for (int q = 0; q < kR; q++) x = df2_mac(x, v[q], fh[u * kR + q], fl[u * kR + q], nfh[u * kR + q]);
                    const f2 h = add2(x.h, x.l);
                    *reinterpret_cast<ulonglong2*>(z + u * vs + i) = make_ulonglong2(h, sub2(x.l, sub2(h, x.h)));
                }
            }
        }
        __syncwarp();  // a lane's rows shift by kR from group to group
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    for (int u = 0; u < nv; u++) {
        if (rows > 0 && c0 + u >= rows) break;
        double* o = rows > 0 ? out + (size_t)(c0 + u) * n : out + (size_t)b * n * n + (size_t)(n - 1 - (c0 + u)) * n;
        for (int i = lane; i < vs; i += 32) {
            const float4 x = z[u * vs + i];
            o[2 * i] = (double)x.x + (double)x.z;
            if (2 * i + 1 < n) o[2 * i + 1] = (double)x.y + (double)x.w;
        }
    }
}

// ---------------------------------------------------------------- polish of a dense solve
// E of X <- X (I + E) and the Rayleigh quotients, from G = X^T X and H = X^T S X (Ogita and Aishima,
// Japan J. Indust. Appl. Math. 35 (2018) 1007): with R = I - G, E = R / 2 + K off the diagonal, K_ij =
// (H_ij + (l_i + l_j) R_ij / 2) / (l_j - l_i) the couplings, and E_jj = R_jj / 2 - sum_i K_ij^2 / 2, which keeps
// the norms to second order.  Counted are the vectors for which that is not enough (polish.h, which takes
// them): a coupling above kCloseCoupling that is not rounding, or two with a product above kCloseProduct.
// One warp a column; the k - m columns past the last only count, their couplings to the first m.
__global__ void __launch_bounds__(128) polish_kernel(int k, int m, const double* __restrict__ G, const double* __restrict__ H,
                                                     double* __restrict__ E, double* __restrict__ lam, int* close) {
    const int lane = threadIdx.x & 31;
    const double rounding = kCouplingRounding * fabs(H[0] / G[0]);
    for (int j = blockIdx.x * 4 + (threadIdx.x >> 5); j < k; j += gridDim.x * 4) {
        const double gj = G[(size_t)j * k + j], lj = H[(size_t)j * k + j] / gj;
        double s2 = 0.0, a1 = 0.0, a2 = 0.0;  // sum of squares, the two largest
        bool over = !isfinite(lj);
        for (int i = lane; i < (j < m ? k : m); i += 32) {
            if (i == j) continue;
            const size_t o = i >= j ? (size_t)j * k + i : (size_t)i * k + j;  // lower triangles
            const double g = G[o], li = H[(size_t)i * k + i] / G[(size_t)i * k + i];
            const double h = H[o] - 0.5 * (li + lj) * g, d = lj - li;
            double v = 0.0;
            if (!(fabs(h) <= kCloseCoupling * fabs(d)))
                over |= !(fabs(h) <= rounding);
            else if (d != 0.0)
                v = h / d;
            s2 = fma(v, v, s2);
            a2 = fmax(a2, fmin(a1, fabs(v)));
            a1 = fmax(a1, fabs(v));
            if (j < m) E[(size_t)j * k + i] = v - 0.5 * g;
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            const double b1 = __shfl_xor_sync(0xffffffffu, a1, o), b2 = __shfl_xor_sync(0xffffffffu, a2, o);
            a2 = fmax(fmax(a2, b2), fmin(a1, b1));
            a1 = fmax(a1, b1);
        }
        over = __any_sync(0xffffffffu, over) || a1 * a2 > kCloseProduct;
        if (lane) continue;
        if (j < m) {
            E[(size_t)j * k + j] = 0.5 * (1.0 - gj - s2);
            lam[j] = lj;
        }
        if (over) atomicAdd(close, 1);
    }
}

template <int NV>
void launch_back(const VecArgs& a, const BlockEigVectors& p, int warps, cudaStream_t s) {
    auto k = backtransform_kernel<NV>;
    const size_t per = sizeof(float4) * (kRing + (size_t)NV * ((p.n + 1) / 2));
    OPSEC_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dynamic_smem((const void*)k)));
    k<<<dim3((p.kmax + warps * NV - 1) / (warps * NV), p.nblk), 32 * warps, per * warps, s>>>(
        a, reinterpret_cast<const float4*>(p.V), reinterpret_cast<const float2*>(p.T), p.out, p.rows);
    OPSEC_CUDA(cudaGetLastError());
}

}  // namespace

void launch_polish_coefficients(int k, int m, const double* G, const double* H, double* E, double* lam, int* close,
                                cudaStream_t s, long long* launches) {
    polish_kernel<<<(unsigned)((k + 3) / 4), 128, 0, s>>>(k, m, G, H, E, lam, close);
    OPSEC_CUDA(cudaGetLastError());
    ++*launches;
}

size_t blockeig_reflector_doubles(int n) { return (size_t)((n + 3) & ~3) * ((n + 1) / 2) * 2; }  // whole groups of kR rows

size_t blockeig_rows_doubles(int n, int nblk) { return (size_t)kRowArrays * ((n + kGrp64 - 1) / kGrp64 * kGrp64) * nblk; }

size_t blockeig_compact_doubles(int n, int nblk) { return (size_t)((n - 2 + kR - 1) / kR) * nblk * kT; }

bool blockeig_supported(int n) { return n >= 3 && n <= kMaxN; }

void launch_blockeig_spectrum(int n, int nblk, const double* dg, const double* eg, double* w, double* scale,
                              cudaStream_t s, long long* launches) {
    const size_t smem = sizeof(float4) * (size_t)((n + kGrp32 - 1) / kGrp32 * kGrp32);
    auto run = [&](auto k, int lanes) {
        OPSEC_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dynamic_smem((const void*)k)));
        k<<<dim3(nblk, (n * lanes + 255) / 256), 256, smem, s>>>(n, dg, eg, w, scale);
    };
    // Eight lanes an eigenvalue do 2.8 times the work in a third of the steps: while the chip is not full
    // (18 blocks of 64^2 25 -> 14 us, 10 of 555^2 193 -> 102, one of 1728^2 585 -> 193, of 3150^2 1062 -> 350;
    // 34 of 512^2 178 and 176).
    if ((long long)n * nblk <= 16000)
        run(spectrum_kernel<8>, 8);
    else
        run(spectrum_kernel<2>, 1);
    OPSEC_CUDA(cudaGetLastError());
    ++*launches;
}

void launch_blockeig_vectors(const BlockEigVectors& p, cudaStream_t s, long long* launches) {
    VecArgs a{p.n, p.nblk, p.ktot, p.kc, p.koff, p.dg, p.eg, p.scale, p.w, p.Z, p.K, p.X, p.Y, p.rows > 0, p.status};
    int dev = 0, nsm = 0;
    OPSEC_CUDA(cudaGetDevice(&dev));
    OPSEC_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const int per = std::min(16, std::max(1, (p.ktot + 4 * nsm - 1) / (4 * nsm)));
    int team = 32;  // lanes a candidate
    while (team * per > 32) team /= 2;
    const dim3 grid(p.nblk, (p.kmax + 4 * per - 1) / (4 * per));
    if (g_clock) g_clock->begin("blockeig_pairs", s);
    const int np = (p.n + kGrp64 - 1) / kGrp64 * kGrp64;
    rows_kernel<<<(np * p.nblk + 127) / 128, 128, 0, s>>>(p.n, p.nblk, p.dg, p.eg, p.scale, p.w, p.R);
    OPSEC_CUDA(cudaGetLastError());
    const size_t rows = sizeof(double) * 10 * (size_t)np;
    const size_t room = (size_t)max_dynamic_smem((const void*)vectors_kernel<true>);
    if (rows <= room) {
        OPSEC_CUDA(cudaFuncSetAttribute(vectors_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room));
        vectors_kernel<true><<<grid, 128, rows, s>>>(a, p.R, per, team);
    } else {
        vectors_kernel<false><<<grid, 128, 0, s>>>(a, p.R, per, team);
    }
    OPSEC_CUDA(cudaGetLastError());
    if (g_clock) g_clock->end(s);
    cluster_kernel<<<dim3(p.nblk, p.kmax), 256, 0, s>>>(a, 1e-6);
    OPSEC_CUDA(cudaGetLastError());
    if (g_clock) g_clock->begin("blockeig_back", s, 2.0 * p.n * (double)p.n * p.ktot);
    const int groups = (p.n - 2 + kR - 1) / kR * p.nblk;
    compact_kernel<<<(groups + 3) / 4, 128, 0, s>>>(p.n, p.nblk, reinterpret_cast<float4*>(p.V), p.tau,
                                                    reinterpret_cast<float2*>(p.T));
    OPSEC_CUDA(cudaGetLastError());
    // Vectors per warp (times before the packed arithmetic; since, the ones taken: 10 blocks of 555^2 0.53,
    // 34 of 512^2 0.92, one of 1728^2 2.6, of 3150^2 11.7 ms, and the order of the choices is the same).
    // One while the warps do not fill the chip four times over (10 blocks of 555^2,
    // 1,390 vectors: 0.68 ms, two 0.84, four 1.07); two beyond (34 of 1024^2: 10.2 ms, four 13.4: a
    // warp's 40 KB leave five warps an SM); four where their rows still leave nine warps an SM and
    // reading the reflectors half as often counts (34 of 512^2, 4,351 vectors: 1.10 ms, two 1.43, one
    // 1.42; 66 of 256^2: two 0.35, four 0.41).
    const int cap = max_dynamic_smem((const void*)backtransform_kernel<4>);
    const size_t vec = sizeof(float4) * (size_t)((p.n + 1) / 2);
    auto warps_of = [&](int nv) { return (int)std::min<size_t>(4, (size_t)cap / (vec * nv + sizeof(float4) * kRing)); };
    // On one dense matrix the reflectors leave L2 behind: two from 2,400 rows on (2730^2, 890 vectors: 14.3
    // ms, one 17.5, four 22.4; 1728^2, 530 vectors: one 3.6, two 5.8).
    int nv = p.n >= 2400 ? 2 : p.ktot < 16 * nsm ? 1 : p.ktot >= 24 * nsm && p.n > 384 && p.n <= 576 ? 4 : 2;
    while (nv > 1 && warps_of(nv) < 1) nv /= 2;
    if (nv == 4)
        launch_back<4>(a, p, warps_of(4), s);
    else if (nv == 2)
        launch_back<2>(a, p, warps_of(2), s);
    else
        launch_back<1>(a, p, warps_of(1), s);
    if (g_clock) g_clock->end(s);
    *launches += 5;
}

}  // namespace opsec
