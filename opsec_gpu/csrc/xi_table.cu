// xi_table.cu -- xi(r) and band-derivative tables on the GPU, to FP64 accuracy.
//
// xi_l^m(r) = (1/2pi^2) int dk k^m j_l(kr) P(k) exp(-(k/kdamp)^2) by Simpson's
// rule, l = 0, m = 2 (Model.cpp:84-123):
//   table 0   GetXi       Nk = 32768 on [0, 10], P = cubic spline of the pkfile
//   table 1+p GetXiDeriv  Nk = 8192 on [k_p, k_{p+1}], P = 1 on [k_p, k_{p+1})
// (RealModel.cpp:98-127).  The spline is zero outside [x0, x_last) and the
// constant band is zero at k = k_{p+1}, so the last Simpson node of every
// band table contributes nothing, as in the reference.
//
// With c_j = mult_j / k_j a table is (1/r) sum_j c_j sin(k_j r), 1.6e9 terms for the 41 tables of
// the 32k-cell build (2.45 ms of FP32 issue as a term-by-term recurrence).  Most r do not need
// the nodes one by one: over a block of nodes of width Delta centred on K,
//   sum_j c_j sin(k_j r) = sin(K r) E + cos(K r) O,  E + iO = sum_p a_p (i z)^p,
//   z = r Delta / 2,  a_p = sum_j c_j u_j^p / p!,  u_j = (k_j - K) / (Delta / 2) in [-1, 1],
// and at z <= 2 the terms past p = 23 are below 3e-17 of sum |c_j|: 24 moments a block stand for
// all of its nodes.  The blocks are dyadic: xi_moments_kernel forms the moments of the narrowest
// blocks from the nodes and merges them pairwise upwards, xi_eval_kernel takes for each group of
// 32 r the widest blocks that keep z <= 2 (a band of width 0.01 is one to four blocks up to r =
// 400, 64 at r = 20,000).  Where even the narrowest blocks are too wide (table 0 past r = 819) it
// sums the nodes by the three-term recurrence of the sines.  All of it runs in double-FP32 (48
// bits) and is bound by FP32 issue.  41 tables of 4,352 r: 2.51 -> 0.23 ms (moments 0.06, evaluation
// 0.15, sums 0.02); 21 tables of 768 r: 0.71 -> 0.12 ms.
#include <cmath>

#include "df64.h"
#include "engine.h"

namespace opsec {
namespace {

constexpr int kNkXi = 32768;
constexpr int kNkBand = 8192;
constexpr double kTwoPi2 = 2.0 * M_PI * M_PI;
// 2^40: keeps the highest moments clear of FP32 underflow.  Table 0 is summed in units of P(k) besides
// (pk_unit), whose own scale FP32's range would not hold: 2^90 times the ordinary one overflows.
constexpr double kScale = 1099511627776.0;
constexpr int kP = 24;                      // moments per block
constexpr int kAnchor = 16;                 // recurrence steps between rotation anchors
constexpr double kZmax = 2.0;
// Levels: 2^l equal blocks per table.  A CTA of the moments kernel owns a subtree of 2^depth of the
// narrowest blocks (level lmax) and merges them to one (level lmin = lmax - depth): 16 of table
// 0's (256 nodes, 128 CTAs), 8 of a band's (at most 1024 nodes, so that 20 bands fill the chip).
constexpr int kDepthXi = 4, kDepthBand = 3, kSubMax = 16;
constexpr int kLmaxXi = 11;  // 16 nodes a block: below that a block costs more than its nodes
constexpr int kLmaxBandLo = 6, kLmaxBandHi = 9;
// work units (warps) per group of 32 r: parts of the table's blocks or nodes
constexpr int kZxi = 64, kZband = 8;
// sums of mult k^4 over groups of 32 nodes and, after those, of 128 (no CTA of the moments kernel
// holds fewer nodes)
constexpr int kW4Xi = kNkXi / 32 + 1 + kNkXi / 128, kW4Band = kNkBand / 32 + 1 + kNkBand / 128;
static_assert((kNkXi >> (kLmaxXi - kDepthXi)) % 128 == 0 && (kNkBand >> (kLmaxBandHi - kDepthBand)) % 128 == 0, "groups");

struct dconst {
    float h, l;
};
constexpr dconst dsplit(double x) { return dconst{(float)x, (float)(x - (double)(float)x)}; }
constexpr double inv_fact_of(int p) {
    double f = 1.0;
    for (int i = 2; i <= p; i++) f *= i;
    return 1.0 / f;
}
__constant__ dconst kInvFact[kP] = {
    dsplit(inv_fact_of(0)),  dsplit(inv_fact_of(1)),  dsplit(inv_fact_of(2)),  dsplit(inv_fact_of(3)),
    dsplit(inv_fact_of(4)),  dsplit(inv_fact_of(5)),  dsplit(inv_fact_of(6)),  dsplit(inv_fact_of(7)),
    dsplit(inv_fact_of(8)),  dsplit(inv_fact_of(9)),  dsplit(inv_fact_of(10)), dsplit(inv_fact_of(11)),
    dsplit(inv_fact_of(12)), dsplit(inv_fact_of(13)), dsplit(inv_fact_of(14)), dsplit(inv_fact_of(15)),
    dsplit(inv_fact_of(16)), dsplit(inv_fact_of(17)), dsplit(inv_fact_of(18)), dsplit(inv_fact_of(19)),
    dsplit(inv_fact_of(20)), dsplit(inv_fact_of(21)), dsplit(inv_fact_of(22)), dsplit(inv_fact_of(23))};

__device__ __forceinline__ df inv_fact(int p) { return df{kInvFact[p].h, kInvFact[p].l}; }
__device__ __forceinline__ df df_neg(df x) { return df{-x.h, -x.l}; }

// scratch: nodes c_j, per-32-node sums of mult k^4, moments, partial sums
struct XiPlan {
    XiTableArgs a;
    int n, ngrp;     // r values and groups of 32 of them
    int lband;       // narrowest level of the band tables
    float2* c2;      // [table nodes] c_j 2^40 as (hi, lo) pairs
    float* w4;       // [table][node / 32], then [node / 128]: sums of mult k^4
    float2* mom;     // [table][level][block][kP]
    float2* part;    // [table][unit][32 ngrp]
};

struct TableSpec {
    int nk, lmax, depth, nz;
    double kmin, kmax;
    size_t node0;  // first node in c2
    size_t w40;    // first sum in w4
    size_t mom0;   // first block in mom (in blocks)
    size_t part0;  // first row in part
    __device__ int lmin() const { return lmax - depth; }
    // the blocks of level l follow those of the wider levels
    __device__ size_t block(int l, int b) const { return mom0 + ((size_t(1) << l) - (size_t(1) << lmin())) + b; }
};

__host__ __device__ inline size_t blocks_of(int lmax, int depth) {
    return (size_t(2) << lmax) - (size_t(1) << (lmax - depth));
}

__device__ TableSpec table_spec(const XiPlan& p, int t) {
    TableSpec s;
    if (t == 0) {
        s = TableSpec{kNkXi, kLmaxXi, kDepthXi, kZxi, 0.0, 10.0, 0, 0, 0, 0};
    } else {
        const size_t b = t - 1;
        s = TableSpec{kNkBand,
                      p.lband,
                      kDepthBand,
                      kZband,
                      p.a.band_lo[b],
                      p.a.band_hi[b],
                      (size_t)(kNkXi + 1) + b * (kNkBand + 1),
                      (size_t)kW4Xi + b * kW4Band,
                      blocks_of(kLmaxXi, kDepthXi) + b * blocks_of(p.lband, kDepthBand),
                      (size_t)kZxi + b * kZband};
    }
    return s;
}

// exp(-x), x = k^2 >= 0, times 2^40, in double-FP32: the argument is reduced by ln 2 in two parts (Cody and
// Waite, Software Manual for the Elementary Functions, 1980) in FP64, the Taylor series on |y| <= ln 2 / 2 runs to y^13 (the next term is below 5e-18).
__device__ __forceinline__ df exp_neg_scaled(double x) {
    constexpr double kMagic = 6755399441055744.0;  // 1.5 2^52: adding it rounds to an integer
    constexpr double kLn2Hi = 6.93147180559945286227e-01, kLn2Lo = 2.31904681384629955842e-17;
    if (!(x < 110.0)) return df{0.f, 0.f};  // below 2^-118
    const double m = fma(x, -1.0 / M_LN2, kMagic);
    const double n = m - kMagic;
    const df y = df_from(fma(-n, kLn2Lo, fma(-n, kLn2Hi, -x)));
    df e = inv_fact(13);
#pragma unroll
    for (int q = 12; q >= 0; q--) e = df_fma(inv_fact(q), e, y);
    const float sc = __int_as_float((__double2loint(m) + 40 + 127) << 23);
    return df{e.h * sc, e.l * sc};
}

// Simpson weights and moments: one CTA per subtree of narrowest blocks.  FP64 (1/64 of the FP32
// rate) only where a node needs it: k, k^2, the argument of the exponential, table 0's spline.
// c_j = mult_j / k_j is formed as k_j P exp(-k_j^2) times the Simpson constants.
__global__ void __launch_bounds__(256) xi_moments_kernel(XiPlan p) {
    constexpr int kNodes = kNkBand >> (kLmaxBandLo - kDepthBand);
    static_assert((kNkXi >> (kLmaxXi - kDepthXi)) <= kNodes, "node buffer");
    __shared__ float2 c_s[kNodes + 1];
    __shared__ float w4_s[kNodes / 32];
    __shared__ float2 tree[2 * kSubMax - 1][kP];  // the narrowest blocks, then each wider level
    const int cta_xi = 1 << (kLmaxXi - kDepthXi), cta_band = 1 << (p.lband - kDepthBand);
    const int bx = (int)blockIdx.x;
    const int t = bx < cta_xi ? 0 : 1 + (bx - cta_xi) / cta_band;
    const int sub = bx < cta_xi ? bx : (bx - cta_xi) % cta_band;
    const TableSpec s = table_spec(p, t);
    const int nblk = 1 << s.depth;
    const int nsub = s.nk >> s.lmin(), L = s.nk >> s.lmax, j0 = sub * nsub;
    const bool last = sub == (1 << s.lmin()) - 1;  // it also holds node nk, at the end of its last block
    const double dk = (s.kmax - s.kmin) / s.nk;
    const double wc = (dk / 3) / kTwoPi2;
    const df wcd = df_from(wc);
    float* w4 = p.w4 + s.w40;
    for (int jj = threadIdx.x; jj < nsub + (last ? 1 : 0); jj += blockDim.x) {
        const int j = j0 + jj;
        const double k = s.kmin + j * dk, k2 = k * k;
        df P = wcd;
        if (t == 0)
            P = df_from(wc * p.a.pk_unit * spline_eval(p.a.npk, p.a.pk_x, p.a.pk_y, p.a.pk_b, p.a.pk_c, p.a.pk_d, k));
        else if (!(k >= s.kmin && k < s.kmax))  // ConstantSpline(1, kmin, kmax)
            P = df{0.f, 0.f};
        const float mult = 2 + 2 * (j % 2) - (j == 0) - (j == s.nk);
        df c = df_mul(df_mul(exp_neg_scaled(k2), df_from(k)), P);
        if (!(k > 0.0)) c = df{0.f, 0.f};
        const float2 c2 = make_float2(mult * c.h, mult * c.l);
        c_s[jj] = c2;
        p.c2[s.node0 + j] = c2;
        const float kf = (float)k, kf2 = kf * kf;
        float m4 = c2.x * (float)(1.0 / kScale) * kf * (kf2 * kf2);
        if (jj < nsub) {  // whole warps: nsub is a multiple of 32
            for (int o = 16; o > 0; o >>= 1) m4 += __shfl_xor_sync(0xffffffffu, m4, o);
            if ((j & 31) == 0) w4_s[jj >> 5] = w4[j >> 5] = m4;
        } else {
            w4[j >> 5] = m4;
        }
    }
    __syncthreads();
    if ((int)threadIdx.x < nsub / 128) {
        float v = 0.f;
        for (int g = 0; g < 4; g++) v += w4_s[4 * threadIdx.x + g];
        w4[s.nk / 32 + 1 + (j0 >> 7) + threadIdx.x] = v;
    }
    // moments of the narrowest blocks: 256 / nblk (16 or 32) threads each, then a butterfly sum
    {
        const int per = 256 >> s.depth, b = threadIdx.x / per, g = threadIdx.x % per;
        df acc[kP];
#pragma unroll
        for (int q = 0; q < kP; q++) acc[q] = df{0.f, 0.f};
        const float sc = 2.0f / (float)L;
        const int end = L + (last && b == nblk - 1 ? 1 : 0);
        for (int i = g; i < end; i += per) {
            const float u = (float)(i - L / 2) * sc;  // exact: L is a power of two
            df v = df_unpack(c_s[b * L + i]);
#pragma unroll
            for (int q = 0; q < kP; q++) {
                acc[q] = df_add(acc[q], v);
                v = df_mul(v, df{u, 0.f});
            }
        }
        for (int o = per / 2; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < kP; q++)
                acc[q] = df_add(acc[q], df{__shfl_xor_sync(0xffffffffu, acc[q].h, o), __shfl_xor_sync(0xffffffffu, acc[q].l, o)});
#pragma unroll
        for (int q = 0; q < kP; q++)
            if ((q & 15) == g) tree[b][q] = df_pack(df_mul(acc[q], inv_fact(q)));
    }
    __syncthreads();
    // wider blocks: a child at u covers u' = (u -+ 1) / 2 of its parent
    for (int n = nblk / 2, src = 0, dst = nblk; n >= 1; src = dst, dst += n, n >>= 1) {
        const int idx = threadIdx.x;
        if (idx < n * kP) {
            const int b = idx / kP, q = idx % kP;
            df acc{0.f, 0.f};
            for (int k = 0; k <= q; k++) {
                const df l = df_unpack(tree[src + 2 * b][k]), r = df_unpack(tree[src + 2 * b + 1][k]);
                acc = df_fma(acc, df_add(r, ((q - k) & 1) ? df_neg(l) : l), inv_fact(q - k));
            }
            const float sc = 1.0f / (float)(1 << q);
            tree[dst + b][q] = make_float2(acc.h * sc, acc.l * sc);
        }
        __syncthreads();
    }
    for (int idx = threadIdx.x; idx < (2 * nblk - 1) * kP; idx += blockDim.x) {
        const int e = idx / kP, q = idx % kP;
        int l = s.lmax, b = e, n = nblk;
        while (b >= n) {
            b -= n;
            n >>= 1;
            --l;
        }
        p.mom[s.block(l, sub * n + b) * kP + q] = tree[e][q];
    }
}

// sin and cos of the angle quad pi/2 + y, |y| <= pi/4, in double-FP32: Taylor series whose first
// terms left out are below 1e-16.
__device__ __forceinline__ void sincos_reduced(int quad, df y, df* sn, df* cs) {
    const df t = df_neg(df_mul(y, y));
    df s = inv_fact(15), c = inv_fact(16);
#pragma unroll
    for (int q = 13; q >= 1; q -= 2) s = df_fma(inv_fact(q), s, t);
#pragma unroll
    for (int q = 14; q >= 0; q -= 2) c = df_fma(inv_fact(q), c, t);
    s = df_mul(s, y);
    const df ss = (quad & 1) ? c : s, cc = (quad & 1) ? s : c;
    *sn = (quad & 2) ? df_neg(ss) : ss;
    *cs = ((quad + 1) & 2) ? df_neg(cc) : cc;
}

constexpr double kPio2Hi = 1.57079632679489655800e+00, kPio2Lo = 6.12323399573676603587e-17;  // to 2 x 53 bits

// sin and cos of k r: the product and its reduction by pi/2 in FP64 (a dozen instructions; FP64
// issues at 1/64 of the FP32 rate)
__device__ __forceinline__ void sincos_df(double k, double r, df* sn, df* cs) {
    constexpr double kMagic = 6755399441055744.0;  // 1.5 2^52: adding it rounds to an integer
    const double x = k * r, xe = fma(k, r, -x);
    const double m = fma(x, 2.0 / M_PI, kMagic);
    const double n = m - kMagic;
    sincos_reduced(__double2loint(m) & 3, df_from(fma(-n, kPio2Hi, x) + fma(-n, kPio2Lo, xe)), sn, cs);
}

// the same of a double-FP32 angle below 2^20, reduced by pi/2 as three floats
__device__ __forceinline__ void sincos_df(df x, df* sn, df* cs) {
    constexpr float kA = (float)kPio2Hi, kB = (float)(kPio2Hi - (double)kA),
                    kC = (float)(kPio2Hi - (double)kA - (double)kB + kPio2Lo);
    const float n = rintf(x.h * (float)(2.0 / M_PI));
    df y = df_fms(x, df{n, 0.f}, df{kA, kB});
    y = df_fms(y, df{n, 0.f}, df{kC, 0.f});
    sincos_reduced((int)n & 3, y, sn, cs);
}

// How a group of r is summed: level >= 0: the table's 2^level blocks; -1: its nodes.  The units
// (warps) in use follow; both kernels below ask this.
__device__ __forceinline__ int group_level(const TableSpec& s, double rmax, int* units) {
    const float need = fabsf((float)(s.kmax - s.kmin)) * (float)rmax * (float)(0.5 / kZmax);
    int l = s.lmin();
    while (l <= s.lmax && (float)(1 << l) < need) ++l;
    if (!(l <= s.lmax)) {
        *units = s.nz;
        return -1;
    }
    *units = min(s.nz, max(1, (1 << l) >> 3));  // eight blocks a unit, more where the units run out
    return l;
}

// One warp: 32 consecutive r of one table over one unit's blocks or nodes.
__global__ void __launch_bounds__(128) xi_eval_kernel(XiPlan p) {
    const int grp = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (grp >= p.ngrp) return;
    const int y = (int)blockIdx.y;
    const int t = y < kZxi ? 0 : 1 + (y - kZxi) / kZband;
    const int z = y < kZxi ? y : (y - kZxi) % kZband;
    const TableSpec s = table_spec(p, t);
    const double rmax = p.a.r[min(32 * grp + 31, p.n - 1)];  // r ascends
    int units;
    const int lev = group_level(s, rmax, &units);
    if (z >= units) return;
    const double r = p.a.r[min(32 * grp + lane, p.n - 1)];  // past the end: a copy, not read
    const double W = s.kmax - s.kmin;
    df tot{0.f, 0.f};
    if (lev >= 0) {
        const int nb = 1 << lev, b0 = (int)((long long)nb * z / units), b1 = (int)((long long)nb * (z + 1) / units);
        const double wb = W * __hiloint2double((1023 - lev) << 20, 0);  // W / nb
        const df wr = df_mul(df_from(wb), df_from(r));
        df sn, cs, sd, cd;
        sincos_df(s.kmin + (b0 + 0.5) * wb, r, &sn, &cs);
        sincos_df(wr, &sd, &cd);
        df zz{0.5f * wr.h, 0.5f * wr.l}, z2 = df_neg(df_mul(zz, zz));
        const bool r0 = !(r > 0.0);
        if (r0) {  // sum_j c_j k_j: per block K a_0 + (Delta/2) a_1
            sn = df_from(s.kmin + (b0 + 0.5) * wb);
            cs = df_from(0.5 * wb);
            zz = cd = df{1.f, 0.f};
            sd = df{2.f, 0.f};  // K moves by Delta from block to block
        }
        const float4* m = reinterpret_cast<const float4*>(p.mom + s.block(lev, b0) * kP);
        for (int b = b0; b < b1; b++, m += kP / 2) {
            float4 v = __ldg(m + kP / 2 - 1);
            df e{v.x, v.y}, o{v.z, v.w};
#pragma unroll
            for (int q = kP / 2 - 2; q >= 0; q--) {
                v = __ldg(m + q);
                e = df_fma(df{v.x, v.y}, e, z2);
                o = df_fma(df{v.z, v.w}, o, z2);
            }
            tot = df_fma(tot, sn, e);
            tot = df_fma(tot, cs, df_mul(o, zz));
            const df s2 = df_fma(df_mul(sn, cd), cs, sd);  // to the next block's centre
            if (!r0) cs = df_fms(df_mul(cs, cd), sn, sd);
            sn = s2;
        }
    } else {
        // sin(x + (m+1) d) = 2 cos(d) sin(x + m d) - sin(x + (m-1) d), restarted every kAnchor steps from
        // (sin, cos) rotated by kAnchor d: the recurrence's error grows with the square of its length
        const int per = ((s.nk + units) / units + kAnchor - 1) / kAnchor * kAnchor;
        const int j0 = z * per, j1 = min(s.nk + 1, j0 + per);
        const double dk = W / s.nk;
        if (j0 < j1) {
            df sn, cs, sd, cd, sT, cT;
            sincos_df(s.kmin + j0 * dk, r, &sn, &cs);
            const df dr = df_mul(df_from(dk), df_from(r));
            sincos_df(dr, &sd, &cd);
            sincos_df(df{kAnchor * dr.h, kAnchor * dr.l}, &sT, &cT);
            const bool r0 = !(r > 0.0);
            if (r0) {  // sum_j c_j k_j: the same recurrence on k_j itself
                sn = df_from(s.kmin + j0 * dk);
                cs = cd = cT = df{1.f, 0.f};
                sd = df_from(dk);
                sT = df{kAnchor * sd.h, kAnchor * sd.l};
            }
            const df c2{2.f * cd.h, 2.f * cd.l};
            const float2* c = p.c2 + s.node0;
            for (int j = j0; j < j1; j += kAnchor) {
                df cur = sn, prev = df_fms(df_mul(sn, cd), cs, sd);
                const int steps = min(kAnchor, j1 - j);
#pragma unroll 4
                for (int m = 0; m < steps; m++) {
                    tot = df_fma(tot, df_unpack(__ldg(c + j + m)), cur);
                    const df nxt = df_fma(df_neg(prev), c2, cur);
                    prev = cur;
                    cur = nxt;
                }
                const df s2 = df_fma(df_mul(sn, cT), cs, sT);
                if (!r0) cs = df_fms(df_mul(cs, cT), sn, sT);
                sn = s2;
            }
        }
    }
    p.part[(s.part0 + z) * (size_t)(32 * p.ngrp) + 32 * grp + lane] = df_pack(tot);
}

// Sums the units in order, divides by r, and adds what the reference's j0 does below x = kr = 0.01:
// its series there (Model.cpp:56-59) is 1 - x^2/6 - x^4/120 + ..., the sign of the x^4 term
// turned, so every such node adds -mult x^4/60 to the sum of sin(x)/x (x^6/2520 is below 4e-16).
// At r = 0 the units hold sum_j c_j k_j = sum_j mult_j.
__global__ void __launch_bounds__(128) xi_finish_kernel(XiPlan p) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, t = blockIdx.y;
    if (i >= p.n) return;
    const TableSpec s = table_spec(p, t);
    const double r = p.a.r[i];
    int units;
    group_level(s, p.a.r[min((i | 31), p.n - 1)], &units);
    const float2* part = p.part + s.part0 * (size_t)(32 * p.ngrp) + i;
    df sum{0.f, 0.f};
#pragma unroll 8
    for (int z = 0; z < units; z++) sum = df_add(sum, df_unpack(part[z * (size_t)(32 * p.ngrp)]));
    double acc = df_to(sum) * (1.0 / kScale);
    if (r > 0.0) {
        acc /= r;
        const double dk = (s.kmax - s.kmin) / s.nk;
        int jc = 0;  // nodes with (k_j r)^2 < 1e-4: a prefix, as k_j grows with j
        if (dk > 0.0 && s.kmin * r < 0.01) {
            const double jf = (0.01 / r - s.kmin) / dk;
            jc = jf > (double)s.nk ? s.nk + 1 : (int)jf + 1;
            while (jc > 0 && !((s.kmin + (jc - 1) * dk) * r * ((s.kmin + (jc - 1) * dk) * r) < 1e-4)) --jc;
        }
        if (jc > 0) {
            const float* w4 = p.w4 + s.w40;
            const float* w4b = w4 + s.nk / 32 + 1;
            float w = 0.f;
            int g = jc >> 7;
#pragma unroll 8
            for (int b = 0; b < g; b++) w += w4b[b];
            for (g *= 4; g < jc / 32; g++) w += w4[g];
            for (int j = jc & ~31; j < jc; j++) {
                const float k = (float)(s.kmin + j * dk), k2 = k * k;
                w += p.c2[s.node0 + j].x * (float)(1.0 / kScale) * k * (k2 * k2);
            }
            const double r2 = r * r;
            acc -= (double)w * (r2 * r2) * (1.0 / 60.0);
        }
    }
    if (t == 0) acc *= p.a.pk_back;
    p.a.xi64[(size_t)t * p.n + i] = acc;
    p.a.xi32[(size_t)t * p.n + i] = (float)acc;
}

// narrowest level of the band tables: enough blocks for the widest band at the largest r, within
// the range where a block is worth its moments (16 to 128 nodes)
int band_level(const XiTableArgs& a) {
    int l = kLmaxBandLo;
    while (l < kLmaxBandHi && (double)(1 << l) < a.band_wmax * a.xl.r2 * (0.5 / kZmax)) ++l;
    return l;
}

size_t plan(const XiTableArgs& a, XiPlan* p) {
    const int n = a.xl.n(), nb = a.nbands, lband = band_level(a), ngrp = (n + 31) / 32;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o += (bytes + 255) & ~size_t(255);
        return at;
    };
    const size_t c2 = take(sizeof(float2) * ((size_t)(kNkXi + 1) + (size_t)nb * (kNkBand + 1)));
    const size_t w4 = take(sizeof(float) * ((size_t)kW4Xi + (size_t)nb * kW4Band));
    const size_t mom =
        take(sizeof(float2) * kP * (blocks_of(kLmaxXi, kDepthXi) + (size_t)nb * blocks_of(lband, kDepthBand)));
    const size_t part = take(sizeof(float2) * ((size_t)kZxi + (size_t)nb * kZband) * 32 * ngrp);
    if (p) {
        unsigned char* b = reinterpret_cast<unsigned char*>(a.scratch);
        *p = XiPlan{a, n, ngrp, lband, reinterpret_cast<float2*>(b + c2), reinterpret_cast<float*>(b + w4),
                    reinterpret_cast<float2*>(b + mom), reinterpret_cast<float2*>(b + part)};
    }
    return o;
}

}  // namespace

size_t xi_scratch_doubles(const XiTableArgs& a) { return (plan(a, nullptr) + sizeof(double) - 1) / sizeof(double); }

void launch_xi_tables(const XiTableArgs& a, cudaStream_t s, long long* launches) {
    XiPlan p;
    plan(a, &p);
    const unsigned ctas = (1u << (kLmaxXi - kDepthXi)) + (unsigned)a.nbands * (1u << (p.lband - kDepthBand));
    xi_moments_kernel<<<ctas, 256, 0, s>>>(p);
    OPSEC_CUDA(cudaGetLastError());
    xi_eval_kernel<<<dim3((p.ngrp + 3) / 4, kZxi + kZband * a.nbands), 128, 0, s>>>(p);
    OPSEC_CUDA(cudaGetLastError());
    xi_finish_kernel<<<dim3((p.n + 127) / 128, 1 + a.nbands), 128, 0, s>>>(p);
    OPSEC_CUDA(cudaGetLastError());
    *launches += 3;
}

}  // namespace opsec
