// Householder tridiagonalisation A = Q T Q^T of symmetric blocks, in double-FP32 (df64.h).
//
// Two shapes of one kernel: a batch of azimuthal blocks, each on a thread-block cluster, and one
// dense matrix on the whole chip.  The reduction is n dependent steps, and at these sizes the
// step's latency, not its arithmetic, is the time: the kernel is laid out for few and short
// hand-overs.
//   * Rows are dealt to CTAs cyclically and kept whole (both triangles), so that a CTA forms its
//     entries of p = A v by itself.  Each step then has one barrier between CTAs, after which
//     every CTA reads p (n pairs) and the next pivot row; y.v, w, the pivot column and its
//     reflector are formed by every CTA alike, from the same data in the same order, hence with
//     the same bits.  Storing one triangle would take 51 FP32 operations an entry of it against
//     39 here on twice the entries, but every CTA (and every warp) then contributes to every
//     entry of p: partial sums in shared memory and their exchange were most of the step.
//   * One fused pass per step applies the rank-2 update to a CTA's rows and forms their products
//     with the next reflector, four rows at a time against the same 64 columns: the vectors are
//     read from shared memory once for the four, and four independent 16-byte loads hide L2.
//   * The last rows (they stay longest) live in shared memory, as many as fit; the rest in L2.
//   * The reflector's square root and reciprocals are double-FP32 Newton steps from the FP32
//     hardware estimates: in FP64, at 1/64 of the FP32 rate, they were a long chain of each step.
//   * The pass runs on packed FP32 instructions (two columns an issue slot).
// Pairs of floats have FP32's exponent range, so a block is reduced times a power of two that brings its
// largest diagonal entry (S is a covariance: its largest entry) to [1/2, 1), and the reflector of a column
// whose squares would underflow is formed from the column times 2^80.
// Bound by the FP32 pipe in the pass (44 % busy over all, with two warps a scheduler) and by the
// step's chain of reductions (3.3 us of each step).  Against one triangle on clusters of four, with
// partial sums and FP64 scalars: 34 blocks of 512^2 (the 32k-cell build) 8.19 -> 5.18 ms, 34 of
// 1024^2 54.5 -> 35.6, 10 of 555^2 10.3 -> 4.65, 18 of 624^2 13.5 -> 6.99, 18 of 64^2 0.318 -> 0.226.
// One dense matrix on the chip: 990^2 5.5 ms, 1728^2 13.6, 2730^2 39.3 (8 us a step at 1728: the barrier
// over 152 CTAs, the exchange through L2 and the reductions; 512 threads a CTA, spilling: 19.6).
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "df64.h"
#include "engine.h"
#include "packed.h"

namespace cg = cooperative_groups;

namespace opsec {
namespace {

constexpr int kChunk = 64;   // columns of a pass step: two per lane
constexpr int kDepth = 4;    // pass steps of a warp's rows under way from L2 (asynchronous copies)
constexpr int kMaxC = 8;     // largest (portable) cluster
constexpr int kElems = 4;    // vector entries of a thread in a cluster (n <= 4 x 256); 4, 8 or 16 on the chip
constexpr int kChipT = 256;  // threads of a CTA on the chip

// Vectors and matrix rows keep two neighbouring entries as (hi, hi, lo, lo): 16 bytes that load as
// the operands of packed FP32 instructions (add/mul/fma .f32x2: two results an issue slot, each
// rounded as the scalar instruction rounds).
__device__ __forceinline__ int at(int i) { return ((i >> 1) << 2) + (i & 1); }
__device__ __forceinline__ df get(const float* x, int i) { return df{x[at(i)], x[at(i) + 2]}; }
__device__ __forceinline__ df getcg(const float* x, int i) { return df{__ldcg(x + at(i)), __ldcg(x + at(i) + 2)}; }
__device__ __forceinline__ void put(float* x, int i, df v) {
    x[at(i)] = v.h;
    x[at(i) + 2] = v.l;
}

// the factor of a rank-1 update that belongs to a row, twice each: x.h, -x.h, -x.l
struct RowFactor {
    f2 h, nh, nl;
};
__device__ __forceinline__ RowFactor row_factor(df x) { return RowFactor{pk(x.h, x.h), pk(-x.h, -x.h), pk(-x.l, -x.l)}; }
// a - x y - u w: both products exact to the second order, one renormalisation (27 operations)
__device__ __forceinline__ df2 df2_rank2(df2 a, RowFactor x, f2 yh, f2 yl, RowFactor u, f2 wh, f2 wl) {
    const f2 q1 = mul2(x.h, yh), q2 = mul2(u.h, wh);
    f2 e = fma2(x.nh, yl, fma2(x.nh, yh, q1));
    e = fma2(x.nl, yh, e);
    f2 g = fma2(u.nh, wl, fma2(u.nh, wh, q2));
    g = fma2(u.nl, wh, g);
    const f2 s1 = sub2(a.h, q1), s2 = sub2(s1, q2);
    const f2 t = add2(sub2_err(a.h, q1, s1), sub2_err(s1, q2, s2));
    const f2 l = add2(add2(a.l, t), add2(e, g));
    const f2 r = add2(s2, l);
    return df2{r, sub2(l, sub2(r, s2))};
}
struct TridiagArgs {
    int n, ld;         // order, row stride of D (a multiple of kChunk)
    int C;             // CTAs per block
    int kres;          // a warp's rows k >= kres live in shared memory
    int nres;          // resident rows per CTA
    float* D;          // [block][n][2 ld] the matrix in double-FP32, both triangles, zero past column n
    float4* V;         // [block][n up to whole fours][ceil(n/2)] reflector c in row c (v[c+1] = 1), two entries as (hi, hi, lo, lo), zeros
                       // from entry c & ~3 on before it and past entry n - 1
    double *tau, *dg, *eg;  // [block][n]
    const double2* unit;    // [block] the power of two, and its inverse
    // whole-chip form: exchange of p, and the barrier between CTAs
    float2* pbuf;      // [2][n]
    unsigned* count;   // arrivals
    int* err;          // set when a wait ran out
    long long wait_cycles;
};

// (2^-e, 2^e) of each block, 2^e > its largest |diagonal entry| >= 2^(e-1): one CTA a block.  Clears the
// reduction's error word on the way.
__global__ void __launch_bounds__(256) unit_kernel(int n, const double* __restrict__ A, double2* __restrict__ unit, int* err) {
    __shared__ double red[8];
    const double* Ab = A + (size_t)blockIdx.x * n * n;
    double m = 0.0;
    for (int i = threadIdx.x; i < n; i += 256) m = fmax(m, fabs(Ab[(size_t)i * n + i]));
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x) return;
    if (blockIdx.x == 0) *err = 0;
    for (int w = 1; w < 8; w++) m = fmax(m, red[w]);
    int e = 0;
    if (m > 0.0 && isfinite(m)) frexp(m, &e);
    e = max(-1000, min(1000, e));  // both powers are normal numbers
    unit[blockIdx.x] = make_double2(ldexp(1.0, -e), ldexp(1.0, e));
}

// lower triangle of the FP64 blocks, times their unit -> both triangles in double-FP32, rows padded with zeros
__global__ void __launch_bounds__(256) pairs_kernel(int n, int ld, const double* __restrict__ A,
                                                    const double2* __restrict__ unit, float* __restrict__ D) {
    __shared__ float2 tile[32][33];
    const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;  // rows i (the contiguous index of A), columns j
    if (i0 + 31 < j0) return;  // above the diagonal: written with its mirror image
    const double* Ab = A + (size_t)blockIdx.z * n * n;
    float* Db = D + (size_t)blockIdx.z * n * 2 * ld;
    const double u = unit[blockIdx.z].x;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int y = ty; y < 32; y += 8) {
        const int i = i0 + tx, j = j0 + y;
        float2 v = make_float2(0.f, 0.f);
        if (i < n && j < n && i >= j) {
            v = df_pack(df_from(Ab[(size_t)j * n + i] * u));
            put(Db + (size_t)j * 2 * ld, i, df_unpack(v));  // row j, column i
        }
        tile[y][tx] = v;
    }
    __syncthreads();
    for (int y = ty; y < 32; y += 8) {
        const int i = i0 + y, j = j0 + tx;
        if (i < n && j < n && i > j) put(Db + (size_t)i * 2 * ld, j, df_unpack(tile[tx][y]));
    }
    for (int y = ty; y < 32 && i0 == j0; y += 8)  // zeros past the last column
        for (int j = n + tx; j < ld; j += 32)
            if (i0 + y < n) put(Db + (size_t)(i0 + y) * 2 * ld, j, df{0.f, 0.f});
}

__device__ __forceinline__ df shfl_xor_df(df x, int o) {
    return df{__shfl_xor_sync(0xffffffffu, x.h, o), __shfl_xor_sync(0xffffffffu, x.l, o)};
}

// Sum over the CTA with one barrier: a butterfly in each warp, then the warps' sums by every
// thread.  The additions commute exactly, so every thread (and every CTA with the same data) gets
// the same bits.  red holds W pairs and is not reused before another barrier.
template <int W>
__device__ __forceinline__ df cta_sum(df x, float2* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o; o >>= 1) x = df_add(x, shfl_xor_df(x, o));
    if (lane == 0) red[warp] = df_pack(x);
    __syncthreads();
    df y[W];
#pragma unroll
    for (int i = 0; i < W; i += 2) {
        const float4 v = *reinterpret_cast<const float4*>(red + i);
        y[i] = df{v.x, v.y};
        y[i + 1] = df{v.z, v.w};
    }
#pragma unroll
    for (int o = 1; o < W; o *= 2)
#pragma unroll
        for (int i = 0; i + o < W; i += 2 * o) y[i] = df_add(y[i], y[i + o]);
    return y[0];
}

// Reflector of a column with first entry x0 and s2 = the sum of squares below it: H = I - tau v v^T,
// v = (1, scal * rest), maps it onto beta e_1.  tau = 1 + |x0| / nrm, scal = 1 / (x0 - beta).
struct Reflector {
    df tau, beta, scal;
};
__device__ __forceinline__ Reflector reflector(df x0, df s2) {
    if (!(s2.h > 0.f)) return Reflector{df{0.f, 0.f}, x0, df{0.f, 0.f}};
    const df x = df_fma(s2, x0, x0);
    // 1/sqrt(x): y0 (1 + r/2 + 3 r^2/8), r = 1 - x y0^2 ~ 2^-22
    const float y0 = rsqrtf(x.h);
    const df r = df_fms(df{1.f, 0.f}, x, df_mul(df{y0, 0.f}, df{y0, 0.f}));
    const df inv = df_fma(df{y0, 0.f}, df{y0, 0.f}, fast_two_sum(0.5f * r.h, fmaf(0.375f * r.h, r.h, 0.5f * r.l)));
    const df nrm = df_mul(x, inv);
    const bool neg = x0.h < 0.f || (x0.h == 0.f && x0.l < 0.f);
    const df ax = neg ? df{-x0.h, -x0.l} : x0;
    const df tau = df_fma(df{1.f, 0.f}, ax, inv);
    // 1/(|x0| + nrm): q0 (1 + r + r^2)
    const df d = df_add(ax, nrm);
    const float q0 = 1.0f / d.h;
    const df e = df_fms(df{1.f, 0.f}, d, df{q0, 0.f});
    const df q = df_fma(df{q0, 0.f}, df{q0, 0.f}, fast_two_sum(e.h, fmaf(e.h, e.h, e.l)));
    return neg ? Reflector{tau, nrm, df{-q.h, -q.l}} : Reflector{tau, df{-nrm.h, -nrm.l}, q};
}

// Barrier over the CTAs of the whole-chip form (a cooperative launch: all are resident).  Every
// wait ends: past the limit the error word is set and the kernel leaves.
__device__ __forceinline__ bool chip_barrier(unsigned* count, unsigned target, int* err, long long limit) {
    __syncthreads();
    int bad = 0;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        unsigned v;
        long long t0 = 0;
        for (int spin = 0;; spin++) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
            if ((int)(v - target) >= 0) break;
            if ((spin & 255) == 255) {
                const long long now = clock64();
                if (t0 == 0) t0 = now;
                if (now - t0 > limit) {
                    atomicExch(err, 1);
                    bad = 1;
                    break;
                }
            }
        }
    }
    return __syncthreads_or(bad) == 0;
}

// One group of a warp's rows against columns [j0, ld): update (UPD) by (v, w), product with vn
// (SYM).  Row q starts at base + off[q] and takes part when bit q of act is set.  Lane l holds
// columns 64 k + 2 l, +1.  Rows in L2 come through the warp's ring of kDepth steps, each lane
// copying what it will read itself: with one step loaded ahead in registers an SM had 16 KB under
// way, and the pass ran at that over the L2 latency (20 bytes a clock).  Afterwards lanes 32/RG q .. hold row q's product in acc[0].
template <int RG, bool UPD, bool SYM, bool SHARED>
__device__ __forceinline__ void pass_group(int j0, int ld, float* base, const int (&off)[RG], unsigned act,
                                           const df (&vr)[RG], const df (&wr)[RG], const float* v, const float* w,
                                           const float* vn, float* ring, int lane, df (&acc)[RG]) {
    auto load_s = [](const float* x, int j) { return *reinterpret_cast<const ulonglong2*>(x + 2 * j); };
    auto slot = [&](int d, int q) { return ring + ((d * RG + q) * 32 + lane) * 4; };
    auto issue = [&](int j, int d) {
        if (j < ld)
#pragma unroll
            for (int q = 0; q < RG; q++)
                if (act >> q & 1) {
                    const unsigned dst = (unsigned)__cvta_generic_to_shared(slot(d, q));
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(base + 2 * (off[q] + j)) : "memory");
                }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (!SHARED)
        for (int d = 0; d < kDepth - 1; d++) issue(j0 + 2 * lane + d * kChunk, d);
    df2 sum[RG];
    RowFactor fv[RG], fw[RG];
    const f2 minus1 = pk(-1.f, -1.f);
#pragma unroll
    for (int q = 0; q < RG; q++) {
        sum[q] = df2{0ull, 0ull};
        if (UPD) {
            fv[q] = row_factor(vr[q]);
            fw[q] = row_factor(wr[q]);
        }
    }
    for (int j = j0 + 2 * lane, it = 0; j < ld; j += kChunk, it = (it + 1) % kDepth) {
        ulonglong2 a[RG];
        if (!SHARED) asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 2) : "memory");
#pragma unroll
        for (int q = 0; q < RG; q++)
            if (act >> q & 1) a[q] = *reinterpret_cast<const ulonglong2*>(SHARED ? base + 2 * (off[q] + j) : slot(it, q));
        if (!SHARED) issue(j + (kDepth - 1) * kChunk, (it + kDepth - 1) % kDepth);
        const ulonglong2 vj = load_s(v, j), wj = load_s(w, j), nj = load_s(vn, j);
        const f2 nnj = mul2(nj.x, minus1);
#pragma unroll
        for (int q = 0; q < RG; q++)
            if (act >> q & 1) {
                df2 x{a[q].x, a[q].y};
                if (UPD) {
                    x = df2_rank2(x, fv[q], wj.x, wj.y, fw[q], vj.x, vj.y);
                    ulonglong2* p = reinterpret_cast<ulonglong2*>(base + 2 * (off[q] + j));
                    const ulonglong2 o = make_ulonglong2(x.h, x.l);
                    if (SHARED)
                        *p = o;
                    else
                        __stcg(p, o);
                }
                if (SYM) sum[q] = df2_mac(sum[q], x, nj.x, nj.y, nnj);
            }
    }
#pragma unroll
    for (int q = 0; q < RG && SYM; q++) {
        df s0, s1;
        upk(sum[q].h, &s0.h, &s1.h);
        upk(sum[q].l, &s0.l, &s1.l);
        acc[q] = df_add(s0, s1);
    }
    if (SYM) {
        // sum over the lanes, halving the rows held at each of the first steps
        int o = 16;
#pragma unroll
        for (int h = RG / 2; h >= 1; h /= 2, o /= 2) {
            const bool up = lane & o;
#pragma unroll
            for (int q = 0; q < h; q++) {
                const df keep = up ? acc[q + h] : acc[q], give = up ? acc[q] : acc[q + h];
                acc[q] = df_add(keep, shfl_xor_df(give, o));
            }
        }
#pragma unroll
        for (int e = 16 / RG; e; e >>= 1) acc[0] = df_add(acc[0], shfl_xor_df(acc[0], e));
    }
}

// n <= E T: a thread holds its entries of a step's vectors in registers.
template <int T, int RG, int E, bool CHIP>
__global__ void __launch_bounds__(T, 1) tridiag_kernel(TridiagArgs a) {
    constexpr int W = T / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int C = a.C, n = a.n, ld = a.ld;
    const int rank = (int)(blockIdx.x % C), b = (int)(blockIdx.x / C);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    float* D = a.D + (size_t)b * n * 2 * ld;
    const int vs = (n + 1) / 2;
    float4* V = a.V + (size_t)b * ((n + 3) & ~3) * vs;
    float* vcur = reinterpret_cast<float*>(smem_raw);  // v of the step being applied
    float* vnxt = vcur + 2 * ld;                       // the next reflector
    float* w = vnxt + 2 * ld;
    float2* red = reinterpret_cast<float2*>(w + 2 * ld);  // [2][32] (two reductions a step)
    float2* x0s = red + 64;               // [2]: y at the pivot, the column's first entry
    float* ring = reinterpret_cast<float*>(x0s + 2) + warp * (kDepth * RG * 128);  // the warp's rows on their way
    float2* pown = x0s + 2 + W * kDepth * RG * 64;  // [2][nl + 1] this CTA's entries of p (cluster form)
    const int nl = (n - rank + C - 1) / C;  // rows rank, rank + C, ...
    const int nlmax = (n + C - 1) / C;
    float* rres = reinterpret_cast<float*>(pown + 2 * ((nlmax + 1) & ~1));  // [nres][2 ld] resident rows
    cg::cluster_group cluster = cg::this_cluster();
    unsigned epoch = 0;

    // between CTAs: their p entries and the next pivot row are in place
    auto barrier = [&]() -> bool {
        if constexpr (CHIP) {
            epoch += (unsigned)C;
            return chip_barrier(a.count, epoch, a.err, a.wait_cycles);
        } else {
            if (C > 1)
                cluster.sync();
            else
                __syncthreads();
            return true;
        }
    };
    // the fused pass over this CTA's rows >= r0; products into parity `par`
    auto pass = [&](int r0, int par, auto upd_c, auto sym_c) {
        constexpr bool UPD = decltype(upd_c)::value, SYM = decltype(sym_c)::value;
        const int j0 = r0 & ~(kChunk - 1);
        const int lr0 = r0 > rank ? (r0 - rank + C - 1) / C : 0;  // first active local row
        const int k0 = lr0 > warp ? (lr0 - warp + W - 1) / W : 0;
        for (int kg = k0 & ~(RG - 1); warp + W * kg < nl; kg += RG) {
            const bool res = kg >= a.kres;
            int off[RG];
            unsigned act = 0;
            df vr[RG], wr[RG], acc[RG];
#pragma unroll
            for (int q = 0; q < RG; q++) {
                const int k = kg + q, lr = warp + W * k, r = rank + C * lr;
                const bool on = k >= k0 && lr < nl;
                off[q] = res ? (lr - W * a.kres) * ld : r * ld;
                act |= on ? 1u << q : 0u;
                vr[q] = UPD && on ? get(vcur, r) : df{0.f, 0.f};
                wr[q] = UPD && on ? get(w, r) : df{0.f, 0.f};
            }
            if (res)
                pass_group<RG, UPD, SYM, true>(j0, ld, rres, off, act, vr, wr, vcur, w, vnxt, ring, lane, acc);
            else
                pass_group<RG, UPD, SYM, false>(j0, ld, D, off, act, vr, wr, vcur, w, vnxt, ring, lane, acc);
            if (SYM && (lane & (32 / RG - 1)) == 0) {
                const int k = kg + lane / (32 / RG), lr = warp + W * k;
                if (k >= k0 && lr < nl) {
                    if constexpr (CHIP)
                        __stcg(a.pbuf + (size_t)par * n + rank + C * lr, df_pack(acc[0]));
                    else
                        pown[par * nlmax + lr] = df_pack(acc[0]);
                }
            }
        }
        // the next pivot row, when it lives in shared memory, to where every CTA reads it
        if (UPD && r0 % C == rank && r0 / C / W >= a.kres) {
            __syncthreads();
            const float4* src = reinterpret_cast<const float4*>(rres + (size_t)(r0 / C - W * a.kres) * 2 * ld);
            float4* dst = reinterpret_cast<float4*>(D + (size_t)r0 * 2 * ld);
            for (int j = (j0 >> 1) + t; j < ld / 2; j += T) __stcg(dst + j, src[j]);
        }
    };
    using yes = std::true_type;
    using no = std::false_type;

    // resident rows in, vectors cleared
    for (int k = a.kres; warp + W * k < nl; k++) {
        const int lr = warp + W * k;
        const float4* src = reinterpret_cast<const float4*>(D + (size_t)(rank + C * lr) * 2 * ld);
        float4* dst = reinterpret_cast<float4*>(rres + (size_t)(lr - W * a.kres) * 2 * ld);
        for (int j = lane; j < ld / 2; j += 32) dst[j] = src[j];
    }
    for (int i = t; i < 6 * ld; i += T) vcur[i] = 0.f;
    __syncthreads();

    // Reflector of the pivot column c1: x[q] is its entry c1 + t + T q (0 at c1), s this thread's share
    // of the sum of squares below the first entry; the reflector goes to v.  Where the column is below
    // 2^-40 of the block (its squares below 2^-80, whose pairs underflow) it is formed anew times 2^80,
    // twice if need be: the reflector does not depend on the column's scale, beta does.
    df tau{0.f, 0.f};
    auto reflect = [&](int c1, df s, df (&x)[E], float* v) {
        df s2 = cta_sum<W>(s, red + 32), x0 = df_unpack(x0s[1]);
        int k = 0;
        for (; k < 2 && fmaf(x0.h, x0.h, s2.h) < 0x1p-80f; k++) {
            __syncthreads();  // every thread has read red
            s = df{0.f, 0.f};
#pragma unroll
            for (int q = 0; q < E; q++) {
                const int i = c1 + t + T * q;
                if (c1 + T * q >= n) break;
                x[q] = df{x[q].h * 0x1p80f, x[q].l * 0x1p80f};
                if (i > c1 + 1) s = df_fma(s, x[q], x[q]);
            }
            x0 = df{x0.h * 0x1p80f, x0.l * 0x1p80f};
            s2 = cta_sum<W>(s, red + 32);
        }
        const Reflector h = reflector(x0, s2);
#pragma unroll
        for (int q = 0; q < E; q++) {
            const int i = c1 + t + T * q;
            if (c1 + T * q >= n) break;
            if (i < n) put(v, i, i == c1 + 1 ? df{1.f, 0.f} : df_mul(x[q], h.scal));
        }
        if (t == 0 && rank == 0) {
            a.eg[(size_t)b * n + c1] = k ? ldexp(df_to(h.beta), -80 * k) : df_to(h.beta);
            a.tau[(size_t)b * n + c1] = df_to(h.tau);
        }
        tau = h.tau;
    };

    // column 0
    {
        df s{0.f, 0.f}, x[E];
#pragma unroll
        for (int q = 0; q < E; q++) {
            const int i = t + T * q;
            if (T * q >= n) break;
            x[q] = i < n ? getcg(D, i) : df{0.f, 0.f};
            if (i == 0) {
                if (rank == 0) a.dg[(size_t)b * n] = df_to(x[q]);
                x[q] = df{0.f, 0.f};
            }
            if (i == 1) x0s[1] = df_pack(x[q]);
            if (i >= 2) s = df_fma(s, x[q], x[q]);
        }
        reflect(0, s, x, vnxt);
        __syncthreads();
        if (rank == 0)
            for (int i = t; i < vs; i += T) V[i] = reinterpret_cast<const float4*>(vnxt)[i];
        pass(1, 0, no{}, yes{});
        if (!barrier()) return;
    }
    for (int c = 0; c <= n - 3; c++) {
        const int c1 = c + 1, par = c & 1;
        float* sw = vcur;
        vcur = vnxt;
        vnxt = sw;
        // p = A v from the CTAs and the pivot row before this step's update; y = tau p, y.v
        const float* rowc = D + (size_t)c1 * 2 * ld;
        df y[E], x[E], v[E];
        float2 p2[E];
#pragma unroll
        for (int q = 0; q < E; q++) {
            const int i = c1 + t + T * q;
            if (c1 + T * q >= n) break;
            p2[q] = make_float2(0.f, 0.f);
            x[q] = v[q] = df{0.f, 0.f};
            if (i < n) {
                if constexpr (CHIP)
                    p2[q] = __ldcg(a.pbuf + (size_t)par * n + i);
                else
                    p2[q] = C > 1 ? cluster.map_shared_rank(pown, i % C)[par * nlmax + i / C] : pown[par * nlmax + i];
                x[q] = getcg(rowc, i);
                v[q] = get(vcur, i);
            }
        }
        df part{0.f, 0.f};
#pragma unroll
        for (int q = 0; q < E; q++) {
            if (c1 + T * q >= n) break;
            y[q] = df_mul(tau, df_unpack(p2[q]));
            part = df_fma(part, y[q], v[q]);
        }
        if (t == 0) {
            x0s[0] = df_pack(y[0]);
            put(w, c, df{0.f, 0.f});
            put(vnxt, c, df{0.f, 0.f});
        }
        const df yv = cta_sum<W>(part, red);
        // w = y - (tau/2)(y.v) v; pivot column c1 under the update (v[c1] = 1)
        const df alpha = df_mul(tau, df{0.5f * yv.h, 0.5f * yv.l});
        const df wc = df_add(df_unpack(x0s[0]), df{-alpha.h, -alpha.l});
        df s{0.f, 0.f};
#pragma unroll
        for (int q = 0; q < E; q++) {
            const int i = c1 + t + T * q;
            if (c1 + T * q >= n) break;
            const df wi = df_fms(y[q], alpha, v[q]);
            if (i < n) put(w, i, wi);
            x[q] = df_add(df_fms(x[q], v[q], wc), df{-wi.h, -wi.l});
            if (i == c1) {
                if (rank == 0) a.dg[(size_t)b * n + c1] = df_to(x[q]);
                x[q] = df{0.f, 0.f};
            }
            if (i == c1 + 1) x0s[1] = df_pack(x[q]);
            if (i > c1 + 1) s = df_fma(s, x[q], x[q]);
        }
        reflect(c1, s, x, vnxt);
        __syncthreads();
        if (rank == c1 % C)
            for (int i = (c1 & ~3) / 2 + t; i < vs; i += T) V[(size_t)c1 * vs + i] = reinterpret_cast<const float4*>(vnxt)[i];
        if (c < n - 3)
            pass(c + 2, par ^ 1, yes{}, yes{});
        else
            pass(c + 2, par ^ 1, yes{}, no{});
        if (!barrier()) return;
    }
    // T back in A's own units: not step by step, where its FP64 products (64 cycles each) are in every
    // step's chain (2 % of a 1,728-cell box)
    const double back = a.unit[b].y;
    if (rank == 0)  // which wrote all but the last row
        for (int i = t; i < n - 1; i += T) {
            a.dg[(size_t)b * n + i] *= back;
            a.eg[(size_t)b * n + i] *= back;
        }
    if (rank == (n - 1) % C && t == 0) {
        // the last row is its own next pivot row: its final value is in D whichever way it lived
        a.dg[(size_t)b * n + n - 1] = df_to(getcg(D + (size_t)(n - 1) * 2 * ld, n - 1)) * back;
        a.eg[(size_t)b * n + n - 1] = 0.0;
        a.tau[(size_t)b * n + n - 1] = 0.0;
    }
}

int pad(int n) { return (n + kChunk - 1) / kChunk * kChunk; }

// shared memory without resident rows (W warps, rg rows each a pass)
size_t smem_base(int n, int C, int W, int rg) {
    const int nl = (n + C - 1) / C;
    return sizeof(float2) * (3 * (size_t)pad(n) + 64 + 2 + (size_t)W * kDepth * rg * 64 + 2 * (size_t)((nl + 1) & ~1));
}

// resident rows that fit in `room` bytes: whole groups of rg W rows, the last ones
void residency(TridiagArgs& a, int W, int rg, size_t room) {
    const int nl = (a.n + a.C - 1) / a.C, kn = (nl + W - 1) / W;
    const size_t row = sizeof(float2) * (size_t)a.ld;
    int k = 0;
    while (k < kn && row * (size_t)std::max(0, nl - W * k) > room) k += rg;
    a.kres = k;
    a.nres = std::max(0, nl - W * k);
}

int sm_count() {
    int dev = 0, nsm = 0;
    OPSEC_CUDA(cudaGetDevice(&dev));
    OPSEC_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    return nsm;
}

template <int T, int RG>
cudaLaunchConfig_t block_config(int nblk, int C, size_t smem, cudaStream_t s, cudaLaunchAttribute* at) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(nblk * C));
    cfg.blockDim = dim3(T);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = C;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// Clusters of C CTAs, one CTA to an SM, that the chip holds at once: a cluster lives inside one
// GPC, so the SMs left over in each (19 of them hold two clusters of eight) do not count.
template <int T, int RG>
int max_clusters(int C) {
    static std::atomic<int> cache[64][kMaxC + 1];
    int dev = 0;
    OPSEC_CUDA(cudaGetDevice(&dev));
    int v = dev < 64 ? cache[dev][C].load() : 0;
    if (v <= 0) {
        auto k = tridiag_kernel<T, RG, kElems, false>;
        const int cap = max_dynamic_smem((const void*)k);
        OPSEC_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, cap));
        cudaLaunchAttribute at{};
        const cudaLaunchConfig_t cfg = block_config<T, RG>(1, C, cap, nullptr, &at);
        OPSEC_CUDA(cudaOccupancyMaxActiveClusters(&v, k, &cfg));
        if (v < 1) fail(OPSEC_ERR_CUDA, "tridiagonalisation: no cluster fits");
        if (dev < 64) cache[dev][C] = v;
    }
    return v;
}

// CTAs per block: as many as leave every block its cluster in one wave (18 blocks of 624^2: eight
// 12.9 ms in two waves, six 7.8 in one), with at least 24 rows each; below n = 96 the hand-over
// between CTAs costs what the shorter pass gains (18 blocks of 64^2: one CTA 0.230 ms, two 0.237).
template <int T, int RG>
int cluster_of(int n, int nblk) {
    for (int C = kMaxC; C > 1 && n >= 96; C--)
        if (n >= 24 * C && max_clusters<T, RG>(C) >= nblk) return C;
    return 1;
}

template <int T, int RG>
void launch_blocks(TridiagArgs a, int nblk, cudaStream_t s) {
    a.C = cluster_of<T, RG>(a.n, nblk);
    auto k = tridiag_kernel<T, RG, kElems, false>;
    const size_t cap = (size_t)max_dynamic_smem((const void*)k), base = smem_base(a.n, a.C, T / 32, RG);
    if (base > cap) fail(OPSEC_ERR_CUDA, "tridiagonalisation: block too large for shared memory");
    residency(a, T / 32, RG, cap - base);
    OPSEC_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
    cudaLaunchAttribute at{};
    const cudaLaunchConfig_t cfg =
        block_config<T, RG>(nblk, a.C, base + sizeof(float2) * (size_t)a.ld * a.nres, s, &at);
    OPSEC_CUDA(cudaLaunchKernelEx(&cfg, k, a));
}

template <int E>
void launch_chip(TridiagArgs a, cudaStream_t s) {
    auto k = tridiag_kernel<kChipT, 2, E, true>;
    a.C = std::min(sm_count(), a.n);
    const size_t cap = (size_t)max_dynamic_smem((const void*)k), base = smem_base(a.n, a.C, kChipT / 32, 2);
    if (base > cap) fail(OPSEC_ERR_CUDA, "tridiagonalisation: matrix too large for shared memory");
    residency(a, kChipT / 32, 2, cap - base);
    OPSEC_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
    OPSEC_CUDA(cudaMemsetAsync(a.count, 0, sizeof(unsigned), s));
    void* args[] = {&a};
    OPSEC_CUDA(cudaLaunchCooperativeKernel((const void*)k, dim3((unsigned)a.C), dim3(kChipT), args,
                                           base + sizeof(float2) * (size_t)a.ld * a.nres, s));
}

}  // namespace

size_t tridiag_work_bytes(int n, int nblk) {
    return sizeof(float2) * ((size_t)nblk * n * pad(n) + 2 * (size_t)n) + 64;
}

bool tridiag_chip_supported(int n) {
    return n >= 3 && n <= 4 * kElems * kChipT &&
           smem_base(n, 152, kChipT / 32, 2) <= (size_t)max_dynamic_smem((const void*)tridiag_kernel<kChipT, 2, 4 * kElems, true>);
}

void launch_block_unit(int n, int nblk, const double* A, double* unit, int* err, cudaStream_t s, long long* launches) {
    unit_kernel<<<nblk, 256, 0, s>>>(n, A, reinterpret_cast<double2*>(unit), err);
    OPSEC_CUDA(cudaGetLastError());
    ++*launches;
}

void launch_tridiag(int n, int nblk, bool chip, const double* A, const double* unit, double* V, double* tau, double* dg,
                    double* eg, void* work, int* err, long long wait_cycles, cudaStream_t s, long long* launches) {
    TridiagArgs a{};
    a.n = n;
    a.ld = pad(n);
    a.D = static_cast<float*>(work);
    a.V = reinterpret_cast<float4*>(V);
    a.tau = tau;
    a.dg = dg;
    a.eg = eg;
    a.unit = reinterpret_cast<const double2*>(unit);
    a.pbuf = reinterpret_cast<float2*>(a.D + (size_t)nblk * n * 2 * a.ld);
    a.count = reinterpret_cast<unsigned*>(a.pbuf + 2 * (size_t)n);
    a.err = err;
    a.wait_cycles = wait_cycles;
    pairs_kernel<<<dim3((n + 31) / 32, (n + 31) / 32, nblk), 256, 0, s>>>(n, a.ld, A, a.unit, a.D);
    OPSEC_CUDA(cudaGetLastError());
    ++*launches;
    if (chip && nblk == 1) {
        if (n <= kElems * kChipT)
            launch_chip<kElems>(a, s);
        else if (n <= 2 * kElems * kChipT)
            launch_chip<2 * kElems>(a, s);
        else
            launch_chip<4 * kElems>(a, s);
    } else {
        launch_blocks<256, 4>(a, nblk, s);
    }
    ++*launches;
}

}  // namespace opsec
