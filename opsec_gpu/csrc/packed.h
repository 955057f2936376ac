// Packed FP32: two values an instruction (add/mul/fma .f32x2), each rounded as the scalar instruction
// rounds.  ptxas (13.0) joins a mul2 all of whose uses are additions with these into fma.f32x2, although
// both are .rn; where such a product's own rounding matters, write it as fma2(x, y, z) with z = -0 known
// only at run time, or let it have another use (as df2_mac's has).
#pragma once

#include <cuda_runtime.h>

namespace opsec {

using f2 = unsigned long long;
__device__ __forceinline__ f2 pk(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk(f2 x, float* a, float* b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(*a), "=f"(*b) : "l"(x)); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 add2_rd(f2 a, f2 b) {
    f2 r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// two double-FP32 values (df64.h)
struct df2 {
    f2 h, l;
};
// error of the rounded difference s = a - q
__device__ __forceinline__ f2 sub2_err(f2 a, f2 q, f2 s) {
    const f2 bb = sub2(s, a);
    return sub2(sub2(a, sub2(s, bb)), add2(q, bb));
}
// acc + x y with ny = -y.h; the low parts are only added up (12 operations)
__device__ __forceinline__ df2 df2_mac(df2 acc, df2 x, f2 yh, f2 yl, f2 ny) {
    const f2 nq = mul2(x.h, ny);
    f2 e = fma2(x.h, yl, fma2(x.h, yh, nq));
    e = fma2(x.l, yh, e);
    const f2 s = sub2(acc.h, nq);
    return df2{s, add2(add2(acc.l, e), sub2_err(acc.h, nq, s))};
}

}  // namespace opsec
