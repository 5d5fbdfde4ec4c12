// Two cells per thread in sm_100a's packed FP32 (add/sub/mul/fma.rn.f32x2).
//
// Each half of a packed operation rounds as the scalar instruction does, so
// collide_fast2 gives collide_fast's results (d3q27.cuh) bit for bit, two
// cells per issue slot.  The assembler fuses a packed multiply into a packed
// add that uses it, even with .rn on both and with -fmad=false (measured: a
// quarter of the results of a*b + c*d differ).  A product that feeds an add
// is therefore written as a*b + z with z = -0 in both halves, which rounds as
// the product alone and is a fused operation already; z comes from the
// kernel's arguments, because a constant is folded away again.
#pragma once

#include "d3q27.cuh"

namespace culbm {

// Two FP32 values in one 64-bit register pair: low half cell 0, high half cell 1.
using f32x2 = unsigned long long;
constexpr f32x2 kNegZero2 = 0x8000000080000000ull;   // the argument z

__device__ __forceinline__ f32x2 pk2(float lo, float hi)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo2(f32x2 v)
{
    float a;
    [[maybe_unused]] float b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a;
}
__device__ __forceinline__ float hi2(f32x2 v)
{
    [[maybe_unused]] float a;
    float b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return b;
}
__device__ __forceinline__ f32x2 dup2(float v) { return pk2(v, v); }

__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// cdot_fast on two cells; n* = -u*.
template <int D>
__device__ __forceinline__ f32x2 cdot_fast2(f32x2 ux, f32x2 uy, f32x2 uz, f32x2 nx, f32x2 ny, f32x2 nz)
{
    constexpr int cx = cx_of(D), cy = cy_of(D), cz = cz_of(D);
    f32x2 v = cx == 1 ? ux : nx;
    if constexpr (cy != 0) v = cx == 0 ? (cy == 1 ? uy : ny) : (cy == 1 ? add2(v, uy) : sub2(v, uy));
    if constexpr (cz != 0)
        v = (cx == 0 && cy == 0) ? (cz == 1 ? uz : nz) : (cz == 1 ? add2(v, uz) : sub2(v, uz));
    return v;
}

// collide_fast<E> on two cells.  get(d) is the raw pair of direction d and is
// called twice (moments, then relaxation), so that the caller may keep the
// narrow stored values in registers and widen them on each call (between()
// runs before the second round); terms(t) may replace the macroscopic terms
// of either cell; put(k, a, b) takes the new pairs of directions k and 26 - k, k <= 13 (b = a for 13).
struct FastTerms2 {
    f32x2 rho, dr, ux, uy, uz;   // dr = rho - 1
    f32x2 b[4], om;              // w W_k 2^E by weight class, 1 - w
};

template <int E, class G, class B, class T, class P>
__device__ __forceinline__ void collide_fast2(float w, f32x2 z0, G&& get, B&& between, T&& terms, P&& put)
{
    f32x2 r = get(13);
    f32x2 jx, jy, jz;
#pragma unroll
    for (int d = 0; d < 13; ++d) {
        const f32x2 a = get(d), b = get(26 - d);
        r = add2(r, add2(a, b));
        const f32x2 t = sub2(a, b);
        if (d == 0) {   // c_0 = (-1, -1, -1)
            jx = jy = jz = mul2(dup2(-1.0f), t);
            continue;
        }
        if (cx_of(d) != 0) jx = cx_of(d) == 1 ? add2(jx, t) : sub2(jx, t);
        if (cy_of(d) != 0) jy = cy_of(d) == 1 ? add2(jy, t) : sub2(jy, t);
        if (cz_of(d) != 0) jz = cz_of(d) == 1 ? add2(jz, t) : sub2(jz, t);
    }
    between();
    const f32x2 un = dup2(pow2<float, -E>());
    FastTerms2 t;
    t.dr = mul2(r, un);   // an exact power-of-two product: fusing it changes no bit
    t.rho = add2(dup2(1.0f), t.dr);
    const f32x2 inv = pk2(__fdiv_rn(1.0f, lo2(t.rho)), __fdiv_rn(1.0f, hi2(t.rho)));
    t.ux = fma2(mul2(jx, un), inv, z0);
    t.uy = fma2(mul2(jy, un), inv, z0);
    t.uz = fma2(mul2(jz, un), inv, z0);
    const float W[4] = {8.0f / 27.0f, 2.0f / 27.0f, 1.0f / 54.0f, 1.0f / 216.0f};
#pragma unroll
    for (int k = 0; k < 4; ++k) t.b[k] = dup2(__fmul_rn(__fmul_rn(w, W[k]), pow2<float, E>()));
    t.om = dup2(__fsub_rn(1.0f, w));
    terms(t);
    const f32x2 ux = t.ux, uy = t.uy, uz = t.uz, om = t.om;
    const f32x2 mone = dup2(-1.0f);
    const f32x2 nx = mul2(mone, ux), ny = mul2(mone, uy), nz = mul2(mone, uz);
    f32x2 Ak[4], Ck[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        Ak[k] = mul2(t.b[k], t.rho);
        Ck[k] = mul2(t.b[k], t.dr);
    }
    const f32x2 uu = fma2(ux, ux, fma2(uy, uy, mul2(uz, uz)));
    const f32x2 base = mul2(dup2(-1.5f), uu);
    for_dirs([&](auto dd) {
        constexpr int d = decltype(dd)::value;
        if constexpr (d < 13) {
            constexpr int k = (cx_of(d) != 0) + (cy_of(d) != 0) + (cz_of(d) != 0);
            const f32x2 cu = cdot_fast2<d>(ux, uy, uz, nx, ny, nz);
            const f32x2 q = fma2(mul2(dup2(4.5f), cu), cu, base);
            const f32x2 ed = fma2(Ak[k], fma2(dup2(3.0f), cu, q), Ck[k]);
            const f32x2 ee = fma2(Ak[k], fma2(dup2(-3.0f), cu, q), Ck[k]);
            put(d, fma2(om, get(d), ed), fma2(om, get(26 - d), ee));
        }
    });
    const f32x2 c = fma2(om, get(13), fma2(Ak[0], base, Ck[0]));
    put(13, c, c);
}

}  // namespace culbm
