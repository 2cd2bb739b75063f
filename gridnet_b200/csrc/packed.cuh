// Arithmetic on pairs of floats held in one 64-bit register (fma.rn.f32x2 and relatives).
#pragma once
#include "common.cuh"

namespace gn {

typedef unsigned long long u64;

__device__ __forceinline__ u64 pack2(float a, float b)
{
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(u64 v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ void ffma2(u64 &acc, u64 a, u64 w)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(w));
}
__device__ __forceinline__ u64 fmul2(u64 a, u64 b)
{
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 fadd2(u64 a, u64 b)
{
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 ffma2r(u64 a, u64 b, u64 c)
{
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// cen + sc * act(h) for a pair of samples. silu is done on the pair: the multiplies and adds are packed, only the
// two MUFU operations per value are scalar. 2^t overflows to +inf for very negative h; the reciprocal is then 0
// and h * 0 = -0, the right limit, so no clamp is needed.
template <int ACT>
__device__ __forceinline__ u64 act_residual2(u64 h, float sc, u64 cen)
{
    const u64 sc2 = pack2(sc, sc);
    if (ACT == GN_ACT_SILU) {
        const u64 t = fmul2(h, pack2(-1.4426950408889634f, -1.4426950408889634f));
        float t0, t1, e0, e1, r0, r1;
        unpack2(t, t0, t1);
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(t0));
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(t1));
        const u64 d = fadd2(pack2(e0, e1), pack2(1.0f, 1.0f));
        float d0, d1;
        unpack2(d, d0, d1);
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d0));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(d1));
        return ffma2r(fmul2(h, pack2(r0, r1)), sc2, cen);
    }
    float h0, h1;
    unpack2(h, h0, h1);
    return ffma2r(pack2(Act<ACT, float>::fwd(h0), Act<ACT, float>::fwd(h1)), sc2, cen);
}

// value and derivative for a pair of samples
template <int ACT>
__device__ __forceinline__ void act_both2(u64 h, u64 &f, u64 &d)
{
    if (ACT == GN_ACT_SILU) {
        const u64 t = fmul2(h, pack2(-1.4426950408889634f, -1.4426950408889634f));
        float t0, t1, e0, e1, r0, r1, d0, d1;
        unpack2(t, t0, t1);
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(t0));
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(t1));
        unpack2(fadd2(pack2(e0, e1), pack2(1.0f, 1.0f)), d0, d1);
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d0));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(d1));
        const u64 r = pack2(r0, r1);
        f = fmul2(h, r);
        d = ffma2r(f, ffma2r(r, pack2(-1.0f, -1.0f), pack2(1.0f, 1.0f)), r);  // sg (1 + h (1 - sg))
        return;
    }
    float h0, h1, f0, f1, d0, d1;
    unpack2(h, h0, h1);
    Act<ACT, float>::both(h0, f0, d0);
    Act<ACT, float>::both(h1, f1, d1);
    f = pack2(f0, f1);
    d = pack2(d0, d1);
}

}  // namespace gn
