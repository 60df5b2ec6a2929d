// philox.cuh — counter-based normals: Philox4x32-10 blocks (Salmon, Moraes, Dror, Shaw, SC'11) and the
// Box–Muller transform, two pairs at a time.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "f32x2.cuh"

namespace mcq {

constexpr float kTwoPow24Inv = 5.9604644775390625e-08f;   // 2^-24

__device__ __forceinline__ uint4 philox10(uint4 c, uint2 k) {
#pragma unroll
    for (int r = 0; r < 10; r++) {
        if (r) { k.x += 0x9E3779B9u; k.y += 0xBB67AE85u; }
        const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    }
    return c;
}

// -2 ln u, 2^-25 <= u <= 1: u = 2^e (1 + f) with 1 + f in [sqrt(1/2), sqrt(2)), and log(1 + f) = f + f^2 Q(f),
// Q of degree 7 (Lawson fit, 0.25 units of 2^-23 relative).  The exponent stays scaled by 2^23.
__device__ __forceinline__ f32x2 minus_two_log(float ua, float ub) {
    const int ia = __float_as_int(ua) - 0x3f3504f3, ib = __float_as_int(ub) - 0x3f3504f3;
    const int ea = ia & (int)0xff800000, eb = ib & (int)0xff800000;
    const f32x2 f = add2(pack(__int_as_float(__float_as_int(ua) - ea), __int_as_float(__float_as_int(ub) - eb)),
                         both(-1.0f));
    f32x2 q = fma2(f, both(0x1.65f792p-4f * -2.0f), both(-0x1.250e42p-3f * -2.0f));
    q = fma2(q, f, both(0x1.317fa6p-3f * -2.0f));
    q = fma2(q, f, both(-0x1.535b18p-3f * -2.0f));
    q = fma2(q, f, both(0x1.98d32ap-3f * -2.0f));
    q = fma2(q, f, both(-0x1.0004acp-2f * -2.0f));
    q = fma2(q, f, both(0x1.5556f2p-2f * -2.0f));
    q = fma2(q, f, both(-0x1.fffffap-2f * -2.0f));
    const f32x2 p = fma2(mul2(f, f), q, mul2(f, both(-2.0f)));
    return fma2(pack((float)ea, (float)eb), both(-2.0f * 0x1.62e43p-1f * 0x1p-23f), p);
}

// sqrt(x), x >= 0, to about half an ulp: the hardware's reciprocal root and one Newton step.
__device__ __forceinline__ f32x2 root(f32x2 x) {
    float xa, xb, ya, yb;
    unpack(x, xa, xb);
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(ya) : "f"(fmaxf(xa, 1e-30f)));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yb) : "f"(fmaxf(xb, 1e-30f)));
    const f32x2 y = pack(ya, yb), r = mul2(x, y);
    const f32x2 e = fma2(mul2(r, both(-1.0f)), r, x);
    return fma2(e, mul2(y, both(0.5f)), r);
}

// sin and cos of 2 pi t, 0 <= t <= 1: the nearest quarter turn, then polynomials on an eighth.
__device__ __forceinline__ void sincos_turns(f32x2 t, float (&s)[2], float (&c)[2]) {
    const f32x2 n = fma2(t, both(4.0f), both(12582912.0f));   // 1.5 2^23: the low bits are the quarter
    const f32x2 y = fma2(add2(n, both(-12582912.0f)), both(-0.25f), t);
    const f32x2 w = mul2(y, y);
    f32x2 a = fma2(w, both(-0x1.2db5a6p+6f), both(0x1.465facp+6f));
    a = fma2(a, w, both(-0x1.4abbbep+5f));
    a = fma2(a, w, both(-0x1.777a5cp-23f));   // 2 pi in two parts
    const f32x2 sn = fma2(y, both(0x1.921fb6p+2f), mul2(y, a));
    f32x2 b = fma2(w, both(0x1.d4f7ecp+5f), both(-0x1.55b2b6p+6f));
    b = fma2(b, w, both(0x1.03c1bp+6f));
    b = fma2(b, w, both(-0x1.3bd3ccp+4f));
    const f32x2 cs = fma2(b, w, both(1.0f));
    float sv[2], cv[2], nv[2];
    unpack(sn, sv[0], sv[1]);
    unpack(cs, cv[0], cv[1]);
    unpack(n, nv[0], nv[1]);
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const uint32_t q = __float_as_uint(nv[i]);
        const float u = (q & 1u) ? cv[i] : sv[i], v = (q & 1u) ? sv[i] : cv[i];
        s[i] = __uint_as_float(__float_as_uint(u) ^ (q << 30 & 0x80000000u));
        c[i] = __uint_as_float(__float_as_uint(v) ^ ((q + 1u) << 30 & 0x80000000u));
    }
}

// Two Box–Muller pairs from the four words of a block: u = ((w >> 8) + 0.5) 2^-24, z0 = r sin(2 pi u2), z1 =
// r cos(2 pi u2), r = sqrt(-2 ln u1).  The pairs share the packed instructions: a path-step of the GBM
// European pass issues 32 instructions where logf, sqrtf and sincospif made it 52, and is bound by the wide
// multiplies of the Philox rounds and the packed ones together (0.54 -> 0.40 ms for 2^22 paths of 64 steps).
// Against FP64 over 2^28 normals, an eighth of them near u1 = 1, u1 = 0 and the quarter turns, in units of
// 2^-23 |z|: at most 1.71 (library functions 1.84), root mean square 0.377 (0.383).
__device__ __forceinline__ void box_muller(uint4 w, float& z0, float& z1, float& z2, float& z3) {
    const f32x2 half = both(0.5f), scale = both(kTwoPow24Inv);
    const f32x2 u1 = mul2(add2(pack((float)(w.x >> 8), (float)(w.z >> 8)), half), scale);
    const f32x2 u2 = mul2(add2(pack((float)(w.y >> 8), (float)(w.w >> 8)), half), scale);
    float ua, ub, s[2], c[2];
    unpack(u1, ua, ub);
    const f32x2 r = root(minus_two_log(ua, ub));
    sincos_turns(u2, s, c);
    unpack(mul2(r, pack(s[0], s[1])), z0, z2);
    unpack(mul2(r, pack(c[0], c[1])), z1, z3);
}

// Normals 32t .. 32t+31 of path `path` on stream `stream` (block b = dims 4b..4b+3).
__device__ __forceinline__ void philox_tile(uint32_t seed, uint32_t stream, uint64_t path, int t,
                                            float (&z)[32]) {
    const uint2 key = make_uint2(seed, 0x6D637121u);
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const uint4 o = philox10(make_uint4((uint32_t)(8 * t + q), (uint32_t)path,
                                            (uint32_t)(path >> 32), stream), key);
        box_muller(o, z[4 * q], z[4 * q + 1], z[4 * q + 2], z[4 * q + 3]);
    }
}

}  // namespace mcq
