// inv_normal.cuh — the inverse normal of the scrambled-Sobol generator, one polynomial per 1/32 of
// the unit interval.
//
// A tile of the generator (sobol_tile, path_kernels.cuh) visits its 32 points in the order of their
// top five bits, so at every step of the unrolled tile all 32 lanes hold a u in the same stratum
// [s/32, (s+1)/32), s a compile-time constant.  The quantile of such a u needs no logarithm, no branch
// and no table load: z = P_s(u - c_s) with the coefficients of stratum s as immediate operands,
// degree 4 to 8 (two multiplications and two FMAs beside u = 1/2, where the polynomial is odd).  The
// two end strata, whose quantile runs to infinity, take r = sqrt(-log2 t), t the distance to the
// nearer end, and z = sqrt(2 ln 2) r plus a polynomial of degree 9 in r - 3: one branch-free form from
// 1/32 to 2^-32 (normcdfinvf takes both sides of its branch for nearly every warp there).  The parity form
// of the generator, which the bit-level exports use, takes normcdfinvf everywhere.
//
// What it replaces: normcdfinvf for every u, about 24 of the 37.7 thread instructions of a path-step of
// the raw GBM Asian pass.
//
// Accuracy.  u = fma(float(x), 2^-32, 2^-32) is the stream's definition.  For x >= 2^27 (every stratum
// but the first) the added 2^-32 is less than half an ulp and vanishes, so u is float(x) 2^-32 and
// u - c_s = fma(float(x), 2^-32, -c_s) is exact (both are multiples of u's ulp, the difference below
// 2^-5).  The polynomials are least-squares / Lawson fits of the quantile in FP64, the coefficients
// rounded to FP32 one after another with the rest refitted; c_s is the multiple of 2^-24 near the middle
// of the stratum whose quantile is closest to a float (off by 0.001 ulp at most, so the constant term
// adds no bias).  Fit error at most 0.12 ulp of z.  The strata below 1/2 mirror those above.  The end
// strata's polynomial is fitted to the r that lg2.approx and sqrt.approx return (they lie low by 0.43 and 0.12
// units of 2^-23 on average, which the fit takes back).  Against FP64, over one in 13 of the x of each
// stratum, in units of 2^-23 |z|: strata 1-30 at most 0.89 (normcdfinvf 2.0), mean 0.14-0.26 (0.28-0.57),
// mean signed error below 1e-9 (up to 8e-8); end strata at most 1.9 (3.1), root mean square 1.27e-7
// (1.33e-7), mean signed error 1e-9 (5.6e-8).
#pragma once
#include <cstdint>

namespace mcq {

constexpr float kTwoPow32Inv = 2.3283064365386963e-10f;   // 2^-32

// u = ((float)s + 1) * 2^-32 as in methods_cuda.cu:823; u_cap is 1.0f in reference-compat
// mode (u may be 1 -> +inf) and 1 - 2^-24 otherwise.
// ((float)x + 1) * 2^-32 == fma((float)x, 2^-32, 2^-32) bit for bit: scaling by a power of two
// is exact, so both round the same real number once.
__device__ __forceinline__ float sobol_normal(uint32_t x, float u_cap) {
    const float u = fmaf((float)x, kTwoPow32Inv, kTwoPow32Inv);
    return normcdfinvf(fminf(u, u_cap));
}

struct Stratum {
    int degree;
    float c;      // centre
    float k[9];   // z = k[0] + k[1] v + ... , v = u - c (stratum 16: z = v (k[1] + k[2] v^2 + k[3] v^4))
};
// strata 16 .. 30, u in [s/32, (s+1)/32)
struct StrataTable {
    Stratum s[15] = {
        {3, 0x1p-1f, {0.f, 0x1.40d932p+1f, 0x1.4ffdap+1f, 0x1.72dbd2p+2f, 0.f, 0.f, 0.f, 0.f, 0.f}},
        {4, 0x1.180034p-1f, {0x1.e266c4p-4f, 0x1.4314d2p+1f, 0x1.802be6p-2f, 0x1.60d204p+1f, 0x1.667102p+0f,
         0.f, 0.f, 0.f, 0.f}},
        {4, 0x1.28003p-1f, {0x1.93aa9ap-3f, 0x1.472448p+1f, 0x1.499912p-1f, 0x1.80238p+1f, 0x1.44981cp+1f, 0.f,
         0.f, 0.f, 0.f}},
        {4, 0x1.38016p-1f, {0x1.1c620cp-2f, 0x1.4d769p+1f, 0x1.e28684p-1f, 0x1.b3c5ecp+1f, 0x1.fc8b3cp+1f, 0.f,
         0.f, 0.f, 0.f}},
        {4, 0x1.47ffbp-1f, {0x1.70c438p-2f, 0x1.5657dp+1f, 0x1.49bc2ep+0f, 0x1.014362p+2f, 0x1.7e118p+2f, 0.f,
         0.f, 0.f, 0.f}},
        {4, 0x1.58066p-1f, {0x1.c7eaacp-2f, 0x1.62475cp+1f, 0x1.b49512p+0f, 0x1.3c49c4p+2f, 0x1.1d80a6p+3f,
         0.f, 0.f, 0.f, 0.f}},
        {4, 0x1.67fc6p-1f, {0x1.11109ap-1f, 0x1.71e24p+1f, 0x1.1d06f4p+1f, 0x1.949054p+2f, 0x1.b0e956p+3f, 0.f,
         0.f, 0.f, 0.f}},
        {4, 0x1.77fefep-1f, {0x1.408cfap-1f, 0x1.86509ap+1f, 0x1.7493fp+1f, 0x1.0e6316p+3f, 0x1.52433ep+4f,
         0.f, 0.f, 0.f, 0.f}},
        {4, 0x1.87fdf8p-1f, {0x1.72eceep-1f, 0x1.a120a8p+1f, 0x1.ec654ep+1f, 0x1.7b766ap+3f, 0x1.156bap+5f,
         0.f, 0.f, 0.f, 0.f}},
        {5, 0x1.97ffd2p-1f, {0x1.a93816p-1f, 0x1.c4f9d4p+1f, 0x1.4cd446p+2f, 0x1.193b72p+4f, 0x1.e5fa72p+5f,
         0x1.ce4458p+7f, 0.f, 0.f, 0.f}},
        {5, 0x1.a7fe76p-1f, {0x1.e4ba8ap-1f, 0x1.f64338p+1f, 0x1.d2766ap+2f, 0x1.c1e974p+4f, 0x1.d259fap+6f,
         0x1.089b5ep+9f, 0.f, 0.f, 0.f}},
        {5, 0x1.b7fb58p-1f, {0x1.13cda2p+0f, 0x1.1e9fa8p+2f, 0x1.59ba9p+3f, 0x1.8dc99cp+5f, 0x1.fdc79cp+7f,
         0x1.60091cp+10f, 0.f, 0.f, 0.f}},
        {6, 0x1.c80234p-1f, {0x1.3adde8p+0f, 0x1.55cb48p+2f, 0x1.18a33ep+4f, 0x1.98b48ep+6f, 0x1.4f0ebap+9f,
         0x1.31d6c4p+12f, 0x1.1bd794p+15f, 0.f, 0.f}},
        {6, 0x1.d8030cp-1f, {0x1.6aff3p+0f, 0x1.b6655ap+2f, 0x1.0a21b4p+5f, 0x1.0cd352p+8f, 0x1.35b022p+11f,
         0x1.9520e8p+14f, 0x1.0a93a6p+18f, 0.f, 0.f}},
        {8, 0x1.e7ff6p-1f, {0x1.ad0732p+0f, 0x1.46adfp+3f, 0x1.5d50e4p+6f, 0x1.256932p+10f, 0x1.1ace64p+14f,
         0x1.21f894p+18f, 0x1.397a62p+22f, 0x1.b59ec8p+26f, 0x1.056738p+31f}},
    };
};

// End strata: z = kEndSlope r + sum of k[i] (r - 3)^i.
constexpr float kEndSlope = 0x1.2d6abep+0f;   // sqrt(2 ln 2)
struct EndTable {
    float k[10] = {-0x1.4b0e7ep-1f, 0x1.0d9b8ap-3f, -0x1.01e6p-5f, 0x1.075c9cp-7f, -0x1.1715aap-9f,
                                0x1.3287dcp-11f, -0x1.6131eep-13f, 0x1.8170bep-15f, -0x1.2c50c2p-17f, 0x1.b4e718p-21f};
};

// |z| of the end strata from t = min(u, 1 - u) <= 1/32; t = 0 (u = 1 in reference-compat mode) gives
// +inf: the leading coefficient and the linear term are positive.
__device__ __forceinline__ float end_stratum(float t) {
    float l, r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(t));
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(-l));
    const float d = r - 3.0f;
    constexpr EndTable e{};
    float p = e.k[9];
#pragma unroll
    for (int i = 8; i >= 0; i--) p = fmaf(p, d, e.k[i]);
    return fmaf(kEndSlope, r, p);
}

// The normal of x, whose top five bits are S.
template <int S>
__device__ __forceinline__ float stratum_normal(uint32_t x, float u_cap) {
    if constexpr (S == 0) {   // the added 2^-32 counts here
        return -end_stratum(fmaf((float)x, kTwoPow32Inv, kTwoPow32Inv));
    } else if constexpr (S == 31) {   // 1 - u is exact
        return end_stratum(1.0f - fminf((float)x * kTwoPow32Inv, u_cap));
    } else {
        constexpr bool up = S >= 16;   // below 1/2: z(u) = -z(1 - u), P(v) becomes -P(-v)
        constexpr Stratum q = StrataTable{}.s[up ? S - 16 : 15 - S];
        constexpr float c = up ? q.c : 1.0f - q.c;
        const float v = fmaf((float)x, kTwoPow32Inv, -c);
        if constexpr (S == 15 || S == 16) {
            const float w = v * v;
            return v * fmaf(w, fmaf(w, q.k[3], q.k[2]), q.k[1]);
        } else {
            constexpr float even = up ? 1.0f : -1.0f;   // sign of the even-degree terms
            float z = (q.degree & 1) ? q.k[q.degree] : even * q.k[q.degree];
#pragma unroll
            for (int i = q.degree - 1; i >= 0; i--) z = fmaf(z, v, (i & 1) ? q.k[i] : even * q.k[i]);
            return z;
        }
    }
}

}  // namespace mcq
