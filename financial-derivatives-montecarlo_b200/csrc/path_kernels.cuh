// path_kernels.cuh — the fused path kernel for sm_100a.
//
// One launch prices R replicas x n_points paths end to end: point generation (scrambled
// Sobol or Philox), noise transform (raw, Brownian bridge), Euler stepping of the model,
// running payoff accumulator, payoff / control-variate / importance-sampling weights,
// Kahan accumulation per lane and a warp-shuffle reduction per work item.  No path array
// is ever written to HBM; the only global writes are one partial-sum record per item.
//
// This fuses what the reference does in up to five passes over a D x N array in HBM:
//   kernel_gen_hh_scrambled_sobol_normal / curandGenerateNormal   (methods_cuda.cu:799-825)
//   kernel_scale / kernel_bb_transform                             (:561-594, :714-718)
//   kernel_mc / kernel_mlmc / kernel_gbm_asian_cv / kernel_dupire_gbm_cv / kernel_is_gbm
//   with CUB_REDUCE2/4 + atomicAdd                                 (:359-381, :414-707)
//
// Work layout.  Points are taken in aligned groups of 32 consecutive indices, one group per
// warp at a time (lane i owns point 32h + i).  A work item is a run of `gpi` groups of one
// replica; warps take items round-robin.  Item boundaries depend only on the problem size, so
// the result is bit-reproducible run to run.
//
// Sobol generation (warp-transposed, in strata order).  For a tile of 32 dimensions, lane j owns
// dimension d0 + j and produces its scrambled integers for all 32 points of the group: one XOR per
// point with direction words already multiplied by the replica's Hong–Hickernell matrix (linearity of
// the scramble over F2) instead of 32 splitmix32 rows + 32 popcounts (hh_scramble,
// methods_cuda.cu:781-795).  Each dimension's 32 points of an aligned group fall into the 32 strata
// [s/32, (s+1)/32) once each, so the lanes visit them stratum by stratum, all lanes in the same one at a
// time: the inverse normal is then a polynomial with compile-time coefficients (inv_normal.cuh).  The
// point a lane visits in a stratum is its own; its normal goes to that point's row of a 32x32
// XOR-swizzled shared-memory tile and comes back one row (one path) per lane.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>
#include <utility>
#include <cuda_fp16.h>
#include "inv_normal.cuh"
#include "kparams.h"
#include "philox.cuh"

namespace mcq {

constexpr float kLog2e = 1.4426950408889634f;

// Programmatic dependent launch (launch_dependent): wait for the kernel before; nothing without the launch
// attribute.  No kernel lets its successor start early: pass CTAs placed beside the running prescramble
// CTAs ended up unevenly over the SMs (Heston level 680 -> 714 us).
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ------------------------------------------------------------------ hashing / scrambling

// splitmix32 (methods_cuda.cu:753-759).
__host__ __device__ __forceinline__ uint32_t splitmix32(uint32_t x) {
    x += 0x9E3779B9u;
    x = (x ^ (x >> 16)) * 0x21F0AAADu;
    x = (x ^ (x >> 15)) * 0x735A2D97u;
    return x ^ (x >> 15);
}

// Hong–Hickernell lower-triangular F2 matrix applied to v, row k MSB-first, without the
// digital shift (the linear part of hh_scramble, methods_cuda.cu:781-795).
__device__ __forceinline__ uint32_t hh_linear(uint32_t v, uint32_t base) {
    uint32_t out = 0;
#pragma unroll
    for (int k = 0; k < 32; k++) {
        uint32_t seed = splitmix32(base ^ (uint32_t)k);
        uint32_t mask = (k == 0) ? 0u : (0xFFFFFFFFu << (32 - k));
        uint32_t row = (1u << (31 - k)) | (seed & mask);
        out |= ((uint32_t)__popc(row & v) & 1u) << (31 - k);
    }
    return out;
}

// ------------------------------------------------------------------ transpose buffer

// 32 x 32 floats per warp, 16-byte chunks XOR-swizzled by row so that column writes
// (lane = column) and float4 row reads (lane = row) are both bank-conflict free.  A tile starts at a
// multiple of 4096 bytes of the shared window (kTileBytes; tile_base), so that the byte offset of (row,
// col) is the XOR of row_bits(row) and 4 col and can be walked by XORs alone.
__device__ __forceinline__ int swz(int row, int col) {
    return row * 32 + ((((col >> 2) ^ (row & 7)) << 2) | (col & 3));
}

__host__ __device__ __forceinline__ constexpr uint32_t row_bits(uint32_t row) {
    return (row << 7) ^ ((row & 7u) << 4);
}
// The first tile of a kernel's dynamic shared memory: launches add kTilePad to what they use.
__device__ __forceinline__ float* tile_base(void* smem) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem);
    return reinterpret_cast<float*>(static_cast<char*>(smem) + ((0u - a) & (kTileBytes - 1)));
}

__device__ __forceinline__ void read_row(const float* buf, int lane, float (&z)[32]) {
    const float4* b4 = reinterpret_cast<const float4*>(buf + lane * 32);
#pragma unroll
    for (int c = 0; c < 8; c++) {
        float4 v = b4[c ^ (lane & 7)];
        z[4 * c + 0] = v.x; z[4 * c + 1] = v.y; z[4 * c + 2] = v.z; z[4 * c + 3] = v.w;
    }
}

// The 32 points of an aligned group are x = X ^ (combination of the five words L0..L4), their top five
// bits taking every value once (the scramble is lower, the Sobol matrix upper triangular with unit
// diagonals, so the leading 5 x 5 block of their product is invertible).  k_prescramble therefore
// stores, per dimension, the basis in reduced form: R_k, the combination whose top five bits are bit k
// alone, with the row offset of its points (row_bits of the point index), and every other word and
// the digital shift reduced to zero top bits, where the row of that word goes instead.  A packed word
// is so the group's point of stratum 0: x (top bits zero) and its row, both walked by the same XORs.
//
// Packed start word of group h: shift ^ W_{5+k} over the set bits k of gray(h), and, for odd h,
// the row 31 that bit 4 of gray(32h) contributes.  A caller that generates the same dimension for groups
// h - 1, h, h + 1, ... in order keeps the packed word of each tile in the shared-memory word at address `slot` (0:
// none) and passes cont from the second group on: one word instead of the walk and its chain of
// dependent loads.
struct TileWalk {
    uint32_t x, a;          // point and shared-memory address of the current stratum
    uint2 R0, R1, R2, R3, R4;   // .x: R_k, .y: the row bits of its row
};

// The packed word of group h's point of stratum 0.
__device__ __forceinline__ uint32_t start_word(const uint32_t* __restrict__ dr, int D, int dim, uint64_t h,
                                               uint32_t slot, bool cont) {
    const uint32_t* col = dr + dim;
    if (cont) {
        uint32_t w;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(slot));
        return w ^ 0xF8000000u ^ __ldg(col + (kDirRowW5 - 1 + __ffsll((long long)h)) * D);
    }
    uint32_t s = __ldg(col + kDirRowShift * D) ^ (0u - ((uint32_t)h & 1u) & 0xF8000000u);
    uint32_t g = (uint32_t)(h ^ (h >> 1));
    while (g) {
        s ^= __ldg(col + (kDirRowW5 - 1 + __ffs(g)) * D);
        g &= g - 1;
    }
    return s;
}

// The walk from packed word START() of the tile at `base`.
template <class START>
__device__ __forceinline__ TileWalk tile_walk(const uint32_t* __restrict__ dr, int D, int dim, uint32_t base,
                                              const START& start) {
    const uint2* rk = reinterpret_cast<const uint2*>(dr) + dim;
    TileWalk w;
    w.R0 = __ldg(rk);
    w.R1 = __ldg(rk + D);
    w.R2 = __ldg(rk + 2 * D);
    w.R3 = __ldg(rk + 3 * D);
    w.R4 = __ldg(rk + 4 * D);
    const uint32_t s = start();
    w.x = s & 0x07FFFFFFu;
    w.a = base ^ row_bits(s >> 27);
    return w;
}

// Visits the strata in gray-code order 0, 1, 3, 2, ...: one step per template index.
template <int T, bool PARITY, class STORE>
__device__ __forceinline__ void stratum_step(TileWalk& w, float u_cap, const STORE& store) {
    if constexpr (T > 0) {
        constexpr int k = (T & 1) ? 0 : (T & 2) ? 1 : (T & 4) ? 2 : (T & 8) ? 3 : 4;
        const uint2 R = k == 0 ? w.R0 : k == 1 ? w.R1 : k == 2 ? w.R2 : k == 3 ? w.R3 : w.R4;
        w.x ^= R.x;
        w.a ^= R.y;
    }
    if constexpr (PARITY) store(w.a, sobol_normal(w.x, u_cap));
    else store(w.a, stratum_normal<T ^ (T >> 1)>(w.x, u_cap));
}
template <bool PARITY, class STORE, int... T>
__device__ __forceinline__ void all_strata(TileWalk& w, float u_cap, const STORE& store,
                                           std::integer_sequence<int, T...>) {
    (stratum_step<T, PARITY>(w, u_cap, store), ...);
}

// Lane owns dimension `dim` of replica table `dr` (kDirRows rows of D words); writes the normals of
// points 32h .. 32h+31 into column `lane` of the transpose tile.  PARITY: every normal from
// normcdfinvf, the bits of the reference's generator (the exports); the priced passes take the
// strata's polynomials.  Every lane takes part, one beyond the path's dimensions
// in a column nobody reads (the table covers whole tiles, table_dims): the branch around the tile cost 0.5 of 18.7
// instructions per normal.
template <bool PARITY = false>
__device__ __forceinline__ void sobol_tile(const uint32_t* __restrict__ dr, int D, int dim, uint64_t h,
                                           float u_cap, float* buf, int lane, uint32_t slot = 0,
                                           bool cont = false) {
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(buf) ^ ((uint32_t)lane << 2);
    TileWalk w = tile_walk(dr, D, dim, base, [&] {
        const uint32_t s = start_word(dr, D, dim, h, slot, cont);
        if (slot) asm volatile("st.shared.u32 [%0], %1;" ::"r"(slot), "r"(s) : "memory");
        return s;
    });
    all_strata<PARITY>(
        w, u_cap,
        [](uint32_t a, float z) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(z) : "memory"); },
        std::make_integer_sequence<int, 32>{});
}

// The same with the slot as a pointer, for the baskets compiled for three CTAs per SM (up to eight assets): there the
// address form's volatile accesses cost more than they save.  Address over pointer, 16 x 2^17 paths of about 260
// dimensions, GBM / Dupire: 1 asset 1.013 / 1.025, 2 1.012 / 1.027, 4 1.081 / 1.038, 5 1.136 / 1.085, 7 1.164 / 1.069, 8
// 1.122 / 1.060; 9 to 16 assets 0.98 to 1.01.
__device__ __forceinline__ void sobol_tile_slot(const uint32_t* __restrict__ dr, int D, int dim, uint64_t h, float u_cap,
                                                float* buf, int lane, uint32_t* slot, bool cont) {
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(buf) ^ ((uint32_t)lane << 2);
    TileWalk w = tile_walk(dr, D, dim, base, [&] {
        const uint32_t s = slot != nullptr && cont
                               ? *slot ^ 0xF8000000u ^ __ldg(dr + dim + (kDirRowW5 - 1 + __ffsll((long long)h)) * D)
                               : start_word(dr, D, dim, h, 0, false);
        if (slot != nullptr) *slot = s;
        return s;
    });
    all_strata<false>(
        w, u_cap,
        [](uint32_t a, float z) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(z) : "memory"); },
        std::make_integer_sequence<int, 32>{});
}

// The generator's plain form, for the estimators whose outputs turn on single paths (the book's digital
// deltas, the adjoint's node vegas): points in order and every normal from normcdfinvf, from the plain
// table of 33 rows (words 0..31, shift).  Lane j's start word x(32h) = shift ^ XOR of v_k over the set
// bits k of gray(32h), gray(32h) = gray(h) << 5 | (h & 1) << 4, then x(32h+i+1) = x(32h+i) ^
// v_{ctz(i+1)}; slot and cont as in tile_walk (x(32h) = x(32(h - 1)) ^ v_4 ^ v_{5 + ctz(h)}).  The four
// blocks of eight points are rolled: unrolled, the inlined inverse normal fills the instruction
// cache of these kernels (book 641 -> 602 options/s).
__device__ __forceinline__ void sobol_tile_plain(const uint32_t* __restrict__ dr, int D, int dim, bool active,
                                                 uint64_t h, float u_cap, float* buf, int lane,
                                                 uint32_t* slot = nullptr, bool cont = false) {
    if (!active) return;
    const uint32_t* col = dr + dim;
    const uint32_t L0 = __ldg(col), L1 = __ldg(col + D), L2 = __ldg(col + 2 * D),
                   L3 = __ldg(col + 3 * D), L4 = __ldg(col + 4 * D);
    uint32_t x;
    if (slot != nullptr && cont) {
        x = *slot ^ L4 ^ __ldg(col + (4 + __ffsll((long long)h)) * D);
    } else {
        x = __ldg(col + 32 * D);
        if (h & 1) x ^= L4;
        uint32_t g = (uint32_t)(h ^ (h >> 1));
        while (g) {
            x ^= __ldg(col + (4 + __ffs(g)) * D);
            g &= g - 1;
        }
    }
    if (slot != nullptr) *slot = x;
#pragma unroll 1
    for (int b = 0; b < 4; b++) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            buf[swz(8 * b + i, lane)] = sobol_normal(x, u_cap);
            // word ctz(i + 1) as bit tests of i, which fold (a recursive constexpr ctz of the loop
            // index does not)
            if (i < 7) x ^= (i & 1) == 0 ? L0 : ((i & 2) ? L2 : L1);
            else if (b < 3) x ^= (b == 1) ? L4 : L3;
        }
    }
}

// ------------------------------------------------------------------ accumulation

__device__ __forceinline__ void kadd(float& s, float& c, float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

template <int NST>
struct Acc {
    float s[NST], c[NST];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < NST; i++) s[i] = c[i] = 0.f;
    }
    __device__ __forceinline__ void add(const float (&y)[NST]) {
#pragma unroll
        for (int i = 0; i < NST; i++) kadd(s[i], c[i], y[i]);
    }
    // Warp total in FP64 (fixed shuffle order), lane 0 stores the item record.
    __device__ __forceinline__ void flush(double* out, int lane) {
#pragma unroll
        for (int i = 0; i < NST; i++) {
            double v = (double)s[i] - (double)c[i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) out[i] = v;
        }
    }
};

// Accumulator for consumers with many statistics: each group's 32 values are reduced in FP32
// by shuffles and lane 0 adds the group total to an FP64 record in the warp's shared memory.
template <int NST>
struct AccWarp {
    double* rec;
    __device__ __forceinline__ void bind(double* r, int lane) {
        rec = r;
        if (lane < NST) rec[lane] = 0.0;
        __syncwarp();
    }
    __device__ __forceinline__ void add(const float (&y)[NST], bool valid, int lane) {
#pragma unroll
        for (int i = 0; i < NST; i++) {
            float v = valid ? y[i] : 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) rec[i] += (double)v;
        }
    }
    __device__ __forceinline__ void flush(double* out, int lane) {
        __syncwarp();
        if (lane < NST) out[lane] = rec[lane];
        __syncwarp();
    }
};

// ------------------------------------------------------------------ models and payoffs

// Grid local volatility, bilinear in (S, t) on the uniform axes.  Every path of a step k shares
// t = k h, so the time axis comes from a per-step row {j nK (as float bits), b} that the engine forms
// once per pass (k_lv_rows) with these expressions; the paths then read it instead of clamping,
// truncating and converting t at every step (the same values, bit for bit).
__device__ __forceinline__ float2 lv_time_row(const KParams& p, int k) {
    const float t = (float)k * p.h;
    float y = (t - p.lv_t0) * p.lv_inv_dt;
    y = fminf(fmaxf(y, 0.f), (float)(p.lv_nt - 1));
    const int j = min((int)y, p.lv_nt - 2);
    return make_float2(__int_as_float(j * p.lv_nK), y - (float)j);
}

__device__ __forceinline__ float lv_sigma_row(const KParams& p, float S, float2 row) {
    float x = (S - p.lv_K0) * p.lv_inv_dK;
    x = fminf(fmaxf(x, 0.f), (float)(p.lv_nK - 1));
    const int i = min((int)x, p.lv_nK - 2);
    const float a = x - (float)i;
    const float b = row.y;
    const float* g = p.lv + __float_as_int(row.x) + i;
    const float s00 = __ldg(g), s01 = __ldg(g + 1), s10 = __ldg(g + p.lv_nK),
                s11 = __ldg(g + p.lv_nK + 1);
    const float lo = fmaf(a, s01 - s00, s00), hi = fmaf(a, s11 - s10, s10);
    return fmaf(b, hi - lo, lo);
}

// sqrt(V+) of the Heston step with the hardware's approximate square root (`sqrt.approx.ftz.f32`,
// relative error about 2^-23, exact at 0 and +inf) instead of the correctly rounded one, whose
// refinement and special-case branch cost 9 % of a coupled Heston level pass.  The error scales
// the diffusion coefficient of S and V by 1 +- 1e-7 and does not enter any drift, so it biases
// neither the level means nor their differences.  (ftz: a variance below 2^-126 counts as 0; without
// it each root carries a rescaling of such arguments.)
__device__ __forceinline__ float sqrt_approx(float v) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// Parametric Dupire local volatility sigma0 e^{-alpha t} (S/S0)^(beta - 1) = sigma0 2^{(beta - 1) log2(S/S0)
// + at}, x = S/S0 and at = -alpha t log2(e) (step number times KParams::dup_f or dup_c), with the hardware's
// approximate base-2 logarithm and exponential (`lg2.approx.ftz.f32`, `ex2.approx.ftz.f32`: errors about
// 2^-22, the same special values: log2 of 0 is -inf, of a negative x NaN, 2^-inf = 0).  As with the Heston
// square root, the error scales the volatility (1 +- 1e-6), which multiplies only the mean-zero
// increment: it biases no drift.
__device__ __forceinline__ float dupire_vol(const KParams& p, float x, float at) {
    float l, e;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(x));
    const float a = fmaf(p.bm1, l, at);
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(a));
    return p.sigma0 * e;
}

template <int PAY>
__host__ __device__ constexpr bool path_dep() {
    return PAY == PAY_ASIAN || PAY == PAY_GEOM || PAY == PAY_LOOKBACK || PAY == PAY_UPOUT ||
           PAY == PAY_DOWNOUT;
}

// One discretisation of one single-asset path (d_euler_gbm / d_euler_heston / d_euler_dupire
// and d_running_* / d_apply_bgk / d_payoff, methods_cuda.cu:270-352).  The Euler update is
// S + S (mu h + vol dW), two FMAs; the reference's S + mu S h + vol S dW differs only in
// rounding.  (Folding the drift into a constant 1 + mu h would round that constant once and
// repeat the same relative error on every step: a systematic drift bias of up to 3e-4 of
// mu h per step that does not cancel between the fine and coarse paths of an MLMC level.)
template <int MOD, int PAY>
struct Leg {
    // running accumulator: the Asian sum keeps a plain partial `tp` over at most 32
    // steps that flush() folds into the Kahan pair (r0, r1); extrema live in r0
    float S, V, r0, r1, tp;
    // Geometric average: the running product, its mantissa in r0 (1 <= r0 < 2) and its exponent in ge, one
    // logarithm per path instead of one per step (42.8 -> 20.8 instructions per path-step of the GBM
    // pass).  The product's n roundings of 2^-24 stay below those of n logarithms and their sum.  The mantissa is
    // kept in [2^a, 2^(a+1)), a from S0 (KParams::geo_win): from [1/2, 1) every price from 2^-125 to the largest float
    // has a normal product, from [2^23, 2^24) every positive one below 2^104.  gu: the largest bits(S) - geo_low; from
    // geo_span on, some price was none of these.  (A branch that scales such prices one by one: 856 -> 1032 us for GBM
    // and 1261 -> 2352 us for PCA, 32 x 2^17 paths of 256 steps.)
    int ge;
    uint32_t gu;
    static constexpr bool SUM = (PAY == PAY_ASIAN);
    __device__ __forceinline__ void init(const KParams& p) {
        S = p.S0; V = p.v0; r1 = 0.f; tp = 0.f;
        r0 = (PAY == PAY_LOOKBACK || PAY == PAY_DOWNOUT) ? p.S0 : PAY == PAY_GEOM ? __uint_as_float(p.geo_win) : 0.f;
        ge = 127 - (int)(p.geo_win >> 23);
        gu = 0;
    }
    __device__ __forceinline__ void multiply(const KParams& p, bool on) {
        const uint32_t b = __float_as_uint(r0 * S), u = __float_as_uint(S) - p.geo_low;
        if (on) {
            ge += (int)(b >> 23) - (int)(p.geo_win >> 23);
            r0 = __uint_as_float((b & 0x007fffffu) | p.geo_win);
            gu = max(gu, u);
        }
    }
    __device__ __forceinline__ void flush() {
        if constexpr (SUM) { kadd(r0, r1, tp); tp = 0.f; }
    }
    __device__ __forceinline__ void update(const KParams& p) {
        if constexpr (PAY == PAY_ASIAN) tp += S;
        else if constexpr (PAY == PAY_GEOM) multiply(p, true);
        else if constexpr (PAY == PAY_LOOKBACK || PAY == PAY_DOWNOUT) r0 = fminf(r0, S);
        else if constexpr (PAY == PAY_UPOUT) r0 = fmaxf(r0, S);
    }
    // update() when `on`, as selects rather than a branch per step (the same values)
    __device__ __forceinline__ void update_if(const KParams& p, bool on) {
        if constexpr (PAY == PAY_ASIAN) tp += on ? S : 0.f;
        else if constexpr (PAY == PAY_GEOM) multiply(p, on);
        else if constexpr (PAY == PAY_LOOKBACK || PAY == PAY_DOWNOUT) r0 = on ? fminf(r0, S) : r0;
        else if constexpr (PAY == PAY_UPOUT) r0 = on ? fmaxf(r0, S) : r0;
    }
    // at: step ks's time in the parametric volatility's exponent (the grid model reads its time row ks)
    template <bool RUN>
    __device__ __forceinline__ void step(const KParams& p, float dw1, float dw2, float at,
                                         float muh, float omk, float hstep, int ks) {
        if constexpr (MOD == MOD_GBM) {
            S = fmaf(S, fmaf(p.sigma, dw1, muh), S);
        } else if constexpr (MOD == MOD_DUPIRE) {
            const float sl = dupire_vol(p, S * p.inv_S0, at);
            S = fmaf(S, fmaf(sl, dw1, muh), S);
        } else if constexpr (MOD == MOD_LVGRID) {
            const float sl = lv_sigma_row(p, S, __ldg(p.lv_rows + ks));
            S = fmaf(S, fmaf(sl, dw1, muh), S);
        } else if constexpr (MOD == MOD_HESTON) {
            // S + S (mu h + sqrt(V+) dW1): the drift joins the random increment before the one
            // rounding against S (S + mu h S rounded on its own would quantise the drift of a fine
            // step, a few ulps of S, the same way at every step: a bias at 2^18 steps)
            const float sq = sqrt_approx(fmaxf(V, 0.f));
            const float Sp = S;
            S = fmaf(S, fmaf(sq, dw1, muh), S);
            if (p.flags & MCQ_FLAG_COMPAT_U_INF_CODE) {
                // reference-compat: a path that went infinite (u = 1 point) and whose variance
                // truncates to 0 becomes NaN through the reference's product sqrt(V+) S (:280)
                const float t0 = sq * Sp;
                if (t0 != t0) S = t0;
            }
            // V + (1 - e^{-kappa h}) (theta - V) + xi sqrt(V+) dW2 (+ xi^2/4 (dW2^2 - h) with the
            // Milstein flag): the reference's exact-mean Euler step (:282-283) with 1 - e^{-kappa h}
            // at full relative precision, and every term summed into one increment before the one
            // rounding against V.  A deterministic term rounded against V on its own (V - xi^2 h / 4,
            // or V + (1 - e^{-kappa h})(theta - V)) leaves the same fraction of an ulp every fine
            // step: at 2^18 steps a drift of V of ~0.5 % that the level differences do not cancel.
            // The Milstein choice is a select on the parameter block (no branch per step); without
            // the flag the term is not formed at all, so an infinite normal of the reference-compat
            // u = 1 point leaves V = +inf as the reference's step does, not 0 * inf = NaN.
            float inc = fmaf(p.xi * sq, dw2, omk * (p.theta - V));
            inc = (p.mil != 0.f) ? fmaf(p.mil, fmaf(dw2, dw2, -hstep), inc) : inc;
            V = V + inc;
        }
        if constexpr (RUN && path_dep<PAY>()) update(p);
    }
    // GBM step from a raw normal: S + S (mu h + (sigma sqrt h) z)
    __device__ __forceinline__ void step_gbm_z(const KParams& p, float z, float muh) {
        S = fmaf(S, fmaf(p.sig_sqh, z, muh), S);
        if constexpr (path_dep<PAY>()) update(p);
    }
    // 2^((ge + log2 r0) / n) = 2^q 2^f, q the exponent's integer part and 2^f, 0 <= f <= 1, a polynomial in f - c
    // whose constant 2^c is a float to 1e-5 ulp (fit error 2.5e-9): every path's mean lies in the same narrow
    // range, so an inverse of n or an exponential a little off would bias them all alike.  A path that met a
    // zero, negative, infinite or undefined price (or one outside the product's range) has no geometric mean (NaN,
    // payoff 0), as the compensated sum of logarithms, one of them infinite or undefined, has none.
    __device__ __forceinline__ float geometric_mean(const KParams& p, int n) const {
        if (gu >= p.geo_span) return __int_as_float(0x7fffffff);
        const int g = ge + (int)(p.geo_win >> 23) - 127;
        const float r = __uint_as_float((__float_as_uint(r0) & 0x007fffffu) | 0x3f800000u);
        const int q = min((int)floorf((float)g / (float)n), 127), qn = max(q, -126);
        const float d = ((float)(g - q * n) + log2f(r)) / (float)n - 0x1.00061ap-1f;
        float e = 0x1.c939fcp-13f;
        e = fmaf(e, d, 0x1.f0e27cp-10f);
        e = fmaf(e, d, 0x1.bdbaf4p-7f);
        e = fmaf(e, d, 0x1.4184f2p-4f);
        e = fmaf(e, d, 0x1.5be578p-2f);
        e = fmaf(e, d, 0x1.f5e88cp-1f);
        e = fmaf(e, d, 0x1.6a0ce4p+0f);
        return e * __int_as_float((qn + 127) << 23) * __int_as_float((q - qn + 127) << 23);
    }
    // X - K less what rounding S0 and K to single precision left in the difference (KParams::dK): it shifts
    // every path's payoff alike, so it costs an option at the money 10 to 30 times its relative size.
    __device__ __forceinline__ float over_strike(const KParams& p, float X) const {
        return fmaxf((X - p.K) - p.dK, 0.f);
    }
    // corr, dcorr: the continuity-correction factor and what its rounding leaves out
    __device__ __forceinline__ float payoff(const KParams& p, int n, float corr, float dcorr) const {
        if constexpr (PAY == PAY_EUR || PAY == PAY_BASKET) return over_strike(p, S) * p.disc;
        else if constexpr (PAY == PAY_ASIAN) return over_strike(p, (r0 - r1) / (float)n);
        else if constexpr (PAY == PAY_GEOM) return over_strike(p, geometric_mean(p, n));
        else if constexpr (PAY == PAY_LOOKBACK) return fmaf(-r0, dcorr, fmaf(-r0, corr, S));
        else if constexpr (PAY == PAY_UPOUT) return (r0 / corr >= p.B) ? 0.f : over_strike(p, S) * p.disc;
        else return (r0 * corr <= p.B) ? 0.f : over_strike(p, S) * p.disc;   // PAY_DOWNOUT
    }
};

// ------------------------------------------------------------------ path consumers
// A consumer takes the normals of its path in Sobol-dimension order (raw mode, tile by tile)
// or the time-ordered increments (bridge mode) and produces the estimator's statistics.

// Single-level / coupled fine-coarse path (kernel_mc, kernel_mlmc).
template <int MOD, int PAY, bool COUPLED>
struct PathC {
    // the grid local-vol time rows are those of the fine steps (a coarse leg would need its own)
    static_assert(!(COUPLED && MOD == MOD_LVGRID), "no coupled grid local-vol pass");
    static constexpr int NST = COUPLED ? 4 : 2;
    __device__ __forceinline__ void bind(int, uint64_t) {}
    static constexpr bool HES = (MOD == MOD_HESTON);
    Leg<MOD, PAY> f, c;
    float a1, a2, muh_f, muh_c;   // mu h of the fine and coarse steps
    int k, m, ck;
    bool run_upd;
    __device__ __forceinline__ void init(const KParams& p) {
        f.init(p);
        muh_f = p.mu * p.h;
        k = 0;
        run_upd = !(HES && COUPLED && (p.flags & 2));
        if constexpr (COUPLED) { c.init(p); a1 = a2 = 0.f; m = 0; ck = 0; muh_c = p.mu * p.hc; }
    }
    // one fine step and, coupled, its increments summed for the coarse step
    __device__ __forceinline__ void fine_dw(const KParams& p, float dw1, float dw2) {
        const float t = (float)k * p.dup_f;
        if constexpr (HES && COUPLED) {   // run_upd is a runtime flag only here
            f.template step<false>(p, dw1, dw2, t, muh_f, p.om_f, p.h, k);
            if constexpr (path_dep<PAY>()) f.update_if(p, run_upd);
        } else {
            f.template step<true>(p, dw1, dw2, t, muh_f, p.om_f, p.h, k);
        }
        k++;
        if constexpr (COUPLED) {
            a1 += dw1;
            if constexpr (HES) a2 += dw2;
        }
    }
    // the coarse step on the last M fine increments
    __device__ __forceinline__ void coarse_now(const KParams& p) {
        const float tc = (float)ck * p.dup_c;
        if constexpr (HES) {
            c.template step<false>(p, a1, a2, tc, muh_c, p.om_c, p.hc, ck);
            if constexpr (path_dep<PAY>()) c.update_if(p, run_upd);
        } else {
            c.template step<true>(p, a1, a2, tc, muh_c, p.om_c, p.hc, ck);
        }
        a1 = a2 = 0.f; ck++;
    }
    __device__ __forceinline__ void step_dw(const KParams& p, float dw1, float dw2) {
        fine_dw(p, dw1, dw2);
        if constexpr (COUPLED) {
            if (++m == p.M) {
                coarse_now(p);
                m = 0;
            }
        }
    }
    // A full tile of a coupled pair with M = MM fine steps per coarse step, entered with no fine
    // step pending (m = 0, which holds at every tile boundary when M divides the tile's steps): the
    // coarse steps fall on compile-time positions instead of a counter test per fine step (the same
    // steps in the same order, so the same bits).
    template <int MM>
    __device__ __forceinline__ void tile_mm(const KParams& p, const float (&z)[32]) {
#pragma unroll
        for (int i = 0; i < 32; i++) {
            fine_dw(p, z[i] * p.sqrt_h, 0.f);
            if ((i % MM) == MM - 1) coarse_now(p);
        }
    }
    template <int MM>
    __device__ __forceinline__ void tile_hes_mm(const KParams& p, const float (&z)[32]) {
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const float z1 = z[2 * i], z2 = z[2 * i + 1];
            fine_dw(p, z1 * p.sqrt_h, fmaf(p.L10s, z1, p.L11s * z2));
            if ((i % MM) == MM - 1) coarse_now(p);
        }
    }
    // two Heston steps from a float4 of a transposed tile
    template <int MM>
    __device__ __forceinline__ void tile_smem_mm(const KParams& p, const float4* row4, int lane) {
#pragma unroll 2
        for (int c = 0; c < 8; c++) {
            const float4 v = row4[c ^ (lane & 7)];
            fine_dw(p, v.x * p.sqrt_h, fmaf(p.L10s, v.x, p.L11s * v.y));
            fine_dw(p, v.z * p.sqrt_h, fmaf(p.L10s, v.z, p.L11s * v.w));
            if (MM == 2 || (MM == 4 && (c & 1))) coarse_now(p);
        }
    }
    // raw normals, tile of 32 dimensions starting at a tile boundary
    __device__ __forceinline__ void tile(const KParams& p, const float (&z)[32], int nv) {
        if (nv == 32) {
            if constexpr (HES && COUPLED) {
                if (m == 0 && p.M == 2) {
                    tile_hes_mm<2>(p, z);
                } else if (m == 0 && p.M == 4) {
                    tile_hes_mm<4>(p, z);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        const float z1 = z[2 * i], z2 = z[2 * i + 1];
                        step_dw(p, z1 * p.sqrt_h, fmaf(p.L10s, z1, p.L11s * z2));
                    }
                }
            } else if constexpr (HES) {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const float z1 = z[2 * i], z2 = z[2 * i + 1];
                    step_dw(p, z1 * p.sqrt_h, fmaf(p.L10s, z1, p.L11s * z2));
                }
            } else if constexpr (MOD == MOD_GBM && !COUPLED) {
#pragma unroll
                for (int i = 0; i < 32; i++) f.step_gbm_z(p, z[i], muh_f);
                k += 32;
            } else if constexpr (COUPLED) {
                if (m == 0 && p.M == 2) {
                    tile_mm<2>(p, z);
                } else if (m == 0 && p.M == 4) {
                    tile_mm<4>(p, z);
                } else {
#pragma unroll
                    for (int i = 0; i < 32; i++) step_dw(p, z[i] * p.sqrt_h, 0.f);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 32; i++) step_dw(p, z[i] * p.sqrt_h, 0.f);
            }
        } else {
            if constexpr (HES) {
#pragma unroll
                for (int i = 0; i < 16; i++)
                    if (2 * i < nv) {
                        const float z1 = z[2 * i], z2 = z[2 * i + 1];
                        step_dw(p, z1 * p.sqrt_h, fmaf(p.L10s, z1, p.L11s * z2));
                    }
            } else {
#pragma unroll
                for (int i = 0; i < 32; i++)
                    if (i < nv) step_dw(p, z[i] * p.sqrt_h, 0.f);
            }
        }
        flush();
    }
    // Heston: the same steps fed straight from this lane's row of a transposed tile in shared
    // memory, four normals (two steps) per float4 and the chunk loop rolled; the fully unrolled
    // sixteen steps of tile() (fine and coarse legs) weighed on the instruction cache.  (GBM and Dupire
    // keep tile(): from shared memory they were 2-3 % slower.)
    static constexpr bool SMEM_TILE = HES;
    __device__ __forceinline__ void tile_smem(const KParams& p, const float* buf, int lane, int nv) {
        const float4* row4 = reinterpret_cast<const float4*>(buf + lane * 32);
        if (nv == 32 && (!COUPLED || (m == 0 && (p.M == 2 || p.M == 4)))) {
            if (!COUPLED) tile_smem_mm<0>(p, row4, lane);
            else if (p.M == 2) tile_smem_mm<2>(p, row4, lane);
            else tile_smem_mm<4>(p, row4, lane);
            flush();
            return;
        }
#pragma unroll 2
        for (int c = 0; c < 8; c++) {
            if (4 * c < nv) {
                const float4 v = row4[c ^ (lane & 7)];
                step_dw(p, v.x * p.sqrt_h, fmaf(p.L10s, v.x, p.L11s * v.y));
                if (4 * c + 2 < nv) step_dw(p, v.z * p.sqrt_h, fmaf(p.L10s, v.z, p.L11s * v.w));
            }
        }
        flush();
    }
    // fold the running partial sums (called at least every 32 steps)
    __device__ __forceinline__ void flush() {
        f.flush();
        if constexpr (COUPLED) c.flush();
    }
    __device__ __forceinline__ void finish(const KParams& p, float (&y)[NST]) {
        flush();
        const float pf = f.payoff(p, p.n_steps, p.corr_f, p.dcorr_f);
        if constexpr (COUPLED) {
            const float pc = (p.n_coarse > 0) ? c.payoff(p, p.n_coarse, p.corr_c, p.dcorr_c) : 0.f;
            const float dy = pf - pc;
            y[0] = dy; y[1] = dy * dy; y[2] = pf; y[3] = pf * pf;
        } else {
            y[0] = pf; y[1] = pf * pf;
        }
    }
};

// Arithmetic Asian with geometric-Asian control on the same GBM path (kernel_gbm_asian_cv,
// methods_cuda.cu:601-640): stats {Ya, Ya^2, Ycv, Ycv^2, Yg, Yg^2, Ya*Yg}.
struct CvAsianC {
    __device__ __forceinline__ void flush() {}
    __device__ __forceinline__ void bind(int, uint64_t) {}
    static constexpr int NST = 7;
    float S, sa, ca, sl, cl, muh;
    __device__ __forceinline__ void init(const KParams& p) {
        S = p.S0; sa = ca = sl = cl = 0.f; muh = p.mu * p.h;
    }
    __device__ __forceinline__ void step_dw(const KParams& p, float dw, float) {
        S = fmaf(S, fmaf(p.sigma, dw, muh), S);
        kadd(sa, ca, S);
        kadd(sl, cl, logf(S));
    }
    __device__ __forceinline__ void tile(const KParams& p, const float (&z)[32], int nv) {
#pragma unroll
        for (int i = 0; i < 32; i++)
            if (i < nv) step_dw(p, z[i] * p.sqrt_h, 0.f);
    }
    __device__ __forceinline__ void finish(const KParams& p, float (&y)[NST]) {
        const float n = (float)p.n_steps;
        const float ya = fmaxf((sa - ca) / n - p.K, 0.f);
        const float yg = fmaxf(expf((sl - cl) / n) - p.K, 0.f);
        const float ycv = ya - p.beta_cv * (yg - p.E_ctrl);
        y[0] = ya; y[1] = ya * ya; y[2] = ycv; y[3] = ycv * ycv;
        y[4] = yg; y[5] = yg * yg; y[6] = ya * yg;
    }
};

// Dupire European with a GBM European control on the same increments
// (kernel_dupire_gbm_cv, methods_cuda.cu:642-677).
struct CvDupireC {
    __device__ __forceinline__ void flush() {}
    __device__ __forceinline__ void bind(int, uint64_t) {}
    static constexpr int NST = 7;
    float Sd, Sg, muh;
    int k;
    __device__ __forceinline__ void init(const KParams& p) {
        Sd = Sg = p.S0; muh = p.mu * p.h; k = 0;
    }
    __device__ __forceinline__ void step_dw(const KParams& p, float dw, float) {
        const float sl = dupire_vol(p, Sd * p.inv_S0, (float)k * p.dup_f);
        Sd = fmaf(Sd, fmaf(sl, dw, muh), Sd);
        Sg = fmaf(Sg, fmaf(p.ctrl_sigma, dw, muh), Sg);
        k++;
    }
    __device__ __forceinline__ void tile(const KParams& p, const float (&z)[32], int nv) {
#pragma unroll
        for (int i = 0; i < 32; i++)
            if (i < nv) step_dw(p, z[i] * p.sqrt_h, 0.f);
    }
    __device__ __forceinline__ void finish(const KParams& p, float (&y)[NST]) {
        const float yd = fmaxf(Sd - p.K, 0.f) * p.disc;
        const float yg = fmaxf(Sg - p.K, 0.f) * p.disc;
        const float ycv = yd - p.beta_cv * (yg - p.E_ctrl);
        y[0] = yd; y[1] = yd * yd; y[2] = ycv; y[3] = ycv * ycv;
        y[4] = yg; y[5] = yg * yg; y[6] = yd * yg;
    }
};

// GBM European under the drift-shifted measure Z' = Z + z* with likelihood ratio
// exp(-z* sum Z - N z*^2 / 2) (kernel_is_gbm, methods_cuda.cu:685-707).
struct IsC {
    __device__ __forceinline__ void flush() {}
    __device__ __forceinline__ void bind(int, uint64_t) {}
    static constexpr int NST = 2;
    float S, zs, zc, muh;
    __device__ __forceinline__ void init(const KParams& p) {
        S = p.S0; zs = zc = 0.f; muh = p.mu * p.h;
    }
    __device__ __forceinline__ void tile(const KParams& p, const float (&z)[32], int nv) {
#pragma unroll
        for (int i = 0; i < 32; i++)
            if (i < nv) {
                kadd(zs, zc, z[i]);
                S = fmaf(S, fmaf(p.sigma, (z[i] + p.z_star) * p.sqrt_h, muh), S);
            }
    }
    __device__ __forceinline__ void step_dw(const KParams&, float, float) {}
    __device__ __forceinline__ void finish(const KParams& p, float (&y)[NST]) {
        const float lr = expf(-p.z_star * (zs - zc) - 0.5f * p.z_star * p.z_star * (float)p.n_steps);
        const float v = fmaxf(S - p.K, 0.f) * p.disc * lr;
        y[0] = v; y[1] = v * v;
    }
};

// Multi-asset basket (kernel_multi_dupire, methods_cuda.cu:525-551, with the Cholesky product
// of correlate_multi_dupire :1122-1148 done in registers): dims of step k are k*n + a.
// MOD_MULTI: parametric Dupire per asset; sigma_loc's S0 scale is read per asset from the second
// block of p.bsk (1 / S0 of asset 0 for every asset, the reference's c_p.S0 (:542, :289), or the
// asset's own under MCQ_FLAG_BASKET_OWN_S0); MOD_BASKET: GBM per asset with its own sigma,
// weighted basket.
template <int MOD, int NB>
struct BasketC {
    static constexpr int NST = 2;
    __device__ __forceinline__ void flush() {}
    __device__ __forceinline__ void bind(int, uint64_t) {}
    float S[NB], dw[NB];
    float muh;
    int f, k;
    __device__ __forceinline__ void init(const KParams& p) {
        const int n = p.n_assets;
#pragma unroll
        for (int a = 0; a < NB; a++) { S[a] = (a < n) ? __ldg(p.bsk + a) : 0.f; dw[a] = 0.f; }
        muh = p.mu * p.h;
        f = 0; k = 0;
    }
    __device__ __forceinline__ void feed(const KParams& p, float z) {
        const int n = p.n_assets;
        const float x = z * p.sqrt_h;
        if (p.uncorrelated) {
#pragma unroll
            for (int a = 0; a < NB; a++) if (a == f) dw[a] = x;
        } else {
            const float* Lrow = p.bsk + 3 * n + f;   // L[a][f] at Lrow[a * n]
#pragma unroll
            for (int a = 0; a < NB; a++)
                if (a >= f && a < n) dw[a] = fmaf(__ldg(Lrow + a * n), x, dw[a]);
        }
        if (++f == n) {
            const float t = (float)k * p.dup_f;
#pragma unroll
            for (int a = 0; a < NB; a++) {
                if (a < n) {
                    if constexpr (MOD == MOD_MULTI) {
                        const float sl = dupire_vol(p, S[a] * __ldg(p.bsk + n + a), t);
                        S[a] = fmaf(S[a], fmaf(sl, dw[a], muh), S[a]);
                    } else {
                        S[a] = fmaf(S[a], fmaf(__ldg(p.bsk + n + a), dw[a], muh), S[a]);
                    }
                }
                dw[a] = 0.f;
            }
            f = 0; k++;
        }
    }
    __device__ __forceinline__ void tile(const KParams& p, const float (&z)[32], int nv) {
#pragma unroll
        for (int i = 0; i < 32; i++)
            if (i < nv) feed(p, z[i]);
    }
    __device__ __forceinline__ void step_dw(const KParams&, float, float) {}
    __device__ __forceinline__ void finish(const KParams& p, float (&y)[NST]) {
        const int n = p.n_assets;
        float b = 0.f;
        if constexpr (MOD == MOD_MULTI) {
#pragma unroll
            for (int a = 0; a < NB; a++) if (a < n) b += S[a];
            b = b / (float)n;
        } else {
#pragma unroll
            for (int a = 0; a < NB; a++) if (a < n) b = fmaf(__ldg(p.bsk + 2 * n + a), S[a], b);
        }
        const float v = fmaxf(b - p.K, 0.f) * p.disc;
        y[0] = v; y[1] = v * v;
    }
};

// The same basket on Sobol tiles of whole steps: a tile holds 32 / N steps (32 / N * N of its 32 lanes), so
// every normal of a step sits at a known column of the transposed tile and L x is an unrolled
// triangular product whose factors are constant-bank operands of the parameter block.  BasketC's feed
// takes one normal at a time at a run-time asset index: for five assets it issues eight predicated
// multiply-adds with their loads per normal.  Same operations in the same order.  N is the exact width: at
// 5 assets x 52 steps x 16 x 2^16 paths 1610 -> 324 us a call.
template <int MOD, int N>
struct BasketTileC {
    static constexpr int NST = 2;
    static constexpr bool SMEM_TILE = true;
    static constexpr int TILE_DIMS = 32 / N * N;
    static constexpr bool SLOT_POINTER = N <= 8;   // sobol_tile_slot
    float S[N];
    float muh;
    int k;
    __device__ __forceinline__ void flush() {}
    __device__ __forceinline__ void bind(int, uint64_t) {}
    __device__ __forceinline__ void init(const KParams& p) {
#pragma unroll
        for (int a = 0; a < N; a++) S[a] = p.bkS0[a];
        muh = p.mu * p.h;
        k = 0;
    }
    __device__ __forceinline__ void tile_smem(const KParams& p, const float* buf, int lane, int nv) {
        const float4* row4 = reinterpret_cast<const float4*>(buf + lane * 32);
#pragma unroll
        for (int st = 0; st < 32 / N; st++) {
            if (st * N < nv) {
                float x[N];
#pragma unroll
                for (int c = 0; c < N; c++) {
                    const int col = st * N + c;
                    const float4 v = row4[(col >> 2) ^ (lane & 7)];
                    x[c] = ((col & 3) == 0 ? v.x : (col & 3) == 1 ? v.y : (col & 3) == 2 ? v.z : v.w) * p.sqrt_h;
                }
                const float t = (float)k * p.dup_f;
#pragma unroll
                for (int a = N - 1; a >= 0; a--) {   // the last asset first: x[a] is not needed after asset a
                    float dw = x[a];
                    if (!p.uncorrelated) {
                        dw = 0.f;
#pragma unroll
                        for (int f = 0; f <= a; f++) dw = fmaf(p.bkL[a * (a + 1) / 2 + f], x[f], dw);
                    }
                    const float v = (MOD == MOD_MULTI) ? dupire_vol(p, S[a] * p.bkV[a], t) : p.bkV[a];
                    S[a] = fmaf(S[a], fmaf(v, dw, muh), S[a]);
                }
                k++;
            }
        }
    }
    __device__ __forceinline__ void finish(const KParams& p, float (&y)[NST]) {
        float b = 0.f;
        if constexpr (MOD == MOD_MULTI) {
#pragma unroll
            for (int a = 0; a < N; a++) b += S[a];
            b = b / (float)N;
        } else {
#pragma unroll
            for (int a = 0; a < N; a++) b = fmaf(p.bkW[a], S[a], b);
        }
        const float v = fmaxf(b - p.K, 0.f) * p.disc;
        y[0] = v; y[1] = v * v;
    }
};

// Parity probe: records the normals (raw) or increments (bridge) the pass consumed for one
// path, so tests can compare the fused generation with the reference stream: bit for bit with PARITY
// (the generator's normcdfinvf form), to the last places with the normals the priced passes use.
template <bool PARITY>
struct DumpC {
    __device__ __forceinline__ void flush() {}
    static constexpr int NST = 1;
    float* out;
    int idx;
    bool on;
    __device__ __forceinline__ void init(const KParams&) { idx = 0; }
    __device__ __forceinline__ void bind(const KParams& p, int r, uint64_t n) {
        on = n >= p.offset && n < p.offset + p.n_points;
        out = p.dump + ((size_t)r * p.n_points + (size_t)(n - p.offset)) * (size_t)p.D;
    }
    __device__ __forceinline__ void tile(const KParams&, const float (&z)[32], int nv) {
#pragma unroll
        for (int i = 0; i < 32; i++)
            if (i < nv && on) out[idx + i] = z[i];
        idx += nv;
    }
    __device__ __forceinline__ void step_dw(const KParams&, float dw, float) {
        if (on) out[idx] = dw;
        idx++;
    }
    __device__ __forceinline__ void finish(const KParams&, float (&y)[NST]) { y[0] = 0.f; }
};

// Coupled fine / coarse correlated basket for MLMC / MLQMC levels (the reference refuses
// baskets there, methods_cuda.cu:1318-1320, :1695-1697), with the pathwise delta per asset.
// MOD_BASKET: GBM per asset with its own sigma and a weighted basket.  Euler GBM is linear in
// S0_a, so dS_a(T)/dS0_a = S_a(T)/S0_a and delta_a = disc 1{B > K} w_a S_a(T) / S0_a on each of
// the fine and coarse paths.
// MOD_MULTI: the reference's Dupire basket (parametric local vol per asset, equally weighted
// mean, kernel_multi_dupire :525-551) stepped as kernel_mlmc steps a one-asset Dupire path
// (:471-497): fine steps at t = k h, coarse steps at t = k_c h_c on the summed increments.  Under
// MCQ_FLAG_BASKET_OWN_S0 each asset's volatility is scaled by its own S0, the path is then
// homogeneous of degree one in (S0_a, S_a) and the same delta formula is the total derivative
// dP/dS0_a (the scale inside sigma_loc moving with S0_a, as the one-asset Dupire adjoint); with
// the reference's asset-0 scale it is not, and the deltas are left at 0.
// Statistics: {dY, dY^2, Yf, Yf^2, d delta_0 .. d delta_15}.
template <int MOD, int NB>
struct BasketLevelC {
    static constexpr int NST = 4 + kMaxBasket;
    static constexpr bool WARP_ACC = true;
    float Sf[NB], Sc[NB], dw[NB], acc[NB];
    float muh_f, muh_c;
    int f, m, k, kc;
    __device__ __forceinline__ void bind(int, uint64_t) {}
    __device__ __forceinline__ void flush() {}
    __device__ __forceinline__ void init(const KParams& p) {
        const int n = p.n_assets;
#pragma unroll
        for (int a = 0; a < NB; a++) {
            Sf[a] = Sc[a] = (a < n) ? __ldg(p.bsk + a) : 0.f;
            dw[a] = acc[a] = 0.f;
        }
        muh_f = p.mu * p.h;
        muh_c = p.mu * p.hc;
        f = 0; m = 0; k = 0; kc = 0;
    }
    // sigma_loc(S, t) S-scale: the per-asset inverse reference S0 (second block of p.bsk)
    __device__ __forceinline__ float vol(const KParams& p, int n, int a, float S, float t) const {
        if constexpr (MOD == MOD_MULTI)
            return dupire_vol(p, S * __ldg(p.bsk + n + a), t);
        else
            return __ldg(p.bsk + n + a);
    }
    __device__ __forceinline__ void feed(const KParams& p, float z) {
        const int n = p.n_assets;
        const float x = z * p.sqrt_h;
        if (p.uncorrelated) {
#pragma unroll
            for (int a = 0; a < NB; a++) if (a == f) dw[a] = x;
        } else {
            const float* Lcol = p.bsk + 3 * n + f;
#pragma unroll
            for (int a = 0; a < NB; a++)
                if (a >= f && a < n) dw[a] = fmaf(__ldg(Lcol + a * n), x, dw[a]);
        }
        if (++f == n) {
            const bool coarse = (++m == p.M);
            const float t = (float)k * p.dup_f, tc = (float)kc * p.dup_c;
#pragma unroll
            for (int a = 0; a < NB; a++) {
                if (a < n) {
                    Sf[a] = fmaf(Sf[a], fmaf(vol(p, n, a, Sf[a], t), dw[a], muh_f), Sf[a]);
                    acc[a] += dw[a];
                    if (coarse) {
                        Sc[a] = fmaf(Sc[a], fmaf(vol(p, n, a, Sc[a], tc), acc[a], muh_c), Sc[a]);
                        acc[a] = 0.f;
                    }
                }
                dw[a] = 0.f;
            }
            if (coarse) { m = 0; kc++; }
            f = 0;
            k++;
        }
    }
    __device__ __forceinline__ void tile(const KParams& p, const float (&z)[32], int nv) {
#pragma unroll
        for (int i = 0; i < 32; i++)
            if (i < nv) feed(p, z[i]);
    }
    __device__ __forceinline__ void step_dw(const KParams&, float, float) {}
    __device__ __forceinline__ void finish(const KParams& p, float (&y)[NST]) {
        const int n = p.n_assets;
        float Bf = 0.f, Bc = 0.f;
        if constexpr (MOD == MOD_MULTI) {   // equally weighted mean, as kernel_multi_dupire
#pragma unroll
            for (int a = 0; a < NB; a++)
                if (a < n) { Bf += Sf[a]; Bc += Sc[a]; }
            Bf = Bf / (float)n;
            Bc = Bc / (float)n;
        } else {
#pragma unroll
            for (int a = 0; a < NB; a++)
                if (a < n) {
                    const float w = __ldg(p.bsk + 2 * n + a);
                    Bf = fmaf(w, Sf[a], Bf);
                    Bc = fmaf(w, Sc[a], Bc);
                }
        }
        const bool has_c = p.n_coarse > 0;
        const float yf = fmaxf(Bf - p.K, 0.f) * p.disc;
        const float yc = has_c ? fmaxf(Bc - p.K, 0.f) * p.disc : 0.f;
        const float dy = yf - yc;
        y[0] = dy; y[1] = dy * dy; y[2] = yf; y[3] = yf * yf;
        const bool deltas = (MOD == MOD_BASKET) || (p.flags & MCQ_FLAG_OWN_S0_CODE);
        const float gf = (Bf > p.K) ? p.disc : 0.f, gc = (has_c && Bc > p.K) ? p.disc : 0.f;
#pragma unroll
        for (int a = 0; a < kMaxBasket; a++) {
            float v = 0.f;
            if (a < NB && a < n && deltas) {
                const float wa = __ldg(p.bsk + 2 * n + a) / __ldg(p.bsk + a);
                v = wa * (gf * Sf[a] - gc * Sc[a]);
            }
            y[4 + a] = v;
        }
    }
};

// Wide basket (up to NMAX assets: kMaxWideBasket for the reference's 100-asset example,
// kMaxHugeBasket for its 1000-asset uncorrelated one): the same arithmetic as BasketC with the
// per-asset state in local memory and rolled loops.
template <int MOD, int NMAX = kMaxWideBasket>
struct BasketWideC {
    static constexpr int NST = 2;
    float S[NMAX], dw[NMAX];
    float muh;
    int f, k;
    __device__ __forceinline__ void bind(int, uint64_t) {}
    __device__ __forceinline__ void flush() {}
    __device__ __forceinline__ void init(const KParams& p) {
        const int n = p.n_assets;
#pragma unroll 1
        for (int a = 0; a < n; a++) { S[a] = __ldg(p.bsk + a); dw[a] = 0.f; }
        muh = p.mu * p.h;
        f = 0; k = 0;
    }
    __device__ __forceinline__ void feed(const KParams& p, float z) {
        const int n = p.n_assets;
        const float x = z * p.sqrt_h;
        if (p.uncorrelated) {
            dw[f] = x;
        } else {
            const float* Lcol = p.bsk + 3 * n + f;
#pragma unroll 1
            for (int a = f; a < n; a++) dw[a] = fmaf(__ldg(Lcol + a * n), x, dw[a]);
        }
        if (++f == n) {
            const float t = (float)k * p.dup_f;
#pragma unroll 1
            for (int a = 0; a < n; a++) {
                if constexpr (MOD == MOD_MULTI) {
                    const float sl = dupire_vol(p, S[a] * __ldg(p.bsk + n + a), t);
                    S[a] = fmaf(S[a], fmaf(sl, dw[a], muh), S[a]);
                } else {
                    S[a] = fmaf(S[a], fmaf(__ldg(p.bsk + n + a), dw[a], muh), S[a]);
                }
                dw[a] = 0.f;
            }
            f = 0; k++;
        }
    }
    __device__ __forceinline__ void tile(const KParams& p, const float (&z)[32], int nv) {
#pragma unroll
        for (int i = 0; i < 32; i++)
            if (i < nv) feed(p, z[i]);
    }
    __device__ __forceinline__ void step_dw(const KParams&, float, float) {}
    __device__ __forceinline__ void finish(const KParams& p, float (&y)[NST]) {
        const int n = p.n_assets;
        float b = 0.f;
        if constexpr (MOD == MOD_MULTI) {
#pragma unroll 1
            for (int a = 0; a < n; a++) b += S[a];
            b = b / (float)n;
        } else {
#pragma unroll 1
            for (int a = 0; a < n; a++) b = fmaf(__ldg(p.bsk + 2 * n + a), S[a], b);
        }
        const float v = fmaxf(b - p.K, 0.f) * p.disc;
        y[0] = v; y[1] = v * v;
    }
};

// ------------------------------------------------------------------ Brownian bridge

// Window of 32 increments from the bridge between W_L = W(32q) and W_R = W(32q + 32):
// 31 interior points over five levels, all indices static.  zs[s] is the normal of interior
// slot s (level u = floor(log2(s+1)), position v = s + 1 - 2^u); its Sobol dimension is
// (S << u) + (q << u) + v (bb_precompute's level order, utils.cpp:78-99) and its weights are
// read from the per-dimension table.
template <bool UNI, class C>
__device__ __forceinline__ void bb_window(const KParams& p, C& cons, const float (&zs)[32],
                                          float WL, float WR, int S, int q) {
    float W[33];
    W[0] = WL;
    W[32] = WR;
#pragma unroll
    for (int u = 0; u < 5; u++) {
#pragma unroll
        for (int v = 0; v < (1 << u); v++) {
            const int s = (1 << u) - 1 + v;
            const int half = 16 >> u;
            const int mid = (2 * v + 1) * half, lft = 2 * v * half, rgt = (2 * v + 2) * half;
            float4 w;
            if constexpr (UNI) {   // level weights from the parameter block: no loads
                w = make_float4(p.bbw[u][0], p.bbw[u][1], p.bbw[u][2], 0.f);
            } else {
                w = __ldg(p.bb + (S << u) + (q << u) + v);
            }
            W[mid] = fmaf(w.x, W[lft], fmaf(w.y, W[rgt], w.z * zs[s]));
        }
    }
#pragma unroll
    for (int t = 0; t < 32; t++) cons.step_dw(p, W[t + 1] - W[t], 0.f);
    cons.flush();
}

// ------------------------------------------------------------------ the pass kernel

template <class C, class = void>
struct smem_tile_of { static constexpr bool value = false; };
template <class C>
struct smem_tile_of<C, std::void_t<decltype(C::SMEM_TILE)>> { static constexpr bool value = C::SMEM_TILE; };

template <class C, class = void>
struct tile_dims_of { static constexpr int value = 32; };
template <class C>
struct tile_dims_of<C, std::void_t<decltype(C::TILE_DIMS)>> { static constexpr int value = C::TILE_DIMS; };
template <class C, class = void>
struct slot_pointer_of { static constexpr bool value = false; };
template <class C>
struct slot_pointer_of<C, std::void_t<decltype(C::SLOT_POINTER)>> { static constexpr bool value = C::SLOT_POINTER; };
template <class C>
struct parity_of { static constexpr bool value = false; };
template <>
struct parity_of<DumpC<true>> { static constexpr bool value = true; };
template <class C>
struct is_dump { static constexpr bool value = false; };
template <bool PARITY>
struct is_dump<DumpC<PARITY>> { static constexpr bool value = true; };

// One 32-path group h of a consumer (PLAIN: raw ordering through the generator's plain form).  `carry` (nullptr: none) holds the Sobol start words of
// every tile the group generates, slot 32 t + lane for its t-th tile; cont says that the slots
// hold group h - 1's words of the same replica (see sobol_tile).
template <int GEN, int NOISE, class C, bool PLAIN = false>
__device__ __forceinline__ void run_group(const KParams& p, C& cons, const uint32_t* dr,
                                          uint32_t stream, uint64_t h, uint64_t n, float* buf,
                                          float* skel, int lane, uint32_t* carry = nullptr,
                                          bool cont = false) {
    const int D = p.D;
    constexpr bool PARITY = parity_of<C>::value;
    // this lane's first slot as a shared-memory address (0: no slots)
    const uint32_t slots = carry ? (uint32_t)__cvta_generic_to_shared(carry + lane) : 0u;
    const bool again = slots != 0 && cont;
    if constexpr (NOISE == NOISE_RAW) {
        constexpr int TD = tile_dims_of<C>::value;   // dimensions a tile holds (32 except for baskets)
        for (int d0 = 0, s0 = 0; d0 < D; d0 += TD, s0 += 32) {
            const int nv = min(TD, D - d0);
            if constexpr (GEN == GEN_SOBOL) {
                if constexpr (PLAIN)
                    sobol_tile_plain(dr, p.dstride, d0 + lane, lane < nv, h, p.u_cap, buf, lane,
                                     carry ? carry + s0 + lane : nullptr, cont);
                else if constexpr (slot_pointer_of<C>::value)
                    sobol_tile_slot(dr, p.dstride, d0 + lane, h, p.u_cap, buf, lane, carry ? carry + s0 + lane : nullptr, cont);
                else
                    sobol_tile<PARITY>(dr, p.dstride, d0 + lane, h, p.u_cap, buf, lane, slots ? slots + 4 * s0 : 0, again);
                __syncwarp();
                if constexpr (smem_tile_of<C>::value) {
                    cons.tile_smem(p, buf, lane, nv);
                    __syncwarp();
                } else {
                    float z[32];
                    read_row(buf, lane, z);
                    __syncwarp();
                    cons.tile(p, z, nv);
                }
            } else {
                float z[32];
                philox_tile(p.seed, stream, n, d0 >> 5, z);
                cons.tile(p, z, nv);
            }
        }
    } else if constexpr (NOISE == NOISE_PCA) {
        // N <= 32 (one tile): dW_i = sum_k M[i][k] z_k with z and M rounded to fp16 as the
        // reference's cast + GEMM (methods_cuda.cu:1228-1229); larger N runs in k_pca.
        const int N = D;
        sobol_tile<PARITY>(dr, p.dstride, lane, h, p.u_cap, buf, lane, slots, again);
        __syncwarp();
        float z[32];
        read_row(buf, lane, z);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; j++) z[j] = __half2float(__float2half_rn(z[j]));
        const __half* Mrow = static_cast<const __half*>(p.pca);
        for (int i = 0; i < N; i++) {
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < 32; j++)
                if (j < N) acc = fmaf(__half2float(Mrow[i * N + j]), z[j], acc);
            cons.step_dw(p, acc, 0.f);
        }
        cons.flush();
    } else if constexpr (NOISE == NOISE_DW) {
        // increments produced outside the pass (the large-N PCA product), time-ordered in
        // p.dw_in[i * p.dw_stride + row] for the point offset + row; lanes of a group read
        // consecutive rows (coalesced).  Lanes outside the point range step on zeros.
        const bool valid = n >= p.offset && n < p.offset + p.n_points;
        const float* col = p.dw_in + (valid ? (size_t)(n - p.offset) : (size_t)0);
        for (int t0 = 0; t0 < D; t0 += 32) {
            const int nv = min(32, D - t0);
#pragma unroll 4
            for (int i = 0; i < nv; i++)
                cons.step_dw(p, valid ? __ldg(col + (size_t)(t0 + i) * (size_t)p.dw_stride) : 0.f, 0.f);
            cons.flush();
        }
    } else {   // NOISE_BB, one factor: D == n_steps == N (power of two)
        // Bridge table row j (Sobol dimension j = bb_precompute step j, utils.cpp:54-101):
        // p.bb[j] = {wl, wr, sd, bits(m)} and p.bbi[j] = {l, r}: W[m] = wl W[l] + wr W[r] + sd z_j.
        const int N = D;
        if (N <= 32) {
            // one tile: the literal table-driven bridge (bb_apply, utils.cpp:104-124)
            sobol_tile<PARITY>(dr, p.dstride, lane, h, p.u_cap, buf, lane, slots, again);
            __syncwarp();
            float z[32];
            read_row(buf, lane, z);
            __syncwarp();
            float W[33];
#pragma unroll
            for (int i = 0; i < 33; i++) W[i] = 0.f;
#pragma unroll
            for (int j = 0; j < 32; j++) {
                if (j < N) {
                    const float4 w = __ldg(p.bb + j);
                    const int2 lr = __ldg(p.bbi + j);
                    W[__float_as_int(w.w)] = fmaf(w.x, W[lr.x], fmaf(w.y, W[lr.y], w.z * z[j]));
                }
            }
#pragma unroll
            for (int t = 0; t < 32; t++)
                if (t < N) cons.step_dw(p, W[t + 1] - W[t], 0.f);
            cons.flush();
        } else {
            // Skeleton W(32q), q = 0..S, from dimensions 0..S-1 (all multiples of 32), kept
            // per lane in shared memory at skel[q * 32 + lane]; then S windows of 32 steps.
            const int S = N >> 5;
            skel[lane] = 0.f;
            // carry slots: the skeleton tiles first, then one per window
            const int ns = (S + 31) & ~31;
            for (int t0 = 0; t0 < S; t0 += 32) {
                sobol_tile<PARITY>(dr, p.dstride, t0 + lane, h, p.u_cap, buf, lane,
                           slots ? slots + 4 * t0 : 0, again);
                __syncwarp();
                float z[32];
                read_row(buf, lane, z);
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const int dim = t0 + j;
                    if (dim < S) {
                        const float4 w = __ldg(p.bb + dim);
                        const int2 lr = __ldg(p.bbi + dim);
                        const int mi = __float_as_int(w.w) >> 5, li = lr.x >> 5, ri = lr.y >> 5;
                        skel[mi * 32 + lane] = fmaf(w.x, skel[li * 32 + lane],
                                                    fmaf(w.y, skel[ri * 32 + lane], w.z * z[j]));
                    }
                }
            }
            for (int q = 0; q < S; q++) {
                int dim = 0;
                if (lane < 31) {   // (lane 31: dimension 0 again)
                    const int u = 31 - __clz(lane + 1);
                    dim = (S << u) + (q << u) + (lane + 1 - (1 << u));
                }
                sobol_tile<PARITY>(dr, p.dstride, dim, h, p.u_cap, buf, lane,
                           slots ? slots + 4 * (ns + 32 * q) : 0, again);
                __syncwarp();
                float z[32];
                read_row(buf, lane, z);
                __syncwarp();
                bb_window<NOISE == NOISE_BB_UNI>(p, cons, z, skel[q * 32 + lane], skel[(q + 1) * 32 + lane], S, q);
            }
        }
    }
}

// ------------------------------------------------------------------ assisted passes

// A pass with few 32-path groups and long paths leaves most of the GPU idle: each warp walks its
// paths' whole step sequence alone, and the generation of its normals stalls the sequential
// path arithmetic it cannot overlap with.  Assisted passes give every path-owning warp three
// helper warps that generate its normal tiles ahead into a four-slot shared-memory ring; the
// owner reads each tile (its own row) and runs the consumer.  The normals, the consumer and the
// work items are those of the plain loop, so the sums are the same bits.  Every wait is bounded;
// a warp that gives up records MCQ_ERR_TIMEOUT in p.err and stops.
constexpr uint32_t kAssistWaitLimit = 1u << 26;

__device__ __forceinline__ uint32_t asst_addr(const void* ptr) { return (uint32_t)__cvta_generic_to_shared(ptr); }
__device__ __forceinline__ void asst_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(asst_addr(bar)) : "memory");
}
__device__ __forceinline__ bool asst_wait(uint64_t* bar, uint32_t parity, uint32_t limit = kAssistWaitLimit) {
    const uint32_t a = asst_addr(bar);
    for (uint32_t i = 0; i < limit; i++) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred q;\n mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n"
            " selp.u32 %0, 1, 0, q;\n}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

template <int GEN, class C>
__device__ __forceinline__ void assisted_pass(const KParams& p, unsigned char* smem) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int team = wib / kAssistTeam, role = wib - team * kAssistTeam;   // role 0 owns the paths
    // the teams' tiles first (each at a multiple of kTileBytes), then their mbarriers
    float* tiles = tile_base(smem);
    float* ring = tiles + team * kAssistSlots * 1024;
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + kAssistTeams * kAssistSlots * 1024) + team * 2 * kAssistSlots;
    uint64_t* empty = full + kAssistSlots;
    if (lane == 0 && role == 0) {
        for (int s = 0; s < kAssistSlots; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(asst_addr(&full[s])), "r"(32));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(asst_addr(&empty[s])), "r"(32));
        }
    }
    __syncthreads();
    const int D = p.D, T = (D + 31) >> 5;   // tiles per path
    const uint64_t gend_all = p.g0 + p.G;
    const int total_teams = gridDim.x * kAssistTeams;
    uint32_t u = 0;   // the team's tile sequence number: tile t of group h in item order
    bool stop = false;
    for (int item = blockIdx.x * kAssistTeams + team; item < p.n_items && !stop; item += total_teams) {
        const int r = item / p.items_per_rep;
        const int j = item - r * p.items_per_rep;
        const uint64_t gb = p.g0 + (uint64_t)j * (uint64_t)p.gpi;
        const uint64_t ge = min(gb + (uint64_t)p.gpi, gend_all);
        if (role == 0) {
            Acc<C::NST> acc;
            acc.zero();
            for (uint64_t h = gb; h < ge && !stop; h++) {
                const uint64_t n = h * 32 + (uint64_t)lane;
                C cons;
                cons.init(p);
                cons.bind(r, n);
                for (int t = 0; t < T; t++, u++) {
                    const int s = (int)(u % kAssistSlots);
                    const bool ok = asst_wait(&full[s], (u / kAssistSlots) & 1u);
                    if (!__all_sync(0xffffffffu, ok)) { stop = true; break; }
                    if constexpr (smem_tile_of<C>::value) {
                        cons.tile_smem(p, ring + s * 1024, lane, min(32, D - 32 * t));
                        asst_arrive(&empty[s]);
                    } else {
                        float z[32];
                        read_row(ring + s * 1024, lane, z);
                        asst_arrive(&empty[s]);
                        cons.tile(p, z, min(32, D - 32 * t));
                    }
                }
                if (stop) break;
                float y[C::NST];
                cons.finish(p, y);
                if (n >= p.offset && n < p.offset + p.n_points) acc.add(y);
            }
            if (!stop) acc.flush(p.partials + (size_t)item * C::NST, lane);
        } else {
            const uint32_t* dr = (GEN == GEN_SOBOL) ? p.dirs + (size_t)r * kDirRows * (size_t)p.dstride : nullptr;
            const uint32_t stream = p.stream_base + (uint32_t)r;
            for (uint64_t h = gb; h < ge && !stop; h++) {
                for (int t = 0; t < T; t++, u++) {
                    if ((int)(u % kAssistHelpers) != role - 1) continue;
                    const int s = (int)(u % kAssistSlots);
                    const uint32_t use = u / kAssistSlots;
                    if (use > 0) {   // the owner has read this slot's previous tile
                        const bool ok = asst_wait(&empty[s], (use - 1) & 1u);
                        if (!__all_sync(0xffffffffu, ok)) { stop = true; break; }
                    }
                    float* b = ring + s * 1024;
                    if constexpr (GEN == GEN_SOBOL) {
                        sobol_tile(dr, p.dstride, 32 * t + lane, h, p.u_cap, b, lane);
                    } else {
                        float z[32];
                        philox_tile(p.seed, stream, h * 32 + (uint64_t)lane, t, z);
                        float4* row = reinterpret_cast<float4*>(b + lane * 32);
#pragma unroll
                        for (int c = 0; c < 8; c++)
                            row[c ^ (lane & 7)] = make_float4(z[4 * c], z[4 * c + 1], z[4 * c + 2], z[4 * c + 3]);
                    }
                    asst_arrive(&full[s]);
                }
            }
        }
    }
    if (stop && lane == 0) *(volatile int*)p.err = MCQ_ERR_TIMEOUT_CODE;
}

__host__ __device__ constexpr bool noise_is_bb(int noise) { return noise == NOISE_BB || noise == NOISE_BB_UNI; }

// MINB: resident CTAs per SM the register budget is set for (0: 2 for the bridge, whose
// window keeps 33 W values live, kMinBlocks otherwise).  Variants differ only in register
// allocation and scheduling, never in arithmetic, so they produce identical sums.
template <class C>
struct warp_acc_of { static constexpr bool value = false; };
template <int MOD, int NB>
struct warp_acc_of<BasketLevelC<MOD, NB>> { static constexpr bool value = true; };

template <int GEN, int NOISE, class C, int MINB = 0>
__global__ void __launch_bounds__(kThreads, MINB ? MINB : (noise_is_bb(NOISE) ? 2 : kMinBlocks))
    k_pass(const __grid_constant__ KParams p) {
    extern __shared__ float4 smem4[];
    grid_dependency_wait();
    if constexpr (NOISE == NOISE_ASSIST) {
        assisted_pass<GEN, C>(p, reinterpret_cast<unsigned char*>(smem4));
        return;
    }
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    constexpr bool WACC = warp_acc_of<C>::value;
    const int skel_floats = (noise_is_bb(NOISE) && p.D > 32) ? ((p.D >> 5) + 1) * 32 : 0;
    const int acc_floats = WACC ? ((2 * C::NST + 3) & ~3) : 0;
    // the warps' transpose tiles, then per warp the bridge skeleton, the FP64 record and the carried words
    float* tiles = tile_base(smem4);
    float* buf = tiles + wib * 1024;
    float* skel = tiles + kWarpsPerBlock * 1024 + wib * (skel_floats + acc_floats + p.carry);
    double* wrec = reinterpret_cast<double*>(skel + skel_floats);
    uint32_t* carry = p.carry ? reinterpret_cast<uint32_t*>(skel + skel_floats + acc_floats) : nullptr;
    const int total_warps = gridDim.x * kWarpsPerBlock;
    const uint64_t gend_all = p.g0 + p.G;
    for (int item = blockIdx.x * kWarpsPerBlock + wib; item < p.n_items; item += total_warps) {
        const int r = item / p.items_per_rep;
        const int j = item - r * p.items_per_rep;
        const uint64_t gb = p.g0 + (uint64_t)j * (uint64_t)p.gpi;
        const uint64_t ge = min(gb + (uint64_t)p.gpi, gend_all);
        const uint32_t* dr = (GEN == GEN_SOBOL) ? p.dirs + (size_t)r * kDirRows * (size_t)p.dstride : nullptr;
        const uint32_t stream = p.stream_base + (uint32_t)r;
        Acc<WACC ? 1 : C::NST> acc;
        AccWarp<C::NST> wacc;
        if constexpr (WACC) wacc.bind(wrec, lane);
        else acc.zero();
        if constexpr (NOISE == NOISE_PACKED) {
            // Paths of D <= 16 normals: one Sobol tile holds Q = 32 / D groups (lane j makes
            // dimension j mod D of group h + j / D), and each lane then runs its Q paths from the
            // transposed tile.  The normals and the order of the paths are those of the
            // one-group-per-tile loop below; only the idle lanes of its tiles are put to work.
            const int D = p.D, Q = 32 / D;
            const int qj = lane / D, dj = lane - qj * D;
            for (uint64_t h = gb; h < ge; h += (uint64_t)Q) {
                sobol_tile(dr, p.dstride, dj, min(h + (uint64_t)qj, ge - 1), p.u_cap, buf, lane);
                __syncwarp();
                const int nq = (int)min((uint64_t)Q, ge - h);
                for (int q = 0; q < nq; q++) {
                    const uint64_t n = (h + (uint64_t)q) * 32 + (uint64_t)lane;
                    C cons;
                    cons.init(p);
                    cons.bind(r, n);
                    float z[32];
#pragma unroll
                    for (int c = 0; c < 32; c++) z[c] = (c < 16 && c < D) ? buf[swz(lane, q * D + c)] : 0.f;
                    cons.tile(p, z, D);
                    float y[C::NST];
                    cons.finish(p, y);
                    if (n >= p.offset && n < p.offset + p.n_points) acc.add(y);
                }
                __syncwarp();
            }
        } else {
            for (uint64_t h = gb; h < ge; h++) {
                const uint64_t n = h * 32 + (uint64_t)lane;
                C cons;
                cons.init(p);
                if constexpr (is_dump<C>::value) cons.bind(p, r, n);
                else cons.bind(r, n);
                run_group<GEN, NOISE, C>(p, cons, dr, stream, h, n, buf, skel, lane, carry, h != gb);
                float y[C::NST];
                cons.finish(p, y);
                const bool valid = n >= p.offset && n < p.offset + p.n_points;
                if constexpr (WACC) wacc.add(y, valid, lane);
                else if (valid) acc.add(y);
            }
        }
        if constexpr (WACC) wacc.flush(p.partials + (size_t)item * C::NST, lane);
        else acc.flush(p.partials + (size_t)item * C::NST, lane);
    }
}

}  // namespace mcq
