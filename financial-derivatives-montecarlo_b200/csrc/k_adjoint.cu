// k_adjoint.cu — pathwise adjoint Greeks on scrambled-Sobol paths (no counterpart in the
// reference, which computes no sensitivities).
//
// For each path (lane) the forward sweep steps S_k -> S_{k+1} = S_k (1 + mu h + sigma_k dW_k),
// keeps the payoff state and writes every (S_k, z_k) to the warp's stretch of a scratch array in device
// memory.  The reverse sweep reads them back from the last step to the first and propagates
//     Sbar_k = Sbar_{k+1} dS_{k+1}/dS_k + dP/dS_k,
//     mubar += Sbar_{k+1} S_k h,            sigmabar += Sbar_{k+1} dS_{k+1}/dsigma,
// and, for the grid local-vol model, adds Sbar_{k+1} S_k dW_k w_n to the four bilinear nodes n of
// (S_k, t_k) in an FP32 shared-memory array per CTA (summed per lane over the consecutive steps
// that stay in one grid cell, then added with one native float atomic per node; a path changes
// cell about once a step on the benchmark's grid, and the FP64 shared atomics this replaced were
// the kernel's top stall), whose totals go to the FP64 output once per CTA.  Payoffs are the Lipschitz ones:
// European (discounted), arithmetic Asian and floating-strike lookback (BGK factor constant).
// Per path it yields P, delta = Sbar_0 (plus, for the parametric Dupire model, whose volatility
// (S/S0)^(beta-1) is scaled by S0, the sensitivity through that scale, so that delta is the
// derivative of the price with respect to the model's S0), rho = mubar (+ -T P for the discounted European, the
// drift and the discount sharing the rate) and vega (GBM: d/dsigma; Dupire: d/dsigma0; grid:
// the parallel shift = sum of node vegas; Heston: d/dv0, see k_adjoint_heston).
#include "adjoint.h"
#include "path_kernels.cuh"

namespace mcq {

// Why the whole path is kept: 8 bytes written and read per path-step are a third of the device memory's
// bandwidth at the rate this kernel runs, while generating the normals a second time and recomputing each
// segment from a checkpoint were half of its 271 instructions per path-step.  And because a path is at hand
// until its stretch is written again, the reverse sweep can wait until 32 paths of two groups are in the
// money: the others have no sensitivities.  Local-vol Asian, 512 steps, 16 x 60000 paths: 7.43 ms a call with
// checkpoints, 4.98 with kept paths, 4.70 with several copies of the node array, 3.55 with waiting paths (157
// instructions per path-step).

struct LvEval {
    float sig, dsig;
    int n00;              // node index (j * nK + i) of the lower-left corner
    float w00, w01, w10, w11;
};

// Bilinear sigma(S, t) on the uniform grid exactly as the pricing pass's lv_sigma_row, with dsigma/dS
// and the weights.  The time axis comes from the same per-step rows {j nK (as float bits), b}
// (lv_time_row, path_kernels.cuh), which the CTA forms once in shared memory; the sweeps read them
// instead of clamping, truncating and converting t in both evaluations of a step.
__device__ __forceinline__ LvEval lv_eval_row(const KParams& p, float S, float2 row) {
    LvEval e;
    float x = (S - p.lv_K0) * p.lv_inv_dK;
    const bool inside = x > 0.f && x < (float)(p.lv_nK - 1);
    x = fminf(fmaxf(x, 0.f), (float)(p.lv_nK - 1));
    const int i = min((int)x, p.lv_nK - 2);
    const float a = x - (float)i;
    const int jn = __float_as_int(row.x);
    const float b = row.y;
    const float* g = p.lv + jn + i;
    const float s00 = __ldg(g), s01 = __ldg(g + 1), s10 = __ldg(g + p.lv_nK), s11 = __ldg(g + p.lv_nK + 1);
    const float lo = fmaf(a, s01 - s00, s00), hi = fmaf(a, s11 - s10, s10);
    e.sig = fmaf(b, hi - lo, lo);
    e.dsig = inside ? ((1.f - b) * (s01 - s00) + b * (s11 - s10)) * p.lv_inv_dK : 0.f;
    e.n00 = jn + i;
    e.w00 = (1.f - a) * (1.f - b);
    e.w01 = a * (1.f - b);
    e.w10 = (1.f - a) * b;
    e.w11 = a * b;
    return e;
}

// local volatility and its S-derivative / sigma-parameter derivative for the model at step k
// (t = k h; the grid model reads its time row from `trow`)
template <int MOD>
__device__ __forceinline__ float local_sigma(const KParams& p, float S, int k, const float2* trow, float* dsig_dS,
                                             float* dsig_dpar, LvEval* lv) {
    const float t = (float)k * p.h;
    if constexpr (MOD == MOD_GBM) {
        *dsig_dS = 0.f;
        *dsig_dpar = 1.f;
        return p.sigma;
    } else if constexpr (MOD == MOD_DUPIRE) {
        const float sl = p.sigma0 * exp2f(fmaf(p.bm1, log2f(S * p.inv_S0), -p.alpha * t * kLog2e));
        *dsig_dS = sl * p.bm1 / S;
        *dsig_dpar = sl / p.sigma0;
        return sl;
    } else {
        *lv = lv_eval_row(p, S, trow[k]);
        *dsig_dS = lv->dsig;
        *dsig_dpar = 1.f;
        return lv->sig;
    }
}

// One CTA of 24 warps per SM (80 registers) rather than three of eight, so that the node array can hold
// several copies: a float atomic on shared memory is a compare-and-swap loop that goes round once for
// each lane of the warp on the same node, and the paths of a warp share cells (all of them in the first steps).
// Where one copy does not fit beside 24 warps' tiles and start words (1024 steps and more than 3836 nodes: 233 KB at
// 4096) a launch takes 16 (213 KB with four copies).
constexpr int kAdjWarps = 24;
constexpr int kAdjThreads = kAdjWarps * 32;
constexpr size_t kAdjSmemMax = 227 * 1024;

// A path that waits for its reverse sweep: where it is (stretch * 32 + lane, in the money or not as the sign)
// and, by payoff, P or the step of the minimum.
struct Pending {
    uint32_t from;
    union { float P; int kmin; };
};
constexpr uint32_t kInMoney = 0x80000000u;
__device__ __forceinline__ int pending_stretch(const Pending& e) { return (int)(e.from >> 5 & 1u); }

__device__ __forceinline__ void add_cell(float* nodes, int cell, int nK, int lc, float v00, float v01, float v10,
                                         float v11) {
    atomicAdd(nodes + (cell << lc), v00);
    atomicAdd(nodes + ((cell + 1) << lc), v01);
    atomicAdd(nodes + ((cell + nK) << lc), v10);
    atomicAdd(nodes + ((cell + nK + 1) << lc), v11);
}

// Writes / reads of the path scratch: streamed, each element is read once.
__device__ __forceinline__ void path_store(float4* p, float4 v) { __stcs(p, v); }
__device__ __forceinline__ float4 path_load(const float4* p) { return __ldcs(p); }

template <int MOD, int PAY>
__global__ void __launch_bounds__(kAdjThreads, 1) k_adjoint(const __grid_constant__ KParams p) {
    extern __shared__ float4 smem4[];
    grid_dependency_wait();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int N = p.n_steps;
    float* buf = reinterpret_cast<float*>(smem4) + wib * 1024;       // 32 x 32 transpose tile
    // FP32 node sums of the CTA, 2^lc copies of each node side by side, lane l adding to copy l mod 2^lc
    float* nodes = reinterpret_cast<float*>(smem4) + warps * 1024;
    const int lc = p.node_copies_log2;
    const int node_floats = (MOD == MOD_LVGRID) ? (((p.lv_nK * p.lv_nt << lc) + 3) & ~3) : 0;
    float* my_nodes = nodes + (lane & ((1 << lc) - 1));
    const int trow_floats = (MOD == MOD_LVGRID) ? ((2 * (N + 1) + 3) & ~3) : 0;
    float2* trow = reinterpret_cast<float2*>(nodes + node_floats);   // [N + 1] time rows (grid model)
    // each tile's Sobol start word, carried from group to group: slot 32 t + lane
    uint32_t* carry = reinterpret_cast<uint32_t*>(nodes + node_floats + trow_floats) + wib * N;
    Pending* pend = reinterpret_cast<Pending*>(reinterpret_cast<uint32_t*>(nodes + node_floats + trow_floats) +
                                               warps * N) + wib * 64;
    if constexpr (MOD == MOD_LVGRID) {
        for (int i = threadIdx.x; i < node_floats; i += blockDim.x) nodes[i] = 0.f;
        for (int k = threadIdx.x; k <= N; k += blockDim.x) trow[k] = lv_time_row(p, k);
        __syncthreads();
    }
    const float h = p.h, sqh = p.sqrt_h, muh = p.mu * p.h;
    const int total_warps = gridDim.x * warps;   // a small call's items go to different SMs first
    // two path stretches, used in turn: steps 2q and 2q + 1 of lane l as {S, z, S, z} at [32 q + l]
    const size_t stretch = (size_t)(N / 2 * 32);
    float4* paths = p.path_scratch + (size_t)(blockIdx.x * warps + wib) * (2 * stretch);
    const uint64_t gend_all = p.g0 + p.G;
    for (int item = wib * gridDim.x + blockIdx.x; item < p.n_items; item += total_warps) {
        const int r = item / p.items_per_rep;
        const int j = item - r * p.items_per_rep;
        const uint64_t gb = p.g0 + (uint64_t)j * (uint64_t)p.gpi;
        const uint64_t ge = min(gb + (uint64_t)p.gpi, gend_all);
        const uint32_t* dr = p.dirs + (size_t)r * kPlainRows * (size_t)N;
        Acc<4> acc;   // {P, delta, rho, vega}
        acc.zero();
        int npend = 0, slot = 0;   // paths waiting for their reverse sweep; the stretch the next group writes
        for (uint64_t hg = gb;; hg++) {
            const bool more = hg < ge;
            bool full = false;     // both stretches hold waiting paths
            if (more) {
                const uint64_t n = hg * 32 + (uint64_t)lane;
                const bool valid = n >= p.offset && n < p.offset + p.n_points;
                // ---------------- forward sweep
                float4* path = paths + slot * stretch + lane;
                float S = p.S0, ts = 0.f, tot = 0.f, comp = 0.f, mn = p.S0;
                int kmin = 0;
                for (int d0 = 0; d0 < N; d0 += 32) {
                    sobol_tile_plain(dr, N, d0 + lane, true, hg, p.u_cap, buf, lane, carry + d0 + lane, hg != gb);
                    __syncwarp();
                    // this lane's row of the tile, four steps per float4 (the swizzled layout makes row
                    // reads conflict-free), rolled over the chunks: fully unrolled, the sweeps overflowed
                    // the instruction cache
                    const float4* row4 = reinterpret_cast<const float4*>(buf + lane * 32);
#pragma unroll 1
                    for (int c = 0; c < 8; c++) {
                        const float4 v4 = row4[c ^ (lane & 7)];
                        const float zc[4] = {v4.x, v4.y, v4.z, v4.w};
                        float Sq[4];
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const int k = d0 + 4 * c + q;
                            Sq[q] = S;
                            float dsS, dsP;
                            LvEval lv;
                            const float sig = local_sigma<MOD>(p, S, k, trow, &dsS, &dsP, &lv);
                            S = fmaf(S, fmaf(sig, zc[q] * sqh, muh), S);
                            if constexpr (PAY == PAY_ASIAN) ts += S;
                            if constexpr (PAY == PAY_LOOKBACK) {
                                if (S < mn) { mn = S; kmin = k + 1; }
                            }
                        }
                        float4* to = path + (d0 / 2 + 2 * c) * 32;
                        path_store(to, make_float4(Sq[0], zc[0], Sq[1], zc[1]));
                        path_store(to + 32, make_float4(Sq[2], zc[2], Sq[3], zc[3]));
                    }
                    if constexpr (PAY == PAY_ASIAN) { kadd(tot, comp, ts); ts = 0.f; }
                    __syncwarp();
                }
                // payoff and its direct derivatives: what the reverse sweep starts from
                float P;
                Pending e;
                e.P = 0.f;
                bool live = true;
                if constexpr (PAY == PAY_EUR) {
                    P = fmaxf(S - p.K, 0.f) * p.disc;
                    live = S > p.K;
                    e.P = P;
                } else if constexpr (PAY == PAY_ASIAN) {
                    const float A = (tot - comp) / (float)N;
                    P = fmaxf(A - p.K, 0.f);
                    live = A > p.K;
                } else {   // floating-strike lookback
                    P = S - mn * p.corr_f;
                    e.kmin = kmin;
                }
                e.from = (uint32_t)(slot * 32 + lane) | (live ? kInMoney : 0u);
                // a path out of the money has no sensitivities, and only the others are swept back, 32 of
                // them at a time whatever group they are from (one that left the positive reals is
                // kept: its NaN belongs in the result)
                live = valid && (live || !(S > 0.f && S < __int_as_float(0x7f800000)));
                if (valid) kadd(acc.s[0], acc.c[0], P);
                const uint32_t m = __ballot_sync(0xffffffffu, live);
                if (live) pend[npend + __popc(m & ((1u << lane) - 1u))] = e;
                __syncwarp();
                full = npend > 0 && m != 0;
                npend += __popc(m);
            }
            const int run = npend >= 32 ? 32 : (full || !more) ? npend : 0;
            if (run > 0) {
                // ---------------- reverse sweep
                const bool on = lane < run;
                const Pending e = pend[on ? lane : 0];
                const float4* path = paths + pending_stretch(e) * stretch + (e.from & 31u);
                const bool itm = on && (e.from & kInMoney);
                const float g_all = (PAY == PAY_ASIAN && itm) ? 1.f / (float)N : 0.f;
                float Sbar = g_all;
                if constexpr (PAY == PAY_EUR) Sbar = itm ? p.disc : 0.f;
                if constexpr (PAY == PAY_LOOKBACK) Sbar = itm ? 1.f + ((e.kmin == N) ? -p.corr_f : 0.f) : 0.f;
                float mubar = 0.f, sigbar = 0.f, s0bar = 0.f;
                // grid local vol: the node sensitivities of consecutive steps in the same cell are
                // summed in registers and added to the CTA's node array when the cell changes
                int vcell = -1;
                float v00 = 0.f, v01 = 0.f, v10 = 0.f, v11 = 0.f;
                // four steps at a time, the next four already on their way
                float4 pa = path_load(path + (N / 2 - 2) * 32), pb = path_load(path + (N / 2 - 1) * 32);
#pragma unroll 1
                for (int k0 = N - 4; k0 >= 0; k0 -= 4) {
                    const float Sq[4] = {pa.x, pa.z, pb.x, pb.z}, zq[4] = {pa.y, pa.w, pb.y, pb.w};
                    if (k0 > 0) {
                        const float4* from = path + (k0 / 2 - 2) * 32;
                        pa = path_load(from);
                        pb = path_load(from + 32);
                    }
#pragma unroll
                    for (int q = 3; q >= 0; q--) {
                        const int k = k0 + q;
                        const float Sk = Sq[q];
                        const float dw = zq[q] * sqh;
                        float dsS, dsP;
                        LvEval lv;
                        const float sig = local_sigma<MOD>(p, Sk, k, trow, &dsS, &dsP, &lv);
                        mubar = fmaf(Sbar, Sk * h, mubar);
                        const float sens = Sbar * Sk * dw;     // dP/dsigma_k through this step
                        sigbar = fmaf(sens, dsP, sigbar);
                        // the parametric Dupire volatility is scaled by the model's S0 itself:
                        // d sigma_k / d S0 = -(beta - 1) sigma_k / S0 enters the delta
                        if constexpr (MOD == MOD_DUPIRE) s0bar = fmaf(sens, -p.bm1 * sig * p.inv_S0, s0bar);
                        if constexpr (MOD == MOD_LVGRID) {
                            if (on && sens != 0.f) {
                                if (lv.n00 != vcell) {
                                    if (vcell >= 0) add_cell(my_nodes, vcell, p.lv_nK, lc, v00, v01, v10, v11);
                                    vcell = lv.n00;
                                    v00 = v01 = v10 = v11 = 0.f;
                                }
                                v00 = fmaf(sens, lv.w00, v00);
                                v01 = fmaf(sens, lv.w01, v01);
                                v10 = fmaf(sens, lv.w10, v10);
                                v11 = fmaf(sens, lv.w11, v11);
                            }
                        }
                        const float dS1 = 1.f + muh + sig * dw + Sk * dw * dsS;
                        float direct = 0.f;
                        if constexpr (PAY == PAY_ASIAN) direct = (k >= 1) ? g_all : 0.f;
                        if constexpr (PAY == PAY_LOOKBACK) direct = (k == e.kmin) ? -p.corr_f : 0.f;
                        Sbar = fmaf(Sbar, dS1, direct);
                    }
                }
                if constexpr (MOD == MOD_LVGRID) {
                    if (vcell >= 0) add_cell(my_nodes, vcell, p.lv_nK, lc, v00, v01, v10, v11);
                }
                if (on) {
                    float rho = mubar;
                    if constexpr (PAY == PAY_EUR) rho -= p.pay_T * e.P;
                    kadd(acc.s[1], acc.c[1], Sbar + s0bar);
                    kadd(acc.s[2], acc.c[2], rho);
                    kadd(acc.s[3], acc.c[3], sigbar);
                }
                __syncwarp();
                npend -= run;   // what is left is all from the newest group
                const Pending rest = pend[32 + lane];
                __syncwarp();
                if (lane < npend) pend[lane] = rest;
                __syncwarp();
            }
            if (!more) break;
            if (npend > 0) slot = pending_stretch(pend[0]) ^ 1;   // the stretch that holds no waiting path
        }
        acc.flush(p.partials + (size_t)item * 4, lane);
    }
    if constexpr (MOD == MOD_LVGRID) {
        __syncthreads();
        for (int i = threadIdx.x; i < p.lv_nK * p.lv_nt; i += blockDim.x) {
            double v = 0.0;
            for (int c = 0; c < 1 << lc; c++) v += (double)nodes[(i << lc) + c];
            if (v != 0.0) atomicAdd(p.node_out + i, v);
        }
    }
}

// Heston (two normals per step: dims 2k for the price, 2k + 1 for the variance, correlated by the
// Cholesky row (L10, L11)), the pricing pass's Euler step with full truncation in the square
// root (and, with MCQ_FLAG_HESTON_MILSTEIN, the Milstein term, which does not depend on V):
//     S' = S + S (mu h + sqrt(V+) dW1),   V' = theta + e^{-kappa h} (V - theta) + xi sqrt(V+) dW2.
// The reverse sweep carries (Sbar, Vbar):
//     Sbar_k = Sbar_{k+1} (1 + mu h + sqrt(V+) dW1) + dP/dS_k,
//     Vbar_k = Sbar_{k+1} S_k dW1 s'(V_k) + Vbar_{k+1} (e^{-kappa h} + xi dW2 s'(V_k)),
// with s'(V) = 1 / (2 sqrt V) for V > 0 and the subgradient 0 where the truncation is active.
// Outputs per path: P, delta = Sbar_0, rho = mubar (- T P for the discounted European) and
// vega = Vbar_0 = dP/dv0.  Each step's (S, V, z1, z2) goes through the path scratch.
__device__ __forceinline__ void heston_adj_step(const KParams& p, float& S, float& V, float dw1, float dw2,
                                                float muh) {
    const float sq = sqrtf(fmaxf(V, 0.f));
    // the pricing pass's operations (Leg::step): one rounding against S and one against V
    S = fmaf(S, fmaf(sq, dw1, muh), S);
    float inc = fmaf(p.xi * sq, dw2, p.om_f * (p.theta - V));
    inc = (p.mil != 0.f) ? fmaf(p.mil, fmaf(dw2, dw2, -p.h), inc) : inc;
    V = V + inc;
}

template <int PAY>
__global__ void __launch_bounds__(kThreads, 3) k_adjoint_heston(const __grid_constant__ KParams p) {
    extern __shared__ float4 smem4[];
    grid_dependency_wait();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int N = p.n_steps, D = 2 * N, n_tiles = D / 32;
    float* buf = reinterpret_cast<float*>(smem4) + wib * 1024;   // 32 x 32 transpose tile
    uint32_t* carry = reinterpret_cast<uint32_t*>(reinterpret_cast<float*>(smem4) + kWarpsPerBlock * 1024) + wib * D;
    const float h = p.h, sqh = p.sqrt_h, muh = p.mu * p.h;
    const int total_warps = gridDim.x * kWarpsPerBlock;
    // this lane's path: step k as {S, V, z1, z2} at path[32 k]
    float4* path = p.path_scratch + (size_t)(blockIdx.x * kWarpsPerBlock + wib) * (size_t)(N * 32) + lane;
    const uint64_t gend_all = p.g0 + p.G;
    for (int item = wib * gridDim.x + blockIdx.x; item < p.n_items; item += total_warps) {
        const int r = item / p.items_per_rep;
        const int j = item - r * p.items_per_rep;
        const uint64_t gb = p.g0 + (uint64_t)j * (uint64_t)p.gpi;
        const uint64_t ge = min(gb + (uint64_t)p.gpi, gend_all);
        const uint32_t* dr = p.dirs + (size_t)r * kPlainRows * (size_t)D;
        Acc<4> acc;
        acc.zero();
        for (uint64_t hg = gb; hg < ge; hg++) {
            const uint64_t n = hg * 32 + (uint64_t)lane;
            const bool valid = n >= p.offset && n < p.offset + p.n_points;
            // ---------------- forward sweep
            float S = p.S0, V = p.v0, ts = 0.f, tot = 0.f, comp = 0.f, mn = p.S0;
            int kmin = 0;
            for (int t = 0; t < n_tiles; t++) {
                sobol_tile_plain(dr, D, t * 32 + lane, true, hg, p.u_cap, buf, lane, carry + t * 32 + lane,
                                 hg != gb);
                __syncwarp();
                const float4* row4 = reinterpret_cast<const float4*>(buf + lane * 32);
#pragma unroll 2
                for (int c = 0; c < 8; c++) {
                    const float4 v4 = row4[c ^ (lane & 7)];
                    const float z1[2] = {v4.x, v4.z}, z2[2] = {v4.y, v4.w};
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        const int k = t * 16 + 2 * c + q;
                        path_store(path + k * 32, make_float4(S, V, z1[q], z2[q]));
                        heston_adj_step(p, S, V, z1[q] * sqh, fmaf(p.L10, z1[q], p.L11 * z2[q]) * sqh, muh);
                        if constexpr (PAY == PAY_ASIAN) ts += S;
                        if constexpr (PAY == PAY_LOOKBACK) {
                            if (S < mn) { mn = S; kmin = k + 1; }
                        }
                    }
                }
                if constexpr (PAY == PAY_ASIAN) { kadd(tot, comp, ts); ts = 0.f; }
                __syncwarp();
            }
            float P, g_all = 0.f, Sbar;
            if constexpr (PAY == PAY_EUR) {
                P = fmaxf(S - p.K, 0.f) * p.disc;
                Sbar = (S > p.K) ? p.disc : 0.f;
            } else if constexpr (PAY == PAY_ASIAN) {
                const float A = (tot - comp) / (float)N;
                P = fmaxf(A - p.K, 0.f);
                g_all = (A > p.K) ? 1.f / (float)N : 0.f;
                Sbar = g_all;
            } else {   // floating-strike lookback
                P = S - mn * p.corr_f;
                Sbar = 1.f + ((kmin == N) ? -p.corr_f : 0.f);
            }
            // ---------------- reverse sweep
            float mubar = 0.f, Vbar = 0.f;
            float4 pa = path_load(path + (N - 1) * 32), pb = path_load(path + (N - 2) * 32);
#pragma unroll 1
            for (int k0 = N - 1; k0 >= 0; k0 -= 2) {
                const float4 cur[2] = {pa, pb};
                if (k0 > 1) {
                    pa = path_load(path + (k0 - 2) * 32);
                    pb = path_load(path + (k0 - 3) * 32);
                }
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const int k = k0 - q;
                    const float Sk = cur[q].x, Vk = cur[q].y, z1 = cur[q].z, z2 = cur[q].w;
                    const float dw1 = z1 * sqh, dw2 = fmaf(p.L10, z1, p.L11 * z2) * sqh;
                    const float sq = sqrtf(fmaxf(Vk, 0.f));
                    const float dsq = (Vk > 0.f) ? 0.5f / sq : 0.f;
                    mubar = fmaf(Sbar, Sk * h, mubar);
                    const float nV = fmaf(Sbar, Sk * dw1 * dsq, Vbar * fmaf(p.xi * dw2, dsq, 1.f - p.om_f));
                    float direct = 0.f;
                    if constexpr (PAY == PAY_ASIAN) direct = (k >= 1) ? g_all : 0.f;
                    if constexpr (PAY == PAY_LOOKBACK) direct = (k == kmin) ? -p.corr_f : 0.f;
                    Sbar = fmaf(Sbar, 1.f + muh + sq * dw1, direct);
                    Vbar = nV;
                }
            }
            float rho = mubar;
            if constexpr (PAY == PAY_EUR) rho -= p.pay_T * P;
            float y[4] = {P, Sbar, rho, Vbar};
            if (valid) acc.add(y);
        }
        acc.flush(p.partials + (size_t)item * 4, lane);
    }
}

template <int MOD>
static const void* adj_payoff(int pay) {
    switch (pay) {
        case PAY_EUR: return (const void*)&k_adjoint<MOD, PAY_EUR>;
        case PAY_ASIAN: return (const void*)&k_adjoint<MOD, PAY_ASIAN>;
        case PAY_LOOKBACK: return (const void*)&k_adjoint<MOD, PAY_LOOKBACK>;
        default: return nullptr;
    }
}

const void* lookup_adjoint(int model, int payoff) {
    switch (model) {
        case MOD_GBM: return adj_payoff<MOD_GBM>(payoff);
        case MOD_DUPIRE: return adj_payoff<MOD_DUPIRE>(payoff);
        case MOD_LVGRID: return adj_payoff<MOD_LVGRID>(payoff);
        case MOD_HESTON:
            switch (payoff) {
                case PAY_EUR: return (const void*)&k_adjoint_heston<PAY_EUR>;
                case PAY_ASIAN: return (const void*)&k_adjoint_heston<PAY_ASIAN>;
                case PAY_LOOKBACK: return (const void*)&k_adjoint_heston<PAY_LOOKBACK>;
                default: return nullptr;
            }
        default: return nullptr;
    }
}

// Shared memory of `warps` warps with 2^lc copies of the nodes: tiles, start words, lists, nodes, time rows.
static size_t adjoint_smem(int model, int warps, int n_steps, int n_nodes, int lc) {
    const int D = (model == MOD_HESTON ? 2 : 1) * n_steps;
    const size_t trow = (model == MOD_LVGRID) ? (size_t)((2 * (n_steps + 1) + 3) & ~3) : 0;
    const size_t nodes = (size_t)(((n_nodes << lc) + 3) & ~3);
    const size_t pend = model == MOD_HESTON ? 0 : 64 * sizeof(Pending) / sizeof(float);
    return (warps * (1024 + (size_t)D + pend) + nodes + trow) * sizeof(float);
}

AdjointShape adjoint_shape(int model, int n_steps, int n_nodes) {
    AdjointShape a;
    a.warps = model == MOD_HESTON ? kWarpsPerBlock : kAdjWarps;
    while (a.warps > 8 && adjoint_smem(model, a.warps, n_steps, n_nodes, 0) > kAdjSmemMax) a.warps -= 8;
    // eight copies of each node where they fit beside the warps' tiles and start words
    a.node_copies_log2 = 3;
    while (a.node_copies_log2 > 0 && adjoint_smem(model, a.warps, n_steps, n_nodes, a.node_copies_log2) > kAdjSmemMax)
        a.node_copies_log2--;
    a.smem = adjoint_smem(model, a.warps, n_steps, n_nodes, a.node_copies_log2);
    return a;
}

size_t adjoint_path_bytes(int model, int n_steps) {
    return (size_t)n_steps * 32 * (model == MOD_HESTON ? sizeof(float4) : 2 * sizeof(float2));   // two stretches
}

}  // namespace mcq
