// k_support.cu — small kernels around the fused pass: per-replica direction-word scrambling,
// the deterministic cross-item reduction, and the Sobol stream export used by parity tests.
#include <cuda_runtime.h>
#include <cstdint>
#include "path_kernels.cuh"
#include "support.h"

namespace mcq {

// Pre-scrambled direction words for salts salt0 .. salt0+R-1 and dims 0..D-1:
// out[r][k][d] = hh_linear(v[d][k], splitmix32(salt) ^ d) for k < 32, and the digital shift
// splitmix32(base ^ 0xA5A5A5A5) at k = 32 (methods_cuda.cu:786-795, :819).  The plain table of the
// stream exports, the book and the adjoint (sobol_tile_plain).
__global__ void k_prescramble_plain(const uint32_t* __restrict__ dv, uint32_t salt0, int R, int D,
                                    uint32_t* __restrict__ out) {
    const long long total = (long long)R * 33 * D;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(idx / (33LL * D));
        const int rem = (int)(idx - (long long)r * 33 * D);
        const int k = rem / D, d = rem - k * D;
        const uint32_t base = splitmix32(salt0 + (uint32_t)r) ^ (uint32_t)d;
        out[idx] = (k < 32) ? hh_linear(__ldg(dv + (size_t)d * 32 + k), base)
                            : splitmix32(base ^ 0xA5A5A5A5u);
    }
}

// The passes' direction table (kDirRows rows per replica, tile_walk in path_kernels.cuh): the same
// words with the first five reduced to a basis of the strata and every other word and the shift
// reduced by it.  One warp per (replica, dimension): lane k forms row k of the scramble matrix and word k
// (32 parities against the rows of all lanes), then one Gauss-Jordan step per stratum bit; the pivots
// are on the diagonal, since the leading 5 x 5 block of (lower x upper) unit triangles has unit leading
// minors.  A block does 32 dimensions of one replica and writes them as rows of 32 (coalesced) from
// shared memory.
__global__ void __launch_bounds__(1024) k_prescramble(const uint32_t* __restrict__ dv, uint32_t salt0, int D,
                                                     uint32_t* __restrict__ out) {
    __shared__ uint32_t st[kDirRows * 33];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int per = (D + 31) >> 5, r = blockIdx.x / per, d0 = (blockIdx.x - r * per) * 32;
    const uint32_t salt = splitmix32(salt0 + (uint32_t)r);
    const int dl = wib, d = d0 + dl;
    if (d < D) {
        const uint32_t base = salt ^ (uint32_t)d;
        const uint32_t mask = lane == 0 ? 0u : 0xFFFFFFFFu << (32 - lane);
        const uint32_t mrow = (1u << (31 - lane)) | (splitmix32(base ^ (uint32_t)lane) & mask);
        const uint32_t v = __ldg(dv + (size_t)d * 32 + lane);
        uint32_t w = 0;
#pragma unroll
        for (int j = 0; j < 32; j++)
            w = (w << 1) | ((uint32_t)__popc(__shfl_sync(0xffffffffu, mrow, j) & v) & 1u);
        uint32_t shift = splitmix32(base ^ 0xA5A5A5A5u), shift_row = 0;
        uint32_t row = lane < 5 ? (2u << lane) - 1u : 0u;   // the point whose gray code is bit `lane`
#pragma unroll
        for (int j = 0; j < 5; j++) {
            const uint32_t pw = __shfl_sync(0xffffffffu, w, j), pr = __shfl_sync(0xffffffffu, row, j);
            if (lane != j && (w >> (31 - j) & 1u)) { w ^= pw; row ^= pr; }
            if (shift >> (31 - j) & 1u) { shift ^= pw; shift_row ^= pr; }
        }
        if (lane < 5) {   // top bits: bit 31 - lane alone, bit 4 - lane of the stratum
            st[(4 - lane) * 66 + 2 * dl] = w;
            st[(4 - lane) * 66 + 2 * dl + 1] = row_bits(row);
        } else {
            st[(kDirRowW5 + lane - 5) * 33 + dl] = w | row << 27;
        }
        if (lane == 0) st[kDirRowShift * 33 + dl] = shift | shift_row << 27;
    }
    __syncthreads();
    uint32_t* o = out + (size_t)r * kDirRows * (size_t)D;
    const int nd = min(32, D - d0);
    for (int i = threadIdx.x; i < kDirRows * 32; i += 1024) {
        if (i < kDirRowW5 * 32) {
            const int k = i >> 6, c = i & 63;
            if (c < 2 * nd) o[2 * ((size_t)k * D + d0) + c] = st[k * 66 + c];
        } else {
            const int row = i >> 5, c = i & 31;
            if (c < nd) o[(size_t)row * D + d0 + c] = st[row * 33 + c];
        }
    }
}

// out[r][s] = sum over j of partials[(r * ipr + j) * nstat + s]; fixed summation order.
__global__ void k_finalize(const double* __restrict__ partials, int ipr, int nstat,
                           double* __restrict__ out) {
    __shared__ double red[256];
    const int r = blockIdx.x, t = threadIdx.x;
    for (int s = 0; s < nstat; s++) {
        double v = 0.0;
        for (int j = t; j < ipr; j += 256) v += partials[((size_t)r * ipr + j) * nstat + s];
        red[t] = v;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if (t < o) red[t] += red[t + o];
            __syncthreads();
        }
        if (t == 0) out[(size_t)r * nstat + s] = red[0];
        __syncthreads();
    }
}

// Scrambled integers / normals of one replica by the direct gray-code form:
// out[d * n + i] for dim dim0 + d and point offset + i.
__global__ void k_sobol_export(const uint32_t* __restrict__ tab, int D, int dim0, int nd,
                               uint32_t offset, long long n, float u_cap, int as_normal,
                               void* out) {
    const long long total = (long long)nd * n;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int d = (int)(idx / n);
        const long long i = idx - (long long)d * n;
        const int dim = dim0 + d;
        const uint32_t pt = offset + (uint32_t)i;
        uint32_t g = pt ^ (pt >> 1);
        uint32_t x = __ldg(tab + 32 * D + dim);
        while (g) {
            const int k = __ffs(g) - 1;
            x ^= __ldg(tab + k * D + dim);
            g &= g - 1;
        }
        if (as_normal) static_cast<float*>(out)[idx] = sobol_normal(x, u_cap);
        else static_cast<uint32_t*>(out)[idx] = x;
    }
}

void launch_prescramble(const uint32_t* dv, uint32_t salt0, int R, int D, uint32_t* out,
                        cudaStream_t s) {
    k_prescramble<<<(unsigned)((D + 31) / 32) * (unsigned)R, 1024, 0, s>>>(dv, salt0, D, out);
}

void launch_prescramble_plain(const uint32_t* dv, uint32_t salt0, int R, int D, uint32_t* out,
                              cudaStream_t s) {
    const long long total = (long long)R * 33 * D;
    int blocks = (int)((total + 255) / 256);
    if (blocks > 148 * 16) blocks = 148 * 16;
    k_prescramble_plain<<<blocks, 256, 0, s>>>(dv, salt0, R, D, out);
}

void launch_finalize(const double* partials, int R, int ipr, int nstat, double* out,
                     cudaStream_t s) {
    k_finalize<<<R, 256, 0, s>>>(partials, ipr, nstat, out);
}

void launch_sobol_export(const uint32_t* tab, int D, int dim0, int nd, uint32_t offset,
                         long long n, float u_cap, int as_normal, void* out, cudaStream_t s) {
    const long long total = (long long)nd * n;
    int blocks = (int)((total + 255) / 256);
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (blocks < 1) blocks = 1;
    k_sobol_export<<<blocks, 256, 0, s>>>(tab, D, dim0, nd, offset, n, u_cap, as_normal, out);
}

// Failure-path probe of the bounded mbarrier wait that the assisted passes (and, with the same
// limit logic, the tensor-core PCA pass) use: one warp waits on a barrier that nothing arrives on,
// gives up after `polls` polls and records MCQ_ERR_TIMEOUT in the status word, which the host's
// check turns into the API error.  No fault, no hang: the wait always returns.
__global__ void k_wait_probe(int* err, uint32_t polls) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(asst_addr(&bar)), "r"(1));
    __syncthreads();
    const bool ok = asst_wait(&bar, 0u, polls);
    if (!__all_sync(0xffffffffu, ok) && threadIdx.x == 0) atomicExch(err, MCQ_ERR_TIMEOUT_CODE);
}

void launch_wait_probe(int* err, uint32_t polls, cudaStream_t s) {
    k_wait_probe<<<1, 32, 0, s>>>(err, polls);
}

// Time rows of the grid local-vol model for steps 0 .. n - 1 of a pass (lv_time_row).
__global__ void k_lv_rows(const __grid_constant__ KParams p, float2* rows, int n) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        rows[k] = lv_time_row(p, k);
}

void launch_lv_rows(const KParams& p, float2* rows, int n, cudaStream_t s) {
    k_lv_rows<<<(n + 255) / 256, 256, 0, s>>>(p, rows, n);
}

}  // namespace mcq
