// k_support.cu — small kernels around the fused pass: per-replica direction-word scrambling,
// the deterministic cross-item reduction, and the Sobol stream export used by parity tests.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstring>
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
        const uint32_t v = __ldg(dv + (size_t)min(d, 19999) * 32 + lane);   // (beyond: lanes nobody reads)
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

// out[r][s] = sum over j of partials[(r * ipr + j) * NST + s]; fixed summation order.  A cluster of CTAs per
// replica, each over every n-th run of 256 records, its sums gathered through distributed shared memory:
// with one CTA a pass of a single replica (plain Monte Carlo, 37,888 records) waited 25 us for it.
// `out` may be host memory: the synchronous passes read their sums there after the stream's end, without a copy.
constexpr int kFinThreads = 256;
template <int NST>
__global__ void __launch_bounds__(kFinThreads) k_finalize(const double* __restrict__ partials, int ipr,
                                                          double* __restrict__ out) {
    __shared__ double red[kFinThreads / 32][NST];
    __shared__ double total[NST];
    auto cluster = cooperative_groups::this_cluster();
    const int nc = (int)cluster.num_blocks(), c = (int)cluster.block_rank(), r = blockIdx.x / nc;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    double v[NST];
#pragma unroll
    for (int s = 0; s < NST; s++) v[s] = 0.0;
    grid_dependency_wait();
    const double* rec = partials + (size_t)r * ipr * NST;
#pragma unroll 4
    for (int j = c * kFinThreads + t; j < ipr; j += nc * kFinThreads) {
#pragma unroll
        for (int s = 0; s < NST; s++) v[s] += rec[(size_t)j * NST + s];
    }
#pragma unroll
    for (int s = 0; s < NST; s++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[s] += __shfl_xor_sync(0xffffffffu, v[s], o);
        if (lane == 0) red[warp][s] = v[s];
    }
    __syncthreads();
    if (t < NST) {
        double x = 0.0;
        for (int w = 0; w < kFinThreads / 32; w++) x += red[w][t];
        total[t] = x;
    }
    if (nc > 1) cluster.sync();
    else __syncthreads();
    if (c == 0 && t < NST) {
        double x = 0.0;
        for (int b = 0; b < nc; b++) x += *cluster.map_shared_rank(&total[t], b);
        out[(size_t)r * NST + t] = x;
    }
    if (nc > 1) cluster.sync();   // the other CTAs' shared memory stays until it has been read
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

// A launch whose CTAs may be placed while the stream's previous kernel drains; the kernel itself waits
// for that kernel's results (grid_dependency_wait).
cudaError_t launch_dependent(const void* fn, unsigned blocks, unsigned threads, void** args, size_t smem,
                             cudaStream_t s, unsigned cluster) {
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
}

void launch_finalize(const double* partials, int R, int ipr, int nstat, double* out,
                     cudaStream_t s) {
    const void* fn = nstat == 1 ? (const void*)&k_finalize<1> : nstat == 2 ? (const void*)&k_finalize<2>
                   : nstat == 4 ? (const void*)&k_finalize<4> : nstat == 7 ? (const void*)&k_finalize<7>
                                                              : (const void*)&k_finalize<4 + kMaxBasket>;
    // up to eight CTAs a replica, four records a thread
    unsigned nc = 1;
    while (nc < 8 && (long long)nc * kFinThreads * 4 < ipr) nc *= 2;
    void* args[] = {&partials, &ipr, &out};
    launch_dependent(fn, (unsigned)R * nc, kFinThreads, args, 0, s, nc);   // errors: cudaGetLastError at the caller
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
    if (!__all_sync(0xffffffffu, ok) && threadIdx.x == 0) *(volatile int*)err = MCQ_ERR_TIMEOUT_CODE;
}

void launch_wait_probe(int* err, uint32_t polls, cudaStream_t s) {
    k_wait_probe<<<1, 32, 0, s>>>(err, polls);
}

// Time rows of the grid local-vol model for steps 0 .. n - 1 of a pass (lv_time_row).  Surfaces of up to
// kLvArgNodes nodes come as a kernel argument and are written to `grid` on the way: no copy from
// pageable host memory, which is staged before the call goes on.
struct LvGrid { float g[kLvArgNodes]; };
template <class G>
__global__ void k_lv_rows(const __grid_constant__ KParams p, const __grid_constant__ G g, float* grid, int nodes,
                          float2* rows, int n) {
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (int k = i0; k < n; k += gridDim.x * blockDim.x) rows[k] = lv_time_row(p, k);
    if constexpr (sizeof(G) > 1)
        for (int i = i0; i < nodes; i += gridDim.x * blockDim.x) grid[i] = g.g[i];
}
struct NoGrid {};

void launch_lv_rows(const KParams& p, const float* host_grid, float* grid, int nodes, float2* rows, int n,
                    cudaStream_t s) {
    const int blocks = std::max(8, (n + 255) / 256);
    if (nodes <= kLvArgNodes) {
        LvGrid g;
        std::memcpy(g.g, host_grid, sizeof(float) * (size_t)nodes);
        k_lv_rows<<<blocks, 256, 0, s>>>(p, g, grid, nodes, rows, n);
    } else {
        k_lv_rows<<<blocks, 256, 0, s>>>(p, NoGrid{}, grid, nodes, rows, n);
    }
}

}  // namespace mcq
