// support.h — host-side launchers for the support kernels in k_support.cu.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace mcq {

// the passes' direction table: [R][kDirRows][D] words (kparams.h)
void launch_prescramble(const uint32_t* dv, uint32_t salt0, int R, int D, uint32_t* out,
                        cudaStream_t s);
// the plain scrambled words and shift, [R][kPlainRows][D]
void launch_prescramble_plain(const uint32_t* dv, uint32_t salt0, int R, int D, uint32_t* out,
                              cudaStream_t s);
void launch_finalize(const double* partials, int R, int ipr, int nstat, double* out,
                     cudaStream_t s);
// one warp waits `polls` times on an mbarrier nothing arrives on, then records MCQ_ERR_TIMEOUT
void launch_wait_probe(int* err, uint32_t polls, cudaStream_t s);
struct KParams;
// the grid local-vol model's time rows of steps 0 .. n - 1 (lv_time_row) into rows[n], and surfaces of at most
// kLvArgNodes nodes into grid[nodes] (larger ones are copied by the caller)
constexpr int kLvArgNodes = 4096;
void launch_lv_rows(const KParams& p, const float* host_grid, float* grid, int nodes, float2* rows, int n,
                    cudaStream_t s);
// a launch that overlaps its set-up with the end of the stream's previous kernel
cudaError_t launch_dependent(const void* fn, unsigned blocks, unsigned threads, void** args, size_t smem,
                             cudaStream_t s, unsigned cluster = 1);
void launch_sobol_export(const uint32_t* tab, int D, int dim0, int nd, uint32_t offset,
                         long long n, float u_cap, int as_normal, void* out, cudaStream_t s);

}  // namespace mcq
