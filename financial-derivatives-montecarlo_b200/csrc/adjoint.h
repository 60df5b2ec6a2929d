// adjoint.h — the pathwise adjoint pass (k_adjoint.cu).
#pragma once
#include <cstddef>

namespace mcq {

const void* lookup_adjoint(int model, int payoff);
struct AdjointShape {
    int warps;              // per CTA
    int node_copies_log2;   // KParams::node_copies_log2
    size_t smem;
};
AdjointShape adjoint_shape(int model, int n_steps, int n_nodes);
// device scratch of one warp's 32 paths (KParams::path_scratch)
size_t adjoint_path_bytes(int model, int n_steps);

}  // namespace mcq
