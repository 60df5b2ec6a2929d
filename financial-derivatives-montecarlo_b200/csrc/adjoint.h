// adjoint.h — the pathwise adjoint pass (k_adjoint.cu).
#pragma once
#include <cstddef>

namespace mcq {

const void* lookup_adjoint(int model, int payoff);
int adjoint_warps(int model);   // per CTA
int adjoint_node_copies_log2(int model, int n_steps, int n_nodes);   // KParams::node_copies_log2
size_t adjoint_smem_bytes(int model, int n_steps, int n_nodes);
// device scratch of one warp's 32 paths (KParams::path_scratch)
size_t adjoint_path_bytes(int model, int n_steps);

}  // namespace mcq
