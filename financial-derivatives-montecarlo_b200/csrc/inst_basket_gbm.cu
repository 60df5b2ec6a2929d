// Single-level Sobol passes of GBM baskets of 1 to 16 assets, one kernel per width (BasketTileC).
#include "inst_common.cuh"
namespace mcq {
// Registers: three CTAs per SM (80) up to eight assets, two (128) beyond.
template <int N>
static const void* basket_width(int n) {
    if (n == N) return (const void*)&k_pass<GEN_SOBOL, NOISE_RAW, BasketTileC<MOD_BASKET, N>, (N <= 8 ? 3 : 2)>;
    if constexpr (N < kMaxBasket) return basket_width<N + 1>(n);
    else return nullptr;
}
const void* lookup_basket_gbm(int n) { return basket_width<1>(n); }
}  // namespace mcq
