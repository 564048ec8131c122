// Single-grid instantiations of the fused kernel with the z-slab terms (a translation unit of its
// own, compiled in parallel with the host code and the batched ones).
#include "yee_fused.cuh"

namespace fdtd {
namespace fused {

bool single_kernels_z(int ty, int ns, FusedKernel out[4]) {
#define FDTD_CASE(TY, NS)                                  \
    if (ty == TY && ns == NS) {                            \
        out[0] = k_yee_fused<TY, NS, false, 4>;            \
        out[1] = k_yee_fused<TY, NS, false, 5>;            \
        out[2] = k_yee_fused<TY, NS, false, 6>;            \
        out[3] = k_yee_fused<TY, NS, false, 7>;            \
        return true;                                       \
    }
    FDTD_FUSED_TILES(FDTD_CASE)
#undef FDTD_CASE
    return false;
}

}  // namespace fused
}  // namespace fdtd
