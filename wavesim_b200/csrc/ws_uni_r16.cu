#include "ws_uni_kernels.cuh"

namespace ws {
namespace uni {
template Kernels kernels_up_to<16>();
}  // namespace uni
}  // namespace ws
