// Warp-MMA kernels (FP64), FP64 storage, any other NC (a translation unit of its own: build time).
#include "mma64_launch.cuh"

namespace askja {
namespace m64 {
ASKJA_M64_ENTRIES(part64, false, double2)
}  // namespace m64
}  // namespace askja
