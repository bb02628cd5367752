// Warp-MMA kernels (FP64), FP64 storage, NC a multiple of 8 (a translation unit of its own: build time).
#include "mma64_launch.cuh"

namespace askja {
namespace m64 {
ASKJA_M64_ENTRIES(full64, true, double2)
}  // namespace m64
}  // namespace askja
