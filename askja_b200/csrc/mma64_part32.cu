// Warp-MMA kernels (FP64 and split TF32), FP32 storage, any other NC (a translation unit of its own: build time).
#include "mma64_launch.cuh"

namespace askja {
namespace m64 {
ASKJA_M64_ENTRIES(part32, false, float2)
}  // namespace m64
}  // namespace askja
