// Plane-resident passes, fused FP32 (complex64) instantiation.
#include "qx_plane_impl.cuh"
namespace qx {
template struct Plane<float>;
}  // namespace qx
