// Plane-resident passes, plain FP64 (complex128) instantiation.
#include "qx_plane_impl.cuh"
namespace qx {
template struct Plane<double>;
}  // namespace qx
