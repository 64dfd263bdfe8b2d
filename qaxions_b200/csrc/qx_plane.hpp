// qx_plane.hpp -- launchers of the plane-resident passes (qx_plane.cuh).  All
// launches go to the caller's stream; nothing allocates.
#pragma once

#include <cuda_runtime.h>

#include "qx_ops.hpp"

namespace qx {

template <typename R> struct Plane {
    using XP = typename Ops<R>::XP;
    using SP = typename Ops<R>::SP;
    // whether an N x N plane of psi fits one SM's shared memory (3D boxes of
    // this size run their x and y transforms in one kernel)
    static bool xy(int N);
    // whether the last-axis pass of this array has a direct-load column kernel
    static bool col(int N, int dim);

    // planes = XP::rows / N.  psi^_xy -> psi (y inverse, x inverse), with r2c
    // also the density's x and y forward transforms into vh
    static void inv(int N, const XP& a, bool r2c, cudaStream_t st);
    // density of psi -> vh, transformed along x and y
    static void r2c(int N, const XP& a, cudaStream_t st);
    // psi (kicked by Vin first if kick) -> psi^_xy
    static void fwd(int N, const XP& a, bool kick, cudaStream_t st);
    // vh (transformed along x and y) -> V, with the flags of Ops::x_c2r; with
    // C2R_FWD psi goes on to psi^_xy
    static void c2r(int N, const XP& a, int flags, cudaStream_t st);
    // y transform (sign -1 forward, +1 inverse) of [planes][N][X], where the grid has one
    static bool ycol(int N, int X, int sign);
    static void y_pass(int N, int planes, const SP& a, int sign, cudaStream_t st);
    // last-axis drift or Poisson pass (OP_DRIFT on psi, OP_POISSON on vh, column 0 included)
    static void col_pass(int N, const SP& a, int op, cudaStream_t st);
};

}  // namespace qx
