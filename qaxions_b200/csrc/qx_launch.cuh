// qx_launch.cuh -- launch helpers shared by the pass launchers.
#pragma once

#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

#include "qx_kernels.cuh"
#include "qx_ops.hpp"

namespace qx {

#define QX_LAUNCH_CHECK()                                                                 \
    do {                                                                                  \
        cudaError_t e_ = cudaGetLastError();                                              \
        if (e_ != cudaSuccess) throw std::runtime_error(std::string("kernel launch: ") + cudaGetErrorString(e_)); \
    } while (0)

// Report a refused call whose status was returned to us.  The runtime also keeps it
// as its last error, which the next launch check of this thread would take for its
// own: clear it.
[[noreturn]] static inline void throw_refused(const char* what, cudaError_t e) {
    cudaGetLastError();
    throw std::runtime_error(what + std::string(cudaGetErrorString(e)));
}

template <typename K>
static void set_smem(K kernel, size_t bytes) {
    if (bytes > 40 * 1024) {  // (48 KB without the attribute, less the kernel's static arrays)
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) throw_refused("smem attribute: ", e);
    }
}

// Launch with programmatic stream serialization: the kernel may start (and
// stage its tables) while the kernel before it in the stream drains; it waits
// for it (pdl_wait) before it touches the state.  Launched one by one, the passes
// of a step then follow one another as closely as in a graph: 256^3 FP32 482 us
// per step without, 460 with; 128^3 FP64 114 -> 108; 2D 256^2 FP64 27 -> 21.
template <typename... KA, typename... A>
static void launch_dep(void (*kern)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<KA>(args)...);
    if (e != cudaSuccess) throw_refused("kernel launch: ", e);
}

template <typename R> static XArgs<R> to_x(const typename Ops<R>::XP& a) {
    XArgs<R> x;
    x.in = a.in; x.out = a.out; x.vh = a.vh; x.Vin = a.Vin; x.Vout = a.Vout;
    x.twN = a.twN; x.twM = a.twM; x.twN_lo = a.twN_lo; x.twM_lo = a.twM_lo; x.twNn = a.twNn;
    x.rows = a.rows; x.dt = a.dt; x.pref = a.pref;
    x.rho_mean = a.rho_mean; x.scale = a.scale;
    return x;
}
template <typename R> static SArgs<R> to_s(const typename Ops<R>::SP& a) {
    SArgs<R> s;
    s.a = a.a; s.tw = a.tw; s.tw_lo = a.tw_lo; s.X = a.X; s.dim = a.dim; s.N = a.N; s.phase_fac = a.phase_fac;
    s.scale = a.scale; s.pois_c = a.pois_c; s.pois_g0 = a.pois_g0;
    return s;
}

}  // namespace qx
