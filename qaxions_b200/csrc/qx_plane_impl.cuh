// qx_plane_impl.cuh -- definitions of Plane<R> (included by qx_plane_f32.cu and
// qx_plane_f64.cu).
#pragma once

#include <stdexcept>
#include <string>

#include "qx_launch.cuh"
#include "qx_plane.cuh"
#include "qx_plane.hpp"

namespace qx {

// grid sizes with plane-resident passes
#define QX_FOR_PLANE_N(N, ...)                                                    \
    switch (N) {                                                                  \
        case 32: { constexpr int NN = 32; __VA_ARGS__; break; }                   \
        case 64: { constexpr int NN = 64; __VA_ARGS__; break; }                   \
        case 96: { constexpr int NN = 96; __VA_ARGS__; break; }                   \
        case 128: {                                                               \
            constexpr int NN = sizeof(R) == 4 ? 128 : 96;                         \
            if (NN == 128) { __VA_ARGS__; break; }                                \
        }                                                                         \
        [[fallthrough]];                                                          \
        default: throw std::logic_error("no plane-resident passes for N=" + std::to_string(N)); \
    }

template <typename R> bool Plane<R>::xy(int N) { return plane_fits(N, sizeof(R)); }

template <int NN, typename R, typename K>
static void launch_plane(K kern, const XArgs<R>& x, cudaStream_t st) {
    using G = PlaneGeo<NN, R>;
    set_smem(kern, G::SMEM);
    launch_dep(kern, dim3((unsigned)(x.rows / NN)), dim3(G::TB), G::SMEM, st, x);
}

template <typename R> void Plane<R>::inv(int N, const XP& a, bool r2c, cudaStream_t st) {
    const XArgs<R> x = to_x<R>(a);
    QX_FOR_PLANE_N(N, {
        if (r2c) launch_plane<NN, R>(k_plane_inv<NN, R, PI_R2C>, x, st);
        else launch_plane<NN, R>(k_plane_inv<NN, R, PI_PLAIN>, x, st);
    });
}

template <typename R> void Plane<R>::r2c(int N, const XP& a, cudaStream_t st) {
    const XArgs<R> x = to_x<R>(a);
    QX_FOR_PLANE_N(N, { launch_plane<NN, R>(k_plane_r2c<NN, R>, x, st); });
}

template <typename R> void Plane<R>::fwd(int N, const XP& a, bool kick, cudaStream_t st) {
    const XArgs<R> x = to_x<R>(a);
    QX_FOR_PLANE_N(N, {
        if (kick) launch_plane<NN, R>(k_plane_fwd<NN, R, true>, x, st);
        else launch_plane<NN, R>(k_plane_fwd<NN, R, false>, x, st);
    });
}

template <typename R> void Plane<R>::c2r(int N, const XP& a, int flags, cudaStream_t st) {
    const XArgs<R> x = to_x<R>(a);
    QX_FOR_PLANE_N(N, {
        switch (flags) {
            case C2R_WRITE_V: launch_plane<NN, R>(k_plane_c2r<NN, R, XC_WRITE_V>, x, st); break;
            case C2R_KICK | C2R_FWD: launch_plane<NN, R>(k_plane_c2r<NN, R, XC_KICK | XC_FWD>, x, st); break;
            case C2R_WRITE_V | C2R_KICK | C2R_WRITE_PSI:
                launch_plane<NN, R>(k_plane_c2r<NN, R, XC_WRITE_V | XC_KICK | XC_WRITE_PSI>, x, st);
                break;
            default: throw std::invalid_argument("plane c2r: unsupported flag combination");
        }
    });
}

// ---- direct-load last-axis passes ----

template <typename R> bool Plane<R>::col(int N, int dim) {
    if (dim == 3) return N == 32 || N == 64 || N == 96 || N == 128;
    return N == 64 || N == 96 || N == 128 || N == 256 || N == 512;
}

template <int NN, typename R, int UX, bool D3>
static void launch_col(const typename Ops<R>::SP& a, int op, cudaStream_t st) {
    using G = ColGeo<NN, R, UX>;
    SArgs<R> s = to_s<R>(a);
    const int nb = a.batch > 0 ? a.batch : 1;
    const unsigned grid = (unsigned)(a.X / (UX * G::PW)) * (unsigned)(D3 ? nb * NN : nb);
    if (a.X % (UX * G::PW)) throw std::logic_error("column pass: columns not a multiple of the tile");
    if (op == OP_DRIFT) {
        if (!a.axy || (sizeof(R) == 4 && !a.tw_lo)) throw std::logic_error("drift pass needs its tables");
        auto kern = k_col<NN, R, OP_DRIFT, UX, D3>;
        const size_t smem = G::smem(OP_DRIFT, D3);
        set_smem(kern, smem);
        launch_dep(kern, dim3(grid), dim3(G::NT), smem, st, s, a.axy);
    } else {
        auto kern = k_col<NN, R, OP_POISSON, UX, D3>;
        const size_t smem = G::smem(OP_POISSON, D3);
        set_smem(kern, smem);
        launch_dep(kern, dim3(grid), dim3(G::NT + (D3 ? G::TX : 0)), smem, st, s, (const double2*)nullptr);
    }
}

template <int NN, typename R>
static void launch_ycol(const typename Ops<R>::SP& a, int planes, int sign, cudaStream_t st) {
    using G = ColGeo<NN, R, 8>;
    SArgs<R> s = to_s<R>(a);
    const unsigned grid = (unsigned)(a.X / (8 * G::PW)) * (unsigned)planes;
    const bool df = sizeof(R) == 4 && a.tw_lo != nullptr;
    auto go = [&](auto kern) {
        const size_t smem = G::smem(OP_FWD, false);
        set_smem(kern, smem);
        launch_dep(kern, dim3(grid), dim3(G::NT), smem, st, s, (const double2*)nullptr);
    };
    if (sign < 0) {
        if (df) go(k_col<NN, R, OP_FWD, 8, false, true>);
        else go(k_col<NN, R, OP_FWD, 8, false, false>);
    } else {
        if (df) go(k_col<NN, R, OP_INV, 8, false, true>);
        else go(k_col<NN, R, OP_INV, 8, false, false>);
    }
}

// FP64 128^3, whose planes do not fit: all y passes (step 106 -> 101 us).  256^3 FP32,
// 128 + 64 MB in and out of L2: psi forward 54 -> 50 us and the half spectrum 31 / 29
// -> 28 / 27; psi inverse is faster from the ring (54 against 59), and so are the
// last-axis passes (z drift 99 against 107); 256^3 FP64 gains nowhere (z Poisson 97
// against 143).
template <typename R> bool Plane<R>::ycol(int N, int X, int sign) {
    if (N == 128) return sizeof(R) == 8;
    return N == 256 && sizeof(R) == 4 && (X < N || sign < 0);
}

template <typename R> void Plane<R>::y_pass(int N, int planes, const SP& a, int sign, cudaStream_t st) {
    if constexpr (sizeof(R) == 8) {
        if (N == 128) return launch_ycol<128, R>(a, planes, sign, st);
    } else {
        if (N == 256) return launch_ycol<256, R>(a, planes, sign, st);
    }
    throw std::logic_error("y column pass: not compiled");
}

template <typename R> void Plane<R>::col_pass(int N, const SP& a, int op, cudaStream_t st) {
    if ((op != OP_DRIFT && op != OP_POISSON) || !col(N, a.dim)) throw std::logic_error("column pass: not compiled");
    if (a.dim == 3) {
        switch (N) {
            case 32: launch_col<32, R, 8, true>(a, op, st); break;
            case 64: launch_col<64, R, 8, true>(a, op, st); break;
            case 96: launch_col<96, R, 8, true>(a, op, st); break;
            default: launch_col<128, R, 8, true>(a, op, st); break;
        }
    } else {
        switch (N) {
            case 64: launch_col<64, R, 4, false>(a, op, st); break;
            case 96: launch_col<96, R, 4, false>(a, op, st); break;
            case 128: launch_col<128, R, 2, false>(a, op, st); break;
            case 256: launch_col<256, R, 2, false>(a, op, st); break;
            default: launch_col<512, R, 2, false>(a, op, st); break;
        }
    }
}

}  // namespace qx
