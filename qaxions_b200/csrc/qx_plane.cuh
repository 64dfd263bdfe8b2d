// qx_plane.cuh -- plane-resident passes for boxes whose (x, y) planes fit one
// SM's shared memory, and direct-load last-axis passes (sm_100a).
//
// A 3D step of a small box is bound by launches and by its passes' fill and
// drain, not by HBM: the whole state sits in L2 and each of the nine row and
// pencil launches of a step moves it once for a few microseconds of work.
// Here one block owns one z plane: the y and x transforms, the density (or the
// potential, the kick) and the next transforms of the plane run in one launch,
// exchanged through shared memory, so a step is four launches:
//   k_col<OP_DRIFT>     psi^_xy: z forward, drift phase, z inverse
//   k_plane_inv         y inverse, x inverse -> psi; density, x r2c, y -> rho^
//   k_col<OP_POISSON>   rho^: z forward, -1/k^2, z inverse (column 0 included)
//   k_plane_c2r         y inverse, x c2r -> V; kick, x forward, y -> psi^_xy
// and L2 sees 16w bytes per site (w = bytes per real: 4w, 5w, 2w, 5w) instead of 28w.
// Between the launches psi is transformed along x and y (psi^_xy).
// Measured (one B200, us per step, nine launches -> these four): 32^3 FP32 45.7
// -> 18.6, 64^3 FP32 45.7 -> 33.0, 128^3 FP32 91 -> 60, 96^3 FP64 99 -> 73.
//
// Column phases (y): lanes run over adjacent column units (pencil pairs in
// FP32, single pencils in FP64), so global accesses are whole lines, shared
// accesses are free of bank conflicts and a warp's twiddle loads are
// broadcasts.  Row phases (x): a row's threads sit in one warp, as in the row
// passes.  The butterflies, twiddles and their order are those of the row and
// pencil passes: psi agrees with theirs bit for bit in FP32, V to 5e-8 (the compiler
// fuses the Poisson scale with the next addition in another order).
//
// Every kernel stages its tables, then waits for the kernel before it
// (griddepcontrol.wait) before it touches the state: launched with programmatic
// stream serialization, its launch and table loads overlap that kernel's tail.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "qx_kernels.cuh"
#include "qx_ops.hpp"
#include "qx_tma.cuh"

namespace qx {

template <int N, typename R> struct PlaneGeo {
    using C = cx_t<R>;
    static constexpr bool F32 = sizeof(R) == 4;
    static constexpr int PW = F32 ? 2 : 1;  // pencils per column unit (16 bytes)
    using P = typename std::conditional<F32, CPair<C>, C>::type;
    static constexpr int M = N / 2;
    static constexpr int E0 = qx_lcm_radices(N);
    static constexpr int EC = (F32 && N == 128) ? 16 : E0;  // values per thread, psi columns
    static constexpr int TC = N / EC, UC = N / PW;           // threads per unit, units
    static constexpr int TH = N / E0, UH = M / PW;           // the same of the half spectrum
    // FP64 96^2: 384 threads with two units each (an E = 24 row needs ~96 registers of values)
    static constexpr int TB = (!F32 && N == 96) ? 384 : UC * TC;
    static constexpr int UPP = TB / TC;  // units per column iteration
    static constexpr int NTH = UH * TH;  // threads of a half-spectrum column phase
    static constexpr int ER = qx_row_efull(N), EH = ER / 2, TR = N / ER;
    static constexpr int RPP = TB / TR;  // rows per row iteration
    // row element x sits at xpad(x): a padding unit of 16 bytes per 128 keeps the
    // 16-byte column accesses aligned and spreads the strided row exchanges; the
    // row pitch offsets the rows that share an access phase
    __host__ __device__ static constexpr int xpad(int x) { return F32 ? x + 2 * (x >> 4) : x + (x >> 3); }
    static constexpr int pitch() {
        if (F32) return N == 32 ? 40 : N == 64 ? 72 : N == 96 ? 120 : 152;  // 8 mod 16
        return N == 32 ? 42 : N == 64 ? 76 : 108;                           // 2 / 4 mod 8
    }
    static constexpr int PITCH = pitch();
    static constexpr int TABLES = N + (F32 ? N : 0) + 2 * M;  // complex elements
    static constexpr size_t SMEM = (size_t)(TABLES + N * PITCH) * sizeof(C);
    static_assert(row_paired<N>(), "row phases chain N- and N/2-point transforms in registers");
    static_assert(UC % UPP == 0 && TB % 32 == 0 && NTH <= TB && NTH % 32 == 0 && (N * TR) % 32 == 0, "plane geometry");
    static_assert(PITCH >= N + (F32 ? 2 * (N / 16) : N / 8), "row pitch");
};

__host__ __device__ constexpr bool plane_fits(int N, int real_bytes) {
    return N == 32 || N == 64 || N == 96 || (N == 128 && real_bytes == 4);
}

// column unit of the plane: element p of its pencils; NT threads share it
template <typename P, typename C, int PITCH, int NT, bool ALL> struct PColAcc {
    static constexpr bool kSplit = false;
    C* base;
    __device__ __forceinline__ P& operator()(int p) const { return *reinterpret_cast<P*>(base + p * PITCH); }
    __device__ __forceinline__ void sync() const {
        if constexpr (ALL) __syncthreads();
        else named_barrier(1, NT);
    }
};
// row of the plane (its threads sit in one warp)
template <typename G> struct PRowAcc {
    static constexpr bool kSplit = false;
    using C = typename G::C;
    C* base;
    __device__ __forceinline__ C& operator()(int p) const { return base[G::xpad(p)]; }
    __device__ __forceinline__ void sync() const { __syncwarp(); }
};

// twiddle tables into shared memory; returns the plane behind them
template <int N, typename R>
__device__ __forceinline__ cx_t<R>* plane_setup(const XArgs<R>& a, unsigned char* smem, XTabs<cx_t<R>>& tb) {
    using C = cx_t<R>;
    C* tN = reinterpret_cast<C*>(smem);
    C* tNl = tN + N;
    C* tM = tNl + (sizeof(R) == 4 ? N : 0);
    C* tNn = tM + N / 2;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        tN[i] = a.twN[i];
        if constexpr (sizeof(R) == 4) tNl[i] = a.twN_lo[i];
    }
    for (int i = threadIdx.x; i < N / 2; i += blockDim.x) {
        tM[i] = a.twM[i];
        tNn[i] = a.twNn[i];
    }
    tb = XTabs<C>{tN, sizeof(R) == 4 ? tNl : tN, tM, tNn};
    return tNn + N / 2;
}

// one z plane's columns, inverse along y: global -> plane (psi^_xy or vh^_xy).
// The loads of a thread are all in flight at once (no staging pass).
// KEEP: the inverse also replaces its source in global memory.
template <int N, typename R, bool HALF, bool KEEP = false>
__device__ __forceinline__ void plane_y_inv(typename std::conditional<KEEP, cx_t<R>*, const cx_t<R>*>::type src,
                                            cx_t<R>* pl, const XTabs<cx_t<R>>& tb) {
    using G = PlaneGeo<N, R>;
    using C = typename G::C;
    using P = typename G::P;
    constexpr int E = HALF ? G::E0 : G::EC;
    constexpr int U = HALF ? G::UH : G::UPP;
    constexpr int NT = HALF ? G::NTH : G::TB;
    constexpr int ITERS = HALF ? 1 : G::UC / G::UPP;
    constexpr int X = HALF ? G::M : N;
    if (threadIdx.x < NT) {
        const int t = threadIdx.x / U;
#pragma unroll 1
        for (int it = 0; it < ITERS; ++it) {
            const int u = threadIdx.x % U + it * U;
            auto* g = src + G::PW * u;
            P v[E];
#pragma unroll
            for (int e = 0; e < E; ++e) v[e] = *reinterpret_cast<const P*>(g + (long)out_pos<N, E>(e, t) * X);
            PColAcc<P, C, G::PITCH, NT, NT == G::TB> acc{pl + G::xpad(G::PW * u)};
            ifft_pencil_rev<N, E>(v, acc, t, tw_src<!HALF>(tb.N, tb.N_lo));
            acc.sync();
#pragma unroll
            for (int e = 0; e < E; ++e) acc(in_pos<N, E, 0>(e, t)) = v[e];
            if constexpr (KEEP) {
#pragma unroll
                for (int e = 0; e < E; ++e) *reinterpret_cast<P*>(g + (long)in_pos<N, E, 0>(e, t) * X) = v[e];
            }
        }
    }
}

// the plane's columns, forward along y: plane -> global
template <int N, typename R, bool HALF>
__device__ __forceinline__ void plane_y_fwd(cx_t<R>* dst, cx_t<R>* pl, const XTabs<cx_t<R>>& tb) {
    using G = PlaneGeo<N, R>;
    using C = typename G::C;
    using P = typename G::P;
    constexpr int E = HALF ? G::E0 : G::EC;
    constexpr int U = HALF ? G::UH : G::UPP;
    constexpr int NT = HALF ? G::NTH : G::TB;
    constexpr int ITERS = HALF ? 1 : G::UC / G::UPP;
    constexpr int X = HALF ? G::M : N;
    if (threadIdx.x < NT) {
        const int t = threadIdx.x / U;
#pragma unroll 1
        for (int it = 0; it < ITERS; ++it) {
            const int u = threadIdx.x % U + it * U;
            PColAcc<P, C, G::PITCH, NT, NT == G::TB> acc{pl + G::xpad(G::PW * u)};
            P v[E];
#pragma unroll
            for (int e = 0; e < E; ++e) v[e] = acc(in_pos<N, E, 0>(e, t));
            fft_pencil<N, E, -1>(v, acc, t, tw_src<!HALF>(tb.N, tb.N_lo));
            C* g = dst + G::PW * u;
#pragma unroll
            for (int e = 0; e < E; ++e) *reinterpret_cast<P*>(g + (long)out_pos<N, E>(e, t) * X) = v[e];
        }
    }
}

// real row (z: pairs 2q, 2q+1 at q = in_pos<M, EH, 0>) -> its packed half
// spectrum in the first N/2 slots of the row (the arithmetic of r2c_post_store)
template <int N, typename R>
__device__ __forceinline__ void plane_row_r2c(cx_t<R> (&z)[PlaneGeo<N, R>::EH], PRowAcc<PlaneGeo<N, R>>& acc, int t,
                                              const XTabs<cx_t<R>>& tb) {
    using G = PlaneGeo<N, R>;
    using C = typename G::C;
    constexpr int M = G::M, EH = G::EH;
    fft_pencil<M, EH, -1>(z, acc, t, tw_src<false>(tb.M, tb.M));
    acc.sync();
#pragma unroll
    for (int e = 0; e < EH; ++e) acc(out_pos<M, EH>(e, t)) = z[e];
    acc.sync();
    C x[EH];
#pragma unroll
    for (int i = 0; i < EH; ++i) {
        const int k = t + i * G::TR;
        const C A = acc(k);
        if (k == 0) {
            x[i] = mk<C>(A.x + A.y, A.x - A.y);
        } else {
            const C B = cconj(acc(M - k));
            const C s = cadd(A, B), d = csub(A, B);
            const C wd = cmul(tb.Nn[k], d);
            x[i] = mk<C>(R(0.5) * (s.x + wd.y), R(0.5) * (s.y - wd.x));
        }
    }
    acc.sync();
#pragma unroll
    for (int i = 0; i < EH; ++i) acc(t + i * G::TR) = x[i];
}

enum PInvMode { PI_PLAIN = 0, PI_R2C = 1 };

// psi^_xy -> psi; with PI_R2C also the density source -> vh (x and y transformed).
// One block per plane.
template <int N, typename R, int MODE>
__global__ void __launch_bounds__((PlaneGeo<N, R>::TB)) k_plane_inv(XArgs<R> a) {
    using G = PlaneGeo<N, R>;
    using C = typename G::C;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    XTabs<C> tb;
    C* pl = plane_setup<N, R>(a, smem_raw, tb);
    pdl_launch();
    pdl_wait();
    __syncthreads();
    const long plane = blockIdx.x;
    plane_y_inv<N, R, false>(a.in + plane * N * N, pl, tb);
    __syncthreads();
    const int t = threadIdx.x % G::TR;
    const R pr = (R)a.pref, rm = (R)a.rho_mean, sc = (R)a.scale;
#pragma unroll 1
    for (int y = threadIdx.x / G::TR; y < N; y += G::RPP) {
        PRowAcc<G> acc{pl + y * G::PITCH};
        C v[G::ER];
#pragma unroll
        for (int e = 0; e < G::ER; ++e) v[e] = acc(out_pos<N, G::ER>(e, t));
        ifft_pencil_rev<N, G::ER, 1>(v, acc, t, tw_src<true>(tb.N, tb.N_lo));
#pragma unroll
        for (int e = 0; e < G::ER; ++e) v[e] = cscale(v[e], sc);
        C* dst = a.out + (plane * N + y) * N;
#pragma unroll
        for (int e = 0; e < G::EH; ++e)
            store_pair(dst, in_pos<G::M, G::EH, 0>(e, t), v[row_pair_idx<N>(e, 0)], v[row_pair_idx<N>(e, 1)]);
        if constexpr (MODE == PI_R2C) {
            auto src_of = [&](const C& u) { return pr * (u.x * u.x + u.y * u.y - rm); };
            C z[G::EH];
#pragma unroll
            for (int e = 0; e < G::EH; ++e)
                z[e] = mk<C>(src_of(v[row_pair_idx<N>(e, 0)]), src_of(v[row_pair_idx<N>(e, 1)]));
            plane_row_r2c<N, R>(z, acc, t, tb);
        }
    }
    if constexpr (MODE == PI_R2C) {
        __syncthreads();
        plane_y_fwd<N, R, true>(a.vh + plane * N * G::M, pl, tb);
    }
}

// density of psi (real space) -> vh
template <int N, typename R>
__global__ void __launch_bounds__((PlaneGeo<N, R>::TB)) k_plane_r2c(XArgs<R> a) {
    using G = PlaneGeo<N, R>;
    using C = typename G::C;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    XTabs<C> tb;
    C* pl = plane_setup<N, R>(a, smem_raw, tb);
    pdl_launch();
    pdl_wait();
    __syncthreads();
    const long plane = blockIdx.x;
    const int t = threadIdx.x % G::TR;
    const R pr = (R)a.pref, rm = (R)a.rho_mean;
#pragma unroll 1
    for (int y = threadIdx.x / G::TR; y < N; y += G::RPP) {
        PRowAcc<G> acc{pl + y * G::PITCH};
        const C* src = a.in + (plane * N + y) * N;
        C z[G::EH];
#pragma unroll
        for (int e = 0; e < G::EH; ++e) {
            C p0, p1;
            load_pair(src, in_pos<G::M, G::EH, 0>(e, t), p0, p1);
            z[e] = mk<C>(pr * (p0.x * p0.x + p0.y * p0.y - rm), pr * (p1.x * p1.x + p1.y * p1.y - rm));
        }
        plane_row_r2c<N, R>(z, acc, t, tb);
    }
    __syncthreads();
    plane_y_fwd<N, R, true>(a.vh + plane * N * G::M, pl, tb);
}

// psi (kicked by Vin first if KICK) -> psi^_xy
template <int N, typename R, bool KICK>
__global__ void __launch_bounds__((PlaneGeo<N, R>::TB)) k_plane_fwd(XArgs<R> a) {
    using G = PlaneGeo<N, R>;
    using C = typename G::C;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    XTabs<C> tb;
    C* pl = plane_setup<N, R>(a, smem_raw, tb);
    pdl_launch();
    pdl_wait();
    __syncthreads();
    const long plane = blockIdx.x;
    const int t = threadIdx.x % G::TR;
#pragma unroll 1
    for (int y = threadIdx.x / G::TR; y < N; y += G::RPP) {
        PRowAcc<G> acc{pl + y * G::PITCH};
        const long row = (plane * N + y) * N;
        C v[G::ER];
#pragma unroll
        for (int e = 0; e < G::EH; ++e) {
            const int q = in_pos<G::M, G::EH, 0>(e, t);
            C p0, p1;
            load_pair(a.in + row, q, p0, p1);
            if constexpr (KICK) {
                const C w = reinterpret_cast<const C*>(a.Vin + row)[q];
                p0 = kick1<R>(p0, w.x, a.dt);
                p1 = kick1<R>(p1, w.y, a.dt);
            }
            v[row_pair_idx<N>(e, 0)] = p0;
            v[row_pair_idx<N>(e, 1)] = p1;
        }
        fft_pencil<N, G::ER, -1, 1>(v, acc, t, tw_src<true>(tb.N, tb.N_lo));
        acc.sync();
#pragma unroll
        for (int e = 0; e < G::ER; ++e) acc(out_pos<N, G::ER>(e, t)) = v[e];
    }
    __syncthreads();
    plane_y_fwd<N, R, false>(a.out + plane * N * N, pl, tb);
}

// vh^_xy -> V, then (FLAGS of XC2RFlags) store V, kick psi, store it in real
// space or transform it along x and y
template <int N, typename R, int FLAGS>
__global__ void __launch_bounds__((PlaneGeo<N, R>::TB)) k_plane_c2r(XArgs<R> a) {
    using G = PlaneGeo<N, R>;
    using C = typename G::C;
    constexpr int M = G::M, EH = G::EH;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    XTabs<C> tb;
    C* pl = plane_setup<N, R>(a, smem_raw, tb);
    pdl_launch();
    pdl_wait();
    __syncthreads();
    const long plane = blockIdx.x;
    // a pass that ends in V leaves vh inverse-transformed along y, as the separate y pass does
    plane_y_inv<N, R, true, (FLAGS & XC_WRITE_V) != 0>(a.vh + plane * N * M, pl, tb);
    __syncthreads();
    const int t = threadIdx.x % G::TR;
#pragma unroll 1
    for (int y = threadIdx.x / G::TR; y < N; y += G::RPP) {
        PRowAcc<G> acc{pl + y * G::PITCH};
        const long row = (plane * N + y) * N;
        C ps[G::ER];  // position 2q + h of psi in ps[row_pair_idx<N>(e, h)]
        if constexpr (FLAGS & XC_KICK) {
#pragma unroll
            for (int e = 0; e < EH; ++e)
                load_pair(a.in + row, in_pos<M, EH, 0>(e, t), ps[row_pair_idx<N>(e, 0)], ps[row_pair_idx<N>(e, 1)]);
        }
        C z[EH];
#pragma unroll
        for (int e = 0; e < EH; ++e) {
            const int k = out_pos<M, EH>(e, t);
            const C X = acc(k);
            if (k == 0) {
                z[e] = mk<C>(X.x + X.y, X.x - X.y);
            } else {
                const C B = cconj(acc(M - k));
                const C s = cadd(X, B), d = csub(X, B);
                const C w = cconj(tb.Nn[k]);
                const C wd = cmul(w, d);
                z[e] = mk<C>(s.x - wd.y, s.y + wd.x);
            }
        }
        ifft_pencil_rev<M, EH>(z, acc, t, tw_src<false>(tb.M, tb.M));
        if constexpr (FLAGS & XC_WRITE_V) {
            C* vrow = reinterpret_cast<C*>(a.Vout + row);
#pragma unroll
            for (int e = 0; e < EH; ++e) vrow[in_pos<M, EH, 0>(e, t)] = z[e];
        }
        if constexpr (FLAGS & XC_KICK) {
#pragma unroll
            for (int e = 0; e < EH; ++e) {
                C& p0 = ps[row_pair_idx<N>(e, 0)];
                C& p1 = ps[row_pair_idx<N>(e, 1)];
                p0 = kick1<R>(p0, z[e].x, a.dt);
                p1 = kick1<R>(p1, z[e].y, a.dt);
            }
            if constexpr (FLAGS & XC_WRITE_PSI) {
#pragma unroll
                for (int e = 0; e < EH; ++e)
                    store_pair(a.out + row, in_pos<M, EH, 0>(e, t), ps[row_pair_idx<N>(e, 0)],
                               ps[row_pair_idx<N>(e, 1)]);
            }
            if constexpr (FLAGS & XC_FWD) {
                fft_pencil<N, G::ER, -1, 1>(ps, acc, t, tw_src<true>(tb.N, tb.N_lo));
                acc.sync();
#pragma unroll
                for (int e = 0; e < G::ER; ++e) acc(out_pos<N, G::ER>(e, t)) = ps[e];
            }
        }
    }
    if constexpr (FLAGS & XC_FWD) {
        __syncthreads();
        plane_y_fwd<N, R, false>(a.out + plane * N * N, pl, tb);
    }
}

// ---------------------------------------------------------------------------
// Last-axis pass without a tile ring: a block loads UX column units x N
// positions straight into registers, transforms, applies the drift phase or
// the Poisson divide, transforms back and stores.  For arrays small enough that
// one tile per block fills the chip a few times at most: the ring of
// k_pencil_tma has nothing to overlap there, and its barrier setup, tensor-map
// fetch and store drain cost more than the loads.  Measured against the ring (us
// per step, the only change): 128^3 FP64 134 -> 118, 2D 256^2 FP64 33 -> 27, 2D
// 512^2 FP32 34 -> 29.
// Block id = tile + tiles * o; 3D: pencils along z, o = box * N + y; 2D: along
// y, o = box.  3D Poisson: the packed kx = 0, N/2 column of row y is combined with its
// mirror mode in row -y, so the tile-0 block of row y, 0 < y < N/2, runs a
// further warp group that carries column 0 of row -y through the whole pass,
// and the tile-0 block of row -y leaves its column 0 alone.
// ---------------------------------------------------------------------------
template <int N, typename R, int UX> struct ColGeo {
    using C = cx_t<R>;
    static constexpr bool F32 = sizeof(R) == 4;
    static constexpr int PW = F32 ? 2 : 1;
    using P = typename std::conditional<F32, CPair<C>, C>::type;
    static constexpr int E = qx_lcm_radices(N), T = N / E;
    static constexpr int NT = UX * T;               // threads of the tile
    static constexpr int TX = (T + 31) / 32 * 32;   // threads of the mirror column
    // exchange rows of UX 16-byte units; narrow tiles pad one row per 8
    __host__ __device__ static constexpr int prow(int p) { return UX == 8 ? p : p + (p >> 3); }
    static_assert(NT % 32 == 0, "whole warps");
    static constexpr size_t smem(int op, bool d3) {
        return (size_t)2 * N * sizeof(C) + (op == OP_DRIFT ? (size_t)N * 16 : (size_t)2 * N * sizeof(C)) +
               (size_t)prow(N) * UX * 16 + (op == OP_POISSON && d3 ? (size_t)(N + N / 8) * 16 : 0);
    }
};

template <typename P> struct ColTileAcc {
    static constexpr bool kSplit = false;
    P* base;
    int pitch, pad, nt;  // row p at base[(p + (pad ? p >> 3 : 0)) * pitch]; nt threads share the buffer
    __device__ __forceinline__ P& operator()(int p) const { return base[(p + (pad ? (p >> 3) : 0)) * pitch]; }
    __device__ __forceinline__ void sync() const { named_barrier(1, nt); }
};

// OP_FWD / OP_INV (D3 = false, o = plane): the y transforms of a 3D array whose
// planes do not fit (FP64 128^3), double-float twiddles when DFT.
template <int N, typename R, int OP, int UX, bool D3, bool DFT = (OP == OP_DRIFT)>
__global__ void __launch_bounds__((ColGeo<N, R, UX>::NT + (OP == OP_POISSON && D3 ? ColGeo<N, R, UX>::TX : 0)))
    k_col(SArgs<R> s, const double2* axy) {
    using G = ColGeo<N, R, UX>;
    using C = typename G::C;
    using P = typename G::P;
    constexpr int E = G::E, PW = G::PW;
    constexpr bool DF = DFT;
    constexpr bool EXTRA = OP == OP_POISSON && D3;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    C* tws = reinterpret_cast<C*>(smem_raw);
    C* tws_lo = tws + N;
    double2* bz = reinterpret_cast<double2*>(tws_lo + N);  // drift: B(nz) / S
    C* mcol = tws_lo + N;                                  // Poisson: column 0 of row y, of row -y
    P* tile = reinterpret_cast<P*>(OP == OP_DRIFT ? reinterpret_cast<unsigned char*>(bz + N)
                                                  : reinterpret_cast<unsigned char*>(mcol + 2 * N));
    const int tid = threadIdx.x;
    const int tiles = s.X / (UX * PW);
    const bool tile0 = blockIdx.x % tiles == 0;
    const int o = blockIdx.x / tiles;  // 3D: box * N + y; 2D: box
    const int yo = D3 ? o % N : 0;
    for (int i = tid; i < N; i += blockDim.x) {
        tws[i] = s.tw[i];
        if constexpr (DF && sizeof(R) == 4) tws_lo[i] = s.tw_lo[i];
    }
    pdl_launch();
    pdl_wait();
    __syncthreads();
    const bool paired = EXTRA && tile0 && yo > 0 && yo < N / 2;  // row -y's column 0 is done here too
    const bool own0 = !(EXTRA && yo > N / 2);                    // this row's column 0 is done here
    const bool extra = EXTRA && tid >= G::NT;
    if (extra && !paired) return;
    const int nt = paired ? G::NT + G::TX : G::NT;
    const int u = extra ? 0 : tid % UX;
    const int t = extra ? (tid - G::NT) % G::T : tid / UX;  // (lanes past T repeat a thread's work)
    const int y = extra ? N - yo : yo;
    const int x0 = (int)((blockIdx.x % tiles) * UX + u) * PW;
    const long pstride = D3 ? (long)N * s.X : (long)s.X;
    C* base = s.a + (D3 ? (long)(o / N) * N * N * s.X + (long)y * s.X : (long)o * N * s.X) + x0;
    P v[E];
    ColTileAcc<P> acc{extra ? tile + (size_t)G::prow(N) * UX : tile + u, extra ? 1 : UX, extra || UX != 8, nt};
    if constexpr (OP == OP_INV) {
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = *reinterpret_cast<const P*>(base + out_pos<N, E>(e, t) * pstride);
        ifft_pencil_rev<N, E>(v, acc, t, tw_src<DF>(tws, tws_lo));
#pragma unroll
        for (int e = 0; e < E; ++e) *reinterpret_cast<P*>(base + in_pos<N, E, 0>(e, t) * pstride) = v[e];
        return;
    }
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = *reinterpret_cast<const P*>(base + in_pos<N, E, 0>(e, t) * pstride);
    if constexpr (OP == OP_FWD) {
        fft_pencil<N, E, -1>(v, acc, t, tw_src<DF>(tws, tws_lo));
#pragma unroll
        for (int e = 0; e < E; ++e) *reinterpret_cast<P*>(base + out_pos<N, E>(e, t) * pstride) = v[e];
        return;
    }
    double2 A[PW];
    if constexpr (OP == OP_DRIFT) {
        const double2* gbz = axy + (D3 ? (long)N * N : (long)N);
        for (int i = tid; i < N; i += G::NT) bz[i] = gbz[i];
#pragma unroll
        for (int h = 0; h < PW; ++h) A[h] = axy[(D3 ? (long)y * N : 0L) + x0 + h];
    }
    fft_pencil<N, E, -1>(v, acc, t, tw_src<DF>(tws, tws_lo));
    if constexpr (OP == OP_DRIFT) {
        // the forward transform's exchanges have synchronised the block since bz was written
#pragma unroll
        for (int h = 0; h < PW; ++h)
#pragma unroll
            for (int e = 0; e < E; ++e) pen_set(v[e], h, cmul_d(pen(v[e], h), dcmul(A[h], bz[out_pos<N, E>(e, t)])));
    } else {
        const bool col0 = tile0 && u == 0 && own0;  // pencil 0 is column 0, finished by this thread
        if (tile0 && own0) {
            if (col0) {
#pragma unroll
                for (int e = 0; e < E; ++e) mcol[(extra ? N : 0) + out_pos<N, E>(e, t)] = pen(v[e], 0);
            }
            acc.sync();
        }
        // the mirror row's column 0: the other of the pair, or the row's own (y = 0, N/2; 2D)
        const C* mir = mcol + (paired && !extra ? N : 0);
        const long ny = D3 ? signed_mode(y, N) : 0;
        if (col0) {
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int p = out_pos<N, E>(e, t);
                const long nz = signed_mode(p, N);
                const long mA = ny * ny + nz * nz, mB = mA + (long)(N / 2) * (N / 2);
                const R gA = pois_mult<R>(mA, s), gB = pois_mult<R>(mB, s);
                const C cm = cconj(mir[(N - p) % N]);
                pen_set(v[e], 0, cadd(cscale(pen(v[e], 0), R(0.5) * (gA + gB)), cscale(cm, R(0.5) * (gA - gB))));
            }
        }
        const bool has_col0 = tile0 && u == 0;
#pragma unroll
        for (int h = 0; h < PW; ++h) {
            if (h == 0 && has_col0) continue;
            const long nx = x0 + h;
            const long mxy = nx * nx + ny * ny;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int nz = signed_mode(out_pos<N, E>(e, t), N);
                pen_set(v[e], h, cscale(pen(v[e], h), pois_mult<R>(mxy + (long)nz * nz, s)));
            }
        }
    }
    ifft_pencil_rev<N, E>(v, acc, t, tw_src<DF>(tws, tws_lo));
    const bool skip0 = tile0 && u == 0 && !own0;  // column 0 belongs to the mirror row's block
    if (EXTRA && (extra || skip0)) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
            C* g = base + in_pos<N, E, 0>(e, t) * pstride;
            if (extra) g[0] = pen(v[e], 0);
            else if (PW == 2) g[1] = pen(v[e], PW - 1);
        }
        return;
    }
#pragma unroll
    for (int e = 0; e < E; ++e) *reinterpret_cast<P*>(base + in_pos<N, E, 0>(e, t) * pstride) = v[e];
}

}  // namespace qx
