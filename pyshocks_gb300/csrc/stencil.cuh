// Shared device templates of the forward and adjoint kernels: shared-memory
// layout, flux phases of one stage, window loader (TMA 1D bulk copies with
// bounded mbarrier waits), CFL time step, fused SSPRK33 tile and the device
// view of a batched plan. See forward.cu for the reference lines followed.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include <type_traits>

#include "device.cuh"
#include "fixed_flux.cuh"
#include "learned.cuh"

namespace shk {

constexpr int kThreads = 256;

constexpr int kDefaultTile = 1024;
// shortest tile of a plan with the learned reconstruction: its warp scratch
// (8 warps x 128 floats forward, x 192 in the reverse step) lives in window
// arrays that the learned phase leaves free (the face-flux array D, at least
// kLearnedScratch floats, in the mixed step; 2W floats in the float step, 3W
// in the reverse step)
constexpr int kLearnedMinTile = 512;
// floats of the forward learned phase's scratch (8 warps, 16-byte alignment slack)
constexpr int kLearnedScratch = (kThreads / 32) * kWarpScratch + 4;
// length of the face-flux array D of the mixed step's layout (the learned
// phase's scratch before it takes the fluxes)
__host__ __device__ constexpr int mixed_d_len(int W) { return W > kLearnedScratch ? W : kLearnedScratch; }

// The FLUX code of kernels whose Rusanov flux runs on fixed_flux.cuh: double
// states, Burgers, WENO-JS5, nu = 1 (fixed_flux_scheme). nu enters that flux as
// 24 a with an integer a; other nu and the other equations keep the FP64
// formula. So do smoothness parameters outside [kFxEpsMin, kFxEpsMax]: the smoothness
// sums are pairs of floats of at least 4 eps, and their lower halves (2^-48 of
// them) must stay above float's smallest number, 2^-149. Against 113-bit
// arithmetic no accepted face is off by more than 4 units of 2^-53 of the largest
// value squared for eps >= 1e-30; at eps = 1e-36 it was 1e4 units, at 1e-40 3e7 (the
// FP64 formula: 4 to 6).
constexpr int kFluxRusanovFx = 100;
constexpr double kFxEpsMin = 1.0e-24, kFxEpsMax = 1.0e24;
// 4-warp CTAs: a stage's warps wait for each other at two barriers, so many small
// CTAs keep the SM busy where few large ones stall (256 threads, 3 CTAs per SM:
// issue 43 %). Us per step at 25.9 M cells by CTAs per SM (tile): 6 (1186) 1247,
// 7 (946) 1229, 8 (946) 1208; 64 registers hold it to 8.
constexpr int kFxThreads = 128;
template <int FLUX>
__host__ __device__ constexpr int flux_threads() { return FLUX == kFluxRusanovFx ? kFxThreads : kThreads; }
inline bool fixed_flux_scheme(const shk_scheme* s, int flux = SHK_FLUX_RUSANOV) {
    return s->flux == flux && s->rec == SHK_REC_WENOJS53 && s->equation == SHK_EQ_BURGERS && s->nu == 1.0 &&
           s->eps >= kFxEpsMin && s->eps <= kFxEpsMax;
}

// halo of a window: 9 cells are needed for three fused stages, rounded up so
// that the window start stays 16-byte aligned for cp.async.bulk
template <class T> __host__ __device__ constexpr int step_halo() { return sizeof(T) == 8 ? 10 : 12; }
template <class T> __host__ __device__ constexpr int op_halo() { return 4; }

__host__ __device__ inline int64_t imin64(int64_t a, int64_t b) { return a < b ? a : b; }

__host__ __device__ inline int64_t imod(int64_t a, int64_t n) {
    int64_t r = a % n;
    return r < 0 ? r + n : r;
}

// the scratch of the learned phase: the nfloats floats of shared memory from
// `region` that the layout leaves free in that phase, from a 16-byte aligned
// start
template <class PR>
__device__ __forceinline__ Win<float> learned_scratch(PR region, int nfloats) {
    float* r = reinterpret_cast<float*>(win_raw(region));
    const uintptr_t a = reinterpret_cast<uintptr_t>(r);
    float* s = reinterpret_cast<float*>((a + 15) & ~uintptr_t(15));
    return make_win(s, nfloats - static_cast<int>(s - r));
}

// ---------------------------------------------------------------------------
// shared-memory layout of one work item (window of W cells)
// ---------------------------------------------------------------------------
constexpr int kFxCounters = 4;  // one per stage, padded

template <class T>
struct Smem {
    Win<T> U;   // u at the start of the step (window)
    Win<T> S;   // stage state k1 / k2
    Win<T> H;   // half differences
    Win<T> D;   // half second differences; reused for face fluxes F
    Win<T> Q;   // 13/12 (2D)^2; reused for ES-WENO omega_0
    Win<T> UL;  // ul (value at the left face of the cell)
    Win<T> UR;  // ur (value at the right face of the cell)
    Win<T> I;   // float states: stage increments (see step_tile); null for double
    Win<float> scr;  // the learned phase's warp scratch (free in that phase)
    Win<int> fx;     // kFluxRusanovFx: counters of the listed faces, then the lists' storage
    int W;      // window length (cells) of every array

    // float states carry one more array (the stage increments)
    static constexpr int kArrays = sizeof(T) == 4 ? 8 : 7;
    __host__ static size_t host_bytes(int W) { return size_t(kArrays) * W * sizeof(T); }
    // the step tile of a double state with the learned reconstruction runs in
    // mixed precision (step_tile_mixed) on the double window and 6 float arrays
    // (kFluxRusanovFx: U, S, D = fluxes, and the list
    // of faces left to the FP64 formula)
    __host__ static size_t step_bytes(int W, int rec, bool fixed = false) {
        if (sizeof(T) == 8 && fixed) return size_t(3) * W * sizeof(T) + size_t(W + kFxCounters) * sizeof(int);
        if (sizeof(T) == 8 && rec == SHK_REC_LEARNED)
            return size_t(W) * sizeof(double) + size_t(5 * W + mixed_d_len(W)) * sizeof(float);
        if (sizeof(T) == 4 && rec == SHK_REC_WENOJS53) return size_t(6) * W * sizeof(T);
        return host_bytes(W);
    }
    // float state with WENO-JS5: the reconstruction works from the window
    // values directly, so H and Q are not needed (6 arrays)
    __device__ void carve_compact(unsigned char* base, int W) {
        T* p = reinterpret_cast<T*>(base);
        U = make_win(p, W); S = make_win(p + W, W); D = make_win(p + 2 * W, W);
        UL = make_win(p + 3 * W, W); UR = make_win(p + 4 * W, W); I = make_win(p + 5 * W, W);
        H = Q = Win<T>();
        scr = Win<float>();
        this->W = W;
    }
    // (one Lax-Friedrichs stage: U, D and the list)
    __host__ static size_t lf_stage_bytes(int W, bool fixed) {
        return fixed ? size_t(2) * W * sizeof(T) + size_t(W + kFxCounters) * sizeof(int) : host_bytes(W);
    }
    __device__ void carve_lf_stage(unsigned char* base, int W) {
        T* p = reinterpret_cast<T*>(base);
        U = make_win(p, W); D = make_win(p + W, W);
        fx = make_win(reinterpret_cast<int*>(p + 2 * W), W + kFxCounters);
        S = H = Q = UL = UR = I = Win<T>();
        scr = Win<float>();
        this->W = W;
        if (threadIdx.x < kFxCounters) fx[threadIdx.x] = 0;  // (the caller's barrier follows)
    }
    __device__ void carve_fixed(unsigned char* base, int W) {
        T* p = reinterpret_cast<T*>(base);
        U = make_win(p, W); S = make_win(p + W, W); D = make_win(p + 2 * W, W);
        fx = make_win(reinterpret_cast<int*>(p + 3 * W), W + kFxCounters);
        H = Q = UL = UR = I = Win<T>();
        scr = Win<float>();
        this->W = W;
        if (threadIdx.x < kFxCounters) fx[threadIdx.x] = 0;  // (the caller's barrier follows)
    }
    // compact layout of that mixed step: U (double window), then as float
    // arrays S (2W: uf, k), I (increments), UL, UR and D (mixed_d_len(W)
    // floats: the learned phase's warp scratch before it takes the face
    // fluxes); no H, and Q aliases D (the learned reconstruction uses neither)
    __device__ void carve_mixed(unsigned char* base, int W) {
        U = make_win(reinterpret_cast<T*>(base), W);
        float* f = reinterpret_cast<float*>(base + size_t(W) * sizeof(double));
        S = win_cast<T>(make_win(f, 2 * W));
        I = win_cast<T>(make_win(f + 2 * W, W));
        UL = win_cast<T>(make_win(f + 3 * W, W));
        UR = win_cast<T>(make_win(f + 4 * W, W));
        D = win_cast<T>(make_win(f + 5 * W, W));
        scr = learned_scratch(make_win(f + 5 * W, mixed_d_len(W)), mixed_d_len(W));
        H = Win<T>();
        Q = D;
        this->W = W;
    }
    __device__ void carve(unsigned char* base, int W) {
        T* p = reinterpret_cast<T*>(base);
        U = make_win(p, W); S = make_win(p + W, W); H = make_win(p + 2 * W, W);
        D = make_win(p + 3 * W, W); Q = make_win(p + 4 * W, W);
        UL = make_win(p + 5 * W, W); UR = make_win(p + 6 * W, W);
        I = kArrays > 7 ? make_win(p + 7 * W, W) : Win<T>();
        const int hd = 2 * W * int(sizeof(T) / sizeof(float));  // H and D as floats
        scr = learned_scratch(make_win(reinterpret_cast<float*>(p + 2 * W), hd), hd);
        this->W = W;
    }
};

template <class T>
struct OpParams {
    T eps, delta, hnu, c;  // WENO eps, ES-WENO delta, nu/2, advection speed
    T hnu_amax;            // LF: nu/2 * global max |f'|
    LearnedParams lp;      // learned reconstruction (float32 state only)
    T fscale;              // face values F are stored as F / fscale (see face_fluxes)
    int lim;               // MUSCL / MUSCLS limiter (SHK_LIM_*)
    T lim_param;           // its theta / van Albada variant
    T atol;                // MUSCL slope-ratio cut
    T dx;                  // cell size (the MUSCLS van Albada variant 2 slope)
    float e4h, e4l;        // 4 eps as the sum of two floats (kFluxRusanovFx)
};

// shared-memory layout of a step tile (see Smem::step_bytes)
template <class T, int REC, int FLUX = SHK_FLUX_RUSANOV>
__device__ __forceinline__ void carve_step(Smem<T>& sm, unsigned char* base, int W) {
    if constexpr (FLUX == kFluxRusanovFx) sm.carve_fixed(base, W);
    else if constexpr (sizeof(T) == 8 && REC == SHK_REC_LEARNED) sm.carve_mixed(base, W);
    else if constexpr (sizeof(T) == 4 && REC == SHK_REC_WENOJS53) sm.carve_compact(base, W);
    else sm.carve(base, W);
}

// ---------------------------------------------------------------------------
// Dirichlet / Neumann boundaries (scalar.py:397-511) on a window. The window
// loader fills every position circularly; for a non-periodic instance the
// three ghost cells of each side (global cells -1-k and n+k, k = 0..2) are
// then overwritten before each operator evaluation. Positions beyond the
// ghosts keep the wrapped values: they reach only ghost outputs, which the
// next overwrite replaces, never an interior output (stencil reach 3).
// ---------------------------------------------------------------------------
struct BcView {
    int left = SHK_BC_PERIODIC, right = SHK_BC_PERIODIC;
    const double* dir = nullptr;  // dir[stage * dir_ss + side * 3 + k]
    int dir_ss = 0;
    const double* neu = nullptr;  // neu[stage * neu_ss + side]
    int neu_ss = 0;
    double dx = 1.0;
    __device__ bool periodic() const { return left == SHK_BC_PERIODIC && right == SHK_BC_PERIODIC; }
};

// S: window array; g0: global cell of window position 0; [wlo, whi): the
// positions holding values of this stage. Call after a barrier; ends with one.
template <class PS>
__device__ void apply_bc(PS S, int64_t g0, int64_t n, int wlo, int whi, const BcView& bc,
                         int stage) {
    using V = elem_t<PS>;
    const int t = threadIdx.x;
    if (t < 6) {
        const int side = t / 3, k = t - 3 * side;
        const int kind = side ? bc.right : bc.left;
        const int64_t w = (side ? n + k : -1 - k) - g0;
        if (kind != SHK_BC_PERIODIC && w >= wlo && w < whi) {
            V val;
            if (kind == SHK_BC_DIRICHLET) {
                val = static_cast<V>(bc.dir[stage * bc.dir_ss + side * 3 + k]);
            } else {
                const int64_t wm = (side ? n - 1 - k : k) - g0;  // mirrored interior cell
                val = S[wm] - static_cast<V>((2 * k + 1) * bc.dx * bc.neu[stage * bc.neu_ss + side]);
            }
            S[w] = val;
        }
    }
    __syncthreads();
}

// Transpose of the ghost fill on a cotangent window z over [wlo, whi): the
// cotangent of a Dirichlet ghost vanishes (its value is data), that of a
// Neumann ghost (mirror - (2k+1) dx g) moves to its mirrored interior cell.
// One thread walks the six ghosts in order (mirrors of the two sides can
// coincide on tiny instances). Call after a barrier; ends with one.
template <class PZ>
__device__ void bc_transpose(PZ z, int64_t g0, int64_t n, int wlo, int whi, const BcView& bc) {
    using V = elem_t<PZ>;
    if (threadIdx.x == 0) {
        for (int t = 0; t < 6; ++t) {
            const int side = t / 3, k = t - 3 * side;
            const int kind = side ? bc.right : bc.left;
            const int64_t w = (side ? n + k : -1 - k) - g0;
            if (kind == SHK_BC_PERIODIC || w < wlo || w >= whi) continue;
            if (kind == SHK_BC_NEUMANN) {
                const int64_t wm = (side ? n - 1 - k : k) - g0;
                if (wm >= wlo && wm < whi) z[wm] += z[w];
            }
            z[w] = V(0);
        }
    }
    __syncthreads();
}

// zero a window array at positions outside the instance [0, n) (the circular
// loader wrapped them in): cotangents of a non-periodic instance
template <class PZ>
__device__ void zero_outside(PZ z, int64_t g0, int64_t n, int wlo, int whi) {
    using V = elem_t<PZ>;
    for (int w = wlo + threadIdx.x; w < whi; w += blockDim.x) {
        const int64_t gi = g0 + w;
        if (gi < 0 || gi >= n) z[w] = V(0);
    }
    __syncthreads();
}

// float copy of the operator parameters (the mixed-precision learned path)
template <class T>
__host__ __device__ inline OpParams<float> float_params(const OpParams<T>& p) {
    OpParams<float> f;
    f.eps = static_cast<float>(p.eps);
    f.delta = static_cast<float>(p.delta);
    f.hnu = static_cast<float>(p.hnu);
    f.c = static_cast<float>(p.c);
    f.hnu_amax = static_cast<float>(p.hnu_amax);
    f.lp = p.lp;
    f.fscale = 1.0f;
    f.lim = p.lim;
    f.lim_param = static_cast<float>(p.lim_param);
    f.atol = static_cast<float>(p.atol);
    f.dx = static_cast<float>(p.dx);
    f.e4h = p.e4h;
    f.e4l = p.e4l;
    return f;
}

// Stage the network of a learned scheme in the block's shared memory (every
// kernel that may run the learned reconstruction, before its first use; the
// whole block; ends with a barrier). BACK: also the backward's fragments.
template <int REC, bool BACK = false>
__device__ __forceinline__ void learned_stage(const LearnedParams& lp) {
    if constexpr (REC == SHK_REC_LEARNED) {
        mlp_stage_forward(lp.mlp, mlp_shared());
        if constexpr (BACK) mlp_stage_back(lp.mlp, mlp_back_shared());
    }
}


// learned reconstruction of cells [clo, chi): one cell per lane, 32 cells per
// warp iteration, both faces of a cell from one network evaluation (the
// network staged by learned_stage). A cell's
// stencil relative to v_c is formed in the state precision straight from the
// window (v_{c+o} - v_c, o = -2..2) and rounded to float; the face values are
// v_c + correction in the state precision.
// scratch: kWarpScratch floats per warp of shared memory (16-byte aligned).
template <class T, class PV, class PO>
__device__ __forceinline__ void learned_phase(PV v, int clo, int chi, PO UL, PO UR,
                                              const LearnedParams& lp, const Win<float>& scratch) {
    const MlpShared& ms = mlp_shared();
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    float* scr = win_span(scratch, warp * kWarpScratch, kWarpScratch);
    const int ncell = chi - clo;
    const int myrow = 16 * (t >> 1) + 8 * (t & 1) + g;  // within the 32-cell block
    for (int q = warp; q * 32 < ncell; q += nw) {
        const int r = q * 32 + myrow;
        const int c = clo + min(r, ncell - 1);
        const T vc = v[c];
        const float ds[5] = {static_cast<float>(v[c - 2] - vc), static_cast<float>(v[c - 1] - vc),
                             0.0f, static_cast<float>(v[c + 1] - vc),
                             static_cast<float>(v[c + 2] - vc)};
        float cr, cl;
        learned_cell32(ms, ds, lp, scr, cr, cl);
        if (r < ncell) {
            UR[c] = vc + static_cast<T>(cr);
            UL[c] = vc + static_cast<T>(cl);
        }
    }
}

// ---------------------------------------------------------------------------
// one evaluation of the numerical fluxes F_j (face j+1/2) for j in [lo-1, hi)
// from the stage input v (valid on [lo-3, hi+3)). Leaves F / p.fscale in sm.D
// (fscale = 1/4 for the FP64 Burgers-Rusanov flux with nu = 1, else 1).
// ---------------------------------------------------------------------------
template <class T, int EQ, int REC, int FLUX, class PV>
__device__ __forceinline__ void face_fluxes(PV v, int lo, int hi, const Smem<T>& sm,
                                            const OpParams<T>& p) {
    const int tid = threadIdx.x, nt = blockDim.x;
    if constexpr (REC == SHK_REC_WENOJS53 && sizeof(T) == 8) {
        // FP64 (pipe-bound): unscaled differences, see weno53_cell_d.
        // phase A: d_c = v_{c+1} - v_c, c in [lo-3, hi+2)
        for (int c = lo - 3 + tid; c < hi + 2; c += nt) sm.H[c] = v[c + 1] - v[c];
        __syncthreads();
        // phase B: E_c = d_c - d_{c-1}, G_c = 13/3 E_c^2 + 4 eps, c in [lo-2, hi+2)
        const T eps4 = T(4) * p.eps;
        for (int c = lo - 2 + tid; c < hi + 2; c += nt) {
            const T e = sm.H[c] - sm.H[c - 1];
            sm.D[c] = e;
            sm.Q[c] = fma(T(13.0 / 3.0) * e, e, eps4);
        }
        __syncthreads();
#pragma unroll 2
        for (int c = lo - 1 + tid; c < hi + 1; c += nt) {
            T ul, ur;
            weno53_cell_d(v[c], sm.H[c - 1], sm.H[c], sm.D[c - 1], sm.D[c], sm.D[c + 1],
                          sm.Q[c - 1], sm.Q[c], sm.Q[c + 1], ul, ur);
            sm.UL[c] = ul;
            sm.UR[c] = ur;
        }
        __syncthreads();
    } else if constexpr (REC == SHK_REC_WENOJS53 && sizeof(T) == 4) {
        // float: each cell's differences straight from its five values (a few
        // more float operations, no barriers and about half the shared-memory
        // traffic of staged difference arrays)
        const float eps4 = 4.0f * p.eps;
#pragma unroll 2
        for (int c = lo - 1 + tid; c < hi + 1; c += nt) {
            const T vm2 = v[c - 2], vm1 = v[c - 1], v0 = v[c], vp1 = v[c + 1], vp2 = v[c + 2];
            T ul, ur;
            weno53_cell_f(v0, vm1 - vm2, v0 - vm1, vp1 - v0, vp2 - vp1, eps4, ul, ur);
            sm.UL[c] = ul;
            sm.UR[c] = ur;
        }
        __syncthreads();
    } else if constexpr (REC == SHK_REC_LEARNED) {
        // warp scratch: sm.scr (free in this phase; with tiles of at least
        // kLearnedMinTile every learned layout gives it kLearnedScratch floats
        // or more)
        learned_phase<T>(v, lo - 1, hi + 1, sm.UL, sm.UR, p.lp, sm.scr);
        __syncthreads();
    } else if constexpr (REC == SHK_REC_CONSTANT) {
        // reconstruction.py:153-163: ul = ur = u
        for (int c = lo - 1 + tid; c < hi + 1; c += nt) {
            sm.UL[c] = v[c];
            sm.UR[c] = v[c];
        }
        __syncthreads();
    } else if constexpr (REC == SHK_REC_MUSCL || REC == SHK_REC_MUSCLS) {
        for (int c = lo - 1 + tid; c < hi + 1; c += nt) {
            T ul, ur;
            if constexpr (REC == SHK_REC_MUSCL)
                muscl_cell<T>(v[c - 1], v[c], v[c + 1], p.lim, p.lim_param, p.atol, ul, ur);
            else
                muscls_cell<T>(v[c - 1], v[c], v[c + 1], p.lim, p.lim_param, p.dx, ul, ur);
            sm.UL[c] = ul;
            sm.UR[c] = ur;
        }
        __syncthreads();
    } else if constexpr (REC == SHK_REC_WENOJS32) {
        for (int c = lo - 1 + tid; c < hi + 1; c += nt) {
            T ul, ur;
            weno32_cell<T>(v[c - 1], v[c], v[c + 1], p.eps, ul, ur);
            sm.UL[c] = ul;
            sm.UR[c] = ur;
        }
        __syncthreads();
    } else {
        for (int c = lo - 1 + tid; c < hi + 1; c += nt) {
            T ul, ur, w0;
            esweno32_cell<T>(v[c - 1], v[c], v[c + 1], p.eps, ul, ur, w0);
            sm.UL[c] = ul;
            sm.UR[c] = ur;
            sm.Q[c] = w0;
        }
        __syncthreads();
    }
    // phase D: F_j, j in [lo-1, hi)
    for (int j = lo - 1 + tid; j < hi; j += nt) {
        T f;
        if constexpr (FLUX == SHK_FLUX_RUSANOV && EQ == SHK_EQ_BURGERS && sizeof(T) == 8) {
            if (p.fscale != T(1)) {
                // nu = 1: 4 F = L^2 + R^2 + 2a (R - L), stored with fscale = 1/4
                const T L = sm.UL[j + 1], R = sm.UR[j];
                const auto ab = abs_bits(v[j]) > abs_bits(v[j + 1]) ? abs_bits(v[j]) : abs_bits(v[j + 1]);
                f = fma(L, L, fma(R, R, twice_abs_bits(ab) * (R - L)));
            } else {
                f = rusanov_face<EQ, T>(sm.UR[j], sm.UL[j + 1], v[j], v[j + 1], p.hnu, p.c);
            }
        } else if constexpr (FLUX == SHK_FLUX_RUSANOV) {
            f = rusanov_face<EQ, T>(sm.UR[j], sm.UL[j + 1], v[j], v[j + 1], p.hnu, p.c);
        } else if constexpr (FLUX == SHK_FLUX_LF) {
            f = lf_face<EQ, T>(sm.UR[j], sm.UL[j + 1], p.hnu_amax, p.c);
        } else if constexpr (FLUX == SHK_FLUX_GODUNOV) {
            f = godunov_face<EQ, T>(sm.UR[j], sm.UL[j + 1], p.c);
        } else if constexpr (FLUX == SHK_FLUX_EO) {
            f = eo_face<EQ, T>(sm.UR[j], sm.UL[j + 1], p.c);
        } else {
            f = esweno_face<EQ, T>(sm.UR[j], sm.UL[j + 1], v[j], v[j + 1], sm.Q[j], sm.Q[j + 1],
                                   p.delta, p.c);
        }
        sm.D[j] = f;
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// window loader: cells g0 .. g0+W-1 of a periodic instance (mod n) into dst.
// Uses cp.async.bulk (TMA 1D, no multicast) into the CTA's own shared memory
// when every piece is 16-byte aligned, plain coalesced loads otherwise.
// Returns false if the bulk copy did not complete within the wait limit.
// ---------------------------------------------------------------------------
// meanwhile() runs on every thread while the copies are in flight.
struct Nothing {
    __device__ void operator()() const {}
};
template <class T, class F = Nothing>
__device__ bool load_window(Win<T> dst, const T* base, int64_t n, int64_t g0, int W,
                            uint64_t* bar, uint32_t& phase, F&& meanwhile = F()) {
    const size_t sz = sizeof(T);
    // a window no longer than its instance wraps at most once: one compare
    // instead of a 64-bit remainder per position
    const bool once = g0 >= -n && g0 + W <= 2 * n;
    auto wrap = [&](int64_t pos) -> int64_t {
        if (once) return pos < 0 ? pos + n : (pos >= n ? pos - n : pos);
        return imod(pos, n);
    };
    // order earlier generic-proxy accesses of dst before the async-proxy writes
    fence_proxy_async();
    // thread 0 decides between bulk copies and plain loads; the barrier that
    // broadcasts the decision also orders the fences before the copies
    bool bulk = false;
    if (threadIdx.x == 0) {
        bulk = (reinterpret_cast<uintptr_t>(base) % 16 == 0) &&
               (reinterpret_cast<uintptr_t>(win_raw(dst)) % 16 == 0);
        int64_t pos = g0;
        const int64_t end = g0 + W;
        int npieces = 0;
        while (pos < end && bulk) {
            const int64_t src = wrap(pos);
            const int64_t len = min(end - pos, n - src);
            if ((src * sz) % 16 || (len * sz) % 16 || ((pos - g0) * sz) % 16) bulk = false;
            pos += len;
            if (++npieces > 8) bulk = false;  // tiny instances: plain loads
        }
    }
    bulk = __syncthreads_or(bulk);
    if (!bulk) {
        for (int w = threadIdx.x; w < W; w += blockDim.x) {
            const int64_t src = wrap(g0 + w);
            if (chk_index(src, n)) dst[w] = base[src];
        }
        meanwhile();
        __syncthreads();
        return true;
    }
    if (threadIdx.x == 0) {
        mbar_expect_tx(bar, static_cast<uint32_t>(W * sz) + test_extra_tx());
        int64_t pos = g0;
        const int64_t end = g0 + W;
        while (pos < end) {
            const int64_t src = wrap(pos);
            const int64_t len = min(end - pos, n - src);
            // (bounds-check build: a piece outside the window or the instance is
            // not copied; the wait for it then expires)
            if (chk_index(src, n) && chk_index(src + len - 1, n) && win_fits(dst, pos - g0, len))
                bulk_g2s(win_raw(dst) + (pos - g0), base + src, static_cast<uint32_t>(len * sz), bar);
            pos += len;
        }
    }
    meanwhile();
    bool ok = mbar_wait_bounded(bar, phase);
    if (!ok) ok = mbar_wait_bounded(bar, phase);  // second bounded wait for copies in flight
    phase ^= 1u;
    return __syncthreads_and(ok) != 0;
}

// ---------------------------------------------------------------------------
// per-instance CFL time step (timestepping.py:139-145 with the Rusanov
// estimate of burgers/schemes.py:121-127 and the driver's theta)
// ---------------------------------------------------------------------------
struct DtState {
    double dt;
    bool active;  // t < tfinal (timestepping.py:133-134)
    bool finite;
};
__host__ __device__ inline DtState compute_dt(double smax, double cfl, double theta, double t,
                                              double tfinal) {
    DtState s;
    s.active = t < tfinal;
    double dt = theta * (cfl / smax);
    if (tfinal != INFINITY) {
        const double dtmin = tfinal - t;
        dt = (dt < dtmin ? dt : dtmin) + 1.0e-15;
    }
    s.dt = dt;
    s.finite = isfinite(dt);
    return s;
}

// ---------------------------------------------------------------------------
// What a replayed step hands to the reverse sweep (pointers to the tile's
// interior cells; null: not wanted): the stage states k1, k2 and, for the
// double WENO-JS5 step, the face values of u, k1 and k2. Their element type is
// the stage precision: float for the learned or float steps, double otherwise.
// ---------------------------------------------------------------------------
template <class S>
struct StageOut {
    Win<S> k1 = nullptr;
    Win<S> k2 = nullptr;
    Win<S> ulu = nullptr;
    Win<S> uru = nullptr;
    Win<S> ul1 = nullptr;
    Win<S> ur1 = nullptr;
    Win<S> ul2 = nullptr;  // face values of k2
    Win<S> ur2 = nullptr;
};
template <class T, int REC>
using stage_t = typename std::conditional<sizeof(T) == 8 && REC != SHK_REC_LEARNED, double, float>::type;

// the tile's interior [HL, HL + te) of a window array into out
template <class PO, class PW>
__device__ __forceinline__ void store_interior(PO out, PW w, int HL, int te) {
    using S = elem_t<PO>;
    if (out)
        for (int i = HL + threadIdx.x; i < HL + te; i += blockDim.x) out[i - HL] = static_cast<S>(w[i]);
}

// ---------------------------------------------------------------------------
// fused SSPRK33 step of one tile: window [s - HL, s + te + HL) -> u_out[s, s + te)
// returns the thread's max |f'(u_new)| bits
// ---------------------------------------------------------------------------
// Mixed precision (double state, learned reconstruction): the operator runs in
// float on the float-rounded stage states and each stage is an increment about
// the step's start state u, accumulated in float and added to u in double
// once per step:
//   k1 = u + i1,  k2 = 3/4 u + 1/4 (k1 + i2) = u + d2,  d2 = (i1 + i2) / 4,
//   u+ = 1/3 u + 2/3 (k2 + i3) = u + 2/3 (d2 + i3),
// with i_s = dt/dx (F_{j-1/2} - F_{j+1/2}) of stage s. Rounding the operator's
// inputs to float perturbs the increments only (the state itself is never
// rounded), and the learned reconstruction works in float/bfloat16 anyway;
// the double pipe then carries three operations per cell and step instead of
// the whole operator. Layout (Smem::carve_mixed, or the full double layout):
// U is the loaded double window, S holds the float window uf and the float
// stage state, I the increments.
// so (optional): the float stage states k1, k2 for a reverse step that then
// skips their recompute; gout may be null when only those are wanted (the
// last stage is skipped).
template <int EQ, int FLUX>
__device__ unsigned long long step_tile_mixed(const Smem<double>& sm, Win<double> gout, int te,
                                              double dtdx, const OpParams<double>& p,
                                              const BcView& bc, int64_t g0, int64_t n,
                                              const StageOut<float>& so = StageOut<float>()) {
    constexpr int HL = step_halo<double>();
    const int tid = threadIdx.x, nt = blockDim.x, W = sm.W;
    const OpParams<float> pf = float_params(p);
    Smem<float> fs;
    fs.U = win_cast<float>(sm.S);
    fs.S = fs.U + W;
    fs.H = win_cast<float>(sm.H);
    fs.D = win_cast<float>(sm.D);
    fs.Q = win_cast<float>(sm.Q);
    fs.UL = win_cast<float>(sm.UL);
    fs.UR = win_cast<float>(sm.UR);
    fs.I = win_cast<float>(sm.I);
    fs.scr = sm.scr;
    fs.W = W;
    const Win<float> inc = fs.I;
    const float dtf = static_cast<float>(dtdx);
    for (int i = tid; i < te + 2 * HL; i += nt) fs.U[i] = static_cast<float>(sm.U[i]);
    __syncthreads();
    if (!bc.periodic()) apply_bc(fs.U, g0, n, 0, te + 2 * HL, bc, 0);
    {
        const int lo = HL - 6, hi = HL + te + 6;
        face_fluxes<float, EQ, SHK_REC_LEARNED, FLUX>(fs.U, lo, hi, fs, pf);
        for (int i = lo + tid; i < hi; i += nt) {
            const float d = dtf * (fs.D[i - 1] - fs.D[i]);
            inc[i] = d;
            fs.S[i] = fs.U[i] + d;
        }
        __syncthreads();
        if (!bc.periodic()) apply_bc(fs.S, g0, n, lo, hi, bc, 1);
        store_interior(so.k1, fs.S, HL, te);
    }
    {
        const int lo = HL - 3, hi = HL + te + 3;
        face_fluxes<float, EQ, SHK_REC_LEARNED, FLUX>(fs.S, lo, hi, fs, pf);
        for (int i = lo + tid; i < hi; i += nt) {
            const float d = 0.25f * (inc[i] + dtf * (fs.D[i - 1] - fs.D[i]));
            inc[i] = d;
            fs.S[i] = fs.U[i] + d;
        }
        __syncthreads();
        if (!bc.periodic()) apply_bc(fs.S, g0, n, lo, hi, bc, 2);
        store_interior(so.k2, fs.S, HL, te);
    }
    unsigned long long mx = 0;
    if (!gout) return mx;
    {
        const int lo = HL, hi = HL + te;
        face_fluxes<float, EQ, SHK_REC_LEARNED, FLUX>(fs.S, lo, hi, fs, pf);
        for (int i = lo + tid; i < hi; i += nt) {
            const float d = (2.0f / 3.0f) * (inc[i] + dtf * (fs.D[i - 1] - fs.D[i]));
            const double un = sm.U[i] + static_cast<double>(d);
            gout[i - HL] = un;
            const unsigned long long b = abs_bits(wave_speed<EQ>(un, p.c));
            mx = b > mx ? b : mx;
        }
    }
    return mx;
}

// Float state, WENO-JS5 + Rusanov: each stage in one pass over the window,
// two adjacent cells per lane. A warp reconstructs the 64 cells r0 .. r0+63
// (r0 even), lane L the pair c0 = r0 + 2L, c0 + 1: its six window values come
// in three aligned 8-byte loads, and the pair shares its differences d,
// second differences E and the terms G = 13/3 E^2 + 4 eps (weno53_cell_fg).
// Each lane forms the fluxes of both its cells' right faces (the left face
// value of the next pair comes from the lane above by shuffle) and takes the
// flux of its first cell's left face from the lane below. The warp updates
// the 62 cells r0+1 .. r0+62. One barrier per stage, the same operations in
// the same order per cell as the one-cell-per-lane stage, so the same results
// bit for bit. The stages ping-pong between S (k1) and UL (k2), since a warp's
// output cells are other warps' stencil inputs.
template <int EQ>
__device__ unsigned int step_tile_f32_weno(const Smem<float>& sm, Win<float> gout, int te, float dtdx,
                                           const OpParams<float>& p, const BcView& bc, int64_t g0,
                                           int64_t n, const StageOut<float>& so) {
    constexpr int HL = step_halo<float>();
    constexpr unsigned kFull = 0xffffffffu;
    const bool np = !bc.periodic();
    if (np) apply_bc(sm.U, g0, n, 0, te + 2 * HL, bc, 0);
    dtdx *= p.fscale;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const float eps4 = 4.0f * p.eps;
    const Win<float> K2 = sm.UL;
    unsigned int mx = 0;
    auto ld2 = [](const Win<float>& a, int i) {  // a[i], a[i+1]; i even
        return *reinterpret_cast<const float2*>(win_span(a, i, 2));
    };
    // stage s reads v on [lo-3, hi+3) and updates [lo, hi); pairs past hi
    // are clamped to the last even start at or below hi (their values only
    // feed unused faces), which keeps every load inside [lo-4, hi+4)
    auto stage = [&](const Win<float>& v, int lo, int hi, int s) {
        const int cmax = hi & ~1;
        for (int r0 = ((lo - 1) & ~1) + 62 * warp; r0 + 1 < hi; r0 += 62 * nw) {
            const int c0 = r0 + 2 * lane;
            const int cc = c0 < cmax ? c0 : cmax;
            const float2 wa = ld2(v, cc - 2), wb = ld2(v, cc), wc = ld2(v, cc + 2);
            const float dA = wa.y - wa.x, dB = wb.x - wa.y, dC = wb.y - wb.x, dD = wc.x - wb.y,
                        dE = wc.y - wc.x;
            const float EB = dB - dA, EC = dC - dB, ED = dD - dC, EE = dE - dD;
            const float GB = weno53_g_f(EB, eps4), GC = weno53_g_f(EC, eps4), GD = weno53_g_f(ED, eps4),
                        GE = weno53_g_f(EE, eps4);
            float ula, ura, ulb, urb;
            weno53_cell_fg(wb.x, dB, dC, EB, EC, ED, GB, GC, GD, ula, ura);
            weno53_cell_fg(wb.y, dC, dD, EC, ED, EE, GC, GD, GE, ulb, urb);
            const float uln = __shfl_down_sync(kFull, ula, 1);  // left face value of cell c0 + 2
            const float fa = rusanov_face<EQ, float>(ura, ulb, wb.x, wb.y, p.hnu, p.c);  // c0 + 1/2
            const float fb = rusanov_face<EQ, float>(urb, uln, wb.y, wc.x, p.hnu, p.c);  // c0 + 3/2
            const float fl = __shfl_up_sync(kFull, fb, 1);                               // c0 - 1/2
            const bool va = lane >= 1 && c0 >= lo && c0 < hi;
            const bool vb = lane <= 30 && c0 + 1 >= lo && c0 + 1 < hi;
            if (!(va || vb)) continue;
            const float2 u = ld2(sm.U, cc);
            const float ra = dtdx * (fl - fa), rb = dtdx * (fa - fb);
            if (s == 3) {
                const float2 inc = ld2(sm.I, cc);
                const float una = u.x + (2.0f / 3.0f) * (inc.x + ra);
                const float unb = u.y + (2.0f / 3.0f) * (inc.y + rb);
                if (va) {
                    gout[c0 - HL] = una;
                    const unsigned int bb = abs_bits(wave_speed<EQ>(una, p.c));
                    mx = bb > mx ? bb : mx;
                }
                if (vb) {
                    gout[c0 + 1 - HL] = unb;
                    const unsigned int bb = abs_bits(wave_speed<EQ>(unb, p.c));
                    mx = bb > mx ? bb : mx;
                }
                continue;
            }
            float da, db;
            if (s == 1) {
                da = ra;
                db = rb;
            } else {
                const float2 inc = ld2(sm.I, cc);
                da = 0.25f * (inc.x + ra);
                db = 0.25f * (inc.y + rb);
            }
            const Win<float>& out = s == 1 ? sm.S : K2;
            if (va && vb) {
                *reinterpret_cast<float2*>(win_span(sm.I, c0, 2)) = make_float2(da, db);
                *reinterpret_cast<float2*>(win_span(out, c0, 2)) = make_float2(u.x + da, u.y + db);
            } else if (va) {
                sm.I[c0] = da;
                out[c0] = u.x + da;
            } else {
                sm.I[c0 + 1] = db;
                out[c0 + 1] = u.y + db;
            }
        }
        __syncthreads();
    };
    stage(sm.U, HL - 6, HL + te + 6, 1);
    if (np) apply_bc(sm.S, g0, n, HL - 6, HL + te + 6, bc, 1);
    store_interior(so.k1, sm.S, HL, te);
    stage(sm.S, HL - 3, HL + te + 3, 2);
    if (np) apply_bc(K2, g0, n, HL - 3, HL + te + 3, bc, 2);
    store_interior(so.k2, K2, HL, te);
    if (!gout) return mx;
    stage(K2, HL, HL + te, 3);
    return mx;
}

// ---------------------------------------------------------------------------
// double state, Burgers + Rusanov (nu = 1) + WENO-JS5: the stages on the fluxes
// of fixed_flux.cuh
// ---------------------------------------------------------------------------
// The faces that fixed_flux.cuh leaves, in FP64: six times the corrections that
// WENO-JS5 adds to the middle cell for its two face values, tR = 6 (ur - v) and
// tL = 6 (ul - v), as the middle sub-stencil's plus weighted third differences (product
// form, P_k = 1 / (4 (eps + beta_k))^2 up to a common factor). From the differences a, b
// on the left and right, E and G = 13/3 E^2 + 4 eps of the cell and of those beside.
// The mirrored input gives the mirrored values bit for bit.
struct WenoTerms {
    double P0, P1, P2, A, B, S;
};
__device__ __forceinline__ WenoTerms weno53_terms(double a, double b, double Em, double E, double Ep, double Gm,
                                                  double G, double Gp) {
    const double h0 = fma(2.0, a, Em), h1 = b + a, h2 = fma(-2.0, b, Ep);
    const double e0 = fma(h0, h0, Gm), e1 = fma(h1, h1, G), e2 = fma(h2, h2, Gp);
    const double p0 = e1 * e2, p1 = e0 * e2, p2 = e0 * e1;
    WenoTerms w;
    w.P0 = p0 * p0;
    w.P1 = p1 * p1;
    w.P2 = p2 * p2;
    w.A = w.P0 * (E - Em);
    w.B = w.P2 * (Ep - E);
    w.S = __dadd_rn(w.A, w.B);  // (not contracted: that would not mirror)
    return w;
}
__device__ __forceinline__ double weno53_right(const WenoTerms& w, double a, double b) {
    return fma(-fma(2.0, w.S, w.B), rcp_nr(fma(6.0, w.P1, fma(3.0, w.P2, w.P0))), fma(2.0, b, a));
}
__device__ __forceinline__ double weno53_left(const WenoTerms& w, double a, double b) {
    return fma(fma(2.0, w.S, w.A), rcp_nr(fma(6.0, w.P1, fma(3.0, w.P0, w.P2))), -fma(2.0, a, b));
}
__device__ __forceinline__ double weno53_g(double E, double eps4) { return fma((13.0 / 3.0) * E, E, eps4); }

// the flux of such a face from its two corrections (LF: with the speed aglob)
template <bool LF, class PV, class FaceOut>
__device__ __forceinline__ void fx_listed_flux(PV v, Win<double> G, int j, double tR, double tL, double aglob,
                                               const FaceOut& out) {
    const double v0 = v[j], v1 = v[j + 1];
    double g;
    bool ok;
    if constexpr (LF) ok = fx::listed_flux_lf(tR, tL, v0, v1, fx::speed_begin(aglob), g);
    else ok = fx::listed_flux(tR, tL, v0, v1, g);
    if (!ok || out.ul) {
        const double R = fma(tR, 1.0 / 6.0, v0), L = fma(tL, 1.0 / 6.0, v1);
        if (!ok) {
            auto ab = abs_bits(v0) > abs_bits(v1) ? abs_bits(v0) : abs_bits(v1);
            if constexpr (LF) ab = ab > abs_bits(aglob) ? ab : abs_bits(aglob);
            g = 72.0 * fma(L, L, fma(R, R, twice_abs_bits(ab) * (R - L)));
        }
        if (out.ul) out(j, R, L);
    }
    G[j] = g;
}

// few: two lanes per face, one for each side (38 FP64 instructions for 16 faces)
template <bool LF, class PV, class FaceOut>
__device__ __noinline__ void fx_listed_faces(PV v, Win<double> G, Win<int> list, int cnt, double eps,
                                             double aglob, FaceOut out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const double eps4 = 4.0 * eps;
    for (int q0 = 16 * warp; q0 < cnt; q0 += 16 * nw) {
        const int q = q0 + (lane >> 1);
        const int j = list[q < cnt ? q : q0];
        const int c = j + (lane & 1), o = (lane & 1) ? -1 : 1;  // cell and direction of this side
        const double x = v[c], vm = v[c - o], vp = v[c + o];
        const double dm2 = vm - v[c - 2 * o], dm1 = x - vm, d0 = vp - x, dp1 = v[c + 2 * o] - vp;
        const double Em = dm1 - dm2, E0 = d0 - dm1, Ep = dp1 - d0;
        const WenoTerms w = weno53_terms(dm1, d0, Em, E0, Ep, weno53_g(Em, eps4), weno53_g(E0, eps4),
                                         weno53_g(Ep, eps4));
        const double t = weno53_right(w, dm1, d0), t1 = __shfl_xor_sync(0xffffffffu, t, 1);
        if (q < cnt && (lane & 1) == 0) fx_listed_flux<LF>(v, G, j, t, t1, aglob, out);
    }
}

// many: both sides of every cell, two cells per lane (74 FP64 instructions for 60
// faces), the neighbours' differences by shuffle; chunks without a listed face are
// skipped. The same operations on the same values give a side's correction, so it does
// not depend on how many others are listed.
// Taken for more than half of a window's faces where it has more than one
// chunk and a half: an FP64 instruction holds a quarter of an SM for 64 clocks, and the
// list spreads the faces of a short window further. Measured (us per step: FP64 formula
// for every face / all listed faces by two one-sided product-form evaluations / this),
// 1024 instances, 6.4 M cells: 0.5 % noise 1948 / 2794 / 1606, random cells 1948 / 3016 /
// 1611, smooth 1948 / 285 / 284; 24 instances of 100 to 1000 cells: noise 57 / 40 / 36,
// random 57 / 78 / 49; 1000 random instances of 128 cells: 71 / 81 / 55, of 64 cells:
// 57 / 47 / 47. (Each warp taking its own chunk at once, before the barrier: noise 5 %
// faster on 300 ragged instances, smooth states 1 % slower.)
__device__ __forceinline__ bool fx_many(int cnt, int faces) { return 2 * cnt > faces && faces > 90; }
template <bool LF, class PV, class FaceOut>
__device__ __noinline__ void fx_listed_tile(PV v, Win<double> G, Win<int> list, int cnt, int jlo, int jhi, int W,
                                            double eps, double aglob, FaceOut out) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int kMark = 0x7ff80001;  // upper word of a listed face's place in G
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const double eps4 = 4.0 * eps;
    for (int q = threadIdx.x; q < cnt; q += blockDim.x) G[list[q]] = __hiloint2double(kMark, 0);
    __syncthreads();
    for (int r0 = (jlo & ~1) - 2 + 60 * warp; r0 + 2 < jhi; r0 += 60 * nw) {
        const int c0 = r0 + 2 * lane;
        const bool inner = lane >= 1 && lane <= 30;
        const bool l0 = inner && c0 >= jlo && c0 < jhi && __double2hiint(G[c0]) == kMark;
        const bool l1 = inner && c0 + 1 >= jlo && c0 + 1 < jhi && __double2hiint(G[c0 + 1]) == kMark;
        if (!__any_sync(kFull, l0 || l1)) continue;
        // (cells outside the window only feed faces that are not stored)
        const int ca = c0 < 0 ? 0 : (c0 < W - 2 ? c0 : W - 2);
        const double vm = v[ca > 0 ? ca - 1 : 0], v0 = v[ca], v1 = v[ca + 1], v2 = v[ca < W - 2 ? ca + 2 : ca + 1];
        const double dm = v0 - vm, d0 = v1 - v0, d1 = v2 - v1;
        const double E0 = d0 - dm, E1 = d1 - d0;
        const double G0 = weno53_g(E0, eps4), G1 = weno53_g(E1, eps4);
        const double Em = __shfl_up_sync(kFull, E1, 1), Gm = __shfl_up_sync(kFull, G1, 1);
        const double Ep = __shfl_down_sync(kFull, E0, 1), Gp = __shfl_down_sync(kFull, G0, 1);
        const WenoTerms a = weno53_terms(dm, d0, Em, E0, E1, Gm, G0, G1);
        const WenoTerms b = weno53_terms(d0, d1, E0, E1, Ep, G0, G1, Gp);
        const double L2 = __shfl_down_sync(kFull, weno53_left(a, dm, d0), 1);
        const double R0 = weno53_right(a, dm, d0), L1 = weno53_left(b, d0, d1), R1 = weno53_right(b, d0, d1);
        if (l0) fx_listed_flux<LF>(v, G, c0, R0, L1, aglob, out);
        if (l1) fx_listed_flux<LF>(v, G, c0 + 1, R1, L2, aglob, out);
    }
}

// face values of the cells [lo, hi) of a window to ul, ur (indexed from the
// cell `at`; null: not wanted)
template <class PO>
struct StoreFaces {
    PO ul, ur;
    int lo, hi, at;
    __device__ void operator()(int j, double R, double L) const {
        if (j >= lo && j < hi) ur[j - at] = R;
        if (j + 1 >= lo && j + 1 < hi) ul[j + 1 - at] = L;
    }
};

// 288 F of the faces [jlo, jhi) into sm.D from v (valid on [jlo-2, jhi+3)): two
// adjacent cells per lane, a warp covers 64 cells and the 60 faces of lanes
// 1..30, neighbours' terms by shuffle. Faces that fixed_flux.cuh leaves go to
// the list of counter `slot` and are evaluated after a barrier. Ends with a
// barrier. The counter of the next stage is cleared on the way: its last
// readers are past this stage's first barrier. LF: the global Lax-Friedrichs
// flux with the speed aglob (at least every |v|).
template <bool LF = false, class PV, class FaceOut>
__device__ __forceinline__ void fx_fluxes(PV v, int jlo, int jhi, const Smem<double>& sm,
                                          const OpParams<double>& p, int slot, const FaceOut& out,
                                          double aglob = 0.0) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const Win<int> list = sm.fx + kFxCounters;
    const fx::FF eps4{fx::dup(p.e4h), fx::dup(p.e4l)};
    fx::Speed speed{0, 0u, true};
    if constexpr (LF) speed = fx::speed_begin(aglob);
    for (int r0 = (jlo & ~1) - 2 + 60 * warp; r0 + 2 < jhi; r0 += 60 * nw) {
        const int c0 = r0 + 2 * lane;
        // (positions outside the window only feed faces that are not stored)
        const int ca = c0 < 0 ? 0 : (c0 < sm.W - 2 ? c0 : sm.W - 2);
        const int cb = ca < sm.W - 4 ? ca + 2 : sm.W - 2;
        const double2 a = *reinterpret_cast<const double2*>(win_span(v, ca, 2));
        const double2 b = *reinterpret_cast<const double2*>(win_span(v, cb, 2));
        const fx::Lane s = fx::lane_begin(v[ca > 0 ? ca - 1 : 0], a.x, a.y, b.x, b.y, eps4);
        const float amh = __shfl_up_sync(kFull, fx::p2y(s.a.h), 1), aml = __shfl_up_sync(kFull, fx::p2y(s.a.l), 1);
        const float gph = __shfl_down_sync(kFull, fx::p2x(s.g.h), 1), gpl = __shfl_down_sync(kFull, fx::p2x(s.g.l), 1);
        const float Tmh = __shfl_up_sync(kFull, fx::p2y(s.T.h), 1), Tml = __shfl_up_sync(kFull, fx::p2y(s.T.l), 1);
        fx::FF pR, pL;
        fx::lane_cells(s, amh, aml, gph, gpl, Tmh, Tml, pR, pL);
        const float nLh = __shfl_down_sync(kFull, fx::p2x(pL.h), 1), nLl = __shfl_down_sync(kFull, fx::p2x(pL.l), 1);
        // faces c0 and c0 + 1: R from the lane's two cells, L from cell c0 + 1 and
        // the next lane's first
        const fx::Sums u = fx::face_units(pR, fx::FF{fx::p2(fx::p2y(pL.h), nLh), fx::p2(fx::p2y(pL.l), nLl)},
                                          fx::p2(s.x.iu, s.y.iu));
        const bool inner = lane >= 1 && lane <= 30;
        const bool m0 = inner && c0 >= jlo && c0 < jhi, m1 = inner && c0 + 1 >= jlo && c0 + 1 < jhi;
        // (the flux of a face left to the list is overwritten after the barrier)
        auto face = [&](int j, const fx::Cell& c, bool mine, float xR, float xL, float tR, float tL, float rs,
                        float rd) -> double {
            int64_t Z, D, Q;
            const bool ok = fx::face_sums(c, xR, xL, tR, tL, rs, rd, Z, D, Q) && speed.in;
            if (mine) {
                if (!ok) list[atomicAdd(&sm.fx[slot], 1)] = j;
                else if (out.ul)
                    out(j, fx::to_double(Z + D, c.kz) * (1.0 / 12.0), fx::to_double(Z - D, c.kz) * (1.0 / 12.0));
            }
            if constexpr (LF) return fx::face_flux_lf(c, Z, D, speed);
            else return fx::face_flux(c.k, Z, D, Q);
        };
        const double f0 = face(c0, s.x, m0, fx::p2x(u.xR), fx::p2x(u.xL), fx::p2x(u.tR), fx::p2x(u.tL),
                               fx::p2x(u.rs), fx::p2x(u.rd));
        const double f1 = face(c0 + 1, s.y, m1, fx::p2y(u.xR), fx::p2y(u.xL), fx::p2y(u.tR), fx::p2y(u.tL),
                               fx::p2y(u.rs), fx::p2y(u.rd));
        if (m0 && m1) *reinterpret_cast<double2*>(win_span(sm.D, c0, 2)) = make_double2(f0, f1);
        else if (m0) sm.D[c0] = f0;
        else if (m1) sm.D[c0 + 1] = f1;
    }
    __syncthreads();
    const int cnt = sm.fx[slot];
    if (threadIdx.x == 0) {
        sm.fx[slot == 2 ? 0 : slot + 1] = 0;
        if (slot == 1) sm.fx[0] = 0;  // (a step may end before its third stage)
    }
    if (cnt > 0) {
        if (fx_many(cnt, jhi - jlo)) fx_listed_tile<LF>(v, sm.D, list, cnt, jlo, jhi, sm.W, p.eps, aglob, out);
        else fx_listed_faces<LF>(v, sm.D, list, cnt, p.eps, aglob, out);
        __syncthreads();
    }
}

// the reference's stage formulas (timestepping.py:312-320) on those fluxes, in
// one loop over the stages: the flux code is long, and three copies of it
// missed the instruction cache. The updates stay in these textbook formulas:
// sums of increments doubled the FP64 work's error (3e-15 against 7e-16 after
// 50 steps). Bound by issue (65 % of the slots) with the integer pipe 50 %, FMA
// 47 % and FP64 49 % of its cycles busy: 10 of the 12.8 FP64 instructions per
// cell-step are the update's, the rest the listed faces'.
__device__ __forceinline__ unsigned long long step_tile_fx(const Smem<double>& sm, Win<double> gout, int te,
                                                           double dtdx, const OpParams<double>& p,
                                                           const BcView& bc, int64_t g0, int64_t n,
                                                           const StageOut<double>& so) {
    constexpr int HL = step_halo<double>();
    const int tid = threadIdx.x, nt = blockDim.x;
    const bool np = !bc.periodic();
    if (np) apply_bc(sm.U, g0, n, 0, te + 2 * HL, bc, 0);
    const double c = dtdx * (1.0 / 288.0);
    unsigned long long mx = 0;
#pragma unroll 1
    for (int s = 0; s < 3; ++s) {
        if (s == 2 && !gout && !so.ul2) break;
        const int lo = HL - 6 + 3 * s, hi = HL + te + 6 - 3 * s;
        const Win<double> v = s == 0 ? sm.U : sm.S;
        const Win<double> ul = s == 0 ? so.ulu : (s == 1 ? so.ul1 : so.ul2);
        const Win<double> ur = s == 0 ? so.uru : (s == 1 ? so.ur1 : so.ur2);
        fx_fluxes(v, lo - 1, hi, sm, p, s, StoreFaces<Win<double>>{ul, ur, HL, HL + te, HL});
        if (s == 2 && !gout) break;
        // the stage formula at the cells i, i + 1 (i even; hi <= W - 4): one value
        // per cell, vector accesses
        auto ld2 = [](const Win<double>& a, int i) { return *reinterpret_cast<const double2*>(win_span(a, i, 2)); };
        for (int i = (lo & ~1) + 2 * tid; i < hi; i += 2 * nt) {
            const double2 f = ld2(sm.D, i), u = ld2(sm.U, i);
            const double r0 = sm.D[i - 1] - f.x, r1 = f.x - f.y;
            double2 w;
            if (s == 0) {
                w = make_double2(fma(c, r0, u.x), fma(c, r1, u.y));
            } else {
                const double2 k = ld2(sm.S, i);
                const double a = s == 1 ? 1.0 / 4.0 : 2.0 / 3.0, b = s == 1 ? 3.0 / 4.0 : 1.0 / 3.0;
                w = make_double2(fma(a, fma(c, r0, k.x), b * u.x), fma(a, fma(c, r1, k.y), b * u.y));
            }
            const bool v0 = i >= lo, v1 = i + 1 < hi;
            if (s < 2) {
                if (v0 && v1) *reinterpret_cast<double2*>(win_span(sm.S, i, 2)) = w;
                else if (v0) sm.S[i] = w.x;
                else sm.S[i + 1] = w.y;
            } else {
                if (v0) {
                    gout[i - HL] = w.x;
                    const unsigned long long b0 = abs_bits(w.x);
                    mx = b0 > mx ? b0 : mx;
                }
                if (v1) {
                    gout[i + 1 - HL] = w.y;
                    const unsigned long long b1 = abs_bits(w.y);
                    mx = b1 > mx ? b1 : mx;
                }
            }
        }
        if (s == 2) break;
        __syncthreads();
        if (np) apply_bc(sm.S, g0, n, lo, hi, bc, s + 1);
        store_interior(s == 0 ? so.k1 : so.k2, sm.S, HL, te);
    }
    return mx;
}

// g0: global cell of window position 0 (s - HL); n: cells of the instance;
// bc: its boundary (periodic: nothing to overwrite)
// so: what the reverse sweep keeps of this step (StageOut); gout may then be
// null (the last stage is skipped)
template <class T, int EQ, int REC, int FLUX>
__device__ typename Bits<T>::type step_tile(const Smem<T>& sm, Win<T> gout, int te, T dtdx,
                                            const OpParams<T>& p, const BcView& bc = BcView(),
                                            int64_t g0 = 0, int64_t n = 0,
                                            const StageOut<stage_t<T, REC>>& so = StageOut<stage_t<T, REC>>()) {
    if constexpr (FLUX == kFluxRusanovFx) {
        return step_tile_fx(sm, gout, te, dtdx, p, bc, g0, n, so);
    } else {
    if constexpr (sizeof(T) == 8 && REC == SHK_REC_LEARNED)
        return step_tile_mixed<EQ, FLUX>(sm, gout, te, dtdx, p, bc, g0, n, so);
    if constexpr (sizeof(T) == 4 && REC == SHK_REC_WENOJS53 && FLUX == SHK_FLUX_RUSANOV)
        return step_tile_f32_weno<EQ>(sm, gout, te, dtdx, p, bc, g0, n, so);
    constexpr int HL = step_halo<T>();
    const int tid = threadIdx.x, nt = blockDim.x;
    const bool np = !bc.periodic();
    if (np) apply_bc(sm.U, g0, n, 0, te + 2 * HL, bc, 0);
    dtdx *= p.fscale;
    if constexpr (sizeof(T) == 4) {
        // float state: the stages as increments about u (as step_tile_mixed).
        // In float 1/3 + 2/3 rounds to 1 + 3e-8, so the textbook combination
        // would scale the mass by that every step; the increments telescope,
        // and conservation holds to rounding.
        {
            const int lo = HL - 6, hi = HL + te + 6;
            face_fluxes<T, EQ, REC, FLUX>(sm.U, lo, hi, sm, p);
            for (int i = lo + tid; i < hi; i += nt) {
                const T d = dtdx * (sm.D[i - 1] - sm.D[i]);
                sm.I[i] = d;
                sm.S[i] = sm.U[i] + d;
            }
            __syncthreads();
            if (np) apply_bc(sm.S, g0, n, lo, hi, bc, 1);
            store_interior(so.k1, sm.S, HL, te);
        }
        {
            const int lo = HL - 3, hi = HL + te + 3;
            face_fluxes<T, EQ, REC, FLUX>(sm.S, lo, hi, sm, p);
            for (int i = lo + tid; i < hi; i += nt) {
                const T d = T(0.25) * (sm.I[i] + dtdx * (sm.D[i - 1] - sm.D[i]));
                sm.I[i] = d;
                sm.S[i] = sm.U[i] + d;
            }
            __syncthreads();
            if (np) apply_bc(sm.S, g0, n, lo, hi, bc, 2);
            store_interior(so.k2, sm.S, HL, te);
        }
        using B = typename Bits<T>::type;
        B mx = 0;
        if (!gout) return mx;
        const int lo = HL, hi = HL + te;
        face_fluxes<T, EQ, REC, FLUX>(sm.S, lo, hi, sm, p);
        for (int i = lo + tid; i < hi; i += nt) {
            const T un = sm.U[i] + T(2.0 / 3.0) * (sm.I[i] + dtdx * (sm.D[i - 1] - sm.D[i]));
            gout[i - HL] = un;
            const B b = abs_bits(wave_speed<EQ>(un, p.c));
            mx = b > mx ? b : mx;
        }
        return mx;
    }
    // double state: the reference's stage formulas (timestepping.py:312-320)
    // stage 1: k1 = u + dt L(u) on [HL-6, HL+te+6)
    {
        const int lo = HL - 6, hi = HL + te + 6;
        face_fluxes<T, EQ, REC, FLUX>(sm.U, lo, hi, sm, p);
        store_interior(so.ulu, sm.UL, HL, te);
        store_interior(so.uru, sm.UR, HL, te);
        for (int i = lo + tid; i < hi; i += nt) sm.S[i] = fma(dtdx, sm.D[i - 1] - sm.D[i], sm.U[i]);
        __syncthreads();
        if (np) apply_bc(sm.S, g0, n, lo, hi, bc, 1);
        store_interior(so.k1, sm.S, HL, te);
    }
    // stage 2: k2 = 3/4 u + 1/4 (k1 + dt L(k1)) on [HL-3, HL+te+3) (in place over k1)
    {
        const int lo = HL - 3, hi = HL + te + 3;
        face_fluxes<T, EQ, REC, FLUX>(sm.S, lo, hi, sm, p);
        store_interior(so.ul1, sm.UL, HL, te);
        store_interior(so.ur1, sm.UR, HL, te);
        for (int i = lo + tid; i < hi; i += nt) {
            const T k = fma(dtdx, sm.D[i - 1] - sm.D[i], sm.S[i]);
            sm.S[i] = fma(T(1.0 / 4.0), k, T(3.0 / 4.0) * sm.U[i]);
        }
        __syncthreads();
        if (np) apply_bc(sm.S, g0, n, lo, hi, bc, 2);
        store_interior(so.k2, sm.S, HL, te);
    }
    // stage 3: u+ = 1/3 u + 2/3 (k2 + dt L(k2)) on the tile
    using B = typename Bits<T>::type;
    B mx = 0;
    if (!gout && !so.ul2) return mx;
    {
        const int lo = HL, hi = HL + te;
        face_fluxes<T, EQ, REC, FLUX>(sm.S, lo, hi, sm, p);
        store_interior(so.ul2, sm.UL, HL, te);
        store_interior(so.ur2, sm.UR, HL, te);
        if (!gout) return mx;
        for (int i = lo + tid; i < hi; i += nt) {
            const T k = fma(dtdx, sm.D[i - 1] - sm.D[i], sm.S[i]);
            const T un = fma(T(2.0 / 3.0), k, T(1.0 / 3.0) * sm.U[i]);
            gout[i - HL] = un;
            const B b = abs_bits(wave_speed<EQ>(un, p.c));
            mx = b > mx ? b : mx;
        }
    }
    return mx;
    }
}

// one work item: tile `tile` of the `tiles` of instance b (te cells of it), whose n
// cells start at off
struct __align__(16) PlanItem {
    int64_t off, n;
    int32_t b, te, tile, tiles;
};

// device view of a batched plan (see shk_plan in forward.cu)
struct PlanDev {
    const int32_t* item_inst;
    const int32_t* item_tile;
    const int64_t* offsets;  // [B+1]
    const double* cfl;       // [B] 0.5 dx^(2-alpha)
    const double* inv_dx;    // [B]
    const double* tfinal;    // [B]
    double theta;
    unsigned long long* amax;  // [2][B] bits of max |f'(u)| (as double)
    double* t;                 // [B]
    double* dt_hist;           // [max_steps][B] or null
    int64_t* step;
    unsigned int* done;
    int32_t* status;
    double* partial;  // [nitems]
    const double* dt_fixed;  // [fixed_steps][B] prescribed steps, or null (CFL steps)
    int64_t fixed_steps;
    int bc_left, bc_right;   // SHK_BC_* of every instance
    const double* bc_dir;    // [B][2][3] Dirichlet ghost values, or [bc_steps][3][B][2][3]
    const double* bc_neu;    // [B][2] Neumann gradients, or [bc_steps][3][B][2]
    int64_t bc_steps;        // 0: time-independent data; else per-step, per-stage tables
    const PlanItem* items;      // [nitems] longest first (dynamic scheduling)
    unsigned int* left;         // [B] tiles of the running step that are done
    unsigned int* sched;        // [8] item counters of the scheduled kernels
    int32_t B, nitems, tile, max_steps;
};

// Dynamic item scheduling. A CTA takes the items of the plan's longest-first
// list from the counter sched[slot]; uneven items (partial tiles, copied-through
// instances) then balance over the persistent grid, where a fixed stride would
// hand some CTAs only long items. The first item is the CTA's own index. EARLY:
// the next one is requested when an item begins, so the counter's latency is
// behind it; kernels with few, long and unequal items take it when an item ends
// (bound early, the learned reverse step lost 12 % to the imbalance).
// s: two words of shared memory (a thread may still read one when the next is
// written).
template <bool EARLY = true>
struct ItemQueue {
    const PlanDev& P;
    int slot;
    int* s;
    int q, par = 0;
    unsigned next = 0;
    __device__ __forceinline__ ItemQueue(const PlanDev& P_, int slot_, int* s_)
        : P(P_), slot(slot_), s(s_), q(static_cast<int>(blockIdx.x)) {}
    __device__ __forceinline__ bool more() const { return q < P.nitems; }
    __device__ __forceinline__ PlanItem begin() {
        if (EARLY && threadIdx.x == 0) next = atomicAdd(P.sched + slot, 1u) + gridDim.x;
        return P.items[q];
    }
    // a barrier
    __device__ __forceinline__ void end() {
        if (threadIdx.x == 0) s[par] = static_cast<int>(EARLY ? next : atomicAdd(P.sched + slot, 1u) + gridDim.x);
        __syncthreads();
        q = s[par];
        par ^= 1;
    }
};

// end of a scheduled launch: the CTA that finishes last (counter
// sched[slot + 1]) resets both counters for the next launch
__device__ __forceinline__ void finish_items(const PlanDev& P, int slot) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(P.sched + slot + 1, 1u) == gridDim.x - 1) {
            atomicExch(P.sched + slot, 0u);
            atomicExch(P.sched + slot + 1, 0u);
            __threadfence();
        }
    }
}

// the boundary of instance b at step k: time-independent data (one set for
// all three stages), or the step's row of a per-step table (steps past the
// table take its last row)
__device__ __forceinline__ BcView plan_bc(const PlanDev& P, int b, int64_t k) {
    BcView v;
    v.left = P.bc_left;
    v.right = P.bc_right;
    if (!v.periodic()) {
        if (P.bc_steps > 0) {
            const int64_t kk = k < P.bc_steps ? k : P.bc_steps - 1;
            const size_t row = size_t(kk) * 3 * P.B + b;
            v.dir = P.bc_dir ? P.bc_dir + row * 6 : nullptr;
            v.dir_ss = 6 * P.B;
            v.neu = P.bc_neu ? P.bc_neu + row * 2 : nullptr;
            v.neu_ss = 2 * P.B;
        } else {
            v.dir = P.bc_dir ? P.bc_dir + size_t(b) * 6 : nullptr;
            v.neu = P.bc_neu ? P.bc_neu + size_t(b) * 2 : nullptr;
        }
        v.dx = 1.0 / P.inv_dx[b];
    }
    return v;
}

// time step k of instance b: the prescribed step when the plan has a dt table
// (a step <= 0 or past the table's end leaves the instance unchanged, a
// non-finite one is an error), else the CFL step clipped at tfinal
__device__ __forceinline__ DtState plan_dt(const PlanDev& P, int64_t k, int b, double smax) {
    if (P.dt_fixed) {
        DtState s;
        s.dt = k < P.fixed_steps ? P.dt_fixed[size_t(k) * P.B + b] : 0.0;
        s.active = !(s.dt <= 0.0);
        s.finite = isfinite(s.dt);
        return s;
    }
    return compute_dt(smax, P.cfl[b], P.theta, P.t[b], P.tfinal[b]);
}

template <class T>
__device__ __forceinline__ unsigned long long to_double_bits(typename Bits<T>::type b) {
    if constexpr (sizeof(T) == 8) return b;
    else return abs_bits(static_cast<double>(from_bits(b)));
}

// read-only view of a plan's device state (defined in forward.cu)
int plan_view(shk_plan* plan, PlanDev* dev, int* dtype, int* grid, shk_scheme* scheme,
              int64_t* total_cells, int64_t* host_steps);

}  // namespace shk
