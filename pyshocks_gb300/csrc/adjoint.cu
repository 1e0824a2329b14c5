// Discrete adjoint of the SSPRK33 / WENO-JS5 / Rusanov step (dt frozen).
//
// Reference: adjoint_step (src/pyshocks/timestepping.py:155-215) builds the
// dense Jacobian of one step with jax.jacfwd(advance) (:174) and applies
// p <- jac.T @ p (:206), with dt re-read from the forward checkpoints
// (:200-201), i.e. not differentiated. Here the transpose Jacobian-vector
// product of one step is evaluated matrix-free, one tile per work item:
//
//   forward:  k1 = u + dt L(u)
//             k2 = 3/4 u + 1/4 (k1 + dt L(k1))
//             u+ = 1/3 u + 2/3 (k2 + dt L(k2))          (timestepping.py:318-320)
//   reverse:  k2b = 2/3 (p + dt J(k2)^T p)
//             k1b = 1/4 (k2b + dt J(k1)^T k2b)
//             ub  = 1/3 p + 3/4 k2b + k1b + dt J(u)^T k1b
//
// J(v)^T w of L(v) = -(F_{i+1/2} - F_{i-1/2})/dx is assembled from the
// derivatives of the Rusanov flux (scalar.py:248, a = max(|f'(v_i)|,
// |f'(v_{i+1})|) from cell values, scalar.py:243-246) and of the WENO-JS5
// reconstruction (weno.py:114-157,247-256), differentiated by hand in the
// product form of device.cuh. Non-differentiable points follow the JAX/torch
// conventions: d|x|/dx = 0 at 0, and max() splits the cotangent evenly at
// ties. The states k1, k2 come from the segment replay's stage storage, or are
// recomputed from u in shared memory (halo 18).
//
// Periodic boundaries are circular indexing, and cotangents live on interior
// cells only (the reference's ghost rows carry zero cotangent when J only
// involves interior cells, see pyshocks_gb300/adjoint.py).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

#include "adjoint_math.cuh"

namespace shk {

constexpr int kAdjTile = 512;
template <class T> __host__ __device__ constexpr int adj_uhalo() { return 20; }  // 18 needed
template <class T> __host__ __device__ constexpr int adj_phalo() { return sizeof(T) == 8 ? 10 : 12; }  // 9 needed
constexpr int kAdjArrays = 24;

template <class T>
struct AdjSmem {
    Win<T> U, K1, K2, PB, CB, Z, ACC;
    Win<T> H, D, Q, UL, UR;
    Win<T> GL, GR, GA;
    Win<T> T0, T1, T2, T3, T4;
    Win<T> CLu, CRu, CL1, CR1;  // face values of u and k1 from the forward recompute
    int W;  // window length (cells) of every array

    __host__ static size_t host_bytes(int W) { return size_t(kAdjArrays) * W * sizeof(T); }
    __device__ void carve(unsigned char* base, int W) {
        T* p = reinterpret_cast<T*>(base);
        Win<T>* slots[kAdjArrays] = {&U, &K1, &K2, &PB, &CB, &Z, &ACC, &H, &D, &Q,
                                     &UL, &UR, &GL, &GR, &GA, &T0, &T1, &T2, &T3, &T4,
                                     &CLu, &CRu, &CL1, &CR1};
        for (int i = 0; i < kAdjArrays; ++i) *slots[i] = make_win(p + size_t(i) * W, W);
        this->W = W;
    }
    // forward-stage view (face_fluxes writes the face fluxes into D and the
    // face values into ul, ur: UL, UR unless given)
    __device__ Smem<T> fwd(Win<T> state_out, Win<T> ul = Win<T>(), Win<T> ur = Win<T>()) const {
        Smem<T> s;
        s.U = U; s.S = state_out; s.H = H; s.D = D; s.Q = Q;
        s.UL = ul ? ul : UL; s.UR = ur ? ur : UR;
        // the learned phase's scratch: H and D (contiguous in both layouts)
        const int hd = 2 * W * int(sizeof(T) / sizeof(float));
        s.scr = learned_scratch(make_win(reinterpret_cast<float*>(win_raw(H)), hd), hd);
        s.W = W;
        return s;
    }
};

// z_i = dt (J_L(v)^T w)_i for i in [lo, hi); v valid on [lo-6, hi+6), w on
// [lo-3, hi+3). Rusanov flux, WENO-JS5 or learned reconstruction.
// cul, cur (WENO-JS5): the face values of v on [lo-3, hi+3) as the forward's
// face pass forms them (stored by the replay, or kept by the recompute)
template <class T, int EQ, int REC, class PV, class PW, class PZ, class PC = Win<const T>>
__device__ void vjp_stage(PV v, PW w, PZ z, int lo, int hi, const AdjSmem<T>& a,
                          const OpParams<T>& p, T dtdx, PC cul = PC(), PC cur = PC()) {
    const int tid = threadIdx.x, nt = blockDim.x;
    if constexpr (REC == SHK_REC_LEARNED) {
        static_assert(sizeof(T) == 4, "the learned VJP runs on float stage states");
        // One pass per cell: the network forward (recomputed with the
        // inference's own mma sequence) gives the cell's face values, from
        // which the flux VJP seeds of its two faces follow, then the network
        // backward. Face j+1/2 (L = ul_{j+1}, R = ur_j) seeds cell j with
        //   gR_j = fb_j (f'(R)/2 + a_j), and cell j+1 with gL = fb_j (f'(L)/2 - a_j),
        // fb_j = dt/dx (w_{j+1} - w_j), a_j = nu/2 max(|f'(v_j)|, |f'(v_{j+1})|).
        // The face values are kept for the wave-speed terms below.
        const MlpShared& ms = mlp_shared();
        const MlpBackShared& bk = mlp_back_shared();
        // warp scratch: GL, GR, GA (3W floats, unused by this branch)
        float* scr = win_span(learned_scratch(a.GL, 3 * a.W), (tid >> 5) * kWarpScratchVjp,
                              kWarpScratchVjp);
        const int lane = tid & 31, g = lane >> 2, tq = lane & 3;
        const int myrow = 16 * (tq >> 1) + 8 * (tq & 1) + g;
        const int c0 = lo - 2, ncell = hi + 2 - c0;
        for (int qb = tid >> 5; qb * 32 < ncell; qb += nt >> 5) {
            const int r = qb * 32 + myrow;
            const int c = c0 + min(r, ncell - 1);
            // the stencil relative to v_c as the forward forms it (learned_phase)
            const float vm = v[c - 1], vc = v[c], vp = v[c + 1];
            const float sc[5] = {v[c - 2] - vc, vm - vc, 0.0f, vp - vc, v[c + 2] - vc};
            const float wm = w[c - 1], wc = w[c], wp = w[c + 1];
            float ul = 0.0f, ur = 0.0f;
            auto seed = [&](float cr, float cl, float& gR, float& gL) {
                ur = vc + cr;
                ul = vc + cl;
                const float wsc = wave_speed<EQ>(vc, p.c);
                const float hp = p.hnu * absmax(wsc, wave_speed<EQ>(vp, p.c));
                const float hm = p.hnu * absmax(wave_speed<EQ>(vm, p.c), wsc);
                gR = ((wp - wc) * dtdx) * fmaf(0.5f, flux_prime<EQ>(ur, p.c), hp);
                gL = ((wc - wm) * dtdx) * fmaf(0.5f, flux_prime<EQ>(ul, p.c), -hm);
            };
            float dd[5];
            learned_cell_vjp32(ms, bk, sc, seed, p.lp, scr, dd);
            if (r < ncell) {
                a.T0[c] = dd[0]; a.T1[c] = dd[1]; a.T2[c] = dd[2]; a.T3[c] = dd[3]; a.T4[c] = dd[4];
                a.UL[c] = ul;
                a.UR[c] = ur;
            }
        }
        __syncthreads();
        for (int i = lo + tid; i < hi; i += nt) {
            T acc = (a.T0[i + 2] + a.T1[i + 1]) + a.T2[i] + (a.T3[i - 1] + a.T4[i - 2]);
            // wave-speed terms: face i-1/2 (cells i-1, i) and face i+1/2 (cells i, i+1)
            const T gam = -(((w[i] - w[i - 1]) * dtdx) * p.hnu) * (a.UL[i] - a.UR[i - 1]);
            const T gap = -(((w[i + 1] - w[i]) * dtdx) * p.hnu) * (a.UL[i + 1] - a.UR[i]);
            acc = fma(gam, damax_dx<EQ>(v[i], v[i - 1], p.c), acc);
            acc = fma(gap, damax_dx<EQ>(v[i], v[i + 1], p.c), acc);
            z[i] = acc;
        }
        __syncthreads();
        return;
    }
    for (int c = lo - 5 + tid; c < hi + 4; c += nt) a.H[c] = T(0.5) * (v[c + 1] - v[c]);
    __syncthreads();
    for (int c = lo - 4 + tid; c < hi + 4; c += nt) {
        const T d = a.H[c] - a.H[c - 1];
        a.D[c] = d;
        a.Q[c] = (T(13.0 / 3.0) * d) * d;
    }
    __syncthreads();
    const PC UL = cul;
    const PC UR = cur;
    // face j+1/2: F = 1/2 (f(L) + f(R)) - nu/2 a (L - R), L = ul_{j+1}, R = ur_j
    for (int j = lo - 3 + tid; j < hi + 2; j += nt) {
        const T fb = (w[j + 1] - w[j]) * dtdx;
        const T L = UL[j + 1], R = UR[j];
        const T ha = p.hnu * absmax(wave_speed<EQ>(v[j], p.c), wave_speed<EQ>(v[j + 1], p.c));
        a.GL[j] = fb * fma(T(0.5), flux_prime<EQ>(L, p.c), -ha);
        a.GR[j] = fb * fma(T(0.5), flux_prime<EQ>(R, p.c), ha);
        a.GA[j] = -(fb * p.hnu) * (L - R);
    }
    __syncthreads();
    for (int c = lo - 2 + tid; c < hi + 2; c += nt) {
        T t0, t1, t2, t3, t4;
        weno53_cell_vjp<T>(a.H[c - 2], a.H[c - 1], a.H[c], a.H[c + 1], a.D[c - 1], a.D[c],
                           a.D[c + 1], a.Q[c - 1], a.Q[c], a.Q[c + 1], p.eps, a.GR[c],
                           a.GL[c - 1], t0, t1, t2, t3, t4);
        a.T0[c] = t0; a.T1[c] = t1; a.T2[c] = t2; a.T3[c] = t3; a.T4[c] = t4;
    }
    __syncthreads();
    for (int i = lo + tid; i < hi; i += nt) {
        T acc = (a.T0[i + 2] + a.T1[i + 1]) + a.T2[i] + (a.T3[i - 1] + a.T4[i - 2]);
        // wave-speed terms: face i-1/2 (cells i-1, i) and face i+1/2 (cells i, i+1)
        acc = fma(a.GA[i - 1], damax_dx<EQ>(v[i], v[i - 1], p.c), acc);
        acc = fma(a.GA[i], damax_dx<EQ>(v[i], v[i + 1], p.c), acc);
        z[i] = acc;
    }
    __syncthreads();
}

// The FP64 backward of a cell's two face values for the listed cells of fx_vjp_stage
// (113 operations; weno53_cell_vjp with its inputs 147): the taps t_o of v_{c+o},
// o = -2..2, for gR, gL = 1/6 of the cotangents of the right and left face value. On
// c_k = 6 (sub-stencil value - v), their weights rho_k, lam_k times the seed and the
// sums e_k = 4 (eps + beta_k), e = h^2 + 13/3 E^2 + 4 eps: a weight's part is
// -2 rho_k (c_k - mean) / e_k in e_k. The taps sum to 6 (gR + gL).
template <class PV>
__device__ __forceinline__ void weno53_listed_vjp(PV v, int c, double eps4, double gR, double gL, double& t0,
                                                  double& t1, double& t2, double& t3, double& t4) {
    const double vm = v[c - 1], x = v[c], vp = v[c + 1];
    const double dm = vm - v[c - 2], a = x - vm, b = vp - x, dp = v[c + 2] - vp;
    const double Em = a - dm, E = b - a, Ep = dp - b;
    const double h0 = fma(2.0, a, Em), h1 = b + a, h2 = fma(-2.0, b, Ep);
    const double f0 = (13.0 / 3.0) * Em, f1 = (13.0 / 3.0) * E, f2 = (13.0 / 3.0) * Ep;
    const double e0 = fma(h0, h0, fma(f0, Em, eps4));
    const double e1 = fma(h1, h1, fma(f1, E, eps4));
    const double e2 = fma(h2, h2, fma(f2, Ep, eps4));
    const double e12 = e1 * e2, e02 = e0 * e2, e01 = e0 * e1;
    const double P0 = e12 * e12, P1 = 6.0 * (e02 * e02), P2 = e01 * e01, Q0 = 3.0 * P0, Q2 = 3.0 * P2;
    const double c0 = fma(2.0, h0, -a), c1 = fma(2.0, b, a), c2 = b - h2;
    const double l0 = fma(2.0, h2, b), l1 = -fma(2.0, a, b), l2 = -(h0 + a);
    const double iR = rcp_nr(P0 + P1 + Q2), iL = rcp_nr(P2 + P1 + Q0);
    const double cR = fma(P0, c0, fma(P1, c1, Q2 * c2)) * iR, cL = fma(P2, l0, fma(P1, l1, Q0 * l2)) * iL;
    const double gsum = gR + gL;
    gR *= iR;
    gL *= iL;
    const double rho0 = gR * P0, rho1 = gR * P1, rho2 = gR * Q2;
    const double lam0 = gL * P2, lam1 = gL * P1, lam2 = gL * Q0;
    const double q = rcp_nr(e01 * e2);
    const double k0 = fma(rho0, c0 - cR, lam2 * (l2 - cL)) * (e12 * q);
    const double k1 = fma(rho1, c1 - cR, lam1 * (l1 - cL)) * (e02 * q);
    const double k2 = fma(rho2, c2 - cR, lam0 * (l0 - cL)) * (e01 * q);
    const double kh0 = k0 * h0, kh1 = k1 * h1, kh2 = k2 * h2, kE0 = k0 * f0, kE1 = k1 * f1, kE2 = k2 * f2;
    // h_0 (1, -4, 3, 0, 0), h_1 (0, -1, 0, 1, 0), h_2 (0, 0, 3, -4, 1), E_k (1, -2, 1);
    // c_0 (2, -7, 5, 0, 0), c_1 (0, -1, -1, 2, 0), c_2 (0, 0, -4, 5, -1), l_k mirrored
    t0 = fma(-4.0, kh0 + kE0, fma(2.0, rho0, -lam2));
    t1 = fma(-4.0, fma(-4.0, kh0, fma(-2.0, kE0, kE1 - kh1)),
             fma(5.0, lam2, fma(2.0, lam1, fma(-7.0, rho0, -rho1))));
    t3 = fma(-4.0, fma(-4.0, kh2, fma(-2.0, kE2, kE1 + kh1)),
             fma(5.0, rho2, fma(2.0, rho1, fma(-7.0, lam0, -lam1))));
    t4 = fma(-4.0, kh2 + kE2, fma(2.0, lam0, -rho2));
    t2 = fma(6.0, gsum, -((t0 + t1) + (t3 + t4)));
}

// vjp_stage for the schemes of fixed_flux_scheme. The FP64 pipe bounded the
// reverse step at 159 operations per cell and stage, most of them in the
// reconstruction's backward. Its linear (ideal-weight) part, the flux seeds and
// the sums stay in FP64 (25 operations); the rest, small where the state is
// smooth, is formed in pairs of floats two cells per lane (lane_grad). Cells
// with a weight change |x0| + |x2| above 1/8 or a third difference out of range
// are listed and take the FP64 backward, without the linear part. In units of
// g / 60: GR, GL, GA hold the flux seeds of the faces; a.H takes the pair part of
// z, a.D the list, a.Q the flags of the listed cells, T0..T4 their taps.
// The pairs hold the seeds relative to the warp's largest. Where a warp's cells span
// more than kPairRange powers of two (then the lower halves of the smallest near
// float's smallest number, 2^-149) or leave 2^+-823, every cell of the window is listed:
// warps share cells, so one warp alone cannot list its own.
// A warp whose cells are all listed skips its pairs. Reverse sweep of ten steps, 96
// instances (0.4 M cells), us (FP64 backward everywhere / the pairs in vain and the linear
// part twice / this): 0.5 % noise 5327 / 6680 / 4725, random 5326 / 7032 / 4741, smooth 5324 /
// 1444 / 1456.
constexpr float kSmoothWeights = 0.125f;
constexpr unsigned kPairRange = 80u;
template <class PV, class PW, class PZ, class PC>
__device__ void fx_vjp_stage(PV v, PW w, PZ z, int lo, int hi, const AdjSmem<double>& a, const OpParams<double>& p,
                             double dtdx, PC UL, PC UR) {
    constexpr unsigned kFull = 0xffffffffu;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    // list[0]: count, list[1]: list every cell, from list[4]: the cells
    const Win<int> list = win_cast<int>(a.D), flag = win_cast<int>(a.Q);
    if (tid == 0) list[0] = list[1] = 0;
    const double cf = dtdx * (1.0 / 120.0);
    for (int j = lo - 3 + tid; j < hi + 2; j += nt) {
        const double fb = (w[j + 1] - w[j]) * cf;
        const double L = UL[j + 1], R = UR[j], s = absmax(v[j], v[j + 1]);
        a.GL[j] = fb * (L - s);
        a.GR[j] = fb * (R + s);
        a.GA[j] = fb * (R - L);
    }
    __syncthreads();
    const fx::FF eps4{fx::dup(p.e4h), fx::dup(p.e4l)};
    // a warp takes 64 cells and finishes z of 58 (those at 4 .. 61)
    const int first = (lo & ~1) - 4;
    for (int r0 = first + 58 * warp; r0 + 4 < hi; r0 += 58 * nw) {
        const int c0 = r0 + 2 * lane;
        const int ca = c0 < a.W - 2 ? c0 : a.W - 2, cb = ca < a.W - 4 ? ca + 2 : a.W - 2;
        auto ld2 = [](const auto& q, int i) { return *reinterpret_cast<const double2*>(win_span(q, i, 2)); };
        const double2 va = ld2(v, ca), vb = ld2(v, cb), gr = ld2(a.GR, ca);
        const double gl0 = a.GL[ca - 1], gl1 = a.GL[ca];
        // the seeds relative to a power of two of the warp's largest (exact: the
        // backward is linear in them). Every cell whose seeds are used counts, by
        // itself: [lo - 2, hi + 2) may begin or end inside a lane's pair, and beyond it
        // the seeds are not written
        unsigned em, least;
        {
            auto top = [&](int c, double r, double l) -> unsigned {
                const unsigned hr = static_cast<unsigned>(__double2hiint(r)) & 0x7fffffffu;
                const unsigned hl = static_cast<unsigned>(__double2hiint(l)) & 0x7fffffffu;
                const bool used = static_cast<unsigned>(c - (lo - 2)) < static_cast<unsigned>(hi - lo + 4);
                return used ? (hr > hl ? hr : hl) : 0u;
            };
            const unsigned h0 = top(c0, gr.x, gl0), h1 = top(c0 + 1, gr.y, gl1);
            em = __reduce_max_sync(kFull, h0 > h1 ? h0 : h1) >> 20;
            // (zeros do not count)
            least = __reduce_min_sync(kFull, h0 - 1u < h1 - 1u ? h0 - 1u : h1 - 1u) >> 20;
        }
        if (lane == 0 && (em > 1846u || least < 200u || least + kPairRange < em)) list[1] = 1;
        em = em < 200u ? 200u : em;
        fx::CellGrad g;
        bool b0, b1;
        {
            fx::Cell x, y;
            {
                const fx::Mag m0 = fx::mag(v[ca - 1]), m1 = fx::mag(va.x), m2 = fx::mag(va.y), m3 = fx::mag(vb.x),
                              m4 = fx::mag(vb.y);
                x = fx::cell_begin(m0, m1, m2, m3);
                y = fx::cell_begin(m1, m2, m3, m4);
            }
            const fx::P2 u0 = fx::p2(x.u0, y.u0), u12 = u0 * fx::dup(0x1p12f), u36 = u0 * fx::dup(0x1p36f);
            const float nan = fx::bitsf(0x7fffffffu);
            fx::FF T0 = fx::to_ff50(x.T, y.T, u0 * fx::dup(0x1p26f), u0);
            T0.h = fx::p2(x.ok ? fx::p2x(T0.h) : nan, y.ok ? fx::p2y(T0.h) : nan);
            const float Tmh = __shfl_up_sync(kFull, fx::p2y(T0.h), 1), Tml = __shfl_up_sync(kFull, fx::p2y(T0.l), 1);
            const fx::FF Tm{fx::p2(Tmh, fx::p2x(T0.h)), fx::p2(Tml, fx::p2x(T0.l))};
            const fx::FF S = fx::to_ff(x.S, y.S, u36, u12, u0), E = fx::to_ff(x.E, y.E, u36, u12, u0);
            const fx::CellWeights cw = fx::lane_weights(S, E, Tm, T0, eps4);
            // listed cells: nothing here
            b0 = !(fx::p2x(cw.x) <= kSmoothWeights);
            b1 = !(fx::p2y(cw.x) <= kSmoothWeights);
            auto mark = [&](int q, int c, bool bad) {
                const bool mine = (q >= 4 && q < 62) || (r0 == first && q >= 2 && q < 4) || (r0 + 62 >= hi && q >= 62);
                if (mine && c >= lo - 2 && c < hi + 2) {
                    flag[c] = bad ? 1 : 0;
                    if (bad) list[4 + atomicAdd(&list[0], 1)] = c;
                }
            };
            mark(2 * lane, c0, b0);
            mark(2 * lane + 1, c0 + 1, b1);
            // (noise: all of them)
            const bool out0 = c0 < lo - 2 || c0 >= hi + 2, out1 = c0 + 1 < lo - 2 || c0 + 1 >= hi + 2;
            if (__all_sync(kFull, lane == 0 || ((b0 || out0) && (b1 || out1)))) {
                if (lane >= 2 && lane <= 30) {
                    if (c0 >= lo && c0 < hi) a.H[c0] = 0.0;
                    if (c0 + 1 >= lo && c0 + 1 < hi) a.H[c0 + 1] = 0.0;
                }
                continue;
            }
            float h0, l0, h1, l1;
            fx::split_double(gr.x, em, h0, l0);
            fx::split_double(gr.y, em, h1, l1);
            const fx::FF gR{fx::p2(h0, h1), fx::p2(l0, l1)};
            fx::split_double(gl0, em, h0, l0);
            fx::split_double(gl1, em, h1, l1);
            const fx::FF gL{fx::p2(h0, h1), fx::p2(l0, l1)};
            g = fx::lane_grad(cw, S, E, Tm, T0, gR, gL);
        }
        auto keep = [&](fx::P2 q) { return fx::p2(b0 ? 0.0f : fx::p2x(q), b1 ? 0.0f : fx::p2y(q)); };
        auto keep2 = [&](fx::FF q) { return fx::FF{keep(q.h), keep(q.l)}; };
        const fx::FF tm = keep2(g.tm), t0 = keep2(g.t0), sg = keep2(g.sg), et = keep2(g.et);
        // transposes of T, E and S: the cotangent of T_c, of E_c, then z (neighbours'
        // values from the lanes beside)
        auto dn = [&](float q) { return __shfl_down_sync(kFull, q, 1); };
        auto up = [&](float q) { return __shfl_up_sync(kFull, q, 1); };
        const fx::FF tn{fx::p2(fx::p2y(tm.h), dn(fx::p2x(tm.h))), fx::p2(fx::p2y(tm.l), dn(fx::p2x(tm.l)))};
        const fx::FF th = fx::add(t0, tn);
        const fx::FF tp{fx::p2(up(fx::p2y(th.h)), fx::p2x(th.h)), fx::p2(up(fx::p2y(th.l)), fx::p2x(th.l))};
        const fx::FF H = fx::add(et, fx::sub(tp, th));
        const fx::FF P = fx::add(H, sg), M = fx::sub(H, sg);
        const fx::FF Pp{fx::p2(up(fx::p2y(P.h)), fx::p2x(P.h)), fx::p2(up(fx::p2y(P.l)), fx::p2x(P.l))};
        const fx::FF Mn{fx::p2(fx::p2y(M.h), dn(fx::p2x(M.h))), fx::p2(fx::p2y(M.l), dn(fx::p2x(M.l)))};
        const fx::FF zz = fx::sub(fx::add(Pp, Mn), fx::twice(H));
        const fx::P2 zh = zz.h + zz.l, zl = zz.l - (zh - zz.h);
        if (lane >= 2 && lane <= 30) {
            if (c0 >= lo && c0 < hi) a.H[c0] = fx::join_double(fx::p2x(zh), fx::p2x(zl), em);
            if (c0 + 1 >= lo && c0 + 1 < hi) a.H[c0 + 1] = fx::join_double(fx::p2y(zh), fx::p2y(zl), em);
        }
    }
    __syncthreads();
    int cnt = list[0];
    if (list[1] != 0) {
        cnt = hi - lo + 4;
        for (int c = lo - 2 + tid; c < hi + 2; c += nt) {
            list[4 + c - (lo - 2)] = c;
            flag[c] = 1;
            if (c >= lo && c < hi) a.H[c] = 0.0;
        }
        __syncthreads();
    }
    // (the seeds of a listed cell are its own: they are taken out of the linear part below)
    for (int q = tid; q < cnt; q += nt) {
        const int c = list[4 + q];
        double t0, t1, t2, t3, t4;
        weno53_listed_vjp(v, c, 4.0 * p.eps, a.GR[c], a.GL[c - 1], t0, t1, t2, t3, t4);
        a.T0[c] = t0;
        a.T1[c] = t1;
        a.T2[c] = t2;
        a.T3[c] = t3;
        a.T4[c] = t4;
        a.GR[c] = 0.0;
        a.GL[c - 1] = 0.0;
    }
    if (cnt > 0) __syncthreads();
    // the cotangent of max(x, y) that x takes, by the magnitudes' bits: all, half at
    // a tie, none
    auto share = [](double g, unsigned long long x, unsigned long long y) {
        const int h = __double2hiint(g);
        const int half = (h & 0x7ff00000) > 0x00100000 ? h - 0x00100000 : 0;
        return __hiloint2double(x > y ? h : (x == y ? half : 0), x >= y ? __double2loint(g) : 0);
    };
    for (int i = lo + tid; i < hi; i += nt) {
        double s = 0.0;
        bool all = cnt > 0;
        if (cnt > 0) {
            const bool f0 = flag[i - 2], f1 = flag[i - 1], f2 = flag[i], f3 = flag[i + 1], f4 = flag[i + 2];
            all = f0 && f1 && f2 && f3 && f4;
            double t = f4 ? a.T0[i + 2] : 0.0;
            if (f3) t += a.T1[i + 1];
            if (f2) t += a.T2[i];
            if (f1) t += a.T3[i - 1];
            if (f0) t += a.T4[i - 2];
            s = 10.0 * t;
        }
        if (!all) {
            // ideal weights: taps (2, -13, 47, 27, -3) of the right face values, mirrored
            // of the left ones
            s = fma(2.0, a.GR[i + 2] + a.GL[i - 3], s);
            s = fma(47.0, a.GR[i] + a.GL[i - 1], s);
            s = fma(-13.0, a.GR[i + 1] + a.GL[i - 2], s);
            s = fma(27.0, a.GR[i - 1] + a.GL[i], s);
            s = fma(-3.0, a.GR[i - 2] + a.GL[i + 1], s);
            s = fma(10.0, a.H[i], s);
        }
        // wave speed terms of the two faces, 60 GA d max(|v_i|, |v_i+-1|) / dv_i
        // (compared, halved and signed on the integer pipe)
        const double vi = v[i];
        const auto bi = abs_bits(vi), bm = abs_bits(v[i - 1]), bp = abs_bits(v[i + 1]);
        const double q = share(a.GA[i - 1], bi, bm) + share(a.GA[i], bi, bp);
        const int sgn60 = bi == 0 ? 0 : 0x404e0000 | (__double2hiint(vi) & static_cast<int>(0x80000000u));
        s = fma(__hiloint2double(sgn60, 0), q, s);
        z[i] = s;
    }
    __syncthreads();
}

// Stage storage of one replayed step: k1, k2 (learned or float steps, in
// float), plus the face values of u and k1 (double WENO-JS5 steps, in double),
// each an array of the plan's `total` cells.
template <class T, int REC>
__host__ __device__ constexpr int kStageArrays() {
    return (sizeof(T) == 8 && REC != SHK_REC_LEARNED) ? 8 : 2;
}
template <class T, int REC>
__device__ __forceinline__ StageOut<stage_t<T, REC>> stage_out(void* base, int64_t total,
                                                               int64_t at) {
    using S = stage_t<T, REC>;
    StageOut<S> so;
    if (!base) return so;
    const Win<S> b = make_win(static_cast<S*>(base), kStageArrays<T, REC>() * total) + at;
    so.k1 = b;
    so.k2 = b + total;
    if constexpr (kStageArrays<T, REC>() == 8) {
        so.ulu = b + 2 * total;
        so.uru = b + 3 * total;
        so.ul1 = b + 4 * total;
        so.ur1 = b + 5 * total;
        so.ul2 = b + 6 * total;
        so.ur2 = b + 7 * total;
    }
    return so;
}

template <class S>
__device__ __forceinline__ StageOut<const S> as_const(const StageOut<S>& so) {
    StageOut<const S> c;
    c.k1 = so.k1; c.k2 = so.k2; c.ulu = so.ulu; c.uru = so.uru; c.ul1 = so.ul1; c.ur1 = so.ur1;
    c.ul2 = so.ul2; c.ur2 = so.ur2;
    return c;
}

// window positions [lo, hi) of a stage array stored per instance cell
// (position i is cell g0 + i, periodically)
template <class PD, class PS>
__device__ __forceinline__ void load_stage(PD dst, PS src, int64_t n, int64_t g0,
                                           int lo, int hi) {
    const bool once = g0 + lo >= -n && g0 + hi <= 2 * n;
    for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        const int64_t pos = g0 + i;
        dst[i] = src[once ? (pos < 0 ? pos + n : (pos >= n ? pos - n : pos)) : imod(pos, n)];
    }
}

// Adjoint step of the mixed-precision learned step (step_tile_mixed): the
// forward stages are recomputed exactly as that step computes them (float
// operator on float stage states, increments about u), the three reverse
// stages run in float on float copies of u and p, and the result
//   ub = p + 2/3 Z3 + 1/4 Z2 + Z1
// (Z_s the stage VJPs dt J^T(.) of the reverse sweep below) adds the float
// increment to the double p once. Of the double arrays only the loaded windows
// a.U and a.PB are read; af holds the float arrays (af.K1, af.K2 may overlay
// a.U, which is dead once af.U is written).
// st (optional): the instance's stored float stage states (replay with stage
// storage), which replace the recompute of k1 and k2 bit for bit.
template <int EQ>
__device__ void adjoint_tile_mixed(const AdjSmem<double>& a, const AdjSmem<float>& af, Win<double> gout,
                                   int te, double dtdx, const OpParams<double>& p,
                                   const BcView& bc = BcView(), int64_t g0 = 0, int64_t n = 0,
                                   const StageOut<const float>& st = StageOut<const float>()) {
    constexpr int HU = adj_uhalo<double>(), HP = adj_phalo<double>();
    constexpr int REC = SHK_REC_LEARNED;
    const int tid = threadIdx.x, nt = blockDim.x;
    const bool np = !bc.periodic();
    const OpParams<float> pf = float_params(p);
    const float dtf = static_cast<float>(dtdx);
    for (int i = tid; i < te + 2 * HU; i += nt) af.U[i] = static_cast<float>(a.U[i]);
    for (int i = HU - HP + tid; i < HU + te + HP; i += nt) af.PB[i] = static_cast<float>(a.PB[i]);
    __syncthreads();
    if (np) {
        apply_bc(af.U, g0, n, 0, te + 2 * HU, bc, 0);
        zero_outside(af.PB, g0, n, HU - HP, HU + te + HP);
    }
    // forward recompute: k1 on [HU-15, HU+te+15), k2 on [HU-12, HU+te+12), or
    // the stored stage states there
    if (st.k1) {
        load_stage(af.K1, st.k1, n, g0, HU - 15, HU + te + 15);
        load_stage(af.K2, st.k2, n, g0, HU - 12, HU + te + 12);
        __syncthreads();
        if (np) {
            apply_bc(af.K1, g0, n, HU - 15, HU + te + 15, bc, 1);
            apply_bc(af.K2, g0, n, HU - 12, HU + te + 12, bc, 2);
        }
    } else {
        {
            const int lo = HU - 15, hi = HU + te + 15;
            face_fluxes<float, EQ, REC, SHK_FLUX_RUSANOV>(af.U, lo, hi, af.fwd(af.K1), pf);
            for (int i = lo + tid; i < hi; i += nt) {
                const float d = dtf * (af.D[i - 1] - af.D[i]);
                af.T0[i] = d;
                af.K1[i] = af.U[i] + d;
            }
            __syncthreads();
            if (np) apply_bc(af.K1, g0, n, lo, hi, bc, 1);
        }
        {
            const int lo = HU - 12, hi = HU + te + 12;
            face_fluxes<float, EQ, REC, SHK_FLUX_RUSANOV>(af.K1, lo, hi, af.fwd(af.K2), pf);
            for (int i = lo + tid; i < hi; i += nt) {
                const float d = 0.25f * (af.T0[i] + dtf * (af.D[i - 1] - af.D[i]));
                af.K2[i] = af.U[i] + d;
            }
            __syncthreads();
            if (np) apply_bc(af.K2, g0, n, lo, hi, bc, 2);
        }
    }
    // reverse stage 3: k2b = 2/3 (p + Z3), Z3 = dt J(k2)^T p
    {
        const int lo = HU - 6, hi = HU + te + 6;
        vjp_stage<float, EQ, REC>(af.K2, af.PB, af.Z, lo, hi, af, pf, dtf);
        if (np) bc_transpose(af.Z, g0, n, lo, hi, bc);
        for (int i = lo + tid; i < hi; i += nt) af.CB[i] = (2.0f / 3.0f) * (af.PB[i] + af.Z[i]);
        for (int i = HU + tid; i < HU + te; i += nt) af.ACC[i] = (2.0f / 3.0f) * af.Z[i];
        __syncthreads();
    }
    // reverse stage 2: k1b = 1/4 (k2b + Z2), Z2 = dt J(k1)^T k2b
    {
        const int lo = HU - 3, hi = HU + te + 3;
        vjp_stage<float, EQ, REC>(af.K1, af.CB, af.Z, lo, hi, af, pf, dtf);
        if (np) bc_transpose(af.Z, g0, n, lo, hi, bc);
        for (int i = HU + tid; i < HU + te; i += nt) af.ACC[i] = fmaf(0.25f, af.Z[i], af.ACC[i]);
        for (int i = lo + tid; i < hi; i += nt) af.CB[i] = 0.25f * (af.CB[i] + af.Z[i]);
        __syncthreads();
    }
    // reverse stage 1: Z1 = dt J(u)^T k1b; ub = p + (2/3 Z3 + 1/4 Z2 + Z1)
    // (and on the ghosts of a boundary tile)
    {
        int lo = HU, hi = HU + te;
        if (np) {
            for (int i = tid; i < 3; i += nt) {  // k1b beyond its range: zero
                af.CB[HU - 6 + i] = 0.0f;
                af.CB[HU + te + 3 + i] = 0.0f;
            }
            __syncthreads();
            if (g0 + HU == 0) lo -= 3;
            if (g0 + HU + te == n) hi += 3;
        }
        vjp_stage<float, EQ, REC>(af.U, af.CB, af.Z, lo, hi, af, pf, dtf);
        if (np) bc_transpose(af.Z, g0, n, lo, hi, bc);
        for (int i = HU + tid; i < HU + te; i += nt)
            gout[i - HU] = a.PB[i] + static_cast<double>(af.ACC[i] + af.Z[i]);
    }
}

// one adjoint step of a tile: p_out[s, s+te) from u_m (window, halo 20) and
// p_next (window, halo 10/12). gout points at p_out + s.
// With a Dirichlet / Neumann boundary (bc; g0 = s - HU the global cell of
// window position 0, n the instance's cells) the forward recompute applies the
// boundary at each stage, the cotangent window is zeroed outside the instance,
// each reverse stage is followed by the boundary's transpose, and the first
// reverse stage of a boundary tile also covers the ghost cells (their
// cotangents reach the interior through the Neumann mirrors).
template <class T, int EQ, int REC, int FLUX>
__device__ void adjoint_tile(const AdjSmem<T>& a, Win<T> gout, int te, T dtdx, const OpParams<T>& p,
                             const BcView& bc = BcView(), int64_t g0 = 0, int64_t n = 0,
                             const StageOut<const stage_t<T, REC>>& st =
                                 StageOut<const stage_t<T, REC>>()) {
    if constexpr (sizeof(T) == 8 && REC == SHK_REC_LEARNED) {
        // full double layout: the float arrays fit from CB on (24 in 20 double ones)
        AdjSmem<float> af;
        af.carve(reinterpret_cast<unsigned char*>(win_raw(a.CB)), a.W);
        adjoint_tile_mixed<EQ>(a, af, gout, te, dtdx, p, bc, g0, n, st);
        return;
    }
    const bool np = !bc.periodic();
    // stored stage states (and, for WENO-JS5, face values) replace the forward
    // recompute bit for bit; the stored faces of a boundary instance lack its
    // ghost cells, so WENO-JS5 steps with a boundary recompute
    constexpr bool kStoreable = (sizeof(T) == 4 && REC == SHK_REC_LEARNED) ||
                                (sizeof(T) == 8 && REC == SHK_REC_WENOJS53);
    const bool stored = kStoreable && st.k1 && (REC == SHK_REC_LEARNED || !np);
    if (np) {
        constexpr int HU0 = adj_uhalo<T>(), HP0 = adj_phalo<T>();
        apply_bc(a.U, g0, n, 0, te + 2 * HU0, bc, 0);
        zero_outside(a.PB, g0, n, HU0 - HP0, HU0 + te + HP0);
    }
    constexpr int HU = adj_uhalo<T>();
    // the forward recompute's face values of u, k1 and k2 serve the reverse
    // stages (they cover [HU-16, HU+te+16), [HU-13, HU+te+13) and
    // [HU-9, HU+te+9); the stages read [HU-6, HU+te+6), k2's [HU-9, HU+te+9))
    constexpr bool kCache = REC == SHK_REC_WENOJS53;
    const int tid = threadIdx.x, nt = blockDim.x;
    const T fdt = dtdx * p.fscale;  // face fluxes are stored as F / fscale
    // forward recompute: k1 on [HU-15, HU+te+15), k2 on [HU-12, HU+te+12),
    // with the forward step's own formulas (increments about u for float)
    if constexpr (kStoreable) {
        if (stored) {
            load_stage(a.K1, st.k1, n, g0, HU - 15, HU + te + 15);
            load_stage(a.K2, st.k2, n, g0, HU - 12, HU + te + 12);
            if constexpr (kCache) {
                load_stage(a.CLu, st.ulu, n, g0, HU - 6, HU + te + 6);
                load_stage(a.CRu, st.uru, n, g0, HU - 6, HU + te + 6);
                load_stage(a.CL1, st.ul1, n, g0, HU - 6, HU + te + 6);
                load_stage(a.CR1, st.ur1, n, g0, HU - 6, HU + te + 6);
                // k2's face values in UL/UR (free: no reconstruction runs here)
                load_stage(a.UL, st.ul2, n, g0, HU - 9, HU + te + 9);
                load_stage(a.UR, st.ur2, n, g0, HU - 9, HU + te + 9);
            }
            __syncthreads();
            if (np) {
                apply_bc(a.K1, g0, n, HU - 15, HU + te + 15, bc, 1);
                apply_bc(a.K2, g0, n, HU - 12, HU + te + 12, bc, 2);
            }
        }
    }
    if (!stored) {
    if constexpr (FLUX == kFluxRusanovFx) {
        // the stages of step_tile_fx on this window (T1: the listed faces)
        Smem<T> f = a.fwd(a.K1);
        f.fx = win_cast<int>(a.T1);
        if (tid < kFxCounters) f.fx[tid] = 0;
        __syncthreads();
        const T c = dtdx * (1.0 / 288.0);
        {
            const int lo = HU - 15, hi = HU + te + 15;
            fx_fluxes(a.U, lo - 1, hi, f, p, 0, StoreFaces<Win<T>>{a.CLu, a.CRu, HU - 6, HU + te + 6, 0});
            for (int i = lo + tid; i < hi; i += nt) a.K1[i] = fma(c, a.D[i - 1] - a.D[i], a.U[i]);
            __syncthreads();
            if (np) apply_bc(a.K1, g0, n, lo, hi, bc, 1);
        }
        {
            const int lo = HU - 12, hi = HU + te + 12;
            fx_fluxes(a.K1, lo - 1, hi, f, p, 1, StoreFaces<Win<T>>{a.CL1, a.CR1, HU - 6, HU + te + 6, 0});
            for (int i = lo + tid; i < hi; i += nt) {
                const T k = fma(c, a.D[i - 1] - a.D[i], a.K1[i]);
                a.K2[i] = fma(1.0 / 4.0, k, (3.0 / 4.0) * a.U[i]);
            }
            __syncthreads();
            if (np) apply_bc(a.K2, g0, n, lo, hi, bc, 2);
        }
        fx_fluxes(a.K2, HU - 10, HU + te + 9, f, p, 2, StoreFaces<Win<T>>{a.UL, a.UR, HU - 9, HU + te + 9, 0});
    } else {
    {
        const int lo = HU - 15, hi = HU + te + 15;
        // WENO-JS5: the face values of u stay in CLu/CRu for reverse stage 1
        face_fluxes<T, EQ, REC, SHK_FLUX_RUSANOV>(a.U, lo, hi, kCache ? a.fwd(a.K1, a.CLu, a.CRu)
                                                                      : a.fwd(a.K1), p);
        for (int i = lo + tid; i < hi; i += nt) {
            if constexpr (sizeof(T) == 4) {
                const T d = fdt * (a.D[i - 1] - a.D[i]);
                a.T0[i] = d;
                a.K1[i] = a.U[i] + d;
            } else {
                a.K1[i] = fma(fdt, a.D[i - 1] - a.D[i], a.U[i]);
            }
        }
        __syncthreads();
        if (np) apply_bc(a.K1, g0, n, lo, hi, bc, 1);
    }
    {
        const int lo = HU - 12, hi = HU + te + 12;
        // and those of k1 in CL1/CR1 for reverse stage 2
        face_fluxes<T, EQ, REC, SHK_FLUX_RUSANOV>(a.K1, lo, hi, kCache ? a.fwd(a.K2, a.CL1, a.CR1)
                                                                       : a.fwd(a.K2), p);
        for (int i = lo + tid; i < hi; i += nt) {
            if constexpr (sizeof(T) == 4) {
                a.K2[i] = a.U[i] + T(0.25) * (a.T0[i] + fdt * (a.D[i - 1] - a.D[i]));
            } else {
                const T k = fma(fdt, a.D[i - 1] - a.D[i], a.K1[i]);
                a.K2[i] = fma(T(1.0 / 4.0), k, T(3.0 / 4.0) * a.U[i]);
            }
        }
        __syncthreads();
        if (np) apply_bc(a.K2, g0, n, lo, hi, bc, 2);
    }
    if constexpr (kCache) {
        // the face values of k2 on [HU-9, HU+te+9) as the forward's face pass
        // forms them (as the stored ones; the fluxes it also leaves in D are
        // not used)
        face_fluxes<T, EQ, REC, SHK_FLUX_RUSANOV>(a.K2, HU - 8, HU + te + 8, a.fwd(a.K2, a.UL, a.UR), p);
    }
    }
    }
    auto vjp = [&](auto v, auto w, auto z, int lo, int hi, const AdjSmem<T>& a_, const OpParams<T>& p_, T dtdx_,
                   Win<T> ul, Win<T> ur) {
        if constexpr (FLUX == kFluxRusanovFx) fx_vjp_stage(v, w, z, lo, hi, a_, p_, dtdx_, ul, ur);
        else vjp_stage<T, EQ, REC>(v, w, z, lo, hi, a_, p_, dtdx_, ul, ur);
    };
    // reverse stage 3: k2b = 2/3 (p + dt J(k2)^T p) on [HU-6, HU+te+6)
    {
        const int lo = HU - 6, hi = HU + te + 6;
        vjp(a.K2, a.PB, a.Z, lo, hi, a, p, dtdx, kCache ? a.UL : Win<T>(),
                              kCache ? a.UR : Win<T>());
        if (np) bc_transpose(a.Z, g0, n, lo, hi, bc);
        for (int i = lo + tid; i < hi; i += nt) a.CB[i] = T(2.0 / 3.0) * (a.PB[i] + a.Z[i]);
        __syncthreads();
        for (int i = HU + tid; i < HU + te; i += nt)
            a.ACC[i] = fma(T(3.0 / 4.0), a.CB[i], T(1.0 / 3.0) * a.PB[i]);
        __syncthreads();
    }
    // reverse stage 2: k1b = 1/4 (k2b + dt J(k1)^T k2b) on [HU-3, HU+te+3)
    {
        const int lo = HU - 3, hi = HU + te + 3;
        vjp(a.K1, a.CB, a.Z, lo, hi, a, p, dtdx, kCache ? a.CL1 : Win<T>(),
                              kCache ? a.CR1 : Win<T>());
        if (np) bc_transpose(a.Z, g0, n, lo, hi, bc);
        for (int i = lo + tid; i < hi; i += nt) a.CB[i] = T(1.0 / 4.0) * (a.CB[i] + a.Z[i]);
        __syncthreads();
    }
    // reverse stage 1: ub = 1/3 p + 3/4 k2b + k1b + dt J(u)^T k1b on the tile
    // (and on the ghosts of a boundary tile)
    {
        int lo = HU, hi = HU + te;
        if (np) {
            for (int i = tid; i < 3; i += nt) {  // k1b beyond its range: zero
                a.CB[HU - 6 + i] = T(0);
                a.CB[HU + te + 3 + i] = T(0);
            }
            __syncthreads();
            if (g0 + HU == 0) lo -= 3;
            if (g0 + HU + te == n) hi += 3;
        }
        vjp(a.U, a.CB, a.Z, lo, hi, a, p, dtdx, kCache ? a.CLu : Win<T>(),
                              kCache ? a.CRu : Win<T>());
        if (np) bc_transpose(a.Z, g0, n, lo, hi, bc);
        for (int i = HU + tid; i < HU + te; i += nt) gout[i - HU] = a.ACC[i] + (a.CB[i] + a.Z[i]);
    }
}

// compact layout of the mixed-precision learned adjoint (22 float arrays of W):
// a.U (double, slots 0-1, dead after the float copy, then af.K1/af.K2),
// a.PB (double, slots 2-3), af.U, af.PB, then the other 16 float arrays
constexpr int kMixedAdjSlots = 22;
__device__ inline void carve_mixed(unsigned char* base, int W, AdjSmem<double>& a, AdjSmem<float>& af) {
    float* f = reinterpret_cast<float*>(base);
    a.U = win_cast<double>(make_win(f, 2 * W));
    a.PB = win_cast<double>(make_win(f + 2 * W, 2 * W));
    a.K1 = a.K2 = a.CB = a.Z = a.ACC = a.H = a.D = a.Q = a.UL = a.UR = Win<double>();
    a.GL = a.GR = a.GA = a.T0 = a.T1 = a.T2 = a.T3 = a.T4 = Win<double>();
    a.W = W;
    af.K1 = make_win(f, W);
    af.K2 = make_win(f + W, W);
    af.U = make_win(f + 4 * W, W);
    af.PB = make_win(f + 5 * W, W);
    Win<float>* rest[] = {&af.CB, &af.Z, &af.ACC, &af.H, &af.D, &af.Q, &af.UL, &af.UR,
                          &af.GL, &af.GR, &af.GA, &af.T0, &af.T1, &af.T2, &af.T3, &af.T4};
    for (int i = 0; i < 16; ++i) *rest[i] = make_win(f + (6 + i) * W, W);
    af.W = W;
}

template <class T>
__device__ __forceinline__ bool adjoint_load(const AdjSmem<T>& a, const T* um, const T* pn,
                                             int64_t n, int64_t s0, int te, uint64_t* bar,
                                             uint32_t& phase) {
    constexpr int HU = adj_uhalo<T>(), HP = adj_phalo<T>();
    if (!load_window<T>(a.U, um, n, s0 - HU, te + 2 * HU, bar, phase)) return false;
    return load_window<T>(a.PB + (HU - HP), pn, n, s0 - HP, te + 2 * HP, bar, phase);
}

template <class T, int EQ, int REC, int FLUX>
__global__ void __launch_bounds__(kThreads, REC == SHK_REC_LEARNED || FLUX == kFluxRusanovFx ? 2 : 1) batched_adjoint_kernel(PlanDev P, const T* __restrict__ um,
                                                                   const T* __restrict__ pnext,
                                                                   T* __restrict__ pout,
                                                                   const double* __restrict__ dt_row,
                                                                   OpParams<T> p,
                                                                   const void* stages,
                                                                   int64_t total, int64_t step) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    constexpr bool kMixed = sizeof(T) == 8 && REC == SHK_REC_LEARNED;
    AdjSmem<T> a;
    AdjSmem<float> af;
    if constexpr (kMixed) carve_mixed(smem_raw, P.tile + 2 * adj_uhalo<T>(), a, af);
    else a.carve(smem_raw, P.tile + 2 * adj_uhalo<T>());
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    learned_stage<REC, true>(p.lp);
    uint32_t phase = 0;
    const Win<const T> gpnext = make_win(pnext, total);
    const Win<T> gpout = make_win(pout, total);
    __shared__ int s_item[2];
    for (ItemQueue<REC != SHK_REC_LEARNED> items(P, 2, s_item); items.more(); items.end()) {
        const PlanItem it = items.begin();
        const int b = it.b, te = it.te;
        const int64_t off = it.off, n = it.n, s0 = int64_t(it.tile) * P.tile;
        const double dt = dt_row[b];
        if (dt == 0.0) {  // no step was taken: identity
            for (int i = threadIdx.x; i < te; i += blockDim.x) gpout[off + s0 + i] = gpnext[off + s0 + i];
            continue;
        }
        if (!adjoint_load<T>(a, um + off, pnext + off, n, s0, te, &bar, phase)) {
            if (threadIdx.x == 0) atomicOr(P.status, ERR_TIMEOUT);
            break;
        }
        const T dtdx = static_cast<T>(dt * P.inv_dx[b]);
        const BcView bc = plan_bc(P, b, step);
        const int64_t g0 = s0 - adj_uhalo<T>();
        const StageOut<const stage_t<T, REC>> st =
            as_const(stage_out<T, REC>(const_cast<void*>(stages), total, off));
        if constexpr (kMixed) adjoint_tile_mixed<EQ>(a, af, gpout + (off + s0), te, dtdx, p, bc, g0, n, st);
        else adjoint_tile<T, EQ, REC, FLUX>(a, gpout + (off + s0), te, dtdx, p, bc, g0, n, st);
        __syncthreads();
    }
    finish_items(P, 2);
}

// The reverse step of a periodic instance of a fixed_flux_scheme plan from the
// replay's stored stages, bound by latency (FP64 pipe 52 % busy, 40 % of the issue
// slots; loads, shared memory and barriers are the top stalls; 240 B of spills at the 80
// registers of three CTAs): one loop over the reverse stages, each loading its own
// state and face values, in 13 windows (batched_adjoint_kernel keeps 24, for its
// recompute) so that three CTAs fit an SM. UL/UR hold T0/T1 once the seeds are
// formed; the cotangent is updated in place; Z overwrites the pair part. 96
// instances, 0.4 M cells: 471 us per reverse step with the FP64 backward, 202 with
// the float pairs in 24 windows (two CTAs), 147 here, about 139 since the listed cells
// have a backward of their own.
constexpr int kAdjFxArrays = 13;
constexpr int kAdjFxThreads = 256, kAdjFxCtas = 3;
__device__ __forceinline__ void carve_adjoint_fx(AdjSmem<double>& a, unsigned char* base, int W) {
    double* p = reinterpret_cast<double*>(base);
    Win<double>* slots[kAdjFxArrays] = {&a.U, &a.UL, &a.UR, &a.CB, &a.ACC, &a.GL, &a.GR,
                                        &a.GA, &a.H, &a.D, &a.T2, &a.T3, &a.T4};
    for (int i = 0; i < kAdjFxArrays; ++i) *slots[i] = make_win(p + size_t(i) * W, W);
    a.T0 = a.UL;
    a.T1 = a.UR;
    a.Z = a.H;
    // the list and the flags share one window: W ints each
    Win<double> d = a.D;
    a.Q = make_win(win_raw(d) + W / 2, W / 2);
    a.D = make_win(win_raw(d), W / 2);
    a.W = W;
}
__global__ void __launch_bounds__(kAdjFxThreads, kAdjFxCtas) batched_adjoint_fx_kernel(PlanDev P, const double* __restrict__ um,
                                                                         const double* __restrict__ pnext,
                                                                         double* __restrict__ pout,
                                                                         const double* __restrict__ dt_row,
                                                                         OpParams<double> p, const void* stages,
                                                                         int64_t total) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int HU = adj_uhalo<double>();
    AdjSmem<double> a;
    carve_adjoint_fx(a, smem_raw, P.tile + 2 * HU);
    const Win<const double> gum = make_win(um, total), gpnext = make_win(pnext, total);
    const Win<double> gpout = make_win(pout, total);
    __shared__ int s_item[2];
    for (ItemQueue<> items(P, 2, s_item); items.more(); items.end()) {
        const PlanItem it = items.begin();
        const int b = it.b, te = it.te;
        const int64_t off = it.off, n = it.n, s0 = int64_t(it.tile) * P.tile;
        const double dt = dt_row[b];
        if (dt == 0.0) {  // no step was taken: identity
            for (int i = threadIdx.x; i < te; i += blockDim.x) gpout[off + s0 + i] = gpnext[off + s0 + i];
            continue;
        }
        const double dtdx = dt * P.inv_dx[b];
        const int64_t g0 = s0 - HU;
        const StageOut<const double> st =
            as_const(stage_out<double, SHK_REC_WENOJS53>(const_cast<void*>(stages), total, off));
        load_stage(a.CB, gpnext + off, n, g0, HU - 9, HU + te + 9);
#pragma unroll 1
        for (int s = 2; s >= 0; --s) {
            // z on [lo, hi) from the state on 6 and the face values on 3 cells more
            const int lo = HU - 3 * s, hi = HU + te + 3 * s;
            load_stage(a.U, s == 2 ? st.k2 : (s == 1 ? st.k1 : gum + off), n, g0, lo - 6, hi + 6);
            load_stage(a.UL, s == 2 ? st.ul2 : (s == 1 ? st.ul1 : st.ulu), n, g0, lo - 3, hi + 3);
            load_stage(a.UR, s == 2 ? st.ur2 : (s == 1 ? st.ur1 : st.uru), n, g0, lo - 3, hi + 3);
            __syncthreads();
            fx_vjp_stage(a.U, a.CB, a.Z, lo, hi, a, p, dtdx, a.UL, a.UR);
            for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
                const double q = a.CB[i], z = a.Z[i];
                if (s == 2) {
                    // k2b = 2/3 (p + Z), acc = 3/4 k2b + 1/3 p
                    const double k = (2.0 / 3.0) * (q + z);
                    a.CB[i] = k;
                    a.ACC[i] = fma(3.0 / 4.0, k, (1.0 / 3.0) * q);
                } else if (s == 1) {
                    a.CB[i] = (1.0 / 4.0) * (q + z);
                } else {
                    gpout[off + s0 + i - HU] = a.ACC[i] + (q + z);
                }
            }
            __syncthreads();
        }
    }
    finish_items(P, 2);
}

// forward step with a recorded dt (no CFL, no time update): recompute of the
// states between checkpoints
// stages (optional): the step's stage storage, kStageArrays<T, REC> arrays of
// P's cells in the stage precision (stage_arrays), for a reverse step that
// skips its forward recompute; uout may then be null.
template <class T, int EQ, int REC, int FLUX>
__global__ void __launch_bounds__(flux_threads<FLUX>(), REC == SHK_REC_LEARNED ? 3 : (FLUX == kFluxRusanovFx ? 6 : 1)) replay_step_kernel(PlanDev P, const T* __restrict__ uin,
                                                               T* __restrict__ uout,
                                                               const double* __restrict__ dt_row,
                                                               OpParams<T> p, void* stages,
                                                               int64_t total, int64_t step) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    constexpr int HL = step_halo<T>();
    Smem<T> sm;
    carve_step<T, REC, FLUX>(sm, smem_raw, P.tile + 2 * HL);
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    learned_stage<REC>(p.lp);
    uint32_t phase = 0;
    const Win<const T> guin = make_win(uin, total);
    const Win<T> guout = make_win(uout, total);
    __shared__ int s_item[2];
    for (ItemQueue<REC != SHK_REC_LEARNED> items(P, 4, s_item); items.more(); items.end()) {
        const PlanItem it = items.begin();
        const int b = it.b, te = it.te;
        const int64_t off = it.off, n = it.n, s0 = int64_t(it.tile) * P.tile;
        const double dt = dt_row[b];
        if (dt == 0.0) {  // no step: the reverse step is the identity, stage states unused
            if (uout)
                for (int i = threadIdx.x; i < te; i += blockDim.x) guout[off + s0 + i] = guin[off + s0 + i];
            continue;
        }
        if (!load_window<T>(sm.U, uin + off, n, s0 - HL, te + 2 * HL, &bar, phase)) {
            if (threadIdx.x == 0) atomicOr(P.status, ERR_TIMEOUT);
            break;
        }
        const T dtdx = static_cast<T>(dt * P.inv_dx[b]);
        step_tile<T, EQ, REC, FLUX>(sm, uout ? guout + (off + s0) : Win<T>(), te, dtdx, p,
                                                plan_bc(P, b, step), s0 - HL, n,
                                                stage_out<T, REC>(stages, total, off + s0));
        __syncthreads();
    }
    finish_items(P, 4);
}

// single instance on the reference's ghosted layout (drop-in adjoint_step)
template <class T, int EQ, int FLUX>
__global__ void __launch_bounds__(kThreads) single_vjp_kernel(const T* __restrict__ u, const T* __restrict__ pn,
                                                              T* __restrict__ pout, int64_t n, int g,
                                                              int tile, T dtdx, OpParams<T> p,
                                                              int32_t* err, shk_boundary bcp, double dx) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    AdjSmem<T> a;
    a.carve(smem_raw, tile + 2 * adj_uhalo<T>());
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    uint32_t phase = 0;
    const int64_t s0 = int64_t(blockIdx.x) * tile;
    const int te = static_cast<int>(imin64(tile, n - s0));
    if (!adjoint_load<T>(a, u + g, pn + g, n, s0, te, &bar, phase)) {
        if (threadIdx.x == 0 && err) atomicOr(err, ERR_TIMEOUT);
        return;
    }
    BcView bc;
    bc.left = bcp.left;
    bc.right = bcp.right;
    bc.dir = &bcp.dirichlet[0][0][0];
    bc.dir_ss = 6;
    bc.neu = &bcp.neumann[0][0];
    bc.neu_ss = 2;
    bc.dx = dx;
    const Win<T> gpout = make_win(pout, n + 2 * g);
    adjoint_tile<T, EQ, SHK_REC_WENOJS53, FLUX>(a, gpout + (g + s0), te, dtdx, p, bc, s0 - adj_uhalo<T>(), n);
    // ghost cotangents are zero (interior-only adjoint)
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < g; i += blockDim.x) {
            gpout[i] = T(0);
            gpout[g + n + i] = T(0);
        }
}

}  // namespace shk

// ===========================================================================
// host side
// ===========================================================================
using namespace shk;

namespace {

int acuda(cudaError_t e) {
    if (e != cudaSuccess) {
        std::fprintf(stderr, "libshocks: CUDA error %s\n", cudaGetErrorString(e));
        return SHK_ECUDA;
    }
    return SHK_OK;
}
#define ADJ_CUDA(call)                          \
    do {                                        \
        int _st = acuda(call);                  \
        if (_st != SHK_OK) return _st;          \
    } while (0)

template <class T>
OpParams<T> adj_params(const shk_scheme* s) {
    OpParams<T> p;
    p.eps = static_cast<T>(s->eps);
    p.delta = static_cast<T>(s->delta);
    p.hnu = static_cast<T>(0.5 * s->nu);
    p.c = static_cast<T>(s->speed);
    p.hnu_amax = T(0);
    p.lp = LearnedParams{s->mlp, static_cast<float>(s->eps), s->tau, s->band, s->dev,
                         norm_floor(s->norm_eps)};
    p.fscale = (sizeof(T) == 8 && s->flux == SHK_FLUX_RUSANOV && s->rec == SHK_REC_WENOJS53 &&
                s->equation == SHK_EQ_BURGERS && s->nu == 1.0) ? T(0.25) : T(1);
    p.lim = s->limiter;
    p.lim_param = static_cast<T>(s->delta);
    p.atol = static_cast<T>(s->eps);
    p.dx = T(1);
    p.e4h = static_cast<float>(4.0 * s->eps);
    p.e4l = static_cast<float>(4.0 * s->eps - static_cast<double>(p.e4h));
    return p;
}

bool adjoint_supported(const shk_scheme* s) {
    return s && s->flux == SHK_FLUX_RUSANOV &&
           (s->rec == SHK_REC_WENOJS53 || (s->rec == SHK_REC_LEARNED && s->mlp)) &&
           s->equation >= 0 && s->equation <= SHK_EQ_LWR;
}

template <class T, int REC, class F>
int by_equation_rec(int eq, F&& f) {
    switch (eq) {
        case SHK_EQ_BURGERS: return f.template operator()<T, SHK_EQ_BURGERS, REC>();
        case SHK_EQ_ADVECTION: return f.template operator()<T, SHK_EQ_ADVECTION, REC>();
        case SHK_EQ_LWR: return f.template operator()<T, SHK_EQ_LWR, REC>();
    }
    return SHK_EINVAL;
}

// WENO-JS53 for both precisions, the learned reconstruction for float32 states
template <class T, class F>
int by_scheme(const shk_scheme& sch, F&& f) {
    if (sch.rec == SHK_REC_LEARNED) return by_equation_rec<T, SHK_REC_LEARNED>(sch.equation, f);
    return by_equation_rec<T, SHK_REC_WENOJS53>(sch.equation, f);
}

template <class T, class F>
int by_equation(int eq, F&& f) {
    return by_equation_rec<T, SHK_REC_WENOJS53>(eq, f);
}

// instances with a kFluxRusanovFx form (used for the schemes of fixed_flux_scheme)
template <class T, int EQ, int REC>
constexpr bool kHasFixed = sizeof(T) == 8 && EQ == SHK_EQ_BURGERS && REC == SHK_REC_WENOJS53;

template <class TS>
struct AdjLaunch {
    PlanDev D; const void* um; const void* pn; void* po; const double* dt_row; OpParams<TS> p;
    size_t smem; int grid; cudaStream_t st; const void* stages = nullptr; int64_t total = 0;
    int64_t step = 0;  // index of the forward step (its boundary data)
    bool fixed = false;
    template <class T, int EQ, int REC> int operator()() {
        auto k = batched_adjoint_kernel<T, EQ, REC, SHK_FLUX_RUSANOV>;
        if constexpr (kHasFixed<T, EQ, REC>)
            if (fixed) k = batched_adjoint_kernel<T, EQ, REC, kFluxRusanovFx>;
        ADJ_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k<<<grid, kThreads, smem, st>>>(D, static_cast<const T*>(um), static_cast<const T*>(pn),
                                         static_cast<T*>(po), dt_row, p, stages, total, step);
        return acuda(cudaGetLastError());
    }
};

template <class TS>
struct ReplayLaunch {
    PlanDev D; const void* uin; void* uout; const double* dt_row; OpParams<TS> p;
    size_t smem; int grid; cudaStream_t st; void* stages = nullptr; int64_t total = 0;
    int64_t step = 0;  // index of the replayed step (its boundary data)
    bool fixed = false;
    template <class T, int EQ, int REC> int operator()() {
        auto k = replay_step_kernel<T, EQ, REC, SHK_FLUX_RUSANOV>;
        if constexpr (kHasFixed<T, EQ, REC>)
            if (fixed) k = replay_step_kernel<T, EQ, REC, kFluxRusanovFx>;
        ADJ_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        const int threads = kHasFixed<T, EQ, REC> && fixed ? kFxThreads : kThreads;
        k<<<grid, threads, smem, st>>>(D, static_cast<const T*>(uin), static_cast<T*>(uout), dt_row, p,
                                         stages, total, step);
        return acuda(cudaGetLastError());
    }
};

struct SingleVjpLaunch {
    const double* u; const double* pn; double* po; int64_t n; int g; int tile; double dtdx;
    OpParams<double> p; size_t smem; int blocks; cudaStream_t st; shk_boundary bc; double dx;
    bool fixed = false;
    template <class T, int EQ, int REC> int operator()() {
        auto k = single_vjp_kernel<T, EQ, SHK_FLUX_RUSANOV>;
        if constexpr (kHasFixed<T, EQ, REC>)
            if (fixed) k = single_vjp_kernel<T, EQ, kFluxRusanovFx>;
        ADJ_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k<<<blocks, kThreads, smem, st>>>(u, pn, po, n, g, tile, dtdx, p, nullptr, bc, dx);
        return acuda(cudaGetLastError());
    }
};

}  // namespace

extern "C" {

// longest array that the single transposed step leaves to the FP64 backward, as the single
// step does (us, FP64 / float pairs, smooth and random states: 64 cells 31 / 47, 41; 96
// 34 / 47, 45; 128 42 / 47, 52; 192 50 / 46, 56; 256 80 / 47, 72)
static constexpr int64_t kFxVjpCells = 128;

int shk_ssprk33_vjp_bc_f64(const shk_scheme* scheme, const shk_boundary* bc, const double* u,
                           const double* p_next, double* p_out, int64_t n, int32_t nghosts,
                           double dx, double dt, void* stream) {
    if (!adjoint_supported(scheme) || scheme->rec != SHK_REC_WENOJS53 || !u || !p_next || !p_out || n < 3 || nghosts < 3 ||
        !(dx > 0) || !(dt >= 0))
        return SHK_EINVAL;
    shk_boundary b;
    std::memset(&b, 0, sizeof(b));
    if (bc) b = *bc;
    if (b.left < SHK_BC_PERIODIC || b.left > SHK_BC_NEUMANN || b.right < SHK_BC_PERIODIC ||
        b.right > SHK_BC_NEUMANN || ((b.left == SHK_BC_PERIODIC) != (b.right == SHK_BC_PERIODIC)))
        return SHK_EINVAL;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int tile = kAdjTile;
    const int W = tile + 2 * adj_uhalo<double>();
    const size_t smem = AdjSmem<double>::host_bytes(W);
    const int blocks = static_cast<int>((n + tile - 1) / tile);
    SingleVjpLaunch f{u, p_next, p_out, n, nghosts, tile, dt / dx, adj_params<double>(scheme),
                      smem, blocks, st, b, dx, fixed_flux_scheme(scheme) && n > kFxVjpCells};
    return by_equation<double>(scheme->equation, f);
}

int shk_ssprk33_vjp_f64(const shk_scheme* scheme, const double* u, const double* p_next,
                        double* p_out, int64_t n, int32_t nghosts, double dx, double dt,
                        void* stream) {
    return shk_ssprk33_vjp_bc_f64(scheme, nullptr, u, p_next, p_out, n, nghosts, dx, dt, stream);
}

int shk_plan_forward_checkpointed(shk_plan* plan, void* u_a, void* u_b, int32_t nsteps,
                                  void* ckpt, int32_t stride, void* stream) {
    PlanDev D;
    int dtype = 0, grid = 0;
    shk_scheme sch;
    int64_t total = 0;
    if (!plan || !u_a || !u_b || !ckpt || nsteps < 0 || stride <= 0) return SHK_EINVAL;
    int64_t hsteps = 0;
    int r = plan_view(plan, &D, &dtype, &grid, &sch, &total, &hsteps);
    if (r != SHK_OK) return r;
    // checkpoints and the dt history are indexed from the last reset
    if (!D.dt_hist || D.max_steps < nsteps || hsteps != 0) return SHK_EINVAL;
    const size_t bytes = size_t(total) * (dtype == SHK_F64 ? 8 : 4);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    for (int k = 0; k < nsteps; k += stride) {
        // the state before step k is in u_a for even k, u_b for odd k
        const void* cur = (k % 2 == 0) ? u_a : u_b;
        ADJ_CUDA(cudaMemcpyAsync(static_cast<char*>(ckpt) + size_t(k / stride) * bytes, cur,
                                 bytes, cudaMemcpyDeviceToDevice, st));
        r = shk_plan_step(plan, u_a, u_b, std::min(stride, nsteps - k), stream);
        if (r != SHK_OK) return r;
    }
    return SHK_OK;
}

int shk_plan_adjoint(shk_plan* plan, const void* ckpt, int32_t stride, int32_t nsteps, void* seg,
                     void* p_a, void* p_b, void* stream) {
    return shk_plan_adjoint_staged(plan, ckpt, stride, nsteps, seg, nullptr, p_a, p_b, stream);
}

// bytes of stage storage per replayed step (0: the plan recomputes)
static int64_t stage_bytes(const PlanDev& D, int dtype, const shk_scheme& sch, int64_t total) {
    if (sch.rec == SHK_REC_LEARNED) return 2 * total * int64_t(sizeof(float));
    const bool periodic = D.bc_left == SHK_BC_PERIODIC && D.bc_right == SHK_BC_PERIODIC;
    if (dtype == SHK_F64 && sch.rec == SHK_REC_WENOJS53 && periodic)
        return 8 * total * int64_t(sizeof(double));
    return 0;
}

int shk_plan_adjoint_stage_bytes(shk_plan* plan, int64_t* nbytes) {
    PlanDev D;
    int dtype = 0, grid = 0;
    shk_scheme sch;
    int64_t total = 0;
    if (!plan || !nbytes) return SHK_EINVAL;
    int r = plan_view(plan, &D, &dtype, &grid, &sch, &total, nullptr);
    if (r != SHK_OK) return r;
    *nbytes = stage_bytes(D, dtype, sch, total);
    return SHK_OK;
}

int shk_plan_adjoint_staged(shk_plan* plan, const void* ckpt, int32_t stride, int32_t nsteps,
                            void* seg, void* stages, void* p_a, void* p_b, void* stream) {
    PlanDev D;
    int dtype = 0, grid = 0;
    shk_scheme sch;
    int64_t total = 0;
    if (!plan || !ckpt || !seg || !p_a || !p_b || p_a == p_b || nsteps < 0 || stride <= 0)
        return SHK_EINVAL;
    int r = plan_view(plan, &D, &dtype, &grid, &sch, &total, nullptr);
    if (r != SHK_OK) return r;
    if (!adjoint_supported(&sch)) return SHK_EUNSUPPORTED;
    const int64_t sbytes = stage_bytes(D, dtype, sch, total);
    if (stages && sbytes == 0) return SHK_EINVAL;  // this plan has no stage storage
    if (!D.dt_hist || D.max_steps < nsteps) return SHK_EINVAL;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t esz = dtype == SHK_F64 ? 8 : 4;
    const size_t bytes = size_t(total) * esz;
    const int W = D.tile + 2 * adj_uhalo<double>();
    const bool mixed = dtype == SHK_F64 && sch.rec == SHK_REC_LEARNED;
    const size_t asmem = mixed ? sizeof(float) * kMixedAdjSlots * size_t(W)
                               : (dtype == SHK_F64 ? AdjSmem<double>::host_bytes(W)
                                                   : AdjSmem<float>::host_bytes(W));
    {
        // the reverse step keeps ~24 windows of the tile in shared memory: plans
        // with longer tiles can step forward but not run the adjoint
        int dev0 = 0, optin = 0;
        cudaGetDevice(&dev0);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev0);
        if (asmem > static_cast<size_t>(optin)) return SHK_EUNSUPPORTED;
    }
    const size_t fsmem = dtype == SHK_F64 ? Smem<double>::step_bytes(D.tile + 2 * step_halo<double>(), sch.rec, fixed_flux_scheme(&sch))
                                          : Smem<float>::step_bytes(D.tile + 2 * step_halo<float>(), sch.rec);
    // adjoint grid: resident CTAs for its larger shared-memory footprint
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int per_sm = std::max(1, static_cast<int>((220 * 1024) / std::max<size_t>(asmem, 1)));
    // stored stages of a fixed-flux plan: batched_adjoint_fx_kernel
    const bool fixed_stored = stages && dtype == SHK_F64 && fixed_flux_scheme(&sch);
    const size_t xsmem = sizeof(double) * kAdjFxArrays * size_t(W);
    if (fixed_stored) {
        ADJ_CUDA(cudaFuncSetAttribute(batched_adjoint_fx_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(xsmem)));
        ADJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batched_adjoint_fx_kernel, kAdjFxThreads, xsmem));
        per_sm = std::max(1, per_sm);
    }
    const int agrid = std::max(1, std::min(D.nitems, per_sm * sms));
    auto seg_at = [&](int j) { return static_cast<char*>(seg) + size_t(j) * bytes; };
    // stage storage of segment step j
    auto stage_at = [&](int j) -> void* {
        return stages ? static_cast<char*>(stages) + size_t(j) * size_t(sbytes) : nullptr;
    };
    const int nseg = (nsteps + stride - 1) / stride;
    void* cur = p_a;
    void* nxt = p_b;
    for (int sgi = nseg - 1; sgi >= 0; --sgi) {
        const int base = sgi * stride;
        const int cnt = std::min(stride, nsteps - base);
        ADJ_CUDA(cudaMemcpyAsync(seg_at(0), static_cast<const char*>(ckpt) + size_t(sgi) * bytes,
                                 bytes, cudaMemcpyDeviceToDevice, st));
        // replay: the states u_1 .. u_{cnt-1} of the segment and, with stage
        // storage, the stage states of every step (the last step's without u_out)
        for (int j = 1; j < cnt + (stages ? 1 : 0); ++j) {
            const double* row = D.dt_hist + size_t(base + j - 1) * D.B;
            void* out = j < cnt ? seg_at(j) : nullptr;
            if (dtype == SHK_F64) {
                ReplayLaunch<double> f{D, seg_at(j - 1), out, row, adj_params<double>(&sch), fsmem, grid, st,
                                       stage_at(j - 1), total, base + j - 1, fixed_flux_scheme(&sch)};
                r = by_scheme<double>(sch, f);
            } else {
                ReplayLaunch<float> f{D, seg_at(j - 1), out, row, adj_params<float>(&sch), fsmem, grid, st,
                                      stage_at(j - 1), total, base + j - 1};
                r = by_scheme<float>(sch, f);
            }
            if (r != SHK_OK) return r;
        }
        for (int j = cnt - 1; j >= 0; --j) {
            const double* row = D.dt_hist + size_t(base + j) * D.B;
            if (fixed_stored) {
                batched_adjoint_fx_kernel<<<agrid, kAdjFxThreads, xsmem, st>>>(
                    D, reinterpret_cast<const double*>(seg_at(j)), static_cast<const double*>(cur),
                    static_cast<double*>(nxt), row, adj_params<double>(&sch), stage_at(j), total);
                r = acuda(cudaGetLastError());
            } else if (dtype == SHK_F64) {
                AdjLaunch<double> f{D, seg_at(j), cur, nxt, row, adj_params<double>(&sch), asmem, agrid, st,
                                    stage_at(j), total, base + j, fixed_flux_scheme(&sch)};
                r = by_scheme<double>(sch, f);
            } else {
                AdjLaunch<float> f{D, seg_at(j), cur, nxt, row, adj_params<float>(&sch), asmem, agrid, st,
                                   stage_at(j), total, base + j};
                r = by_scheme<float>(sch, f);
            }
            if (r != SHK_OK) return r;
            std::swap(cur, nxt);
        }
    }
    return SHK_OK;
}

}  // extern "C"

#ifdef SHOCKS_BOUNDS_CHECK
// this translation unit's bounds log (read by shk_check_bounds in forward.cu)
extern "C" int shk_check_tu_adjoint(shk::BoundsLog* out, int32_t reset) {
    return acuda(shk::bounds_log_read(out, reset != 0));
}
#endif
