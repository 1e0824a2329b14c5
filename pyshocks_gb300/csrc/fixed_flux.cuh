// Face fluxes of a double state without the FP64 pipe (Burgers, WENO-JS5,
// Rusanov or global Lax-Friedrichs with nu = 1).
//
// GB300's FP64 pipe takes 16 clocks per warp instruction and SM, 64 times an
// FP32 or integer instruction's share, so the flux is formed from 64-bit
// integers and pairs of floats. With E_k = v_{k+1} - 2 v_k + v_{k-1} and
// T_k = E_{k+1} - E_k, the two face values of WENO-JS5 (R = ur_j, L = ul_{j+1})
// on the middle sub-stencil's value plus weighted third differences give
//   Z = 6 (R + L) = 6 (v_j + v_{j+1}) - (E_j + E_{j+1}) + pR_j + pL_{j+1}
//   D = 6 (R - L) = T_j + pR_j - pL_{j+1}
//   288 F = Z^2 + D (D + 24 a),  a = max(|v_j|, |v_{j+1}|) (Lax-Friedrichs: the
//                                instance's maximum)
//   pR = -(2 r0 T_{c-1} + 3 r2 T_c) / (r0 + 6 + 3 r2)
//   pL =  (2 r2 T_c + 3 r0 T_{c-1}) / (r2 + 6 + 3 r0)
// with r0 = (e1/e0)^2, r2 = (e1/e2)^2, e_k = 4 (eps + beta_k). Only pR and pL
// are nonlinear, and they carry the factor T, the third difference:
//   * v, E, T, Z and D are 64-bit integers in units of 2^-57 of the largest of
//     a lane's cells (a power of two per lane), finer than a double near that
//     size; sums and differences of them are exact;
//   * pR and pL are unevaluated sums of two floats (about 45 bits). A face is
//     accepted while |T| <= 2^-7 of the lane's scale: their error then stays
//     below 2^-54 of it, under the rounding of a double evaluation. Other faces
//     (shocks, noise, non-finite values, scales outside 2^+-60) are left to
//     the FP64 formula.
// The two cells of a lane run in the two halves of the packed float
// instructions (add/mul/fma.f32x2).
// Measured on the batched step (4096 instances, 25.9 M cells, us per step): 8010
// with the FP64 formula (156 FP64 instructions per cell-step, that pipe 86 %
// busy), 1199 with this. Error of the states against runs in 113-bit arithmetic
// (relative L2, FP64 formula / this): Fourier modes and a jump, 24 instances of 100 to
// 1000 cells, 30 steps 1.806e-15 / 1.799e-15; 16 of 500 to 9000, 6 steps 3.941e-16 /
// 3.957e-16; with 0.5 % noise, 10 steps 6.189e-16 / 6.196e-16; jumps between constants
// 4.587e-16 / 4.387e-16; random cells, all left to FP64, 6.291e-16 / 6.238e-16.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define SHK_FX __device__ __forceinline__
#else
#include <cmath>
#include <cstring>
#define SHK_FX static inline
#endif

namespace shk {
namespace fx {

// ---- pairs of floats in one register pair ------------------------------------
#ifdef __CUDACC__
struct P2 {
    unsigned long long b;
};
SHK_FX P2 p2(float x, float y) {
    P2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.b) : "f"(x), "f"(y));
    return r;
}
SHK_FX float p2x(P2 a) {
    return __uint_as_float(static_cast<unsigned>(a.b));
}
SHK_FX float p2y(P2 a) {
    return __uint_as_float(static_cast<unsigned>(a.b >> 32));
}
SHK_FX P2 operator+(P2 a, P2 b) {
    P2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
    return r;
}
SHK_FX P2 operator*(P2 a, P2 b) {
    P2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
    return r;
}
SHK_FX P2 operator-(P2 a, P2 b) {
    P2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
    return r;
}
SHK_FX P2 fma2(P2 a, P2 b, P2 c) {
    P2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.b) : "l"(a.b), "l"(b.b), "l"(c.b));
    return r;
}
SHK_FX float rcp1(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
SHK_FX uint32_t fbits(float x) { return __float_as_uint(x); }
SHK_FX float bitsf(uint32_t x) { return __uint_as_float(x); }
SHK_FX int32_t f2i(float x) { return __float2int_rn(x); }
SHK_FX uint32_t umulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
SHK_FX uint32_t clz32(uint32_t a) { return static_cast<uint32_t>(__clz(static_cast<int>(a))); }
SHK_FX int dhi(double x) { return __double2hiint(x); }
SHK_FX uint32_t dlo(double x) { return static_cast<uint32_t>(__double2loint(x)); }
SHK_FX double hilo(int hi, uint32_t lo) { return __hiloint2double(hi, static_cast<int>(lo)); }
SHK_FX uint64_t shr64(uint64_t x, uint32_t s) {  // 0 for s >= 64
    uint64_t r;
    asm("shr.b64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
    return r;
}
#else
struct P2 {
    float x, y;
};
SHK_FX P2 p2(float x, float y) { return P2{x, y}; }
SHK_FX float p2x(P2 a) { return a.x; }
SHK_FX float p2y(P2 a) { return a.y; }
SHK_FX P2 operator+(P2 a, P2 b) { return P2{a.x + b.x, a.y + b.y}; }
SHK_FX P2 operator-(P2 a, P2 b) { return P2{a.x - b.x, a.y - b.y}; }
SHK_FX P2 operator*(P2 a, P2 b) { return P2{a.x * b.x, a.y * b.y}; }
SHK_FX P2 fma2(P2 a, P2 b, P2 c) { return P2{std::fmaf(a.x, b.x, c.x), std::fmaf(a.y, b.y, c.y)}; }
SHK_FX float rcp1(float x) { return 1.0f / x; }
SHK_FX uint32_t fbits(float x) { uint32_t r; std::memcpy(&r, &x, 4); return r; }
SHK_FX float bitsf(uint32_t x) { float r; std::memcpy(&r, &x, 4); return r; }
SHK_FX int32_t f2i(float x) { return x == x ? static_cast<int32_t>(std::nearbyintf(x)) : 0; }
SHK_FX uint32_t clz32(uint32_t a) { return a ? static_cast<uint32_t>(__builtin_clz(a)) : 32u; }
SHK_FX uint32_t umulhi(uint32_t a, uint32_t b) { return static_cast<uint32_t>((uint64_t(a) * b) >> 32); }
SHK_FX int dhi(double x) { int64_t r; std::memcpy(&r, &x, 8); return static_cast<int>(r >> 32); }
SHK_FX uint32_t dlo(double x) { uint64_t r; std::memcpy(&r, &x, 8); return static_cast<uint32_t>(r); }
SHK_FX double hilo(int hi, uint32_t lo) {
    const uint64_t r = (uint64_t(uint32_t(hi)) << 32) | lo;
    double d;
    std::memcpy(&d, &r, 8);
    return d;
}
SHK_FX uint64_t shr64(uint64_t x, uint32_t s) { return s >= 64 ? 0 : x >> s; }
#endif
SHK_FX P2 dup(float x) { return p2(x, x); }
SHK_FX P2 neg(P2 a) { return a * dup(-1.0f); }

// ---- unevaluated sums h + l of two floats (error-free transformations of
// Dekker and Knuth) -------------------------------------------------------------
struct FF {
    P2 h, l;
};
SHK_FX FF add(FF a, FF b) {
    const P2 s = a.h + b.h;
    const P2 bb = s - a.h;
    const P2 e = (a.h - (s - bb)) + (b.h - bb);
    return FF{s, e + (a.l + b.l)};
}
SHK_FX FF sub(FF a, FF b) {
    const P2 s = a.h - b.h;
    const P2 bb = s - a.h;
    const P2 e = (a.h - (s - bb)) - (b.h + bb);
    return FF{s, e + (a.l - b.l)};
}
// |a| >= |b|
SHK_FX FF add_ordered(FF a, FF b) {
    const P2 s = a.h + b.h;
    const P2 e = b.h - (s - a.h);
    return FF{s, e + (a.l + b.l)};
}
SHK_FX FF mul(FF a, FF b) {
    const P2 p = a.h * b.h;
    P2 e = fma2(a.h, b.h, neg(p));
    e = fma2(a.h, b.l, e);
    e = fma2(a.l, b.h, e);
    return FF{p, e};
}
SHK_FX FF sqr(FF a) {
    const P2 p = a.h * a.h;
    P2 e = fma2(a.h, a.h, neg(p));
    e = fma2(a.h + a.h, a.l, e);
    return FF{p, e};
}
SHK_FX FF twice(FF a) { return FF{a.h + a.h, a.l + a.l}; }
SHK_FX FF scale(FF a, P2 s) { return FF{a.h * s, a.l * s}; }  // s a power of two
// n / d, sign s = +1 or -1 of the result
SHK_FX FF quot(FF n, FF d, float s) {
    const P2 y = p2(rcp1(p2x(d.h)), rcp1(p2y(d.h)));
    const P2 q = n.h * y;
    const P2 nq = neg(q);
    P2 r = fma2(nq, d.h, n.h);
    r = fma2(nq, d.l, r + n.l);
    const P2 q1 = r * y;
    return s > 0.0f ? FF{q, q1} : FF{nq, neg(q1)};
}

// ---- 64-bit integers -----------------------------------------------------------
// magnitude and exponent of a double: m 2^(e - 1080) with m < 2^58
struct Mag {
    uint64_t m;
    uint32_t e;
    int32_t s;  // 0 or -1
};
SHK_FX Mag mag(double v) {
    const uint32_t hi = static_cast<uint32_t>(dhi(v)) & 0x7fffffffu;
    return Mag{((uint64_t((hi & 0xfffffu) | 0x100000u) << 32) | dlo(v)) << 5, hi >> 20, dhi(v) >> 31};
}
// |v| truncated to units of 2^(exm - 1079) (exponents up to exm + 1 fit; 0
// stays 0, since the scale is far above the subnormals), and with its sign
SHK_FX uint64_t fix_abs(const Mag& v, uint32_t exm) { return shr64(v.m, exm + 1u - v.e); }
SHK_FX int64_t with_sign(uint64_t m, const Mag& v) {
    const int64_t s = v.s;
    return (static_cast<int64_t>(m) ^ s) - s;
}
// X u as two floats from pieces above bit 36, 24 bits and 12 bits (|X| < 2^60)
SHK_FX FF to_ff(int64_t X, int64_t Y, P2 u36, P2 u12, P2 u0) {
    const P2 h = p2(static_cast<float>(static_cast<int32_t>(X >> 36)),
                    static_cast<float>(static_cast<int32_t>(Y >> 36))) * u36;
    const P2 m = p2(static_cast<float>(static_cast<uint32_t>(X >> 12) & 0xffffffu),
                    static_cast<float>(static_cast<uint32_t>(Y >> 12) & 0xffffffu));
    const P2 l = p2(static_cast<float>(static_cast<uint32_t>(X) & 0xfffu),
                    static_cast<float>(static_cast<uint32_t>(Y) & 0xfffu));
    const P2 s = fma2(m, u12, h);           // |h| >= |m u12| or h = 0
    const P2 e = fma2(m, u12, h - s);   // exact
    return FF{s, fma2(l, u0, e)};
}
// (third differences, |X| < 2^50: two pieces)
SHK_FX FF to_ff50(int64_t X, int64_t Y, P2 u26, P2 u0) {
    const P2 h = p2(static_cast<float>(static_cast<int32_t>(X >> 26)),
                    static_cast<float>(static_cast<int32_t>(Y >> 26))) * u26;
    const P2 l = p2(static_cast<float>(static_cast<uint32_t>(X) & 0x3ffffffu),
                    static_cast<float>(static_cast<uint32_t>(Y) & 0x3ffffffu)) * u0;
    const P2 s = h + l;
    return FF{s, l + (h - s)};
}

// one cell c of a lane: integers in units of 2^(exm - 1079), the scale taken
// from cells c - 1 .. c + 1
struct Cell {
    int64_t VV;   // v_c + v_{c+1}
    int64_t EE;   // E_c + E_{c+1}
    int64_t T;    // E_{c+1} - E_c
    int64_t S, E; // v_{c+1} - v_{c-1}, E_c
    uint64_t A;   // max(|v_c|, |v_{c+1}|)
    uint32_t exm;
    float u0;     // 2^(exm - 1079)
    float iu;     // 1 / u0
    int kz, k;    // binary exponents of the units and of the flux units
    bool in;      // the scale is in range
    bool ok;      // and v_{c+2} fits it, and |T| < 2^50
};
SHK_FX Cell cell_begin(const Mag& vm, const Mag& v0, const Mag& v1, const Mag& v2) {
    Cell c;
    uint32_t exm = v0.e > v1.e ? v0.e : v1.e;
    exm = exm > vm.e ? exm : vm.e;
    // scales 2^-60 .. 2^60; a zero state takes the smallest
    c.in = exm - (1023u - 60u) <= 120u || exm == 0u;
    exm = exm == 0u || !c.in ? 1023u - 60u : exm;
    c.exm = exm;
    c.u0 = bitsf((exm - 952u) << 23);
    c.iu = bitsf((1206u - exm) << 23);
    c.kz = static_cast<int>(exm) - 1079;
    c.k = 2 * static_cast<int>(exm) - 2094;
    const uint64_t A0 = fix_abs(v0, exm), A1 = fix_abs(v1, exm);
    c.A = A0 > A1 ? A0 : A1;
    const int64_t Vm = with_sign(fix_abs(vm, exm), vm), V0 = with_sign(A0, v0);
    const int64_t V1 = with_sign(A1, v1), V2 = with_sign(fix_abs(v2, exm), v2);
    const int64_t dm = V0 - Vm, d0 = V1 - V0, d1 = V2 - V1;
    const int64_t E1 = d1 - d0;
    c.E = d0 - dm;
    c.S = d0 + dm;
    c.T = E1 - c.E;
    c.EE = c.E + E1;
    c.VV = V0 + V1;
    c.ok = c.in && v2.e <= exm + 1u && static_cast<uint32_t>((c.T >> 32) + 0x40000) < 0x80000u;
    return c;
}

// the two cells c0, c0 + 1 of a lane between the exchanges with its neighbours
struct Lane {
    Cell x, y;
    FF T;        // (T_{c0}, T_{c0+1}); NaN where out of range
    FF a, b, g;  // e0 of cell k+1, e1 of cell k, e2 of cell k-1 for k = c0, c0+1
};

// part 1: from v_{c0-1} .. v_{c0+3}. Every quantity of cell c depends on its
// own cells c-1 .. c+2 alone (not on the lane that holds it), so a flux is a
// function of its face's six-cell stencil.
SHK_FX Lane lane_begin(double vm, double v0, double v1, double v2, double v3, FF eps4) {
    Lane s;
    {
        const Mag a = mag(vm), b = mag(v0), c = mag(v1), d = mag(v2), e = mag(v3);
        s.x = cell_begin(a, b, c, d);
        s.y = cell_begin(b, c, d, e);
    }
    const P2 u0 = p2(s.x.u0, s.y.u0);
    const P2 u12 = u0 * dup(0x1p12f), u36 = u0 * dup(0x1p36f);
    const FF Sf = to_ff(s.x.S, s.y.S, u36, u12, u0);
    const FF Ef = to_ff(s.x.E, s.y.E, u36, u12, u0);
    const float nan = bitsf(0x7fffffffu);
    s.T = to_ff50(s.x.T, s.y.T, u0 * dup(0x1p26f), u0);
    s.T.h = p2(s.x.ok ? p2x(s.T.h) : nan, s.y.ok ? p2y(s.T.h) : nan);
    // b = S^2 + 13/3 E^2 + 4 eps, a / g = b + 4 E^2 +- 4 S E
    const FF Q = sqr(Sf), W = sqr(Ef), C = mul(Sf, Ef);
    const FF c133{dup(4.33333349f), dup(-1.58945718e-07f)};  // 13/3
    s.b = add(add(Q, mul(W, c133)), eps4);
    // (b >= 13/3 W, and b + 4 W >= 2 sqrt(25/3) |S E| > 4 |S E|)
    const FF base = add_ordered(s.b, scale(W, dup(4.0f)));
    s.a = add_ordered(base, scale(C, dup(4.0f)));
    s.g = add_ordered(base, scale(C, dup(-4.0f)));
    s.g.h = p2(s.x.in ? p2x(s.g.h) : nan, s.y.in ? p2y(s.g.h) : nan);
    return s;
}

// part 2: pR and pL of cells c0, c0+1 from the neighbours' am = a of cell c0-1,
// gp = g of cell c0+2, Tm = T_{c0-1} (each as two floats)
SHK_FX void lane_cells(const Lane& s, float amh, float aml, float gph, float gpl, float Tmh, float Tml,
                       FF& pR, FF& pL) {
    const FF e0{p2(amh, p2x(s.a.h)), p2(aml, p2x(s.a.l))};
    const FF e2{p2(p2y(s.g.h), gph), p2(p2y(s.g.l), gpl)};
    const FF Tm{p2(Tmh, p2x(s.T.h)), p2(Tml, p2x(s.T.l))};
    const FF r0 = sqr(quot(s.b, e0, 1.0f)), r2 = sqr(quot(s.b, e2, 1.0f));
    const FF A = mul(r0, Tm), B = mul(r2, s.T);
    const FF X2 = twice(add(A, B));
    const FF Y6 = add(add(r0, r2), FF{dup(6.0f), dup(0.0f)});
    pR = quot(add(X2, B), add(Y6, twice(r2)), -1.0f);
    pL = quot(add(X2, A), add(Y6, twice(r0)), 1.0f);
}

// ---- reverse mode of a lane's two cells --------------------------------------------
// The smoothness sums and weights' derivatives of both face values of a cell as
// cotangents of S, E, T_{c-1} and T_c. The linear (ideal-weight) part of the
// reconstruction is left to the caller: with x_k = r_k - 1, formed without
// cancellation from e_1 - e_0 = T_{c-1} (2S - T_{c-1} + 13/3 (2E - T_{c-1})) and
// e_1 - e_2 = T_c (2S - T_c - 13/3 (2E + T_c)), the remaining weights
//   r0/D_R - 1/10 = 3 (3 x0 - x2) / 10 D_R,  r2/D_R - 1/10 = (7 x2 - x0) / 10 D_R
// (and mirrored on the left) are small where the state is smooth, and every term
// below carries one of them or a third difference. lane_weights: the weights and `x` =
// |x0| + |x2|, the caller's measure of smooth; lane_grad: the rest, gR, gL 1/6 of the
// cotangents of the face values.
struct CellWeights {
    FF h0, h2, E0, E2, e0, e1, e2, x0, x2;
    P2 x;
};
struct CellGrad {
    FF tm, t0, sg, et;
};
// a times a constant of few bits
SHK_FX FF mul_const(FF a, float c) {
    const P2 C = dup(c);
    const P2 p = a.h * C;
    return FF{p, fma2(a.l, C, fma2(a.h, C, neg(p)))};
}
SHK_FX P2 abs2(P2 a) { return p2(bitsf(fbits(p2x(a)) & 0x7fffffffu), bitsf(fbits(p2y(a)) & 0x7fffffffu)); }
SHK_FX CellWeights lane_weights(FF S, FF E, FF Tm, FF T0, FF eps4) {
    const FF c133{dup(4.33333349f), dup(-1.58945718e-07f)};  // 13/3
    CellWeights w;
    w.h0 = sub(S, Tm);
    w.h2 = sub(S, T0);
    w.E0 = sub(E, Tm);
    w.E2 = add(E, T0);
    w.e1 = add(add(sqr(S), mul(sqr(E), c133)), eps4);
    w.e0 = add(add(sqr(w.h0), mul(sqr(w.E0), c133)), eps4);
    w.e2 = add(add(sqr(w.h2), mul(sqr(w.E2), c133)), eps4);
    const FF b0 = mul(Tm, add(add(S, w.h0), mul(add(E, w.E0), c133)));
    const FF b2 = mul(T0, sub(add(S, w.h2), mul(add(E, w.E2), c133)));
    w.x0 = mul(quot(b0, w.e0, 1.0f), quot(add(w.e1, w.e0), w.e0, 1.0f));
    w.x2 = mul(quot(b2, w.e2, 1.0f), quot(add(w.e1, w.e2), w.e2, 1.0f));
    w.x = abs2(w.x0.h) + abs2(w.x2.h);
    return w;
}
SHK_FX CellGrad lane_grad(const CellWeights& w, FF S, FF E, FF Tm, FF T0, FF gR, FF gL) {
    const FF c263{dup(8.66666698f), dup(-3.17891436e-07f)};  // 26/3
    const FF c03{dup(0.300000012f), dup(-1.19209291e-08f)};  // 3/10
    const FF one{dup(1.0f), dup(0.0f)}, ten{dup(10.0f), dup(0.0f)};
    const FF h0 = w.h0, h2 = w.h2, E0 = w.E0, E2 = w.E2, e0 = w.e0, e1 = w.e1, e2 = w.e2, x0 = w.x0, x2 = w.x2;
    CellGrad g;
    const FF X = add(ten, add(x0, x2));
    const FF DR = add(X, twice(x2)), DL = add(X, twice(x0));
    const FF r0 = add(one, x0), r2 = add(one, x2);
    const FF A = mul(r0, Tm), B = mul(r2, T0), X2 = twice(add(A, B));
    const FF pR = quot(add(X2, B), DR, -1.0f), pL = quot(add(X2, A), DL, 1.0f);
    const FF a = quot(gR, DR, 1.0f), b = quot(gL, DL, 1.0f);
    const FF a3 = add_ordered(twice(a), a), b3 = add_ordered(twice(b), b);
    const FF u0 = sub(b3, twice(a)), u2 = sub(twice(b), a3);
    // cotangents of r0, r2, then of e0, e1, e2
    const FF m0 = add(mul(a, pR), mul(b3, pL)), m2 = add(mul(a3, pR), mul(b, pL));
    const FF w0 = twice(mul(r0, sub(mul(Tm, u0), m0))), w2 = twice(mul(r2, sub(mul(T0, u2), m2)));
    const FF k0 = quot(w0, e0, -1.0f), k2 = quot(w2, e2, -1.0f), k1 = quot(add(w0, w2), e1, 1.0f);
    const FF hk0 = twice(mul(h0, k0)), hk2 = twice(mul(h2, k2));
    const FF Ek0 = mul(mul(E0, k0), c263), Ek2 = mul(mul(E2, k2), c263);
    // the weights beyond the ideal ones
    const FF d = sub(x0, x2);
    const FF y0 = add(twice(x0), d), y2 = sub(twice(x2), d);                        // 3 x0 - x2, 3 x2 - x0
    const FF z0 = add(mul_const(x0, 4.0f), y0), z2 = add(mul_const(x2, 4.0f), y2);  // 7 x0 - x2, 7 x2 - x0
    const FF o0 = mul(sub(mul(z0, b), twice(mul(y0, a))), c03);
    const FF o2 = mul(sub(twice(mul(y2, b)), mul(z2, a)), c03);
    g.sg = add(twice(mul(S, k1)), add(hk0, hk2));
    g.et = add(mul(mul(E, k1), c263), add(Ek0, Ek2));
    g.tm = sub(o0, add(hk0, Ek0));
    g.t0 = add(o2, sub(Ek2, hk2));
    return g;
}

// v 2^(1023 - em) as two floats (truncated upper part, the rest rounded to 24 bits: 48
// bits in all), on the integer pipe; em the biased exponent of the largest value of the warp, 200 .. 1846. 2^-120
// below it and less: zero.
SHK_FX void split_double(double v, uint32_t em, float& h, float& l) {
    const uint32_t hi = static_cast<uint32_t>(dhi(v)), lo = dlo(v);
    const uint32_t mag = hi & 0x7fffffffu;
    const uint32_t fb = ((hi << 3) | (lo >> 29)) + ((0x400u - em + 0x7fu) << 23);
    const uint32_t b = mag < ((em - 120u) << 20) ? 0u : ((fb & 0x7fffffffu) | (hi & 0x80000000u));
    h = bitsf(b);
    // the lower 29 bits of the mantissa, in units of 2^-52 of the upper part's
    // power of two
    l = (static_cast<float>(lo & 0x1fffffffu) * 0x1p-52f) * bitsf(b & 0xff800000u);
}
// (h + l) 2^(em - 1023) as a double, |l| at most a unit of h, on the integer pipe; down to
// |h| = 2^-97, where l's units reach float's smallest number
SHK_FX double join_double(float h, float l, uint32_t em) {
    const uint32_t b = fbits(h), e = (b >> 23) & 0xffu;
    // l in units of 2^-52 of h's power of two, in two factors where one would overflow
    const uint32_t ec = e > 52u ? e : 52u;
    const int32_t li = f2i((l * bitsf((306u - ec) << 23)) * bitsf((127u + ec - e) << 23));
    const int64_t u = (static_cast<int32_t>(b) < 0) ? -int64_t(li) : int64_t(li);
    const uint64_t d = (uint64_t(((b & 0x7fffffffu) >> 3) + ((em - 127u) << 20)) << 32 | uint64_t(b << 29)) +
                       static_cast<uint64_t>(u);
    const bool zero = (b & 0x7fffffffu) == 0u;
    return hilo(zero ? 0 : static_cast<int>(static_cast<uint32_t>(d >> 32) | (b & 0x80000000u)),
                zero ? 0u : static_cast<uint32_t>(d));
}

// the sums and differences of the corrections of a lane's two faces, pR + pL
// and pR - pL, in units: n 2^30 + r each, |p| < 2^52 units
struct Sums {
    P2 xR, xL;  // pR, pL in units
    P2 tR, tL;  // rounded to multiples of 2^30, plus the rounding constant
    P2 rs, rd;  // sum and difference of the rests
};
constexpr float kRound30 = 0x1.8p53f;  // bits 0x5a400000
SHK_FX Sums face_units(FF pR, FF pL, P2 iu) {
    Sums u;
    u.xR = pR.h * iu;
    u.xL = pL.h * iu;
    u.tR = u.xR + dup(kRound30);
    u.tL = u.xL + dup(kRound30);
    const P2 rR = fma2(pR.l, iu, u.xR - (u.tR - dup(kRound30)));
    const P2 rL = fma2(pL.l, iu, u.xL - (u.tL - dup(kRound30)));
    u.rs = rR + rL;
    u.rd = rR - rL;
    return u;
}

// Z = 6 (R + L), D = 6 (R - L) and Q = D + 24 a of face c + 1/2; false where the
// face is left to the FP64 formula
SHK_FX bool face_sums(const Cell& c, float xR, float xL, float tR, float tL, float rs, float rd, int64_t& Z,
                      int64_t& D, int64_t& Q) {
    const uint32_t bR = fbits(tR), bL = fbits(tL);
    const int32_t ns = static_cast<int32_t>(bR + bL - 2u * 0x5a400000u), nd = static_cast<int32_t>(bR - bL);
    Z = int64_t(ns) * (int64_t(1) << 30) + (6 * c.VV - c.EE) + f2i(rs);
    D = int64_t(nd) * (int64_t(1) << 30) + c.T + f2i(rd);
    Q = D + static_cast<int64_t>(24u * c.A);
#ifdef __CUDACC__
    const float x = fabsf(xR) + fabsf(xL);
#else
    const float x = std::fabs(xR) + std::fabs(xL);
#endif
    return x <= 0x1p52f && Q >= 0;
}

// a 64-bit integer X in units of 2^k as a double, rounded to nearest (ties
// away), on the integer pipe
SHK_FX double pack_double(uint32_t hi, uint32_t lo, int e, uint32_t sign) {
    const uint32_t n = clz32(hi);
    const uint64_t t = ((uint64_t(hi) << 32) | lo) << n;  // top bit set
    // the top bit adds one to the exponent field, a rounding carry likewise
    const uint64_t bits = (t >> 11) + ((t >> 10) & 1u) + (uint64_t(uint32_t(e) - n) << 52);
    return hilo(static_cast<int>(static_cast<uint32_t>(bits >> 32) | sign), static_cast<uint32_t>(bits));
}
SHK_FX double to_double(int64_t X, int k) {
    const int e = 1022 + 63 + k;
    if (static_cast<int32_t>(X >> 32) > 0)
        return pack_double(static_cast<uint32_t>(X >> 32), static_cast<uint32_t>(X), e, 0u);
    const uint32_t s = X < 0 ? 0x80000000u : 0u;
    const uint64_t m = X < 0 ? -static_cast<uint64_t>(X) : static_cast<uint64_t>(X);
    const uint32_t hi = static_cast<uint32_t>(m >> 32), lo = static_cast<uint32_t>(m);
    if (hi != 0u) return pack_double(hi, lo, e, s);
    return lo != 0u ? pack_double(lo, 0u, e - 32, s) : 0.0;
}

// the upper 64 of 128 bits of Z^2 and of D Q, 0 <= Q < 2^63
SHK_FX int64_t square_hi(int64_t Z) {
    const int32_t zh = static_cast<int32_t>(Z >> 32), zl = static_cast<int32_t>(static_cast<uint32_t>(Z) >> 1);
    return int64_t(zh) * zh + ((int64_t(zh) * zl) >> 30);
}
SHK_FX int64_t product_hi(int64_t D, int64_t Q) {
    const int32_t dh = static_cast<int32_t>(D >> 32);
    const int32_t qh = static_cast<int32_t>(Q >> 32), ql = static_cast<int32_t>(static_cast<uint32_t>(Q) >> 1);
    return int64_t(dh) * qh + ((int64_t(dh) * ql) >> 31) + umulhi(static_cast<uint32_t>(D), static_cast<uint32_t>(qh));
}
// 288 F = Z^2 + D Q with Q = D + 24 a, in units of 2^k
SHK_FX double face_flux(int k, int64_t Z, int64_t D, int64_t Q) {
    return to_double(square_hi(Z) + product_hi(D, Q), k);
}

// the Lax-Friedrichs speed: 24 a = M units of 2^(e - 1079), M < 2^62
struct Speed {
    int64_t M;
    uint32_t e;
    bool in;  // the scale is in range
};
SHK_FX Speed speed_begin(double a) {
    const Mag m = mag(a);
    return Speed{static_cast<int64_t>(24u * fix_abs(m, m.e)), m.e, m.e <= 1023u + 60u};
}
// 288 F = Z^2 + D^2 + 24 a D with the speed's own scale (at least the cell's):
// in units 2^(k + sh), sh the distance of the two scales. dt / dx times the
// speed is at most 1/2, so a resolution of 2^-57 of (speed x local value) in F
// is one of 2^-57 of the local value in the state.
SHK_FX double lf_flux(uint32_t exm, int k, int64_t Z, int64_t D, const Speed& sp) {
    const uint32_t d = sp.e > exm ? sp.e - exm : 0u, sh = d < 63u ? d : 63u;
    return to_double(((square_hi(Z) + square_hi(D)) >> sh) + product_hi(D, sp.M), k + static_cast<int>(d));
}
SHK_FX double face_flux_lf(const Cell& c, int64_t Z, int64_t D, const Speed& sp) {
    return lf_flux(c.exm, c.k, Z, D, sp);
}

// Z and D of a face from six times the corrections tR = 6 (R - v0), tL = 6 (L - v1) of its
// face values formed in double (v0, v1: the face's cells; A: max of their magnitudes), on
// the scale of the cells and of a quarter of the corrections (|R - v| is a sixth of
// them): the corrections' integers stay below 2^59, Z and D below 2^62, D + 24 A below
// 2^63. False where the integers do not hold it.
struct ListedSums {
    int64_t Z, D;
    uint64_t A;
    uint32_t exm;
};
SHK_FX bool listed_sums(double tR, double tL, double v0, double v1, ListedSums& s) {
    const Mag r = mag(tR), l = mag(tL), a = mag(v0), b = mag(v1);
    uint32_t exm = a.e > b.e ? a.e : b.e;
    exm = exm + 2u > r.e ? exm : r.e - 2u;
    exm = exm + 2u > l.e ? exm : l.e - 2u;
    if (exm == 0u) exm = 1023u - 60u;
    s.exm = exm;
    if (exm - (1023u - 60u) > 120u) return false;
    const int64_t x = with_sign(shr64(r.m << 2, exm + 3u - r.e), r), y = with_sign(shr64(l.m << 2, exm + 3u - l.e), l);
    const uint64_t A0 = fix_abs(a, exm), A1 = fix_abs(b, exm);
    const int64_t V0 = with_sign(A0, a), V1 = with_sign(A1, b);
    s.A = A0 > A1 ? A0 : A1;
    s.Z = 6 * (V0 + V1) + (x + y);
    s.D = 6 * (V0 - V1) + (x - y);
    return true;
}
// 288 F with the integer arithmetic of the other faces: next to a constant state, where
// R = L = v, the flux equals theirs and the difference vanishes exactly
SHK_FX bool listed_flux(double tR, double tL, double v0, double v1, double& G) {
    ListedSums s;
    if (!listed_sums(tR, tL, v0, v1, s)) return false;
    const int64_t Q = s.D + static_cast<int64_t>(24u * s.A);
    if (Q < 0) return false;
    G = face_flux(2 * static_cast<int>(s.exm) - 2094, s.Z, s.D, Q);
    return true;
}
// (with the speed's own scale, as face_flux_lf; a face value may exceed it by a few powers
// of two)
SHK_FX bool listed_flux_lf(double tR, double tL, double v0, double v1, const Speed& sp, double& G) {
    ListedSums s;
    if (!listed_sums(tR, tL, v0, v1, s) || !sp.in) return false;
    const uint32_t up = s.exm > sp.e ? s.exm - sp.e : 0u;
    const Speed scaled{static_cast<int64_t>(shr64(static_cast<uint64_t>(sp.M), up)), sp.e + up, true};
    G = lf_flux(s.exm, 2 * static_cast<int>(s.exm) - 2094, s.Z, s.D, scaled);
    return true;
}

}  // namespace fx
}  // namespace shk
