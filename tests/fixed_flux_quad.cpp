// The host half of csrc/fixed_flux.cuh against 113-bit arithmetic. Prints lines
// "name value"; the test holds the bars.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "fixed_flux.cuh"

#if defined(__aarch64__)
typedef long double quad;
#else
typedef __float128 quad;
#endif
using namespace shk::fx;

static quad qabs(quad x) { return x < 0 ? -x : x; }
static quad qmax(quad a, quad b) { return a > b ? a : b; }

// six times the corrections of cell v[2] of five, on either side
static void corrections(const quad* v, quad eps, quad& right, quad& left) {
    auto side = [&](quad a, quad b, quad c, quad d, quad e) {
        const quad t = quad(13) / 12, q = quad(1) / 4;
        const quad b0 = t * (a - 2 * b + c) * (a - 2 * b + c) + q * (a - 4 * b + 3 * c) * (a - 4 * b + 3 * c);
        const quad b1 = t * (b - 2 * c + d) * (b - 2 * c + d) + q * (b - d) * (b - d);
        const quad b2 = t * (c - 2 * d + e) * (c - 2 * d + e) + q * (3 * c - 4 * d + e) * (3 * c - 4 * d + e);
        const quad w0 = 1 / ((eps + b0) * (eps + b0)), w1 = 6 / ((eps + b1) * (eps + b1)), w2 = 3 / ((eps + b2) * (eps + b2));
        return (w0 * (2 * a - 7 * b + 5 * c) + w1 * (2 * d - c - b) + w2 * (5 * d - 4 * c - e)) / (w0 + w1 + w2);
    };
    right = side(v[0], v[1], v[2], v[3], v[4]);
    left = side(v[4], v[3], v[2], v[1], v[0]);
}
static quad flux288(quad R, quad L, quad a) { return 72 * (R * R + L * L) - 144 * a * (L - R); }

// the FP64 formula of the same face (weno53_cell_d of csrc/device.cuh)
static void cell_double(const double* v, double eps, double& ul, double& ur) {
    const double dm2 = v[1] - v[0], dm1 = v[2] - v[1], d0 = v[3] - v[2], dp1 = v[4] - v[3];
    const double Em = dm1 - dm2, E0 = d0 - dm1, Ep = dp1 - d0, e4 = 4.0 * eps;
    auto G = [&](double E) { return std::fma(13.0 / 3.0 * E, E, e4); };
    const double h0 = std::fma(2.0, dm1, Em), h1 = d0 + dm1, h2 = std::fma(-2.0, d0, Ep);
    double s0 = std::fma(h0, h0, G(Em)), s1 = std::fma(h1, h1, G(E0)), s2 = std::fma(h2, h2, G(Ep));
    s0 *= s0; s1 *= s1; s2 *= s2;
    const double P0 = s1 * s2, P1 = s0 * s2, P2 = s0 * s1;
    const double cr1 = std::fma(12.0, d0, 6.0 * dm1);
    const double nr = std::fma(P0, std::fma(2.0, h0, -dm1), std::fma(P1, cr1, P2 * (3.0 * (d0 - h2))));
    const double nl = std::fma(P2, std::fma(2.0, h2, d0), std::fma(P1, std::fma(6.0, E0, -cr1), P0 * (-3.0 * (h0 + dm1))));
    const double m = 36.0 * P1, dr = std::fma(6.0, P0, std::fma(18.0, P2, m)), dl = std::fma(6.0, P2, std::fma(18.0, P0, m));
    const double r = 1.0 / (dr * dl);
    ur = std::fma(nr * dl, r, v[2]);
    ul = std::fma(nl * dr, r, v[2]);
}

struct Sum;
static void add_listed(Sum& sum, const double* v, double eps);
struct Sum {
    double n = 0, s = 0, top = 0;
    void add(double e) { n += 1; s += e * e; top = std::max(top, e); }
    void print(const char* name) const { std::printf("%s.count %.0f\n%s.rms %.6g\n%s.max %.6g\n", name, n, name, std::sqrt(s / std::max(n, 1.0)), name, top); }
};

static Sum lf_rough;
static int state_shift = 0;

// the flux of the face between v[2] and v[3] of six from its rounded corrections, in units
// of the largest of its four cells and face values
static void add_listed(Sum& sum, const double* v, double eps) {
    quad q[6], tR, tL, x;
    for (int i = 0; i < 6; ++i) q[i] = v[i];
    corrections(q, eps, tR, x);
    corrections(q + 1, eps, x, tL);
    const double tr = double(tR), tl = double(tL);
    const quad R = q[2] + quad(tr) / 6, L = q[3] + quad(tl) / 6, am = qmax(qabs(q[2]), qabs(q[3]));
    quad top = qmax(qmax(qabs(R), qabs(L)), am);
    double g;
    if (!listed_flux(tr, tl, v[2], v[3], g)) return;
    sum.add(double(qabs(quad(g) - flux288(R, L, am)) / (quad(0x1p-53) * 288 * top * top)));
    // Lax-Friedrichs with a speed at least the cells': in units of speed x size
    const double speed = std::ldexp(double(am), state_shift++ % 40) * 1.25;
    if (!listed_flux_lf(tr, tl, v[2], v[3], speed_begin(speed), g)) return;
    lf_rough.add(double(qabs(quad(g) - flux288(R, L, speed)) / (quad(0x1p-53) * 288 * top * qmax(top, speed))));
}

int main() {
    std::mt19937_64 gen(7);
    std::normal_distribution<double> N(0.0, 1.0);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    const double unit = 0x1p-53;
    Sum pair, plain, lf, listed, rough, faces, grad;
    double bad_double = 0, bad_split = 0;
    for (double eps : {1e-24, 1e-12, 1e-6, 1.0, 1e24}) {
        const FF eps4{dup(static_cast<float>(4.0 * eps)), dup(static_cast<float>(4.0 * eps - double(static_cast<float>(4.0 * eps))))};
        for (int state = 0; state < 240; ++state) {
            // smooth waves with a little noise, a mean, and any amplitude of 2^-58 .. 2^58
            const int n = 128;
            const double amp = std::ldexp(1.0 + U(gen), int(std::floor(116.0 * U(gen))) - 58);
            const double mean = (state % 3) ? N(gen) : 0.0, noise = std::pow(10.0, -2.0 - 8.0 * U(gen));
            double ph[4], a[4], w[4];
            for (int k = 0; k < 4; ++k) { ph[k] = 7.0 * U(gen); a[k] = N(gen); w[k] = 0.4 * U(gen); }
            std::vector<double> v(n);
            for (int i = 0; i < n; ++i) {
                double x = mean + noise * N(gen);
                for (int k = 0; k < 4; ++k) x += a[k] * std::sin(w[k] * i + ph[k]);
                v[i] = amp * x;
            }
            double speed_d = 0;
            for (double x : v) speed_d = std::max(speed_d, std::fabs(x));
            const Speed speed = speed_begin(speed_d);
            // as the lanes of fx_fluxes: two cells each
            const int lanes = n / 2 - 2;
            std::vector<Lane> s(lanes);
            std::vector<FF> pR(lanes), pL(lanes);
            for (int l = 1; l < lanes; ++l) s[l] = lane_begin(v[2 * l - 1], v[2 * l], v[2 * l + 1], v[2 * l + 2], v[2 * l + 3], eps4);
            for (int l = 2; l + 1 < lanes; ++l)
                lane_cells(s[l], p2y(s[l - 1].a.h), p2y(s[l - 1].a.l), p2x(s[l + 1].g.h), p2x(s[l + 1].g.l), p2y(s[l - 1].T.h), p2y(s[l - 1].T.l), pR[l], pL[l]);
            for (int l = 2; l + 2 < lanes; ++l) {
                const Sums u = face_units(pR[l], FF{p2(p2y(pL[l].h), p2x(pL[l + 1].h)), p2(p2y(pL[l].l), p2x(pL[l + 1].l))}, p2(s[l].x.iu, s[l].y.iu));
                for (int k = 0; k < 2; ++k) {
                    const int j = 2 * l + k;
                    const Cell& c = k ? s[l].y : s[l].x;
                    auto el = [&](P2 q) { return k ? p2y(q) : p2x(q); };
                    int64_t Z, D, Q;
                    const bool ok = face_sums(c, el(u.xR), el(u.xL), el(u.tR), el(u.tL), el(u.rs), el(u.rd), Z, D, Q);
                    quad w5[6];
                    double top = 0;
                    for (int i = 0; i < 6; ++i) w5[i] = v[j - 2 + i];
                    for (int i = 1; i < 5; ++i) top = std::max(top, std::fabs(v[j - 2 + i]));
                    quad tR, tL, x;
                    corrections(w5, eps, tR, x);
                    corrections(w5 + 1, eps, x, tL);
                    const quad R = w5[2] + tR / 6, L = w5[3] + tL / 6, am = qmax(qabs(w5[2]), qabs(w5[3]));
                    const quad size = quad(unit) * 288 * quad(top) * quad(top);
                    if (ok) {
                        const quad F = flux288(R, L, am);
                        pair.add(double(qabs(quad(face_flux(c.k, Z, D, Q)) - F) / size));
                        double ul, ur, dummy;
                        cell_double(&v[j - 2], eps, dummy, ur);
                        cell_double(&v[j - 1], eps, ul, dummy);
                        const double ad = std::max(std::fabs(v[j]), std::fabs(v[j + 1]));
                        const double f = 72.0 * std::fma(ul, ul, std::fma(ur, ur, 2.0 * ad * (ur - ul)));
                        plain.add(double(qabs(quad(f) - F) / size));
                        lf.add(double(qabs(quad(face_flux_lf(c, Z, D, speed)) - flux288(R, L, speed_d)) / (quad(unit) * 288 * quad(top) * quad(speed_d))));
                        faces.add(double(qmax(qabs(quad(to_double(Z + D, c.kz) * (1.0 / 12.0)) - R), qabs(quad(to_double(Z - D, c.kz) * (1.0 / 12.0)) - L)) / (quad(unit) * quad(top))));
                    }
                    // the flux of a left face from its rounded corrections
                    add_listed(listed, &v[j - 2], eps);
                }
                // the backward of the two cells' weights
                const Cell &cx = s[l].x, &cy = s[l].y;
                const P2 u0 = p2(cx.u0, cy.u0), u12 = u0 * dup(0x1p12f), u36 = u0 * dup(0x1p36f);
                const FF T0 = s[l].T, Tm{p2(p2y(s[l - 1].T.h), p2x(T0.h)), p2(p2y(s[l - 1].T.l), p2x(T0.l))};
                const FF S = to_ff(cx.S, cy.S, u36, u12, u0), E = to_ff(cx.E, cy.E, u36, u12, u0);
                const CellWeights cw = lane_weights(S, E, Tm, T0, eps4);
                const double gr = N(gen), gl = N(gen);
                float h, lo;
                split_double(gr, 1023 + 3, h, lo);
                const FF gR{dup(h), dup(lo)};
                split_double(gl, 1023 + 3, h, lo);
                const FF gL{dup(h), dup(lo)};
                const CellGrad g = lane_grad(cw, S, E, Tm, T0, gR, gL);
                for (int k = 0; k < 2; ++k) {
                    auto val = [&](const FF& q) { return k ? quad(p2y(q.h)) + quad(p2y(q.l)) : quad(p2x(q.h)) + quad(p2x(q.l)); };
                    if (!((k ? p2y(cw.x) : p2x(cw.x)) <= 0.125f)) continue;
                    // the same quantities in quad, from the cells
                    const int c = 2 * l + k;
                    auto V = [&](int i) { return quad(v[c + i]); };
                    const quad qS = V(1) - V(-1), qE = V(1) - 2 * V(0) + V(-1), Em = V(0) - 2 * V(-1) + V(-2), Ep = V(2) - 2 * V(1) + V(0);
                    const quad qTm = qE - Em, qT0 = Ep - qE, h0 = qS - qTm, h2 = qS - qT0, c133 = quad(13) / 3;
                    const quad e0 = h0 * h0 + c133 * Em * Em + 4 * quad(eps), e1 = qS * qS + c133 * qE * qE + 4 * quad(eps), e2 = h2 * h2 + c133 * Ep * Ep + 4 * quad(eps);
                    const quad r0 = (e1 / e0) * (e1 / e0), r2 = (e1 / e2) * (e1 / e2), DR = r0 + 6 + 3 * r2, DL = r2 + 6 + 3 * r0;
                    const quad A = r0 * qTm, B = r2 * qT0, qpR = -(2 * A + 3 * B) / DR, qpL = (3 * A + 2 * B) / DL;
                    const quad sc = 8, a = quad(gr) / sc / DR, b = quad(gl) / sc / DL, k0 = 3 * b - 2 * a, k2 = 2 * b - 3 * a;
                    const quad w0 = 2 * r0 * (qTm * k0 - (a * qpR + 3 * b * qpL)), w2 = 2 * r2 * (qT0 * k2 - (3 * a * qpR + b * qpL));
                    const quad i0 = -w0 / e0, i2 = -w2 / e2, i1 = (w0 + w2) / e1;
                    // (less the ideal weights' part: -2/10 gR + 3/10 gL in T_m, -3/10 gR + 2/10 gL in T_0)
                    const quad gm = r0 * k0 - (3 * quad(gl) - 2 * quad(gr)) / sc / 10, g0 = r2 * k2 - (2 * quad(gl) - 3 * quad(gr)) / sc / 10;
                    const quad sg = 2 * (qS * i1 + h0 * i0 + h2 * i2), et = 2 * c133 * (qE * i1 + Em * i0 + Ep * i2);
                    const quad tm = gm - 2 * (h0 * i0 + c133 * Em * i0), t0 = g0 + 2 * (c133 * Ep * i2 - h2 * i2);
                    const quad size = qmax(qabs(quad(gr)), qabs(quad(gl))) / sc;
                    const quad err = qmax(qmax(qabs(val(g.tm) - tm), qabs(val(g.t0) - t0)), qmax(qabs(val(g.sg) - sg), qabs(val(g.et) - et)));
                    grad.add(double(err / size / quad(unit)));
                }
            }
        }
    }
    // left faces of random cells, also where one side is much the larger
    for (int i = 0; i < 100000; ++i) {
        double v[6];
        for (double& x : v) x = N(gen) * (i % 2 ? 1.0 : std::pow(10.0, -6.0 * U(gen)));
        add_listed(rough, v, 1e-6);
    }
    for (int i = 0; i < 200000; ++i) {
        // integers to doubles: within half a unit in the last place
        const int sh = int(gen() % 63);
        const int64_t X = int64_t(gen()) >> sh;
        const int k = int(gen() % 200) - 100;
        const double d = to_double(X, k);
        const quad e = X == 0 ? qabs(quad(d)) : qabs(quad(std::ldexp(d, -k)) - quad(X)) / (qabs(quad(X)) * quad(unit));
        bad_double = std::max(bad_double, double(e));
        // doubles to pairs and back, relative to any scale above
        const double v = N(gen) * std::ldexp(1.0, int(gen() % 60));
        const uint32_t em = ((static_cast<uint32_t>(dhi(v)) & 0x7fffffffu) >> 20) + uint32_t(gen() % 80);
        float h, l;
        split_double(v, em, h, l);
        const double w = join_double(h, l, em);
        bad_split = std::max(bad_split, std::fabs(w - v) / std::fabs(v) / unit);
    }
    pair.print("rusanov");
    plain.print("formula");
    lf.print("lf");
    faces.print("faces");
    listed.print("listed");
    rough.print("rough");
    lf_rough.print("lf_rough");
    grad.print("grad");
    std::printf("to_double.max %.6g\nsplit.max %.6g\n", bad_double, bad_split);
    return 0;
}
