// gfk_solver.cuh — the per-(f, k) layered boundary-value solve, as device code.
//
// Two formulations of the reference's Medium.SurfaceResponse
// (internal/fk/fk.go:276-327):
//   direct_u  — the reference algorithm restated: 4x4 complex eigenvector
//               propagators and a pivoted 4x4 surface solve (fk.go:138-327,
//               internal/fk/cmat.go:57-96).
//   dunkin_u  — the complex second-compound (minor) propagation of the
//               half-space's decaying 2-plane up to the surface, in closed form
//               with no k*h limit (design source internal/propmat/propmat.go:168-315),
//               started at the shallowest layer thick enough to isolate the
//               layers beneath it.
#pragma once
#include "gfk_math.cuh"

namespace gfk {

constexpr double kTwoPi = 6.283185307179586476925286766559;
constexpr double kPi = 3.141592653589793238462643383280;
constexpr int kMaxLayers = 64;

// Per-(frequency, layer) constants, written once per build by the layer kernel.
// Dunkin:  c[0] = 1/alpha^2, c[1] = 1/beta^2, c[2] = beta^2/alpha^2, c[3] = rho beta^2/mu_ref
// direct:  c[0] = alpha,     c[1] = beta,     c[2] = mu = rho beta^2, c[3] = (rho, 0)
struct LayerC {
    cd c[4];
    double h;
    double pad;
};

// Layer description on the device (mirrors gfk_layer).
struct LayerP {
    double h, vp, vs, rho, qs, qp;
};

// One medium of a plan: fk.Medium's defaults plus what the kernels derive.
struct MediumP {
    double ref_freq, default_q, tau_sigma, tau_eps;
    double mu_ref;  // max rho Vs^2 (fk.go:216-222)
    int count;      // stack entries, the last one the half-space
    int sls;        // nonzero: SLS relaxation replaces constant Q
    int lp_off;     // first layer in the plan's LayerP table
    int pad;
};

// One frequency of a plan (a bank row).
struct FreqDesc {
    double freq;     // Hz
    double dk;       // wavenumber step; k_i = i dk, i = 1..nk
    double kfar;     // k of the static coefficient (fk.go:515-521); 0 skips the row
    int64_t off;     // integrand row offset within its chunk
    int64_t lc_off;  // first of the row's layer constants
    int nk;          // wavenumber samples
    int soil;        // index into the medium table
};

GFK_HD double q_of(const MediumP& m, const LayerP& l) {  // fk.go:67-75
    if (l.qs > 0) return l.qs;
    if (m.default_q > 0) return m.default_q;
    return 30.0;
}

GFK_HD double ref_freq(const MediumP& m) { return m.ref_freq > 0 ? m.ref_freq : 30.0; }

GFK_HD cd sls_modulus(const MediumP& m, cd w) {  // visco.go:78-81 at complex w
    cd iw = cmul_i(w);
    return (1.0 + iw * m.tau_eps) / (1.0 + iw * m.tau_sigma);
}

// Medium.complexVelocity (fk.go:96-110) at the complex frequency 2 pi f - i wi.
// Kjartansson c0 (i w_c / w_ref)^gamma on the principal branch; with wi = 0 the
// reference's own factorisation c0 (f/f_ref)^gamma e^(i pi gamma/2) is used.
GFK_HD cd complex_velocity(const MediumP& m, double v, double q, double f, double wi) {
    if (m.sls) {
        cd rel = 1.0 / csqrt_(sls_modulus(m, mk(kTwoPi * ref_freq(m))));
        double relaxed = v * rel.re;  // visco.go:100-102
        if (f <= 0) return mk(relaxed);
        return relaxed * csqrt_(sls_modulus(m, mk(kTwoPi * f, -wi)));  // visco.go:106-108
    }
    if (q <= 0 || f <= 0) return mk(v);
    double gam = atan(1.0 / q) / kPi;
    double c0 = v * cos(kPi * gam / 2);
    if (wi == 0.0) return (c0 * pow(f / ref_freq(m), gam)) * cexp_(mk(0.0, kPi * gam / 2));
    cd z = cmul_i(mk(kTwoPi * f, -wi)) / (kTwoPi * ref_freq(m));
    return c0 * cexp_(gam * clog_(z));
}

// ---------------------------------------------------------------- Dunkin --
//
// Minor order n <-> row pair: 0:(0,1) 1:(0,2) 2:(0,3) 3:(1,2) 4:(1,3) 5:(2,3)
// (propmat.go:168-174). Each layer's eigen-basis is F = [pd, g, pu, h]:
//   pd, pu = P eigenvectors (fk.go:158-159)
//   g = (sd - rb pd)/eb = (0, -u1, -mu' x2,  mu' rb)
//   h = (su + rb pu)/eb = (0, -u1, -mu' x2, -mu' rb)
// with eb = c^2/beta^2 = 1 - rb^2, u1 = (1 - ra rb)/eb, x2 = (1 + rb^2 - 2 ra rb)/eb
// and mu' = rho beta^2/mu_ref. In F the system matrix is block upper
// triangular, T = [[-ra, tau, 0, 0], [0, -rb, 0, 0], [0, 0, ra, tau], [0, 0, 0, rb]],
// tau = rb (ra - rb)/eb, so the layer's compound C(F) C(exp(-T k h)) C(F)^-1
// is closed form with no 0/0 as c -> 0 and a single growth exp((ra + rb) k h),
// divided out: C(exp(-T zeta)) = 1 (+) (P Y Q^T on the middle four minors)
// (+) (Ea Eb)^2, with Ea = exp(-ra zeta), Eb = exp(-rb zeta),
// P = [[Eb, -W], [0, Ea]], Q = [[Ea, -W], [0, Eb]], W = rb (Eb - Ea)/eb.
//
// The basis changes are applied in factored form:
//
// 1. F = G S with S a constant matrix of +-1 (pd = c0 - c1, g = c2 + c3,
//    pu = c0 + c1, h = c2 - c3) and
//      c0 = (1, 0, 0, mu'(1 + rb^2)),  c1 = (0, ra, 2 mu' ra, 0),
//      c2 = (0, -u1, -mu' x2, 0),      c3 = (0, 0, 0, mu' rb),
//    so G is block diagonal on the row sets {0, 3} and {1, 2}:
//      B03 = [[1, 0], [mu'(1 + rb^2), mu' rb]],  B12 = [[ra, -u1], [2 mu' ra, -mu' x2]],
//    det B03 = mu' rb and det B12 = mu' ra (2 u1 - x2 = 1). The compound of a
//    block-diagonal matrix keeps the pure pairs (0,3) and (1,2) apart (scaled
//    by the block determinants) and maps the mixed minors, as the 2x2 matrix
//    V[a][b] = M_ab (a in {0,3}, b in {1,2}), to B03 V B12^T. C(S) has only
//    0, +-1 and +-2 entries, and C(S^-1) = C(S)^T / 4.
// 2. C(G)^-1 is applied as C(adj G) over det B03 det B12: the pure pairs
//    scale by det B12 and det B03, the mixed minors go to
//    adj(B03) V adj(B12)^T. det F and every other common scale cancel in the
//    surface ratio M_12/M_23.
// 3. The propagation keeps M_02 + M_13 = 0 (five independent minors, the
//    Dunkin reduction; checked to rounding on random stacks), so V is
//    symmetric, M_13 is never formed and five minors are carried.
// 4. u1, x2 and ra - rb have forms without cancellation through
//    A = 1/(1 + ra) and B = 1/(1 + rb) (|1 + r| >= 1 on the principal
//    branch): 1 - ra rb = ea A + eb B - ea eb A B gives
//      u1 = kap A + ra B,  ra - rb = eb (B - kap A),  x2 = 2 u1 - 1,
//    and r2 = ((1 + rb^2)^2 - 4 ra rb)/eb = 4 u1 - 4 + eb, with
//    kap = ea/eb = beta^2/alpha^2 <= 1/2. For |eb| >= 0.35 the direct forms
//    (1 - ra rb)/eb and (eb - ea)/(ra + rb) are used instead.
// Against the previous unfactored step this runs 26% fewer FP64 instructions
// per layer; against 40-3000-digit evaluations of the reference algorithm it
// is as accurate or better.

struct Terms {
    cd ra, rb, mu, u1, x2, delta, ieb, eb;
};

GFK_HD Terms layer_terms(const LayerC& L, cd c2) {
    Terms t;
    const cd ea = c2 * L.c[0];
    const cd eb = c2 * L.c[1];
    const cd kap = L.c[2];
    t.mu = L.c[3];
    t.eb = eb;
    t.ra = csqrt_fast(1.0 - ea);  // principal root: Re >= 0, the decaying branch
    t.rb = csqrt_fast(1.0 - eb);
    t.ieb = crcp_(eb);
    if (cnorm1(eb) < 0.35) {
        const cd A = crcp_(1.0 + t.ra), B = crcp_(1.0 + t.rb);
        const cd kA = kap * A;
        t.u1 = cmadd(t.ra, B, kA);
        t.delta = eb * (B - kA);
    } else {
        t.u1 = cnmadd(t.ra, t.rb, mk(1.0)) * t.ieb;
        t.delta = (eb - ea) * crcp_(t.ra + t.rb);
    }
    t.x2 = 2.0 * t.u1 - 1.0;
    return t;
}

// The five independent minors (M01, M02, M03, M12, M23) of a layer's two
// downward-decaying solutions pd ^ g (M13 = -M02).
GFK_HD void decaying_minors(const Terms& t, cd m[5]) {
    const cd mu = t.mu;
    const cd r2 = 4.0 * t.u1 - 4.0 + t.eb;
    m[0] = -t.u1;
    m[1] = -(mu * t.x2);
    m[2] = mu * t.rb;
    m[3] = -(mu * t.ra);
    m[4] = (mu * mu) * r2;
}

// One layer's step, the part that does not depend on the minors: the basis
// entries and the layer's exponentials over exp((ra + rb) zeta).
struct Step {
    cd ra, u1, mrb, mra, mx2, mq, Ea, Eb, W, EaEb2;
};

GFK_HD Step layer_step(const Terms& t, double zeta) {
    Step s;
    const cd rb = t.rb, mu = t.mu;
    s.ra = t.ra;
    s.u1 = t.u1;
    s.mrb = mu * rb;
    s.mra = mu * t.ra;
    s.mx2 = mu * t.x2;
    s.mq = mu * (2.0 - t.eb);  // 1 + rb^2 with rb^2 = 1 - eb exactly
    const cd Eb = cexp_(-(rb * zeta));
    const cd dz = t.delta * zeta;  // (ra - rb) zeta
    cd Ea, W;
    if (cnorm1(dz) < 0.5) {
        const cd e = Eb * cexpm1_(-dz);  // Ea - Eb without cancellation
        Ea = Eb + e;
        W = (rb * (-e)) * t.ieb;
    } else {
        Ea = cexp_(-(t.ra * zeta));
        W = (rb * (Eb - Ea)) * t.ieb;
    }
    s.Ea = Ea;
    s.Eb = Eb;
    s.W = W;
    const cd EaEb = Ea * Eb;
    s.EaEb2 = EaEb * EaEb;
    return s;
}

// m <- C(exp(-A zeta)) m up to a scalar: one layer, bottom to top, on the
// five minors (M01, M02, M03, M12, M23). With renorm the result is rescaled by
// a power of two (exact) so its largest part is in [1, 2); a layer changes the
// magnitude by a bounded factor, so callers rescale every few layers
// (kRenormEvery) and at the surface.
GFK_HD void apply_step(const Step& s, cd m[5], bool renorm) {
    const cd ra = s.ra, u1 = s.u1, mrb = s.mrb, mra = s.mra, mx2 = s.mx2, mq = s.mq;
    const cd Ea = s.Ea, Eb = s.Eb, W = s.W;
    const cd mra2 = 2.0 * mra;
    // v = C(adj G) m: pure pairs by the other block's determinant, mixed
    // V = [[M01, M02], [M02, -M23]] to adj(B03) V adj(B12)^T with
    // adj(B03) = [[mu' rb, 0], [-mu'(1 + rb^2), 1]], adj(B12) = [[-mu' x2, u1], [-2 mu' ra, ra]]
    const cd v03 = mra * m[2];
    const cd v12 = mrb * m[3];
    const cd T00 = cmul2_sub(u1, m[1], mx2, m[0]);
    const cd T01 = cmul2_sub(ra, m[1], mra2, m[0]);
    const cd nT10 = cmul2_add(mx2, m[1], u1, m[4]);
    const cd nT11 = cmul2_add(mra2, m[1], ra, m[4]);
    const cd v01 = mrb * T00;
    const cd v02 = mrb * T01;
    const cd v13 = cmadd(mq, T00, nT10);
    const cd v23 = cmadd(mq, T01, nT11);
    // y = C(S)^T v (F-basis pairs)
    const cd sab = v02 - v13, pab = v02 + v13, scd = v03 - v12, pcd = v03 + v12;
    const cd y0 = sab + scd;
    const cd y1 = 2.0 * v01;
    const cd y2 = pab - pcd;
    const cd y3 = -(pab + pcd);
    const cd y4 = -2.0 * v23;
    const cd y5 = sab - scd;
    // middle minors Z = P Y Q^T, Y = [[y1, y2], [y3, y4]]; the outer pairs
    // scale by 1 and (Ea Eb)^2
    const cd p00 = cmul2_sub(Eb, y1, W, y3), p01 = cmul2_sub(Eb, y2, W, y4);
    const cd p10 = Ea * y3, p11 = Ea * y4;
    const cd z1 = cmul2_sub(Ea, p00, W, p01);
    const cd z2 = Eb * p01;
    const cd z3 = cmul2_sub(Ea, p10, W, p11);
    const cd z4 = Eb * p11;
    // w = C(S) z (G-basis pairs)
    const cd s05 = cmadd(s.EaEb2, y5, y0), d05 = cnmadd(s.EaEb2, y5, y0);  // y0 +- z5
    const cd s23 = z2 + z3, d23 = z2 - z3;
    const cd w01 = 2.0 * z1;
    const cd w02 = s05 + d23;
    const cd w03 = d05 - s23;
    const cd w12 = -(d05 + s23);
    const cd w13 = d23 - s05;
    const cd w23 = -2.0 * z4;
    // m = C(G) w: pure pairs by the block determinants, mixed
    // [[w01, w02], [-w13, -w23]] to B03 (.) B12^T (its (3,1) entry, -M13, not formed)
    const cd U00 = cmul2_sub(ra, w01, u1, w02);
    const cd U01 = cmul2_sub(mra2, w01, mx2, w02);
    const cd U11 = cmul2_sub(mx2, w23, mra2, w13);
    m[0] = U00;
    m[1] = U01;
    m[2] = mrb * w03;
    m[3] = mra * w12;
    m[4] = -cmul2_add(mq, U01, mrb, U11);
    // renormalise by a power of two (exact; the common scale cancels)
    if (!renorm) return;
    double mx = 0.0;
#pragma unroll
    for (int i = 0; i < 5; i++) mx = fmax(mx, cnorm1(m[i]));
    if (mx > 0.0 && mx < INFINITY) {
        const double sc = pow2i(-ilogb(mx));
#pragma unroll
        for (int i = 0; i < 5; i++) m[i] = m[i] * sc;
    }
}

GFK_HD void dunkin_layer_up(const Terms& t, double zeta, cd m[5], bool renorm = true) {
    apply_step(layer_step(t, zeta), m, renorm);
}

// Thick-layer start. Through a finite layer whose P and S factors
// exp(-Re(ra) k h) and exp(-Re(rb) k h) are both below e^-kThick, the
// minors leave as z0 C(F) e0 plus terms carrying products of two such
// factors (z1..z5 in dunkin_layer_up). C(F) e0 is the layer's own decaying
// minors, so above that layer the minors are those of a half-space of its
// material up to scale, to ~e^(-2 kThick) relative, and the layers beneath it
// cannot reach the surface in FP64. Propagation therefore starts at the
// shallowest such layer. Re(sqrt(1 - e)) >= sqrt(Re(1 - e)) gives a cheap
// sufficient test without the square roots. Against the full propagation on
// the graded, single and 40 seeded uneven soils the difference stays at
// rounding level down to kThick = 20; below that it grows as C e^(-2 kThick)
// with C = 260-550 at kThick = 8-12 (rising slowly with kThick). On 90,000
// random (stack, frequency, wavenumber) points (2-12 layers, Q 10-1200,
// real and complex frequencies) the differences from the full propagation
// have the same mean (1.9e-16) and 99th percentile (8e-16) at every
// threshold from 20 to 32 — rounding — and grow at 18 (mean 3x, 99.99th
// percentile 40x). 23 keeps five units of margin above that onset; the
// neglected part, ~C e^-46, is ~1e-17 relative.
constexpr double kThick = 23.0;

// Layers between power-of-two rescalings of the minor vector (the scale is
// exact and cancels, so the result does not depend on it while nothing
// overflows; one layer changes the magnitude by far less than 2^64).
constexpr int kRenormEvery = 4;

GFK_HD bool thick_layer(const LayerC& L, cd c2, double zeta) {
    const double pa = 1.0 - (c2.re * L.c[0].re - c2.im * L.c[0].im);  // Re(1 - ea)
    const double pb = 1.0 - (c2.re * L.c[1].re - c2.im * L.c[1].im);  // Re(1 - eb)
    return fmin(pa, pb) * (zeta * zeta) > kThick * kThick;
}

// The layer the upward propagation starts from: the shallowest thick finite
// layer, else the half-space.
GFK_HD int start_layer(const LayerC* L, int n, cd c2, double k) {
    for (int i = 0; i < n - 1; i++)
        if (thick_layer(L[i], c2, k * L[i].h)) return i;
    return n - 1;
}

// Surface vertical displacement per newton (fk.go:276-327) by minor
// propagation: u_z = i b4 M_12/M_23 with b4 = -i/(2 pi mu_ref k).
GFK_HD cd dunkin_u(const LayerC* L, int n, cd wc2, double k, double mu_ref) {
    const cd c2 = wc2 * rcp_(k * k);
    const int top = start_layer(L, n, c2, k);
    cd m[5];
    {
        Terms t = layer_terms(L[top], c2);
        decaying_minors(t, m);
    }
    for (int i = top - 1; i >= 0; i--) {
        Terms t = layer_terms(L[i], c2);
        dunkin_layer_up(t, k * L[i].h, m, i % kRenormEvery == 0);
    }
    // the minors end rescaled into [1, 2), so |denominator|^2 stays in range
    // for one real reciprocal
    return cdiv_fast(m[3], (kTwoPi * mu_ref * k) * m[4]);
}

// ------------------------------------------------------ reference direct --

struct M4 {
    cd a[4][4];
};

// cmat.solve (cmat.go:57-96): Gaussian elimination with partial pivoting.
__device__ __forceinline__ bool m4_solve(M4 m, cd x[4], cd out[4]) {
#pragma unroll
    for (int col = 0; col < 4; col++) {
        double best = 0.0;
        int brow = col;
#pragma unroll
        for (int r = col; r < 4; r++) {
            double v = cabs_(m.a[r][col]);
            if (v > best) { best = v; brow = r; }
        }
        if (best == 0.0) return false;
#pragma unroll
        for (int r = col + 1; r < 4; r++) {
            if (r == brow) {
#pragma unroll
                for (int c = 0; c < 4; c++) { cd t = m.a[col][c]; m.a[col][c] = m.a[r][c]; m.a[r][c] = t; }
                cd t = x[col]; x[col] = x[r]; x[r] = t;
            }
        }
        const cd p = m.a[col][col];
#pragma unroll
        for (int r = col + 1; r < 4; r++) {
            const cd f = m.a[r][col] / p;
            if (f.re == 0.0 && f.im == 0.0) continue;
#pragma unroll
            for (int c = col; c < 4; c++) m.a[r][c] -= f * m.a[col][c];
            x[r] -= f * x[col];
        }
    }
#pragma unroll
    for (int i = 3; i >= 0; i--) {
        cd s = x[i];
#pragma unroll
        for (int j = i + 1; j < 4; j++) s -= m.a[i][j] * out[j];
        out[i] = s / m.a[i][i];
    }
    return true;
}

// The inverse as fk.go:195-213 takes it: one solve per unit vector. The four
// solves share the matrix, so its elimination runs once for the four
// right-hand sides: the operations on each are m4_solve's, in its order.
__device__ __forceinline__ bool m4_inverse(M4 m, M4& x) {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) x.a[i][j] = mk(i == j ? 1.0 : 0.0);
#pragma unroll
    for (int col = 0; col < 4; col++) {
        double best = 0.0;
        int brow = col;
#pragma unroll
        for (int r = col; r < 4; r++) {
            const double v = cabs_(m.a[r][col]);
            if (v > best) { best = v; brow = r; }
        }
        if (best == 0.0) return false;
#pragma unroll
        for (int r = col + 1; r < 4; r++) {
            if (r == brow) {
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    cd t = m.a[col][c]; m.a[col][c] = m.a[r][c]; m.a[r][c] = t;
                    t = x.a[col][c]; x.a[col][c] = x.a[r][c]; x.a[r][c] = t;
                }
            }
        }
        const cd p = m.a[col][col];
#pragma unroll
        for (int r = col + 1; r < 4; r++) {
            const cd f = m.a[r][col] / p;
            if (f.re == 0.0 && f.im == 0.0) continue;
#pragma unroll
            for (int c = col; c < 4; c++) m.a[r][c] -= f * m.a[col][c];
#pragma unroll
            for (int c = 0; c < 4; c++) x.a[r][c] -= f * x.a[col][c];
        }
    }
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
        for (int i = 3; i >= 0; i--) {
            cd s = x.a[i][c];
#pragma unroll
            for (int j = i + 1; j < 4; j++) s -= m.a[i][j] * x.a[j][c];
            x.a[i][c] = s / m.a[i][i];
        }
    return true;
}

// props.eigen (fk.go:138-168): columns (P down, SV down, P up, SV up).
__device__ __forceinline__ void eigen4(const LayerC& L, double k, double omega, double mu_ref, cd lam[4], M4& e) {
    const cd alpha = L.c[0], beta = L.c[1], mu = L.c[2];
    const double rho = L.c[3].re;
    const double w2 = omega * omega;
    const double k2 = k * k;
    cd ra = csqrt_(1.0 - mk(w2) / ((k2 * alpha) * alpha));
    cd rb = csqrt_(1.0 - mk(w2) / ((k2 * beta) * beta));
    if (ra.re < 0) ra = -ra;
    if (rb.re < 0) rb = -rb;
    const double rc2 = rho * w2 / k2;
    const cd mr = mk(mu_ref);
    lam[0] = -ra; lam[1] = -rb; lam[2] = ra; lam[3] = rb;
    const cd two_mu_mr = (2.0 * mu) / mr;
    const cd p3 = (2.0 * mu - rc2) / mr;
    const cd s2 = (rc2 - 2.0 * mu) / mr;
    e.a[0][0] = mk(1.0);            e.a[0][1] = rb;               e.a[0][2] = mk(1.0);          e.a[0][3] = -rb;
    e.a[1][0] = -ra;                e.a[1][1] = mk(-1.0);         e.a[1][2] = ra;               e.a[1][3] = mk(-1.0);
    e.a[2][0] = -(two_mu_mr * ra);  e.a[2][1] = s2;               e.a[2][2] = two_mu_mr * ra;   e.a[2][3] = s2;
    e.a[3][0] = p3;                 e.a[3][1] = two_mu_mr * rb;   e.a[3][2] = p3;               e.a[3][3] = -(two_mu_mr * rb);
}

// Medium.SurfaceResponse restated (fk.go:276-327). ok = false where the
// reference reports a singular propagator or surface system.
__device__ __forceinline__ cd direct_u(const LayerC* L, int n, double omega, double k, double mu_ref, bool& ok) {
    M4 total;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) total.a[i][j] = mk(i == j ? 1.0 : 0.0);
    ok = true;
    for (int l = 0; l < n - 1; l++) {
        cd lam[4];
        M4 e;
        eigen4(L[l], k, omega, mu_ref, lam, e);
        const double zeta = k * L[l].h;
        double max_re = 0.0;
#pragma unroll
        for (int i = 0; i < 4; i++) max_re = fmax(max_re, lam[i].re);
        cd d[4];
#pragma unroll
        for (int i = 0; i < 4; i++) d[i] = cexp_((lam[i] - max_re) * zeta);
        M4 inv;
        if (!m4_inverse(e, inv)) { ok = false; return mk(0.0); }
        // p = (e d) inv; total = p total
        M4 p;
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                cd s = mk(0.0);
#pragma unroll
                for (int q = 0; q < 4; q++) s += (e.a[i][q] * d[q]) * inv.a[q][j];
                p.a[i][j] = s;
            }
        M4 nt;
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                cd s = mk(0.0);
#pragma unroll
                for (int q = 0; q < 4; q++) s += p.a[i][q] * total.a[q][j];
                nt.a[i][j] = s;
            }
        total = nt;
    }
    cd lam[4];
    M4 e;
    eigen4(L[n - 1], k, omega, mu_ref, lam, e);
    const cd b4 = mk(0.0, -1.0 / (kTwoPi * mu_ref * k));
    M4 a;
    cd rhs[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        a.a[i][0] = total.a[i][0];
        a.a[i][1] = total.a[i][1];
        a.a[i][2] = -e.a[i][0];
        a.a[i][3] = -e.a[i][1];
        rhs[i] = -(b4 * total.a[i][3]);
    }
    cd x[4];
    if (!m4_solve(a, rhs, x)) { ok = false; return mk(0.0); }
    return mk(x[1].im, -x[1].re);  // -i * x1
}

}  // namespace gfk
