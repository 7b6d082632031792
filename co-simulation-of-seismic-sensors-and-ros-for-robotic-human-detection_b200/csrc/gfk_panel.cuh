// gfk_panel.cuh — the integrand k u - C at 128 consecutive wavenumbers (a
// panel) from its values at 16 or 32 Chebyshev nodes.
//
// u(k) is analytic in k away from the surface-wave poles and the branch points
// k = w/alpha, w/beta of the layers. The wavenumber grid resolves the
// narrowest pole; over most of the grid (all of it past the slowest wave's
// k = w/0.87 Vs, and wherever the waves are damped) it oversamples the
// integrand many times, and a panel is a polynomial to rounding. So each panel
// is first evaluated at 16 nodes; if its last Chebyshev coefficients are at
// rounding level the panel is interpolated from them, else, where their decay
// says that twice the degree will do, at 16 more nodes; else every wavenumber
// is solved as before. A pole 1/(k - p) puts a tail on the coefficients of its
// whole neighbourhood (it decays as slowly as the pole is near), so a panel
// with a narrow pole between its nodes cannot pass.
//
// The 32 nodes are the Chebyshev points cos((j + 1/2) pi / 32); the first 16
// are the even j, whose Lebesgue constant is 3.6 (full set: 2.7). Measured on the
// CPU over 24 bins of the graded soil, 60 random uneven soils and 60 Sobol
// soils: against direct evaluation the interpolated values differ by 4e-16 (p50),
// 2e-15 (p99), 5e-15 (largest) of |C| + max|k u - C|; moving k by one ulp moves
// the direct values by 2e-16, 3e-15 and 7e-15. Solves per wavenumber
// weighted by their cost: 2.7x fewer on the graded soil, 1.7x on the uneven
// soils, 2.1x on the Sobol soils. 16 nodes serve 81-85% of the panels, 32
// another 5-12%. Panels of 256 with 32/16 nodes were within 12% of these; 64/32
// nodes save less.
#pragma once
#include <cmath>
#include <utility>
#include <vector>

#include "gfk_math.cuh"

namespace gfk {

constexpr int kPanel = 128;        // wavenumbers per panel
constexpr int kPanelE = 16;        // nodes of the first try
constexpr int kPanelN = 32;        // nodes of both
constexpr int kPanelLeast = 33;    // a shorter last panel is solved directly: no more solves than its second try
constexpr double kPanelTol = 1e-15;  // last coefficients against |C| + max |k u - C|

// Whether a panel may be interpolated: `tail` its largest last coefficient (infinite
// where one is not finite, which every node that is not makes it), `scale` |C| + max |k u - C|
// over its nodes. Strictly below: a node that overflowed makes both infinite, and a refused
// panel's wavenumbers are solved one by one and flagged there. (A test of the scale by itself
// cost 8 bytes of spills a thread, 1% of the Sobol rows' time.)
GFK_HD bool panel_passes(double tail, double scale) { return tail < kPanelTol * scale; }

// Offsets (doubles) into the table every context keeps on the device.
constexpr int kPtX = 0;                              // node abscissae, first 16 then the other 16
// coefficient rows as m8n8k4 A fragments [node/4][lane], lane = 4 row + node%4:
// rows 0-2 the last three coefficients, rows 3-5 (16-node fit) coefficients 7..9
constexpr int kPtRowsE = kPtX + kPanelN;
constexpr int kPtRowsN = kPtRowsE + 8 * kPanelE;
constexpr int kPtFragE = kPtRowsN + 8 * kPanelN;     // interpolation matrices as m8n8k4 A fragments:
constexpr int kPtFragN = kPtFragE + kPanel * kPanelE;  // [point/8][node/4][lane], lane = 4 (point%8) + node%4
constexpr int kPtSize = kPtFragN + kPanel * kPanelN;

GFK_HD int panel_frag(int point, int node, int nodes) {
    return ((point >> 3) * (nodes >> 2) + (node >> 2)) * 32 + 4 * (point & 7) + (node & 3);
}

// The table, in long double: the 16-node fit by its Lagrange polynomials and
// the inverse of its Chebyshev-Vandermonde matrix, the 32-node fit by the
// discrete orthogonality of the Chebyshev points.
inline std::vector<double> panel_table() {
    using L = long double;
    const L pi = 3.141592653589793238462643383279502884L;
    std::vector<double> t(kPtSize);
    L x[kPanelN];
    for (int j = 0; j < kPanelN; j++) {  // first the even Chebyshev points, then the odd ones
        const int c = j < kPanelE ? 2 * j : 2 * (j - kPanelE) + 1;
        x[j] = cosl((c + 0.5L) * pi / kPanelN);
        t[kPtX + j] = (double)x[j];
    }
    auto cheb = [](L v, L* out, int n) {
        out[0] = 1;
        out[1] = v;
        for (int m = 2; m < n; m++) out[m] = 2 * v * out[m - 1] - out[m - 2];
    };
    L T[kPanelN][kPanelN];
    for (int j = 0; j < kPanelN; j++) cheb(x[j], T[j], kPanelN);
    for (int c = 0; c < 3; c++)
        for (int j = 0; j < kPanelN; j++)
            t[kPtRowsN + (j >> 2) * 32 + 4 * c + (j & 3)] = (double)(2.0L / kPanelN * T[j][kPanelN - 3 + c]);
    // inverse of V[a][m] = T_m(x_a), a, m < 16 (Gauss-Jordan, partial pivoting)
    L V[kPanelE][2 * kPanelE];
    for (int a = 0; a < kPanelE; a++)
        for (int m = 0; m < kPanelE; m++) {
            V[a][m] = T[a][m];
            V[a][kPanelE + m] = a == m;
        }
    for (int c = 0; c < kPanelE; c++) {
        int p = c;
        for (int r = c + 1; r < kPanelE; r++)
            if (fabsl(V[r][c]) > fabsl(V[p][c])) p = r;
        for (int m = 0; m < 2 * kPanelE; m++) std::swap(V[c][m], V[p][m]);
        const L d = V[c][c];
        for (int m = 0; m < 2 * kPanelE; m++) V[c][m] /= d;
        for (int r = 0; r < kPanelE; r++) {
            if (r == c) continue;
            const L f = V[r][c];
            for (int m = 0; m < 2 * kPanelE; m++) V[r][m] -= f * V[c][m];
        }
    }
    for (int c = 0; c < 3; c++)
        for (int j = 0; j < kPanelE; j++) {
            t[kPtRowsE + (j >> 2) * 32 + 4 * c + (j & 3)] = (double)V[kPanelE - 3 + c][kPanelE + j];
            t[kPtRowsE + (j >> 2) * 32 + 4 * (c + 3) + (j & 3)] = (double)V[kPanelE - 9 + c][kPanelE + j];
        }
    for (int p = 0; p < kPanel; p++) {
        const L v = (2.0L * p - (kPanel - 1)) / kPanel;  // wavenumber a + 1 + p of a panel centred at a + 64.5
        L Tv[kPanelN];
        cheb(v, Tv, kPanelN);
        for (int j = 0; j < kPanelE; j++) {
            L l = 1;
            for (int b = 0; b < kPanelE; b++)
                if (b != j) l *= (v - x[b]) / (x[j] - x[b]);
            t[kPtFragE + panel_frag(p, j, kPanelE)] = (double)l;
        }
        for (int j = 0; j < kPanelN; j++) {
            L s = 0.5L;
            for (int m = 1; m < kPanelN; m++) s += T[j][m] * Tv[m];
            t[kPtFragN + panel_frag(p, j, kPanelN)] = (double)(2.0L / kPanelN * s);
        }
    }
    return t;
}

}  // namespace gfk
