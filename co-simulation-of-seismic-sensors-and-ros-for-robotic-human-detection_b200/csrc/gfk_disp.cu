// gfk_disp.cu — Rayleigh dispersion curves on the GPU: the secular function of
// internal/propmat and the bracketing root search of internal/disp, a
// scan of every (frequency, velocity) and one block per frequency for the roots.
//
// Secular (propmat.go:82-315), in FP64 per (f, c): for every finite layer the
// dimensionless 4x4 system matrix A (SystemMatrix), its exponential over the
// layer shifted by the largest vertical-P growth so it stays bounded
// (LayerPropagator), that matrix's 6x6 second compound applied to the minor
// vector of the free-surface two-plane and renormalised to max |m| = 1, then
// the generalised Laplace expansion against the half-space's closed-form
// decaying minors. The scale factors are positive and are dropped, as the
// reference does. The exponential is closed form: A couples (u_x, s_zz) with
// (u_z, s_xz) only, so exp(z A) is made of cosh(z sqrt(M)) and sinh(z sqrt(M))/
// sqrt(M) of the 2x2 products M = B C, C B of its blocks, which by
// Cayley-Hamilton are c0 + c1 M and s0 + s1 M with divided differences over M's
// eigenvalues ra^2 = 1 - c^2/alpha^2 and rb^2 = 1 - c^2/beta^2 (layer_functions).
// About 230 FP64 operations a layer; scaling and squaring with a degree-16
// Taylor polynomial took about 2800 and bounded the root search (2.6 ms of 3.3
// on 512 frequencies of a ten-layer soil, every mode).
//
// Modes (disp.go:62-103, bisect disp.go:194-217): the secular function on
// samples + 1 evenly spaced velocities in [0.85 Vs_min, Vs_halfspace (1 - 1e-9)]
// (k_scan), the sign changes between defined neighbours in order, and one bisection per bracket (a group of lanes each, evaluating
// several steps' midpoints at once, below) with the reference's stopping
// rules; a bracket whose bisection meets an undefined value yields no root, as
// in the reference.
#include <algorithm>
#include <cmath>
#include <vector>

#include <math_constants.h>

#include "../../include/gfk.h"
#include "gfk_ctx.h"
#include "gfk_kernels.cuh"

namespace gfk {
namespace disp {

constexpr int kMaxLayers = 64;
constexpr int kThreads = 128;
constexpr int kMaxModes = 64;
constexpr int kMaxSamples = 16384;

// One layer of the dimensionless system matrix (propmat.go:82-106), what does
// not depend on the phase velocity c: A[0][2] = p, A[1][0] = q = -A[2][3],
// A[1][3] = r, A[2][0] = s - t c^2, A[3][1] = -t c^2.
struct LayerK {
    double h, ia2, ib2, p, q, r, s, t;
};

struct Stack {
    LayerK l[kMaxLayers];  // the finite layers
    int n;                 // entries including the half-space
    double mu_ref;         // referenceModulus (propmat.go:109-115)
    double hvp, hvs, hrho;
};

// c0 + c1 M = cosh(z sqrt(M)) and s0 + s1 M = sinh(z sqrt(M))/sqrt(M) for a
// 2x2 M with eigenvalues A = ra^2 > B = rb^2 (negative where the wave
// propagates), both over exp(z Re ra), the layer's largest growth:
//   c1 = (cosh z ra - cosh z rb)/(A - B),  s1 likewise with sinh(z r)/r.
// Where z^2 |A|, z^2 |B| <= 1, by their power series (divided differences of
// powers by recurrence); where A - B < 1/4 (then rb > 0.7), by products of
// functions of half the sum and half the difference of z ra and z rb, free of
// cancellation; else as written.
__device__ __forceinline__ void layer_functions(double A, double B, double z, double& c0, double& c1, double& s0,
                                                double& s1) {
    const double u = z * z, D = A - B;
    double Cb, Sb;
    if (u * fmax(fabs(A), fabs(B)) <= 1.0) {
        const double a = u * A, b = u * B;
        // 1/(2n)! and 1/(2n + 1)!; h_n = sum_i a^i b^(n - i)
        const double ic[11] = {1.0, 1.0 / 2, 1.0 / 24, 1.0 / 720, 1.0 / 40320, 1.0 / 3628800, 1.0 / 479001600,
                               1.0 / 87178291200.0, 1.0 / 20922789888000.0, 1.0 / 6402373705728000.0,
                               1.0 / 2432902008176640000.0};
        double bn = 1.0, h = 0.0, cs = 0.0, ss = 0.0, cb = 1.0, sb = 1.0;
#pragma unroll
        for (int n = 1; n <= 10; n++) {
            h = fma(a, h, bn);  // h_(n - 1)
            bn *= b;
            const double c = ic[n], d = ic[n] / (2 * n + 1);
            cs = fma(c, h, cs);
            ss = fma(d, h, ss);
            cb = fma(c, bn, cb);
            sb = fma(d, bn, sb);
        }
        const double e = A > 0.0 ? exp(-z * sqrt(A)) : 1.0;
        c1 = e * u * cs;
        s1 = e * z * u * ss;
        Cb = e * cb;
        Sb = e * z * sb;
    } else if (D < 0.25 && B > 0.0) {
        const double ra = sqrt(A), rb = sqrt(B), sum = ra + rb;
        const double S2 = z * sum, d2 = z * D / sum;  // twice the half sum and half difference
        const double eS = expm1(-S2), ed = expm1(-d2);
        const double shS = -0.5 * eS, chS = 1.0 + 0.5 * eS, shd = -0.5 * ed, chd = 1.0 + 0.5 * ed;  // over their growth
        const double hS = 2.0 * shS / S2, hd = d2 > 0.0 ? 2.0 * shd / d2 : 1.0;
        c1 = 0.5 * u * hS * hd;
        s1 = z * (chS * hd - hS * chd) / (2.0 * ra * rb);
        Cb = chS * chd - shS * shd;
        Sb = (shS * chd - chS * shd) / rb;
    } else {
        double Ca, Sa, shift = 0.0;
        if (A > 0.0) {
            const double r = sqrt(A), e = expm1(-2.0 * z * r);
            shift = z * r;
            Ca = 1.0 + 0.5 * e;
            Sa = -0.5 * e / r;
        } else {
            const double r = sqrt(-A);
            double sn, cs;
            sincos(z * r, &sn, &cs);
            Ca = cs;
            Sa = r > 0.0 ? sn / r : z;
        }
        if (B > 0.0) {
            const double r = sqrt(B), e = expm1(-2.0 * z * r), g = exp(z * r - shift);
            Cb = (1.0 + 0.5 * e) * g;
            Sb = -0.5 * e * g / r;
        } else {
            const double r = sqrt(-B), g = exp(-shift);
            double sn, cs;
            sincos(z * r, &sn, &cs);
            Cb = g * cs;
            Sb = g * (r > 0.0 ? sn / r : z);
        }
        c1 = (Ca - Cb) / D;
        s1 = (Sa - Sb) / D;
    }
    c0 = fma(-B, c1, Cb);
    s0 = fma(-B, s1, Sb);
}

// propmat.Secular; false where the reference returns an error. Not inlined:
// the scan, the bisection and the pointwise call run the same instructions.
__device__ __noinline__ bool secular(const Stack& st, double omega, double k, double* out) {
    if (!(k > 0.0) || !(omega > 0.0)) return false;
    const double c2 = (omega * omega) / (k * k);
    // minors 0:(0,1) 1:(0,2) 2:(0,3) 3:(1,2) 4:(1,3) 5:(2,3); the layers keep
    // M_02 + M_13 = 0 (the Dunkin reduction), so the fifth is not carried
    double m0 = 1.0, m1 = 0.0, m2 = 0.0, m3 = 0.0, m5 = 0.0;
    for (int li = 0; li + 1 < st.n; li++) {
        const LayerK L = st.l[li];
        const double z = k * L.h;
        double c0, c1, s0, s1;
        layer_functions(fma(-c2, L.ia2, 1.0), fma(-c2, L.ib2, 1.0), z, c0, c1, s0, s1);
        const double a20 = fma(-L.t, c2, L.s), tc = L.t * c2;
        // B = [[-1, p], [-tc, 1]] on (x1, x2) -> (x0, x3); C = [[q, r], [a20, -q]]
        const double q = L.q, r = L.r, p = L.p;
        const double n00 = fma(p, a20, -q), n01 = -fma(p, q, r);          // B C
        const double n10 = fma(-tc, q, a20), n11 = -fma(tc, r, q);
        const double k00 = -fma(r, tc, q), k01 = fma(q, p, r);            // C B
        const double k10 = fma(q, tc, -a20), k11 = fma(a20, p, -q);
        const double E00 = fma(c1, n00, c0), E01 = c1 * n01, E10 = c1 * n10, E11 = fma(c1, n11, c0);
        const double F00 = fma(c1, k00, c0), F01 = c1 * k01, F10 = c1 * k10, F11 = fma(c1, k11, c0);
        const double f00 = fma(s1, k00, s0), f01 = s1 * k01, f10 = s1 * k10, f11 = fma(s1, k11, s0);
        const double e00 = fma(s1, n00, s0), e01 = s1 * n01, e10 = s1 * n10, e11 = fma(s1, n11, s0);
        const double G00 = fma(p, f10, -f00), G01 = fma(p, f11, -f01);    // B (s0 + s1 C B)
        const double G10 = fma(-tc, f00, f10), G11 = fma(-tc, f01, f11);
        const double H00 = fma(q, e00, r * e10), H01 = fma(q, e01, r * e11);  // C (s0 + s1 B C)
        const double H10 = fma(a20, e00, -q * e10), H11 = fma(a20, e01, -q * e11);
        // rows of P: 0 (E00, G00, G01, E01), 1 (H00, F00, F01, H01), 2 (H10, F10, F11, H11), 3 (E10, G10, G11, E11)
        auto row = [&](double i0, double i1, double i2, double i3, double j0, double j1, double j2, double j3) {
            double v = fma(i0, j1, -i1 * j0) * m0;
            v = fma(fma(i0, j2, -i2 * j0) - fma(i1, j3, -i3 * j1), m1, v);
            v = fma(fma(i0, j3, -i3 * j0), m2, v);
            v = fma(fma(i1, j2, -i2 * j1), m3, v);
            return fma(fma(i2, j3, -i3 * j2), m5, v);
        };
        const double x0 = row(E00, G00, G01, E01, H00, F00, F01, H01);
        const double x1 = row(E00, G00, G01, E01, H10, F10, F11, H11);
        const double x2 = row(E00, G00, G01, E01, E10, G10, G11, E11);
        const double x3 = row(H00, F00, F01, H01, H10, F10, F11, H11);
        const double x5 = row(H10, F10, F11, H11, E10, G10, G11, E11);
        const double norm = fmax(fmax(fmax(fabs(x0), fabs(x1)), fmax(fabs(x2), fabs(x3))), fabs(x5));
        if (norm == 0.0) return false;
        const double inv = 1.0 / norm;
        m0 = x0 * inv;
        m1 = x1 * inv;
        m2 = x2 * inv;
        m3 = x3 * inv;
        m5 = x5 * inv;
    }
    if (omega / k >= st.hvs) return false;
    const double a_ = sqrt(fmax(0.0, 1.0 - c2 / (st.hvp * st.hvp))), b_ = sqrt(fmax(0.0, 1.0 - c2 / (st.hvs * st.hvs)));
    const double mu = st.hrho * st.hvs * st.hvs / st.mu_ref;
    const double rc2 = st.hrho * c2 / st.mu_ref;
    const double pv[4] = {1.0, -a_, -2.0 * mu * a_, 2.0 * mu - rc2};
    const double sv[4] = {b_, -1.0, rc2 - 2.0 * mu, 2.0 * mu * b_};
    const double m[6] = {m0, m1, m2, m3, -m1, m5}, sign[6] = {1, -1, 1, 1, -1, 1};
    const int pi_[6] = {0, 0, 0, 1, 1, 2}, pj_[6] = {1, 2, 3, 2, 3, 3};
    double f = 0.0;
#pragma unroll
    for (int n = 0; n < 6; n++) {
        const int c = 5 - n;  // complement pair
        const double e = pv[pi_[c]] * sv[pj_[c]] - pv[pj_[c]] * sv[pi_[c]];
        f += sign[n] * m[n] * e;
    }
    *out = f;
    return true;
}

__device__ inline bool secular_c(const Stack& st, double freq, double c, double* out) {
    const double omega = 2.0 * 3.14159265358979323846 * freq;
    double v;
    if (!secular(st, omega, omega / c, &v) || isnan(v) || isinf(v)) return false;
    *out = v;
    return true;
}

__device__ inline bool sign_change(double a, double b) { return (a < 0.0 && b > 0.0) || (a > 0.0 && b < 0.0); }

struct ModeArgs {
    const double* freqs;
    int nf, samples, max_modes;
    double tol, lo, hi;
    double* vals;  // [nf][samples + 1] the scan's values, NaN where undefined
    double* vel;   // [nf][max_modes]
    int* count;    // [nf]; -1 - found when more than max_modes
};

// The scan's velocities with one rounding per operation (no contraction into
// FMAs), so the host can form the very same doubles: lo + i step.
__device__ __forceinline__ double scan_step(const ModeArgs& a) {
    return __dsub_rn(__dmul_rn(a.hi, 1.0 - 1e-9), a.lo) / a.samples;
}
__device__ __forceinline__ double scan_velocity(const ModeArgs& a, double step, int i) {
    return i == 0 ? a.lo : __dadd_rn(a.lo, __dmul_rn((double)i, step));
}

// The scan, one thread per (frequency, velocity): its own launch, so that one
// frequency's 2001 evaluations spread over 16 blocks and 512 frequencies fill
// every SM evenly (a block per frequency left 3 or 4 blocks an SM).
__global__ void __launch_bounds__(kThreads) k_scan(const __grid_constant__ Stack st, ModeArgs a) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i > a.samples) return;
    double v;
    if (!secular_c(st, a.freqs[blockIdx.y], scan_velocity(a, scan_step(a), i), &v)) v = CUDART_NAN;
    a.vals[(size_t)blockIdx.y * (a.samples + 1) + i] = v;
}

__global__ void __launch_bounds__(kThreads) k_modes(const __grid_constant__ Stack st, ModeArgs a) {
    __shared__ int br[kMaxModes + 1], found[kThreads / 32][kMaxModes], nfound[kThreads / 32];
    __shared__ double root[kMaxModes];
    const int fi = blockIdx.x;
    const double freq = a.freqs[fi];
    const double step = scan_step(a);
    const double* vals = a.vals + (size_t)fi * (a.samples + 1);
    // the sign changes in order: each warp takes a contiguous stretch of the
    // samples, 32 at a time, then the warps' lists are put one after the other
    {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int per = (a.samples + kThreads / 32 - 1) / (kThreads / 32);
        const int i0 = 1 + warp * per, i1 = min(i0 + per, a.samples + 1);
        int n = 0;
        for (int at = i0; at < i1; at += 32) {
            const int i = at + lane;
            const bool hit = i < i1 && sign_change(vals[i - 1], vals[i]);  // false for a NaN
            const unsigned b = __ballot_sync(0xffffffffu, hit);
            const int k = n + __popc(b & ((1u << lane) - 1));
            if (hit && k < kMaxModes) found[warp][k] = i;
            n += __popc(b);
        }
        if (lane == 0) nfound[warp] = n;
    }
    __syncthreads();
    int nbr = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; w++) {
        for (int k = threadIdx.x; k < nfound[w] && k < kMaxModes && nbr + k < kMaxModes; k += kThreads)
            br[nbr + k] = found[w][k];
        nbr += nfound[w];
    }
    __syncthreads();
    const int nb = nbr < kMaxModes ? nbr : kMaxModes;
    // Bisection, `depth` steps per round: the 2^depth - 1 lanes of a group
    // evaluate every midpoint the next `depth` steps could visit (a complete
    // binary tree of brackets, each computed by the same halvings the
    // sequential search would make), then each lane walks the path the
    // sequential search takes through them. The midpoints, the decisions and
    // the stopping rules are those of the one-thread search, so the roots are
    // the same doubles; the dependent chain is `depth` times shorter. Few
    // brackets leave lanes for four steps a round.
    const int depth = nb <= kThreads / 16 ? 4 : 3, lanes = 1 << depth;
    const int lane = threadIdx.x & 31, grp = lane / lanes, node = lane % lanes;
    const int groups = (blockDim.x / 32) * (32 / lanes);
    const int gid = (threadIdx.x / 32) * (32 / lanes) + grp;
    for (int b0 = 0; b0 < nb; b0 += groups) {
        const int b = b0 + gid;
        const bool active = b < nb;
        double lo = 0.0, hi = 0.0, flo = 0.0, r = -1.0;
        bool done = !active;
        if (active) {
            const int i = br[b];
            lo = scan_velocity(a, step, i - 1);
            hi = scan_velocity(a, step, i);
            flo = vals[i - 1];  // the scan's value at this very velocity (defined: a bracket end)
        }
        int it = 0;
        while (__any_sync(0xffffffffu, !done)) {
            // this lane's tree node: heap index h = node + 1 at depth floor(log2 h)
            double v = 0.0;
            int vok = 0;
            if (!done && node < lanes - 1) {
                const int h = node + 1, d = 31 - __clz(h);
                double nlo = lo, nhi = hi;
                for (int sh = d - 1; sh >= 0; sh--) {
                    const double mid = 0.5 * (nlo + nhi);
                    if ((h >> sh) & 1) nlo = mid; else nhi = mid;
                }
                vok = secular_c(st, freq, 0.5 * (nlo + nhi), &v) ? 1 : 0;
            }
            int h = 1;
            for (int step_ = 0; step_ < depth; step_++) {
                const int src = (lane & ~(lanes - 1)) + (h - 1);
                const double hv = __shfl_sync(0xffffffffu, v, src);
                const int hok = __shfl_sync(0xffffffffu, vok, src);
                if (done) continue;
                if (it >= 200) {
                    r = 0.5 * (lo + hi);
                    done = true;
                    continue;
                }
                const double mid = 0.5 * (lo + hi);
                if (mid == lo || mid == hi || (hi - lo) < a.tol * mid) {
                    r = mid;
                    done = true;
                    continue;
                }
                it++;
                if (!hok) {
                    done = true;  // undefined inside the bracket: no root
                    continue;
                }
                if (sign_change(flo, hv)) {
                    hi = mid;
                    h = 2 * h;
                } else {
                    lo = mid;
                    flo = hv;
                    h = 2 * h + 1;
                }
            }
        }
        if (active && node == 0) root[b] = r;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int n = 0;
        for (int b = 0; b < nb; b++)
            if (root[b] > 0.0) {
                if (n < a.max_modes) a.vel[(size_t)fi * a.max_modes + n] = root[b];
                n++;
            }
        a.count[fi] = (nbr > kMaxModes || n > a.max_modes) ? -1 - n : n;
    }
}

__global__ void k_secular(const __grid_constant__ Stack st, const double* f, const double* c, long long n,
                          double* out, int* ok) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v = 0.0;
    ok[i] = secular_c(st, f[i], c[i], &v) ? 1 : 0;
    out[i] = v;
}

}  // namespace disp
}  // namespace gfk

namespace {

int dfail(gfk_ctx* ctx, int status, const std::string& msg) {
    if (ctx) ctx->last_error = msg;
    return status;
}

#define DS_CUDA(ctx, call)                                                                         \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return dfail(ctx, e_ == cudaErrorMemoryAllocation ? GFK_ENOMEM : GFK_ECUDA,            \
                         std::string(#call ": ") + cudaGetErrorString(e_));                        \
    } while (0)

int make_stack(gfk_ctx* ctx, const gfk_medium* m, gfk::disp::Stack* st) {
    if (!m || !m->layers || m->count < 1) return dfail(ctx, GFK_ESTACK, "layer: empty stack");
    const int v = gfk_stack_validate(m);
    if (v != GFK_OK) return dfail(ctx, v, "layer: stack failed validation");
    if (m->count > gfk::disp::kMaxLayers) return dfail(ctx, GFK_ELIMIT, "disp: more than 64 stack entries");
    st->n = m->count;
    st->mu_ref = 0.0;
    for (int i = 0; i < m->count; i++) {
        const gfk_layer& l = m->layers[i];
        st->mu_ref = std::max(st->mu_ref, l.density_kgm3 * l.vs_mps * l.vs_mps);
    }
    for (int i = 0; i + 1 < m->count; i++) {
        const gfk_layer& l = m->layers[i];
        const double mu = l.density_kgm3 * l.vs_mps * l.vs_mps, lam = l.density_kgm3 * l.vp_mps * l.vp_mps - 2.0 * mu;
        const double l2m = lam + 2.0 * mu;
        st->l[i] = gfk::disp::LayerK{l.thickness_m, 1.0 / (l.vp_mps * l.vp_mps), 1.0 / (l.vs_mps * l.vs_mps),
                                     st->mu_ref / mu, lam / l2m, st->mu_ref / l2m,
                                     4.0 * mu * (lam + mu) / l2m / st->mu_ref, l.density_kgm3 / st->mu_ref};
    }
    const gfk_layer& hs = m->layers[m->count - 1];
    st->hvp = hs.vp_mps;
    st->hvs = hs.vs_mps;
    st->hrho = hs.density_kgm3;
    return GFK_OK;
}

struct DBuf {
    gfk_ctx* ctx;
    void* p = nullptr;
    ~DBuf() {
        if (p) cudaFreeAsync(p, ctx->stream);
    }
};

}  // namespace

extern "C" {

int gfk_dispersion_modes(gfk_ctx* ctx, const gfk_medium* m, const double* freqs, int32_t nf, gfk_search opt,
                         int32_t max_modes, double* velocities, int32_t* counts) {
    if (!ctx || !m || !freqs || !velocities || !counts) return GFK_EARG;
    if (nf < 0 || max_modes < 1 || max_modes > gfk::disp::kMaxModes)
        return dfail(ctx, GFK_EARG, "disp: max_modes must lie in [1, 64]");
    gfk::disp::Stack st;
    int s0 = make_stack(ctx, m, &st);
    if (s0) return s0;
    for (int i = 0; i < nf; i++)
        if (!(freqs[i] > 0)) {
            char buf[96];
            snprintf(buf, sizeof buf, "disp: frequency must be positive, got %g Hz", freqs[i]);
            return dfail(ctx, GFK_EARG, buf);
        }
    const int samples = opt.samples > 0 ? opt.samples : 2000;
    const double tol = opt.tolerance > 0 ? opt.tolerance : 1e-10;
    if (samples > gfk::disp::kMaxSamples) return dfail(ctx, GFK_ELIMIT, "disp: at most 16384 samples");
    if (nf == 0) return GFK_OK;
    double vmin = m->layers[0].vs_mps;
    for (int i = 0; i < m->count; i++) vmin = std::min(vmin, m->layers[i].vs_mps);
    const double lo = 0.85 * vmin, hi = m->layers[m->count - 1].vs_mps;  // disp.go:62-65
    cudaSetDevice(ctx->device);
    cudaStream_t s = ctx->stream;
    DBuf d_f{ctx}, d_v{ctx}, d_c{ctx}, d_s{ctx};
    DS_CUDA(ctx, cudaMallocAsync(&d_f.p, sizeof(double) * nf, s));
    DS_CUDA(ctx, cudaMallocAsync(&d_v.p, sizeof(double) * nf * max_modes, s));
    DS_CUDA(ctx, cudaMallocAsync(&d_c.p, sizeof(int) * nf, s));
    DS_CUDA(ctx, cudaMemcpyAsync(d_f.p, freqs, sizeof(double) * nf, cudaMemcpyHostToDevice, s));
    // the scan's values, up to 64 MB of them (or one frequency's) at a time
    const int chunk = (int)std::max<size_t>(1, std::min<size_t>({(size_t)nf, (size_t(64) << 20) / (sizeof(double) * (samples + 1)),
                                                                 (size_t)65535}));
    DS_CUDA(ctx, cudaMallocAsync(&d_s.p, sizeof(double) * (samples + 1) * chunk, s));
    for (int f0 = 0; f0 < nf; f0 += chunk) {
        const int n = std::min(chunk, nf - f0);
        gfk::disp::ModeArgs a{static_cast<const double*>(d_f.p) + f0, n, samples, max_modes, tol, lo, hi,
                              static_cast<double*>(d_s.p), static_cast<double*>(d_v.p) + (size_t)f0 * max_modes,
                              static_cast<int*>(d_c.p) + f0};
        gfk::disp::k_scan<<<dim3(samples / gfk::disp::kThreads + 1, n), gfk::disp::kThreads, 0, s>>>(st, a);
        gfk::disp::k_modes<<<n, gfk::disp::kThreads, 0, s>>>(st, a);
        ctx->launches += 2;
        DS_CUDA(ctx, cudaGetLastError());
    }
    std::vector<int> cnt(nf);
    DS_CUDA(ctx, cudaMemcpyAsync(velocities, d_v.p, sizeof(double) * nf * max_modes, cudaMemcpyDeviceToHost, s));
    DS_CUDA(ctx, cudaMemcpyAsync(cnt.data(), d_c.p, sizeof(int) * nf, cudaMemcpyDeviceToHost, s));
    DS_CUDA(ctx, cudaStreamSynchronize(s));
    int status = GFK_OK;
    for (int i = 0; i < nf; i++) {
        counts[i] = cnt[i] < 0 ? -1 - cnt[i] : cnt[i];
        if (cnt[i] < 0) status = GFK_ELIMIT;
    }
    if (status) dfail(ctx, status, "disp: more modes than max_modes at some frequency");
    return status;
}

int gfk_secular(gfk_ctx* ctx, const gfk_medium* m, const double* freqs, const double* velocities, int64_t n,
                double* out, int32_t* ok) {
    if (!ctx || !m || !freqs || !velocities || !out || !ok || n < 0) return GFK_EARG;
    gfk::disp::Stack st;
    int s0 = make_stack(ctx, m, &st);
    if (s0) return s0;
    if (n == 0) return GFK_OK;
    cudaSetDevice(ctx->device);
    cudaStream_t s = ctx->stream;
    DBuf d_f{ctx}, d_c{ctx}, d_o{ctx}, d_k{ctx};
    DS_CUDA(ctx, cudaMallocAsync(&d_f.p, sizeof(double) * n, s));
    DS_CUDA(ctx, cudaMallocAsync(&d_c.p, sizeof(double) * n, s));
    DS_CUDA(ctx, cudaMallocAsync(&d_o.p, sizeof(double) * n, s));
    DS_CUDA(ctx, cudaMallocAsync(&d_k.p, sizeof(int) * n, s));
    DS_CUDA(ctx, cudaMemcpyAsync(d_f.p, freqs, sizeof(double) * n, cudaMemcpyHostToDevice, s));
    DS_CUDA(ctx, cudaMemcpyAsync(d_c.p, velocities, sizeof(double) * n, cudaMemcpyHostToDevice, s));
    gfk::disp::k_secular<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(
        st, static_cast<const double*>(d_f.p), static_cast<const double*>(d_c.p), n, static_cast<double*>(d_o.p),
        static_cast<int*>(d_k.p));
    ctx->launches++;
    DS_CUDA(ctx, cudaGetLastError());
    DS_CUDA(ctx, cudaMemcpyAsync(out, d_o.p, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
    DS_CUDA(ctx, cudaMemcpyAsync(ok, d_k.p, sizeof(int) * n, cudaMemcpyDeviceToHost, s));
    DS_CUDA(ctx, cudaStreamSynchronize(s));
    return GFK_OK;
}

}  // extern "C"
