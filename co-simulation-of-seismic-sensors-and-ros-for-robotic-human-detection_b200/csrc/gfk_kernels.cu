// gfk_kernels.cu — FP64 kernels of the Green's-function bank path.
//
//   k_layer_consts  per (frequency, layer): complex velocities -> solver constants
//                   (fk.go:96-128 hoisted out of the wavenumber loop)
//   k_static        per frequency: C = k_far u(k_far) (fk.go:365-371, 521)
//   k_prop          per (frequency, wavenumber): the layered solve and the
//                   static-subtracted integrand k u - C (fk.go:534-544)
//   k_j0_table      the shared-grid Hankel weights w_i J0(k_i r_j) dk (fk.go:540-546)
//   k_quad_gemm     the shared-grid wavenumber sum as an FP64 complex x real GEMM
//   k_quad_rows     per-frequency grids: the same sum with J0 in the loop, over
//                   items of a row's wavenumbers
//   k_bank_pack     FP64 [f][r] -> float32 range-major bank payload
//                   (internal/bank/format.go:185-193)
#include "gfk_kernels.cuh"
#include "gfk_j0.cuh"
#include "gfk_panel.cuh"


#include <algorithm>
#include <atomic>

namespace gfk {

// ------------------------------------------------------------ constants --

// One layer's constants at one frequency.
__device__ __forceinline__ LayerC layer_const(const MediumP& med, const LayerP& L, double fr, double wi,
                                              int formulation) {
    const double q = q_of(med, L);
    LayerC out;
    if (formulation == 0) {
        // Medium.propsOf (fk.go:119-128): Qp = 2.25 Qs, real frequency
        const cd a = complex_velocity(med, L.vp, 2.25 * q, fr, 0.0);
        const cd b = complex_velocity(med, L.vs, q, fr, 0.0);
        out.c[0] = a;
        out.c[1] = b;
        out.c[2] = (L.rho * b) * b;
        out.c[3] = mk(L.rho);
    } else {
        const double qp = L.qp > 0 ? L.qp : 2.25 * q;
        const cd a = complex_velocity(med, L.vp, qp, fr, wi);
        const cd b = complex_velocity(med, L.vs, q, fr, wi);
        const cd a2 = a * a, b2 = b * b;
        out.c[0] = 1.0 / a2;
        out.c[1] = 1.0 / b2;
        out.c[2] = b2 / a2;
        out.c[3] = (L.rho * b2) / med.mu_ref;
    }
    out.h = L.h;
    out.pad = 0.0;
    return out;
}

__global__ void k_layer_consts(const LayerP* __restrict__ lp, const MediumP* __restrict__ media,
                               const FreqDesc* __restrict__ fd, int nf, double wi, int formulation,
                               LayerC* __restrict__ lc, cd* __restrict__ wc2) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const FreqDesc d = fd[f];
    const MediumP med = media[d.soil];
    const double fr = d.freq;
    for (int l = 0; l < med.count; l++) lc[d.lc_off + l] = layer_const(med, lp[med.lp_off + l], fr, wi, formulation);
    const cd wc = mk(kTwoPi * fr, -wi);
    wc2[f] = wc * wc;
}

void launch_layer_consts(cudaStream_t s, const LayerP* lp, const MediumP* media, const FreqDesc* fd, int nf,
                         double wi, int formulation, LayerC* lc, cd* wc2) {
    if (nf <= 0) return;
    k_layer_consts<<<(nf + 127) / 128, 128, 0, s>>>(lp, media, fd, nf, wi, formulation, lc, wc2);
}

// The same constants with one thread per (frequency, layer): a few hundred
// frequencies of a thin stack otherwise leave most SMs idle while each thread
// walks its layers' transcendental functions in sequence.
__global__ void k_layer_consts_fl(const LayerP* __restrict__ lp, const MediumP* __restrict__ media,
                                  const FreqDesc* __restrict__ fd, int nf, double wi, int formulation,
                                  LayerC* __restrict__ lc, cd* __restrict__ wc2) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    const int l = blockIdx.y;
    if (f >= nf) return;
    const FreqDesc d = fd[f];
    const MediumP med = media[d.soil];
    if (l < med.count) lc[d.lc_off + l] = layer_const(med, lp[med.lp_off + l], d.freq, wi, formulation);
    if (l == 0) {
        const cd wc = mk(kTwoPi * d.freq, -wi);
        wc2[f] = wc * wc;
    }
}

void launch_layer_consts_fl(cudaStream_t s, const LayerP* lp, const MediumP* media, const FreqDesc* fd, int nf,
                            int max_layers, double wi, int formulation, LayerC* lc, cd* wc2) {
    if (nf <= 0 || max_layers <= 0) return;
    dim3 grid((nf + 63) / 64, max_layers);
    k_layer_consts_fl<<<grid, 64, 0, s>>>(lp, media, fd, nf, wi, formulation, lc, wc2);
}

__device__ __forceinline__ bool finite_cd(cd a) { return isfinite(a.re) && isfinite(a.im); }

// ------------------------------------------------------ static coefficient --

__device__ __forceinline__ void static_row(const LayerC* __restrict__ lc, const MediumP* __restrict__ media,
                                           const FreqDesc* __restrict__ fd, const cd* __restrict__ wc2, int f,
                                           int formulation, cd* __restrict__ C, int* __restrict__ status) {
    const FreqDesc d = fd[f];
    const double k = d.kfar;
    if (!(k > 0)) {
        C[f] = mk(0.0);
        return;
    }
    const MediumP med = media[d.soil];
    cd u;
    if (formulation == 0) {
        bool ok;
        u = direct_u(lc + d.lc_off, med.count, kTwoPi * d.freq, k, med.mu_ref, ok);
        if (!ok) atomicOr(status + f, kStSingular);
    } else {
        u = dunkin_u(lc + d.lc_off, med.count, wc2[f], k, med.mu_ref);
    }
    cd c = k * u;
    if (!finite_cd(c)) {
        atomicOr(status + f, kStNonfinite);
        c = mk(0.0);
    }
    C[f] = c;
}

__global__ void k_static(const LayerC* __restrict__ lc, const MediumP* __restrict__ media,
                         const FreqDesc* __restrict__ fd, const cd* __restrict__ wc2, int nf, int formulation,
                         cd* __restrict__ C, int* __restrict__ status) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f < nf) static_row(lc, media, fd, wc2, f, formulation, C, status);
}

void launch_static(cudaStream_t s, const LayerC* lc, const MediumP* media, const FreqDesc* fd, const cd* wc2, int nf,
                   int formulation, cd* C, int* status) {
    if (nf <= 0) return;
    k_static<<<(nf + 63) / 64, 64, 0, s>>>(lc, media, fd, wc2, nf, formulation, C, status);
}

// ------------------------------------------------------------ propagator --
//
// The work item is (row f, run): 8 panels of 128 wavenumbers per 128 threads
// (gfk_panel.cuh). Pass 0 solves the 16 first nodes of every panel, one per
// thread, a half-warp per panel, which tests its coefficients;
// pass 1 the other 16 nodes of the panels that may be served by 32; the passes
// after that every wavenumber of the remaining panels. One loop holds the
// three, so the solve is compiled once. The interpolation of the accepted
// panels is a product of a fixed 128 x 16 (or 32) matrix and the node values,
// 4 panels (re, im) wide, on the FP64 tensor path: as many FP64-pipe cycles as
// FMAs, an eighth of the issue slots and no operand traffic (the matrix
// fragments come from L1).
//
// k_prop serves one item per block (blockIdx = (run, f)); k_prop_q is
// persistent: each resident block takes items from a device queue, last row
// first, until none are left. The row's layer constants are staged in shared memory.
// Launch shapes are template parameters; the plan times them once and keeps
// the fastest. The direct formulation (FORM 0) solves every wavenumber: its parity with
// the reference includes the digits its eigenbasis loses. So does FORM 2, the Dunkin
// solve of short rows and small banks (direct_variant), SWEEPS runs of THREADS
// wavenumbers a block, a wavenumber per thread in each.

constexpr int kNodeStride = kPanelN + 4;  // of the node values in shared memory: conflict-free B fragments

// Shared memory of one propagator block.
template <int THREADS, bool SLICE>
struct PropSmem {
    LayerC lc[kMaxLayers];
    union {
        cd tile[SLICE ? THREADS * 8 : 1];
        cd nodes[THREADS / 16 * kNodeStride];
    };
    unsigned char mode[THREADS / 16];
    int last, item;
    __device__ PropSmem() {}
};

// FP64 tensor-path product D = A B + D, m8n8k4: lane t holds A[t/4][t%4],
// B[t%4][t/4] and D[t/4][2(t%4) + {0,1}]. Not volatile: the result is used, and
// the compiler may move the next step's fragment loads ahead of these MMAs.
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

// The three last (and, MID, three middle) Chebyshev coefficients of the warp's
// two panels, lane 16 p + j holding node j of panel p in v[] (one value per 16
// nodes): an 8 x 16 T times 16 T x 4 product on the FP64 tensor path, whose B
// fragments are shuffled out of the lanes (half the shuffles of a reduction
// tree per coefficient, and 4 T instructions for the sums). rows: the table's
// coefficient rows as A fragments. Returns this lane's panel's largest
// |part| of a last coefficient, and of a middle one in mid; NaN where one is.
template <int T, bool MID>
__device__ __forceinline__ double panel_tail(const double* __restrict__ rows, const cd (&v)[T], double& mid) {
    const int lane = threadIdx.x & 31;
    const int src = ((lane >> 3) & 1) * 16 + (lane & 3);  // column lane/4: panel, part
    const bool im = (lane >> 2) & 1;
    double c0 = 0.0, c1 = 0.0;
#pragma unroll
    for (int t = 0; t < T; t++)
#pragma unroll
        for (int kk = 0; kk < 4; kk++) {
            const double re = __shfl_sync(0xffffffffu, v[t].re, src + 4 * kk);
            const double iv = __shfl_sync(0xffffffffu, v[t].im, src + 4 * kk);
            dmma(c0, c1, rows[(4 * t + kk) * 32 + lane], im ? iv : re);
        }
    // lane 4 row + p (p < 2) holds (re, im) of coefficient `row` of panel p
    double m = fmax(fabs(c0), fabs(c1));
    if (isnan(c0) || isnan(c1)) m = INFINITY;
    const int p = lane >> 4;
    mid = 0.0;
    if (MID)
        mid = fmax(__shfl_sync(0xffffffffu, m, 12 + p),
                   fmax(__shfl_sync(0xffffffffu, m, 16 + p), __shfl_sync(0xffffffffu, m, 20 + p)));
    return fmax(__shfl_sync(0xffffffffu, m, p), fmax(__shfl_sync(0xffffffffu, m, 4 + p), __shfl_sync(0xffffffffu, m, 8 + p)));
}

// The largest of the half-warp's non-negative values, to 2^-20 (its high word).
__device__ __forceinline__ double half_max(double v) {
    int h = __double2hiint(v);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) h = max(h, __shfl_xor_sync(0xffffffffu, h, o));
    return __hiloint2double(h, 0);
}

// The panels of one item, [base, lim) of row f's n wavenumbers (lim a panel's
// end or n). NR = 0: the integrand goes to row[]; NR > 0: each value is added
// to acc times the range's weights, W[wavenumber][nr] or, for a whole panel,
// Wp[panel][48][nr] (the weights carried over to its 16 or 32 nodes). SUB: the
// values are k u - c, else k u. WIDE: a warp per panel solves all 32 nodes in
// the first pass (the same decisions from the same values): more solves, but
// an item is half as many wavenumbers and passes, for banks of few items.
template <int THREADS, bool WIDE, int NR, bool SUB, class SMEM>
__device__ __forceinline__ void panel_item(const double* __restrict__ tab, SMEM& sm, int nl, double mu_ref, cd w2,
                                           cd c, double d, int n, int base, int lim, cd* __restrict__ row,
                                           const double* __restrict__ W, const double* __restrict__ Wp, int nr,
                                           double* acc, double& mre, double& mim, int& bad) {
    constexpr int PANELS = THREADS / (WIDE ? 32 : 16);
    const int tid = threadIdx.x, hp = tid >> (WIDE ? 5 : 4), hj = tid & 15;
    const int pa = base + kPanel * hp;
    const bool use = pa < lim && n - pa >= kPanelLeast;
    const double cabs1 = SUB ? cnorm1(c) : 0.0;
    cd first = mk(0.0), other = mk(0.0);
    double big = 0.0;
    bool more = false;
    int mode = 0;
    unsigned direct = 0;  // panels to be solved, or (64 threads) their halves
#pragma unroll 1
    for (int pass = 0;; pass++) {
        double x;  // wavenumber / d
        bool live;
        int i = 0;
        if (pass < 2) {
            live = pass == 0 ? use : !WIDE && more;
            x = fma(64.0, tab[kPtX + (WIDE ? tid & 31 : pass * kPanelE + hj)], (double)pa + 64.5);
        } else {
            if (direct == 0) break;
            constexpr int STEP = THREADS < kPanel ? THREADS : kPanel;
            i = base + STEP * (__ffs(direct) - 1) + (tid & (STEP - 1)) + 1;
            if constexpr (THREADS > kPanel) {  // the upper threads take the next panel
                const unsigned rest = direct & (direct - 1);
                if (tid >= kPanel) i = rest ? base + kPanel * (__ffs(rest) - 1) + (tid & (kPanel - 1)) + 1 : n + 1;
                direct = rest;
            }
            direct &= direct - 1;
            live = i <= n;
            x = (double)i;
        }
        cd r = mk(0.0);
        if (live) {
            const double k = x * d;
            r = k * dunkin_u(sm.lc, nl, w2, k, mu_ref);
            if (SUB) r -= c;
        }
        if (pass == 0) {
            if constexpr (NR == 0) sm.nodes[hp * kNodeStride + (WIDE ? tid & 31 : hj)] = r;
            if (WIDE) {  // both half-warps hold the panel's pairs of first and other nodes from here on
                const cd v = r;
                r = cd{__shfl_sync(0xffffffffu, v.re, hj), __shfl_sync(0xffffffffu, v.im, hj)};
                other = cd{__shfl_sync(0xffffffffu, v.re, 16 + hj), __shfl_sync(0xffffffffu, v.im, 16 + hj)};
            }
            first = r;
            big = half_max(cnorm1(r));
            const cd v[1] = {r};
            double mid;
            const double tail = panel_tail<1, true>(tab + kPtRowsE, v, mid);
            const double scale = cabs1 + big;
            mode = use && panel_passes(tail, scale);
            // decay per 6 orders, q = tail/mid; at order 31: tail q^(16/6) <= 10 tol scale
            const float s = (float)(1.0 / scale), tl = (float)tail * s, q = tl / ((float)mid * s);
            const float room = (float)(10.0 * kPanelTol) / tl, q2 = q * q, q4 = q2 * q2;
            more = use && !mode && q < 1.0f && q4 * q4 <= room * room * room;
        } else if (pass == 1) {
            if (WIDE) r = other;
            if (__any_sync(0xffffffffu, more)) {
                const double m2 = half_max(cnorm1(r));
                const cd v[2] = {first, r};
                double none;
                const double tail = panel_tail<2, false>(tab + kPtRowsN, v, none);
                if (more && panel_passes(tail, cabs1 + fmax(big, m2))) mode = 2;
            }
            if constexpr (NR > 0) {
                if (mode) {
                    const double* w = Wp + ((size_t)(pa / kPanel) * 48 + (mode == 1 ? 0 : kPanelE) + hj) * nr;
#pragma unroll
                    for (int q = 0; q < NR; q++)
                        if (q < nr) {
                            acc[2 * q] = fma(first.re, w[q], acc[2 * q]);
                            acc[2 * q + 1] = fma(first.im, w[q], acc[2 * q + 1]);
                            if (mode == 2) {
                                const double w1 = w[kPanelE * nr + q];
                                acc[2 * q] = fma(r.re, w1, acc[2 * q]);
                                acc[2 * q + 1] = fma(r.im, w1, acc[2 * q + 1]);
                            }
                        }
                }
            } else {
                if (!WIDE) sm.nodes[hp * kNodeStride + kPanelE + hj] = r;
            }
            if (hj == 0) sm.mode[hp] = (unsigned char)mode;
            __syncthreads();
#pragma unroll
            for (int p = 0; p < PANELS; p++)
                if (sm.mode[p] == 0 && base + kPanel * p < lim)
                    direct |= THREADS >= kPanel ? 1u << p : (base + kPanel * p + 64 < lim ? 3u : 1u) << (2 * p);
        } else if (live) {
            if (!(isfinite(r.re) && isfinite(r.im))) { bad |= kStNonfinite; r = mk(0.0); }
            if constexpr (NR > 0) {
#pragma unroll
                for (int q = 0; q < NR; q++) {
                    const double w = q < nr ? W[(size_t)(i - 1) * nr + q] : 0.0;
                    acc[2 * q] = fma(r.re, w, acc[2 * q]);
                    acc[2 * q + 1] = fma(r.im, w, acc[2 * q + 1]);
                }
            } else {
                row[i - 1] = r;
                mre = fmax(mre, fabs(r.re));
                mim = fmax(mim, fabs(r.im));
            }
        }
    }
    if constexpr (NR == 0) {
        // a warp takes points 32 wq .. + 31 of 4 panels at a time: C fragment
        // row = point, columns 2 (panel) + part
        const int lane = tid & 31;
#pragma unroll 1
        for (int job = tid >> 5; job < PANELS; job += THREADS / 32) {
            const int g = job & ~3, wq = job & 3;
            const int bm = sm.mode[g + (lane >> 3)];
            const bool any1 = __any_sync(0xffffffffu, bm == 1), any2 = __any_sync(0xffffffffu, bm == 2);
            if (!any1 && !any2) continue;
            const double* v = reinterpret_cast<const double*>(sm.nodes + (g + (lane >> 3)) * kNodeStride + (lane & 3)) +
                              ((lane >> 2) & 1);
            double y[4][2];
#pragma unroll
            for (int m = 0; m < 4; m++) y[m][0] = y[m][1] = 0.0;
            if (any1) {
#pragma unroll
                for (int kk = 0; kk < kPanelE / 4; kk++) {
                    const double bv = bm == 1 ? v[8 * kk] : 0.0;
#pragma unroll
                    for (int m = 0; m < 4; m++)
                        dmma(y[m][0], y[m][1], tab[kPtFragE + ((4 * wq + m) * (kPanelE / 4) + kk) * 32 + lane], bv);
                }
            }
            if (any2) {
#pragma unroll
                for (int kk = 0; kk < kPanelN / 4; kk++) {
                    const double bv = bm == 2 ? v[8 * kk] : 0.0;
#pragma unroll
                    for (int m = 0; m < 4; m++)
                        dmma(y[m][0], y[m][1], tab[kPtFragN + ((4 * wq + m) * (kPanelN / 4) + kk) * 32 + lane], bv);
                }
            }
            const int p = g + (lane & 3);
            if (sm.mode[p])
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    const int at = base + kPanel * p + (4 * wq + m) * 8 + (lane >> 2);
                    if (at < n) {
                        row[at] = mk(y[m][0], y[m][1]);
                        mre = fmax(mre, fabs(y[m][0]));
                        mim = fmax(mim, fabs(y[m][1]));
                    }
                }
        }
    }
}

// `stage`: the block's staged layer constants are not row f's (uniform).
template <int FORM, int THREADS, bool WIDE, bool SLICE, int SWEEPS = 1>
__device__ __forceinline__ void prop_item(const LayerC* __restrict__ lc, const MediumP* __restrict__ media,
                                          const FreqDesc* __restrict__ fd, const cd* __restrict__ wc2,
                                          const cd* __restrict__ C, const double* __restrict__ tab,
                                          cd* __restrict__ rem, int* __restrict__ status, const SliceOut& so, int f,
                                          int run, int runs, bool stage, PropSmem<THREADS, SLICE>& sm) {
    const FreqDesc fdesc = fd[f];
    const MediumP med = media[fdesc.soil];
    const int nl = med.count;
    const double mu_ref = med.mu_ref;
    if (stage) {
        for (int l = threadIdx.x; l < nl; l += blockDim.x) sm.lc[l] = lc[fdesc.lc_off + l];
        __syncthreads();
    }
    const int n = fdesc.kfar > 0 ? fdesc.nk : 0;
    const double d = fdesc.dk;
    const cd c = C ? C[f] : mk(0.0);
    cd* row = rem + fdesc.off;
    int bad = 0;
    double mre = 0.0, mim = 0.0;
    if constexpr (FORM != 1) {
#pragma unroll 1
        for (int sweep = 0; sweep < SWEEPS; sweep++) {
            const int i = (run * SWEEPS + sweep) * THREADS + threadIdx.x + 1;
            if (i > n) break;
            const double k = (double)i * d;
            cd r;
            if constexpr (FORM == 0) {
                bool ok;
                cd u = direct_u(sm.lc, nl, kTwoPi * fdesc.freq, k, mu_ref, ok);
                if (!ok) bad |= kStSingular;
                r = k * u - c;
            } else {
                r = k * dunkin_u(sm.lc, nl, wc2[f], k, mu_ref) - c;
            }
            if (!finite_cd(r)) { bad |= kStNonfinite; r = mk(0.0); }
            row[i - 1] = r;
            mre = fmax(mre, fabs(r.re));
            mim = fmax(mim, fabs(r.im));
        }
    } else {
        panel_item<THREADS, WIDE, 0, true>(tab, sm, nl, mu_ref, wc2[f], c, d, n, run * THREADS * (WIDE ? 4 : 8), n, row,
                                           nullptr, nullptr, 0, nullptr, mre, mim, bad);
    }
    if (bad) atomicOr(status + f, bad);
    if constexpr (SLICE) {
        // The tensor-core sum's integer slicing, by the row's last block: the
        // row's maxima (the bits of a non-negative double order like the value),
        // then a device-scope fence and the row's count of finished blocks; the
        // block that finishes the row slices it while it is still in L2. No block
        // waits for another. (The pattern of a grid barrier's arrival: block
        // barrier, one thread's fence, the atomic count.)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mre = fmax(mre, __shfl_xor_sync(0xffffffffu, mre, o));
            mim = fmax(mim, __shfl_xor_sync(0xffffffffu, mim, o));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMax(so.rowmax + 2 * f, (unsigned long long)__double_as_longlong(mre));
            atomicMax(so.rowmax + 2 * f + 1, (unsigned long long)__double_as_longlong(mim));
        }
        // the barrier orders every thread's stores before thread 0's fence
        // (cumulative), which orders them before the count
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            const bool last = atomicAdd(so.done + f, 1ull) == (unsigned long long)(runs - 1);
            if (last) __threadfence();
            sm.last = last;
        }
        __syncthreads();
        if (!sm.last) return;
        const unsigned long long b0 = __ldcg(so.rowmax + 2 * f), b1 = __ldcg(so.rowmax + 2 * f + 1);
        const int e[2] = {slice_exp(__longlong_as_double((long long)b0)), slice_exp(__longlong_as_double((long long)b1))};
        if (threadIdx.x == 0) {
            so.row_exp[2 * f] = e[0];
            so.row_exp[2 * f + 1] = e[1];
            so.done[f] = 0;  // every block of the row has counted: ready for the next launch
        }
        // a row with no device work (both maxima 0) slices to zeros without
        // reading its integrand slot
        slice_row<THREADS>(row, n, b0 != 0 || b1 != 0, e, so, f, sm.tile);
    }
}

template <int FORM, int THREADS, int MINB, bool WIDE, bool SLICE, int SWEEPS = 1>
__global__ __launch_bounds__(THREADS, MINB) void k_prop(const LayerC* __restrict__ lc,
                                                       const MediumP* __restrict__ media,
                                                       const FreqDesc* __restrict__ fd, const cd* __restrict__ wc2,
                                                       const cd* __restrict__ C, const double* __restrict__ tab,
                                                       cd* __restrict__ rem, int* __restrict__ status, SliceOut so,
                                                       PropQueue) {
    __shared__ PropSmem<THREADS, SLICE> sm;
    prop_item<FORM, THREADS, WIDE, SLICE, SWEEPS>(lc, media, fd, wc2, C, tab, rem, status, so,
                                                  gridDim.y - 1 - blockIdx.y, blockIdx.x, gridDim.x, true, sm);
}

// Rows of uneven length: block (item, y) serves the y-th run of 128
// wavenumbers of that item. A grid over (longest row, rows) is mostly empty
// blocks when the rows differ a hundredfold (2.46M blocks for 57k runs on the
// loam bank). The static coefficients are solved beside the integrand, by the
// blocks past the last item: one solve is a serial chain (89 us alone in the
// direct formulation), so the integrand is stored as k u and the sum takes
// C off.
// Block (item, y): the y-th 128 wavenumbers (solved one by one) or 1024 (by
// panels, PANEL) of the item.
template <int FORM, bool PANEL>
__global__ __launch_bounds__(128, FORM == 0 ? 1 : 5) void k_prop_rows(const LayerC* __restrict__ lc,
                                                                     const MediumP* __restrict__ media,
                                                                     const FreqDesc* __restrict__ fd, int nf,
                                                                     const cd* __restrict__ wc2, cd* __restrict__ C,
                                                                     const double* __restrict__ tab,
                                                                     cd* __restrict__ ku, int* __restrict__ status,
                                                                     RowItems it) {
    constexpr int RUN = PANEL ? 8 * kPanel : 128;
    __shared__ PropSmem<128, false> sm;
    const int item = blockIdx.x;
    if (item >= it.items) {
        const int f = (item - it.items) * 128 + threadIdx.x;
        if (blockIdx.y == 0 && f < nf) static_row(lc, media, fd, wc2, f, FORM, C, status);
        return;
    }
    const int f = it.row ? it.row[item] - it.row0 : 0;
    const int first = (item - (it.begin ? it.begin[f] - it.item0 : 0)) * it.kc;
    const FreqDesc fdesc = fd[f];
    const int base = first + blockIdx.y * RUN, lim = min(first + it.kc, fdesc.nk);
    if (base >= lim) return;
    const MediumP med = media[fdesc.soil];
    for (int l = threadIdx.x; l < med.count; l += 128) sm.lc[l] = lc[fdesc.lc_off + l];
    __syncthreads();
    cd* row = ku + fdesc.off;
    int bad = 0;
    if constexpr (PANEL) {
        double mre = 0.0, mim = 0.0;
        panel_item<128, false, 0, false>(tab, sm, med.count, med.mu_ref, wc2[f], mk(0.0), fdesc.dk, fdesc.nk, base, lim, row,
                                  nullptr, nullptr, 0, nullptr, mre, mim, bad);
    } else {
        const int i = base + threadIdx.x + 1;
        if (i <= lim) {
            const double k = (double)i * fdesc.dk;
            cd u;
            if (FORM == 0) {
                bool ok;
                u = direct_u(sm.lc, med.count, kTwoPi * fdesc.freq, k, med.mu_ref, ok);
                if (!ok) bad |= kStSingular;
            } else {
                u = dunkin_u(sm.lc, med.count, wc2[f], k, med.mu_ref);
            }
            cd r = k * u;
            if (!finite_cd(r)) { bad |= kStNonfinite; r = mk(0.0); }
            row[i - 1] = r;
        }
    }
    if (bad) atomicOr(status + f, bad);
}

// Persistent: items (f, run), row by row, from q.next (zero at launch), so a
// row's items run together and the row is sliced while it is in L2. Blocks
// never wait for one another; each leaves when the queue is empty.
template <int FORM, int THREADS, int MINB, bool WIDE, bool SLICE>
__global__ __launch_bounds__(THREADS, MINB) void k_prop_q(const LayerC* __restrict__ lc,
                                                         const MediumP* __restrict__ media,
                                                         const FreqDesc* __restrict__ fd, const cd* __restrict__ wc2,
                                                         const cd* __restrict__ C, const double* __restrict__ tab,
                                                         cd* __restrict__ rem, int* __restrict__ status, SliceOut so,
                                                         PropQueue q) {
    __shared__ PropSmem<THREADS, SLICE> sm;
    int cur = -1;
    for (;;) {
        __syncthreads();  // every thread is done with the previous item's shared memory
        if (threadIdx.x == 0) sm.item = (int)atomicAdd(q.next, 1u);
        __syncthreads();
        const int item = sm.item;
        if (item >= q.items) return;
        // the last rows first: a medium's higher frequencies, whose poles reach
        // further, are its costlier rows, and the queue ends on cheap items
        const int rf = item / q.runs, run = item - rf * q.runs, f = q.items / q.runs - 1 - rf;
        prop_item<FORM, THREADS, WIDE, SLICE>(lc, media, fd, wc2, C, tab, rem, status, so, f, run, q.runs, f != cur, sm);
        cur = f;
    }
}

namespace {
using PropFn = void (*)(const LayerC*, const MediumP*, const FreqDesc*, const cd*, const cd*, const double*, cd*, int*,
                        SliceOut, PropQueue);
struct PropVariant {
    PropFn fn, fn_slice;  // without and with the fused slicing
    int threads, minb;
    bool wide;        // all 32 nodes in the first pass
    bool persistent;  // k_prop_q: one block per resident slot, items from a queue
};
#define GFK_PROP_SHAPE(T, B, W) {k_prop<1, T, B, W, false>, k_prop<1, T, B, W, true>, T, B, W, false}
#define GFK_PROP_QUEUE(T, B, W) {k_prop_q<1, T, B, W, false>, k_prop_q<1, T, B, W, true>, T, B, W, true}
// 80 registers spill up to 220 bytes a thread and still lead: six blocks of four
// warps hide the FP64 latency. On the 2048-row graded bank (ms, with the sum's
// 0.48): 256 threads at 3 blocks per SM 2.44, 128 at 4, 5, 6, 7 blocks 2.50,
// 2.45, 2.41, 2.46, 64 at 10 and 12 2.51, 2.52; one item per warp without
// barriers 2.82 (an item is then up to 20 solves in series). All nodes at once
// for plans of few items: 317 rows x 3001, 11 layers 188 -> 140 us.
const PropVariant kDunkinVariants[] = {
    GFK_PROP_SHAPE(64, 12, false),  // 4 panels per item, <= 80 registers
    GFK_PROP_SHAPE(128, 5, false),  // 8 panels per item, <= 96 registers
    GFK_PROP_SHAPE(128, 6, false),  // <= 80 registers
    GFK_PROP_SHAPE(256, 3, false),  // 16 panels per item
    GFK_PROP_SHAPE(128, 5, true),   // 4 panels per item, all nodes at once
    GFK_PROP_SHAPE(256, 2, true),
    GFK_PROP_QUEUE(64, 12, false),
    GFK_PROP_QUEUE(128, 5, false),
    GFK_PROP_QUEUE(128, 6, false),
    GFK_PROP_QUEUE(256, 3, false),
    GFK_PROP_QUEUE(128, 5, true),
};
constexpr int kPropVariants = sizeof(kDunkinVariants) / sizeof(kDunkinVariants[0]);

// The launches that solve every wavenumber (FORM 2), variants kPropFixed + index.
struct DirectVariant {
    PropFn fn, fn_slice;
    int threads, minb, sweeps;
};
#define GFK_DIRECT(T, B, S) {k_prop<2, T, B, false, false, S>, k_prop<2, T, B, false, true, S>, T, B, S}
const DirectVariant kDirectVariants[] = {
    GFK_DIRECT(128, 4, 1),           // <= 128 registers
    GFK_DIRECT(128, 5, 1),           // <= 96 registers
    GFK_DIRECT(128, 5, kRowSweeps),  // a short row per block
    GFK_DIRECT(256, 2, 1),           // <= 128 registers
};
constexpr int kDirectCount = sizeof(kDirectVariants) / sizeof(kDirectVariants[0]);
#undef GFK_DIRECT
static_assert(kPropFixed + kDirectCount == kPropFused, "fixed variants follow one another");

// The launches with the sum fused in (k_prop_fused), variants kPropFused + index:
// `sweeps` runs of 128 wavenumbers a block, or panels of 128.
struct FusedVariant {
    int minb, sweeps;
    bool panel;
};
const FusedVariant kFusedVariants[] = {
    {4, 1, false}, {4, 2, false}, {4, kRowSweeps, false}, {6, 8, true}, {4, 8, true},  // up to 2 ranges, up to 8
};
constexpr int kFusedCount = sizeof(kFusedVariants) / sizeof(kFusedVariants[0]);
#undef GFK_PROP_SHAPE
#undef GFK_PROP_QUEUE

// Resident blocks of a persistent shape on the whole device (queried once per
// kernel; concurrent first calls compute the same value).
int persistent_grid(int variant, bool slice) {
    static std::atomic<int> cache[kPropVariants][2] = {};
    std::atomic<int>& slot = cache[variant][slice ? 1 : 0];
    int g = slot.load(std::memory_order_relaxed);
    if (g == 0) {
        const PropVariant& v = kDunkinVariants[variant];
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)(slice ? v.fn_slice : v.fn), v.threads,
                                                      0);
        g = std::max(1, sms * std::max(per_sm, 1));
        slot.store(g, std::memory_order_relaxed);
    }
    return g;
}
}  // namespace

int prop_variant_count() { return kPropVariants; }

bool prop_variant_persistent(int variant) {
    return variant >= 0 && variant < kPropVariants && kDunkinVariants[variant].persistent;
}

// Which of kDirectVariants a plan of `rows` rows of nk wavenumbers takes. Execute of a
// plan as a graph, on either side of each line (us; first the fastest of the 13 shapes that
// used to be timed for each plan, then these four in turn; 2 us are one tick of the timer):
//   rows of two runs: 256 threads hold one while every block is resident (two on each of 148
//     SMs), then a block per row. 157 x 208, 12 layers 70: 76 / 76 / 72 / 70;
//     538 x 166, 9 layers 69: 76 / 78 / 70 / 78;  2412 x 186, 9 layers 138: 150 / 142 / 132 / 186
//   many short rows: a block per row, no block of a few live threads at a row's end. The
//     longer the rows the later, as few rows are few blocks; with the split sum, whose
//     last block of a row cuts its digits, earlier. 423 x 488, 7 layers, split 69: 74 / 72 / 68 / 76;
//     403 x 469, 5 layers 80: 82 / 81 / 82 / 84;  564 x 1118, 2 layers, split 68: 74 / 70 / 64 / 79;
//     467 x 1046, 9 layers, split 123: 125 / 121 / 132 / 131;  755 x 1050, 4 layers 99: 103 / 99 / 109 / 109;
//     2590 x 964, 5 layers 360: 378 / 363 / 356 / 389
//   rows of four runs, plain sum: two blocks of 256 threads from the second wave on
//     (175 x 422, 12 layers 84: 89 / 96 / 96 / 84)
//   a half-space alone: a solve is so short that a block wants many (112 x 4150, split 54:
//     65 / 65 / 56 / 65)
//   rows of one run: five blocks per SM where four leave a second wave, and for many
//     (740 x 100, 8 layers, split 73: 70 / 62 / 63 / 84;  800 x 100 74: 72 / 74 / 74 / 89;
//     1332 x 100 86: 84 / 76 / 78 / 113)
//   long rows, few of them, split: 256 threads cut a row's digits (33 x 2608, 12 layers 74:
//     78 / 84 / 176 / 72;  21 x 10767, 3 layers 69: 73 / 74 / 94 / 68)
//   else few blocks: more registers, a shorter chain (91 x 1477, 11 layers, split 77: 76 / 80 /
//     135 / 77); many: the fifth block (113 x 1553, 10 layers, split 84: 84 / 80 / 141 / 88)
// Over 400 random plans the geometric mean is 1.004 of the fastest shape's speed, 0.998 with
// 128 threads only and one line for all short rows; below 0.96 are 15 instead of 36.
int direct_variant(int nl, long long rows, int nk, bool split) {
    constexpr int kRun = 128, kShort = kRun * kRowSweeps, kManyLong = 240;
    const long long runs = rows * ((nk + kRun - 1) / kRun), longs = rows * ((nk + kShort - 1) / kShort);
    enum { kFew = kPropFixed, kMany, kRow, kPair };
    if (nk <= kRun) return runs <= 4 * 148 || (runs > 5 * 148 && runs <= 8 * 148) ? kFew : kMany;
    if (nk <= 2 * kRun) return rows <= 2 * 148 ? kPair : kRow;
    if (nk <= kShort && rows >= (nk <= 4 * kRun ? 400 : split ? 540 : 1000)) return kRow;
    if (nl == 1 && longs >= kManyLong) return kRow;
    if (!split && nk > 3 * kRun && nk <= 4 * kRun && runs > 4 * 148 && runs <= 8 * 148) return kPair;
    if (split && nk > 16 * kRun && runs > 3 * 148 && runs <= 13 * 148) return kPair;
    return runs <= 8 * 148 ? kFew : kMany;
}

bool prop_variant_shape(int variant, int* threads, int* blocks_per_sm, int* ilp, int* sweeps, int* persistent) {
    if (variant >= kPropFixed && variant < kPropFixed + kDirectCount) {
        const DirectVariant& v = kDirectVariants[variant - kPropFixed];
        *threads = v.threads;
        *blocks_per_sm = v.minb;
        *ilp = 1;
        *sweeps = v.sweeps;
        *persistent = 0;
        return true;
    }
    if (variant >= kPropFused && variant < kPropFused + kFusedCount) {
        const FusedVariant& v = kFusedVariants[variant - kPropFused];
        *threads = 128;
        *blocks_per_sm = v.minb;
        *ilp = 1;
        *sweeps = v.sweeps;
        *persistent = 0;
        return true;
    }
    if (variant < 0 || variant >= kPropVariants) return false;
    const PropVariant& v = kDunkinVariants[variant];
    *threads = v.threads;
    *blocks_per_sm = v.minb;
    *ilp = 1;
    *sweeps = v.threads / (v.wide ? 32 : 16);  // a panel of 128 wavenumbers per 16 threads
    *persistent = v.persistent ? 1 : 0;
    return true;
}

void launch_prop(cudaStream_t s, const LayerC* lc, const MediumP* media, const FreqDesc* fd, const cd* wc2, int nf,
                 int max_nk, const cd* C, int formulation, const double* tab, cd* rem, int* status, int variant,
                 const SliceOut* slice, unsigned int* queue) {
    if (nf <= 0 || max_nk <= 0) return;
    const SliceOut so = slice ? *slice : SliceOut{};
    if (formulation == 0) {
        dim3 grid((max_nk + 127) / 128, nf);
        if (slice)
            k_prop<0, 128, 1, false, true><<<grid, 128, 0, s>>>(lc, media, fd, wc2, C, tab, rem, status, so, PropQueue{});
        else
            k_prop<0, 128, 1, false, false><<<grid, 128, 0, s>>>(lc, media, fd, wc2, C, tab, rem, status, so, PropQueue{});
        return;
    }
    if (variant >= kPropFixed && variant < kPropFixed + kDirectCount) {
        const DirectVariant& v = kDirectVariants[variant - kPropFixed];
        const int per_block = v.threads * v.sweeps;
        (slice ? v.fn_slice : v.fn)<<<dim3((max_nk + per_block - 1) / per_block, nf), v.threads, 0, s>>>(
            lc, media, fd, wc2, C, tab, rem, status, so, PropQueue{});
        return;
    }
    if (variant < 0 || variant >= kPropVariants) variant = 0;
    if (kDunkinVariants[variant].persistent && !queue) variant = 2;  // no queue: one item per block
    const PropVariant& v = kDunkinVariants[variant];
    const int per_item = v.threads * (v.wide ? 4 : 8);
    const int runs = (max_nk + per_item - 1) / per_item;
    const PropFn fn = slice ? v.fn_slice : v.fn;
    if (v.persistent) {
        const PropQueue q{queue, nf * runs, runs};
        fn<<<std::min(persistent_grid(variant, slice != nullptr), nf * runs), v.threads, 0, s>>>(
            lc, media, fd, wc2, C, tab, rem, status, so, q);
    } else {
        fn<<<dim3(runs, nf), v.threads, 0, s>>>(lc, media, fd, wc2, C, tab, rem, status, so, PropQueue{});
    }
}

void launch_prop_rows(cudaStream_t s, const LayerC* lc, const MediumP* media, const FreqDesc* fd, int nf,
                      const cd* wc2, cd* C, int formulation, const double* tab, cd* ku, int* status,
                      const RowItems& it) {
    if (nf <= 0) return;
    const int extra = (nf + 127) / 128;
    const dim3 grid(it.items + extra, it.kc / 128);
    if (formulation == 0)
        k_prop_rows<0, false><<<grid, 128, 0, s>>>(lc, media, fd, nf, wc2, C, tab, ku, status, it);
    else if (tab)
        k_prop_rows<1, true><<<dim3(it.items + extra, (it.kc + 1023) / 1024), 128, 0, s>>>(lc, media, fd, nf, wc2, C,
                                                                                        tab, ku, status, it);
    else
        k_prop_rows<1, false><<<grid, 128, 0, s>>>(lc, media, fd, nf, wc2, C, tab, ku, status, it);
}

// ------------------------------------------------- fused propagator + sum --
//
// For a handful of ranges the wavenumber sum is a dot product per range: each
// thread accumulates its values k u - C times the Hankel weights over its
// block's 1024 wavenumbers (8 panels), the block reduces in a fixed order (warp
// tree, then warps), and one partial per (row, k block, range) is written. A
// panel taken from its nodes is never interpolated: the weights of its 128
// wavenumbers are carried over to the nodes once per grid (k_panel_weights).
// Short rows and small plans (fused_variant) solve every wavenumber, 1, 2 or
// kRowSweeps runs of 128 a block, and need no node weights.
// The integrand never reaches HBM; k_fused_finish adds the partials in block
// order (deterministic) and the closed k = 0 panel (fk.go:529-532).

constexpr int kFuseThreads = 128;
constexpr int kFuseSpan = 8 * kFuseThreads;  // wavenumbers of its row a block of panels covers

// Wp[panel][48][nr]: sum over the panel's wavenumbers of the interpolation
// matrix times W, for the 16-node and then the 32-node fit.
__global__ void k_panel_weights(const double* __restrict__ W, const double* __restrict__ tab, int nk, int nr,
                                double* __restrict__ Wp) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int panels = (nk + kPanel - 1) / kPanel;
    if (t >= (int64_t)panels * 48 * nr) return;
    const int q = (int)(t % nr), j = (int)(t / nr % 48), p = (int)(t / nr / 48);
    double s = 0.0;
    for (int i = 0; i < kPanel && p * kPanel + i < nk; i++) {
        const double m = j < kPanelE ? tab[kPtFragE + panel_frag(i, j, kPanelE)]
                                     : tab[kPtFragN + panel_frag(i, j - kPanelE, kPanelN)];
        s = fma(m, W[(size_t)(p * kPanel + i) * nr + q], s);
    }
    Wp[t] = s;
}

size_t panel_weight_count(int nk, int nr) { return (size_t)((nk + kPanel - 1) / kPanel) * 48 * nr; }

void launch_panel_weights(cudaStream_t s, const double* W, const double* tab, int nk, int nr, double* Wp) {
    const size_t n = panel_weight_count(nk, nr);
    k_panel_weights<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(W, tab, nk, nr, Wp);
}

// PANEL: `sweeps` is not read; else the runs of 128 wavenumbers a block covers.
template <int NR, bool PANEL>
__global__ __launch_bounds__(kFuseThreads, PANEL && NR <= 2 ? 6 : 4) void k_prop_fused(const LayerC* __restrict__ lc,
                                                                const MediumP* __restrict__ media,
                                                                const FreqDesc* __restrict__ fd,
                                                                const cd* __restrict__ wc2, const cd* __restrict__ C,
                                                                const double* __restrict__ tab,
                                                                const double* __restrict__ W,
                                                                const double* __restrict__ Wp, int nr, int nkb,
                                                                int sweeps, cd* __restrict__ partial,
                                                                int* __restrict__ status) {
    __shared__ PropSmem<kFuseThreads, false> sm;
    __shared__ double s_red[2 * NR][kFuseThreads / 32];
    const int f = gridDim.y - 1 - blockIdx.y;  // the costlier rows first
    const FreqDesc fdesc = fd[f];
    const MediumP med = media[fdesc.soil];
    const int nl = med.count;
    for (int l = threadIdx.x; l < nl; l += blockDim.x) sm.lc[l] = lc[fdesc.lc_off + l];
    __syncthreads();
    const int n = fdesc.kfar > 0 ? fdesc.nk : 0;
    double acc[2 * NR];
#pragma unroll
    for (int q = 0; q < 2 * NR; q++) acc[q] = 0.0;
    int bad = 0;
    if constexpr (PANEL) {
        double mre = 0.0, mim = 0.0;
        panel_item<kFuseThreads, false, NR, true>(tab, sm, nl, med.mu_ref, wc2[f], C[f], fdesc.dk, n,
                                                  blockIdx.x * kFuseSpan, n, nullptr, W, Wp, nr, acc, mre, mim, bad);
    } else {
        const cd w2 = wc2[f], c = C[f];
#pragma unroll 1
        for (int sweep = 0; sweep < sweeps; sweep++) {
            const int i = (blockIdx.x * sweeps + sweep) * kFuseThreads + threadIdx.x + 1;
            if (i > n) break;
            const double k = (double)i * fdesc.dk;
            cd r = k * dunkin_u(sm.lc, nl, w2, k, med.mu_ref) - c;
            if (!finite_cd(r)) { bad |= kStNonfinite; r = mk(0.0); }
#pragma unroll
            for (int q = 0; q < NR; q++) {
                const double w = q < nr ? W[(size_t)(i - 1) * nr + q] : 0.0;
                acc[2 * q] = fma(r.re, w, acc[2 * q]);
                acc[2 * q + 1] = fma(r.im, w, acc[2 * q + 1]);
            }
        }
    }
    if (bad) atomicOr(status + f, bad);
    // warp tree, then the block's warps in order: a fixed summation order
#pragma unroll
    for (int q = 0; q < 2 * NR; q++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_down_sync(0xffffffffu, acc[q], o);
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int q = 0; q < 2 * NR; q++) s_red[q][warp] = acc[q];
    __syncthreads();
    if (threadIdx.x < nr) {
        const int j = threadIdx.x;
        double re = 0.0, im = 0.0;
#pragma unroll
        for (int w = 0; w < kFuseThreads / 32; w++) {
            re += s_red[2 * j][w];
            im += s_red[2 * j + 1][w];
        }
        partial[((size_t)f * nkb + blockIdx.x) * nr + j] = mk(re, im);
    }
}

__global__ void k_fused_finish(const cd* __restrict__ partial, const cd* __restrict__ C,
                               const double* __restrict__ ranges, const FreqDesc* __restrict__ fd, int nf, int nr,
                               int nkb, cd* __restrict__ G) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)nf * nr) return;
    const int f = (int)(t / nr), j = (int)(t - (int64_t)f * nr);
    const cd c = C[f];
    const double d = fd[f].dk;
    cd acc = c / ranges[j] - (0.5 * d) * c;
#pragma unroll 8
    for (int b = 0; b < nkb; b++) acc += partial[((size_t)f * nkb + b) * nr + j];
    G[(size_t)f * nr + j] = acc;
}

int fused_max_ranges() { return 8; }

// Many short rows take a block each, rows of two runs earlier: as blocks of their own
// a full and a nearly empty run alternate over the SMs. A solve of one or two finite layers is short
// beside a block's table load and reduction: two runs a block there. Execute of a plan
// with 1 / 2 / 4 / 8 runs a block (us):
//   552 rows x 207, 8 layers 66 / 57 / 57 / 57    245 x 252, 9 layers 64 / 55 / 55 / 55
//   141 x 359, 10 layers 60 / 70 / 66 / 66        283 x 760, 6 layers 68 / 70 / 82 / 67
//   129 x 3608, 8 layers 115 / 118 / 128 / 201    25 x 5823, 4 layers 55 / 53 / 63 / 70
//   21 x 4616, 2 layers 46 / 44 / 44 / 52         26 x 3437, half-space 43 / 39 / 39 / 42
int fused_variant(int nl, long long rows, int nk, int nr, bool direct) {
    constexpr int kManyRows = 400, kManyPairs = 148;
    if (!direct) return kPropFused + (nr <= 2 ? 3 : 4);
    const bool is_short = nk <= 128 * kRowSweeps;
    return kPropFused + (is_short && rows >= (nk <= 256 ? kManyPairs : kManyRows) ? 2 : !is_short && nl <= 3 ? 1 : 0);
}

int fused_span(int variant) { return kFuseThreads * kFusedVariants[variant - kPropFused].sweeps; }

namespace {
template <int NR>
void launch_fused(cudaStream_t s, dim3 grid, bool panel, const LayerC* lc, const MediumP* media, const FreqDesc* fd,
                  const cd* wc2, const cd* C, const double* tab, const double* W, const double* Wp, int nr, int sweeps,
                  cd* partial, int* status) {
    (panel ? k_prop_fused<NR, true> : k_prop_fused<NR, false>)<<<grid, kFuseThreads, 0, s>>>(
        lc, media, fd, wc2, C, tab, W, Wp, nr, (int)grid.x, sweeps, partial, status);
}
}  // namespace

void launch_prop_fused(cudaStream_t s, const LayerC* lc, const MediumP* media, const FreqDesc* fd, const cd* wc2,
                       int nf, int nk, const cd* C, const double* tab, const double* W, const double* Wp,
                       const double* ranges, int nr, int variant, cd* partial, int* status, cd* G) {
    if (nf <= 0 || nk <= 0 || nr <= 0 || nr > 8) return;
    const FusedVariant& v = kFusedVariants[variant - kPropFused];
    const int span = fused_span(variant), nkb = (nk + span - 1) / span;
    const auto fn = nr <= 1 ? launch_fused<1> : nr <= 2 ? launch_fused<2> : nr <= 4 ? launch_fused<4> : launch_fused<8>;
    fn(s, dim3(nkb, nf), v.panel, lc, media, fd, wc2, C, tab, W, Wp, nr, v.sweeps, partial, status);
    const int64_t nt = (int64_t)nf * nr;
    k_fused_finish<<<(unsigned)((nt + 255) / 256), 256, 0, s>>>(partial, C, ranges, fd, nf, nr, nkb, G);
}

// -------------------------------------------------------------- J0 table --

__global__ void k_j0_table(const double* __restrict__ ranges, int nr, int nk, double dk, double* __restrict__ W) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)nk * nr) return;
    const int i = (int)(idx / nr) + 1;
    const int j = (int)(idx - (int64_t)(i - 1) * nr);
    const double k = (double)i * dk;
    const double w = i == nk ? 0.5 : 1.0;
    W[idx] = (w * j0(k * ranges[j])) * dk;
}

void launch_j0_table(cudaStream_t s, const double* ranges, int nr, int nk, double dk, double* W) {
    const int64_t n = (int64_t)nk * nr;
    k_j0_table<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(ranges, nr, nk, dk, W);
}

// ----------------------------------------------------- FP64 quadrature --
//
// G[f][j] = C_f/r_j - (dk/2) C_f + sum_i rem[f][i] W[i][j]:
// a complex (nf x nk) by real (nk x nr) product, computed as the real GEMM of
// the 2 nf rows (re, im) of the integrand on the FP64 tensor cores:
// mma.sync m8n8k4 f64 (A 8x4 row-major, B 4x8 column-major, FP64 accumulate;
// lane t holds A[t/4][t%4], B[t%4][t/4] and C[t/4][2(t%4) + {0,1}]). Block
// tile 128 real rows (64 frequencies) x 16 TNW ranges x 16 wavenumbers, 8
// warps as 4 (rows) x 2 (ranges), a warp owning 32 x 8 TNW of the output
// (4 x TNW 8x8 accumulator tiles). The tiles move global -> shared with
// cp.async in a 3-stage ring; a stage holds the integrand as [k][2f + part]
// and the weights as [k][r], both with a row stride of 8 mod 16 doubles, so
// each fragment load (4 wavenumber rows x 8 consecutive doubles) takes the
// minimum two shared-memory wavefronts.

namespace qd {
constexpr int BM = 128, BK = 16, STAGES = 3, THREADS = 256;  // real rows, wavenumbers per stage
constexpr int ASTR = BM + 8;
template <int TNW>
__host__ __device__ constexpr int bstr() { return 16 * TNW + 8; }
template <int TNW>
constexpr int smem_bytes() { return STAGES * (BK * ASTR + BK * bstr<TNW>()) * (int)sizeof(double); }

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(s), "l"(src), "r"(valid ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
}  // namespace qd

template <int TNW>
__global__ __launch_bounds__(qd::THREADS, TNW == 8 ? 1 : 2) void k_quad_gemm(const cd* __restrict__ rem,
                                                              const double* __restrict__ W,
                                                              const cd* __restrict__ C,
                                                              const double* __restrict__ ranges, int nf, int nk,
                                                              int nr, double dk, cd* __restrict__ G,
                                                              cd* __restrict__ part) {
    using namespace qd;
    constexpr int BN = 16 * TNW, BSTR = bstr<TNW>();
    extern __shared__ __align__(16) double d_smem[];
    double* const sA = d_smem;                       // [STAGES][BK][ASTR]
    double* const sB = d_smem + STAGES * BK * ASTR;  // [STAGES][BK][BSTR]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp & 3, wn = warp >> 2;
    const int f0 = blockIdx.y * (BM / 2);
    const int n0 = blockIdx.x * BN;
    const int ntiles = (nk + BK - 1) / BK;
    const int kt0 = (int)((long long)blockIdx.z * ntiles / gridDim.z);
    const int nt = (int)((long long)(blockIdx.z + 1) * ntiles / gridDim.z) - kt0;

    auto load = [&](int stage, int kt) {
        const int kb = kt * BK;
        double* a = sA + stage * BK * ASTR;
        double* b = sB + stage * BK * BSTR;
        const int fr = tid >> 2, kq = (tid & 3) * 4;
        const int gf = f0 + fr;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int k = kb + kq + q;
            const bool ok = gf < nf && k < nk;
            qd::cp_async16(a + (kq + q) * ASTR + 2 * fr,
                           ok ? (const void*)(rem + (size_t)gf * nk + k) : (const void*)rem, ok);
        }
        const int kr = tid >> 4, c0 = (tid & 15) * 2;
        const int k = kb + kr;
#pragma unroll
        for (int q = 0; q < BN / 32; q++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int col = c0 + 32 * q + e, gc = n0 + col;
                const bool ok = k < nk && gc < nr;
                qd::cp_async8(b + kr * BSTR + col, ok ? (const void*)(W + (size_t)k * nr + gc) : (const void*)W, ok);
            }
    };

    double acc[4][TNW][2];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < TNW; j++) acc[i][j][0] = acc[i][j][1] = 0.0;

#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) {
        if (s < nt) load(s, kt0 + s);
        qd::cp_commit();
    }
    const int fa = (lane & 3) * ASTR + wm * 32 + (lane >> 2);       // this lane's A fragment element
    const int fb = (lane & 3) * BSTR + wn * 8 * TNW + (lane >> 2);  // and B fragment element
    for (int t = 0; t < nt; t++) {
        qd::cp_wait<STAGES - 2>();
        __syncthreads();
        if (t + STAGES - 1 < nt) load((t + STAGES - 1) % STAGES, kt0 + t + STAGES - 1);
        qd::cp_commit();
        const double* a = sA + (t % STAGES) * BK * ASTR + fa;
        const double* b = sB + (t % STAGES) * BK * BSTR + fb;
        // fragments of step k4 + 1 are loaded while step k4's MMAs issue
        double av[2][4], bv[2][TNW];
#pragma unroll
        for (int i = 0; i < 4; i++) av[0][i] = a[8 * i];
#pragma unroll
        for (int j = 0; j < TNW; j++) bv[0][j] = b[8 * j];
#pragma unroll
        for (int k4 = 0; k4 < BK / 4; k4++) {
            const int c = k4 & 1;
            if (k4 + 1 < BK / 4) {
#pragma unroll
                for (int i = 0; i < 4; i++) av[c ^ 1][i] = a[4 * (k4 + 1) * ASTR + 8 * i];
#pragma unroll
                for (int j = 0; j < TNW; j++) bv[c ^ 1][j] = b[4 * (k4 + 1) * BSTR + 8 * j];
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < TNW; j++) dmma(acc[i][j][0], acc[i][j][1], av[c][i], bv[c][j]);
        }
    }
    qd::cp_wait<0>();

    // lane holds real row wm*32 + 8i + lane/4 (frequency f0 + row/2, part row&1)
    // and ranges wn*8 TNW + 8j + 2(lane%4) + {0,1}
    double* const dst = reinterpret_cast<double*>(part ? part + (size_t)blockIdx.z * nf * nr : G);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = wm * 32 + 8 * i + (lane >> 2);
        const int f = f0 + (row >> 1), pr = row & 1;
        if (f >= nf) continue;
        const double cp = pr ? C[f].im : C[f].re;
#pragma unroll
        for (int j = 0; j < TNW; j++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int jj = n0 + wn * 8 * TNW + 8 * j + 2 * (lane & 3) + e;
                if (jj >= nr) continue;
                double v = acc[i][j][e];
                if (!part) v = (cp / ranges[jj] - (0.5 * dk) * cp) + v;  // fk.go:529-532
                dst[2 * ((size_t)f * nr + jj) + pr] = v;
            }
    }
}

int quad_gemm_splits(int nf, int nk, int nr) {
    // one block per SM of 148: the smallest split count (<= 64, each split
    // >= 8 wavenumber tiles) whose blocks fill the waves within 2% of the best
    // count's (more splits only add partial sums); banks of many waves keep one
    const int bn = nr > 64 ? 128 : 64;
    const long long tiles = (long long)((nr + bn - 1) / bn) * ((2 * nf + qd::BM - 1) / qd::BM);
    const int ntiles = (nk + qd::BK - 1) / qd::BK;
    if (tiles >= 8 * 148) return 1;
    const int smax = std::min(64, std::max(1, ntiles / 8));
    auto eff = [&](int s) {
        const long long blocks = tiles * s;
        return (double)blocks / ((double)((blocks + 147) / 148) * 148.0);
    };
    double best = 0.0;
    for (int s = 1; s <= smax; s++) best = std::max(best, eff(s));
    for (int s = 1; s <= smax; s++)
        if (eff(s) >= best - 0.02) return s;
    return 1;
}

namespace {
template <class K>
void set_smem_once(K kernel, int bytes, std::atomic<bool>* done) {
    if (!done->load(std::memory_order_relaxed) &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess)
        done->store(true, std::memory_order_relaxed);
}
}  // namespace

void launch_quad_gemm(cudaStream_t s, const cd* rem, const double* W, const cd* C, const double* ranges, int nf,
                      int nk, int nr, double dk, cd* G, int splits, cd* part) {
    if (nf <= 0 || nr <= 0) return;
    if (splits < 1 || !part) splits = 1;
    cd* const p = splits > 1 ? part : nullptr;
    // a failed attribute call leaves the launch to fail, and the caller's
    // cudaGetLastError to report it
    static std::atomic<bool> a8{false}, a4{false};
    if (nr > 64) {
        set_smem_once(k_quad_gemm<8>, qd::smem_bytes<8>(), &a8);
        dim3 grid((nr + 127) / 128, (2 * nf + qd::BM - 1) / qd::BM, splits);
        k_quad_gemm<8><<<grid, qd::THREADS, qd::smem_bytes<8>(), s>>>(rem, W, C, ranges, nf, nk, nr, dk, G, p);
    } else {
        set_smem_once(k_quad_gemm<4>, qd::smem_bytes<4>(), &a4);
        dim3 grid((nr + 63) / 64, (2 * nf + qd::BM - 1) / qd::BM, splits);
        k_quad_gemm<4><<<grid, qd::THREADS, qd::smem_bytes<4>(), s>>>(rem, W, C, ranges, nf, nk, nr, dk, G, p);
    }
    if (splits > 1) launch_quad_finish(s, part, splits, C, ranges, nf, nr, dk, G);
}

__global__ void k_quad_finish(const cd* __restrict__ part, int splits, const cd* __restrict__ C,
                              const double* __restrict__ ranges, int nf, int nr, double dk, cd* __restrict__ G) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nf * nr) return;
    const int f = (int)(i / nr), j = (int)(i % nr);
    cd acc = part[i];
    for (int z = 1; z < splits; z++) acc = acc + part[(size_t)z * nf * nr + i];
    const cd c = C[f];
    G[i] = (c / ranges[j] - (0.5 * dk) * c) + acc;  // fk.go:529-532
}

void launch_quad_finish(cudaStream_t s, const cd* part, int splits, const cd* C, const double* ranges, int nf,
                        int nr, double dk, cd* G) {
    const long long n = (long long)nf * nr;
    if (n <= 0) return;
    k_quad_finish<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(part, splits, C, ranges, nf, nr, dk, G);
}

// ---------------------------------------------- per-frequency-grid sum --
//
// Rows whose grids differ share no weight table: J0 is evaluated in the loop
// (fk.go:529-548), so the FP64 pipe bounds the sum (about 35 instructions per
// wavenumber and range for J0, 2 for the sum). One block serves one item (kc
// consecutive wavenumbers of one row) and RT ranges: its threads run over the
// wavenumbers, so the lanes of a warp take the same J0 branch, and each loads
// an integrand value once for RT ranges; then a fixed-order reduction and one
// partial per (item, range), which k_rows_finish adds in item order
// (deterministic). Items, not rows, are the unit because row lengths differ a
// hundredfold (a low bin's step is set by its own k/8Q): one thread per range
// walking its row took 242 ms on a 614-bin x 270-range loam bank (7.3M
// wavenumbers), most of it one block per SM on the longest rows; this takes
// 5.7 ms, 70% of what 39 FP64 instructions per value allow. Where all RT
// arguments are in the asymptotic range the J0s run as RT branchless chains
// side by side: with a branch per value they ran one after the other and the
// FP64 latency showed (10.2 ms).

constexpr int kRowThreads = 128;

template <int RT>
__global__ __launch_bounds__(kRowThreads) void k_quad_rows(const cd* __restrict__ ku, const cd* __restrict__ C,
                                                          const double* __restrict__ ranges, int nr,
                                                          const FreqDesc* __restrict__ fd, RowItems it,
                                                          cd* __restrict__ part) {
    __shared__ double s_red[kRowThreads / 32][2 * RT];
    const int tiles = (nr + RT - 1) / RT;
    const int item = blockIdx.x / tiles, tid = threadIdx.x;
    const int f = it.row ? it.row[item] - it.row0 : 0;
    const int first = (item - (it.begin ? it.begin[f] - it.item0 : 0)) * it.kc;
    const FreqDesc fdesc = fd[f];
    const int n = fdesc.nk, last = min(first + it.kc, n);
    const double d = fdesc.dk;
    const int r0 = (blockIdx.x - item * tiles) * RT, nv = min(RT, nr - r0);
    double r[RT], acc[2 * RT];
    double rmin = INFINITY, rmax = 0.0;
#pragma unroll
    for (int q = 0; q < RT; q++) {
        r[q] = ranges[r0 + min(q, nv - 1)];  // past the last range: its sums again, not stored
        rmin = fmin(rmin, r[q]);
        rmax = fmax(rmax, r[q]);
        acc[2 * q] = acc[2 * q + 1] = 0.0;
    }
    const cd* row = ku + fdesc.off;
    const cd c = C[f];
    for (int i = first + tid + 1; i <= last; i += kRowThreads) {
        const double k = (double)i * d;
        const cd v = (row[i - 1] - c) * (i == n ? 0.5 * d : d);
        if (k * rmin >= kJ0Asymptotic && k * rmax < kJ0Largest) {  // RT independent chains, no branch among them
#pragma unroll
            for (int q = 0; q < RT; q++) {
                const double w = j0_modulus_phase(k * r[q]);
                acc[2 * q] = fma(w, v.re, acc[2 * q]);
                acc[2 * q + 1] = fma(w, v.im, acc[2 * q + 1]);
            }
        } else {
#pragma unroll
            for (int q = 0; q < RT; q++) {
                const double w = j0_(k * r[q]);
                acc[2 * q] = fma(w, v.re, acc[2 * q]);
                acc[2 * q + 1] = fma(w, v.im, acc[2 * q + 1]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 2 * RT; q++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_down_sync(0xffffffffu, acc[q], o);
    if ((tid & 31) == 0)
#pragma unroll
        for (int q = 0; q < 2 * RT; q++) s_red[tid >> 5][q] = acc[q];
    __syncthreads();
    if (tid < 2 * nv) {
        double t = s_red[0][tid];
#pragma unroll
        for (int w = 1; w < kRowThreads / 32; w++) t += s_red[w][tid];
        reinterpret_cast<double*>(part)[2 * ((size_t)item * nr + r0) + tid] = t;
    }
}

__global__ void k_rows_finish(const cd* __restrict__ part, const cd* __restrict__ C,
                              const double* __restrict__ ranges, int nf, int nr, const FreqDesc* __restrict__ fd,
                              RowItems it, cd* __restrict__ G) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nf * nr) return;
    const int f = (int)(t / nr), j = (int)(t - (long long)f * nr);
    const int b = it.begin ? it.begin[f] - it.item0 : 0;
    const int e = it.begin ? it.begin[f + 1] - it.item0 : it.items;
    cd acc = mk(0.0);
#pragma unroll 8
    for (int i = b; i < e; i++) acc += part[(size_t)i * nr + j];
    const cd c = C[f];
    G[t] = (c / ranges[j] - (0.5 * fd[f].dk) * c) + acc;  // fk.go:529-532
}

void launch_quad_rows(cudaStream_t s, const cd* ku, const cd* C, const double* ranges, int nf, int nr,
                      const FreqDesc* fd, const RowItems& it, cd* part, cd* G) {
    if (nf <= 0 || nr <= 0) return;
    if (it.items > 0) {
        // 8 ranges per block: one integrand load and one reduction per 8 J0s
        // (16 accumulators); fewer ranges take the smallest tile holding them
        if (nr <= 1)
            k_quad_rows<1><<<it.items, kRowThreads, 0, s>>>(ku, C, ranges, nr, fd, it, part);
        else if (nr <= 2)
            k_quad_rows<2><<<it.items, kRowThreads, 0, s>>>(ku, C, ranges, nr, fd, it, part);
        else if (nr <= 4)
            k_quad_rows<4><<<it.items, kRowThreads, 0, s>>>(ku, C, ranges, nr, fd, it, part);
        else
            k_quad_rows<8><<<(unsigned)it.items * ((nr + 7) / 8), kRowThreads, 0, s>>>(ku, C, ranges, nr, fd, it, part);
    }
    k_rows_finish<<<(unsigned)(((long long)nf * nr + 127) / 128), 128, 0, s>>>(part, C, ranges, nf, nr, fd, it, G);
}

int rows_item_size(long long wavenumbers, int nr) {
    // about 16 blocks per SM of 148 over the launch's (item, range tile) blocks,
    // between 2 wavenumbers a thread (a single response: latency) and 64 (the
    // reduction, ~200 instructions a thread, is then under 1% of 64 x 8 J0s)
    const long long tiles = nr <= 8 ? 1 : (nr + 7) / 8;
    long long kc = wavenumbers * tiles / (148 * 16);
    kc = (kc + kRowThreads - 1) / kRowThreads * kRowThreads;
    return (int)std::min<long long>(std::max<long long>(kc, 2 * kRowThreads), 64 * kRowThreads);
}

// ------------------------------------------------------------ bank pack --

__global__ void k_bank_pack(const cd* __restrict__ G, int nf, int nr, int first_bin, int bins,
                            float* __restrict__ payload) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)nf * nr) return;
    const int j = (int)(idx / nf);
    const int f = (int)(idx - (int64_t)j * nf);
    const int bin = first_bin + f;
    if (bin < 0 || bin >= bins) return;
    const cd v = G[(size_t)f * nr + j];
    const size_t o = 2 * ((size_t)j * bins + bin);
    payload[o] = (float)v.re;
    payload[o + 1] = (float)v.im;
}

void launch_bank_pack(cudaStream_t s, const cd* G, int nf, int nr, int first_bin, int bins, float* payload) {
    const int64_t n = (int64_t)nf * nr;
    k_bank_pack<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(G, nf, nr, first_bin, bins, payload);
}

}  // namespace gfk
