// gfk_fft.cuh — FP64 complex FFTs of one power-of-two record in shared
// memory, by the block that calls it: fft_pow2 by radix-2 passes between two
// buffers, fft_block by radix-8 passes through registers in one.
//
// fft_pow2 is the autosort (Stockham) formulation of Govindaraju et al., SC 2008: at the
// stage with sub-transform length ns, butterfly j (< n/2) reads x[j] and
// x[j + n/2] and writes y[2 ns (j / ns) + j % ns] and that + ns, with twiddle
// e^{-2 pi i (j % ns) / (2 ns)} = tw[(j % ns) (n / (2 ns))], tw[m] =
// e^{-2 pi i m / n}. Results come out in natural order.
#pragma once
#include "gfk_math.cuh"

namespace gfk {

// Forward transform (e^{-i}) of x[0, n); y is scratch of the same size. The
// result ends in x when log2(n) is even, in y otherwise; the return value
// points at it. Every thread of the block must call it.
__device__ inline cd* fft_pow2(cd* x, cd* y, int n, const cd* __restrict__ tw) {
    cd* src = x;
    cd* dst = y;
    for (int ns = 1; ns < n; ns <<= 1) {
        for (int j = threadIdx.x; j < n / 2; j += blockDim.x) {
            const int k = j & (ns - 1);
            const cd w = tw[k * (n / (2 * ns))];
            const cd a0 = src[j];
            const cd a1 = src[j + n / 2] * w;
            const int d = ((j - k) << 1) + k;
            dst[d] = a0 + a1;
            dst[d + ns] = a0 - a1;
        }
        __syncthreads();
        cd* t = src;
        src = dst;
        dst = t;
    }
    return src;
}

// Forward DFT (e^{-i}) of R = 2, 4 or 8 values in registers.
template <int R>
__device__ __forceinline__ void dft_small(cd (&v)[R]) {
    if constexpr (R == 2) {
        const cd t = v[1];
        v[1] = v[0] - t;
        v[0] = v[0] + t;
    } else if constexpr (R == 4) {
        const cd a = v[0] + v[2], b = v[0] - v[2], c = v[1] + v[3], d = v[1] - v[3];
        v[0] = a + c;
        v[2] = a - c;
        v[1] = cd{b.re + d.im, b.im - d.re};  // b - i d
        v[3] = cd{b.re - d.im, b.im + d.re};
    } else {
        static_assert(R == 8, "radix");
        cd e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        dft_small<4>(e);
        dft_small<4>(o);
        constexpr double h = 0.70710678118654752440;
        o[1] = cd{h * (o[1].re + o[1].im), h * (o[1].im - o[1].re)};
        o[2] = cd{o[2].im, -o[2].re};
        o[3] = cd{h * (o[3].im - o[3].re), -h * (o[3].re + o[3].im)};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            v[i] = e[i] + o[i];
            v[i + 4] = e[i] - o[i];
        }
    }
}

// Element i of a record in shared memory lies at fft_at(i): a gap of one
// (16-byte) element after every eight, so that neither the radix-8 passes'
// strided stores nor their contiguous loads conflict.
__device__ __forceinline__ int fft_at(int i) { return i + (i >> 3); }
__host__ __device__ constexpr int fft_room(int m) { return m + m / 8 + 1; }

// One radix-R Stockham pass over m values by the block's first max(32, m / 8)
// threads, each with up to 8 / R butterflies: loads x, then (all threads) emit(element, value)
// for every output. tw[q] = e^{-2 pi i q / tn}, q < tn/2, tn a multiple of m;
// ns is the product of the radices before. Twiddles: w, w^2, w^4 from the
// table, the others as their products.
template <int R, class Emit>
__device__ __forceinline__ void fft_pass(const cd* x, int m, int ns, const cd* __restrict__ tw, int tn, Emit emit) {
    constexpr int B = 8 / R;
    const int stride = m / R, tid = threadIdx.x, nt = m >= 256 ? m / 8 : 32;
    cd v[B][R];
#pragma unroll
    for (int b = 0; b < B; b++) {
        const int j = tid + b * nt;
        if ((B == 1 || tid < nt) && j < stride) {
#pragma unroll
            for (int r = 0; r < R; r++) v[b][r] = x[fft_at(j + r * stride)];
        }
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < B; b++) {
        const int j = tid + b * nt;
        if ((B > 1 && tid >= nt) || j >= stride) continue;
        const int k = j & (ns - 1);
        if (ns > 1) {
            const int q = k * (tn / (ns * R));
            cd w[R];
            w[1] = tw[q];
            if constexpr (R >= 4) {
                w[2] = tw[2 * q];  // 2 q < 2 tn / R <= tn / 2
                w[3] = w[1] * w[2];
            }
            if constexpr (R == 8) {
                const int q4 = 4 * q;  // < tn / 2
                w[4] = tw[q4];
                w[5] = w[4] * w[1];
                w[6] = w[4] * w[2];
                w[7] = w[4] * w[3];
            }
#pragma unroll
            for (int r = 1; r < R; r++) v[b][r] = v[b][r] * w[r];
        }
        dft_small<R>(v[b]);
        const int d = (j - k) * R + k;
#pragma unroll
        for (int r = 0; r < R; r++) emit(d + r * ns, v[b][r]);
    }
}

// Forward transform (e^{-i}) of the m = 2^logm values at x[fft_at(i)], the last
// pass handing its outputs, in natural order, to emit(i, value) instead of
// shared memory. The block has at least max(32, m / 8) threads; all must call it, with
// x written and a barrier passed. Every pass but the first is radix 8: a third of the
// passes (and of the shared-memory traffic and barriers) of radix 2.
template <class Emit>
__device__ __forceinline__ void fft_block(cd* x, int logm, const cd* __restrict__ tw, int tn, Emit emit) {
    const int m = 1 << logm;
    const int head = logm % 3;
    auto keep = [&](int i, cd v) { x[fft_at(i)] = v; };
    if (logm == 0) {
        if (threadIdx.x == 0) emit(0, x[0]);
        return;
    }
    if (logm == 1) return fft_pass<2>(x, m, 1, tw, tn, emit);
    if (logm == 2) return fft_pass<4>(x, m, 1, tw, tn, emit);
    int ns = 1;
    if (head == 1) fft_pass<2>(x, m, 1, tw, tn, keep), ns = 2;
    if (head == 2) fft_pass<4>(x, m, 1, tw, tn, keep), ns = 4;
    if (head) __syncthreads();
    for (; ns * 8 < m; ns *= 8) {
        fft_pass<8>(x, m, ns, tw, tn, keep);
        __syncthreads();
    }
    fft_pass<8>(x, m, ns, tw, tn, emit);
}

}  // namespace gfk
