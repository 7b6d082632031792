// gfk_fdtd.cu — the reference's axisymmetric finite-difference validator
// (internal/fdtd) on the GPU: a vertical point force on the free surface of a
// layered, optionally viscoelastic (one standard linear solid) half-space, in
// cylindrical coordinates, Virieux staggering, C-PML absorbing layers.
//
// What is restated, from internal/fdtd:
//   grid, time step, materials   fdtd.go:45-98, model.go:30-246 (host)
//   C-PML profiles                pml.go:30-70 (host), update pml.go:66-70
//   velocities                    fdtd.go:149-216
//   stresses and memory variables fdtd.go:218-320
//   surface velocity read-out     fdtd.go:330-345, Run's loop run.go:78-127
//
// Every phase of a step is a pure function of the previous phase's fields. A
// step's new stresses depend on the old ones at most one cell away, so a block
// that loads a tile and a halo of S cells can take S steps in shared memory
// before it writes its tile back (k_tiles): one launch and one pass over memory
// per S steps. The fields are double-buffered, because neighbouring tiles read
// what this one writes. Where the second copy does not fit the device (or
// GFK_FDTD_COPIES=1 asks for one), each phase is one kernel over the grid in place (k_velocities, which also writes
// the prescribed surface traction, and k_stresses, which also records the
// receivers: their velocities are final by then). The arithmetic of every cell is the
// reference's, in the same order, except that divisions by the spacing, the
// radius and the density are multiplications by precomputed reciprocals (the
// same values to a rounding); FP64 throughout. Every 256 steps a max-speed
// reduction checks for divergence, as Run does.
#include <cmath>
#include <complex>
#include <cstdlib>
#include <string>
#include <utility>
#include <vector>

#include <math_constants.h>

#include "../../include/gfk.h"
#include "gfk_ctx.h"
#include "gfk_kernels.cuh"

namespace gfk {
namespace fdtd {

struct Args {
    int nr, nz;
    double dr, dz, dt, src_area;
    bool lossy;
    double mem_decay, mem_drive;
    // materials per row; the time step over the densities, precomputed
    const double *lamU, *muU, *muZ;
    const double *dt_rho, *dt_rhoZ;
    // reciprocal spacings and radii: 1 / dr, 1 / dz, 1 / ((i + 1/2) dr), 1 / (i dr)
    double idr, idz;
    const double *ir_half, *ir_int;
    // C-PML profiles (a, b) and the first damped index of each
    const double *aRi, *bRi, *aRh, *bRh, *aZi, *bZi, *aZh, *bZh;
    int fRi, fRh, fZi, fZh;
    // fields [nz][nr]
    double *vr, *vz, *trr, *tqq, *tzz, *trz;
    double *rrr, *rqq, *rzz, *rrz;
    double *psiTrrR, *psiTrzZ, *psiTrzR, *psiTzzZ, *psiVrR, *psiVzZ, *psiVzR, *psiVrZ;
    // receivers
    const int* cols;
    int nrcv, steps;
    double* traces;  // [nrcv][steps]
};

__device__ __forceinline__ double cpml(double* psi, double a, double b, double deriv) {
    const double p = b * *psi + a * deriv;
    *psi = p;
    return p;
}

__device__ __forceinline__ double relax(const Args& s, double* r, double e) {
    const double next = s.mem_decay * *r - s.mem_drive * e;
    const double avg = 0.5 * (*r + next);
    *r = next;
    return avg;
}

__global__ void k_velocities(Args s, double surface_traction) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= s.nr - 1 || j >= s.nz - 1) return;
    const int nr = s.nr;
    const int k = j * nr + i;
    // radial velocity
    {
        double dtrr = (s.trr[k + 1] - s.trr[k]) * s.idr;
        if (i >= s.fRh) dtrr += cpml(&s.psiTrrR[k], s.aRh[i], s.bRh[i], dtrr);
        double dtrz = j == 0 ? 2 * s.trz[k] * s.idz : (s.trz[k] - s.trz[k - nr]) * s.idz;
        if (j >= s.fZi) dtrz += cpml(&s.psiTrzZ[k], s.aZi[j], s.bZi[j], dtrz);
        const double hoop = 0.5 * ((s.trr[k] - s.tqq[k]) + (s.trr[k + 1] - s.tqq[k + 1])) * s.ir_half[i];
        s.vr[k] += s.dt_rho[j] * (dtrr + dtrz + hoop);
    }
    // vertical velocity
    {
        const double tzz_k = k == 0 ? surface_traction : s.tzz[k];
        if (k == 0) s.tzz[0] = surface_traction;  // fdtd.go:144
        double dtzz = (s.tzz[k + nr] - tzz_k) * s.idz;
        if (j >= s.fZh) dtzz += cpml(&s.psiTzzZ[k], s.aZh[j], s.bZh[j], dtzz);
        double radial;
        if (i == 0) {
            radial = 4 * s.trz[k] * s.idr;
        } else {
            double d = (s.trz[k] - s.trz[k - 1]) * s.idr;
            if (i >= s.fRi) d += cpml(&s.psiTrzR[k], s.aRi[i], s.bRi[i], d);
            radial = d + 0.5 * (s.trz[k] + s.trz[k - 1]) * s.ir_int[i];
        }
        s.vz[k] += s.dt_rhoZ[j] * (dtzz + radial);
    }
}

__device__ double surface_velocity(const Args& s, int i) {
    double dvr, vrr;
    if (i == 0) {
        dvr = 2 * s.vr[0] / s.dr;
        vrr = dvr;
    } else {
        dvr = (s.vr[i] - s.vr[i - 1]) / s.dr;
        vrr = 0.5 * (s.vr[i] + s.vr[i - 1]) / (double(i) * s.dr);
    }
    const double lam = s.lamU[0], mu = s.muU[0];
    const double dvz = -lam / (lam + 2 * mu) * (dvr + vrr);
    return s.vz[i] - 0.5 * s.dz * dvz;
}

__global__ void k_stresses(Args s, double dTdt, int step) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.y == 0)
        for (int q = threadIdx.x; q < s.nrcv; q += blockDim.x)
            s.traces[(size_t)q * s.steps + step] = surface_velocity(s, s.cols[q]);
    if (i >= s.nr || j >= s.nz) return;
    const int nr = s.nr;
    const int k = j * nr + i;
    const double lam = s.lamU[j], mu = s.muU[j];
    const double lam2mu = lam + 2 * mu;
    // normal stresses
    double dvr, vrr;
    if (i == 0) {
        dvr = 2 * s.vr[k] * s.idr;
        vrr = dvr;
    } else {
        dvr = (s.vr[k] - s.vr[k - 1]) * s.idr;
        vrr = 0.5 * (s.vr[k] + s.vr[k - 1]) * s.ir_int[i];
    }
    if (i >= s.fRi) dvr += cpml(&s.psiVrR[k], s.aRi[i], s.bRi[i], dvr);
    double dvz;
    if (j == 0) {
        const double applied = i == 0 ? dTdt : 0.0;
        dvz = (applied - lam * (dvr + vrr)) / lam2mu;
    } else {
        dvz = (s.vz[k] - s.vz[k - nr]) * s.idz;
        if (j >= s.fZi) dvz += cpml(&s.psiVzZ[k], s.aZi[j], s.bZi[j], dvz);
    }
    const double err = lam2mu * dvr + lam * (vrr + dvz);
    const double eqq = lam * (dvr + dvz) + lam2mu * vrr;
    if (s.lossy) {
        s.trr[k] += s.dt * (err + relax(s, &s.rrr[k], err));
        s.tqq[k] += s.dt * (eqq + relax(s, &s.rqq[k], eqq));
    } else {
        s.trr[k] += s.dt * err;
        s.tqq[k] += s.dt * eqq;
    }
    if (j != 0) {
        const double ezz = lam * (dvr + vrr) + lam2mu * dvz;
        if (s.lossy)
            s.tzz[k] += s.dt * (ezz + relax(s, &s.rzz[k], ezz));
        else
            s.tzz[k] += s.dt * ezz;
    }
    // shear stress
    if (i < nr - 1 && j < s.nz - 1) {
        double dvzdr = (s.vz[k + 1] - s.vz[k]) * s.idr;
        if (i >= s.fRh) dvzdr += cpml(&s.psiVzR[k], s.aRh[i], s.bRh[i], dvzdr);
        double dvrdz = (s.vr[k + nr] - s.vr[k]) * s.idz;
        if (j >= s.fZh) dvrdz += cpml(&s.psiVrZ[k], s.aZh[j], s.bZh[j], dvrdz);
        const double e = s.muZ[j] * (dvzdr + dvrdz);
        if (s.lossy)
            s.trz[k] += s.dt * (e + relax(s, &s.rrz[k], e));
        else
            s.trz[k] += s.dt * e;
    }
}

// ---- S steps per pass over memory --
//
// A block of 512 threads holds a 32 x 32 window of the fields: its tile of
// (32 - 2S)^2 cells and the halo. A thread keeps its two cells' velocities,
// stresses, memory variables and constants in registers; what the neighbours
// read (velocities and stresses) and the C-PML variables also lie in shared
// memory. Per step the valid part of the window shrinks by one cell on every
// side that is not a domain edge; each phase runs over what is still valid.
// Cells of the window's rim lack a neighbour and are skipped, which is what the
// shrinking accounts for. With every field in shared memory a step read and
// wrote it 50 times a cell and its bandwidth bound the step. On a
// 281 x 201 grid one launch per phase left 13.6 us a step, nearly all launch
// and L2 latency on 382 cells an SM; on 6 million cells the two phases moved
// 208 bytes a cell and step, here 220 per 4 steps.

constexpr int kTileW = 32, kTileCells = kTileW * kTileW, kTileThreads = kTileCells / 2, kOwn = 2;
constexpr int kFields = 18, kMaxTileSteps = 10;
enum : int { kVr, kVz, kTrr, kTqq, kTzz, kTrz, kRrr, kRqq, kRzz, kRrz, kTrrR, kTrzZ, kTrzR, kTzzZ, kVrR, kVzZ, kVzR, kVrZ };
constexpr int kTileSmem = (6 + 8) * kTileCells * (int)sizeof(double);

struct Tiles {
    const double* in[kFields];
    double* out[kFields];
    const double* force;  // [steps + 1]
    int S, n, step0;      // halo, steps of this launch (<= S), first step
};

template <bool LOSSY>
__global__ void __launch_bounds__(kTileThreads, 1) k_tiles(Args s, Tiles t) {
    extern __shared__ double sm[];
    double* const vr = sm;
    double* const vz = vr + kTileCells;
    double* const trr = vz + kTileCells;
    double* const tqq = trr + kTileCells;
    double* const tzz = tqq + kTileCells;
    double* const trz = tzz + kTileCells;
    double* const psi = trz + kTileCells;  // [8]: kTrrR .. kVrZ
    const int li = threadIdx.x & (kTileW - 1);
    const int tw = kTileW - 2 * t.S;
    const int x0 = blockIdx.x * tw, z0 = blockIdx.y * tw;  // the tile's first cell
    const int gx = x0 - t.S, gz = z0 - t.S;                // the window's
    const int i = gx + li, ic = min(max(i, 0), s.nr - 1);
    // whether the window reaches the damped columns or rows (the psi fields are zero elsewhere)
    const bool damp_r = gx + kTileW > min(s.fRi, s.fRh), damp_z = gz + kTileW > min(s.fZi, s.fZh);
    const bool radial_psi[8] = {true, false, true, false, true, false, true, false};
    // this thread's two cells (rows lj and lj + 16 of the window)
    double ovr[kOwn], ovz[kOwn], orr[kOwn], oqq[kOwn], ozz[kOwn], orz[kOwn], m[kOwn][4];
    double dt_rho[kOwn], dt_rhoZ[kOwn], lam[kOwn], mu[kOwn], muZ[kOwn];
    double ps[kOwn][8];
    // every load first, then the stores to shared memory: nothing tells the
    // compiler that these pointers cannot reach shared memory, and it keeps the
    // order of what might overlap (8 us a launch when they alternated)
#pragma unroll
    for (int c = 0; c < kOwn; c++) {
        const int j = gz + (int)(threadIdx.x >> 5) + 16 * c;
        const bool in = i >= 0 && i < s.nr && j >= 0 && j < s.nz;
        const size_t k = (size_t)j * s.nr + i;
        ovr[c] = in ? __ldg(t.in[kVr] + k) : 0.0;
        ovz[c] = in ? __ldg(t.in[kVz] + k) : 0.0;
        orr[c] = in ? __ldg(t.in[kTrr] + k) : 0.0;
        oqq[c] = in ? __ldg(t.in[kTqq] + k) : 0.0;
        ozz[c] = in ? __ldg(t.in[kTzz] + k) : 0.0;
        orz[c] = in ? __ldg(t.in[kTrz] + k) : 0.0;
#pragma unroll
        for (int f = 0; f < 4; f++) m[c][f] = LOSSY && in ? __ldg(t.in[kRrr + f] + k) : 0.0;
#pragma unroll
        for (int f = 0; f < 8; f++) ps[c][f] = in && (radial_psi[f] ? damp_r : damp_z) ? __ldg(t.in[kTrrR + f] + k) : 0.0;
        const int jc = min(max(j, 0), s.nz - 1);
        dt_rho[c] = __ldg(s.dt_rho + jc);
        dt_rhoZ[c] = __ldg(s.dt_rhoZ + jc);
        lam[c] = __ldg(s.lamU + jc);
        mu[c] = __ldg(s.muU + jc);
        muZ[c] = __ldg(s.muZ + jc);
    }
#pragma unroll
    for (int c = 0; c < kOwn; c++) {
        const int e = ((threadIdx.x >> 5) + 16 * c) * kTileW + li;
        vr[e] = ovr[c];
        vz[e] = ovz[c];
        trr[e] = orr[c];
        tqq[e] = oqq[c];
        tzz[e] = ozz[c];
        trz[e] = orz[c];
#pragma unroll
        for (int f = 0; f < 8; f++)
            if (radial_psi[f] ? damp_r : damp_z) psi[f * kTileCells + e] = ps[c][f];
    }
    const double ir_half = s.ir_half[ic], ir_int = s.ir_int[ic];
    __syncthreads();
    const bool source = gx <= 0 && gz <= 0;  // the window holds cell (0, 0)
    auto damp = [&](int f, int e, const double* a, const double* b, int at, double d) {
        return cpml(psi + (f - kTrrR) * kTileCells + e, a[at], b[at], d);
    };
    for (int n = 0; n < t.n; n++) {
        const int step = t.step0 + n;
        double traction = 0.0, rate = 0.0;  // at cell (0, 0) only
        if (source) {
            traction = -t.force[step] / s.src_area;
            rate = (t.force[step + 1] - t.force[step]) / s.dt;
        }
        // the part still valid, in window coordinates
        const int l0 = gx <= 0 ? -gx : n, l1 = gx + kTileW >= s.nr ? s.nr - gx : kTileW - n;
        const int h0 = gz <= 0 ? -gz : n, h1 = gz + kTileW >= s.nz ? s.nz - gz : kTileW - n;
        const bool col = li >= l0 && li < l1;
        // both cells' neighbours are read before either is written (as above);
        // an index past the window's rim is clamped, its cell is skipped below
        double n1[kOwn], n2[kOwn], n3[kOwn], n4[kOwn], n5[kOwn];
#pragma unroll
        for (int c = 0; c < kOwn; c++) {
            const int lj = (threadIdx.x >> 5) + 16 * c, e = lj * kTileW + li;
            const int er = min(e + 1, kTileCells - 1), eu = max(e - kTileW, 0), ed = min(e + kTileW, kTileCells - 1);
            n1[c] = trr[er];
            n2[c] = tqq[er];
            n3[c] = trz[eu];
            n4[c] = tzz[ed];
            n5[c] = trz[max(e - 1, 0)];
        }
#pragma unroll
        for (int c = 0; c < kOwn; c++) {
            const int lj = (threadIdx.x >> 5) + 16 * c, e = lj * kTileW + li, j = gz + lj;
            if (!col || lj < h0 || lj >= h1 || i >= s.nr - 1 || j >= s.nz - 1) continue;
            if (li + 1 < kTileW && (lj > 0 || j == 0)) {  // radial velocity
                double dtrr = (n1[c] - orr[c]) * s.idr;
                if (i >= s.fRh) dtrr += damp(kTrrR, e, s.aRh, s.bRh, i, dtrr);
                double dtrz = j == 0 ? 2 * orz[c] * s.idz : (orz[c] - n3[c]) * s.idz;
                if (j >= s.fZi) dtrz += damp(kTrzZ, e, s.aZi, s.bZi, j, dtrz);
                const double hoop = 0.5 * ((orr[c] - oqq[c]) + (n1[c] - n2[c])) * ir_half;
                ovr[c] += dt_rho[c] * (dtrr + dtrz + hoop);
            }
            if (lj + 1 < kTileW && (li > 0 || i == 0)) {  // vertical velocity
                if (i == 0 && j == 0) ozz[c] = traction;  // fdtd.go:144
                double dtzz = (n4[c] - ozz[c]) * s.idz;
                if (j >= s.fZh) dtzz += damp(kTzzZ, e, s.aZh, s.bZh, j, dtzz);
                double radial;
                if (i == 0) {
                    radial = 4 * orz[c] * s.idr;
                } else {
                    double d = (orz[c] - n5[c]) * s.idr;
                    if (i >= s.fRi) d += damp(kTrzR, e, s.aRi, s.bRi, i, d);
                    radial = d + 0.5 * (orz[c] + n5[c]) * ir_int;
                }
                ovz[c] += dt_rhoZ[c] * (dtzz + radial);
            }
        }
#pragma unroll
        for (int c = 0; c < kOwn; c++) {
            const int e = ((threadIdx.x >> 5) + 16 * c) * kTileW + li;
            vr[e] = ovr[c];
            vz[e] = ovz[c];
        }
        __syncthreads();
        // receivers of this tile's surface cells
        if (z0 == 0)
            for (int q = threadIdx.x; q < s.nrcv; q += kTileThreads) {
                const int ri = s.cols[q];
                if (ri < x0 || ri >= x0 + tw) continue;
                const int e = -gz * kTileW + ri - gx;
                double dvr, vrr;
                if (ri == 0) {
                    dvr = 2 * vr[e] / s.dr;
                    vrr = dvr;
                } else {
                    dvr = (vr[e] - vr[e - 1]) / s.dr;
                    vrr = 0.5 * (vr[e] + vr[e - 1]) / (double(ri) * s.dr);
                }
                const double l = s.lamU[0], g = s.muU[0];
                const double dvz = -l / (l + 2 * g) * (dvr + vrr);
                s.traces[(size_t)q * s.steps + step] = vz[e] - 0.5 * s.dz * dvz;
            }
#pragma unroll
        for (int c = 0; c < kOwn; c++) {
            const int lj = (threadIdx.x >> 5) + 16 * c, e = lj * kTileW + li;
            n1[c] = vr[max(e - 1, 0)];
            n2[c] = vz[max(e - kTileW, 0)];
            n3[c] = vz[min(e + 1, kTileCells - 1)];
            n4[c] = vr[min(e + kTileW, kTileCells - 1)];
        }
#pragma unroll
        for (int c = 0; c < kOwn; c++) {
            const int lj = (threadIdx.x >> 5) + 16 * c, e = lj * kTileW + li, j = gz + lj;
            if (!col || lj < h0 || lj >= h1) continue;
            const double lam2mu = lam[c] + 2 * mu[c];
            if ((li > 0 || i == 0) && (lj > 0 || j == 0)) {  // normal stresses
                double dvr, vrr;
                if (i == 0) {
                    dvr = 2 * ovr[c] * s.idr;
                    vrr = dvr;
                } else {
                    dvr = (ovr[c] - n1[c]) * s.idr;
                    vrr = 0.5 * (ovr[c] + n1[c]) * ir_int;
                }
                if (i >= s.fRi) dvr += damp(kVrR, e, s.aRi, s.bRi, i, dvr);
                double dvz;
                if (j == 0) {
                    const double applied = i == 0 ? rate : 0.0;
                    dvz = (applied - lam[c] * (dvr + vrr)) / lam2mu;
                } else {
                    dvz = (ovz[c] - n2[c]) * s.idz;
                    if (j >= s.fZi) dvz += damp(kVzZ, e, s.aZi, s.bZi, j, dvz);
                }
                const double err = lam2mu * dvr + lam[c] * (vrr + dvz);
                const double eqq = lam[c] * (dvr + dvz) + lam2mu * vrr;
                orr[c] += s.dt * (LOSSY ? err + relax(s, &m[c][0], err) : err);
                oqq[c] += s.dt * (LOSSY ? eqq + relax(s, &m[c][1], eqq) : eqq);
                if (j != 0) {
                    const double ezz = lam[c] * (dvr + vrr) + lam2mu * dvz;
                    ozz[c] += s.dt * (LOSSY ? ezz + relax(s, &m[c][2], ezz) : ezz);
                }
            }
            if (i < s.nr - 1 && j < s.nz - 1 && li + 1 < kTileW && lj + 1 < kTileW) {  // shear stress
                double dvzdr = (n3[c] - ovz[c]) * s.idr;
                if (i >= s.fRh) dvzdr += damp(kVzR, e, s.aRh, s.bRh, i, dvzdr);
                double dvrdz = (n4[c] - ovr[c]) * s.idz;
                if (j >= s.fZh) dvrdz += damp(kVrZ, e, s.aZh, s.bZh, j, dvrdz);
                const double g = muZ[c] * (dvzdr + dvrdz);
                orz[c] += s.dt * (LOSSY ? g + relax(s, &m[c][3], g) : g);
            }
        }
#pragma unroll
        for (int c = 0; c < kOwn; c++) {
            const int e = ((threadIdx.x >> 5) + 16 * c) * kTileW + li;
            trr[e] = orr[c];
            tqq[e] = oqq[c];
            tzz[e] = ozz[c];
            trz[e] = orz[c];
        }
        __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < kOwn; c++) {
        const int lj = (threadIdx.x >> 5) + 16 * c, e = lj * kTileW + li, j = gz + lj;
        if (li < t.S || li >= t.S + tw || lj < t.S || lj >= t.S + tw || i >= s.nr || j >= s.nz) continue;
        const size_t k = (size_t)j * s.nr + i;
        t.out[kVr][k] = ovr[c];
        t.out[kVz][k] = ovz[c];
        t.out[kTrr][k] = orr[c];
        t.out[kTqq][k] = oqq[c];
        t.out[kTzz][k] = ozz[c];
        t.out[kTrz][k] = orz[c];
#pragma unroll
        for (int f = 0; f < 4; f++)
            if (LOSSY) t.out[kRrr + f][k] = m[c][f];
#pragma unroll
        for (int f = 0; f < 8; f++)
            if (radial_psi[f] ? damp_r : damp_z) t.out[kTrrR + f][k] = psi[f * kTileCells + e];
    }
}

// Steps per launch: the fewest estimated microseconds a step. A launch takes
// about 8 us for its window's loads and stores and 2.1 per step (fitted on one
// wave of tiles, S = 2 to 8), times its waves of one tile per SM of 148. On
// 281 x 201 cells S = 2, 3, 4, 5, 6 took 6.3, 4.6, 4.2, 4.2, 5.9 us a step, on 6.1
// million cells 223, 208, 209, 228, 259; one launch per phase 13.6 and 321.
int tile_steps(int nr, int nz) {
    int best = 1;
    double least = INFINITY;
    for (int S = 1; S <= kMaxTileSteps; S++) {
        const double tw = kTileW - 2 * S, tiles = ceil(nr / tw) * ceil(nz / tw);
        const double cost = ceil(tiles / 148) * (8.0 + 2.1 * S) / S;
        if (cost < least) {
            least = cost;
            best = S;
        }
    }
    return best;
}

// Block maxima of |vz| and |vr| (NaN propagates as NaN).
__global__ void k_maxspeed(const double* vz, const double* vr, long long n, double* out) {
    __shared__ double red[256];
    double m = 0.0;
    bool nan = false;
    for (long long q = blockIdx.x * 256LL + threadIdx.x; q < n; q += (long long)gridDim.x * 256) {
        const double a = fabs(vz[q]), b = fabs(vr[q]);
        nan |= isnan(a) || isnan(b);
        m = fmax(m, fmax(a, b));
    }
    red[threadIdx.x] = nan ? CUDART_NAN : m;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            const double x = red[threadIdx.x], y = red[threadIdx.x + w];
            red[threadIdx.x] = (isnan(x) || isnan(y)) ? CUDART_NAN : fmax(x, y);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = red[0];
}

}  // namespace fdtd
}  // namespace gfk

namespace {

using cplx = std::complex<double>;

struct Sls {
    double ts = 0, te = 0;
    bool lossy() const { return te > ts; }
    double delta() const { return te / ts - 1; }
    cplx modulus(double f) const {  // visco.go:78-81
        const cplx w(0, 2 * M_PI * f);
        return (1.0 + w * te) / (1.0 + w * ts);
    }
    double relaxed_velocity(double v, double fref) const {  // visco.go:100-102
        return v * (1.0 / std::sqrt(modulus(fref))).real();
    }
};

struct Grid {
    int nr = 0, nz = 0, pml = 0;
    double h = 0, dt = 0, vmax = 0, dominant = 0, fref = 30, refl = 1e-4;
    Sls sls;
};

int ffail(gfk_ctx* ctx, int st, const std::string& msg) {
    if (ctx) ctx->last_error = msg;
    return st;
}

const gfk_layer& layer_at(const gfk_medium& m, double z) {  // model.go:206-217
    double top = 0;
    for (int i = 0; i + 1 < m.count; i++) {
        top += m.layers[i].thickness_m;
        if (z < top) return m.layers[i];
    }
    return m.layers[m.count - 1];
}

int setup(gfk_ctx* ctx, const gfk_fdtd_model* md, Grid* g) {
    const gfk_medium& m = md->medium;
    if (!m.layers || m.count < 1) return ffail(ctx, GFK_ESTACK, "layer: empty stack");
    const int v = gfk_stack_validate(&m);
    if (v) return ffail(ctx, v, "layer: stack failed validation");
    if (!(md->spacing_m > 0)) return ffail(ctx, GFK_EARG, "fdtd: spacing must be positive");
    if (!(md->max_range_m > 0) || !(md->depth_m > 0)) return ffail(ctx, GFK_EARG, "fdtd: domain must be positive");
    g->sls.ts = m.sls_tau_sigma;
    g->sls.te = m.sls_tau_eps;
    if (g->sls.te < g->sls.ts)
        return ffail(ctx, GFK_EARG, "fdtd: TauEps must be at least TauSigma for a dissipative solid");
    g->fref = m.ref_freq_hz > 0 ? m.ref_freq_hz : 30.0;
    g->pml = md->pml_cells > 0 ? md->pml_cells : 20;
    g->refl = md->pml_reflection > 0 ? md->pml_reflection : 1e-4;
    const double courant = md->courant > 0 ? md->courant : 0.5;
    g->h = md->spacing_m;
    g->nr = (int)std::lround(md->max_range_m / g->h) + 1 + g->pml;
    g->nz = (int)std::lround(md->depth_m / g->h) + 1 + g->pml;
    double vmax = 0;  // model.go:219-233
    for (int i = 0; i < m.count; i++) {
        double vv = m.layers[i].vp_mps;
        if (g->sls.lossy()) vv = g->sls.relaxed_velocity(vv, g->fref) * std::sqrt(1 + g->sls.delta());
        vmax = std::max(vmax, vv);
    }
    g->vmax = vmax;
    g->dt = courant * (g->h / (vmax * M_SQRT2));
    if (md->dominant_freq_hz > 0) {
        g->dominant = md->dominant_freq_hz;
    } else {  // fdtd.go:106-117
        double slow = m.layers[0].vs_mps;
        for (int i = 0; i < m.count; i++) slow = std::min(slow, m.layers[i].vs_mps);
        if (g->sls.lossy()) slow = g->sls.relaxed_velocity(slow, g->fref);
        g->dominant = slow / (20 * g->h);
    }
    return GFK_OK;
}

struct Profile {
    std::vector<double> a, b;
    int first;
};

Profile profile(int n, double h, double offset, double inner, double thickness, double vmax, double refl,
                double dominant, double dt) {  // pml.go:30-62
    Profile p{std::vector<double>(n, 0.0), std::vector<double>(n, 1.0), n};
    if (thickness <= 0) return p;
    const double d0 = -(2 + 1) * vmax * std::log(refl) / (2 * thickness);
    const double amax = M_PI * dominant;
    for (int i = 0; i < n; i++) {
        const double s = (i + offset) * h - inner;
        if (s <= 0) continue;
        const double x = std::min(s / thickness, 1.0);
        const double d = d0 * std::pow(x, 2);
        const double alpha = amax * (1 - x);
        if (d + alpha <= 0) continue;
        const double b = std::exp(-(d + alpha) * dt);
        p.a[i] = d * (b - 1) / (d + alpha);
        p.b[i] = b;
        p.first = std::min(p.first, i);
    }
    return p;
}

}  // namespace

extern "C" {

int gfk_fdtd_grid(const gfk_fdtd_model* m, double* dt, int32_t* nr, int32_t* nz) {
    if (!m || !dt || !nr || !nz) return GFK_EARG;
    Grid g;
    const int st = setup(nullptr, m, &g);
    if (st) return st;
    *dt = g.dt;
    *nr = g.nr;
    *nz = g.nz;
    return GFK_OK;
}

int gfk_fdtd_run(gfk_ctx* ctx, const gfk_fdtd_model* md, const double* force, int32_t nforce, const double* ranges,
                 int32_t nrcv, int32_t steps, double* traces, double* snapped, double* meta) {
    if (!ctx || !md || (!force && nforce > 0) || (!ranges && nrcv > 0) || (!traces && nrcv > 0) || !meta)
        return GFK_EARG;
    Grid g;
    int st = setup(ctx, md, &g);
    if (st) return st;
    if (steps <= 0) return ffail(ctx, GFK_EARG, "fdtd: a shot needs a positive number of steps");
    const int nr = g.nr, nz = g.nz;
    const double h = g.h;
    std::vector<int> cols(std::max(nrcv, 1));
    for (int q = 0; q < nrcv; q++) {  // fdtd.go:135-139, run.go:90-96
        int c = (int)std::lround(ranges[q] / h);
        c = std::max(0, std::min(c, nr - 2));
        const double sn = c * h;
        if (sn >= md->max_range_m) {
            char buf[160];
            snprintf(buf, sizeof buf, "fdtd: receiver at %g m is outside the interior (%g m)", ranges[q],
                     md->max_range_m);
            return ffail(ctx, GFK_EARG, buf);
        }
        cols[q] = c;
        if (snapped) snapped[q] = sn;
    }
    // materials per row (model.go:150-204)
    const gfk_medium& m = md->medium;
    std::vector<double> rho(nz), lamU(nz), muU(nz), rhoZ(nz), muZ(nz);
    for (int j = 0; j < nz; j++) {
        const gfk_layer& l = layer_at(m, j * h);
        const double r = l.density_kgm3, vp = l.vp_mps, vs = l.vs_mps;
        double mp, ms;
        if (g.sls.lossy()) {
            const double cp = g.sls.relaxed_velocity(vp, g.fref), cs = g.sls.relaxed_velocity(vs, g.fref);
            mp = r * cp * cp * (1 + g.sls.delta());
            ms = r * cs * cs * (1 + g.sls.delta());
        } else {
            mp = r * vp * vp;
            ms = r * vs * vs;
        }
        rho[j] = r;
        muU[j] = ms;
        lamU[j] = mp - 2 * ms;
    }
    for (int j = 0; j < nz; j++) {
        const int k = std::min(j + 1, nz - 1);
        rhoZ[j] = 0.5 * (rho[j] + rho[k]);
        muZ[j] = (muU[j] <= 0 || muU[k] <= 0) ? 0.0 : 2 * muU[j] * muU[k] / (muU[j] + muU[k]);
    }
    const double thick = g.pml * h;
    const Profile pRi = profile(nr, h, 0, md->max_range_m, thick, g.vmax, g.refl, g.dominant, g.dt);
    const Profile pRh = profile(nr, h, 0.5, md->max_range_m, thick, g.vmax, g.refl, g.dominant, g.dt);
    const Profile pZi = profile(nz, h, 0, md->depth_m, thick, g.vmax, g.refl, g.dominant, g.dt);
    const Profile pZh = profile(nz, h, 0.5, md->depth_m, thick, g.vmax, g.refl, g.dominant, g.dt);

    cudaSetDevice(ctx->device);
    cudaStream_t s = ctx->stream;
    const size_t n = (size_t)nr * nz;
    std::vector<void*> owned;
    auto dev = [&](size_t bytes) -> void* {
        void* p = nullptr;
        if (cudaMallocAsync(&p, std::max<size_t>(bytes, 8), s) != cudaSuccess) p = nullptr;
        owned.push_back(p);
        return p;
    };
    // the constants go up in one copy, once all of them are known
    std::vector<double> consts;
    std::vector<std::pair<const double**, size_t>> places;
    auto up = [&](const std::vector<double>& v, const double** where) {
        places.push_back({where, consts.size()});
        consts.insert(consts.end(), v.begin(), v.end());
        consts.resize((consts.size() + 31) / 32 * 32, 0.0);
    };
    auto cleanup = [&]() {
        for (void* p : owned)
            if (p) cudaFreeAsync(p, s);
        cudaStreamSynchronize(s);
    };
    gfk::fdtd::Args a{};
    a.nr = nr;
    a.nz = nz;
    a.dr = h;
    a.dz = h;
    a.dt = g.dt;
    a.src_area = M_PI * h * h / 4;
    a.lossy = g.sls.lossy();
    if (a.lossy) {  // fdtd.go:71-77
        const double tau = g.sls.ts, kappa = g.sls.delta() / (1 + g.sls.delta());
        const double den = 1 + g.dt / (2 * tau);
        a.mem_decay = (1 - g.dt / (2 * tau)) / den;
        a.mem_drive = (g.dt * kappa / tau) / den;
    }
    std::vector<double> dtr(nz), dtrz(nz), irh(nr), iri(nr, 0.0);
    for (int j = 0; j < nz; j++) {
        dtr[j] = g.dt / rho[j];
        dtrz[j] = g.dt / rhoZ[j];
    }
    for (int i = 0; i < nr; i++) {
        irh[i] = 1.0 / ((i + 0.5) * h);
        if (i > 0) iri[i] = 1.0 / (i * h);
    }
    a.idr = 1.0 / h;
    a.idz = 1.0 / h;
    up(dtr, &a.dt_rho);
    up(dtrz, &a.dt_rhoZ);
    up(irh, &a.ir_half);
    up(iri, &a.ir_int);
    up(lamU, &a.lamU);
    up(muU, &a.muU);
    up(muZ, &a.muZ);
    up(pRi.a, &a.aRi);
    up(pRi.b, &a.bRi);
    up(pRh.a, &a.aRh);
    up(pRh.b, &a.bRh);
    up(pZi.a, &a.aZi);
    up(pZi.b, &a.bZi);
    up(pZh.a, &a.aZh);
    up(pZh.b, &a.bZh);
    a.fRi = pRi.first;
    a.fRh = pRh.first;
    a.fZi = pZi.first;
    a.fZh = pZh.first;
    // in the order of the kernel's field enumeration
    double** fields[] = {&a.vr, &a.vz, &a.trr, &a.tqq, &a.tzz, &a.trz, &a.rrr, &a.rqq, &a.rzz, &a.rrz, &a.psiTrrR,
                         &a.psiTrzZ, &a.psiTrzR, &a.psiTzzZ, &a.psiVrR, &a.psiVzZ, &a.psiVzR, &a.psiVrZ};
    static_assert(sizeof fields / sizeof fields[0] == gfk::fdtd::kFields, "fields");
    auto has = [&](int f) { return a.lossy || f < gfk::fdtd::kRrr || f > gfk::fdtd::kRrz; };
    const int nfield = gfk::fdtd::kFields - (a.lossy ? 0 : 4);
    // two copies of the fields, where they take at most half of what is free
    // (asked only for large grids: the query takes up to a millisecond) and can be
    // had; else one. GFK_FDTD_COPIES=<1 or 2> replaces the question.
    gfk::fdtd::Tiles tl{};
    size_t mem_free = 0, mem_all = 0;
    const char* asked = getenv("GFK_FDTD_COPIES");
    const bool fits = asked ? atoi(asked) > 1
                            : 2 * n * 8 * nfield <= (size_t(1) << 30) ||
                                  (cudaMemGetInfo(&mem_free, &mem_all) == cudaSuccess && 2 * n * 8 * nfield <= mem_free / 2);
    bool tiled = fits && cudaFuncSetAttribute(a.lossy ? gfk::fdtd::k_tiles<true> : gfk::fdtd::k_tiles<false>,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              gfk::fdtd::kTileSmem) == cudaSuccess;
    std::vector<double> fpad(force, force + std::max(0, std::min(nforce, steps + 1)));
    fpad.resize((size_t)steps + 1, 0.0);
    const size_t copy = (n * 8 + 255) / 256 * 256;
    size_t all = (tiled ? 2 : 1) * nfield * copy;
    unsigned char* slab = static_cast<unsigned char*>(dev(all));
    if (!slab && tiled) {
        cudaGetLastError();
        owned.clear();
        tiled = false;
        all = nfield * copy;
        slab = static_cast<unsigned char*>(dev(all));
    }
    for (int f = 0, at = 0; slab && f < gfk::fdtd::kFields; f++)
        if (has(f)) {
            *fields[f] = reinterpret_cast<double*>(slab + at * copy);
            tl.in[f] = *fields[f];
            if (tiled) tl.out[f] = reinterpret_cast<double*>(slab + (nfield + at) * copy);
            at++;
        }
    if (tiled) {
        up(fpad, &tl.force);
        tl.S = gfk::fdtd::tile_steps(nr, nz);
    }
    double* d_consts = static_cast<double*>(dev(consts.size() * 8));
    int* d_cols = static_cast<int*>(dev(cols.size() * sizeof(int)));
    double* d_traces = static_cast<double*>(dev((size_t)std::max(nrcv, 1) * steps * 8));
    const int nblk = 296;
    double* d_max = static_cast<double*>(dev(nblk * 8));
    for (void* p : owned)
        if (!p) {
            cleanup();
            return ffail(ctx, GFK_ENOMEM, "fdtd: device allocation failed");
        }
    for (auto& [where, at] : places) *where = d_consts + at;
    cudaMemsetAsync(slab, 0, all, s);
    cudaMemsetAsync(d_traces, 0, (size_t)std::max(nrcv, 1) * steps * 8, s);
    cudaMemcpyAsync(d_consts, consts.data(), consts.size() * 8, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(d_cols, cols.data(), cols.size() * sizeof(int), cudaMemcpyHostToDevice, s);
    a.cols = d_cols;
    a.nrcv = nrcv;
    a.steps = steps;
    a.traces = d_traces;

    const dim3 blk(32, 8), grd((nr + 31) / 32, (nz + 7) / 8);
    double peak = 0;
    std::vector<double> mx(nblk);
    for (int step = 0; step < steps;) {  // fdtd.go:142-147, run.go:98-121
        // up to the next step whose speeds are checked (every 256th), at most S
        int take = 1;
        const double *vz = a.vz, *vr = a.vr;
        if (tiled) {
            take = std::min({tl.S, steps - step, step == 0 ? 1 : 256 - (step - 1) % 256});
            tl.n = take;
            tl.step0 = step;
            const int tw = gfk::fdtd::kTileW - 2 * tl.S;
            const dim3 tiles((nr + tw - 1) / tw, (nz + tw - 1) / tw);
            if (a.lossy)
                gfk::fdtd::k_tiles<true><<<tiles, gfk::fdtd::kTileThreads, gfk::fdtd::kTileSmem, s>>>(a, tl);
            else
                gfk::fdtd::k_tiles<false><<<tiles, gfk::fdtd::kTileThreads, gfk::fdtd::kTileSmem, s>>>(a, tl);
            ctx->launches++;
            for (int f = 0; f < gfk::fdtd::kFields; f++) {
                double* o = tl.out[f];
                tl.out[f] = const_cast<double*>(tl.in[f]);
                tl.in[f] = o;
            }
            vz = tl.in[gfk::fdtd::kVz];
            vr = tl.in[gfk::fdtd::kVr];
        } else {
            gfk::fdtd::k_velocities<<<grd, blk, 0, s>>>(a, -fpad[step] / a.src_area);
            gfk::fdtd::k_stresses<<<grd, blk, 0, s>>>(a, (fpad[step + 1] - fpad[step]) / g.dt, step);
            ctx->launches += 2;
        }
        step += take;
        const int done = step - 1;
        if (done % 256 == 0) {
            gfk::fdtd::k_maxspeed<<<nblk, 256, 0, s>>>(vz, vr, (long long)n, d_max);
            ctx->launches++;
            if (cudaMemcpyAsync(mx.data(), d_max, nblk * 8, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
                cudaStreamSynchronize(s) != cudaSuccess) {
                cleanup();
                return ffail(ctx, GFK_ECUDA, "fdtd: step kernels failed");
            }
            double p = 0;
            bool bad = false;
            for (double x : mx) {
                bad |= std::isnan(x) || std::isinf(x);
                p = std::max(p, x);
            }
            peak = std::max(peak, p);
            if (bad) {
                cleanup();
                char buf[96];
                snprintf(buf, sizeof buf, "fdtd: diverged at step %d of %d", done, steps);
                return ffail(ctx, GFK_ENONFINITE, buf);
            }
        }
    }
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && nrcv > 0)
        e = cudaMemcpyAsync(traces, d_traces, (size_t)nrcv * steps * 8, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cleanup();
    if (e != cudaSuccess) return ffail(ctx, GFK_ECUDA, std::string("fdtd: ") + cudaGetErrorString(e));
    meta[0] = g.dt;
    meta[1] = 0.5 * g.dt;
    meta[2] = peak;
    meta[3] = nr;
    meta[4] = nz;
    return GFK_OK;
}

}  // extern "C"
