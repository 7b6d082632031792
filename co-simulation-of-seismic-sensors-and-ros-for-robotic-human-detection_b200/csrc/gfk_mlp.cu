// gfk_mlp.cu — the surrogate network's kernels.
//
// The network maps (soil scalars, range, frequency) to the vertical Green's
// spectrum as t0 = log|G| and t1 = -phi/(w r), phi the unwrapped phase: an
// input layer 128 -> 512, four hidden layers 512 -> 512 (all SiLU) and an
// FP32 output layer 512 -> 2. Weights and activations are BF16, accumulation
// FP32 in TMEM, master weights and Adam moments FP32.
//
// Every 512-wide layer runs on one BF16 tcgen05 GEMM kernel with the layer's
// elementwise work fused into its epilogue:
//   forward   Z = X W^T + b, H = silu(Z)       (A = X [B][K], B = W [N][K])
//   backward  dZ' = (dZ W) silu'(Z')          (A = dZ [B][N], B = W^T [K][N])
//   weights   dW = dZ^T X, split over the batch (A = dZ^T, B = X^T)
// so every operand is K-major and is fed by plain TMA tiles: the epilogues
// write the transposed copies (X^T, dZ^T) the weight gradients read, and Adam
// writes W and W^T. The kernel shape is the wavenumber-sum kernel's: one
// 128 x 128 tile per CTA, warp 0 TMA, warp 1 TMEM + MMA issue, warps 2-5
// epilogue, SWIZZLE_64B tiles (32 BF16 = 64 bytes per row), 3-stage ring,
// bounded waits. Inference on many rows has a kernel of its own,
// k_layer_infer. No load is multicast.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <math_constants.h>

#include <algorithm>
#include <atomic>
#include <type_traits>
#include <utility>

#include "gfk_kernels.cuh"
#include "gfk_mlp.cuh"
#include "gfk_tc.cuh"

namespace gfk {
namespace mlp {

using namespace gfk::tc;

constexpr int BM = 128, BN = 128;
constexpr int BKE = 32;                        // BF16 elements per 64-byte swizzled row (one TMA box)
constexpr int BOX = 2;                         // boxes per operand per stage
constexpr int BK = BKE * BOX;                  // 64 elements of K per stage
constexpr int TILE = BM * 64;                  // bytes per box: 128 rows x 64 bytes
constexpr int STAGE_BYTES = 2 * BOX * TILE;    // 32768
constexpr int STAGES = 3;
constexpr int THREADS = 192;
constexpr int TMEM_COLS = BN;                  // 128 FP32 accumulator columns
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256 + BN * 4;
constexpr int kTileLd = BN + 8;  // BF16 row pitch of the epilogue's staging tiles (272 bytes)
static_assert(2 * BM * kTileLd * 2 <= STAGES * STAGE_BYTES, "staging tiles alias the pipeline stages");

// Instruction descriptor: BF16 x BF16 -> F32, both K-major.
__host__ __device__ inline uint32_t idesc_bf16(int m, int n) {
    cute::UMMA::InstrDescriptor id;
    id.desc_ = 0;
    id.c_format_ = 1;  // F32
    id.a_format_ = 1;  // BF16
    id.b_format_ = 1;
    id.a_major_ = 0;   // K-major
    id.b_major_ = 0;
    id.n_dim_ = n >> 3;
    id.m_dim_ = m >> 4;
    return id.desc_;
}

// Programmatic dependent launch. The network's kernels are launched so that
// the next one may be scheduled while the previous one finishes: each calls
// dep_wait() before its first global-memory access (it returns once the
// previous kernel in the stream has completed and its writes are visible; a
// no-op for an ordinary launch) and dep_release() to let its successor start
// its own set-up early.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_release() { asm volatile("griddepcontrol.launch_dependents;" :::); }

template <typename... P, typename... A>
void launch_dep(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

// Hardware exponential and approximate reciprocal (no IEEE division): the
// results are rounded to BF16 (8-bit mantissa) right after.
__device__ __forceinline__ float sigmoid_(float z) { return __fdividef(1.0f, 1.0f + __expf(-z)); }

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float2 t = __bfloat1622float2(h[i]);
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
    }
}

template <int MODE>
__global__ void __launch_bounds__(THREADS, 2)
    k_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, GemmArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
    uint64_t* empty = full + STAGES;
    uint64_t* accf = empty + STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accf + 1);
    int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
    float* bias_s = reinterpret_cast<float*>(smem + STAGES * STAGE_BYTES + 256);  // [BN]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int kbase = blockIdx.z * a.K;
    const int nkb = a.K / BK;

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(accf, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    dep_wait();  // the set-up above overlaps the previous kernel's tail
    dep_release();

    if (warp == 0) {
        if (lane == 0) {
            int issued = 0;
            for (int kb = 0; kb < nkb; kb++) {
                const int st = kb % STAGES;
                const uint32_t ph = (kb / STAGES) & 1;
                if (!mbar_wait(&empty[st], ph ^ 1)) {
                    *abort_flag = 1;
                    break;
                }
                if (*(volatile int*)abort_flag) break;
                mbar_expect_tx(&full[st], STAGE_BYTES);
                uint8_t* base = smem + st * STAGE_BYTES;
                const int kx = kbase + kb * BK;
#pragma unroll
                for (int b = 0; b < BOX; b++) tma_load_2d(base + b * TILE, &tmA, &full[st], kx + b * BKE, m0);
#pragma unroll
                for (int b = 0; b < BOX; b++)
                    tma_load_2d(base + (BOX + b) * TILE, &tmB, &full[st], kx + b * BKE, n0);
                issued = kb + 1;
            }
            for (int kb = issued - 1; kb >= 0 && kb >= issued - STAGES; kb--)
                if (!mbar_wait(&full[kb % STAGES], (kb / STAGES) & 1)) *abort_flag = 1;
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16(BM, BN);
            uint32_t acc = 0;
            for (int kb = 0; kb < nkb; kb++) {
                const int st = kb % STAGES;
                if (!mbar_wait(&full[st], (kb / STAGES) & 1)) {
                    *abort_flag = 1;
                    break;
                }
                if (*(volatile int*)abort_flag) break;
                tc_fence_after();
                const uint32_t base = smem_u32(smem + st * STAGE_BYTES);
#pragma unroll
                for (int b = 0; b < BOX; b++) {
#pragma unroll
                    for (int kk = 0; kk < BKE / 16; kk++) {  // K = 16 per instruction = 32 bytes
                        const uint64_t da = sdesc_k_sw64(base + b * TILE + kk * 32);
                        const uint64_t db = sdesc_k_sw64(base + (BOX + b) * TILE + kk * 32);
                        tc_mma_f16(tmem, da, db, idesc, acc);
                        acc = 1;
                    }
                }
                tc_commit(&empty[st]);
            }
            tc_commit(accf);
        }
    } else {
        // epilogue, phase 1 (warps 2-5): TMEM -> registers -> elementwise work;
        // BF16 results go to a shared-memory tile (the pipeline stages are free
        // once every MMA has completed), FP32 gradient partials straight out
        // the tile's bias columns, read once while the MMAs run
        if (MODE == kFwdTrain || MODE == kFwdInfer) {
            bias_s[threadIdx.x - 64] = a.bias[n0 + threadIdx.x - 64];
            asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        const int q = warp & 3;
        const int rl = q * 32 + lane;
        const int row = m0 + rl;
        // backward-data: this row's pre-activations, one 32-column chunk ahead
        // (the first chunk is in flight while the MMAs run)
        uint4 zcur[4], znext[4];
        if (MODE == kBwdData) {
            const uint4* zs = reinterpret_cast<const uint4*>(a.zin + (size_t)row * a.N + n0);
#pragma unroll
            for (int c = 0; c < 4; c++) zcur[c] = zs[c];
        }
        const bool ok = mbar_wait(accf, 0);
        if (!ok) *(volatile int*)abort_flag = 1;  // the tile stays unwritten: no stores below
        tc_fence_after();
        const bool row_ok = ok && !*(volatile int*)abort_flag;
        bf16* tileO = reinterpret_cast<bf16*>(smem);
        bf16* tileZ = tileO + BM * kTileLd;
#pragma unroll 1
        for (int j = 0; j < BN / 32; j++) {
            uint32_t v[32];
            tmem_ld32(tmem + (static_cast<uint32_t>(q * 32) << 16) + j * 32, v);
            if (MODE == kBwdData && j + 1 < BN / 32) {
                const uint4* zs = reinterpret_cast<const uint4*>(a.zin + (size_t)row * a.N + n0 + (j + 1) * 32);
#pragma unroll
                for (int c = 0; c < 4; c++) znext[c] = zs[c];
            }
            tmem_wait_ld();
            if (!row_ok) continue;
            const int nb = n0 + j * 32;
            if (MODE == kWgrad) {
                float4* dst = reinterpret_cast<float4*>(a.part + ((size_t)blockIdx.z * a.M + row) * a.N + nb);
#pragma unroll
                for (int c = 0; c < 8; c++)
                    dst[c] = make_float4(__uint_as_float(v[4 * c]), __uint_as_float(v[4 * c + 1]),
                                         __uint_as_float(v[4 * c + 2]), __uint_as_float(v[4 * c + 3]));
                continue;
            }
            float y[32];
            if (MODE == kFwdTrain || MODE == kFwdInfer) {
                float zv[32];
#pragma unroll
                for (int c = 0; c < 32; c++) {
                    zv[c] = __uint_as_float(v[c]) + bias_s[j * 32 + c];
                    y[c] = zv[c] * sigmoid_(zv[c]);
                }
                if (MODE == kFwdTrain) {
                    uint4* zd = reinterpret_cast<uint4*>(tileZ + rl * kTileLd + j * 32);
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        zd[c] = make_uint4(pack2(zv[8 * c], zv[8 * c + 1]), pack2(zv[8 * c + 2], zv[8 * c + 3]),
                                           pack2(zv[8 * c + 4], zv[8 * c + 5]), pack2(zv[8 * c + 6], zv[8 * c + 7]));
                }
            } else {  // kBwdData
                float zv[32];
#pragma unroll
                for (int c = 0; c < 4; c++) unpack8(zcur[c], zv + 8 * c);
#pragma unroll
                for (int c = 0; c < 32; c++) {
                    const float sg = sigmoid_(zv[c]);
                    y[c] = __uint_as_float(v[c]) * (sg * (1.0f + zv[c] * (1.0f - sg)));
                }
#pragma unroll
                for (int c = 0; c < 4; c++) zcur[c] = znext[c];
            }
            uint4* od = reinterpret_cast<uint4*>(tileO + rl * kTileLd + j * 32);
#pragma unroll
            for (int c = 0; c < 4; c++)
                od[c] = make_uint4(pack2(y[8 * c], y[8 * c + 1]), pack2(y[8 * c + 2], y[8 * c + 3]),
                                   pack2(y[8 * c + 4], y[8 * c + 5]), pack2(y[8 * c + 6], y[8 * c + 7]));
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // phase 2 (all warps): coalesced stores of the tile, its transpose and Z
    if (MODE != kWgrad && !*(volatile int*)abort_flag) {
        const bf16* tileO = reinterpret_cast<const bf16*>(smem);
        const bf16* tileZ = tileO + BM * kTileLd;
        for (int c = threadIdx.x; c < BM * (BN / 8); c += THREADS) {
            const int r = c / (BN / 8), c8 = (c % (BN / 8)) * 8;
            const size_t g = (size_t)(m0 + r) * a.N + n0 + c8;
            *reinterpret_cast<uint4*>(a.out + g) = *reinterpret_cast<const uint4*>(tileO + r * kTileLd + c8);
            if (MODE == kFwdTrain)
                *reinterpret_cast<uint4*>(a.zout + g) = *reinterpret_cast<const uint4*>(tileZ + r * kTileLd + c8);
        }
        if (MODE != kFwdInfer && a.outT) {
            // 32 bytes (16 rows) of one transposed row per thread; lanes run
            // over columns, so the shared-memory column reads do not conflict
            for (int c = threadIdx.x; c < BN * (BM / 16); c += THREADS) {
                const int n = c % BN, r16 = (c / BN) * 16;
                uint32_t w[8];
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    __nv_bfloat162 v2;
                    v2.x = tileO[(r16 + 2 * e) * kTileLd + n];
                    v2.y = tileO[(r16 + 2 * e + 1) * kTileLd + n];
                    w[e] = *reinterpret_cast<uint32_t*>(&v2);
                }
                uint4* d = reinterpret_cast<uint4*>(a.outT + (size_t)(n0 + n) * a.M + m0 + r16);
                d[0] = make_uint4(w[0], w[1], w[2], w[3]);
                d[1] = make_uint4(w[4], w[5], w[6], w[7]);
            }
        }
    }
    if (threadIdx.x == 0 && *(volatile int*)abort_flag && a.status) atomicOr(a.status, kStTimeout);
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

// ------------------------------------------------- inference layers --
//
// h = silu(x W^T + b) for many rows. A pair of CTAs on a pair of SMs keeps one
// of the layer's 256-column slabs of weights in shared memory, half in each CTA
// and the whole K extent (at most 512: 128 KB), and takes blocks of 256 rows,
// which stream through a ring, again half in each: every SM computes 128 x 256
// from 128 KB loaded. The leader of the pair issues the MMAs and its barriers
// count both CTAs' loads. The accumulator is double-buffered in all 512 columns of
// TMEM, so a tile's epilogue runs while the next one multiplies. Warp 0 loads,
// warp 1 issues, warps 2-17 are the epilogue in two groups of 128 columns; a
// group's 128 x 64 box of shared memory leaves by TMA. The order of K is
// k_gemm's, and so are the results' bits.
//
// For 2^20 rows x 512 x 512 (2.1 GB at least, 0.32 ms of HBM, 0.35 ms of BF16):
//   one tile per CTA (k_gemm), 32-wide K boxes          0.99 ms
//   persistent, rows resident, weights streaming        0.93 ms  all SMs ask L2 for the same lines at a time
//   128-column weights resident in each CTA alone       0.81 ms  256 KB loaded for 128 x 256, L2-bound
//   pairs, 8 epilogue warps / 16                        0.60 / 0.58 ms
// With K = 128 the loads are a quarter and it takes 0.43 ms: what is left is
// the epilogue's chain (TMEM, exponentials, barriers, box) on 4 warps a scheduler.
//
// A producer stops only when a wait of its own has run out, a second after its
// last load: nothing is in flight into a CTA that leaves.

constexpr int kInfStages = 4;                       // row ring: 64 of K a stage
constexpr int kInfKb = 8;                           // K blocks of 64 at most
constexpr int kInfBlock = BM * 128;                 // 16 KB: 128 rows x 64 of K
constexpr int kInfGroups = 2;                       // of eight epilogue warps, 128 columns each
constexpr int kInfThreads = 64 + 256 * kInfGroups;
constexpr int kInfBox = BM * 128;                   // output box: 128 rows x 64 columns
constexpr int kInfN = 2 * BN;                       // columns of a pair's slab
constexpr int kInfSmem = (kInfKb + kInfStages) * kInfBlock + kInfGroups * kInfBox + kInfN * 4 + 256 + 1024;
static_assert(kInfSmem <= 227 * 1024, "shared memory per CTA");

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kInfThreads, 1)
    k_layer_infer(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                  const __grid_constant__ CUtensorMap tmO, GemmArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* ring = smem + kInfKb * kInfBlock;
    uint8_t* outs = ring + kInfStages * kInfBlock;  // one box per group
    float* bias_s = reinterpret_cast<float*>(outs + kInfGroups * kInfBox);
    uint64_t* w_full = reinterpret_cast<uint64_t*>(bias_s + kInfN);
    uint64_t* a_full = w_full + kInfKb;
    uint64_t* a_empty = a_full + kInfStages;
    uint64_t* acc_full = a_empty + kInfStages;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* drained = acc_empty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* stop = abort_flag + 1;  // [kInfGroups] each epilogue group's common answer to it

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x & 1;  // in the pair
    const int nkb = a.K / BK, nslab = a.N / kInfN, nblock = (a.M + 2 * BM - 1) / (2 * BM);
    const int n0 = ((blockIdx.x >> 1) % nslab) * kInfN;                             // the pair's columns
    const int mb0 = (blockIdx.x >> 1) / nslab, mstep = (gridDim.x >> 1) / nslab;    // and row blocks
    if (threadIdx.x == 0) {
        for (int i = 0; i < kInfKb; i++) mbar_init(&w_full[i], 1);
        for (int i = 0; i < kInfStages; i++) {
            mbar_init(&a_full[i], 1);
            mbar_init(&a_empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 16 * kInfGroups);  // one arrival per epilogue warp of the pair
        }
        mbar_init(drained, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(2 * kInfN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    dep_wait();  // the set-up above overlaps the previous kernel's tail
    dep_release();
    for (int n = threadIdx.x; n < kInfN; n += kInfThreads) bias_s[n] = a.bias[n0 + n];
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the leader's barriers are there before the follower's loads count on them
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            const int row0 = rank * BM;
            int st = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int mb = mb0; mb < nblock && ok; mb += mstep)
                for (int kb = 0; kb < nkb; kb++) {
                    if (!mbar_wait(&a_empty[st], ph ^ 1)) {
                        ok = false;
                        break;
                    }
                    if (mb == mb0) {  // the weights come with the first block: its MMAs start on the first K block
                        if (rank == 0) mbar_expect_tx(&w_full[kb], 2 * kInfBlock);
                        tma_load_2d_pair(smem + kb * kInfBlock, &tmB, leader_addr(&w_full[kb]), kb * BK, n0 + row0);
                    }
                    if (rank == 0) mbar_expect_tx(&a_full[st], 2 * kInfBlock);
                    tma_load_2d_pair(ring + st * kInfBlock, &tmA, leader_addr(&a_full[st]), kb * BK, mb * 2 * BM + row0);
                    if (++st == kInfStages) {
                        st = 0;
                        ph ^= 1;
                    }
                }
            if (!ok) *abort_flag = 1;
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            const uint32_t idesc = idesc_bf16(2 * BM, kInfN);
            int st = 0, tile = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int mb = mb0; mb < nblock && ok; mb += mstep, tile++) {
                const int buf = tile & 1;
                if (!leader_wait(&acc_empty[buf], ((tile >> 1) & 1) ^ 1) || *abort_flag) {
                    ok = false;
                    break;
                }
                for (int kb = 0; kb < nkb; kb++) {
                    if ((mb == mb0 && !leader_wait(&w_full[kb], 0)) || !leader_wait(&a_full[st], ph) || *abort_flag) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t ra = smem_u32(ring + st * kInfBlock), rb = smem_u32(smem + kb * kInfBlock);
#pragma unroll
                    for (int kk = 0; kk < BK / 16; kk++)  // K = 16 per instruction = 32 bytes of the row
                        tc_mma_f16_pair(tmem + buf * kInfN, sdesc_k_sw128(ra + kk * 32), sdesc_k_sw128(rb + kk * 32),
                                        idesc, (kb | kk) ? 1u : 0u);
                    tc_commit_pair(&a_empty[st]);
                    if (++st == kInfStages) {
                        st = 0;
                        ph ^= 1;
                    }
                }
                if (ok) tc_commit_pair(&acc_full[buf]);
            }
            if (!ok) *abort_flag = 1;
            tc_commit_pair(drained);  // every MMA issued above, before TMEM is freed
        }
    } else {
        const int q = warp & 3, group = (warp - 2) >> 3, sub = ((warp - 2) >> 2) & 1;
        const bool lead = ((warp - 2) & 7) == 0 && lane == 0;  // issues its group's stores
        uint8_t* const box = outs + group * kInfBox;
        const int rl = q * 32 + lane;
        auto group_sync = [&] { asm volatile("bar.sync %0, 256;" ::"r"(1 + group) : "memory"); };
        int tile = 0;
        for (int mb = mb0; mb < nblock; mb += mstep, tile++) {
            const int buf = tile & 1;
            if (!mbar_wait(&acc_full[buf], (tile >> 1) & 1)) *abort_flag = 1;
            __syncwarp();
            tc_fence_after();
            const uint32_t at = tmem + (static_cast<uint32_t>(q * 32) << 16) + buf * kInfN + group * BN + sub * 32;
            const int row = (mb * 2 + rank) * BM;
            bool run = true;
#pragma unroll
            for (int c = 0; c < 2; c++) {  // 64 columns at a time, 32 in each warp
                uint32_t v[32];
                tmem_ld32(at + c * 64, v);
                tmem_wait_ld();
                if (c == 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) leader_arrive(leader_addr(&acc_empty[buf]));
                }
                uint4 y4[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    float y[8];
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        const float z = __uint_as_float(v[8 * j + e]) + bias_s[group * BN + c * 64 + sub * 32 + 8 * j + e];
                        y[e] = z * sigmoid_(z);
                    }
                    y4[j] = make_uint4(pack2(y[0], y[1]), pack2(y[2], y[3]), pack2(y[4], y[5]), pack2(y[6], y[7]));
                }
                if (lead) {
                    tma_store_wait_read();  // the box is free again
                    stop[group] = *abort_flag;
                }
                group_sync();
                // once a wait has run out the group stops together: the next write of
                // stop[group] comes after the barrier below, when all have read it
                if (stop[group]) {
                    run = false;
                    break;
                }
#pragma unroll
                for (int j = 0; j < 4; j++)
                    *reinterpret_cast<uint4*>(box + rl * 128 + (((sub * 4 + j) ^ (rl & 7)) << 4)) = y4[j];
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                group_sync();
                if (lead && row < a.M) {  // an odd last block has rows in the leader only
                    tma_store_2d(&tmO, box, n0 + group * BN + c * 64, row);
                    tma_store_commit();
                }
            }
            if (!run) break;
        }
        if (lead) tma_store_wait();
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 32 && !mbar_wait(drained, 0)) *abort_flag = 1;
    __syncthreads();
    cluster_sync();  // neither CTA leaves while the other may still signal it or read its operands
    tc_fence_after();
    if (threadIdx.x == 0 && *abort_flag && a.status) atomicOr(a.status, kStTimeout);
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kInfN) : "memory");
}

// ----------------------------------------------------------------- batch --

// splitmix64 finaliser (Steele, Lea, Flood 2014) as a counter-based generator.
__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
    x += 0x9e3779b97f4a7c15ULL;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
    return x ^ (x >> 31);
}

__device__ __forceinline__ int pick(unsigned long long h32, int n) {
    return static_cast<int>(((h32 & 0xffffffffULL) * static_cast<unsigned long long>(n)) >> 32);
}

struct PointScalars {
    float ur, uf, lr, lf, f;
};

__device__ __forceinline__ void range_scalars(PointScalars& p, double r, const FeatureDomain& d) {
    p.ur = static_cast<float>((r - d.r_lo) / (d.r_hi - d.r_lo));
    p.lr = static_cast<float>(2.0 * log(r / d.r_lo) / log(d.r_hi / d.r_lo) - 1.0);
}

__device__ __forceinline__ void freq_scalars(PointScalars& p, double f, const FeatureDomain& d) {
    p.uf = static_cast<float>((f - d.f_lo) / (d.f_hi - d.f_lo));
    p.lf = static_cast<float>(2.0 * log(f / d.f_lo) / log(d.f_hi / d.f_lo) - 1.0);
    p.f = static_cast<float>(f);
}

// sf: one soil table row (scalars at [0, 11), travel times at [16, 22)).
__device__ __forceinline__ float feature(int j, const float* sf, const PointScalars& p, const float* four) {
    if (j < kMaxSoil) return sf[j];
    if (j < kScalars) {
        switch (j) {
            case 11: return 2.0f * p.ur - 1.0f;
            case 12: return 2.0f * p.uf - 1.0f;
            case 13: return p.lr;
            case 14: return p.lf;
            default: return 0.0f;
        }
    }
    if (j < kLogTimeFeat) {
        const int q = (j - kTimeFeat) >> 1;
        float sn, cs;
        sincospif(2.0f * (p.f * sf[kScalars + q]), &sn, &cs);
        return (j & 1) ? cs : sn;
    }
    if (j < kFourierFeat) {
        const float x = p.f * sf[kScalars + (j - kLogTimeFeat)];
        return x > 0.0f ? fminf(fmaxf((logf(x) + 2.0f) / 3.0f, -2.0f), 2.0f) : -2.0f;
    }
    const int q = (j - kFourierFeat) >> 1;
    float sn, cs;
    sincospif(2.0f * (four[2 * q] * p.ur + four[2 * q + 1] * p.uf), &sn, &cs);
    return (j & 1) ? cs : sn;
}

// Features j and j + 1, j even: a sine and cosine share their argument and one call.
__device__ __forceinline__ void feature_pair(int j, const float* sf, const PointScalars& p, const float* four, float& v0,
                                             float& v1) {
    if ((j >= kTimeFeat && j < kLogTimeFeat) || j >= kFourierFeat) {
        const int f = (j - kFourierFeat) >> 1;
        const float arg = j < kLogTimeFeat ? 2.0f * (p.f * sf[kScalars + ((j - kTimeFeat) >> 1)])
                                           : 2.0f * (four[2 * f] * p.ur + four[2 * f + 1] * p.uf);
        sincospif(arg, &v0, &v1);
    } else {
        v0 = feature(j, sf, p, four);
        v1 = feature(j + 1, sf, p, four);
    }
}
static_assert(kTimeFeat % 2 == 0 && kLogTimeFeat % 2 == 0 && kFourierFeat % 2 == 0, "features come in pairs");

// The step's counter and rates. The batch draws with the counter's next value, so
// this one-thread kernel (two FP64 powers) runs beside the last weight
// gradients, before the loss history and Adam, which read what it writes.
__global__ void k_step_begin(TrainScalars* ts) {
    dep_wait();
    dep_release();
    const long long t = ++ts->step;
    float lr;
    if (t <= ts->warmup) {
        lr = ts->lr_max * static_cast<float>(t) / static_cast<float>(ts->warmup > 0 ? ts->warmup : 1);
    } else {
        const double span = ts->total > ts->warmup ? static_cast<double>(ts->total - ts->warmup) : 1.0;
        const double p = fmin(1.0, static_cast<double>(t - ts->warmup) / span);
        lr = static_cast<float>(ts->lr_min + 0.5 * (ts->lr_max - ts->lr_min) * (1.0 + cospi(p)));
    }
    ts->lr = lr;
    ts->bc1 = static_cast<float>(1.0 - pow(static_cast<double>(ts->beta1), static_cast<double>(t)));
    ts->bc2 = static_cast<float>(1.0 - pow(static_cast<double>(ts->beta2), static_cast<double>(t)));
}

// kBatchRows samples per block. A lane per sample of one warp draws the cell and
// gathers its targets while the lanes of another form the samples' scalars (FP64
// logarithms); then a thread fills a pair of features of four samples. Small
// blocks keep many of them resident, so the dependent gathers (soil, cell,
// label) of different blocks overlap. (One warp doing both and a thread per
// feature walking 16 samples: 16.1 us for 8192 samples; 9.0 us here, cold.)
constexpr int kBatchRows = 16;
constexpr int kBatchThreads = 256;
__global__ void __launch_bounds__(kBatchThreads) k_batch(BatchArgs a) {
    dep_wait();
    dep_release();
    __shared__ uint32_t tile[kBatchRows][kIn / 2 + 1];  // pairs of BF16
    __shared__ PointScalars ps[kBatchRows];
    __shared__ int soil_of[kBatchRows];
    const long long t = a.ts->step + 1;
    const int b0 = blockIdx.x * kBatchRows;
    const int tid = threadIdx.x, sample = tid & 31;
    unsigned long long h = 0;
    int ir = 0, jf = 0;
    if (tid < 64 && sample < kBatchRows) {
        h = mix64(a.seed ^ mix64(static_cast<unsigned long long>(t) * a.B + b0 + sample));
        const unsigned long long h2 = mix64(h);
        ir = a.ir0 + pick(h2, a.nir);
        jf = pick(h2 >> 32, a.nf);
    }
    if (tid >= 32 && tid < 32 + kBatchRows) {
        range_scalars(ps[sample], a.ranges[ir], a.dom);
        freq_scalars(ps[sample], a.freqs[jf], a.dom);
    }
    if (tid < kBatchRows) {
        const int b = b0 + sample;
        const int soil = a.train[pick(h, a.ntrain)];
        soil_of[sample] = soil;
        const float* L = a.labels + (((size_t)soil * a.nr + ir) * a.nf + jf) * 2;
        const bool ph = !isnan(L[1]);
        a.Y[2 * b] = (L[0] - a.y_mean0) / a.y_std0;
        a.Y[2 * b + 1] = (L[1] - a.y_mean1) / a.y_std1;  // NaN stays NaN
        float c0 = 1.0f, c1 = ph ? a.phase_weight : 0.0f;
        if (a.loss_mode == 2) {
            const float w = fmaxf(__expf(L[0] - a.lmax[(size_t)soil * a.nr + ir]), a.weight_floor);
            c0 = w;
            c1 = ph ? a.phase_weight * w : 0.0f;
        } else if (a.loss_mode == 1) {
            const float w = fmaxf(__expf(2.0f * (L[0] - a.lmax[(size_t)soil * a.nr + ir])), a.weight_floor);
            const float wr = static_cast<float>(2.0 * 3.14159265358979323846 * a.freqs[jf] * a.ranges[ir]) *
                             (a.y_std1 / a.y_std0);
            c0 = w;
            c1 = ph ? a.phase_weight * w * fminf(wr * wr, a.phase_cap) : 0.0f;
        }
        a.C[2 * b] = c0;
        a.C[2 * b + 1] = c1;
    }
    __syncthreads();
    const int pair = tid & 63;
#pragma unroll
    for (int i = tid >> 6; i < kBatchRows; i += kBatchThreads / 64) {
        float v0, v1;
        feature_pair(2 * pair, a.soilfeat + (size_t)soil_of[i] * kSoilStride, ps[i], a.fourier, v0, v1);
        const uint32_t v = pack2(v0, v1);
        tile[i][pair] = v;
        *reinterpret_cast<uint32_t*>(a.X + (size_t)(b0 + i) * kIn + 2 * pair) = v;
    }
    __syncthreads();
    // X^T: a thread writes 8 consecutive samples of its feature
    const int j = tid & (kIn - 1), half = tid / kIn;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t lo = tile[8 * half + 2 * i][j >> 1], hi = tile[8 * half + 2 * i + 1][j >> 1];
        w[i] = __byte_perm(lo, hi, (j & 1) ? 0x7632 : 0x5410);
    }
    *reinterpret_cast<uint4*>(a.XT + (size_t)j * a.B + b0 + 8 * half) = make_uint4(w[0], w[1], w[2], w[3]);
}
static_assert(kBatchRows == 16 && kBatchThreads == 2 * kIn, "two groups of 8 samples");

// ------------------------------------------------------------------ head --

// 8 warps x 4 rows; lane owns columns u*256 + lane*8 + e (u = 0, 1; e < 8). A
// warp asks for its four rows of H and Z at once and carries the four dot
// products together, then walks the columns with the rows inside, and the
// warps' dW6 parts meet in shared memory in one step, added in warp order. (A row
// after the other, a load and a shuffle chain each, and one barrier per warp for
// the parts: 27.7 us for 8192 rows, 34 MB; 13.1 us here, cold.)
struct HeadShared {
    bf16 tile[kHeadRows][kWidth + 8];
    float part[8][2 * kWidth];
};
__global__ void __launch_bounds__(256, 2) k_head_train(const bf16* __restrict__ H, const bf16* __restrict__ Z,
                                                       const float* __restrict__ W6, const float* __restrict__ b6,
                                                       const float* __restrict__ Y, const float* __restrict__ Cw, int B,
                                                       bf16* __restrict__ dZ, bf16* __restrict__ dZT,
                                                       float* __restrict__ gpart, float* __restrict__ lpart) {
    dep_wait();
    dep_release();
    extern __shared__ __align__(16) uint8_t head_raw[];
    HeadShared& sm = *reinterpret_cast<HeadShared*>(head_raw);
    __shared__ float lred[8][6];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r0 = blockIdx.x * kHeadRows, row = r0 + warp * 4;
    uint4 hq[4][2], zq[4][2];
    float2 yt[4], ct[4];
#pragma unroll
    for (int t = 0; t < 4; t++)
#pragma unroll
        for (int u = 0; u < 2; u++) {
            hq[t][u] = *reinterpret_cast<const uint4*>(H + (size_t)(row + t) * kWidth + u * 256 + lane * 8);
            zq[t][u] = *reinterpret_cast<const uint4*>(Z + (size_t)(row + t) * kWidth + u * 256 + lane * 8);
        }
#pragma unroll
    for (int t = 0; t < 4; t++) {
        yt[t] = *reinterpret_cast<const float2*>(Y + 2 * (row + t));
        ct[t] = *reinterpret_cast<const float2*>(Cw + 2 * (row + t));
    }
    auto load8 = [](const float* src, float (&w)[8]) {
        const float4 x = *reinterpret_cast<const float4*>(src), y = *reinterpret_cast<const float4*>(src + 4);
        w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w, w[4] = y.x, w[5] = y.y, w[6] = y.z, w[7] = y.w;
    };
    float y0[4] = {}, y1[4] = {};
#pragma unroll
    for (int u = 0; u < 2; u++) {
        float w0[8], w1[8];
        load8(W6 + u * 256 + lane * 8, w0);
        load8(W6 + kWidth + u * 256 + lane * 8, w1);
#pragma unroll
        for (int t = 0; t < 4; t++) {
            float h[8];
            unpack8(hq[t][u], h);
#pragma unroll
            for (int e = 0; e < 8; e++) {
                y0[t] = fmaf(h[e], w0[e], y0[t]);
                y1[t] = fmaf(h[e], w1[e], y1[t]);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int t = 0; t < 4; t++) {
            y0[t] += __shfl_xor_sync(0xffffffffu, y0[t], o);
            y1[t] += __shfl_xor_sync(0xffffffffu, y1[t], o);
        }
    float l0 = 0.0f, l1 = 0.0f, sc0 = 0.0f, sc1 = 0.0f, ds0 = 0.0f, ds1 = 0.0f;
    float d0[4], d1[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
        const float c0 = ct[t].x, c1 = ct[t].y;
        const bool ph = !isnan(yt[t].y) && c1 > 0.0f;
        const float e0 = (y0[t] + b6[0]) - yt[t].x, e1 = ph ? (y1[t] + b6[1]) - yt[t].y : 0.0f;
        d0[t] = 2.0f * c0 * e0 / B;
        d1[t] = ph ? 2.0f * c1 * e1 / B : 0.0f;
        l0 += c0 * e0 * e0;
        l1 += ph ? c1 * e1 * e1 : 0.0f;
        sc0 += c0;
        sc1 += ph ? c1 : 0.0f;
        ds0 += d0[t];
        ds1 += d1[t];
    }
    if (lane == 0) {
        lred[warp][0] = l0;
        lred[warp][1] = l1;
        lred[warp][2] = sc0;
        lred[warp][3] = sc1;
        lred[warp][4] = ds0;
        lred[warp][5] = ds1;
    }
    // opaque: else the compiler keeps the first pass's 64 unpacked values and spills
#pragma unroll
    for (int t = 0; t < 4; t++)
#pragma unroll
        for (int u = 0; u < 2; u++)
            asm volatile("" : "+r"(hq[t][u].x), "+r"(hq[t][u].y), "+r"(hq[t][u].z), "+r"(hq[t][u].w));
    asm volatile("" : "+l"(W6));
#pragma unroll
    for (int u = 0; u < 2; u++) {
        float w0[8], w1[8], g0[8] = {}, g1[8] = {};
        load8(W6 + u * 256 + lane * 8, w0);
        load8(W6 + kWidth + u * 256 + lane * 8, w1);
#pragma unroll
        for (int t = 0; t < 4; t++) {
            float h[8], z[8], dz[8];
            unpack8(hq[t][u], h);
            unpack8(zq[t][u], z);
#pragma unroll
            for (int e = 0; e < 8; e++) {
                g0[e] = fmaf(d0[t], h[e], g0[e]);
                g1[e] = fmaf(d1[t], h[e], g1[e]);
                const float dh = d0[t] * w0[e] + d1[t] * w1[e];
                const float sg = sigmoid_(z[e]);
                dz[e] = dh * (sg * (1.0f + z[e] * (1.0f - sg)));
            }
            const uint4 pk = make_uint4(pack2(dz[0], dz[1]), pack2(dz[2], dz[3]), pack2(dz[4], dz[5]),
                                        pack2(dz[6], dz[7]));
            *reinterpret_cast<uint4*>(dZ + (size_t)(row + t) * kWidth + u * 256 + lane * 8) = pk;
            *reinterpret_cast<uint4*>(&sm.tile[warp * 4 + t][u * 256 + lane * 8]) = pk;
        }
#pragma unroll
        for (int k = 0; k < 8; k += 4) {
            const int c = u * 256 + lane * 8 + k;
            *reinterpret_cast<float4*>(&sm.part[warp][c]) = make_float4(g0[k], g0[k + 1], g0[k + 2], g0[k + 3]);
            *reinterpret_cast<float4*>(&sm.part[warp][kWidth + c]) = make_float4(g1[k], g1[k + 1], g1[k + 2], g1[k + 3]);
        }
    }
    __syncthreads();
    // dZ^T: 32 consecutive rows of column c, 64 bytes per store group
    for (int c = threadIdx.x; c < kWidth; c += blockDim.x) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            __nv_bfloat162 v;
            v.x = sm.tile[2 * i][c];
            v.y = sm.tile[2 * i + 1][c];
            w[i] = *reinterpret_cast<uint32_t*>(&v);
        }
        uint4* d = reinterpret_cast<uint4*>(dZT + (size_t)c * B + r0);
#pragma unroll
        for (int i = 0; i < 4; i++) d[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
    }
    for (int i = threadIdx.x; i < kHeadStride; i += blockDim.x) {
        float v = 0.0f;
        if (i < 2 * kWidth + 2)
            for (int w = 0; w < 8; w++) v += i < 2 * kWidth ? sm.part[w][i] : lred[w][4 + i - 2 * kWidth];
        gpart[(size_t)blockIdx.x * kHeadStride + i] = v;
    }
    if (threadIdx.x < 4) {
        float v = 0.0f;
        for (int w = 0; w < 8; w++) v += lred[w][threadIdx.x];
        lpart[blockIdx.x * 4 + threadIdx.x] = v;
    }
}

struct BiasPtrs {
    const bf16* p[8];
};

// One block per (output unit, layer): tree sum of that dz^T row.
__global__ void __launch_bounds__(256) k_bias_grad(BiasPtrs d, int B, float* gb) {
    dep_wait();
    dep_release();
    __shared__ float sm[256];
    const int o = blockIdx.x, l = blockIdx.y;
    const bf16* row = d.p[l] + (size_t)o * B;
    float s = 0.0f;
    for (int b = threadIdx.x * 8; b < B; b += blockDim.x * 8) {
        float v[8];
        unpack8(*reinterpret_cast<const uint4*>(row + b), v);
#pragma unroll
        for (int i = 0; i < 8; i++) s += v[i];
    }
    sm[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) sm[threadIdx.x] += sm[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) gb[l * kWidth + o] = sm[0];
}

// ------------------------------------------------------------------ adam --

// Grids are (blocks over the largest segment, segments): a block works inside
// one segment, whose descriptor it reads from device memory.
// The partials are loaded 32 or 8 at a time before they are added (in the same
// order as one at a time), so a thread has that many loads in flight instead of
// one dependent load per partial (the head's segment sums 256 partials).
__device__ __forceinline__ float seg_grad(const AdamSeg& g, long long j) {
    const float* __restrict__ src = g.src + j;
    float grad = 0.0f;
    int q = 0;
    for (; q + 32 <= g.nsrc; q += 32) {
        float t[32];
#pragma unroll
        for (int u = 0; u < 32; u++) t[u] = __ldg(src + (long long)(q + u) * g.stride);
#pragma unroll
        for (int u = 0; u < 32; u++) grad += t[u];
    }
    for (; q + 8 <= g.nsrc; q += 8) {
        float t[8];
#pragma unroll
        for (int u = 0; u < 8; u++) t[u] = __ldg(src + (long long)(q + u) * g.stride);
#pragma unroll
        for (int u = 0; u < 8; u++) grad += t[u];
    }
    for (; q < g.nsrc; q++) grad += __ldg(src + (long long)q * g.stride);
    return grad;
}

// AdamW (Loshchilov & Hutter 2019) on the FP32 master copy, gradients summed
// from their partials in a fixed order; refreshes the BF16 copies W and W^T.
__device__ __forceinline__ float adam_one(const AdamArgs& a, const TrainScalars& ts, long long i, float m0, float v0, float p,
                                          float grad) {
    const float b1 = ts.beta1, b2 = ts.beta2;
    const float m = b1 * m0 + (1.0f - b1) * grad;
    const float v = b2 * v0 + (1.0f - b2) * grad * grad;
    a.m[i] = m;
    a.v[i] = v;
    p -= ts.lr * ((m / ts.bc1) / (sqrtf(v / ts.bc2) + a.eps) + a.weight_decay * p);
    a.p[i] = p;
    return p;
}

// A block of 256 threads takes a 32 x 32 tile of a weight segment, whose W^T goes
// out through shared memory; 256 parameters of a segment without copies; or 32
// parameters of one with many partials (the head's 256): it loads 128 partials of each at
// a time and a thread adds its parameter's in order. (One parameter per
// thread everywhere and the transposes in a launch of their own: 30.3 + 6.6 us
// for 1.1 M parameters, 36 MB of partials and 31 MB of state; 17.7 us here, cold.)
constexpr int kAdamMany = 32;  // partials from which a block takes 32 parameters
__host__ __device__ inline long long adam_items(const AdamSeg& g) {
    return g.wb ? 1024 : g.nsrc > kAdamMany ? 32 : 256;
}
__global__ void __launch_bounds__(256) k_adam(AdamArgs a) {
    dep_wait();
    dep_release();
    __shared__ union {
        bf16 t[32][33];
        float part[128][33];
    } sm;
    const AdamSeg g = a.dseg[blockIdx.y];
    const long long j0 = blockIdx.x * adam_items(g);
    if (j0 >= g.n) return;
    const TrainScalars ts = *a.ts;
    const int tid = threadIdx.x, x = tid & 31, y = tid >> 5;
    if (g.wb) {
        const int tiles = g.cols / 32, r0 = (blockIdx.x / tiles) * 32, c0 = (blockIdx.x % tiles) * 32;
        float m[4], v[4], p[4], grad[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const long long i = g.off + (long long)(r0 + y + 8 * k) * g.cols + c0 + x;
            m[k] = a.m[i];
            v[k] = a.v[i];
            p[k] = a.p[i];
            grad[k] = 0.0f;
        }
        int q = 0;
        for (; q + 4 <= g.nsrc; q += 4) {  // 16 loads in flight
            float u[4][4];
#pragma unroll
            for (int w = 0; w < 4; w++)
#pragma unroll
                for (int k = 0; k < 4; k++)
                    u[w][k] = __ldg(g.src + (q + w) * g.stride + (long long)(r0 + y + 8 * k) * g.cols + c0 + x);
#pragma unroll
            for (int w = 0; w < 4; w++)
#pragma unroll
                for (int k = 0; k < 4; k++) grad[k] += u[w][k];
        }
        for (; q < g.nsrc; q++)
#pragma unroll
            for (int k = 0; k < 4; k++)
                grad[k] += __ldg(g.src + q * g.stride + (long long)(r0 + y + 8 * k) * g.cols + c0 + x);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const long long j = (long long)(r0 + y + 8 * k) * g.cols + c0 + x;
            const bf16 w = __float2bfloat16_rn(adam_one(a, ts, g.off + j, m[k], v[k], p[k], grad[k]));
            g.wb[j] = w;
            sm.t[y + 8 * k][x] = w;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; k++) g.wt[(size_t)(c0 + y + 8 * k) * g.rows + r0 + x] = sm.t[x][y + 8 * k];
        return;
    }
    if (g.nsrc <= kAdamMany) {
        const long long j = j0 + tid;
        if (j < g.n) adam_one(a, ts, g.off + j, a.m[g.off + j], a.v[g.off + j], a.p[g.off + j], seg_grad(g, j));
        return;
    }
    const long long j = j0 + x, i = g.off + j;
    float grad = 0.0f, m = 0.0f, v = 0.0f, p = 0.0f;
    const bool own = y == 0 && j < g.n;
    if (own) {
        m = a.m[i];
        v = a.v[i];
        p = a.p[i];
    }
    for (int q0 = 0; q0 < g.nsrc; q0 += 128) {
        const int nq = g.nsrc - q0 < 128 ? g.nsrc - q0 : 128;
        if (j < g.n) {
            float u[16];
#pragma unroll
            for (int k = 0; k < 16; k++) u[k] = y + 8 * k < nq ? __ldg(g.src + (q0 + y + 8 * k) * g.stride + j) : 0.0f;
#pragma unroll
            for (int k = 0; k < 16; k++) sm.part[y + 8 * k][x] = u[k];
        }
        __syncthreads();
        if (own) {
            int q = 0;
            for (; q + 16 <= nq; q += 16)
#pragma unroll
                for (int k = 0; k < 16; k++) grad += sm.part[q + k][x];
            for (; q < nq; q++) grad += sm.part[q][x];
        }
        __syncthreads();
    }
    if (own) adam_one(a, ts, i, m, v, p, grad);
}

// W^T from W for every weight segment (parameters set from outside), 32 x 32
// tiles through shared memory.
__global__ void k_transpose_w(AdamArgs a) {
    dep_wait();
    dep_release();
    __shared__ bf16 t[32][33];
    const AdamSeg g = a.dseg[blockIdx.z];
    if (!g.wb) return;
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    if (c0 >= g.cols || r0 >= g.rows) return;
    for (int y = threadIdx.y; y < 32; y += blockDim.y) t[y][threadIdx.x] = g.wb[(size_t)(r0 + y) * g.cols + c0 + threadIdx.x];
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y) g.wt[(size_t)(c0 + y) * g.rows + r0 + threadIdx.x] = t[threadIdx.x][y];
}

__global__ void k_sync_weights(AdamArgs a) {
    const AdamSeg g = a.dseg[blockIdx.y];
    const long long j = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (j >= g.n || !g.wb) return;
    g.wb[j] = __float2bfloat16_rn(a.p[g.off + j]);
}

__global__ void k_grad_flat(AdamArgs a, float* out) {
    const AdamSeg g = a.dseg[blockIdx.y];
    const long long j = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (j >= g.n) return;
    out[g.off + j] = seg_grad(g, j);
}

// One warp: fixed-order sums of the head kernel's loss partials; each slot
// holds the step's two coefficient-weighted mean squared errors.
__global__ void k_loss_hist(const float* lpart, int nblk, int B, const TrainScalars* ts, float* hist, int cap) {
    dep_wait();
    dep_release();
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int b = threadIdx.x; b < nblk; b += 32)
        for (int q = 0; q < 4; q++) s[q] += lpart[4 * b + q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        for (int q = 0; q < 4; q++) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
    if (threadIdx.x == 0) {
        const long long slot = (ts->step - 1) % cap;
        hist[2 * slot] = s[2] > 0.0f ? s[0] / s[2] : 0.0f;
        hist[2 * slot + 1] = s[3] > 0.0f ? s[1] / s[3] : 0.0f;
    }
}

// ------------------------------------------------------------- inference --

// kFeatRows rows per block. Two threads per row form its point scalars (FP64
// logarithms of its range and of its frequency); then the block fills the features kind by
// kind, so that a warp's lanes do the same thing: the Fourier pairs (a sine and
// cosine share their argument and one call), the travel times' pairs, their
// logarithms, the scalars. A warp over half a row went through all kinds
// one after the other: 0.306 ms for 2^20 rows (268 MB written, 0.04 ms of HBM); 0.210 ms here. A
// thread per feature walking the rows repeated each row's logarithms: 1.89 ms.
constexpr int kFeatRows = 64;
constexpr int kFeatThreads = 256;
constexpr int kFourierPairs = (kIn - kFourierFeat) / 2, kTimePairs = (kLogTimeFeat - kTimeFeat) / 2;
constexpr int kLogPairs = (kFourierFeat - kLogTimeFeat) / 2;
__global__ void __launch_bounds__(kFeatThreads) k_features(FeatureArgs a, long long rows_padded) {
    dep_wait();
    dep_release();
    __shared__ PointScalars ps[kFeatRows];
    __shared__ const float* soil[kFeatRows];  // null past the last row
    const long long q0 = (long long)blockIdx.x * kFeatRows;
    const int tid = threadIdx.x;
    if (tid < 2 * kFeatRows) {
        const int i = tid & (kFeatRows - 1);
        const long long q = q0 + i;
        const bool in = q < a.rows;
        const long long p = a.p0 + q, t = p / a.nr;
        if (tid < kFeatRows) {
            soil[i] = in ? a.soilfeat + (t / a.nf) * kSoilStride : nullptr;
            if (in) range_scalars(ps[i], a.ranges[static_cast<int>(p % a.nr)], a.dom);
        } else if (in) {
            freq_scalars(ps[i], a.freqs[static_cast<int>(t % a.nf)], a.dom);
        }
    }
    __syncthreads();
    const int rows = static_cast<int>(rows_padded - q0 < kFeatRows ? rows_padded - q0 : kFeatRows);
    uint32_t* const X = reinterpret_cast<uint32_t*>(a.X + q0 * kIn);
    auto fill = [&](auto kind, int j0) {  // features [j0, j0 + 2 pairs) of all rows
        constexpr int pairs = decltype(kind)::value;
        for (int it = tid; it < rows * pairs; it += kFeatThreads) {
            const int i = it / pairs, j = j0 + 2 * (it - i * pairs);
            float v0 = 0.0f, v1 = 0.0f;
            if (const float* sf = soil[i]) feature_pair(j, sf, ps[i], a.fourier, v0, v1);
            X[i * (kIn / 2) + (j >> 1)] = pack2(v0, v1);
        }
    };
    fill(std::integral_constant<int, kFourierPairs>{}, kFourierFeat);
    fill(std::integral_constant<int, kTimePairs>{}, kTimeFeat);
    fill(std::integral_constant<int, kLogPairs>{}, kLogTimeFeat);
    fill(std::integral_constant<int, kScalars / 2>{}, 0);
}
static_assert(kScalars == kTimeFeat, "the kinds follow one another");

// A warp takes 32 rows, their dot products one after the other (the row's 1 KB
// coalesced, the next row's loads in flight), then each lane turns one row's
// outputs into G: the FP64 exponential and sine-cosine run on 32 lanes instead
// of one (1.13 ms for 2^20 rows with a row per warp).
__global__ void __launch_bounds__(256) k_head_infer(HeadInferArgs a) {
    dep_wait();
    dep_release();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long q0 = (blockIdx.x * 8LL + warp) * 32;
    if (q0 >= a.rows) return;
    const int nrows = static_cast<int>(a.rows - q0 < 32 ? a.rows - q0 : 32);
    float w0[16], w1[16];
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
        for (int e = 0; e < 8; e++) {
            w0[8 * u + e] = a.W6[u * 256 + lane * 8 + e];
            w1[8 * u + e] = a.W6[kWidth + u * 256 + lane * 8 + e];
        }
    const uint4* row = reinterpret_cast<const uint4*>(a.H + q0 * kWidth) + lane;
    uint4 n0 = row[0], n1 = row[32];
    float o0 = 0.0f, o1 = 0.0f;
#pragma unroll 2
    for (int r = 0; r < nrows; r++) {
        float h[16];
        unpack8(n0, h);
        unpack8(n1, h + 8);
        if (r + 1 < nrows) {
            n0 = row[(r + 1) * (kWidth / 8)];
            n1 = row[(r + 1) * (kWidth / 8) + 32];
        }
        float y0 = 0.0f, y1 = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            y0 = fmaf(h[i], w0[i], y0);
            y1 = fmaf(h[i], w1[i], y1);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            y0 += __shfl_xor_sync(0xffffffffu, y0, o);
            y1 += __shfl_xor_sync(0xffffffffu, y1, o);
        }
        if (lane == r) {
            o0 = y0;
            o1 = y1;
        }
    }
    if (lane >= nrows) return;
    const long long q = q0 + lane;
    const double t0 = static_cast<double>(o0 + a.b6[0]) * a.y_std0 + a.y_mean0;
    const double t1 = static_cast<double>(o1 + a.b6[1]) * a.y_std1 + a.y_mean1;
    const long long p = a.p0 + q;
    const int ir = static_cast<int>(p % a.nr);
    const int jf = static_cast<int>((p / a.nr) % a.nf);
    const double phi = -t1 * (2.0 * CUDART_PI * a.freqs[jf]) * a.ranges[ir];
    double sn, cs;
    sincos(phi, &sn, &cs);
    const double amp = exp(t0);
    a.G[p] = mk(amp * cs, amp * sn);
    if (a.T) {
        a.T[2 * q] = static_cast<float>(t0);
        a.T[2 * q + 1] = static_cast<float>(t1);
    }
}

// ---------------------------------------------------------------- labels --

constexpr int kLabelThreads = 128;
constexpr int16_t kBroken = INT16_MIN;

__device__ __forceinline__ double amp_of(cd g) { return hypot(g.re, g.im); }

// One block per soil. Phase unwrapping follows bank.prepare
// (internal/bank/interp.go:66-102): along range, each step folded into
// (-pi, pi]. A 1 m range step spans many cycles at high frequency for slow
// soils, so the fold is taken about a prediction instead of about zero: the
// same range step one frequency bin lower, scaled by f_j / f_{j-1} (the
// step is -k(f) dr and k grows about linearly in f). The first range is
// unwrapped along frequency the same way. Whole-cycle counts are kept as
// integers, so phi = principal value + 2 pi n exactly. A chain stops (the
// phase label becomes NaN) at the first cell below the amplitude floor.
__global__ void __launch_bounds__(kLabelThreads) k_labels(LabelArgs a) {
    extern __shared__ int16_t cyc[];  // [nr][nf]
    __shared__ double red[kLabelThreads];
    const int s = blockIdx.x, tid = threadIdx.x;
    const cd* G = a.G + (size_t)s * a.nf * a.nr;
    const int cells = a.nf * a.nr;
    double mx = 0.0;
    for (int c = tid; c < cells; c += blockDim.x) mx = fmax(mx, amp_of(G[c]));
    red[tid] = mx;
    __syncthreads();
    for (int w = kLabelThreads / 2; w > 0; w >>= 1) {
        if (tid < w) red[tid] = fmax(red[tid], red[tid + w]);
        __syncthreads();
    }
    const double floor_amp = red[0] * a.floor_rel;
    __syncthreads();
    const double two_pi = 2.0 * CUDART_PI;
    if (tid < a.nr) {
        const int i = tid;
        double dprev = 0.0, wprev = 0.0, rmax = 0.0;
        int n = 0;
        bool ok = true;
        for (int j = 0; j < a.nf; j++) {
            const cd g = G[(size_t)j * a.nr + i];
            rmax = fmax(rmax, amp_of(g));
            const double w = atan2(g.im, g.re);
            if (i == 0) {
                if (j > 0) {
                    const double dw = w - wprev;
                    const double m = rint((dprev - dw) / two_pi);
                    dprev = dw + two_pi * m;
                    n += static_cast<int>(m);
                }
                ok = ok && amp_of(g) > floor_amp;
                cyc[j] = ok ? static_cast<int16_t>(n) : kBroken;
                wprev = w;
            } else {
                const cd gp = G[(size_t)j * a.nr + i - 1];
                const double dw = w - atan2(gp.im, gp.re);
                const double pred = j > 0 ? dprev * (a.freqs[j] / a.freqs[j - 1]) : 0.0;
                const double m = rint((pred - dw) / two_pi);
                dprev = dw + two_pi * m;
                ok = ok && amp_of(g) > floor_amp && amp_of(gp) > floor_amp;
                cyc[(size_t)i * a.nf + j] = ok ? static_cast<int16_t>(m) : kBroken;
            }
        }
        a.lmax[(size_t)s * a.nr + i] = static_cast<float>(log(fmax(rmax, 1e-300)));
    }
    __syncthreads();
    double st[6] = {0, 0, 0, 0, 0, 0};
    const float qnan = __int_as_float(0x7fc00000);
    for (int j = tid; j < a.nf; j += blockDim.x) {
        int n = cyc[j];
        bool valid = n != kBroken;
        const double w_r = two_pi * a.freqs[j];
        for (int i = 0; i < a.nr; i++) {
            if (i > 0) {
                const int m = cyc[(size_t)i * a.nf + j];
                if (m == kBroken) valid = false;
                if (valid) n += m;
            }
            const cd g = G[(size_t)j * a.nr + i];
            const double t0 = log(fmax(amp_of(g), floor_amp));
            float* L = a.labels + (((size_t)s * a.nr + i) * a.nf + j) * 2;
            L[0] = static_cast<float>(t0);
            st[0] += 1.0;
            st[1] += t0;
            st[2] += t0 * t0;
            if (valid) {
                const double phi = atan2(g.im, g.re) + two_pi * n;
                const double t1 = -phi / (w_r * a.ranges[i]);
                L[1] = static_cast<float>(t1);
                st[3] += 1.0;
                st[4] += t1;
                st[5] += t1 * t1;
            } else {
                L[1] = qnan;
            }
        }
    }
    for (int q = 0; q < 6; q++) {
        __syncthreads();
        red[tid] = st[q];
        __syncthreads();
        for (int w = kLabelThreads / 2; w > 0; w >>= 1) {
            if (tid < w) red[tid] += red[tid + w];
            __syncthreads();
        }
        if (tid == 0) a.stats[(size_t)s * 6 + q] = red[0];
    }
}

// ------------------------------------------------------------------ eval --

__global__ void __launch_bounds__(256) k_eval(const float* T, const float* labels, const int* soil_ids,
                                              long long p0, long long rows, int nr, int nf, const double* ranges,
                                              const double* freqs, double* acc) {
    __shared__ double sm[6][256];
    double a[6] = {0, 0, 0, 0, 0, 0};
    for (long long q = blockIdx.x * 256LL + threadIdx.x; q < rows; q += (long long)gridDim.x * 256) {
        const long long p = p0 + q;
        const int ir = static_cast<int>(p % nr);
        const int jf = static_cast<int>((p / nr) % nf);
        const long long sl = p / ((long long)nr * nf);
        const float* L = labels + (((size_t)soil_ids[sl] * nr + ir) * nf + jf) * 2;
        const double wr = 2.0 * CUDART_PI * freqs[jf] * ranges[ir];
        const double e0 = (double)T[2 * q] - L[0];
        a[0] += e0 * e0;
        const double al = exp((double)L[0]), ap = exp((double)T[2 * q]);
        if (!isnan(L[1])) {
            const double e1 = (double)T[2 * q + 1] - L[1];
            a[1] += 1.0;
            a[2] += e1 * e1;
            a[3] += (e1 * wr) * (e1 * wr);
            // |ap e^{-i t1p wr} - al e^{-i t1l wr}|^2
            a[4] += ap * ap + al * al - 2.0 * ap * al * cos(e1 * wr);
        } else {
            a[4] += (ap - al) * (ap - al);
        }
        a[5] += al * al;
    }
    for (int k = 0; k < 6; k++) sm[k][threadIdx.x] = a[k];
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w)
            for (int k = 0; k < 6; k++) sm[k][threadIdx.x] += sm[k][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < 6) acc[blockIdx.x * 6 + threadIdx.x] = sm[threadIdx.x][0];
}

// ------------------------------------------------------------------ host --

namespace {
bool make_map_bf16(CUtensorMap* map, const bf16* base, int rows, int K, bool wide = false) {
    auto fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    cuuint32_t box[2] = {(cuuint32_t)(wide ? BK : BKE), (cuuint32_t)BM};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, wide ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MODE>
bool set_attr() {
    return cudaFuncSetAttribute(k_gemm<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) ==
           cudaSuccess;
}

template <int MODE>
void launch_mode(cudaStream_t s, const CUtensorMap& ta, const CUtensorMap& tb, dim3 grid, const GemmArgs& a) {
    // weight gradients run on a second stream behind an event: an ordinary
    // launch, so that event stays a full dependency
    if (MODE == kWgrad)
        k_gemm<MODE><<<grid, THREADS, SMEM_BYTES, s>>>(ta, tb, a);
    else
        launch_dep(k_gemm<MODE>, grid, dim3(THREADS), SMEM_BYTES, s, ta, tb, a);
}
}  // namespace

int prepare_gemm() {
    static std::atomic<bool> done{false};
    if (!done.load(std::memory_order_relaxed) && set_attr<kFwdTrain>() && set_attr<kFwdInfer>() && set_attr<kBwdData>() && set_attr<kWgrad>() &&
        cudaFuncSetAttribute(k_layer_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, kInfSmem) == cudaSuccess &&
        cudaFuncSetAttribute(k_head_train, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(HeadShared)) == cudaSuccess)
        done.store(true, std::memory_order_relaxed);
    return done.load(std::memory_order_relaxed) ? 0 : 3;
}

int launch_gemm(cudaStream_t s, int mode, const bf16* A, const bf16* B, int rowsA, int rowsB, int ktotal, int splits,
                const GemmArgs& a0) {
    if (rowsA <= 0 || rowsB <= 0 || splits <= 0 || rowsA % BM || rowsB % BN || ktotal % (BK * splits)) return 1;
    if (prepare_gemm()) return 3;
    CUtensorMap ta, tb;
    if (!make_map_bf16(&ta, A, rowsA, ktotal) || !make_map_bf16(&tb, B, rowsB, ktotal)) return 2;
    GemmArgs a = a0;
    a.M = rowsA;
    a.N = rowsB;
    a.K = ktotal / splits;
    const dim3 grid(rowsB / BN, rowsA / BM, splits);
    switch (mode) {
        case kFwdTrain: launch_mode<kFwdTrain>(s, ta, tb, grid, a); return 0;
        case kFwdInfer: {
            if (splits != 1 || a.K / BK > kInfKb || a.N % kInfN) return 1;
            int dev = 0, sms = 0;
            if (cudaGetDevice(&dev) != cudaSuccess ||
                cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
                return 3;
            // While every tile has a place of its own (two CTAs per SM) k_gemm is
            // ahead: its CTAs start beside the previous layer's, those with all of an
            // SM's shared memory cannot. A prediction of 1 / 2048 / 8192 rows: 132 / 175 /
            // 236 us, with the pairs 158 / 200 / 248; of 12288 / 16384 / 2^20: 297 / 319 /
            // 5530 against 303 / 319 / 3750.
            if (rowsA / BM * (rowsB / BN) <= 2 * sms) {
                launch_mode<kFwdInfer>(s, ta, tb, grid, a);
                return 0;
            }
            CUtensorMap to;
            if (!make_map_bf16(&ta, A, rowsA, ktotal, true) || !make_map_bf16(&tb, B, rowsB, ktotal, true) ||
                !make_map_bf16(&to, a.out, rowsA, rowsB, true))
                return 2;
            const int slabs = rowsB / kInfN;  // a pair of CTAs per pair of SMs, as many for each slab
            const int pairs = slabs * std::max(1, std::min(sms / 2 / slabs, (rowsA + 2 * BM - 1) / (2 * BM)));
            launch_dep(k_layer_infer, dim3(2 * pairs), dim3(kInfThreads), kInfSmem, s, ta, tb, to, a);
            return 0;
        }
        case kBwdData: launch_mode<kBwdData>(s, ta, tb, grid, a); return 0;
        case kWgrad: launch_mode<kWgrad>(s, ta, tb, grid, a); return 0;
    }
    return 1;
}

void launch_step_begin(cudaStream_t s, TrainScalars* ts) { launch_dep(k_step_begin, dim3(1), dim3(1), 0, s, ts); }

void launch_batch(cudaStream_t s, const BatchArgs& a) {
    launch_dep(k_batch, dim3(a.B / kBatchRows), dim3(kBatchThreads), 0, s, a);
}

void launch_head_train(cudaStream_t s, const bf16* H, const bf16* Z, const float* W6, const float* b6, const float* Y,
                       const float* C, int B, bf16* dZ, bf16* dZT, float* gpart, float* lpart) {
    launch_dep(k_head_train, dim3(B / kHeadRows), dim3(256), sizeof(HeadShared), s,  // prepare_gemm set the limit
               H, Z, W6, b6, Y, C, B, dZ, dZT, gpart, lpart);
}

void launch_bias_grad(cudaStream_t s, const bf16* const* dZT, int layers, int B, float* gb) {
    BiasPtrs d{};
    for (int l = 0; l < layers && l < 8; l++) d.p[l] = dZT[l];
    k_bias_grad<<<dim3(kWidth, layers), 256, 0, s>>>(d, B, gb);  // follows the join of the two streams
}

namespace {
long long max_seg(const AdamArgs& a) {
    long long m = 1;
    for (int s = 0; s < a.nseg; s++) m = a.seg[s].n > m ? a.seg[s].n : m;
    return m;
}
void launch_transposes(cudaStream_t s, const AdamArgs& a) {
    int rows = 32, cols = 32;
    for (int q = 0; q < a.nseg; q++)
        if (a.seg[q].wb) {
            rows = a.seg[q].rows > rows ? a.seg[q].rows : rows;
            cols = a.seg[q].cols > cols ? a.seg[q].cols : cols;
        }
    launch_dep(k_transpose_w, dim3(cols / 32, rows / 32, a.nseg), dim3(32, 8), 0, s, a);
}
}  // namespace

void launch_adam(cudaStream_t s, const AdamArgs& a, long long) {
    long long blocks = 1;
    for (int q = 0; q < a.nseg; q++) {
        const long long per = adam_items(a.seg[q]);
        blocks = std::max(blocks, (a.seg[q].n + per - 1) / per);
    }
    launch_dep(k_adam, dim3((unsigned)blocks, a.nseg), dim3(256), 0, s, a);
}

void launch_sync_weights(cudaStream_t s, const AdamArgs& a, long long) {
    k_sync_weights<<<dim3((unsigned)((max_seg(a) + 255) / 256), a.nseg), 256, 0, s>>>(a);
    launch_transposes(s, a);
}

void launch_grad_flat(cudaStream_t s, const AdamArgs& a, long long, float* out) {
    k_grad_flat<<<dim3((unsigned)((max_seg(a) + 255) / 256), a.nseg), 256, 0, s>>>(a, out);
}

void launch_loss_hist(cudaStream_t s, const float* lpart, int nblk, int B, const TrainScalars* ts, float* hist,
                      int cap) {
    launch_dep(k_loss_hist, dim3(1), dim3(32), 0, s, lpart, nblk, B, ts, hist, cap);
}

void launch_features(cudaStream_t s, const FeatureArgs& a, long long rows_padded) {
    launch_dep(k_features, dim3((unsigned)((rows_padded + kFeatRows - 1) / kFeatRows)), dim3(kFeatThreads), 0, s, a,
               rows_padded);
}

void launch_head_infer(cudaStream_t s, const HeadInferArgs& a) {
    launch_dep(k_head_infer, dim3((unsigned)((a.rows + 255) / 256)), dim3(256), 0, s, a);
}

int launch_labels(cudaStream_t s, const LabelArgs& a) {
    if (a.nr > kLabelThreads || a.nr < 1 || a.nf < 1) return 1;
    const size_t smem = (size_t)a.nr * a.nf * sizeof(int16_t);
    if (smem > 200 * 1024) return 1;
    static size_t attr = 0;
    if (smem > 48 * 1024 && smem > attr) {
        if (cudaFuncSetAttribute(k_labels, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
            return 3;
        attr = smem;
    }
    k_labels<<<a.ns, kLabelThreads, smem, s>>>(a);
    return 0;
}

void launch_eval(cudaStream_t s, const float* T, const float* labels, const int* soil_ids, long long p0,
                 long long rows, int nr, int nf, const double* ranges, const double* freqs, double* acc, int nblk) {
    k_eval<<<nblk, 256, 0, s>>>(T, labels, soil_ids, p0, rows, nr, nf, ranges, freqs, acc);
}

}  // namespace mlp
}  // namespace gfk
