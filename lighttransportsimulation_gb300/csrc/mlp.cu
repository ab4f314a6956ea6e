// Radiance-cache MLP kernels on the 5th-generation tensor cores (tcgen05, BF16 operands in shared
// memory, FP32 accumulators in tensor memory), and a product check of the operand layouts.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "dev_common.cuh"
#include "mlp.cuh"
#include "umma.cuh"

#include <cuda.h>
#include <cuda_bf16.h>
#include <cmath>
#include <cstring>

namespace lts {
namespace {

constexpr int kProbeSmem = 96 * 1024;

__global__ __launch_bounds__(128) void k_umma_probe(const uint16_t* __restrict__ A, const uint16_t* __restrict__ B,
                                                    float* __restrict__ D, int mode, int swap, uint32_t* err) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* sA = smem;
    unsigned char* sB = smem + 32 * 1024;
    uint64_t* mbar = (uint64_t*)(smem + 64 * 1024);
    uint32_t* tslot = (uint32_t*)(smem + 64 * 1024 + 64);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // operand shapes (rows x columns of the stored RC matrices) and the product's M, N, K
    const int ar = 128, ac = mode == 2 ? 96 : 64;
    const int br = mode == 2 ? 128 : 64, bc = mode == 0 ? 64 : (mode == 1 ? 96 : 64);
    const int N = mode == 1 ? 96 : 64, K = mode == 2 ? 128 : 64;
    for (int e = tid; e < ar * ac; e += 128) {
        const int r = e / ac, c = e % ac;
        *(uint16_t*)(sA + rc_offset(r, c, ac)) = A[e];
    }
    for (int e = tid; e < br * bc; e += 128) {
        const int r = e / bc, c = e % bc;
        *(uint16_t*)(sB + rc_offset(r, c, bc)) = B[e];
    }
    if (tid == 0) mbar_init(mbar, 1);
    if (warp == 0) tmem_alloc(tslot, 128);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    if (tid == 0) {
        const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB);
        const uint32_t idesc = umma_idesc_bf16(128, N, mode == 2, mode != 0);
        for (int s = 0; s < K / 16; ++s) {
            uint64_t da, db;
            if (mode == 2) {  // MN-major A: K rows of 16 ac bytes
                const uint32_t lbo = swap ? 128u : 16u * ac, sbo = swap ? 16u * ac : 128u;
                da = umma_desc(a0 + s * 2 * 16 * ac, lbo, sbo);
            } else {
                da = umma_desc(a0 + s * 256, 128, 16 * ac);
            }
            if (mode == 0) {
                db = umma_desc(b0 + s * 256, 128, 16 * bc);
            } else {
                const uint32_t lbo = swap ? 128u : 16u * bc, sbo = swap ? 16u * bc : 128u;
                db = umma_desc(b0 + s * 2 * 16 * bc, lbo, sbo);
            }
            umma_bf16(tmem, da, db, idesc, s > 0);
        }
        umma_commit(mbar);
    }
    const bool ok = mbar_wait(mbar, 0, err);
    if (!ok && tid == 0) mbar_drain(mbar, 0, err);
    tc_fence_after();
    if (ok) {
        const int row = 32 * warp + lane;
        for (int c0 = 0; c0 < N; c0 += 16) {
            float v[16];
            tmem_ld16(tmem + ((uint32_t)(32 * warp) << 16) + c0, v);
            for (int k = 0; k < 16; ++k) D[row * N + c0 + k] = v[k];
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 128);
}


// ------------------------------------------------------------------ the radiance-cache MLP
// Shared memory (bytes).  Weights in RC layout: W0 64x96, W1..W4 64x64, W5 16x64; two input
// tiles X (128 x 96: this tile's and the next one's), hidden activations H1..H5 (128 x 64 each),
// the output-gradient tile Gz (128 x 16) and two hidden-gradient tiles Ga (128 x 64).  MN-major
// reads of a 64- or 96-column buffer with M = 128 run past its end into the next buffer; those
// product rows are never used.
__host__ __device__ constexpr uint32_t kSW(int L) { return L == 0 ? 0u : 12288u + 8192u * (uint32_t)(L - 1); }
constexpr uint32_t kSX = 47104;
constexpr uint32_t kSH = kSX + 2 * 24576;
constexpr uint32_t kSGz = kSH + 5 * 16384;
constexpr uint32_t kSGa = kSGz + 4096;
constexpr uint32_t kTrainBar = kSGa + 2 * 16384;
constexpr uint32_t kTrainSmem = kTrainBar + 64;
// Eight warps, two per 32 rows (columns 0..31 and 32..63), and one warp that issues the products.
constexpr int kTrainThreads = 288;
static_assert(kTrainSmem <= 232448, "training tile exceeds shared memory");
// Inference keeps kFwdGroups tiles in flight per CTA (one CTA per SM), one warpgroup of 128
// threads per tile, sharing the weights: each tile has a 24 KB buffer at fwd_buf(g) for its features
// X (128 x 96), an mbarrier and 96 TMEM columns -- the product D (128 x 64 FP32) and, as the next
// product's A operand, the activations (128 x 64 bf16, two to a column).
constexpr int kFwdGroups = 5;
constexpr uint32_t kFwdTileBytes = 24576;
__host__ __device__ constexpr uint32_t fwd_buf(int g) { return kSX + kFwdTileBytes * (uint32_t)g; }
// then two mbarriers per tile (products, feature copies) and the TMEM slot
constexpr uint32_t kFwdBar = kSX + kFwdTileBytes * kFwdGroups;
constexpr uint32_t kFwdSmem = kFwdBar + 16 * kFwdGroups + 16;
static_assert(kSX % 1024 == 0 && kFwdTileBytes % 1024 == 0, "swizzled copies need 1024-byte aligned buffers");
constexpr uint32_t kFwdCols = 512, kFwdTileCols = 96, kFwdACol = 64;
static_assert(kFwdTileCols * kFwdGroups <= kFwdCols && kFwdSmem <= 232448, "inference tiles exceed TMEM or shared memory");
// TMEM columns: 0..63 the working product; dW_k^T accumulators (training) at kDwCol(k)
__host__ __device__ constexpr uint32_t kDwCol(int L) { return 64u * (uint32_t)(L + 1); }

// Two floats to one word of two bf16, a in the low half.
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
// And ReLU: rounded first, then clamped (the same values; NaN becomes 0 as by fmaxf).
__device__ __forceinline__ uint32_t relu_bf16x2(uint32_t a, uint32_t b) {
    uint32_t r = pack_bf16x2(__uint_as_float(a), __uint_as_float(b));
    asm("max.bf16x2 %0, %0, %1;" : "+r"(r) : "r"(0u));
    return r;
}
// All ones in the halves of w that are > 0.
__device__ __forceinline__ uint32_t positive_bf16x2(uint32_t w) {
    __nv_bfloat162 v;
    memcpy(&v, &w, 4);
    return __hgt2_mask(v, __floats2bfloat162_rn(0.f, 0.f));
}

// Row `row` of an R x C RC-layout buffer: store / load the 8 NJ values (two to a word) from column c0 on.
template <int NJ>
__device__ __forceinline__ void rc_store_row(unsigned char* buf, int row, int C, int c0, const uint32_t* v) {
#pragma unroll
    for (int j = 0; j < NJ; ++j)
        *(uint4*)(buf + rc_offset(row, c0 + 8 * j, C)) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
}
template <int NJ>
__device__ __forceinline__ void rc_load_row(const unsigned char* buf, int row, int C, int c0, uint32_t* v) {
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        const uint4 q = *(const uint4*)(buf + rc_offset(row, c0 + 8 * j, C));
        v[4 * j] = q.x; v[4 * j + 1] = q.y; v[4 * j + 2] = q.z; v[4 * j + 3] = q.w;
    }
}

// Weights (global, bf16 row-major [out][in]) into their RC slots: every copy of a thread in flight
// at once (a loop per layer paid the latency per layer), landed on return.
__device__ void load_weights(uint32_t sbase, const uint16_t* __restrict__ w16) {
    for (int e = threadIdx.x; e < kMlpParams / 8; e += blockDim.x) {
        int L = 0, f = e;
        if (e >= 768) L = 1 + (e - 768) / 512, f = (e - 768) % 512;  // W0 64 x 96, the others 64 (16) x 64
        const int C = mlp_in(L), r = f / (C / 8), j = f % (C / 8);
        cp_async16(sbase + kSW(L) + rc_offset(r, 8 * j, C), w16 + 8 * e, true);
    }
    cp_async_wait();
}

// All threads: makes the shared-memory operands written so far visible to the tensor cores.
__device__ __forceinline__ void publish_smem() {
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
}

// Issue (thread 0) D[128 x N] = A[128 x K] . W^T with A (row-major activations, K-major) at a_off
// (a_cols columns) and W [N x K] (K-major) at w_off.
__device__ __forceinline__ void issue_fwd(uint32_t tmem_d, uint32_t sbase, uint32_t a_off, int a_cols, uint32_t w_off,
                                          int N, int K) {
    const uint32_t idesc = umma_idesc_bf16(128, N, false, false);
    for (int s = 0; s < K / 16; ++s)
        umma_bf16(tmem_d, umma_desc(sbase + a_off + s * 256, 128, 16 * a_cols),
                  umma_desc(sbase + w_off + s * 256, 128, 16 * K), idesc, s > 0);
}

// Named barrier over the 128 threads of warpgroup `id - 1` (barrier 0 is __syncthreads).
__device__ __forceinline__ void wg_sync(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }
__device__ __forceinline__ bool wg_sync_and(int id, bool v) {
    uint32_t r;
    asm volatile(
        "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.and.pred q, %2, 128, p;\nselp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(r)
        : "r"((uint32_t)v), "r"(id)
        : "memory");
    return r != 0;
}
// Inference: out[r * stride + c] = exp(z_c), c < 3, for the feature rows r = rows[i] (rows null:
// r = i), i < n.  Persistent CTAs of kFwdGroups warpgroups; warpgroup g runs tiles
// g * gridDim.x + blockIdx.x, + gridDim.x * kFwdGroups, ..., and synchronises with named barrier 1 + g
// only, so the tiles of a CTA overlap each other's epilogues and waits.  A tile is a chain of six
// dependent products, so what bounds the kernel is that chain's latency over the tiles in flight.
// It is kept short: the hidden activations never leave TMEM (the epilogue loads D, rounds and
// clamps, stores the next product's A operand; no shared-memory stores, no proxy fence, and the
// product reads only the weights from shared memory), one barrier per layer, and the next tile's
// features load while the current tile's hidden layers run.  Features in row order (MAP) come by
// TMA, two swizzled boxes a tile that the first product reads as they are; listed rows (the
// renderer's queries) by cp.async, 64 contiguous bytes per row.  2,073,600 rows, us a call: 235
// through shared memory with the loads in the chain; 140 with the activations in TMEM and cp.async
// for every tile (its address work and L1 traffic slow the chain: 95 without it); 97 with
// TMA.  HBM floor 62, the products alone 64.
template <bool MAP>
__global__ __launch_bounds__(128 * kFwdGroups) void k_mlp_forward(const uint16_t* __restrict__ w16,
                                                                 const uint16_t* __restrict__ feat,
                                                                 const int32_t* __restrict__ rows, int n,
                                                                 const uint32_t* d_n, float* __restrict__ out,
                                                                 int stride, uint32_t* err,
                                                                 const __grid_constant__ CUtensorMap map_a,
                                                                 const __grid_constant__ CUtensorMap map_b) {
    if (d_n) n = min(n, (int)*d_n);  // a count produced on the device (at most n)
    extern __shared__ __align__(1024) unsigned char smem[];
    const int g = threadIdx.x >> 7, row = threadIdx.x & 127, lane = threadIdx.x & 31, bar_id = 1 + g;
    uint64_t* mbar = (uint64_t*)(smem + kFwdBar) + 2 * g;
    uint64_t* xbar = mbar + 1;  // MAP: the tile's features have arrived
    uint32_t* tslot = (uint32_t*)(smem + kFwdBar + 16 * kFwdGroups);
    const uint32_t sbase = smem_u32(smem), buf = fwd_buf(g);
    const int ntiles = (n + 127) / 128, step = gridDim.x * kFwdGroups;
    // A wait that runs out sets the error flag and is not repeated; the tile runs through, row 0 issues
    // nothing more, and at the end it waits for what it has issued.
    bool ok = true;
    bool xpending = false, ppending = false;  // row 0's feature copy / product that nothing has waited for
    uint32_t pphase = 0;                      // that product's phase
    // The features of tile t into the buffer, a warp its 32 rows: each access 8 rows x 64 bytes.
    // Returns this thread's feature row of the tile (-1: none).
    auto load_tile = [&](int t) -> long {
        const long i = (long)t * 128 + row;
        const bool valid = t < ntiles && i < n;
        if (MAP) {
            if (row == 0 && t < ntiles && ok) {
                xpending = true;
                mbar_expect(xbar, kFwdTileBytes);  // rows past n arrive as zeros
                tma_load_2d(sbase + buf, &map_a, 0, t * 128, xbar);
                tma_load_2d(sbase + buf + 16384, &map_b, 64, t * 128, xbar);
            }
            return valid ? i : -1;
        }
        const int mine = valid ? (rows ? __ldg(rows + i) : (int)i) : -1;
        if (t < ntiles) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int sub = 8 * q + (lane & 7), r = __shfl_sync(~0u, mine, sub);
                const uint32_t dst = sbase + buf + rc_offset((row & ~31) + sub, 0, kMlpIn);
#pragma unroll
                for (int j4 = 0; j4 < 3; ++j4) {
                    const int j = 4 * j4 + (lane >> 3);
                    cp_async16(dst + 128u * j, feat + (size_t)max(r, 0) * kMlpIn + 8 * j, r >= 0);
                }
            }
        }
        return mine;
    };
    int tile = g * gridDim.x + blockIdx.x;
    long r = -1;
    if (row == 0) {
        mbar_init(mbar, 1);
        mbar_init(xbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    r = load_tile(tile);
    load_weights(smem_u32(smem), w16);
    if ((threadIdx.x >> 5) == 0) tmem_alloc(tslot, kFwdCols);
    publish_smem();
    const uint32_t tmem = *tslot + kFwdTileCols * (uint32_t)g;
    const uint32_t mine = tmem + ((uint32_t)(32 * ((threadIdx.x >> 5) & 3)) << 16);  // warp w: lanes 32 (w % 4) ..
    uint32_t phase = 0, xphase = 0;  // xphase: row 0's, of the copy it waits for next
    auto product = [&](int L) {  // issue layer L's product and wait for it
        if (row == 0 && ok && L == 0 && MAP) {
            ok = mbar_wait(xbar, xphase, err);
            if (ok) {
                xpending = false;
                xphase ^= 1u;
            }
        }
        if (row == 0 && ok) {
            if (L == 0 && MAP) {
                const uint32_t idesc = umma_idesc_bf16(128, 64, false, false);
                for (int s = 0; s < 6; ++s)
                    umma_bf16(tmem, s < 4 ? umma_desc_swizzled(sbase + buf + 32 * s, 128)
                                          : umma_desc_swizzled(sbase + buf + 16384 + 32 * (s - 4), 64),
                              umma_desc(sbase + kSW(0) + s * 256, 128, 16 * kMlpIn), idesc, s > 0);
            } else if (L == 0) {
                issue_fwd(tmem, sbase, buf, kMlpIn, kSW(0), 64, kMlpIn);
            } else {
                const uint32_t idesc = umma_idesc_bf16(128, mlp_out(L), false, false);
                for (int s = 0; s < 4; ++s)
                    umma_bf16_ta(tmem, tmem + kFwdACol + 8 * s, umma_desc(sbase + kSW(L) + s * 256, 128, 16 * 64), idesc, s > 0);
            }
            umma_commit(mbar);
        }
        if (ok) {
            ok = mbar_wait(mbar, phase, err);
            if (!ok) {
                ppending = row == 0;
                pphase = phase;
            }
        }
        phase ^= 1u;
        __syncwarp();  // the lanes leave the wait one by one; the TMEM accesses are warp-wide
        tc_fence_after();
    };
    for (; tile < ntiles; tile += step) {
        // the features are in (cp.async: published here), and every row of the tile before has read its
        // outputs from TMEM
        if (!MAP) {
            cp_async_wait();
            fence_async_smem();
        }
        tc_fence_before();
        if (!wg_sync_and(bar_id, ok)) break;
        tc_fence_after();
        product(0);
        const long next = load_tile(tile + step);
        for (int L = 1; L < kMlpLayers; ++L) {
            uint32_t v[32], a[32];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                tmem_ld32(mine + 32 * h, v);
                tmem_wait_ld();
#pragma unroll
                for (int k = 0; k < 16; ++k) a[16 * h + k] = relu_bf16x2(v[2 * k], v[2 * k + 1]);
            }
            tmem_st32(mine + kFwdACol, a);
            tmem_wait_st();
            tc_fence_before();
            wg_sync(bar_id);
            tc_fence_after();
            product(L);
        }
        float z[16];
        tmem_ld16(mine, z);
        if (r >= 0)
            for (int c = 0; c < kMlpOut; ++c) out[r * stride + c] = expf(z[c]);
        r = next;
    }
    if (row == 0) {
        if (ppending) mbar_drain(mbar, pphase, err);
        if (xpending) mbar_drain(xbar, xphase, err);
    }
    tc_fence_before();
    __syncthreads();
    if ((threadIdx.x >> 5) == 0) tmem_free(*tslot, kFwdCols);
}

// Training: gradient of mean over samples and channels of (pred - t)^2 / (pred^2 + 0.01)
// (relative L2; the denominator is not differentiated) for every weight, accumulated per CTA in
// TMEM (dW_k^T = H_k^T G_k) and added to grad[] once per CTA.
// A tile of 128 rows is a chain of eleven dependent products, so the chain's latency bounds the
// kernel: TMEM holds one tile's accumulators (448 columns) and shared memory one tile's
// activations.  What is not in the chain is kept off it: a warp of its own issues the products (the
// rows' warps wait only for what they read), two warps share 32 rows, the weight gradients' products
// run behind the epilogue that follows them (two Ga buffers, no commit of their own: the next
// commit covers them), features of the next tile and targets of this one load ahead, and a layer
// costs one barrier; an epilogue works on two values at a time (conversion, ReLU, mask).  65,536
// rows (four rounds of tiles over 152 SMs), us for a step and the parameters' readback: 88.6 with 128
// threads that issued, waited and converted one by one; about 83 with the products taken off the
// chain, 76 with two values at a time, 71.1 with every weight copy in flight at once.  Four warps per 32
// rows were slower (80 against 75, timed together).
__global__ __launch_bounds__(kTrainThreads, 1) void k_mlp_train(const uint16_t* __restrict__ w16,
                                                                const uint16_t* __restrict__ feat,
                                                                const float* __restrict__ target, int n,
                                                                float* __restrict__ grad, float* __restrict__ loss,
                                                                uint32_t* err) {
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* mbar = (uint64_t*)(smem + kTrainBar);
    uint32_t* tslot = (uint32_t*)(smem + kTrainBar + 16);
    const uint32_t sbase = smem_u32(smem);
    const int warp = threadIdx.x >> 5;
    const bool worker = warp < 8, issuer = threadIdx.x == kTrainThreads - 32;
    const int row = threadIdx.x & 127, c0 = 32 * ((threadIdx.x >> 7) & 1);  // a worker's row and first column
    const int ntiles = (n + 127) / 128;
    if (issuer) mbar_init(mbar, 1);
    if (warp == 0) tmem_alloc(tslot, 512);
    // the features of `tile` into X buffer b, half a row per worker
    auto fetch = [&](int tile, int b) {
        const long r = (long)tile * 128 + row;
        if (!worker || tile >= ntiles) return;
        const bool in = r < n;
        const uint16_t* src = feat + (in ? r : 0) * kMlpIn;
        for (int j = c0 ? 6 : 0, e = j + 6; j < e; ++j)
            cp_async16(sbase + kSX + 24576 * b + rc_offset(row, 8 * j, kMlpIn), src + 8 * j, in);
    };
    fetch(blockIdx.x, 0);
    load_weights(sbase, w16);
    uint32_t phase = 0, commits = 0;  // commits: the issuer's
    bool any = false, ok = true;
    // Shared-memory operands to the tensor cores, TMEM reads done; false when a wait ran out in any thread.
    auto publish = [&]() {
        fence_async_smem();
        tc_fence_before();
        ok = __syncthreads_and(ok);
        tc_fence_after();
        return ok;
    };
    auto wait = [&]() {
        ok = mbar_wait(mbar, phase, err) && ok;
        phase ^= 1u;
        __syncwarp();
        tc_fence_after();
    };
    publish();
    const uint32_t tmem = *tslot, mine = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + c0;
    auto commit = [&]() {
        umma_commit(mbar);
        ++commits;
    };
    // D = activations . W_L^T
    auto forward = [&](int L, int b) {
        if (!issuer) return;
        issue_fwd(tmem, sbase, L == 0 ? kSX + 24576 * b : kSH + (L - 1) * 16384, mlp_in(L), kSW(L), mlp_out(L), mlp_in(L));
        commit();
    };
    float loss_acc = 0.0f;
    const float inv_count = 1.0f / (3.0f * (float)n);
    int b = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, b ^= 1) {
        const long grow = (long)tile * 128 + row;
        const bool valid = grow < n;
        float t[kMlpOut] = {};
        if (worker && c0 == 0 && valid)
            for (int c = 0; c < kMlpOut; ++c) t[c] = __ldg(target + grow * 3 + c);
        uint32_t d[32], a[16];
        cp_async_wait();
        if (!publish()) break;
        forward(0, b);
        for (int L = 0; L < kMlpLayers - 1; ++L) {
            if (worker) {
                wait();
                // the tile before has now left its X buffer and everything else to this one
                if (L == 0) fetch(tile + gridDim.x, b ^ 1);
                tmem_ld32(mine, d);
                tmem_wait_ld();
#pragma unroll
                for (int k = 0; k < 16; ++k) a[k] = relu_bf16x2(d[2 * k], d[2 * k + 1]);
                rc_store_row<4>(smem + kSH + L * 16384, row, 64, c0, a);
            }
            if (!publish()) break;
            forward(L + 1, b);
        }
        if (!ok) break;
        if (worker) {
            wait();
            if (c0 == 0) {  // output gradient
                float z[16], g[kMlpOut] = {};
                tmem_ld16(mine, z);
                if (valid) {
                    for (int c = 0; c < kMlpOut; ++c) {
                        const float pred = expf(z[c]);
                        const float dif = pred - t[c], den = pred * pred + 0.01f;
                        loss_acc += dif * dif / den;
                        g[c] = 2.0f * dif / den * pred * inv_count;  // d/dz through exp
                    }
                }
                a[0] = pack_bf16x2(g[0], g[1]);
                a[1] = pack_bf16x2(g[2], 0.0f);
#pragma unroll
                for (int k = 2; k < 8; ++k) a[k] = 0u;
                rc_store_row<2>(smem + kSGz, row, 16, 0, a);
            }
        }
        if (!publish()) break;
        // layer 5: G_h5 = Gz . W5 ; dW5^T += H5^T . Gz
        if (issuer) {
            umma_bf16(tmem, umma_desc(sbase + kSGz, 128, 16 * 16), umma_desc(sbase + kSW(5), 16 * 64, 128),
                      umma_idesc_bf16(128, 64, false, true), false);
            commit();
            const uint32_t h5 = kSH + 4 * 16384;
            for (int s = 0; s < 8; ++s)
                umma_bf16(tmem + kDwCol(5), umma_desc(sbase + h5 + s * 2 * 16 * 64, 16 * 64, 128),
                          umma_desc(sbase + kSGz + s * 2 * 16 * 16, 16 * 16, 128), umma_idesc_bf16(128, 16, true, true),
                          any || s != 0);
        }
        for (int L = 4; L >= 0; --L) {
            // D holds G_h(L+1) for the activations feeding W_(L+1); mask with H(L+1) > 0
            const uint32_t ga = kSGa + (L & 1) * 16384;
            if (worker) {
                rc_load_row<4>(smem + kSH + L * 16384, row, 64, c0, a);  // H(L+1)
#pragma unroll
                for (int k = 0; k < 16; ++k) a[k] = positive_bf16x2(a[k]);
                wait();
                tmem_ld32(mine, d);
                tmem_wait_ld();
#pragma unroll
                for (int k = 0; k < 16; ++k) a[k] &= pack_bf16x2(__uint_as_float(d[2 * k]), __uint_as_float(d[2 * k + 1]));
                rc_store_row<4>(smem + ga, row, 64, c0, a);
            }
            if (!publish()) break;
            if (issuer) {
                const uint32_t a_in = L == 0 ? kSX + 24576 * b : kSH + (L - 1) * 16384;  // input of W_L
                const int cin = mlp_in(L);
                if (L > 0) {  // G_h(L) = Ga . W_L (W_L [64 out x 64 in] as MN-major B)
                    for (int s = 0; s < 4; ++s)
                        umma_bf16(tmem, umma_desc(sbase + ga + s * 256, 128, 16 * 64),
                                  umma_desc(sbase + kSW(L) + s * 2 * 16 * cin, 16 * cin, 128),
                                  umma_idesc_bf16(128, cin, false, true), s > 0);
                    commit();
                }
                for (int s = 0; s < 8; ++s)  // dW_L^T += A_in^T . Ga
                    umma_bf16(tmem + kDwCol(L), umma_desc(sbase + a_in + s * 2 * 16 * cin, 16 * cin, 128),
                              umma_desc(sbase + ga + s * 2 * 16 * 64, 16 * 64, 128), umma_idesc_bf16(128, 64, true, true),
                              any || s != 0);
            }
        }
        if (!ok) break;
        any = true;
    }
    cp_async_wait();
    if (ok && any) {  // the last tile's dW_0
        if (issuer) commit();
        if (worker) wait();
    }
    ok = __syncthreads_and(ok);
    if (!ok && issuer && commits > 0) {
        // a wait ran out: let what is in flight end, the weight gradients behind the last commit too
        mbar_drain(mbar, (commits - 1u) & 1u, err);
        commit();
        mbar_drain(mbar, (commits - 1u) & 1u, err);
    }
    // flush the accumulated weight gradients (rows = input features, columns = outputs), every CTA
    // from another layer on
    if (any && ok && worker) {
        for (int i = 0; i < kMlpLayers; ++i) {
            const int L = (i + (int)blockIdx.x) % kMlpLayers, in = mlp_in(L);
            float* dst = grad + mlp_offset(L) + row;
            if (L == 5) {
                if (c0 == 0) {
                    float v[16];
                    tmem_ld16(mine + kDwCol(5), v);
                    if (row < in)
                        for (int o = 0; o < kMlpOut; ++o) atomicAdd(dst + o * in, v[o]);
                }
            } else {
                uint32_t v[32];
                tmem_ld32(mine + kDwCol(L), v);
                tmem_wait_ld();
                if (row < in) {
#pragma unroll
                    for (int o = 0; o < 32; ++o) atomicAdd(dst + (c0 + o) * in, __uint_as_float(v[o]));
                }
            }
        }
    }
    float tot = loss_acc;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(~0u, tot, o);
    if ((threadIdx.x & 31) == 0 && tot != 0.0f) atomicAdd(loss, tot / (3.0f * (float)n));
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 512);
}

__global__ void k_adam(float* __restrict__ w, float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       uint16_t* __restrict__ w16, float* __restrict__ e32, uint16_t* __restrict__ e16, int n, float lr,
                       float b1, float b2, float c1, float c2, float eps, float ema) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi, vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    w16[i] = __bfloat16_as_ushort(__float2bfloat16_rn(wi));
    const float ei = ema > 0.0f ? ema * e32[i] + (1.0f - ema) * wi : wi;
    e32[i] = ei;
    e16[i] = __bfloat16_as_ushort(__float2bfloat16_rn(ei));
    g[i] = 0.0f;
}

__global__ void k_to_bf16(const float* __restrict__ w, uint16_t* __restrict__ w16, float* __restrict__ e32,
                          uint16_t* __restrict__ e16, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint16_t b = __bfloat16_as_ushort(__float2bfloat16_rn(w[i]));
    w16[i] = b;
    e32[i] = w[i];
    e16[i] = b;
}

// Check of the bounded mbarrier wait itself: an mbarrier expecting one arrival that never comes.
__global__ void k_debug_mbar_timeout(uint32_t* err) {
    __shared__ __align__(8) uint64_t mbar;
    if (threadIdx.x == 0) mbar_init(&mbar, 1);
    __syncthreads();
    (void)mbar_wait(&mbar, 0, err);
}

}  // namespace

#define TRY(call)                                                                       \
    do {                                                                                \
        cudaError_t e_ = (call);                                                        \
        if (e_ != cudaSuccess) return std::string(#call ": ") + cudaGetErrorString(e_); \
    } while (0)

std::string umma_probe(int mode, int swap, const uint16_t* a, const uint16_t* b, float* d, uint32_t* d_err,
                       cudaStream_t s) {
    if (mode < 0 || mode > 2) return "umma_probe: mode must be 0, 1 or 2";
    const size_t na = 128 * (mode == 2 ? 96 : 64), nb = mode == 2 ? 128 * 64 : 64 * (mode == 1 ? 96 : 64);
    const size_t nd = 128 * (mode == 1 ? 96 : 64);
    void *da = nullptr, *db = nullptr, *dd = nullptr;
    std::string e;
    auto fail = [&](const std::string& m) {
        dev_free(da);
        dev_free(db);
        dev_free(dd);
        return m;
    };
    if (dev_alloc(&da, 2 * na) != cudaSuccess || dev_alloc(&db, 2 * nb) != cudaSuccess ||
        dev_alloc(&dd, 4 * nd) != cudaSuccess)
        return fail("umma_probe: allocation failed");
    cudaError_t c = cudaMemcpyAsync(da, a, 2 * na, cudaMemcpyHostToDevice, s);
    if (c == cudaSuccess) c = cudaMemcpyAsync(db, b, 2 * nb, cudaMemcpyHostToDevice, s);
    if (c == cudaSuccess) c = cudaFuncSetAttribute(k_umma_probe, cudaFuncAttributeMaxDynamicSharedMemorySize, kProbeSmem);
    if (c != cudaSuccess) return fail(std::string("umma_probe: ") + cudaGetErrorString(c));
    k_umma_probe<<<1, 128, kProbeSmem, s>>>((const uint16_t*)da, (const uint16_t*)db, (float*)dd, mode, swap, d_err);
    c = cudaGetLastError();
    if (c == cudaSuccess) c = cudaMemcpyAsync(d, dd, 4 * nd, cudaMemcpyDeviceToHost, s);
    if (c == cudaSuccess) c = cudaStreamSynchronize(s);
    if (c != cudaSuccess) return fail(std::string("umma_probe: ") + cudaGetErrorString(c));
    return fail("");
}


void Mlp::release() {
    for (void* p : {(void*)w32_, (void*)grad_, (void*)m_, (void*)v_, (void*)w16_, (void*)e32_, (void*)e16_, (void*)loss_}) dev_free(p);
    w32_ = grad_ = m_ = v_ = e32_ = loss_ = nullptr;
    w16_ = e16_ = nullptr;
    allocated_ = false;
}

Mlp::~Mlp() { release(); }

std::string Mlp::init(uint32_t seed, cudaStream_t s) {
    if (!allocated_) {
        release();  // what an init that failed part way has left
        TRY(dev_alloc((void**)&w32_, 4 * kMlpParams));
        TRY(dev_alloc((void**)&grad_, 4 * kMlpParams));
        TRY(dev_alloc((void**)&m_, 4 * kMlpParams));
        TRY(dev_alloc((void**)&v_, 4 * kMlpParams));
        TRY(dev_alloc((void**)&w16_, 2 * kMlpParams));
        TRY(dev_alloc((void**)&e32_, 4 * kMlpParams));
        TRY(dev_alloc((void**)&e16_, 2 * kMlpParams));
        TRY(dev_alloc((void**)&loss_, 4));
        int dev = 0, sms = 0;
        TRY(cudaGetDevice(&dev));
        TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        TRY(cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrainSmem));
        TRY(cudaFuncSetAttribute(k_mlp_forward<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem));
        TRY(cudaFuncSetAttribute(k_mlp_forward<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem));
        blocks_train_ = sms;
        blocks_fwd_ = sms;  // one CTA of kFwdGroups tiles per SM
        allocated_ = true;
    }
    // He-uniform weights, xorshift32 stream from the seed; W5 rows 3..15 zero
    std::vector<float> w(kMlpParams, 0.0f);
    uint32_t x = seed ? seed : 0x9e3779b9u;
    for (int L = 0; L < kMlpLayers; ++L) {
        const int in = mlp_in(L), out = L == 5 ? kMlpOut : mlp_out(L);
        const float a = std::sqrt(6.0f / in) * (L == 5 ? 0.1f : 1.0f);
        for (int o = 0; o < out; ++o)
            for (int i = 0; i < in; ++i) {
                x ^= x << 13;
                x ^= x >> 17;
                x ^= x << 5;
                w[mlp_offset(L) + o * in + i] = a * (2.0f * ((x >> 8) * (1.0f / 16777216.0f)) - 1.0f);
            }
    }
    steps = 0;
    return set_params(w.data(), s);
}

std::string Mlp::sync_bf16(cudaStream_t s) {
    k_to_bf16<<<(kMlpParams + 255) / 256, 256, 0, s>>>(w32_, w16_, e32_, e16_, kMlpParams);
    TRY(cudaGetLastError());
    return "";
}

std::string Mlp::set_params(const float* host, cudaStream_t s) {
    if (!allocated_) return "MLP not initialised";
    TRY(cudaMemcpyAsync(w32_, host, 4 * kMlpParams, cudaMemcpyHostToDevice, s));
    TRY(cudaMemsetAsync(grad_, 0, 4 * kMlpParams, s));
    TRY(cudaMemsetAsync(m_, 0, 4 * kMlpParams, s));
    TRY(cudaMemsetAsync(v_, 0, 4 * kMlpParams, s));
    steps = 0;
    const std::string e = sync_bf16(s);
    if (!e.empty()) return e;
    TRY(cudaStreamSynchronize(s));
    return "";
}

std::string Mlp::get_params(float* host, cudaStream_t s) {
    if (!allocated_) return "MLP not initialised";
    TRY(cudaMemcpyAsync(host, w32_, 4 * kMlpParams, cudaMemcpyDeviceToHost, s));
    TRY(cudaStreamSynchronize(s));
    return "";
}

std::string Mlp::get_grad(float* host, cudaStream_t s) {
    if (!allocated_) return "MLP not initialised";
    TRY(cudaMemcpyAsync(host, grad_, 4 * kMlpParams, cudaMemcpyDeviceToHost, s));
    TRY(cudaStreamSynchronize(s));
    return "";
}

namespace {
// A tensor map of n feature rows in boxes of 128 rows x `cols` columns (false: none could be made,
// and the kernel copies the rows itself).
bool feature_map(const uint16_t* d_feat, int n, int cols, CUtensorMapSwizzle swizzle, CUtensorMap* map) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<Encode>(f);
    }();
    if (!encode) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)kMlpIn, (cuuint64_t)n}, strides[1] = {2 * (cuuint64_t)kMlpIn};
    const cuuint32_t box[2] = {(cuuint32_t)cols, 128}, one[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t*>(d_feat), dims, strides, box, one,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

std::string Mlp::forward(const uint16_t* d_feat, int n, float* d_out, uint32_t* d_err, cudaStream_t s,
                         const int32_t* d_rows, int out_stride, const uint32_t* d_n) {
    if (!allocated_) return "MLP not initialised";
    if (n <= 0) return "";
    const int tiles = (n + 127) / 128;
    // features in row order come through tensor maps of this call's buffer (96 columns as 64 + 32)
    CUtensorMap map_a{}, map_b{};
    const bool map = !d_rows && feature_map(d_feat, n, 64, CU_TENSOR_MAP_SWIZZLE_128B, &map_a) &&
                     feature_map(d_feat, n, 32, CU_TENSOR_MAP_SWIZZLE_64B, &map_b);
    auto k = map ? k_mlp_forward<true> : k_mlp_forward<false>;
    k<<<std::min(tiles, blocks_fwd_), 128 * kFwdGroups, kFwdSmem, s>>>(e16_, d_feat, d_rows, n, d_n, d_out, out_stride, d_err,
                                                                      map_a, map_b);
    TRY(cudaGetLastError());
    return "";
}

std::string Mlp::train_step(const uint16_t* d_feat, const float* d_target, int n, float lr, float* d_loss,
                            uint32_t* d_err, cudaStream_t s) {
    if (!allocated_) return "MLP not initialised";
    if (n <= 0) return "";
    TRY(cudaMemsetAsync(grad_, 0, 4 * kMlpParams, s));
    TRY(cudaMemsetAsync(d_loss, 0, 4, s));
    const int tiles = (n + 127) / 128;
    k_mlp_train<<<std::min(tiles, blocks_train_), kTrainThreads, kTrainSmem, s>>>(w16_, d_feat, d_target, n, grad_, d_loss, d_err);
    TRY(cudaGetLastError());
    return lr > 0 ? adam(lr, s) : std::string();
}

std::string Mlp::adam(float lr, cudaStream_t s) {
    if (!allocated_) return "MLP not initialised";
    ++steps;
    const float b1 = 0.9f, b2 = 0.99f;
    const float c1 = 1.0f - std::pow(b1, (float)steps), c2 = 1.0f - std::pow(b2, (float)steps);
    k_adam<<<(kMlpParams + 255) / 256, 256, 0, s>>>(w32_, grad_, m_, v_, w16_, e32_, e16_, kMlpParams, lr, b1, b2, c1,
                                                     c2, 1e-8f, ema);
    TRY(cudaGetLastError());
    return "";
}

std::string mlp_set_spin_limit(int limit) {
    const int v = limit > 0 ? limit : kSpinLimit;
    TRY(cudaMemcpyToSymbol(g_mbar_spin_limit, &v, sizeof v));
    return "";
}

std::string mlp_debug_mbar_timeout(uint32_t* d_err, cudaStream_t s) {
    k_debug_mbar_timeout<<<1, 32, 0, s>>>(d_err);
    TRY(cudaGetLastError());
    TRY(cudaStreamSynchronize(s));
    return "";
}

}  // namespace lts
