// LBVH build kernels (sm_103a).  Stages and the reference code each one restates:
//   1 k_scene_bounds   per-triangle AABB + scene AABB            BVH.cuh:92-97, Triangle.cuh:48-53,
//                                                                 Geometry.cuh:647-655
//   2 k_morton         centroid -> 30-bit Morton code + ids, and the 4x256 radix histograms
//                                                                 BVH.cuh:101-116,134-137, Bound.cuh:169-175
//   3 4 x k_onesweep   stable LSD radix sort of (code, id), 8-bit digits, decoupled look-back, after
//                      k_digit_prefix above 500,000 keys (replaces thrust::stable_sort_by_key,
//                      BVH.cuh:140-146); up to 4,096 keys 1 to 3 are one block, k_small_sort
//   4 k_tree           Karras topology and bottom-up AABBs in one climb
//                                                                 BVH.cuh:173-262
//   5 k_dump           the reference's flattened order            BVH.cuh:311-329
// Output layout: one 64-byte node per interior node carrying both child boxes (see lbvh.cuh).
#include <cuda/atomic>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <mutex>
#include <string>

#include "../../include/lts_capi.h"

#include "dev_common.cuh"
#include "lbvh.cuh"

namespace lts {
namespace {

constexpr int kBlock = 256;
constexpr uint32_t kFlagAgg = 1u << 30, kFlagPrefix = 2u << 30, kCountMask = (1u << 30) - 1;

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Stage a block's run of `count` triangles (9 floats each) into shared memory with 16-byte
// loads when the run start is 16-byte aligned, scalar loads otherwise.
// Poll limit of the waits on another block's flag: kSpinLimit, unless a test shrinks it
// (lts_set_option "debug_spin_limit") to see a wait run out.
__device__ int g_spin_limit = kSpinLimit;

// One poll of a bounded wait: counts it and backs off, or, past the limit, sets
// DEV_ERR_LOOKBACK_TIMEOUT (and the build's own *gave_up) and returns false so that the caller
// gives up.
__device__ __forceinline__ bool spin_or_give_up(int& spins, uint32_t* err, uint32_t* gave_up = nullptr) {
    if (++spins > g_spin_limit) {
        atomicOr(err, DEV_ERR_LOOKBACK_TIMEOUT);
        if (gave_up) atomicOr(gave_up, 1u);
        return false;
    }
    __nanosleep(32);
    return true;
}

// Check of the bounded wait itself: one thread waits on a flag word that nothing sets.
__global__ void k_debug_wait_flag(const uint32_t* flag, uint32_t* err) {
    int spins = 0;
    while (ld_relaxed(flag) == 0u)
        if (!spin_or_give_up(spins, err)) return;
}

__device__ __forceinline__ void stage_tris(const float* __restrict__ tri, long first, int count, float* s) {
    const long f0 = first * 9;
    const int nf = count * 9;
    const float* src = tri + f0;
    if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
        const int n4 = nf >> 2;
        const float4* s4 = reinterpret_cast<const float4*>(src);
        for (int i = threadIdx.x; i < n4; i += blockDim.x) reinterpret_cast<float4*>(s)[i] = __ldg(s4 + i);
        for (int i = (n4 << 2) + threadIdx.x; i < nf; i += blockDim.x) s[i] = __ldg(src + i);
    } else {
        for (int i = threadIdx.x; i < nf; i += blockDim.x) s[i] = __ldg(src + i);
    }
}

__device__ __forceinline__ void tri_bounds(const float* t, float mn[3], float mx[3]) {
    // Triangle::worldBound: bUnion(Bounds3f(p0, p1), p2)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mn[k] = fminf(fminf(t[k], t[3 + k]), t[6 + k]);
        mx[k] = fmaxf(fmaxf(t[k], t[3 + k]), t[6 + k]);
    }
}

// Box of triangle `prim` gathered from an array of n triangles (9 floats each).  With a 16-byte
// aligned array, the 48-byte aligned window [floor16(36 prim), +48) always holds the triangle and
// lies inside the array for prim <= n - 2, so three 16-byte loads replace nine 4-byte ones (a third
// of the L1 wavefronts of a random gather); the last triangle and unaligned arrays load floats.
__device__ __forceinline__ void gather_tri_bounds(const float* __restrict__ tri, int n, bool aligned16, int prim,
                                                  float mn[3], float mx[3]) {
    float t[9];
    if (aligned16 && prim <= n - 2) {
        const long f = 9L * prim;
        const float4* w = reinterpret_cast<const float4*>(tri + (f & ~3L));
        const float4 w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2);
        const float v[12] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w, w2.x, w2.y, w2.z, w2.w};
        const int sh = (int)(f & 3L);
#pragma unroll
        for (int k = 0; k < 9; ++k) t[k] = sh == 0 ? v[k] : sh == 1 ? v[k + 1] : sh == 2 ? v[k + 2] : v[k + 3];
    } else {
#pragma unroll
        for (int k = 0; k < 9; ++k) t[k] = __ldg(tri + 9L * prim + k);
    }
    tri_bounds(t, mn, mx);
}

// ------------------------------------------------------------------ 1. scene bounds
__global__ __launch_bounds__(kBlock) void k_scene_bounds(const float* __restrict__ tri, int n,
                                                         uint32_t* __restrict__ gb) {
    __shared__ float s_tri[kBlock * 9];
    uint32_t kmn[3] = {~0u, ~0u, ~0u}, kmx[3] = {0u, 0u, 0u};
    for (long first = (long)blockIdx.x * kBlock; first < n; first += (long)gridDim.x * kBlock) {
        const int cnt = (int)min((long)kBlock, n - first);
        __syncthreads();
        stage_tris(tri, first, cnt, s_tri);
        __syncthreads();
        if (threadIdx.x < cnt) {
            float mn[3], mx[3];
            tri_bounds(s_tri + 9 * threadIdx.x, mn, mx);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                kmn[k] = min(kmn[k], float_key(mn[k]));
                kmx[k] = max(kmx[k], float_key(mx[k]));
            }
        }
    }
    // warp, then block reduction: one atomic per block and bound (same-address atomics serialise)
    __shared__ uint32_t s_red[kBlock / 32][6];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        for (int o = 16; o > 0; o >>= 1) {
            kmn[k] = min(kmn[k], __shfl_xor_sync(0xffffffffu, kmn[k], o));
            kmx[k] = max(kmx[k], __shfl_xor_sync(0xffffffffu, kmx[k], o));
        }
    }
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            s_red[threadIdx.x >> 5][k] = kmn[k];
            s_red[threadIdx.x >> 5][3 + k] = kmx[k];
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        uint32_t v = s_red[0][threadIdx.x];
        for (int w = 1; w < kBlock / 32; ++w)
            v = threadIdx.x < 3 ? min(v, s_red[w][threadIdx.x]) : max(v, s_red[w][threadIdx.x]);
        atomicMax(gb + threadIdx.x, threadIdx.x < 3 ? ~v : v);  // gb starts zeroed: minima as their complements
    }
}

// ------------------------------------------------------------------ 2. Morton codes + histograms
__device__ __forceinline__ uint32_t left_shift3(uint32_t x) {
    // BVH.cuh:101-109
    if (x == (1u << 10)) --x;
    x = (x | (x << 16)) & 0b00000011000000000000000011111111u;
    x = (x | (x << 8)) & 0b00000011000000001111000000001111u;
    x = (x | (x << 4)) & 0b00000011000011000011000011000011u;
    x = (x | (x << 2)) & 0b00001001001001001001001001001001u;
    return x;
}

__device__ __forceinline__ uint32_t morton_code(const float mn[3], const float mx[3], const float gmn[3], const float gmx[3]) {
    uint32_t q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float c = mn[k] * 0.5f + mx[k] * 0.5f;        // BVH.cuh:95
        float o = c - gmn[k];                                // Bound.cuh:169-175
        if (gmx[k] > gmn[k]) o = __fdiv_rn(o, gmx[k] - gmn[k]);
        const float s = __fmul_rn((float)(1 << 10), o);     // * mortonScale (BVH.cuh:136)
        q[k] = (uint32_t)s;                                  // float -> uint32_t truncation
    }
    return left_shift3(q[0]) | (left_shift3(q[1]) << 1) | (left_shift3(q[2]) << 2);
}

__global__ __launch_bounds__(kBlock) void k_morton(const float* __restrict__ tri, int n, const uint32_t* __restrict__ gb,
                                                   int code_limit, uint32_t* __restrict__ codes,
                                                   int32_t* __restrict__ ids, uint32_t* __restrict__ hist) {
    __shared__ float s_tri[kBlock * 9];
    __shared__ uint32_t s_hist[4 * 256];
    for (int i = threadIdx.x; i < 4 * 256; i += kBlock) s_hist[i] = 0;
    float gmn[3], gmx[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        gmn[k] = key_float(~gb[k]);
        gmx[k] = key_float(gb[3 + k]);
    }
    for (long first = (long)blockIdx.x * kBlock; first < n; first += (long)gridDim.x * kBlock) {
        const int cnt = (int)min((long)kBlock, n - first);
        __syncthreads();
        stage_tris(tri, first, cnt, s_tri);
        __syncthreads();
        if (threadIdx.x < cnt) {
            const long i = first + threadIdx.x;
            uint32_t code = 0;
            int32_t id = 0;
            if (code_limit < 0 || i < code_limit) {
                float mn[3], mx[3];
                tri_bounds(s_tri + 9 * threadIdx.x, mn, mx);
                code = morton_code(mn, mx, gmn, gmx);
                id = (int32_t)i;
            }
            codes[i] = code;
            if (ids) ids[i] = id;  // null: every id is its position, generated by the first sort pass
#pragma unroll
            for (int p = 0; p < 4; ++p) atomicAdd(&s_hist[p * 256 + ((code >> (8 * p)) & 255u)], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * 256; i += kBlock)
        if (s_hist[i]) atomicAdd(hist + i, s_hist[i]);
}

// ------------------------------------------------------------------ 3. radix sort
__device__ __forceinline__ uint32_t block_excl_scan256(uint32_t v, uint32_t* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    uint32_t wsum = 0;
    for (int w = 0; w < warp; ++w) wsum += s_warp[w];
    __syncthreads();
    return wsum + x - v;
}

#ifndef LTS_SORT_MIN_BLOCKS
#define LTS_SORT_MIN_BLOCKS 4  // resident sort tiles per SM the register budget is cut for
#endif
#ifndef LTS_SORT_BALLOT_MATCH
#define LTS_SORT_BALLOT_MATCH 1  // 0: __match_any_sync
#endif
// Lanes of the warp whose valid key has the same 8-bit digit d (only valid lanes: `valid`).  One
// ballot per digit bit: a lane keeps the lanes that agree with it on every bit.  MATCH.ANY is
// issued on the slow ADU pipe; the ballots are not.
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, bool valid) {
#if LTS_SORT_BALLOT_MATCH
    uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? m : ~m;
    }
    return valid ? peers : (1u << (threadIdx.x & 31));  // an invalid lane ranks alone (unused)
#else
    return __match_any_sync(0xffffffffu, valid ? d : 256u);
#endif
}

__global__ void k_digit_prefix(const uint32_t* __restrict__ hist, uint32_t* __restrict__ prefix) {
    __shared__ uint32_t s_warp[8];
    const uint32_t v = hist[blockIdx.x * 256 + threadIdx.x];
    prefix[blockIdx.x * 256 + threadIdx.x] = block_excl_scan256(v, s_warp);
}

// vin null: every value is its key's position (the identity ids of the first pass).  ITEMS keys per
// thread; LOOKBACK predecessor tiles read per look-back round trip.
// A look-back that runs out leaves digits counted too low: its pass writes some positions twice and
// others not at all.  The keys are then no longer the ones that were counted, and the passes after it would
// write past the arrays: every position is checked before its write.  *gave_up tells the tree.  (Asking it
// at the start of every tile instead cost 2 us a pass.)
template <int ITEMS, int LOOKBACK, bool SCAN>
__global__ __launch_bounds__(kSortThreads, LTS_SORT_MIN_BLOCKS) void k_onesweep(const uint32_t* __restrict__ kin, const int32_t* __restrict__ vin,
                                                           uint32_t* __restrict__ kout, int32_t* __restrict__ vout,
                                                           int n, int shift, const uint32_t* __restrict__ prefix,
                                                           uint32_t* __restrict__ status, uint32_t* __restrict__ tile_counter,
                                                           uint32_t* gave_up, uint32_t* __restrict__ err) {
    constexpr int kTile = kSortThreads * ITEMS;
    __shared__ uint32_t s_keys[kTile];
    __shared__ int32_t s_vals[kTile];
    __shared__ uint32_t s_whist[kSortThreads / 32][256];
    __shared__ uint32_t s_tile_start[256];
    __shared__ uint32_t s_dst[256];
    __shared__ uint32_t s_warp[8];
    __shared__ int s_tile;

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = (int)atomicAdd(tile_counter, 1u);
    for (int i = threadIdx.x; i < (kSortThreads / 32) * 256; i += kSortThreads) (&s_whist[0][0])[i] = 0;
    __syncthreads();
    const int tile = s_tile;
    const long base = (long)tile * kTile;
    const long wbase = base + (long)warp * 32 * ITEMS;

    uint32_t key[ITEMS];
    int32_t val[ITEMS];
    uint32_t rank[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const long idx = wbase + i * 32 + lane;
        if (idx < n) {
            key[i] = __ldg(kin + idx);
            val[i] = vin ? __ldg(vin + idx) : (int32_t)idx;
        } else {
            key[i] = 0;
            val[i] = 0;
        }
    }
    // the digits' first output positions: an exclusive scan of the pass' histogram, by every tile
    // (SCAN) or made before the passes
    const uint32_t gprefix = SCAN ? block_excl_scan256(__ldg(prefix + threadIdx.x), s_warp) : __ldg(prefix + threadIdx.x);
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const long idx = wbase + i * 32 + lane;
        const bool valid = idx < n;
        const uint32_t d = (key[i] >> shift) & 255u;
        const uint32_t peers = digit_peers(d, valid);
        const int leader = __ffs(peers) - 1;
        uint32_t b = 0;
        if (valid && lane == leader) {
            b = s_whist[warp][d];
            s_whist[warp][d] = b + __popc(peers);
        }
        b = __shfl_sync(0xffffffffu, b, leader);
        rank[i] = b + __popc(peers & lt);
    }
    __syncthreads();
    const uint32_t dig = threadIdx.x;
    uint32_t tot = 0;
#pragma unroll
    for (int w = 0; w < kSortThreads / 32; ++w) {
        const uint32_t c = s_whist[w][dig];
        s_whist[w][dig] = tot;
        tot += c;
    }
    uint32_t* st = status + (size_t)tile * 256;
    st_relaxed(st + dig, (tile == 0 ? kFlagPrefix : kFlagAgg) | tot);
    const uint32_t start = block_excl_scan256(tot, s_warp);
    s_tile_start[dig] = start;
    uint32_t excl = 0;
    if (tile > 0) {
        // look back LOOKBACK predecessors per round trip (each status word carries its flag and
        // count together), consumed newest first until an inclusive prefix; a predecessor that
        // has published nothing yet is re-read (bounded wait)
        int k = tile - 1, spins = 0;
        while (k >= 0) {
            uint32_t v[LOOKBACK];
#pragma unroll
            for (int j = 0; j < LOOKBACK; ++j)
                v[j] = k - j >= 0 ? ld_relaxed(status + (size_t)(k - j) * 256 + dig) : kFlagPrefix;
            int used = LOOKBACK;
            bool done = false;
#pragma unroll
            for (int j = 0; j < LOOKBACK; ++j) {
                if (done || used < LOOKBACK) continue;
                const uint32_t f = v[j] & ~kCountMask;
                if (f == 0) {
                    used = j;
                } else {
                    excl += v[j] & kCountMask;
                    done = f == kFlagPrefix;
                }
            }
            if (done) break;
            k -= used;
            if (used < LOOKBACK && !spin_or_give_up(spins, err, gave_up)) break;
        }
        st_relaxed(st + dig, kFlagPrefix | (excl + tot));
    }
    s_dst[dig] = gprefix + excl;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const long idx = wbase + i * 32 + lane;
        if (idx < n) {
            const uint32_t d = (key[i] >> shift) & 255u;
            const uint32_t pos = s_tile_start[d] + s_whist[warp][d] + rank[i];
            s_keys[pos] = key[i];
            s_vals[pos] = val[i];
        }
    }
    __syncthreads();
    const int tile_n = (int)min((long)kTile, n - base);
    for (int j = threadIdx.x; j < tile_n; j += kSortThreads) {
        const uint32_t k = s_keys[j];
        const uint32_t d = (k >> shift) & 255u;
        const uint32_t dst = s_dst[d] + (uint32_t)j - s_tile_start[d];
        if (dst < (uint32_t)n) {
            kout[dst] = k;
            vout[dst] = s_vals[j];
        }
    }
}

// ------------------------------------------------------------------ 1-3 in one block
// Scene bounds, Morton codes and the stable sort of up to kSmallSort primitives by one block: a
// bitonic sort of (code, position) words in shared memory.  For so few primitives the six
// launches, six clears and the sort tiles' latencies were all there is to the time (a build of 1,280
// triangles, launch to finish: 107 us, 4 x 8 us of it in sort passes over one tile; 38 now).
constexpr int kSmallThreads = 1024, kSmallSort = 4096;
__global__ __launch_bounds__(kSmallThreads) void k_small_sort(const float* __restrict__ tri, int n, int code_limit,
                                                              uint32_t* __restrict__ codes, int32_t* __restrict__ ids,
                                                              uint32_t* __restrict__ group_done, int ngroups) {
    __shared__ uint64_t s_key[kSmallSort];
    __shared__ uint32_t s_red[kSmallThreads / 32][6];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < ngroups; i += kSmallThreads) group_done[i] = 0u;  // the tree's counters
    uint32_t key[6] = {0u, 0u, 0u, 0u, 0u, 0u};  // complements of the minima, maxima
    for (int i = tid; i < n; i += kSmallThreads) {
        float t[9], mn[3], mx[3];
#pragma unroll
        for (int k = 0; k < 9; ++k) t[k] = __ldg(tri + 9L * i + k);
        tri_bounds(t, mn, mx);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            key[k] = max(key[k], ~float_key(mn[k]));
            key[3 + k] = max(key[3 + k], float_key(mx[k]));
        }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        key[k] = __reduce_max_sync(~0u, key[k]);
        if (lane == 0) s_red[warp][k] = key[k];
    }
    __syncthreads();
    float gmn[3], gmx[3];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const uint32_t v = __reduce_max_sync(~0u, s_red[lane][k]);
        if (k < 3) gmn[k] = key_float(~v);
        else gmx[k - 3] = key_float(v);
    }
    int p2 = 64;
    while (p2 < n) p2 <<= 1;
    for (int i = tid; i < p2; i += kSmallThreads) {
        uint64_t w = ~0ull;
        if (i < n) {
            uint32_t code = 0;
            if (code_limit < 0 || i < code_limit) {
                float t[9], mn[3], mx[3];
#pragma unroll
                for (int k = 0; k < 9; ++k) t[k] = __ldg(tri + 9L * i + k);
                tri_bounds(t, mn, mx);
                code = morton_code(mn, mx, gmn, gmx);
            }
            w = ((uint64_t)code << 32) | (uint32_t)i;
        }
        s_key[i] = w;
    }
    __syncthreads();
    // pair p of a stage of stride j joins elements e and e + j, e = 2 j (p / j) + p % j; strides up to
    // 32 stay within the 64 elements of a warp's pairs, so those stages need no block barrier
    for (int k = 2; k <= p2; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int p = tid; p < p2 / 2; p += kSmallThreads) {
                const int e = 2 * (p & ~(j - 1)) + (p & (j - 1));
                const uint64_t a = s_key[e], b = s_key[e + j];
                if ((a > b) == ((e & k) == 0)) {
                    s_key[e] = b;
                    s_key[e + j] = a;
                }
            }
            const bool next_in_warp = j > 1 ? (j >> 1) <= 32 : k <= 32;  // the next stage's stride (k itself after j = 1)
            if (j <= 32 && next_in_warp) __syncwarp();
            else __syncthreads();
        }
    __syncthreads();
    for (int i = tid; i < n; i += kSmallThreads) {
        const uint64_t w = s_key[i];
        const int pos = (int)(uint32_t)w;
        codes[i] = (uint32_t)(w >> 32);
        ids[i] = code_limit < 0 || pos < code_limit ? pos : 0;
    }
}

// ------------------------------------------------------------------ 4+5. tree: topology and refit
// delta (BVH.cuh:173-190): common-prefix length of the Morton codes at sorted positions a and b;
// for equal codes 40 + the common prefix of the positions; -1 when b lies outside [0, n).
__device__ __forceinline__ int delta_codes(uint32_t ca, uint32_t cb, int a, int b) {
    uint32_t x = ca ^ cb;
    int extra = 0;
    if (x == 0) {
        extra = 40;
        x = (uint32_t)(a ^ b);
    }
    return __clz((int)x) + extra;
}
__device__ __forceinline__ int delta(const uint32_t* __restrict__ c, int n, int a, int b) {
    if (b < 0 || b >= n) return -1;
    return delta_codes(__ldg(c + a), __ldg(c + b), a, b);
}

// The reference builds the tree in two passes: every interior node i finds its leaf range and
// split by binary searches over delta (BVH.cuh:192-236), then every leaf climbs to the root
// through parent links, the second child to arrive forming the union (BVH.cuh:238-262).  The
// result is the binary radix tree of the sorted codes: node [lo, hi] with split g has children
// [lo, g] and [g+1, hi]; an interior child sits at index g when it is a left child (its last
// position) and at g+1 when it is a right child (its first position); the root, [0, n-1], at 0.
// The same tree is built here in ONE bottom-up pass (the agglomerative order of Apetrei, "Fast
// and Simple Agglomerative LBVH Construction", 2014, with the indices above): node [L, R] is the
// left child of a parent split at R when delta(R, R+1) > delta(L-1, L) and the right child of a
// parent split at L-1 otherwise (the two deltas differ for distinct augmented keys), which also
// gives the node's own index (R or L).  Each thread climbs from one leaf; the two children of a
// parent meet at the parent's split g, the first to arrive stops, the second forms the union,
// writes the parent's whole 64-byte record (both child boxes, children, range) and climbs on:
//  * a block of kTreeBlock threads owns kTreeBlock consecutive leaves; when g and g+1 both lie in
//    the block the children meet in a shared-memory slot of g (box, child reference, far range
//    end; a block-scope fence and a shared arrival bitmask), without barriers;
//  * what is left of the block is its forest, the subtrees whose parents reach into another block:
//    at most kForestCap - 1 of them (each side's deltas rise strictly outwards, and a delta takes
//    54 values: 2..31 for distinct codes, 40 + 8..31 for equal ones), consecutive and covering the
//    block.  The block writes them, in order, to device memory (a count beyond the capacity, which
//    sorted codes cannot give, is cut and reported); the last block of a group of
//    kTreeGroup to finish takes the group's forests as its items (subtrees instead of leaves) and
//    climbs again, the last group of a group of groups likewise, up to the root.  No block waits:
//    the others of a group just end.  (The ancestors of the block edges used to meet in a second
//    kernel through arrival words in device memory, one dependent chain of exchanges per edge:
//    24 us for 1,280 triangles, 47 for 200,000, 94 for 16M.)
// Leaves (threads) per block: 512, or 256 above kTreeLarge leaves, where shorter longest climbs beat
// the levels of merging they add (16M, sorted: 0.96 ms against 1.04; 1M: 0.097 against 0.094; the line lies
// between the two, its crossing is not measured).
constexpr int kTreeLarge = 4000000;
__host__ __device__ constexpr int tree_block(long n) { return n > kTreeLarge ? 256 : 512; }
// Forests merged by one block.  Random triangles leave 9.3 subtrees a block of 512 at the first level, 223 items
// for the 512 threads, and longer forests above it; codes that close in on a block's edges leave up to 26, which
// the merge then takes in chunks.
constexpr int kTreeGroup = 24;
constexpr int kForestCap = 128;  // entries of 32 bytes per block: up to 127 subtrees, the last word their count

// One subtree of a forest: box, reference, last leaf (it begins after its predecessor's).
struct alignas(16) ForestEntry {
    float4 a;  // min.xyz, max.x
    float4 b;  // max.yz, reference bits, last leaf bits
};
constexpr long tree_blocks(long n, int block) { return (n + block - 1) / block; }
constexpr size_t forest_bytes(long n, int block) { return (size_t)tree_blocks(n, block) * kForestCap * sizeof(ForestEntry); }
// Completion counters: one per group of every level.
constexpr long tree_counters(long n, int block) {
    long c = 0;
    for (long m = tree_blocks(n, block); m > 1; m = (m + kTreeGroup - 1) / kTreeGroup) c += (m + kTreeGroup - 1) / kTreeGroup;
    return c;
}

__device__ __forceinline__ void put_root(float* __restrict__ root_bounds, const float* mn, const float* mx) {
    for (int k = 0; k < 3; ++k) {
        root_bounds[k] = mn[k];
        root_bounds[3 + k] = mx[k];
    }
}

// Slot k of the boundary between items k and k + 1 holds what the record of the node split there
// needs: both child boxes, both child references, the far items of the node's range and, once
// both children arrived, the node's index.  The climbs touch only shared memory (so the
// block-scope fences wait on nothing in flight to device memory); the records go out after the
// block's barrier, one 64-byte line per thread.
//   slot[k][2 side + 0] = (min.x, min.y, min.z, max.x)      side 0: left child, 1: right
//   slot[k][2 side + 1] = (max.y, max.z, reference, far item)
//   slot[k][4]          = (node index, arrival bits: 1 left, 2 right, -, -)
// Five 16-byte words per slot put eight consecutive slots in distinct bank groups.
template <int kTreeBlock>
struct TreeShared {
    float4 slot[kTreeBlock][5];
    int delta[kTreeBlock + 1];    // delta across the boundary before item k (-1 outside the array)
    int pos[kTreeBlock + 1];      // first leaf of item k (item count: one past the last leaf)
    int root[kTreeBlock];         // forest: 0, or where the subtree beginning at item k is: slot * 2 + side + 1,
                                  // or -1 / -2: edge[0] / edge[1]
    float4 edge[2][2];            // the subtrees whose parent lies beyond the first / last boundary
    int warp[kTreeBlock / 32];
    int list[kTreeGroup + 1];     // a group's forests: entries before forest j
    int last;
};

// The climb over the block's `cnt` items (thread i < cnt holds item i: reference, box), the node
// records, and the forest into `out` (entries in order, then their count; the whole tree gives 0).
// Every thread of the block calls it.
template <int kTreeBlock>
__device__ void tree_climb(TreeShared<kTreeBlock>& sh, int cnt, int n, int ref, float* mn, float* mx, BvhNode* __restrict__ nodes,
                           float* __restrict__ root_bounds, ForestEntry* __restrict__ out, uint32_t* err) {
    const int i = threadIdx.x;
    auto have_of = [&](int slot) -> uint32_t* { return reinterpret_cast<uint32_t*>(&sh.slot[slot][4]) + 1; };
    sh.slot[i][4] = make_float4(0.f, 0.f, 0.f, 0.f);
    sh.root[i] = 0;
    __syncthreads();
    if (i < cnt) {
        int li = i, ri = i;
        for (;;) {
            const bool left = sh.delta[ri + 1] > sh.delta[li];
            const int bound = left ? ri + 1 : li;  // the boundary its parent is split at
            if (bound == 0 || bound == cnt) {      // the parent reaches out of the block
                const int e = bound == 0 ? 0 : 1;
                sh.edge[e][0] = make_float4(mn[0], mn[1], mn[2], mx[0]);
                sh.edge[e][1] = make_float4(mx[1], mx[2], __int_as_float(ref), __int_as_float(sh.pos[ri + 1] - 1));
                sh.root[li] = -1 - e;
                break;
            }
            const int side = left ? 0 : 1, slot = bound - 1;
            sh.slot[slot][2 * side] = make_float4(mn[0], mn[1], mn[2], mx[0]);
            sh.slot[slot][2 * side + 1] = make_float4(mx[1], mx[2], __int_as_float(ref), __int_as_float(left ? li : ri));
            __threadfence_block();
            if (!(atomicOr(have_of(slot), 1u << side) & (2u >> side))) break;  // first arrival stops
            __threadfence_block();
            const float4 e0 = sh.slot[slot][2 * (side ^ 1)], e1 = sh.slot[slot][2 * (side ^ 1) + 1];
            const float smn[3] = {e0.x, e0.y, e0.z}, smx[3] = {e0.w, e1.x, e1.y};
#pragma unroll
            for (int k = 0; k < 3; ++k) {  // bUnion(left, right), operands in that order
                mn[k] = left ? fminf(mn[k], smn[k]) : fminf(smn[k], mn[k]);
                mx[k] = left ? fmaxf(mx[k], smx[k]) : fmaxf(smx[k], mx[k]);
            }
            if (left) ri = __float_as_int(e1.w);
            else li = __float_as_int(e1.w);
            const int L = sh.pos[li], R = sh.pos[ri + 1] - 1;
            int* idx = reinterpret_cast<int*>(&sh.slot[slot][4]);
            if (L == 0 && R == n - 1) {
                *idx = 0;
                put_root(root_bounds, mn, mx);
                break;
            }
            ref = sh.delta[ri + 1] > sh.delta[li] ? R : L;
            *idx = ref;
        }
    }
    __syncthreads();
    if (i + 1 < cnt) {
        const float4 w = sh.slot[i][4];
        const uint32_t have = __float_as_uint(w.y);
        if (have == 3u) {  // the record of the node formed here
            const float4 a0 = sh.slot[i][0], a1 = sh.slot[i][1], c0 = sh.slot[i][2], c1 = sh.slot[i][3];
            float4* P = reinterpret_cast<float4*>(nodes + __float_as_int(w.x));
            P[0] = a0;
            P[1] = make_float4(a1.x, a1.y, c0.x, c0.y);
            P[2] = make_float4(c0.z, c0.w, c1.x, c1.y);
            reinterpret_cast<int4*>(P)[3] = make_int4(__float_as_int(a1.z), __float_as_int(c1.z), sh.pos[__float_as_int(a1.w)],
                                                      sh.pos[__float_as_int(c1.w) + 1] - 1);  // (left ref, right ref, lo, hi)
        } else if (have == 1u) {  // a left child alone: its sibling reaches out of the block
            sh.root[__float_as_int(sh.slot[i][1].w)] = 2 * i + 1;
        } else if (have == 2u) {  // a right child alone
            sh.root[i + 1] = 2 * i + 2;
        }
    }
    __syncthreads();
    const int r = i < cnt ? sh.root[i] : 0, lane = i & 31, warp = i >> 5;
    const unsigned m = __ballot_sync(~0u, r != 0);
    if (lane == 0) sh.warp[warp] = __popc(m);
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < kTreeBlock / 32; ++w) {
        const int c = sh.warp[w];
        before += w < warp ? c : 0;
        total += c;
    }
    if (r != 0) {
        const int at = before + __popc(m & ((1u << lane) - 1u));
        float4 a, b;
        if (r < 0) {
            a = sh.edge[-1 - r][0];
            b = sh.edge[-1 - r][1];
        } else {  // a lone child: its far item becomes its last leaf
            const int slot = (r - 1) >> 1, side = (r - 1) & 1;
            a = sh.slot[slot][2 * side];
            b = sh.slot[slot][2 * side + 1];
            b.w = __int_as_float(sh.pos[(side == 0 ? slot : __float_as_int(b.w)) + 1] - 1);
        }
        if (at < kForestCap - 1) {
            out[at].a = a;
            out[at].b = b;
        }
    }
    if (i == 0) {
        if (total > kForestCap - 1) atomicOr(err, DEV_ERR_CAPACITY);
        out[kForestCap - 1].a.x = __int_as_float(min(total, kForestCap - 1));
    }
    __syncthreads();
}

template <int kTreeBlock>
__global__ __launch_bounds__(kTreeBlock, 2048 / kTreeBlock) void k_tree(const float* __restrict__ tri, int n, int mode,
                                                     const int32_t* __restrict__ ids, const uint32_t* __restrict__ codes,
                                                     BvhNode* __restrict__ nodes, ForestEntry* __restrict__ forest,
                                                     uint32_t* __restrict__ group_done, int32_t* __restrict__ leaf_prim,
                                                     float* __restrict__ root_bounds, const uint32_t* __restrict__ gave_up,
                                                     uint32_t* err) {
    __shared__ TreeShared<kTreeBlock> sh;
    const int b0 = blockIdx.x * kTreeBlock, cnt = min(kTreeBlock, n - b0);
    const int i = threadIdx.x, l = b0 + i;
    // deltas across the block's boundaries b0 .. b0 + cnt, each thread's from its own two codes
    if (i <= cnt) {
        sh.delta[i] = l == 0 || l >= n ? -1 : delta_codes(__ldg(codes + l - 1), __ldg(codes + l), l - 1, l);
        sh.pos[i] = l;
    }
    if (i == 0 && cnt == kTreeBlock) {
        sh.delta[cnt] = delta(codes, n, b0 + cnt - 1, b0 + cnt);
        sh.pos[cnt] = b0 + cnt;
    }
    float mn[3], mx[3];
    if (i < cnt) {
        // (an id outside the triangles comes from a sort that gave up, below)
        const int prim = (mode == BVH_MODE_REFERENCE) ? l : (int)min((uint32_t)__ldg(ids + l), (uint32_t)(n - 1));
        leaf_prim[l] = prim;
        gather_tri_bounds(tri, n, (reinterpret_cast<uintptr_t>(tri) & 15u) == 0, prim, mn, mx);
        if (n == 1) put_root(root_bounds, mn, mx);
    }
    if (n == 1) return;
    long first = blockIdx.x;  // the first block of the forest this block has written
    tree_climb(sh, cnt, n, ~l, mn, mx, nodes, root_bounds, forest + first * kForestCap, err);
    long span = 1;            // blocks per forest of this level
    for (long count = gridDim.x; count > 1;) {
        // publish the forest; the last of its group goes on with the group's
        const long groups = (count + kTreeGroup - 1) / kTreeGroup, group = first / span / kTreeGroup;
        const int nlists0 = (int)min((long)kTreeGroup, count - group * kTreeGroup);
        if (i == 0) {
            __threadfence();
            const bool last = (int)atomicAdd(group_done + group, 1u) == nlists0 - 1;
            // The sort gave up: there is no tree.  A block's own climb stays within its items whatever their
            // codes are (a subtree grows with every step, and its far ends are items), but what it left is
            // no forest to go on with.
            sh.last = last && !(gave_up && __ldg(gave_up));
            __threadfence();
        }
        __syncthreads();
        if (!sh.last) return;
        group_done += groups;
        first = group * kTreeGroup * span;
        // the group's subtrees as items, kTreeBlock at a time; the forests of several chunks (more
        // subtrees than threads) are written over the lists read before, and merged again
        int nlists = nlists0;
        long step = span;
        for (;;) {
            if (i < nlists) sh.list[i + 1] = __float_as_int(__ldcg(&forest[(first + i * step) * kForestCap + kForestCap - 1].a.x));
            __syncthreads();
            if (i == 0) {
                sh.list[0] = 0;
                for (int j = 0; j < nlists; ++j) sh.list[j + 1] += sh.list[j];
            }
            __syncthreads();
            const int total = sh.list[nlists], chunks = (total + kTreeBlock - 1) / kTreeBlock;
            for (int c = 0; c < chunks; ++c) {
                const int c0 = c * kTreeBlock, m = min(kTreeBlock, total - c0);
                auto entry = [&](int k) -> const ForestEntry* {
                    int j = 0;
                    while (k >= sh.list[j + 1]) ++j;
                    return forest + (first + j * step) * kForestCap + (k - sh.list[j]);
                };
                int ref = 0;
                if (i < m) {
                    const ForestEntry* e = entry(c0 + i);
                    const float4 a = __ldcg(&e->a), b = __ldcg(&e->b);
                    mn[0] = a.x; mn[1] = a.y; mn[2] = a.z;
                    mx[0] = a.w; mx[1] = b.x; mx[2] = b.y;
                    ref = __float_as_int(b.z);
                    const int end = __float_as_int(b.w) + 1;
                    sh.pos[i + 1] = end;
                    sh.delta[i + 1] = end >= n ? -1 : delta_codes(__ldg(codes + end - 1), __ldg(codes + end), end - 1, end);
                }
                if (i == 0) {
                    const int p = c0 == 0 ? (int)(first * kTreeBlock) : __float_as_int(__ldcg(&entry(c0 - 1)->b).w) + 1;
                    sh.pos[0] = p;
                    sh.delta[0] = p == 0 ? -1 : delta_codes(__ldg(codes + p - 1), __ldg(codes + p), p - 1, p);
                }
                __syncthreads();
                // chunk c's forest over list c: at most 127 entries a list, so the chunks up to c
                // have read every list up to c
                tree_climb(sh, m, n, ref, mn, mx, nodes, root_bounds, forest + (first + c * step) * kForestCap, err);
            }
            if (chunks <= 1) break;
            nlists = chunks;
            __threadfence_block();
            __syncthreads();
        }
        span *= kTreeGroup;
        count = groups;
    }
}

inline int grid_for(long items, int per_block) { return (int)((items + per_block - 1) / per_block); }

// The build in the reference's flattened order (BVH.cuh:311-329: interior 0 .. n - 2, leaves
// n - 1 .. 2n - 2): each interior node writes its children's indices and, at their indices, their
// boxes.
__global__ __launch_bounds__(kBlock) void k_dump(const BvhNode* __restrict__ nodes, int n, const float* __restrict__ root_bounds,
                                                 int32_t* __restrict__ left, int32_t* __restrict__ right,
                                                 float* __restrict__ bounds) {
    const long i = (long)blockIdx.x * kBlock + threadIdx.x;
    if (i < n) left[n - 1 + i] = right[n - 1 + i] = -1;
    if (i < 6) bounds[i] = root_bounds[i];
    if (i >= n - 1) return;
    const float4 a = nodes[i].a, b = nodes[i].b, c = nodes[i].c;
    const int4 d = nodes[i].d;
    const int lc = d.x < 0 ? n - 1 + ~d.x : d.x, rc = d.y < 0 ? n - 1 + ~d.y : d.y;
    left[i] = lc;
    right[i] = rc;
    float2* const lb = reinterpret_cast<float2*>(bounds + 6 * (size_t)lc);
    float2* const rb = reinterpret_cast<float2*>(bounds + 6 * (size_t)rc);
    lb[0] = make_float2(a.x, a.y);
    lb[1] = make_float2(a.z, a.w);
    lb[2] = make_float2(b.x, b.y);
    rb[0] = make_float2(b.z, b.w);
    rb[1] = make_float2(c.x, c.y);
    rb[2] = make_float2(c.z, c.w);
}

// Sort tiles: kSortItems keys per thread once the tiles fill the SMs' resident blocks; smaller tiles
// below that, whose passes are a tile's latency (a chain of ranking steps) and the look-back over
// all tiles at once (400,000 keys, ms of the four passes: 15 keys and 4 tiles a round trip 0.055, 4
// and 16 0.059, 8 and 16 0.051, 8 and 32 0.066, 10 and 16 0.051; at 700,000 15 keys are faster;
// the line lies between the two, its crossing is not measured).
constexpr int kSortSmallMax = 500000, kSortSmallItems = 8, kSortSmallLookback = 16, kSortLookback = 4;
// Triangles per thread of the two streaming kernels before every SM has its eight blocks: each block
// ends with atomics on the same words (400,000 triangles: Morton codes 12.2 us, 18.4 at one).
constexpr int kStreamItems = 4;
constexpr long sort_tile(long n) { return kSortThreads * (n <= kSortSmallMax ? kSortSmallItems : kSortItems); }
constexpr long sort_tiles(long n) { return (n + sort_tile(n) - 1) / sort_tile(n); }

// The words every build starts from zero, in one buffer: scene box (8), sort tile counters (4),
// whether the sort gave up (4), histograms (4 x 256), the tree's group counters, then the sort's
// look-back table.
constexpr size_t kZeroGaveUp = 12, kZeroHist = 16, kZeroGroups = kZeroHist + 4 * 256;
constexpr size_t zero_status(long n) { return kZeroGroups + ((size_t)tree_counters(n, tree_block(n)) + 7) / 8 * 8; }
constexpr size_t zero_words(long n) { return zero_status(n) + 4 * 256 * (size_t)sort_tiles(n); }

// The build's launches, shared by Lbvh and the allocation-free entry point.  kalt / valt: the sort's
// second key and value buffers; `zero`: zero_words(n) words; `block`: leaves per block of the tree,
// tree_block(n) or 512; `forest`: forest_bytes(n, block).  mark(k) is called before stage k (bounds, Morton
// codes, sort, clear, tree) and after the last.
template <class Mark>
cudaError_t build_launches(const float* tri, int n, int mode, int code_limit, uint32_t* codes, int32_t* ids, uint32_t* kalt,
                           int32_t* valt, uint32_t* zero, int block, ForestEntry* forest, BvhNode* nodes, int32_t* leaf_prim,
                           float* root_bounds, uint32_t* err, int sms, cudaStream_t s, int* launches, Mark mark) {
    uint32_t* const groups = zero + kZeroGroups;
    uint32_t* gave_up = nullptr;  // the one-block sort waits for nothing
    mark(0);
    if (n <= kSmallSort) {
        mark(1);
        mark(2);
        k_small_sort<<<1, kSmallThreads, 0, s>>>(tri, n, code_limit, codes, ids, groups, (int)tree_counters(n, block));
        *launches = 2;
    } else {
        cudaError_t e = cudaMemsetAsync(zero, 0, 4 * zero_words(n), s);
        if (e != cudaSuccess) return e;
        const int stream_grid = std::min(grid_for(n, kBlock * kStreamItems), sms * 8);
        k_scene_bounds<<<stream_grid, kBlock, 0, s>>>(tri, n, zero);
        mark(1);
        const bool identity = code_limit < 0 || code_limit >= n;  // every id is its position
        uint32_t* const hist = zero + kZeroHist;
        k_morton<<<stream_grid, kBlock, 0, s>>>(tri, n, zero, code_limit, codes, identity ? nullptr : ids, hist);
        mark(2);
        uint32_t* const status = zero + zero_status(n);
        const size_t tiles = (size_t)sort_tiles(n);
        gave_up = zero + kZeroGaveUp;
        if (n > kSortSmallMax) k_digit_prefix<<<4, 256, 0, s>>>(hist, hist);
        uint32_t *kin = codes, *kout = kalt;
        int32_t *vin = ids, *vout = valt;
        for (int p = 0; p < 4; ++p) {
            auto k = n <= kSortSmallMax ? k_onesweep<kSortSmallItems, kSortSmallLookback, true> : k_onesweep<kSortItems, kSortLookback, false>;
            k<<<(int)tiles, kSortThreads, 0, s>>>(kin, (p == 0 && identity) ? nullptr : vin, kout, vout, n, 8 * p, hist + 256 * p,
                                                  status + (size_t)p * 256 * tiles, zero + 8 + p, gave_up, err);
            std::swap(kin, kout);
            std::swap(vin, vout);
        }
        *launches = n > kSortSmallMax ? 8 : 7;
    }
    mark(3);
    mark(4);
    auto tree = block == 512 ? k_tree<512> : k_tree<256>;
    tree<<<(int)tree_blocks(n, block), block, 0, s>>>(tri, n, mode, ids, codes, nodes, forest, groups, leaf_prim, root_bounds,
                                                                  gave_up, err);
    mark(5);
    return cudaGetLastError();
}

}  // namespace

#define LTS_TRY(call)                                                                   \
    do {                                                                                \
        cudaError_t e_ = (call);                                                        \
        if (e_ != cudaSuccess) return std::string(#call ": ") + cudaGetErrorString(e_); \
    } while (0)

void Lbvh::release() {
    void* ptrs[] = {nodes, root_bounds, leaf_prim, codes, ids, codes_alt_, zero_};
    for (void* p : ptrs) dev_free(p);
    nodes = nullptr;
    root_bounds = nullptr;
    leaf_prim = ids = ids_alt_ = nullptr;
    codes = codes_alt_ = zero_ = nullptr;
    cap_ = 0;
    bytes_ = 0;
}

Lbvh::~Lbvh() {
    release();
    for (auto& e : ev_)
        if (e) cudaEventDestroy(e);
}

std::string Lbvh::reserve(int nn) {
    if (!ev_[0])
        for (auto& e : ev_) LTS_TRY(cudaEventCreate(&e));
    if (nn <= cap_) return "";
    release();  // if an allocation below fails, the next build starts from nothing
    const size_t N = (size_t)nn;
    auto al = [&](void** p, size_t b) -> cudaError_t {
        bytes_ += b;
        return dev_alloc(p, b);
    };
    LTS_TRY(al((void**)&nodes, sizeof(BvhNode) * (N > 1 ? N - 1 : 1)));
    LTS_TRY(al((void**)&root_bounds, 6 * sizeof(float)));
    LTS_TRY(al((void**)&leaf_prim, 4 * N));
    LTS_TRY(al((void**)&codes, 4 * N));
    LTS_TRY(al((void**)&ids, 4 * N));
    // the sort's ping-pong keys and ids, one allocation: after the sort it holds the tree's forests.  Those of
    // blocks of 256 leaves need twice what the sort does (134 MB more at 16M); where that cannot be had, the
    // tree is built by blocks of 512.
    const size_t sort_bytes = std::max(8 * N, forest_bytes(nn, 512));
    small_blocks_ = tree_block(nn) == 256;
    if (small_blocks_) {
        const cudaError_t e = al((void**)&codes_alt_, std::max(sort_bytes, forest_bytes(nn, 256)));
        if (e != cudaSuccess) {
            if (e != cudaErrorMemoryAllocation) LTS_TRY(e);
            cudaGetLastError();
            small_blocks_ = false;
            bytes_ -= std::max(sort_bytes, forest_bytes(nn, 256));
        }
    }
    if (!small_blocks_) LTS_TRY(al((void**)&codes_alt_, sort_bytes));
    ids_alt_ = reinterpret_cast<int32_t*>(codes_alt_ + N);
    // a smaller build may take smaller sort tiles, hence more of them than a larger one
    LTS_TRY(al((void**)&zero_, 4 * std::max(zero_words(nn), zero_words(std::min(nn, kSortSmallMax)))));
    cap_ = nn;
    return "";
}

std::string Lbvh::build(const float* d_tri, int nn, int md, int code_limit, cudaStream_t s, uint32_t* d_error) {
    if (nn < 1) return "LBVH needs at least one primitive";
    if (nn > (1 << 24)) return "LBVH is limited to 2^24 primitives (the reference's float index arithmetic)";
    std::string e = reserve(nn);
    if (!e.empty()) return e;
    n = nn;
    mode = md;
    launches = 0;
    ++serial;
    int dev = 0, sms = 0;
    LTS_TRY(cudaGetDevice(&dev));
    LTS_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    cudaError_t me = cudaSuccess;
    LTS_TRY(build_launches(d_tri, nn, md, code_limit, codes, ids, codes_alt_, ids_alt_, zero_,
                           small_blocks_ ? tree_block(nn) : 512,
                           reinterpret_cast<ForestEntry*>(codes_alt_), nodes, leaf_prim, root_bounds, d_error, sms, s, &launches,
                           [&](int k) {
                               const cudaError_t e = cudaEventRecord(ev_[k], s);
                               if (e != cudaSuccess) me = e;
                           }));
    LTS_TRY(me);
    return "";
}

std::string Lbvh::flatten(int32_t* d_left, int32_t* d_right, float* d_bounds, cudaStream_t s) const {
    k_dump<<<grid_for(n, kBlock), kBlock, 0, s>>>(nodes, n, root_bounds, d_left, d_right, d_bounds);
    LTS_TRY(cudaGetLastError());
    return "";
}

std::string lbvh_set_spin_limit(int limit) {
    const int v = limit > 0 ? limit : kSpinLimit;
    LTS_TRY(cudaMemcpyToSymbol(g_spin_limit, &v, sizeof v));
    return "";
}

std::string lbvh_debug_wait_flag(uint32_t* d_err, cudaStream_t s) {
    uint32_t* flag = nullptr;
    LTS_TRY(dev_alloc((void**)&flag, 4));
    cudaError_t e = cudaMemsetAsync(flag, 0, 4, s);
    if (e == cudaSuccess) {
        k_debug_wait_flag<<<1, 1, 0, s>>>(flag, d_err);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    dev_free(flag);
    return e == cudaSuccess ? std::string() : std::string("debug wait: ") + cudaGetErrorString(e);
}

void Lbvh::stage_ms(float out[5]) const {
    for (int i = 0; i < 5; ++i) {
        out[i] = 0.f;
        if (ev_[i] && ev_[i + 1]) {
            cudaEventSynchronize(ev_[i + 1]);
            cudaEventElapsedTime(&out[i], ev_[i], ev_[i + 1]);
        }
    }
}

}  // namespace lts

// ---------------------------------------------------------------------------------------------
// Allocation-free LBVH build.
//
// Some callers cannot allocate device memory at all: code running inside a host allocator or
// memory-pool callback, real-time render loops that forbid cudaMalloc/cudaFree (both can
// synchronise the whole device), and plugins whose host application owns every device
// allocation.  This variant keeps all of the build's scratch (the sort's ping-pong buffers and
// look-back table, histograms, the tree's forests and group counters, the scene box and an error word) in
// one file-scope device array of fixed size, so a call allocates nothing; the caller supplies the
// triangles and every output buffer.
//
// Limits and sharing: at most kNoAllocMaxPrims primitives (about 2.5 MiB of device memory that
// every GPU which loads the library keeps until process exit).  All calls share the one array and
// it keeps the previous call's contents, so everything that must start at zero is cleared at the
// start of each call, and two calls that overlap on the GPU (different streams, or different host
// threads) race on it.  The first call on a device looks up the array's device address with
// cudaGetSymbolAddress (which may load the module), so that first call should be made before any
// stream capture begins.  The address is kept for the life of the process: after
// cudaDeviceReset on a device, its next call would use a stale address, so a program that resets
// a device does not call this entry point on it again.  Every call blocks until its work on the
// given stream has finished (it reads the kernels' error word back before returning).
// ---------------------------------------------------------------------------------------------
namespace lts {
namespace {

constexpr int kNoAllocMaxPrims = 1 << 18;
constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kOffCodes = 0;
constexpr size_t kOffIds = kOffCodes + 4ull * kNoAllocMaxPrims;
static_assert(tree_block(kNoAllocMaxPrims) == 512 && kOffIds + 4ull * kNoAllocMaxPrims >= forest_bytes(kNoAllocMaxPrims, 512), "the tree's forests lie in both sort buffers");
constexpr size_t kOffZero = align256(kOffIds + 4ull * kNoAllocMaxPrims);
constexpr size_t kOffError = kOffZero + align256(4 * zero_words(kNoAllocMaxPrims));
constexpr size_t kNoAllocBytes = kOffError + 256;
static_assert(kNoAllocMaxPrims <= kSortSmallMax, "one tile size, so the largest build has the most tiles");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

}  // namespace

int lbvh_noalloc_limit() { return kNoAllocMaxPrims; }

}  // namespace lts





namespace {
std::mutex g_noalloc_mu;
void* g_noalloc_addr[256] = {nullptr};
}  // namespace

extern "C" int lts_bvh_build_noalloc(const float* d_tri, int32_t n, int32_t mode, int32_t code_limit,
                                     uint32_t* d_codes, int32_t* d_ids, void* d_nodes, int32_t* d_leaf_prim,
                                     float* d_root_bounds, void* stream) {
    using namespace lts;
    if (!d_tri || !d_codes || !d_ids || !d_leaf_prim || !d_root_bounds || n < 1) return LTS_ERR_ARG;
    if (n > kNoAllocMaxPrims) return LTS_ERR_ARG;
    if (n > 1 && !d_nodes) return LTS_ERR_ARG;
    if (mode != BVH_MODE_REFERENCE && mode != BVH_MODE_SORTED) return LTS_ERR_ARG;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) return LTS_ERR_CUDA;
    unsigned char* base;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_addr[dev]) {
            void* p = nullptr;
            if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return LTS_ERR_CUDA;
            g_noalloc_addr[dev] = p;
        }
        base = static_cast<unsigned char*>(g_noalloc_addr[dev]);
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    uint32_t* codes_alt = reinterpret_cast<uint32_t*>(base + kOffCodes);
    int32_t* ids_alt = reinterpret_cast<int32_t*>(base + kOffIds);
    uint32_t* zero = reinterpret_cast<uint32_t*>(base + kOffZero);
    uint32_t* err = reinterpret_cast<uint32_t*>(base + kOffError);
    int sms = 0, launches = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return LTS_ERR_CUDA;
    const bool waits = n > kSmallSort;  // the sort's look-back: the only wait that can run out
    if (waits && cudaMemsetAsync(err, 0, 4, s) != cudaSuccess) return LTS_ERR_CUDA;
    if (build_launches(d_tri, n, mode, code_limit, d_codes, d_ids, codes_alt, ids_alt, zero, 512,
                       reinterpret_cast<ForestEntry*>(codes_alt), static_cast<BvhNode*>(d_nodes), d_leaf_prim, d_root_bounds, err,
                       sms, s, &launches, [](int) {}) != cudaSuccess)
        return LTS_ERR_CUDA;
    uint32_t h_err = 0;
    if (waits && cudaMemcpyAsync(&h_err, err, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess) return LTS_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return LTS_ERR_CUDA;
    return h_err ? LTS_ERR_DEVICE : LTS_OK;
}
