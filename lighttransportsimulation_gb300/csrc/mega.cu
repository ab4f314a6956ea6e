// The float integrators beside the wavefront (sm_103a): the path-tracing megakernel, one launch (one
// thread per pixel and slice of its samples, as the reference's PathTracingKernel, intergrators/
// IntegratorKernels.cu:17-23), and the bidirectional integrator, five launches a chunk (bdpt.cuh).
//
// Differences in mechanism, not in arithmetic:
//  - scene tables are SoA arrays and materials/lights are `switch`-dispatched records, so the
//    per-bounce device `new`/`free` of BSDFs and BxDFs (materials/Material.cuh:41-52) is gone;
//  - traversal reads 64-byte two-child nodes and triangles in leaf order, visits the nearer
//    child first and keeps its node stack in shared memory; the closest hit is the same as the
//    reference's left-first visit (edges are excluded by the epsilon test, so exact-t ties
//    between neighbouring triangles cannot occur);
//  - the closest-hit SurfaceInteraction is built once from the winning triangle rather than on
//    every closer hit (it is a pure function of the ray and the triangle);
//  - the film accumulates each pixel's own 2x2 splat footprint in compensated FP32 (Kahan) in
//    shared memory and flushes it once per pixel to FP64 sums; the rare wider splats go straight
//    to FP64 atomics.  The resolve divides in FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "dev_common.cuh"
#include "dev_math.cuh"
#include "once_per_device.hpp"
#include "tracer.cuh"
#include "tracer_dev.cuh"
#include "megakernel.cuh"
#include "shade.cuh"
#include "bdpt.cuh"

namespace lts {
namespace {

#define TRY(call)                                                                       \
    do {                                                                                \
        cudaError_t e_ = (call);                                                        \
        if (e_ != cudaSuccess) return std::string(#call ": ") + cudaGetErrorString(e_); \
    } while (0)

}  // namespace

// This translation unit's copies of the procedural textures' tables on the current device.
std::string mega_init() {
    static OncePerDevice once;
    int dev = 0;
    TRY(cudaGetDevice(&dev));
    return once.run(dev, []() -> std::string {
        unsigned char p2[512];
        const float* mc = nullptr;
        texture_tables(p2, &mc);
        TRY(cudaMemcpyToSymbol(c_perm, p2, 512));
        TRY(cudaMemcpyToSymbol(c_marble, mc, 30 * sizeof(float)));
        return "";
    });
}

namespace {

// Where shade_scatter's rays and weights go: the thread's registers, until the warp traces them.
struct MegaScatter {
    Spec nee_beta, sh_c, mis_fv;
    float lpdf, mis_w, mis_pdf;
    V3 so, sd, mo, md, ro, rd;
    int light;
    bool has_nee, has_sh, sh_on, has_mis;
    __device__ __forceinline__ void nee(Spec beta, float p) {
        has_nee = true;
        nee_beta = beta;
        lpdf = p;
    }
    __device__ __forceinline__ void shadow(V3 o, V3 d, Spec c, bool on) {
        has_sh = true;
        so = o;
        sd = d;
        sh_c = c;
        sh_on = on;
    }
    __device__ __forceinline__ void mis(V3 o, V3 d, Spec fv, float w, float pdf, int l) {
        has_mis = true;
        mo = o;
        md = d;
        mis_fv = fv;
        mis_w = w;
        mis_pdf = pdf;
        light = l;
    }
    __device__ __forceinline__ void ray(V3 o, V3 d) {
        ro = o;
        rd = d;
    }
};

// The path tracer without record mode: the samples of the wavefront and of k_pathtrace bit for
// bit.  Its body is far larger than the instruction caches, and with warps at different places of
// it the kernel waited on instruction fetch (19.5 stall cycles per issue, 15 % issue active).  So
// the block's warps go through its phases together: extension rays, shading, shadow rays, MIS
// rays, with a block barrier between them (0.4 stall cycles, 37 % issue active).  Besides:
//  * one loop over bounces, not one per sample: a lane whose path has ended starts its pixel's
//    next sample in the next turn instead of waiting for the longest path of its warp;
//  * a vertex's scattering draws everything first (shade_scatter), so no surface or BSDF is held
//    in registers while the rays are traced, each kind in step over the warp (trace_warp);
//  * compiled for the lobes and textures the scene has (LM, TEX) and for the 8-wide flat tree
//    (WIDE), which leaves out the rest of the code;
//  * a pixel's samples are split over gridDim.z slices, so that a small film fills the chip.
// The box scene at 256 x 256, 16 spp: k_pathtrace (one loop per sample, 512 blocks of 128, two per
// SM) 14.6 ms; this kernel with warps running free 11.7, with the barriers 6.4 at one 128-thread
// tile per block (four blocks per SM), 5.0 at two, 5.3 at four, 5.8 at three (168 registers);
// the materials scene at 183 x 104, 15 spp: 5.4 free, 3.4, 2.3, 1.8, 1.9.  Four tiles it is.
constexpr int kMegaTiles = 4;                      // most 16 x 8 pixel tiles of a block
constexpr int kMegaWaves = 8;                      // tiles wanted per resident tile of the chip (2: +4 %)
constexpr int kMegaWords = (kStack + 32) * kThreads;  // shared words per tile: stacks, film accumulators
template <int LM, bool TEX, bool WIDE>
__global__ __launch_bounds__(kThreads * kMegaTiles, 1) void k_mega(const SceneView sv, const RenderParams rp, int nleaf,
                                                                                int tiles_x, int tiles) {
    // per tile of kThreads threads: the traversal stacks, then the film accumulators
    extern __shared__ uint32_t s_mega[];
    const int tid = threadIdx.x % kThreads, group = threadIdx.x / kThreads;
    uint32_t* stack = s_mega + group * kMegaWords + tid;
    float* acc = reinterpret_cast<float*>(s_mega + group * kMegaWords + kStack * kThreads) + tid;
    const int tile = blockIdx.x * (blockDim.x / kThreads) + group;
    const int i = rp.x0 + (tile % tiles_x) * kBX + tid % kBX;
    const int j = rp.y0 + (tile / tiles_x) * kBY + tid / kBX;
    const int W = sv.width, H = sv.height;
    const bool inside = tile < tiles && i < rp.x1 && j < rp.y1;
    bool alive = inside;
    unsigned rays = 0;
    Work wk{0u, 0u};
#pragma unroll
    for (int k = 0; k < 32; ++k) acc[k * kThreads] = 0.0f;
    const float* cam = sv.cam;
    const V3 co = v3(cam[0], cam[1], cam[2]), cright = v3(cam[3], cam[4], cam[5]), cup = v3(cam[6], cam[7], cam[8]),
             cllc = v3(cam[9], cam[10], cam[11]);
    const float rx = (float)(W - 1), ry = (float)(H - 1);
    Rng rng;
    rng.key = rp.seed + wang_hash((uint32_t)(j * W + i));
    int s = (int)blockIdx.z, bounce = -1;  // -1: the next sample has not begun
    float pfx = 0, pfy = 0;
    V3 ro = co, rd = co;
    Spec L = spec(0.0f), beta = spec(1.0f);
    bool specular = false;
    for (;;) {
        if (alive && bounce < 0) {
            if (s < rp.spp) {  // camera ray (PathTracingIntegrator.cuh:40-46, Camera.cu:51-81)
                rng.sample = (uint32_t)s;
                rng.draw = 0;
                const F2 fs = rng_2d(rng);
                (void)rng_2d(rng);  // the lens sample: drawn, moves nothing at aperture 0
                pfx = (float)(i + fs.x);
                pfy = (float)(j + fs.y);
                ro = co;
                rd = normalize(cllc + cright * (pfx / rx) + cup * (pfy / ry) - co);
                L = spec(0.0f);
                beta = spec(1.0f);
                specular = false;
                bounce = 0;
            } else {
                alive = false;
            }
        }
        if (!__syncthreads_or(alive)) break;
        // extension rays, then each hit's emission, material and scattering
        bool done = bounce >= rp.max_bounce;
        const bool ext = alive && !done;
        Trav t;
        warp_rays<false, WIDE>(ext, t, sv, nleaf, ro, rd, INFINITY, stack, rp.err, wk);
        __syncthreads();
        MegaScatter out;
        out.has_nee = out.has_sh = out.has_mis = false;
        if (ext) {
            ++rays;
            const int prim = t.best;
            const bool hit = prim >= 0;
            SI si;
            if (hit) make_si(sv, prim, rd, t.bu, t.bv, t.binv, si, &ro);
            if (bounce == 0 || specular) {
                if (hit) {
                    Spec le = spec(0.0f);
                    if (si.light >= 0) {
                        const DevLight& Lt = sv.lights[si.light];
                        if (dot(si.n, -rd) > 0.f) le = Spec{Lt.L[0], Lt.L[1], Lt.L[2]};
                    }
                    L = L + beta * le;
                } else {
                    for (int l = 0; l < sv.nlight; ++l) {
                        const DevLight& Lt = sv.lights[l];
                        L = L + beta * (Lt.kind == 1 ? Spec{Lt.L[0], Lt.L[1], Lt.L[2]} : spec(0.0f));
                    }
                }
            }
            done = !hit;
            if (hit) {
                if (bounce == 0) {  // camera-ray differentials (Ray.cuh:35-40, Interaction.cuh:118-160)
                    const V3 dx0 = normalize(cllc + cright * ((pfx + 1) / rx) + cup * (pfy / ry) - co);
                    const V3 dy0 = normalize(cllc + cright * (pfx / rx) + cup * ((pfy + 1) / ry) - co);
                    const V3 rxd = rd + (dx0 - rd) * rp.spp_scale, ryd = rd + (dy0 - rd) * rp.spp_scale;
                    const V3 n = si.n;
                    const float d = -dot(n, si.p);
                    const float tx = (-dot(n, ro) - d) / dot(n, rxd);
                    const float ty = (-dot(n, ro) - d) / dot(n, ryd);
                    si.dpdx = (ro + rxd * tx) - si.p;
                    si.dpdy = (ro + ryd * ty) - si.p;
                } else {
                    si.dpdx = v3(0, 0, 0);
                    si.dpdy = v3(0, 0, 0);
                }
                Bsdf f;
                uint64_t ev0 = 0, ev1 = 0;
                if (!make_bsdf<LM, TEX>(sv, si, f, nullptr))
                    done = true;
                else
                    done = shade_scatter<false, LM>(sv, rp, si, f, bounce, beta, specular, rng, out, nullptr, ev0, ev1);
            }
        }
        // direct light (IntegratorHelper.cuh:51-149): shadow rays, MIS BSDF rays
        Spec Ld = spec(0.0f);
        __syncthreads();
        if (__any_sync(~0u, out.has_sh)) {
            warp_rays<true, WIDE>(out.has_sh, t, sv, nleaf, out.so, out.sd, 1 - kShadowEps, stack, rp.err, wk);
            if (out.has_sh) {
                ++rays;
                if (t.best != 1 && out.sh_on) Ld = Ld + out.sh_c;
            }
        }
        __syncthreads();
        if (__any_sync(~0u, out.has_mis)) {
            warp_rays<false, WIDE>(out.has_mis, t, sv, nleaf, out.mo, out.md, INFINITY, stack, rp.err, wk);
            if (out.has_mis) {
                ++rays;
                const DevLight& Lt = sv.lights[out.light];
                Spec Li = spec(0.0f);
                if (t.best >= 0) {
                    if (Lt.kind == 0 && prim_word(sv, t.best).z == out.light) {
                        SI lit;
                        make_si(sv, t.best, out.md, t.bu, t.bv, t.binv, lit, &out.mo);
                        if (dot(lit.n, -out.md) > 0.f) Li = Spec{Lt.L[0], Lt.L[1], Lt.L[2]};
                    }
                } else if (Lt.kind == 1) {
                    Li = Spec{Lt.L[0], Lt.L[1], Lt.L[2]};
                }
                if (!is_black(Li)) Ld = Ld + out.mis_fv * Li * spec(1.0f) * out.mis_w / out.mis_pdf;
            }
        }
        if (out.has_nee) L = L + out.nee_beta * (Ld / out.lpdf);
        if (alive && !done) {
            ro = out.ro;
            rd = out.rd;
            ++bounce;
        }
        if (alive && done) {  // film (Camera::addSample, Camera.cu:192-218)
            const int px0 = max((int)ceilf(pfx - 1.0f), 0), py0 = max((int)ceilf(pfy - 1.0f), 0);
            const int px1 = min((int)floorf(pfx + 1.0f) + 1, W), py1 = min((int)floorf(pfy + 1.0f) + 1, H);
            for (int y = py0; y < py1; ++y) {
                for (int x = px0; x < px1; ++x) {
                    const float fdx = fabsf((x - pfx - 0.5f) * 1.0f * 16);
                    const float fdy = fabsf((y - pfy - 0.5f) * 1.0f * 16);
                    const int ix = min((int)floorf(fdx), 15), iy = min((int)floorf(fdy), 15);
                    const float wgt = __ldg(sv.filter + iy * 16 + ix);
                    const Spec c = L * wgt;
                    const int ox = x - i, oy = y - j;
                    if (ox >= 0 && ox <= 1 && oy >= 0 && oy <= 1) {
                        const int base = (oy * 2 + ox) * 4;
                        kahan_add(acc + (base + 0) * kThreads, acc + (16 + base + 0) * kThreads, c.r);
                        kahan_add(acc + (base + 1) * kThreads, acc + (16 + base + 1) * kThreads, c.g);
                        kahan_add(acc + (base + 2) * kThreads, acc + (16 + base + 2) * kThreads, c.b);
                        kahan_add(acc + (base + 3) * kThreads, acc + (16 + base + 3) * kThreads, wgt);
                    } else {
                        double* fp = rp.film + 4 * ((size_t)y * W + x);
                        atomicAdd(fp + 0, (double)c.r);
                        atomicAdd(fp + 1, (double)c.g);
                        atomicAdd(fp + 2, (double)c.b);
                        atomicAdd(fp + 3, (double)wgt);
                    }
                }
            }
            s += (int)gridDim.z;
            bounce = -1;
        }
    }
    // flush the 2x2 core accumulators (sum minus compensation) to the FP64 film
    if (inside) {
        for (int oy = 0; oy < 2; ++oy)
            for (int ox = 0; ox < 2; ++ox) {
                const int x = i + ox, y = j + oy;
                if (x >= W || y >= H) continue;
                double* fp = rp.film + 4 * ((size_t)y * W + x);
                const int base = (oy * 2 + ox) * 4;
                for (int c = 0; c < 4; ++c) {
                    const float sum = acc[(base + c) * kThreads], cmp = acc[(16 + base + c) * kThreads];
                    if (sum != 0.0f || cmp != 0.0f) atomicAdd(fp + c, (double)sum - (double)cmp);
                }
            }
    }
    const unsigned tot = __reduce_add_sync(~0u, rays);
    const unsigned tn = __reduce_add_sync(~0u, wk.nodes), tt = __reduce_add_sync(~0u, wk.tris);
    if ((tid & 31) == 0 && rp.counters) {
        atomicAdd(rp.counters, (unsigned long long)tot);
        atomicAdd(rp.counters + 1, (unsigned long long)tn);
        atomicAdd(rp.counters + 2, (unsigned long long)tt);
    }
}

}  // namespace

std::string mega_set_libm_double(int on) {
    const int v = on ? 1 : 0;
    TRY(cudaMemcpyToSymbol(c_libm_double, &v, sizeof v));
    return "";
}

// matte_only: every material is Lambertian / Oren-Nayar with constant textures.
std::string mega_launch(const SceneView& sv, const RenderParams& rp, int nleaf, bool matte_only, cudaStream_t s) {
    // sample slices until every SM's four tiles are filled kMegaWaves times over; blocks of fewer
    // tiles when there are not four tiles for every SM (a thumbnail's few blocks would leave most SMs
    // idle)
    const dim3 grid((rp.x1 - rp.x0 + kBX - 1) / kBX, (rp.y1 - rp.y0 + kBY - 1) / kBY);
    int dev = 0, sms = 0;
    TRY(cudaGetDevice(&dev));
    TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const long tiles = (long)grid.x * grid.y, want = (long)kMegaWaves * kMegaTiles * sms;
    const long z = std::max(1L, std::min<long>({(long)rp.spp, (want + tiles - 1) / tiles, 65535L}));
    const long per = std::max(1L, std::min<long>(kMegaTiles, tiles * z / sms));
    const bool wide = sv.wnodes != nullptr && sv.ninst == 0;
    auto k = !wide ? k_mega<LM_ALL, true, false> : matte_only ? k_mega<LM_MATTE, false, true> : k_mega<LM_ALL, true, true>;
    TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kMegaWords * kMegaTiles));
    k<<<dim3((unsigned)((tiles + per - 1) / per), 1, (unsigned)z), (unsigned)(kThreads * per), 4 * kMegaWords * per, s>>>(
        sv, rp, nleaf, (int)grid.x, (int)tiles);
    TRY(cudaGetLastError());
    return "";
}

namespace {
// The strategies (s, t) of a path of at most maxb + 2 vertices (only >= 0: the one s = only / 100,
// t = only % 100), camera vertices outer, light vertices inner.
BdptStrategies bdpt_strategies(int maxb, int only) {
    BdptStrategies st;
    st.n = 0;
    for (int t = 1; t <= maxb + 2; ++t)
        for (int s = 0; s <= maxb + 1; ++s) {
            const int depth = t + s - 2;
            if ((s == 1 && t == 1) || depth < 0 || depth > maxb) continue;
            if (only >= 0 && (s != only / 100 || t != only % 100)) continue;
            if (st.n < kBdptMaxStrategies) {
                st.s[st.n] = (unsigned char)s;
                st.t[st.n] = (unsigned char)t;
                ++st.n;
            }
        }
    return st;
}
static_assert((kBdptMaxBounce + 2) * (kBdptMaxBounce + 3) / 2 + kBdptMaxBounce <= kBdptMaxStrategies,
              "every strategy of the longest path fits the list");
}  // namespace

size_t bdpt_sample_bytes(int max_bounce, int strategy) {
    const int maxb = std::min(max_bounce, kBdptMaxBounce);
    return (size_t)(2 * maxb + 2) * (16 * kBvWordsAll + 8) + (16 + 36) * (size_t)bdpt_strategies(maxb, strategy).n + 20;
}

std::string bdpt_launch(const SceneView& sv, const RenderParams& rp, int nleaf, double* splat, int strategy,
                        bool matte_only, void* ws, long cap, uint32_t* d_count, cudaStream_t s, int* launches) {
    *launches = 0;
    const int maxb = std::min(rp.max_bounce, kBdptMaxBounce);
    const BdptStrategies st = bdpt_strategies(maxb, strategy);
    const bool wide = sv.wnodes != nullptr && sv.ninst == 0;
    const size_t slots = 2 * (size_t)maxb + 2, words = matte_only && wide ? kBvWordsMatte : kBvWordsAll;
    BdptBuf buf;
    buf.cap = (int)cap;
    buf.vert = static_cast<uint4*>(ws);
    buf.head = buf.vert + slots * words * cap;
    buf.contrib = reinterpret_cast<float4*>(buf.head + cap);
    buf.ray_o = buf.contrib + (size_t)st.n * cap;
    buf.ray_d = buf.ray_o + (size_t)st.n * cap;
    buf.pdf = reinterpret_cast<float2*>(buf.ray_d + (size_t)st.n * cap);
    buf.delta = reinterpret_cast<uint32_t*>(buf.pdf + slots * cap);
    buf.sees = buf.delta + cap;
    buf.count = d_count;
    const long total = (long)(rp.x1 - rp.x0) * (rp.y1 - rp.y0) * rp.spp;
    int dev = 0, sms = 0;
    TRY(cudaGetDevice(&dev));
    TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    for (long first = 0; first < total; first += cap) {
        const int n = (int)std::min(cap, total - first);
        const unsigned gw = (unsigned)((n + kBdptWalkThreads - 1) / kBdptWalkThreads), gs = (unsigned)((n + kThreads - 1) / kThreads);
        auto kw = !wide ? k_bdpt_walk<LM_ALL, true, false> : matte_only ? k_bdpt_walk<LM_MATTE, false, true> : k_bdpt_walk<LM_ALL, true, true>;
        const bool matte = wide && matte_only;
        kw<<<gw, kBdptWalkThreads, 0, s>>>(sv, rp, nleaf, buf, first, n);
        if (st.n > 0) {
            TRY(cudaMemsetAsync(buf.count, 0, 8, s));
            auto kc = matte ? k_bdpt_connect<LM_MATTE> : k_bdpt_connect<LM_ALL>;
            kc<<<dim3(gs, (unsigned)st.n), kThreads, 0, s>>>(sv, rp, buf, st, first, n, strategy);
            auto ks = wide ? k_bdpt_shadow : k_bdpt_shadow_any;
            ks<<<kBdptShadowBlocks * sms, kThreads, 0, s>>>(sv, rp, nleaf, buf);
            auto kt = matte ? k_bdpt_weight<LM_MATTE> : k_bdpt_weight<LM_ALL>;
            kt<<<kBdptConnectBlocks * 4 * sms, kThreads, 0, s>>>(sv, rp, buf, st, first, strategy, splat);
        }
        k_bdpt_film<<<gs, kThreads, 0, s>>>(sv, rp, buf, st, n);
        *launches += st.n > 0 ? 5 : 2;
        TRY(cudaGetLastError());
    }
    return "";
}

}  // namespace lts
