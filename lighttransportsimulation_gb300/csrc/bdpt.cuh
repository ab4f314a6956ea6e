// Bidirectional path tracing (sm_103a): every sample builds a camera subpath and a light subpath
// and combines every connection strategy (s light vertices, t camera vertices) with
// multiple-importance weights -- the algorithm of Veach's thesis as PBRT v3 states it (ch. 16.3:
// random walks with forward / reverse area densities, ConnectBDPT, MISWeight's ratio chain).
//
// Five kernels over a chunk of samples:
//   k_bdpt_walk     one thread per sample: both random walks in one loop, the vertices written to
//                   a structure of arrays in device memory
//   k_bdpt_connect  one thread per (strategy, sample), the strategy uniform over a block: the
//                   connection's unweighted contribution and its shadow ray, listed
//   k_bdpt_shadow   persistent warps over the listed rays (k_bdpt_shadow_any: trees other than the
//                   8-wide flat one)
//   k_bdpt_weight   one thread per listed connection: the MIS weight of those that see each other
//   k_bdpt_film     one thread per sample: the contributions summed in strategy order and filtered
//                   into the film
// As one kernel (a thread per pixel with its vertices in local memory) the same work ran at 4.7
// of 32 lanes and waited on instruction fetch (39.5 stall cycles per issue): lanes were at
// different strategies of different samples and the body is far larger than the instruction
// caches.  Here a warp is at one strategy, and a kernel's body is one stage: the box lit by one
// triangle, 256 x 256, 16 spp, 5 bounces, 81.2 -> 12.0 ms with the same contributions bit for bit
// while the connection still traced its ray and weighted its result (10.5 of 32 lanes, waiting for
// a warp's longest ray: 1.78 ms a chunk), 8.6 ms with the rays listed
// (0.41 ms a chunk connecting, 0.25 the rays, 0.31 the weights, beside 1.11 for the walks).
//
// The reference ships this integrator disabled and unfinished (intergrators/
// BidirectionalPathIntegrator.cuh:285-660, LightTransportSimulation.cu:116-121): its light walk
// starts on top of the light vertex (`randomWalk(..., path, id)` overwrites path[0]), its
// strategy loops stop one vertex short (`t < nCamera`, `s < nLight`), and its camera importance
// (Camera.cu:88-186) divides by the raster's pixel count instead of the image plane's area.  Here
// the published algorithm is built over this renderer's own pieces -- the traversal, make_si,
// the materials' BSDFs, the area and point lights -- so that it estimates the same image as the
// path tracer: tests compare the two films.
//
// The reference's dielectric is not reciprocal (its "reflection" continues straight through the
// surface with the Fresnel term of the arriving side, Specular.cuh:112), so paths through glass
// are weighted differently when traced from the light: where glass shapes the image (a caustic)
// this estimator and the path tracer's differ.
//
// Scope: area and point lights (the reference's infinite light has no consistent emission
// density: its sampleLi draws a hemisphere about +y with a latitude-longitude pdf about +z, so a
// scene with one is refused).  The camera is the reference's pinhole (lens radius 0): importance
// We = 1 / (A cos^4), direction density 1 / (A cos^3) with A the film's area on the plane at unit
// distance.  Subpaths have no Russian roulette (MIS needs the plain densities); camera subpaths
// carry up to max_bounce + 2 vertices, light subpaths up to max_bounce + 1.  Connections to the
// camera (t = 1) land anywhere on the film and are splatted, unfiltered, into a separate buffer
// scaled by 1 / spp at resolve.
#pragma once

#include "shade.cuh"
#include "tracer_dev.cuh"

namespace lts {
namespace {

enum : int { BV_CAMERA = 0, BV_LIGHT = 1, BV_SURFACE = 2 };

struct BVert {
    int type;        // BV_*
    int light;       // light vertices and emitting surfaces: light index, else -1
    V3 p, n, perr;   // position, geometric normal (zero: not on a surface), position error bound
    V3 wo;           // surface: direction toward the vertex it was reached from
    Spec beta;       // throughput up to and including this vertex
    real pdf_fwd;    // area density of a resampled light point (the walks' densities are in BdptBuf::pdf)
    Bsdf f;          // surface: its scattering functions
};

// Camera model (rendering/Camera.cu:9-43, lens radius 0): origin, screen corner and edge vectors
// at the focal distance, viewing direction -w.
struct BCam {
    V3 o, right, up, llc, w;
    real focal, area;  // film area on the plane at unit distance
    int W, H;
};
__device__ __forceinline__ BCam bdpt_camera(const SceneView& sv) {
    BCam c;
    const float* m = sv.cam;
    c.o = v3(m[0], m[1], m[2]);
    c.right = v3(m[3], m[4], m[5]);
    c.up = v3(m[6], m[7], m[8]);
    c.llc = v3(m[9], m[10], m[11]);
    c.w = v3(m[18], m[19], m[20]);
    c.focal = m[22];
    c.W = sv.width;
    c.H = sv.height;
    // rays go through llc + right * px / (W - 1) + up * py / (H - 1) for px in [0, W), py in [0, H)
    const real sx = xsqrt(len2(c.right)) * ((real)c.W / (real)(c.W - 1));
    const real sy = xsqrt(len2(c.up)) * ((real)c.H / (real)(c.H - 1));
    c.area = sx * sy / (c.focal * c.focal);
    return c;
}
// The film position of direction d from the camera (false: behind the camera or off the film),
// and cos(theta) to the viewing axis.
__device__ __forceinline__ bool bdpt_raster(const BCam& c, V3 d, real& px, real& py, real& cos_t) {
    cos_t = -dot(d, c.w);
    if (cos_t <= 0) return false;
    const V3 s = c.o + d * (c.focal / cos_t) - c.llc;
    px = dot(s, c.right) / len2(c.right) * (real)(c.W - 1);
    py = dot(s, c.up) / len2(c.up) * (real)(c.H - 1);
    return px >= 0 && px < (real)c.W && py >= 0 && py < (real)c.H;
}
__device__ __forceinline__ real bdpt_we(const BCam& c, real cos_t) {
    const real c2 = cos_t * cos_t;
    return 1 / (c.area * c2 * c2);
}
__device__ __forceinline__ real bdpt_pdf_dir(const BCam& c, real cos_t) { return 1 / (c.area * cos_t * cos_t * cos_t); }

// Light choice with the power distribution (Distribution1D, sampling/Sampling.cuh:104-198) over
// every light -- without the reference's findInterval clamp that never picks the last light.
__device__ __forceinline__ int bdpt_pick_light(const SceneView& sv, real u, real& pdf) {
    const int n = sv.nlight;
    int first = 0, len = n + 1;
    while (len > 0) {
        const int half = len >> 1, middle = first + half;
        if (__ldg(sv.light_cdf + middle) <= u) {
            first = middle + 1;
            len -= half + 1;
        } else {
            len = half;
        }
    }
    const int i = max(0, min(first - 1, n - 1));
    pdf = __ldg(sv.light_func + i) / (sv.light_func_int * n);
    return i;
}
__device__ __forceinline__ real bdpt_light_pdf(const SceneView& sv, int i) {
    return __ldg(sv.light_func + i) / (sv.light_func_int * sv.nlight);
}

__device__ __forceinline__ bool bv_on_surface(const BVert& v) { return v.n.x != 0 || v.n.y != 0 || v.n.z != 0; }
__device__ __forceinline__ bool bv_delta_light(const SceneView& sv, const BVert& v) {
    return v.type == BV_LIGHT && sv.lights[v.light].kind == 2;  // a point light's position
}
__device__ __forceinline__ bool bv_is_light(const BVert& v) {
    return v.type == BV_LIGHT || (v.type == BV_SURFACE && v.light >= 0);
}
__device__ __forceinline__ bool bv_connectible(const BVert& v) {
    if (v.type != BV_SURFACE) return true;
    return v.f.lobe != LOBE_NONE && (v.f.type & (BSDF_DIFFUSE | BSDF_GLOSSY)) != 0;
}
// Vertex::ConvertDensity: a solid-angle density at `from` toward `to` in area measure at `to`.
__device__ __forceinline__ real bv_convert(real pdf, const BVert& from, const BVert& to) {
    const V3 d = to.p - from.p;
    const real l2 = len2(d);
    if (l2 == 0) return 0;
    const real inv = 1 / l2;
    if (bv_on_surface(to)) pdf *= absdot(to.n, d * xsqrt(inv));
    return pdf * inv;
}
// PBRT's CorrectShadingNormal for importance transport (the reference's correctShadingNormal,
// BidirectionalPathIntegrator.cuh:11-22).
__device__ __forceinline__ real bdpt_shading_fix(const Bsdf& f, V3 wo, V3 wi) {
    const real den = absdot(wo, f.ng) * absdot(wi, f.ns);
    if (den == 0) return 0;
    return absdot(wo, f.ns) * absdot(wi, f.ng) / den;
}
// Vertex::f: scattering at surface vertex v toward `next`.  LM (and TEX below): the lobes (and
// textures) the scene's materials can have -- the kernel is compiled for them only, as the
// wavefront's shade kernels are.
template <int LM>
__device__ __forceinline__ Spec bv_f(const BVert& v, const BVert& next, bool importance) {
    const V3 wi = normalize(next.p - v.p);
    Spec c = bsdf_f<LM>(v.f, v.wo, wi, BSDF_ALL, nullptr);
    if (importance) c = c * bdpt_shading_fix(v.f, v.wo, wi);
    return c;
}
// Emitted radiance of light vertex or emitting surface v toward w (DiffuseAreaLight::L: one-sided
// along the surface normal; a point light's intensity is reached only by connections).
__device__ __forceinline__ Spec bv_le(const SceneView& sv, const BVert& v, V3 w) {
    if (v.light < 0) return spec(0.0f);
    const DevLight& L = sv.lights[v.light];
    if (L.kind != 0) return spec(0.0f);
    return dot(v.n, w) > 0 ? Spec{L.L[0], L.L[1], L.L[2]} : spec(0.0f);
}
// Vertex::PdfLight: density (area measure at `to`) of light vertex v emitting toward `to`.
__device__ __forceinline__ real bv_pdf_light(const SceneView& sv, const BVert& v, const BVert& to) {
    const V3 d = to.p - v.p;
    const real l2 = len2(d);
    if (l2 == 0) return 0;
    const V3 w = d * xsqrt(1 / l2);
    const DevLight& L = sv.lights[v.light];
    real pdf = L.kind == 0 ? xmax(0.0f, dot(v.n, w)) * LTS_INV_PI_F : (real)(0.25 * LTS_INV_PI_F);
    pdf /= l2;
    if (bv_on_surface(to)) pdf *= absdot(to.n, w);
    return pdf;
}
// Vertex::PdfLightOrigin: light choice times the position density (0 for a point light's delta).
__device__ __forceinline__ real bv_pdf_light_origin(const SceneView& sv, const BVert& v) {
    const DevLight& L = sv.lights[v.light];
    return L.kind == 0 ? bdpt_light_pdf(sv, v.light) / L.area : 0.0f;
}
// Vertex::Pdf: density (area measure at `next`) of sampling `next` from v, which was reached from
// `prev` (null for an endpoint).
template <int LM>
__device__ __forceinline__ real bv_pdf(const SceneView& sv, const BCam& cam, const BVert& v, const BVert* prev,
                                       const BVert& next) {
    if (v.type == BV_LIGHT) return bv_pdf_light(sv, v, next);
    const V3 d = next.p - v.p;
    if (len2(d) == 0) return 0;
    const V3 wn = normalize(d);
    real pdf;
    if (v.type == BV_CAMERA) {
        real px, py, cos_t;
        if (!bdpt_raster(cam, wn, px, py, cos_t)) return 0;
        pdf = bdpt_pdf_dir(cam, cos_t);
    } else {
        if (!prev) return 0;
        const V3 wp = normalize(prev->p - v.p);
        pdf = bsdf_pdf<LM>(v.f, wp, wn, BSDF_ALL, nullptr);
    }
    return bv_convert(pdf, v, next);
}

// The chunk's buffers.  A vertex is kBvWords 16-byte words, word w of vertex slot v of sample k at
// vert[(v * words + w) * cap + k] (lanes of a warp read neighbouring samples); slots: camera
// vertices 1 .. maxb + 1, then light vertices 0 .. maxb.  Matte scenes leave out the last words.
constexpr int kBvWordsMatte = 8, kBvWordsAll = 11;
struct BdptBuf {
    uint4* vert;
    float2* pdf;    // (pdf_fwd, pdf_rev) of vertex slot v of sample k at [v * cap + k]
    uint4* head;    // per sample: film x, y bits; draw after both walks; n_cam | n_light << 4 |
                    // connectible camera vertices << 8 (bit 8 + c: vertex c)
    uint32_t* delta;  // per sample: delta camera vertices (bit c), delta light vertices (bit 16 + l)
    float4* contrib;  // [strategy * cap + k]
    // the connections with a contribution, in list order (count[0] of them): the ray's origin and its
    // sample, its direction and its strategy | kConnFree (no ray to trace), 1 when it sees
    float4 *ray_o, *ray_d;
    uint32_t* sees;
    uint32_t* count;  // [0] listed, [1] trace fetch
    int cap;
};
constexpr uint32_t kConnFree = 256u;
// The strategies rendered, in the order their contributions are summed (t outer, s inner).
constexpr int kBdptMaxStrategies = 64;
struct BdptStrategies {
    int n;
    unsigned char s[kBdptMaxStrategies], t[kBdptMaxStrategies];
};

template <int LM>
__device__ __forceinline__ int bv_words() {
    return (LM & ~LM_MATTE) ? kBvWordsAll : kBvWordsMatte;
}
template <int LM>
__device__ __forceinline__ void bv_store(const BdptBuf& b, int slot, int k, const BVert& v) {
    uint4* o = b.vert + (size_t)slot * bv_words<LM>() * b.cap + k;
    auto put = [&](int w, V3 a, uint32_t x) {
        o[(size_t)w * b.cap] = make_uint4(__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(a.z), x);
    };
    put(0, v.p, (uint32_t)v.type | ((uint32_t)v.f.lobe << 4) | (v.f.type << 8));
    put(1, v.n, (uint32_t)v.light);
    put(2, v.perr, __float_as_uint(v.f.a));
    put(3, v.wo, __float_as_uint(v.f.b));
    put(4, v3(v.beta.r, v.beta.g, v.beta.b), __float_as_uint(v.f.R.r));
    put(5, v.f.ns, __float_as_uint(v.f.R.g));
    put(6, v.f.ss, __float_as_uint(v.f.R.b));
    put(7, v.f.ts, __float_as_uint(v.f.eta));
    if (LM & ~LM_MATTE) {
        put(8, v3(v.f.T.r, v.f.T.g, v.f.T.b), __float_as_uint(v.f.alpha));
        put(9, v3(v.f.k.r, v.f.k.g, v.f.k.b), 0u);
        put(10, v3(v.f.eta3.r, v.f.eta3.g, v.f.eta3.b), 0u);
    }
}
// The stored vertex (the words of fields the caller does not use are not read).
template <int LM>
__device__ __forceinline__ void bv_load(const BdptBuf& b, int slot, int k, BVert& v) {
    const uint4* o = b.vert + (size_t)slot * bv_words<LM>() * b.cap + k;
    auto get = [&](int w, V3& a) -> uint32_t {
        const uint4 q = __ldg(o + (size_t)w * b.cap);
        a = v3(__uint_as_float(q.x), __uint_as_float(q.y), __uint_as_float(q.z));
        return q.w;
    };
    V3 c;
    const uint32_t m = get(0, v.p);
    v.type = (int)(m & 15u);
    v.f.lobe = (int)((m >> 4) & 15u);
    v.f.type = m >> 8;
    v.light = (int)get(1, v.n);
    v.f.ng = v.n;
    v.f.a = __uint_as_float(get(2, v.perr));
    v.f.b = __uint_as_float(get(3, v.wo));
    v.f.R.r = __uint_as_float(get(4, c));
    v.beta = Spec{c.x, c.y, c.z};
    v.f.R.g = __uint_as_float(get(5, v.f.ns));
    v.f.R.b = __uint_as_float(get(6, v.f.ss));
    v.f.eta = __uint_as_float(get(7, v.f.ts));
    if (LM & ~LM_MATTE) {
        v.f.alpha = __uint_as_float(get(8, c));
        v.f.T = Spec{c.x, c.y, c.z};
        get(9, c);
        v.f.k = Spec{c.x, c.y, c.z};
        get(10, c);
        v.f.eta3 = Spec{c.x, c.y, c.z};
    }
}
__device__ __forceinline__ BVert bv_camera(const BCam& cam) {
    BVert v;
    v.type = BV_CAMERA;
    v.light = -1;
    v.p = cam.o;
    v.n = v3(0, 0, 0);
    v.perr = v3(0, 0, 0);
    v.beta = spec(1.0f);
    v.pdf_fwd = 0;
    v.f.lobe = LOBE_NONE;
    v.f.type = 0;
    return v;
}

// The pixel of batch sample `idx` (all pixels of sample 0, then of sample 1, ...; pixels in 8 x 4
// tiles) and its sample number.
__device__ __forceinline__ void bdpt_pixel(const RenderParams& rp, long idx, int& i, int& j, int& s) {
    const int cw = rp.x1 - rp.x0, ch = rp.y1 - rp.y0;
    const long npix = (long)cw * ch;
    s = (int)(idx / npix);
    int ci, cj;
    tile_pixel(idx - s * npix, cw, ch, ci, cj);
    i = rp.x0 + ci;
    j = rp.y0 + cj;
}

// GenerateCameraSubpath and GenerateLightSubpath (the random walks of RandomWalk) of samples
// first .. first + n - 1.  One loop: a lane whose camera walk has ended starts its light walk in the
// next turn; the block's warps trace and extend together (barriers), as in the path tracer's
// megakernel.
constexpr int kBdptWalkThreads = 256;
#ifndef LTS_BDPT_WALK_BLOCKS
#define LTS_BDPT_WALK_BLOCKS 2
#endif
template <int LM, bool TEX, bool WIDE>
__global__ __launch_bounds__(kBdptWalkThreads, LTS_BDPT_WALK_BLOCKS) void k_bdpt_walk(const SceneView sv, const RenderParams rp,
                                                                                      int nleaf, BdptBuf buf, long first, int n) {
    __shared__ uint32_t s_stack[kStack * kBdptWalkThreads];
    uint32_t* stack = s_stack + (threadIdx.x / kThreads) * (kStack * kThreads) + threadIdx.x % kThreads;
    const int k = blockIdx.x * kBdptWalkThreads + threadIdx.x;
    const bool in = k < n;
    const BCam cam = bdpt_camera(sv);
    const int maxb = min(rp.max_bounce, kBdptMaxBounce);
    unsigned rays = 0;
    Work wk{0u, 0u};
    int i = 0, j = 0, s_ix = 0;
    if (in) bdpt_pixel(rp, first + k, i, j, s_ix);
    Rng rng;
    rng.key = rp.seed + wang_hash((uint32_t)(j * sv.width + i));
    rng.sample = (uint32_t)s_ix;
    rng.draw = 0;
    const real rx = (real)(cam.W - 1), ry = (real)(cam.H - 1);
    // camera subpath: the path tracer's primary ray
    const F2 fs = rng_2d(rng);
    (void)rng_2d(rng);
    const real pfx = (real)(i + fs.x), pfy = (real)(j + fs.y);
    V3 ro = cam.o, rd = normalize(cam.llc + cam.right * (pfx / rx) + cam.up * (pfy / ry) - cam.o);
    Spec beta = spec(1.0f);
    real cpx, cpy, cos_t;
    bdpt_raster(cam, rd, cpx, cpy, cos_t);
    real pdf_fwd = bdpt_pdf_dir(cam, cos_t);
    V3 prev_p = cam.o, prev_n = v3(0, 0, 0);
    int phase = in ? 0 : 2, bounces = 0, max_depth = maxb + 1;  // phase 0: camera walk, 1: light walk, 2: done
    int n_cam = 1, n_light = 0;
    uint32_t conn = 0, delta = 0;
    while (__syncthreads_or(phase < 2)) {
        const bool on = phase < 2 && bounces < max_depth;
        Trav t;
        warp_rays<false, WIDE>(on, t, sv, nleaf, ro, rd, INFINITY, stack, rp.err, wk);
        __syncthreads();
        bool end = phase < 2;
        if (on) {
            ++rays;
            if (t.best >= 0 && !is_black(beta)) {
                SI si;
                make_si(sv, t.best, rd, t.bu, t.bv, t.binv, si, &ro);
                if (phase == 0 && bounces == 0) {  // camera-ray differentials for the first hit's textures
                    const V3 dx0 = normalize(cam.llc + cam.right * ((pfx + 1) / rx) + cam.up * (pfy / ry) - cam.o);
                    const V3 dy0 = normalize(cam.llc + cam.right * (pfx / rx) + cam.up * ((pfy + 1) / ry) - cam.o);
                    const V3 rxd = rd + (dx0 - rd) * rp.spp_scale, ryd = rd + (dy0 - rd) * rp.spp_scale;
                    const V3 nn = si.n;
                    const real d = -dot(nn, si.p);
                    const real tx = (-dot(nn, ro) - d) / dot(nn, rxd);
                    const real ty = (-dot(nn, ro) - d) / dot(nn, ryd);
                    si.dpdx = (ro + rxd * tx) - si.p;
                    si.dpdy = (ro + ryd * ty) - si.p;
                } else {
                    si.dpdx = v3(0, 0, 0);
                    si.dpdy = v3(0, 0, 0);
                }
                BVert v, prev;
                v.type = BV_SURFACE;
                v.light = si.light;
                v.p = si.p;
                v.n = si.n;
                v.perr = si.perr;
                v.wo = -rd;
                v.beta = beta;
                v.f = Bsdf{};
                prev.p = prev_p;
                prev.n = prev_n;
                if (!make_bsdf<LM, TEX>(sv, si, v.f, nullptr)) v.f.lobe = LOBE_NONE;
                v.f.ng = si.n;
                const int slot = phase == 0 ? bounces : maxb + 2 + bounces;  // camera vertex bounces + 1, light bounces + 1
                buf.pdf[(size_t)slot * buf.cap + k] = make_float2(bv_convert(pdf_fwd, prev, v), 0.f);
                bv_store<LM>(buf, slot, k, v);
                if (phase == 0 && bv_connectible(v)) conn |= 1u << (bounces + 1);
                ++bounces;
                if (bounces < max_depth && v.f.lobe != LOBE_NONE) {
                    V3 wi;
                    uint32_t stype = 0;
                    real pdf = 0;
                    const Spec fv = bsdf_sample<LM>(v.f, v.wo, wi, rng_2d(rng), pdf, BSDF_ALL, stype, nullptr);
                    if (!is_black(fv) && pdf != 0) {
                        end = false;
                        beta = beta * (fv * absdot(wi, v.f.ns) / pdf);
                        pdf_fwd = pdf;
                        real pdf_rev = bsdf_pdf<LM>(v.f, wi, v.wo, BSDF_ALL, nullptr);
                        if (stype & BSDF_SPECULAR) {
                            delta |= phase == 0 ? 1u << bounces : 0x10000u << bounces;
                            pdf_fwd = pdf_rev = 0;
                        }
                        if (phase == 1) {  // importance
                            beta = beta * bdpt_shading_fix(v.f, v.wo, wi);
                            // specular transmission scales radiance by (eta_i / eta_t)^2 (the BSDF applies
                            // it); importance is not scaled (PBRT's TransportMode), so light paths undo it
                            if (v.f.lobe == LOBE_FRESNEL_SPECULAR && (stype & BSDF_TRANSMISSION)) {
                                const bool entering = dot(v.wo, v.f.ns) > 0;
                                const real ei = entering ? 1.0f : v.f.eta, et = entering ? v.f.eta : 1.0f;
                                beta = beta * ((et * et) / (ei * ei));
                            }
                        }
                        // the vertex before: camera vertex 0 has no slot
                        if (slot > 0) buf.pdf[(size_t)(slot - 1) * buf.cap + k].y = bv_convert(pdf_rev, v, prev);
                        ro = offset_origin(si.p, si.perr, si.n, wi);
                        rd = wi;
                        prev_p = v.p;
                        prev_n = v.n;
                    }
                }
            }
        }
        if (end && phase == 1) {
            n_light = 1 + bounces;
            phase = 2;
        } else if (end) {  // the camera walk is over: the light walk's start
            n_cam = 1 + bounces;
            phase = 2;
            bounces = 0;
            max_depth = maxb;
            real lpick;
            const int li = bdpt_pick_light(sv, rng_1d(rng), lpick);
            const F2 u1 = rng_2d(rng), u2 = rng_2d(rng);
            const DevLight& L = sv.lights[li];
            BVert l0 = bv_camera(cam);
            l0.type = BV_LIGHT;
            l0.light = li;
            l0.f = Bsdf{};
            l0.wo = v3(0, 0, 0);
            V3 dir, nl;
            real pdf_pos = 0, pdf_dir = 0;
            const Spec Le = Spec{L.L[0], L.L[1], L.L[2]};
            if (L.kind == 0) {  // point on the triangle (Triangle::sample), cosine-weighted direction
                // weights of p0, p1, p2 as Triangle::sample draws them (Triangle.cu:232-259); the
                // emitting side is the surface normal make_si gives a hit there
                const real su = xsqrt(u1.x);
                const real w0 = 1 - su, w1 = u1.y * su, w2 = 1 - w0 - w1;
                V3 p0, p1, p2;
                prim_tri(sv, L.prim, p0, p1, p2);
                SI ls;
                make_si(sv, L.prim, v3(0, 0, 1), w1, w2, 1.0f, ls);
                nl = ls.n;
                l0.p = p0 * w0 + p1 * w1 + p2 * w2;
                l0.perr = (vabs(p0 * w0) + vabs(p1 * w1) + vabs(p2 * w2)) * gamma_n(6);
                l0.n = nl;
                const real r = xsqrt(u2.x), th = mul_dc(u2.y, LTS_2PI);
                const real lx = r * xcos(th), ly = r * xsin(th), lz = xsqrt(xmax(0.0f, 1 - lx * lx - ly * ly));
                V3 a, b;
                coordinate_system(nl, a, b);
                dir = normalize(a * lx + b * ly + nl * lz);
                pdf_pos = 1 / L.area;
                pdf_dir = lz * LTS_INV_PI_F;
            } else {  // point light: uniform sphere of directions
                const real z = 1 - 2 * u1.x, r = xsqrt(xmax(0.0f, 1 - z * z)), ph = mul_dc(u1.y, LTS_2PI);
                dir = v3(r * xcos(ph), r * xsin(ph), z);
                nl = dir;
                l0.p = v3(L.p[0], L.p[1], L.p[2]);
                pdf_pos = 1;
                pdf_dir = (real)(0.25 * LTS_INV_PI_F);
            }
            if (pdf_pos > 0 && pdf_dir > 0 && !is_black(Le)) {
                l0.beta = Le;
                buf.pdf[(size_t)(maxb + 1) * buf.cap + k] = make_float2(pdf_pos * lpick, 0.f);
                bv_store<LM>(buf, maxb + 1, k, l0);
                beta = Le * (absdot(nl, dir) / (lpick * pdf_pos * pdf_dir));
                pdf_fwd = pdf_dir;
                ro = offset_origin(l0.p, l0.perr, l0.n, dir);
                rd = dir;
                prev_p = l0.p;
                prev_n = l0.n;
                phase = 1;  // a walk of no surface vertices (max_bounce 0) ends in the next turn
            }
        }
    }
    if (in) {
        buf.head[k] = make_uint4(__float_as_uint(pfx), __float_as_uint(pfy), rng.draw,
                                 (uint32_t)n_cam | ((uint32_t)n_light << 4) | (conn << 8));
        buf.delta[k] = delta;
    }
    const unsigned tot = __reduce_add_sync(~0u, rays);
    if ((threadIdx.x & 31) == 0 && rp.counters) atomicAdd(rp.counters, (unsigned long long)tot);
}

// MISWeight: the balance heuristic over every strategy that could have made the same path, from
// the ratio chain of forward and reverse densities; the connection endpoints' densities (and the
// resampled endpoint of s = 1 or t = 1) replace the stored ones for the evaluation.  qs / pt: the
// connected light and camera vertices (s, t > 0), qsm / ptm the ones before them (s, t > 1).
template <int LM>
__device__ real bdpt_mis(const SceneView& sv, const BCam& cam, const BdptBuf& buf, int k, int maxb, int s, int t,
                         const BVert& qs, const BVert& pt, const BVert& qsm, const BVert& ptm) {
    if (s + t == 2) return 1;
    // overridden reverse densities of the four vertices around the connection
    real pt_rev = 0, ptm_rev = 0, qs_rev = 0, qsm_rev = 0;
    if (s > 0) pt_rev = bv_pdf<LM>(sv, cam, qs, s > 1 ? &qsm : nullptr, pt);
    else pt_rev = bv_pdf_light_origin(sv, pt);  // pt is an emitting surface
    if (t > 1) {
        if (s > 0) ptm_rev = bv_pdf<LM>(sv, cam, pt, &qs, ptm);
        else ptm_rev = bv_pdf_light(sv, pt, ptm);  // PdfLight of the emitting surface pt toward ptm
    }
    if (s > 0) qs_rev = bv_pdf<LM>(sv, cam, pt, t > 1 ? &ptm : nullptr, qs);
    if (s > 1) qsm_rev = bv_pdf<LM>(sv, cam, qs, &pt, qsm);
    const uint32_t delta = buf.delta[k];
    auto remap0 = [](real f) -> real { return f != 0 ? f : 1; };
    real sum = 0, ri = 1;
    for (int i = t - 1; i > 0; --i) {
        const float2 w = __ldg(buf.pdf + (size_t)(i - 1) * buf.cap + k);
        const real rev = i == t - 1 ? pt_rev : (i == t - 2 ? ptm_rev : w.y);
        ri *= remap0(rev) / remap0(w.x);
        const bool d_i = i == t - 1 ? false : ((delta >> i) & 1u) != 0;
        const bool d_im = ((delta >> (i - 1)) & 1u) != 0;
        if (!d_i && !d_im) sum += ri;
    }
    ri = 1;
    for (int i = s - 1; i >= 0; --i) {
        const float2 w = __ldg(buf.pdf + (size_t)(maxb + 1 + i) * buf.cap + k);
        const real fwd = s == 1 ? qs.pdf_fwd : w.x;  // s = 1: the resampled light point
        const real rev = i == s - 1 ? qs_rev : (i == s - 2 ? qsm_rev : w.y);
        ri *= remap0(rev) / remap0(fwd);
        const bool d_i = i == s - 1 ? false : ((delta >> (16 + i)) & 1u) != 0;
        bool d_light;
        if (i > 0) {
            d_light = ((delta >> (16 + i - 1)) & 1u) != 0;
        } else if (s == 1) {
            d_light = bv_delta_light(sv, qs);
        } else {
            const uint32_t li = __ldg(buf.vert + ((size_t)(maxb + 1) * bv_words<LM>() + 1) * buf.cap + k).w;
            d_light = sv.lights[li].kind == 2;
        }
        if (!d_i && !d_light) sum += ri;
    }
    return 1 / (1 + sum);
}

// Film writes: a camera sample through the reference's Gaussian filter (Camera::addSample), with
// its footprint and table lookup; a light-to-camera splat through the same footprint and weights,
// without a weight sum: the resolve divides it by the weight the camera samples of spp per pixel
// put on that pixel in expectation (film_weight_1d), so that both parts estimate the same filtered
// image, borders included.
__device__ __forceinline__ void bdpt_add_sample(const SceneView& sv, const RenderParams& rp, real pfx, real pfy, Spec L) {
    const int W = sv.width, H = sv.height;
    const int px0 = max((int)xceil(pfx - 1.0f), 0), py0 = max((int)xceil(pfy - 1.0f), 0);
    const int px1 = min((int)xfloor(pfx + 1.0f) + 1, W), py1 = min((int)xfloor(pfy + 1.0f) + 1, H);
    for (int y = py0; y < py1; ++y)
        for (int x = px0; x < px1; ++x) {
            const real fdx = xabs((x - pfx - 0.5f) * 1.0f * 16);
            const real fdy = xabs((y - pfy - 0.5f) * 1.0f * 16);
            const int ix = min((int)xfloor(fdx), 15), iy = min((int)xfloor(fdy), 15);
            const real wgt = __ldg(sv.filter + iy * 16 + ix);
            double* fp = rp.film + 4 * ((size_t)y * W + x);
            atomicAdd(fp + 0, (double)(L.r * wgt));
            atomicAdd(fp + 1, (double)(L.g * wgt));
            atomicAdd(fp + 2, (double)(L.b * wgt));
            atomicAdd(fp + 3, (double)wgt);
        }
}

__device__ __forceinline__ void bdpt_add_splat(const SceneView& sv, real rx, real ry, Spec L, double* splat) {
    const int W = sv.width, H = sv.height;
    const int px0 = max((int)xceil(rx - 1.0f), 0), py0 = max((int)xceil(ry - 1.0f), 0);
    const int px1 = min((int)xfloor(rx + 1.0f) + 1, W), py1 = min((int)xfloor(ry + 1.0f) + 1, H);
    for (int y = py0; y < py1; ++y)
        for (int x = px0; x < px1; ++x) {
            const real fdx = xabs((x - rx - 0.5f) * 1.0f * 16);
            const real fdy = xabs((y - ry - 0.5f) * 1.0f * 16);
            const int ix = min((int)xfloor(fdx), 15), iy = min((int)xfloor(fdy), 15);
            const real wgt = __ldg(sv.filter + iy * 16 + ix);
            double* sp = splat + 3 * ((size_t)y * W + x);
            atomicAdd(sp + 0, (double)(L.r * wgt));
            atomicAdd(sp + 1, (double)(L.g * wgt));
            atomicAdd(sp + 2, (double)(L.b * wgt));
        }
}

// only >= 0 (here and below): the single strategy s = only / 100, t = only % 100, unweighted (each strategy
// alone estimates its own paths; a debugging view of the estimator, as PBRT's visualizeStrategies).
// s = 1: the light point sampled from camera vertex pt of strategy (1, t), into qs; false: no light
// reaches pt from it.
template <int LM>
__device__ __forceinline__ bool bdpt_light_point(const SceneView& sv, const RenderParams& rp, const BdptBuf& buf, long first, int k,
                                                 int t, int only, const BVert& pt, BVert& qs, V3* wi = nullptr) {
    const uint4 h = __ldg(buf.head + k);
    // three draws for each connectible camera vertex before this one
    int i, j, s_ix;
    bdpt_pixel(rp, first + k, i, j, s_ix);
    Rng rng;
    rng.key = rp.seed + wang_hash((uint32_t)(j * sv.width + i));
    rng.sample = (uint32_t)s_ix;
    rng.draw = h.z;
    if (only < 0) rng.draw += 3u * (uint32_t)__popc((h.w >> 8) & ((1u << (t - 1)) - 1u));
    rng_resume(rng);
    real lpick;
    const int li = bdpt_pick_light(sv, rng_1d(rng), lpick);
    const F2 ul = rng_2d(rng);
    const DevLight& Lt = sv.lights[li];
    SI psi;
    psi.p = pt.p;
    psi.perr = pt.perr;
    psi.n = pt.n;
    LightSample ls;
    const bool dl = sample_li(sv, Lt, psi, ul, ls);
    if (!(ls.pdf > 0) || is_black(ls.Li)) return false;
    qs.type = BV_LIGHT;
    qs.light = li;
    qs.p = ls.p1;
    qs.n = dl ? v3(0, 0, 0) : ls.n1;
    qs.perr = ls.perr1;
    qs.beta = ls.Li / (ls.pdf * lpick);
    qs.pdf_fwd = bv_pdf_light_origin(sv, qs);
    if (wi) *wi = ls.wi;
    return true;
}

// The part of ConnectBDPT before visibility, for strategy (s, t) = strategies[blockIdx.y] and samples
// first .. first + n - 1.
// Resident blocks per SM the register budgets are cut for.  The box above: 3, 4 and 5 blocks of the
// connection and of the weight are within 2 % of each other, 6 and 10 of the rays 1 and 3 % slower
// than 8; fetching at 8 or 16 idle lanes costs the same as at 12.
constexpr int kBdptConnectBlocks = 4, kBdptShadowBlocks = 8;
template <int LM>
__global__ __launch_bounds__(kThreads, kBdptConnectBlocks) void k_bdpt_connect(const SceneView sv, const RenderParams rp,
                                                                               BdptBuf buf, const BdptStrategies st, long first,
                                                                               int n, int only) {
    const int k = blockIdx.x * kThreads + threadIdx.x;
    const int s = st.s[blockIdx.y], t = st.t[blockIdx.y];
    const int maxb = min(rp.max_bounce, kBdptMaxBounce);
    const bool in = k < n;
    const uint4 h = in ? __ldg(buf.head + k) : make_uint4(0u, 0u, 0u, 0u);
    const int n_cam = (int)(h.w & 15u), n_light = (int)((h.w >> 4) & 15u);
    const bool have = in && t <= n_cam && s <= n_light;
    const BCam cam = bdpt_camera(sv);
    Spec c = spec(0.0f);
    BVert qs, pt, ptm;
    real spx = 0, spy = 0, geo = 1;
    bool vis = false;  // the connection needs its shadow ray
    if (have) {
        if (t == 1) pt = bv_camera(cam);
        else bv_load<LM>(buf, t - 2, k, pt);
        if (t == 2) ptm = bv_camera(cam);
        else if (t > 2) bv_load<LM>(buf, t - 3, k, ptm);
        if (s == 1) qs = bv_camera(cam);  // resampled below
        else if (s > 1) bv_load<LM>(buf, maxb + s, k, qs);
        if (s == 0) {  // the camera path's end is on a light
            if (bv_is_light(pt)) c = bv_le(sv, pt, normalize(ptm.p - pt.p)) * pt.beta;
        } else if (t == 1) {  // connect the light path's end to the camera
            if (bv_connectible(qs)) {
                const V3 d = cam.o - qs.p;
                const real l2 = len2(d);
                const V3 wi = d * xsqrt(1 / l2);
                real cos_c;
                if (l2 > 0 && bdpt_raster(cam, -wi, spx, spy, cos_c)) {
                    const real pdf = l2 / cos_c;  // solid angle at qs (lens area 1)
                    pt.beta = spec(bdpt_we(cam, cos_c) / pdf);
                    // qs is a surface vertex: s >= 2 whenever t = 1
                    c = qs.beta * bv_f<LM>(qs, pt, true) * pt.beta * absdot(wi, qs.f.ns);
                    vis = !is_black(c);
                }
            }
        } else if (s == 1) {  // connect the camera path's end to a sampled light point
            if (bv_connectible(pt)) {
                V3 wi;
                if (bdpt_light_point<LM>(sv, rp, buf, first, k, t, only, pt, qs, &wi)) {
                    c = pt.beta * bv_f<LM>(pt, qs, false) * qs.beta;
                    c = c * absdot(wi, pt.f.ns);
                    vis = !is_black(c);
                }
            }
        } else if (bv_connectible(qs) && bv_connectible(pt)) {  // connect two surface vertices (s >= 2, t >= 2)
            c = qs.beta * bv_f<LM>(qs, pt, true) * bv_f<LM>(pt, qs, false) * pt.beta;
            if (!is_black(c)) {  // generalized geometry term G with visibility
                V3 d = qs.p - pt.p;
                real g = 1 / len2(d);
                d = d * xsqrt(g);
                g *= absdot(qs.f.ns, d) * absdot(pt.f.ns, d);
                geo = g;
                vis = true;
            }
        }
    }
    // VisibilityTester::unoccluded between the vertices (offset origins as spawnRayTo), from the
    // camera path's end (t = 1 and surface connections: from the light path's)
    const bool keep = have && !is_black(c);
    const unsigned m = __ballot_sync(~0u, keep);
    if (m) {
        const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(buf.count, (uint32_t)__popc(m));
        base = __shfl_sync(~0u, base, leader);
        if (keep) {
            const uint32_t at = base + (uint32_t)__popc(m & ((1u << lane) - 1u));
            V3 org = v3(0, 0, 0), dir = v3(0, 0, 1);
            if (vis) {
                const BVert &a = t == 1 || s >= 2 ? qs : pt, &b = t == 1 || s >= 2 ? pt : qs;
                org = offset_origin(a.p, a.perr, a.n, b.p - a.p);
                dir = offset_origin(b.p, b.perr, b.n, org - b.p) - org;
            }
            buf.ray_o[at] = make_float4(org.x, org.y, org.z, __int_as_float(k));
            buf.ray_d[at] = make_float4(dir.x, dir.y, dir.z, __uint_as_float(blockIdx.y | (vis ? 0u : kConnFree)));
            if (!vis) buf.sees[at] = 1u;
        }
    }
    // geo: what a surface connection that sees is multiplied with
    if (in) buf.contrib[(size_t)blockIdx.y * buf.cap + k] = keep ? make_float4(c.r, c.g, c.b, geo) : make_float4(0, 0, 0, 0);
    const unsigned tot = __popc(__ballot_sync(~0u, vis));
    if ((threadIdx.x & 31) == 0 && tot && rp.counters) atomicAdd(rp.counters, (unsigned long long)tot);
}

// The listed rays through the 8-wide flat tree: persistent warps that fetch new rays for lanes whose
// ray has finished (as the wavefront's trace kernel).
__global__ __launch_bounds__(kThreads, kBdptShadowBlocks) void k_bdpt_shadow(const SceneView sv, const RenderParams rp, int nleaf, BdptBuf buf) {
    __shared__ uint32_t s_stack[kStack * kThreads];
    uint32_t* stack = s_stack + threadIdx.x;
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t n = *buf.count;
    Trav t;
    Work wk{0u, 0u};
    uint32_t i = 0;
    bool active = false, exhausted = false;
    constexpr int kIdle = 12;  // lanes without a ray that make the warp fetch
    for (;;) {
        const unsigned idle = __ballot_sync(~0u, !active);
        if (!exhausted && __popc(idle) >= kIdle) {
            const uint32_t take = (uint32_t)__popc(idle);
            const int leader = __ffs(idle) - 1;
            uint32_t base = 0;
            if ((int)lane == leader) base = atomicAdd(buf.count + 1, take);
            base = __shfl_sync(~0u, base, leader);
            if (base + take >= n) exhausted = true;
            i = active ? i : base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
            if (!active && i < n) {
                const float4 d = __ldcs(buf.ray_d + i);
                if (!(__float_as_uint(d.w) & kConnFree)) {
                    const float4 o = __ldcs(buf.ray_o + i);
                    active = trav_begin(true, t, sv, nleaf, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), 1 - kShadowEps, wk);
                    if (!active) buf.sees[i] = t.best == 1 ? 0u : 1u;
                }
            }
        }
        if (__ballot_sync(~0u, active) == 0u) {
            if (exhausted) break;
            continue;
        }
        for (;;) {
            if (wide_warp_step(true, active, t, sv, stack, rp.err, wk)) {
                buf.sees[i] = t.best == 1 ? 0u : 1u;
                active = false;
            }
            const unsigned act = __ballot_sync(~0u, active);
            if (act == 0u || (!exhausted && 32 - __popc(act) >= kIdle)) break;
        }
    }
}
__global__ __launch_bounds__(kThreads) void k_bdpt_shadow_any(const SceneView sv, const RenderParams rp, int nleaf, BdptBuf buf) {
    __shared__ uint32_t s_stack[kStack * kThreads];
    const uint32_t n = *buf.count;
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
        const float4 o = buf.ray_o[i], d = buf.ray_d[i];
        if (__float_as_uint(d.w) & kConnFree) continue;
        Work wk{0u, 0u};
        buf.sees[i] = scene_occluded(sv, nleaf, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), 1 - kShadowEps, s_stack + threadIdx.x, rp.err,
                                     wk) ? 0u : 1u;
    }
}

// The part of ConnectBDPT after visibility: the listed connections that see each other, weighted; t = 1
// goes to the film where it lands, the others stay for k_bdpt_film.
template <int LM>
__global__ __launch_bounds__(kThreads, kBdptConnectBlocks) void k_bdpt_weight(const SceneView sv, const RenderParams rp, BdptBuf buf,
                                                                              const BdptStrategies st, long first, int only,
                                                                              double* __restrict__ splat) {
    const uint32_t n = *buf.count;
    const int maxb = min(rp.max_bounce, kBdptMaxBounce);
    const BCam cam = bdpt_camera(sv);
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
        const int k = __float_as_int(buf.ray_o[i].w);
        const uint32_t q = __float_as_uint(buf.ray_d[i].w) & (kConnFree - 1u);
        float4* const slot = buf.contrib + (size_t)q * buf.cap + k;
        if (!buf.sees[i]) {
            *slot = make_float4(0, 0, 0, 0);
            continue;
        }
        const int s = st.s[q], t = st.t[q];
        const float4 c4 = *slot;
        Spec c{c4.x, c4.y, c4.z};
        if (s >= 2 && t >= 2) c = c * c4.w;
        BVert qs, pt, qsm, ptm;
        real spx = 0, spy = 0;
        if (t == 1) pt = bv_camera(cam);
        else bv_load<LM>(buf, t - 2, k, pt);
        if (t == 2) ptm = bv_camera(cam);
        else if (t > 2) bv_load<LM>(buf, t - 3, k, ptm);
        if (s == 1) {
            qs = bv_camera(cam);
            bdpt_light_point<LM>(sv, rp, buf, first, k, t, only, pt, qs);
        }
        if (s > 1) bv_load<LM>(buf, maxb + s, k, qs);
        if (s > 1) bv_load<LM>(buf, maxb + s - 1, k, qsm);
        if (!is_black(c) && only < 0) c = c * bdpt_mis<LM>(sv, cam, buf, k, maxb, s, t, qs, pt, qsm, ptm);
        if (t == 1) {
            real cos_c;
            const V3 d = cam.o - qs.p;
            const V3 wi = d * xsqrt(1 / len2(d));
            bdpt_raster(cam, -wi, spx, spy, cos_c);
            if (!is_black(c)) bdpt_add_splat(sv, spx, spy, c, splat);
        } else {
            *slot = make_float4(c.r, c.g, c.b, 0.f);
        }
    }
}

__global__ __launch_bounds__(kThreads) void k_bdpt_film(const SceneView sv, const RenderParams rp, BdptBuf buf,
                                                        const BdptStrategies st, int n) {
    const int k = blockIdx.x * kThreads + threadIdx.x;
    if (k >= n) return;
    Spec L = spec(0.0f);
    for (int q = 0; q < st.n; ++q) {
        if (st.t[q] == 1) continue;
        const float4 c = __ldg(buf.contrib + (size_t)q * buf.cap + k);
        L = L + Spec{c.x, c.y, c.z};
    }
    const uint4 h = __ldg(buf.head + k);
    bdpt_add_sample(sv, rp, __uint_as_float(h.x), __uint_as_float(h.y), L);
}

}  // namespace
}  // namespace lts
