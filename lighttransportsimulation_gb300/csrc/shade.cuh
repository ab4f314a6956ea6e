// What the wavefront's shade stage and the megakernels share: the sampler's resume, the pixel
// order, one vertex's scattering, and the traversal of a warp's rays in step.
#pragma once

#include "tracer_dev.cuh"

namespace lts {
namespace {

// Resume a (pixel, sample) stream at draw `draw` (regenerates the current Philox block).
__device__ __forceinline__ void rng_resume(Rng& r) {
    const uint32_t k = r.draw & 3u;
    if (k == 0u) return;
    const uint32_t d = r.draw;
    r.draw = d & ~3u;
    philox_block(r);
    r.draw = d;
    for (uint32_t q = 0; q < k; ++q) {
        r.w0 = r.w1;
        r.w1 = r.w2;
        r.w2 = r.w3;
    }
}

// Order in which a slice's samples of one sample index visit the crop's pixels: 8 x 4 tiles
// (one warp each) left to right in bands of four rows, so the rays a warp traces start from a
// compact patch of the image instead of a 32 x 1 strip (partial tiles at the right and bottom
// edges are row-major).  Position k in 0 .. cw * ch - 1 -> crop pixel (ci, cj).
#ifndef LTS_PIXEL_TILES
#define LTS_PIXEL_TILES 1  // 0: row-major pixel order
#endif
constexpr int kTileW = 8, kTileH = 4;
__device__ __forceinline__ void tile_pixel(long k, int cw, int ch, int& ci, int& cj) {
    if (!LTS_PIXEL_TILES) {
        ci = (int)(k % cw);
        cj = (int)(k / cw);
        return;
    }
    const long band_px = (long)kTileH * cw;
    const int band = (int)(k / band_px);
    const int rows = min(kTileH, ch - band * kTileH);
    const int o = (int)(k - band * band_px);
    const int full = cw / kTileW, tile_px = kTileW * rows;
    if (o < full * tile_px) {
        const int tx = o / tile_px, r = o - tx * tile_px;
        ci = tx * kTileW + r % kTileW;
        cj = band * kTileH + r / kTileW;
    } else {  // the narrower last tile of the band
        const int rem = cw - full * kTileW, r = o - full * tile_px;
        ci = full * kTileW + r % rem;
        cj = band * kTileH + r / rem;
    }
}

// One vertex of PathTracingIntegrator::evaluate after its material is known
// (PathTracingIntegrator.cuh:77-103, IntegratorHelper.cuh:51-149): the light sample's shadow ray
// and weight, the MIS BSDF ray and weight, the path's next ray, throughput and Russian roulette.
// `out` receives the rays (nee: this vertex samples a light; shadow, mis, ray); `sig` records the
// events of the light evaluation, ev_mis / ev_main those the caller mixes in later.  Returns true
// when the path ends here.
template <bool RECORD, int LM, class Out>
__device__ __forceinline__ bool shade_scatter(const SceneView& sv, const RenderParams& rp, const SI& si, const Bsdf& f,
                                              int bounce, Spec& beta, bool& specular, Rng& rng, Out& out, EvSink* sig,
                                              uint64_t& ev_mis, uint64_t& ev_main) {
    bool done = false;
    if (sv.nlight > 0) {
        const float ul = rng_1d(rng);
        int off = 0;
        {
            const int size = sv.nlight;
            if (size != 1) {
                int first = 0, len = size;
                while (len > 0) {
                    const int half = len >> 1, middle = first + half;
                    if (__ldg(sv.light_cdf + middle) <= ul) {
                        first = middle + 1;
                        len -= half + 1;
                    } else {
                        len = half;
                    }
                }
                off = (int)clampf((float)(first - 1), 0.0f, (float)(size - 2));
            }
        }
        const float lpdf_sel = __ldg(sv.light_func + off) / (sv.light_func_int * sv.nlight);
        out.nee(beta, lpdf_sel);
        const F2 ulight = rng_2d(rng);
        const F2 uscat = rng_2d(rng);
        const DevLight& Lt = sv.lights[off];
        const uint32_t fl = specular ? BSDF_ALL : (BSDF_ALL & ~BSDF_SPECULAR);
        LightSample ls;
        const bool delta = sample_li(sv, Lt, si, ulight, ls);
        if (ls.pdf > 0 && !is_black(ls.Li)) {
            const Spec fv = bsdf_f<LM>(f, si.wo, ls.wi, fl, sig) * absdot(ls.wi, si.sn);
            const float spdf = bsdf_pdf<LM>(f, si.wo, ls.wi, fl, sig);
            if (!is_black(fv)) {
                const V3 org = offset_origin(si.p, si.perr, si.n, ls.p1 - si.p);
                const V3 tgt = offset_origin(ls.p1, ls.perr1, ls.n1, org - ls.p1);
                Spec c;
                if (delta) {
                    c = fv * ls.Li / ls.pdf;
                } else {
                    const float fp = 1 * ls.pdf, gp = 1 * spdf;
                    const float wgt = (fp * fp) / (fp * fp + gp * gp);
                    c = fv * ls.Li * wgt / ls.pdf;
                }
                const V3 dir = tgt - org;
                out.shadow(org, dir, c, !is_black(ls.Li));
            }
        }
        if (!delta) {
            V3 wi = ls.wi;
            float spdf = 0;
            uint32_t stype = 0;
            EvSink cap{nullptr, 0};
            Spec fv = bsdf_sample<LM>(f, si.wo, wi, uscat, spdf, fl, stype, RECORD ? &cap : nullptr);
            ev_mis = cap.cap;
            fv = fv * absdot(wi, si.sn);
            const bool sampled_spec = (stype & BSDF_SPECULAR) != 0;
            if (!is_black(fv) && spdf > 0) {
                float wgt = 1;
                bool skip = false;
                if (!sampled_spec) {
                    float lp;
                    if (Lt.kind == 0) lp = area_pdf(sv, Lt, si.p, si.perr, si.n, wi);
                    else if (Lt.kind == 1) lp = sph_pdf_infinite(wi);
                    else lp = 0.0f;
                    if (lp == 0) skip = true;
                    else {
                        const float fp = 1 * spdf, gp = 1 * lp;
                        wgt = (fp * fp) / (fp * fp + gp * gp);
                    }
                }
                if (!skip) {
                    const V3 org = offset_origin(si.p, si.perr, si.n, wi);
                    out.mis(org, wi, fv, wgt, spdf, off);
                }
            }
        }
    }
    // path BSDF sample, throughput, spawn, Russian roulette (PathTracingIntegrator.cuh:80-103)
    V3 wi = v3(0, 0, 0);
    float pdf = 0;
    uint32_t stype = 0;
    const F2 ub = rng_2d(rng);
    EvSink cap{nullptr, 0};
    const Spec fv = bsdf_sample<LM>(f, si.wo, wi, ub, pdf, BSDF_ALL, stype, RECORD ? &cap : nullptr);
    ev_main = cap.cap;
    if (is_black(fv) || pdf == 0) {
        done = true;
    } else {
        specular = (stype & BSDF_SPECULAR) != 0;
        beta = beta * (fv * absdot(wi, si.sn) / pdf);
        const V3 no = offset_origin(si.p, si.perr, si.n, wi);
        out.ray(no, wi);
        if (bounce >= rp.rr_start) {
            const float qq = fmaxf(0.05f, 1 - lum(beta));
            if (rng_1d(rng) < qq) done = true;
            else beta = beta / (1 - qq);
        }
        if (bounce + 1 >= rp.max_bounce) done = true;
    }
    return done;
}

#if !LTS_FP64
// Traversal of one ray per lane, the whole warp in step (every lane calls; `active` lanes hold a
// ray that trav_begin accepted): as in the wavefront's trace kernel the warp runs node visits or
// triangle tests, whichever more of its lanes wait for, so a lane's triangle tests do not hold up
// the others' node visits.  8-wide flat tree only.
__device__ __forceinline__ void trace_warp(const bool any, bool active, Trav& t, const SceneView& sv, uint32_t* stack,
                                           uint32_t* err, Work& wk) {
    for (;;) {
        if (__ballot_sync(~0u, active) == 0u) return;
        if (wide_warp_step(any, active, t, sv, stack, err, wk)) active = false;
    }
}

// Rays of a warp's lanes (on: the lane has one) against the scene; WIDE: the 8-wide flat tree, in
// step; else whichever tree the scene has, lane by lane.  ANY: t.best == 1 on a hit; else t.best is
// the closest hit's primitive (-1 none) with its barycentrics, 1 / det and distance.
template <bool ANY, bool WIDE>
__device__ __forceinline__ void warp_rays(bool on, Trav& t, const SceneView& sv, int nleaf, V3 o, V3 d, real tmax,
                                          uint32_t* stack, uint32_t* err, Work& wk) {
    t.best = -1;
    if (WIDE) {
        if (on) on = trav_begin(ANY, t, sv, nleaf, o, d, tmax, wk);
        trace_warp(ANY, on, t, sv, stack, err, wk);
        if (!ANY) t.best = hit_prim(t.best);
    } else if (on) {
        t.tmax = tmax;
        t.best = traverse<ANY, true>(sv, nleaf, make_trace_ray(o, d), t.tmax, t.bu, t.bv, t.binv, stack, err, wk);
    }
    __syncwarp();
}
#endif

}  // namespace
}  // namespace lts
