// One camera sample, traced to the end in forward (loop) form.
//
// Renderer.TraceRay (Rendering/Renderer.cs:1581-1783) is recursive; the value
// it returns for the camera ray is
//     L0 = W0 * (e0 + d0 + clampInd(att0 * S(L1)))     (first vertex on a surface)
//     Lk = Wk * (ek + dk + attk * S(L(k+1)))             (deeper vertices)
// with W the segment factors (medium beta, interior Beer-Lambert), S the
// per-frame sanitize and clampInd the primary-surface indirect clamp
// (Renderer.cs:1378-1381). The loop below accumulates the same sum front to
// back: terms of the first vertex go to Lp, deeper terms to La weighted by the
// product of the attenuations after the first vertex, and the clamp is applied
// to att0 * La at the end. The RNG dimension sequence, the throughput used by
// Russian roulette and every branch decision are those of the recursion; only
// the order of the final additions differs.
#pragma once

#include "device.cuh"

namespace rt {

struct RenderConst {
    Camera cam;
    int width, height;
    int max_depth;
    float max_rad, ind_max;
    int mis_power;
    int rr_min_bounces;
    float rr_min_survival;
    int opaque;        // no material transmits shadow rays: any-hit shadows
    int dielectrics;   // a solid dielectric exists: keep the IOR stack
    int light_pick;    // RT_LIGHTS_*: 0 every light, 1 / 2 one light by power / uniformly
};

// LightDistribution.Sample (LightDistribution.cs:104-122): the light whose CDF
// entry is the first not below xi, and its pick probability.
RT_D int pick_light(const SceneView& s, int mode, float xi, float& pdf) {
    int n = s.num_lights;
    const float* cdf = s.pick_cdf + (size_t)(mode - 1) * n;
    const float* pp = s.pick_pdf + (size_t)(mode - 1) * n;
    if (n == 1) {
        pdf = pp[0];
        return 0;
    }
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi) / 2;
        if (cdf[mid] < xi) lo = mid + 1;
        else hi = mid;
    }
    pdf = pp[lo];
    return lo;
}

struct IorStackD {   // Volumetrics/IorStack.cs (capacity 8)
    float slot[8];
    int n;
    RT_D float top() const { return n == 0 ? 1.0f : slot[n - 1]; }
    RT_D float enclosing() const { return n >= 2 ? slot[n - 2] : 1.0f; }
    RT_D void push(float v) {
        if (n >= 8) {
            for (int i = 0; i < 7; i++) slot[i] = slot[i + 1];
            slot[7] = v;
            return;
        }
        slot[n++] = v;
    }
    RT_D void pop() {
        if (n > 0) n--;
    }
};

RT_D float shadow_terminator(V3 ng, V3 ns, V3 w) {   // Core/MathUtils.cs:44-61
    float ng_w = dot(ng, w);
    if (ng_w <= 0.0f) return 0.0f;
    float ns_w = dot(ns, w);
    if (ns_w <= 0.0f) return 0.0f;
    float ng_ns = dot(ng, ns);
    if (ng_ns >= 0.9999f) return 1.0f;
    float g = ng_w / (ns_w * fmaxf(ng_ns, 1e-4f));
    if (g >= 1.0f) return 1.0f;
    if (g <= 0.0f) return 0.0f;
    float g2 = g * g;
    return (-g2 * g) + g2 + g;
}

// Renderer.WeightEmission (:1549-1565). Out of line: it runs only when a ray
// hits an emitter, and keeping it out of the shading code that every vertex
// runs eases the instruction cache (wavefront shade -1.7%, megakernel -6.8%
// per frame on the icosphere field).
__device__ __noinline__ V3 weight_emission(const SceneView& s, const RenderConst& rc, V3 raw, int mat, V3 o, V3 d, float prev_pdf,
                        int prev_delta) {
    if (prev_delta) return raw;
    int li = s.emitter_light[RT_IX(mat, s.n_materials)];
    if (li >= 0) {
        float pl = light_pdf(s, s.lights[RT_IX(li, s.num_lights)], o, d);
        if (prev_pdf + pl <= 1e-20f) return v3(0.0f);
        return raw * mis_weight(prev_pdf, pl, rc.mis_power);
    }
    return raw;
}

// SampleSky (Renderer.cs:1820-1861) for a flat sky: its radiance, MIS-weighted
// against the EnvironmentLight's uniform-sphere pdf unless the bounce before
// was delta (or no EnvironmentLight samples the sky).
RT_D V3 weight_sky(const SceneView& s, const RenderConst& rc, float prev_pdf, int prev_delta) {
    if (prev_delta || s.env_light < 0) return s.sky;
    float pl = 1.0f / (4.0f * kPi);   // EnvironmentLight.PdfSolidAngle -> FlatSky.Pdf
    if (prev_pdf + pl <= 1e-20f) return v3(0.0f);
    return s.sky * mis_weight(prev_pdf, pl, rc.mis_power);
}

// Path state carried from vertex to vertex. The megakernel and the adjoint's
// replay keep it whole; the forward wavefront's shade keeps the part a vertex
// works on (LeanPath, wavefront.cuh), with the same members shade_vertex uses.
struct PathState {
    V3 o, d;          // current ray
    V3 beta;          // path throughput used by RR and the dead-path test
    V3 w;             // weight of the next vertex's terms (segment factors x attenuations)
    V3 lp, la;        // first-vertex terms; deeper terms relative to att0
    V3 pre, att0;     // first-vertex weight and attenuation (primary clamp)
    V3 cur_abs;       // interior Beer-Lambert sigma_a of the current segment
    V3 mask;          // channels still live in la (per-frame sanitize)
    float prev_pdf;
    int prev_delta;
    int first;        // no scattering vertex yet
    int clamp_mode;   // the first vertex was a surface
    int depth;        // TraceRay depth of the next segment
    Sampler rng;
    IorStackD iors;

    // Adds a term of the current vertex (already weighted) to lp or la.
    RT_D void add(V3 x, int to_la) {
        if (!to_la) {
            lp = lp + x;
            return;
        }
        if (!isfinite(x.x)) mask.x = 0.0f;
        if (!isfinite(x.y)) mask.y = 0.0f;
        if (!isfinite(x.z)) mask.z = 0.0f;
        la = la + v3(mask.x != 0.0f ? x.x : 0.0f, mask.y != 0.0f ? x.y : 0.0f, mask.z != 0.0f ? x.z : 0.0f);
    }
    RT_D float ior_top() const { return iors.top(); }
    RT_D float ior_enclosing() const { return iors.enclosing(); }
    RT_D void ior_push(float v) { iors.push(v); }
    RT_D void ior_pop() { iors.pop(); }
    // The first surface vertex: its weight and attenuation, for the primary clamp.
    RT_D void set_primary(V3 att) {
        pre = w;
        att0 = att;
    }
};

// Camera sample setup (Renderer.cs:615-653): pixel seed, 2 jitter draws,
// pinhole ray (Camera.cs:127-139).
RT_D void path_init(PathState& ps, const RenderConst& rc, int px, int py, uint32_t sample_index) {
    uint32_t seed = ((uint32_t)px * 73856093u) ^ ((uint32_t)py * 19349663u);
    ps.rng = Sampler{seed, sample_index, 0u};
    float ju = ps.rng.next();
    float jv = ps.rng.next();
    float u = ((float)px + ju) / (float)rc.width;
    float v = ((float)(rc.height - py - 1) + jv) / (float)rc.height;
    V3 target = rc.cam.llc + u * rc.cam.horizontal + v * rc.cam.vertical;
    ps.o = rc.cam.origin;
    ps.d = target - rc.cam.origin;
    ps.beta = v3(1.0f);
    ps.w = v3(1.0f);
    ps.lp = v3(0.0f);
    ps.la = v3(0.0f);
    ps.pre = v3(1.0f);
    ps.att0 = v3(0.0f);
    ps.cur_abs = v3(0.0f);
    ps.mask = v3(1.0f);
    ps.prev_pdf = 0.0f;
    ps.prev_delta = 1;
    ps.first = 1;
    ps.clamp_mode = 0;
    ps.depth = rc.max_depth;
    ps.iors.n = 0;
}

// Entry test of TraceRay (Renderer.cs:1589-1603): depth and dead path.
template <class PS>
RT_D bool path_alive(const PS& ps) {
    return ps.depth > 0 && max3(ps.beta) >= 1e-4f;
}

// The clamped sample radiance (ClampRadianceIndirect at the primary surface,
// then ClampRadiance; Renderer.cs:670, 1380-1381).
RT_D V3 path_resolve(const PathState& ps, const RenderConst& rc) {
    V3 L = ps.lp;
    if (ps.clamp_mode) L = L + ps.pre * clamp_lum(ps.att0 * sanitize(ps.la), rc.ind_max);
    return clamp_lum(L, rc.max_rad);
}

// Russian roulette on the projected throughput (Renderer.cs:1283-1294).
// q_used: the survival probability a surviving path was drawn against, 0 when
// the roulette did not run.
RT_D bool russian_roulette(const RenderConst& rc, int depth, V3& att, V3& next_beta, Sampler& rng, float& q_used) {
    int used = rc.max_depth - depth;
    q_used = 0.0f;
    if (used >= rc.rr_min_bounces) {
        float q = fmaxf(next_beta.x, fmaxf(next_beta.y, next_beta.z));
        q = fmaxf(q, rc.rr_min_survival);
        q = fminf(q, 0.95f);
        if (rng.next() > q) return false;
        q_used = q;
        float inv = 1.0f / q;
        att = att * inv;
        next_beta = next_beta * inv;
    }
    return true;
}

RT_D V3 bl_factor(V3 sigma, float t) { return beer_lambert(v3(1.0f), sigma, t); }

// Adjoint hooks. shade_vertex reports every factor that multiplies the path
// weight and every term it adds, so that the path-replay adjoint can run the
// same code; the forward sinks inherit these empty versions, which compile
// away.
enum : int { SEG_ABSORPTION = 0, SEG_MEDIUM_PASS = 1, SEG_MEDIUM_SCATTER = 2 };
enum : int { SCATTER_SAMPLED = 0, SCATTER_DELTA = 1, SCATTER_LEGACY = 2 };
struct NoAdjoint {
    // ps.w is about to be multiplied by the factors of a segment of length t:
    // interior Beer-Lambert (all modes but SEG_MEDIUM_PASS) and the medium.
    template <class PS>
    RT_D void segment(const PS&, float, int) {}
    // The interior absorption now belongs to material `mat` (-1: none).
    RT_D void interior(int) {}
    // An emitted-radiance term ps.w * we was just added.
    template <class PS>
    RT_D void emission(const PS&, int, V3, int) {}
    // A surface NEE sample: the term coef * brdf * term * tr_m * tr went through shadow().
    template <class PS>
    RT_D void nee_surface(const PS&, int, const Material&, const Surface&, V3, V3, float, V3, float, V3,
                          int) {}
    template <class PS>
    RT_D void nee_medium(const PS&, int, float, int) {}
    // A path survived Russian roulette drawn against q = clamp(max(thr)); its
    // throughput now carries 1/q. first: the roulette of the first surface
    // vertex (whose attenuation becomes att0).
    template <class PS>
    RT_D void roulette(const PS&, V3, float, int) {}
    // The vertex attenuation: att_pre before Russian roulette, att after. For
    // the legacy path, the lobe and direction of the null sample before it.
    template <class PS>
    RT_D void scatter(const PS&, const Material&, const Surface&, V3, V3, int, int, float, V3, V3, int, V3) {}

    // Capture hooks (the AOV probe, Renderer.cs:1051-1054, 1139-1145,
    // 1271-1277, 1657-1662, 1716-1724, 1849-1850). None of them draws from
    // the sampler, so a capturing render traces the same paths.
    // The closest hit of the current ray (d its direction).
    RT_D void aov_ray(const Hit&, V3) {}
    // A medium scattering event at distance t along direction d.
    RT_D void aov_medium(float, V3) {}
    // The ray left the scene (the flat sky's radiance).
    RT_D void aov_miss(V3) {}
    // The surface ShadeSurface is about to shade.
    RT_D void aov_surface(V3, const Material&) {}
    // The bounce decision: a delta lobe with attenuation f, or a non-delta one.
    RT_D void aov_bounce(bool, V3) {}
};

// One vertex of TraceRay given the closest hit of the current ray: the
// volumetric branch (Renderer.cs:1704-1782), ShadeSurface (:1008-1228) and
// ShadeSampleBounce (:1235-1383). Returns true when the path continues with
// ps.o/ps.d as the next ray (ps.depth already decremented). MEDIUM = false
// compiles the volumetric branch out; TRANSMIT = false the specular
// transmission lobe, the interior absorption it starts and the IOR stack (no
// material has specTrans > 0).
//
// The vertex's draws run through one loop: a turn per light sample (NEE:
// ComputeDirectLighting :1894-2036 and, at a medium scattering point,
// ComputeDirectLightingMedium :2099-2206, over every light or one picked
// light), then one for Sample and, when that is null, one for the legacy
// Scatter draw (:1127-1225). The turns share their two Sobol draws, the light
// samplers and the BSDF's evaluation, so each long stretch of code is compiled
// once and the lanes of a warp run it together: shading is bound by
// instruction supply (with a copy of the evaluation and the samplers at each of
// their uses, shade took 8.9 against 7.2 ms on a Cornell box of 256x256x64
// samples and 62.3 against 52.3 ms on four foggy views of 256x256x64). The NEE
// integrand and its MIS weight are evaluated
// before the shadow ray and the ray is dropped when they are zero (the
// reference casts it first; only the cost differs: every draw happens in the
// light sampler).
template <bool MEDIUM = true, bool TRANSMIT = true, class PS, class Sink>
__device__ __forceinline__ bool shade_vertex(const SceneView& s, const RenderConst& rc, PS& ps, const Hit& h,
                                             Sink& sink) {
    bool hit = h.kind != HIT_NONE;
    V3 beta_s = ps.beta;   // the throughput at the vertex
    sink.aov_ray(h, ps.d);
    bool med = false;      // a medium scattering vertex
    Surface rec;
    if (MEDIUM && s.has_medium) {
        float tmax = hit ? h.t : 1e30f;
        float tmed;
        V3 mb;
        med = medium_sample(s, tmax, ps.rng, tmed, mb);
        if (med) {
            rec.p = ps.o + ps.d * tmed;
            rec.n = v3(0.0f);
            sink.aov_medium(tmed, ps.d);
            sink.segment(ps, tmed, SEG_MEDIUM_SCATTER);
            if constexpr (TRANSMIT) ps.w = ps.w * bl_factor(ps.cur_abs, tmed);
            ps.w = ps.w * mb;
        } else {
            sink.segment(ps, tmax, SEG_MEDIUM_PASS);
            ps.w = ps.w * mb;
        }
        beta_s = ps.beta * mb;
    }
    V3 view;
    const Material* mp = s.materials;
    BsdfView bv;
    float rel_eta = 0.0f;
    bool dielectric = false;
    if (!MEDIUM || !med) {
        if (!hit) {   // SampleSky, then TraceRay's Beer-Lambert over an infinite segment
            if (s.sky_on) {
                V3 x = ps.w * weight_sky(s, rc, ps.prev_pdf, ps.prev_delta);
                if constexpr (TRANSMIT) x = x * bl_factor(ps.cur_abs, INFINITY);
                ps.add(x, ps.clamp_mode);
            }
            sink.aov_miss(s.sky);
            return false;
        }
        sink.segment(ps, h.t, SEG_ABSORPTION);
        if constexpr (TRANSMIT) ps.w = ps.w * bl_factor(ps.cur_abs, h.t);
        rec = make_surface(s, h, ps.o, ps.d);
        mp += rec.material;
        sink.aov_surface(rec.n, *mp);
        if (mp->type != 0) {   // Emissive: Emit (front face only), no NEE, no scatter
            int to_la = ps.clamp_mode;
            V3 em = mp->emission;
            if (rec.front && (em.x > 0.0f || em.y > 0.0f || em.z > 0.0f)) {
                V3 we = weight_emission(s, rc, em, rec.material, ps.o, ps.d, ps.prev_pdf, ps.prev_delta);
                ps.add(ps.w * we, to_la);
                sink.emission(ps, rec.material, we, to_la);
            }
            return false;
        }
        view = normalize(-ps.d);
        if constexpr (TRANSMIT) {
            dielectric = !mp->thin_walled && mp->spec_trans_raw > 0.0f;
            if (dielectric) rel_eta = rec.front ? (ps.ior_top() / mp->ior_raw) : (mp->ior_raw / ps.ior_enclosing());
        }
        bv = bsdf_view(*mp, rec, view);
    }
    const Material& m = *mp;
    const int to_la = ps.clamp_mode;
    int li = 0, l1 = s.num_lights, si = 0;
    float p_pick = 1.0f, inv_pick = 1.0f;
    if (rc.light_pick && l1 > 0) {   // single-light picking (Renderer.cs:1907-1974, 2110-2160): lightAccum / pPick
        li = pick_light(s, rc.light_pick, ps.rng.next(), p_pick);
        l1 = li + 1;
        inv_pick = p_pick > 0.0f ? 1.0f / p_pick : 0.0f;
    }
    BsdfSample bs;
    bs.transition = 0;
    bs.has_next_absorption = 0;
    V3 att, sdir;
    int lobe = -1, pass = 0;
#pragma unroll 1
    for (;;) {
        while (li < l1 && si >= s.lights[RT_IX(li, s.num_lights)].shadow_samples) {
            li++;
            si = 0;
        }
        const bool nee = li < l1;
        if (MEDIUM && !nee && med) break;
        const Light* l = nullptr;
        V3 vs;   // ScatterInternal's view vector
        bool two;
        if (nee) {
            l = s.lights + RT_IX(li, s.num_lights);
            two = light_two_draws(*l);
        } else {
            vs = normalize(pass == 0 ? view : -ps.d);
            lobe = bsdf_pick_lobe<TRANSMIT>(m, ps.rng.next());
            two = bsdf_two_draws<TRANSMIT>(m, rec, vs, lobe);
        }
        float u1 = 0.0f, u2 = 0.0f;
        if (two) {
            u1 = ps.rng.next();
            u2 = ps.rng.next();
        }
        LightSample ls;
        V3 L;
        if (nee) {
            ls = light_sample(s, *l, rec.p, rec.n, si, u1, u2, ps.rng);
            si++;
            if (ls.occluded || !ls.has_ray) continue;
            L = ls.dir;
        } else {
            V3 tried = rec.n;
            bool ok = bsdf_scatter<TRANSMIT>(m, rec, bv.fr, vs, pass == 0 ? -view : ps.d, rel_eta, lobe, u1, u2, ps.rng,
                                             att, sdir, tried);
            if (pass == 1) {   // the legacy draw ends the vertex either way
                if (!ok) return false;
                break;
            }
            bs.lobe = lobe;
            bs.tried = tried;
            int kind = ok ? bsdf_sample_kind<TRANSMIT>(m, rec, att, sdir, lobe, bs) : SAMPLE_NULL;
            if (kind == SAMPLE_NULL) {
                pass = 1;
                continue;
            }
            if (kind == SAMPLE_DELTA) break;
            L = sdir;
        }
        V3 f;
        float pb;   // the density of L under the vertex's own sampler
        if (MEDIUM && med) {
            pb = hg_eval(s.hg_g, ps.d, L);
        } else {
            bsdf_eval_pdf(m, rec, bv, L, nee, f, pb);
            if (!nee) {
                bsdf_sample_value(att, f, pb, lobe, bs);
                break;
            }
        }
        float term = 1.0f;
        if (!MEDIUM || !med) {
            term = shadow_terminator(rec.n, rec.n, view) * shadow_terminator(rec.n, rec.n, L);
            f = f * term;
            if (is_zero(f)) {
                sink.skipped(offset_origin(rec.p, rec.n), L, ls.ray_tmax);
                continue;
            }
        }
        V3 tr_m = v3(1.0f);
        if (MEDIUM && s.has_medium) tr_m = medium_tr(s, ls.dist >= kInf ? 1e30f : ls.dist);
        float wgt = 1.0f;
        if (!l->is_delta && pb > 0.0f) {
            float pl = p_pick * light_pdf(s, *l, rec.p, L);   // pNee = pPick * pLightSample
            if (pl + pb > 0.0f) wgt = mis_weight(pl, pb, rc.mis_power);
        }
        wgt *= inv_pick;
        V3 wc = wgt * ls.color;
        V3 c = (MEDIUM && med) ? wc * pb : wc * f;
        if (MEDIUM) c = c * tr_m;
        sink.shadow(ps, li, offset_origin(rec.p, rec.n), L, ls.ray_tmax, ps.w * c, to_la);
        if (MEDIUM && med) sink.nee_medium(ps, li, ls.dist, to_la);
        else sink.nee_surface(ps, li, m, rec, L, view, term, ps.w * wc, ls.dist, tr_m, to_la);
    }
    if (MEDIUM && med) {
        int used = rc.max_depth - ps.depth;
        float scale = 1.0f;
        if (used >= rc.rr_min_bounces) {
            float q = fmaxf(beta_s.x, fmaxf(beta_s.y, beta_s.z));
            q = fmaxf(q, rc.rr_min_survival);
            q = fminf(q, 0.95f);
            if (ps.rng.next() > q) return false;
            scale = 1.0f / q;
            sink.roulette(ps, beta_s, q, 0);
        }
        float ppdf;
        V3 wi = hg_sample(s.hg_g, ps.d, ps.rng, ppdf);
        float pv = hg_eval(s.hg_g, ps.d, wi);
        float pw = ppdf > 1e-20f ? pv / ppdf : 0.0f;
        ps.beta = beta_s * (pw * scale);
        ps.w = ps.w * (pw * scale);
        ps.o = rec.p;
        ps.d = wi;
        ps.prev_pdf = ppdf;
        ps.prev_delta = 0;
        ps.first = 0;   // a medium first vertex: no primary clamp
        ps.depth -= 1;
        return path_alive(ps);
    }
    const bool sampled = pass == 0;   // ShadeSampleBounce, else the legacy Scatter path
    if (sampled) {
        if (bs.is_delta) {
            att = bs.f;
        } else {
            float a = fabsf(dot(rec.n, bs.wo));
            if (a <= 0.0f || bs.pdf <= 0.0f) return false;
            att = bs.f * a / bs.pdf;
        }
        sink.aov_bounce(bs.is_delta, bs.f);
        sdir = bs.wo;
    } else {
        sink.aov_bounce(false, att);   // Disney's IsDeltaScatter is false
    }
    V3 next_beta = beta_s * att;
    V3 att_pre = att, thr = next_beta;
    float q_rr;
    if (!russian_roulette(rc, ps.depth, att, next_beta, ps.rng, q_rr)) return false;
    if (q_rr > 0.0f) sink.roulette(ps, thr, q_rr, ps.first);
    if (sampled) {
        sink.scatter(ps, m, rec, view, bs.wo, bs.lobe, bs.is_delta ? SCATTER_DELTA : SCATTER_SAMPLED, bs.pdf, att_pre,
                     att, -1, bs.wo);
        V3 off = dot(sdir, rec.n) >= 0.0f ? rec.n : -rec.n;
        ps.o = offset_origin(rec.p, off);
        ps.prev_pdf = bs.is_delta ? 0.0f : bs.pdf;
        ps.prev_delta = bs.is_delta;
        if constexpr (TRANSMIT) {
            if (bs.has_next_absorption) {
                ps.cur_abs = bs.next_absorption;
                sink.interior(near_zero(bs.next_absorption) ? -1 : rec.material);
            }
            if (rc.dielectrics && bs.transition == 1) ps.ior_push(dielectric ? m.ior_raw : ps.ior_top());
            if (rc.dielectrics && bs.transition == 2) ps.ior_pop();
        }
    } else {
        sink.scatter(ps, m, rec, view, sdir, lobe, SCATTER_LEGACY, 1.0f, att_pre, att, bs.lobe, bs.tried);
        ps.o = rec.p;
        ps.prev_pdf = 0.0f;
        ps.prev_delta = 0;
        if constexpr (TRANSMIT) {
            if (rc.dielectrics && dielectric && dot(sdir, rec.n) < 0.0f) {
                if (rec.front) ps.ior_push(m.ior_raw);
                else ps.ior_pop();
            }
        }
    }
    ps.d = sdir;
    if (ps.first) {   // primary surface: deeper terms are clamped as one (:1380-1381)
        ps.first = 0;
        ps.clamp_mode = 1;
        ps.set_primary(att);
        ps.w = v3(1.0f);
    } else {
        ps.w = ps.w * att;
    }
    ps.beta = next_beta;
    ps.depth -= 1;
    return path_alive(ps);
}

// Shadow sink of the megakernel: traces the shadow ray at once.
template <int STACK>
struct InlineShadows : NoAdjoint {
    const SceneView* s;
    int opaque;
    Counters* cnt;
    int* err;
    RT_D void shadow(PathState& ps, int, V3 o, V3 d, float tmax, V3 c, int to_la) {
        V3 tr = shadow_transmittance<STACK>(*s, opaque, o, d, kEps, tmax, cnt, err);
        if (near_zero(tr)) return;
        ps.add(c * tr, to_la);
    }
    // A shadow ray the reference casts but whose contribution is zero: traced
    // only by the counting build, so the work counts are the reference's.
    RT_D void skipped(V3 o, V3 d, float tmax) {
        if (cnt) shadow_transmittance<STACK>(*s, opaque, o, d, kEps, tmax, cnt, err);
    }
};

// Traces one camera sample of pixel (px, py) to the end and returns the
// clamped sample radiance. cnt (counting builds only) accumulates the work.
template <int STACK, bool COUNT>
__device__ V3 trace_sample(const SceneView& s, const RenderConst& rc, int px, int py, uint32_t sample_index,
                           Counters* cnt, int* err) {
    if (!COUNT) cnt = nullptr;
    PathState ps;
    path_init(ps, rc, px, py, sample_index);
    InlineShadows<STACK> sink{{}, &s, rc.opaque, cnt, err};
    while (path_alive(ps)) {
        Hit h;
        if (COUNT) cnt->closest_rays++;
        traverse<false, STACK>(s, ps.o, ps.d, kEps, kInf, h, COUNT ? &cnt->closest : nullptr, err);
        if (!shade_vertex(s, rc, ps, h, sink)) break;
    }
    return path_resolve(ps, rc);
}

// The AOV probe of one camera path (Renderer.cs:776-815): depth at the camera
// ray's first surface hit; albedo and normal at the first non-delta surface,
// with a specular chain's tint folded into weight; a medium scatter commits
// white with no normal, a miss the (black) sky.
struct AovProbe {
    bool pending, have_depth, camera;
    float depth;
    V3 weight, tent_albedo, tent_normal, albedo, normal;
    RT_D void reset() {
        pending = true;
        have_depth = false;
        camera = true;
        depth = -1.0f;
        weight = v3(1.0f);
        tent_albedo = v3(1.0f);
        tent_normal = v3(0.0f);
        albedo = v3(0.0f);
        normal = v3(0.0f);
    }
    RT_D void commit() {
        albedo = weight * tent_albedo;
        normal = tent_normal;
        pending = false;
    }
    RT_D void commit_as(V3 a, V3 n) {
        albedo = weight * a;
        normal = n;
        pending = false;
    }
};

RT_D V3 clamp01(V3 v) {   // Vector3.Clamp(v, Zero, One)
    return v3(fminf(fmaxf(v.x, 0.0f), 1.0f), fminf(fmaxf(v.y, 0.0f), 1.0f), fminf(fmaxf(v.z, 0.0f), 1.0f));
}

// The megakernel's shadow sink plus the capture hooks on a probe.
template <int STACK>
struct CaptureShadows : InlineShadows<STACK> {
    AovProbe* probe;
    RT_D void aov_ray(const Hit& h, V3 d) {
        AovProbe& p = *probe;
        if (p.camera && h.kind != HIT_NONE && p.pending && !p.have_depth) {   // :1657-1662
            p.depth = h.t * length(d);
            p.have_depth = true;
        }
        p.camera = false;
    }
    RT_D void aov_medium(float t, V3 d) {   // :1716-1724
        AovProbe& p = *probe;
        if (!p.pending) return;
        if (!p.have_depth) {
            p.depth = t * length(d);
            p.have_depth = true;
        }
        p.commit_as(v3(1.0f), v3(0.0f));
    }
    RT_D void aov_miss(V3 sky) {   // :1849-1850
        if (probe->pending) probe->commit_as(clamp01(sky), v3(0.0f));
    }
    RT_D void aov_surface(V3 n, const Material& m) {   // :1051-1054
        if (!probe->pending) return;
        probe->tent_normal = n;
        probe->tent_albedo = clamp01(m.base);   // AovAlbedo: baseColor, or an Emissive's colour
    }
    RT_D void aov_bounce(bool delta, V3 f) {   // :1139-1145, 1271-1277
        if (!probe->pending) return;
        if (delta) probe->weight = probe->weight * clamp01(f);
        else probe->commit();
    }
};

// trace_sample with the probe: returns the clamped sample radiance and leaves
// the path's committed features in *probe.
template <int STACK>
__device__ V3 trace_capture(const SceneView& s, const RenderConst& rc, int px, int py, uint32_t sample_index,
                            AovProbe* probe, int* err) {
    PathState ps;
    path_init(ps, rc, px, py, sample_index);
    probe->reset();
    CaptureShadows<STACK> sink{{{}, &s, rc.opaque, nullptr, err}, probe};
    while (path_alive(ps)) {
        Hit h;
        traverse<false, STACK>(s, ps.o, ps.d, kEps, kInf, h, nullptr, err);
        if (!shade_vertex(s, rc, ps, h, sink)) break;
    }
    if (probe->pending) probe->commit();   // CaptureAccumulator.Add (:835-837)
    return path_resolve(ps, rc);
}

}  // namespace rt
