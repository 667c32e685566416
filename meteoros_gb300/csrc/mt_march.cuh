// The raymarch kernel (cloudRayMarch.comp:565-826), templated on the lanes
// per ray and on the storage of the noise volumes:
//   MT_STORAGE_U8    RGBA8 volumes, exact FP32 filtering (the plain form)
//   MT_STORAGE_F16   IEEE half volumes (precision form): the primary fetches
//                    filtered in FP32; the cone-light samples' filtering and
//                    density math (FBM, remaps, coverage) in half2, two
//                    samples per pair
//   MT_STORAGE_BF16  bfloat16 volumes, filtered in FP32 (a storage form)
// Apart from the FP16 form's cone-light density math, everything after the
// filtered texel (FBM, remaps, erosion, lighting, transmittance, radiance,
// accumulation) is FP32.  Each storage is instantiated by its own translation
// unit (mt_march_u8.cu, mt_march_f16.cu, mt_march_bf16.cu).
#pragma once
#include "mt_shared.cuh"

namespace mt {

// Storage-specific volume access.
template <int S> struct Vol;
// T3: the element of the 3D volumes (base, detail), T2: of the 2D images
// (curl, weather), as build_march_args points at them.
template <> struct Vol<MT_STORAGE_U8> {
    using T3 = uint4;  // plane quads (launch_layouts)
    using T2 = uint4;  // bilinear cells (launch_layouts)
    template <int N> static MT_HD f4v tex3(const T3* v, f3 s) { return tex3_u8<N>(v, s); }
    template <int N> static MT_HD f4v tex3_light(const T3* v, f3 s) { return tex3_u8_fused<N>(v, s); }
    template <int N> static MT_HD f4v tex2(const T2* v, float x, float y) { return tex2_u8<N>(v, x, y); }
};
// The 16-bit storages (P the packed pair type): every fetch filters the
// 16-bit texels in FP32, except the FP16 form's six cone-light samples per
// in-cloud step, which reach colour only and run in half2 (lerps and density
// math, sample_light_pair).
template <class P> struct Vol16 {
    using T3 = uint4;  // plane quads (launch_layouts)
    using T2 = uint2;
    template <int N> static MT_HD f4v tex3(const T3* v, f3 s) { return tex3_p16q_f32<N, P>(v, s); }
    // bfloat16 (an 8-bit mantissa) filters its cone-light samples in FP32 too
    template <int N> static MT_HD f4v tex3_light(const T3* v, f3 s) { return tex3_p16q_f32<N, P>(v, s); }
    template <int N> static MT_HD f4v tex2(const T2* v, float x, float y) { return tex2_p16_f32<N, P>(v, x, y); }
};
template <> struct Vol<MT_STORAGE_F16> : Vol16<__half2> {};
template <> struct Vol<MT_STORAGE_BF16> : Vol16<__nv_bfloat162> {};

// The RGBA8 form's tame frames: every special case of the density path's
// arithmetic -- operands of the reciprocals, roots and quotients far from 1, NaN
// in the clamps -- is settled by Frame::tame, so it runs on rcp_core, sqrt_core
// and saturating instructions, value for value the shader's.  (The 16-bit
// forms' compiler settings have approximations there already.)
template <int S, bool TAME> constexpr bool kExact = TAME && S == MT_STORAGE_U8;

struct Weather {
    float lo, mul, type;
    float hgrad;  // height gradient at the primary sample, shared by its light samples
    Rcp r_lo;     // {1 - lo, ~1/(1 - lo)}: the coverage remap's width (b, exact division)
                  // and an approximate reciprocal for the light samples (y)
};

template <int S> struct Tex {
    const typename Vol<S>::T3* base;
    const typename Vol<S>::T3* detail;
    const typename Vol<S>::T2* curl;
    const typename Vol<S>::T2* weather;
};
template <int S> MT_HD Tex<S> make_tex(const MarchArgs& a) {
    return Tex<S>{(const typename Vol<S>::T3*)a.vol[0], (const typename Vol<S>::T3*)a.vol[1],
                  (const typename Vol<S>::T2*)a.vol[2], (const typename Vol<S>::T2*)a.vol[3]};
}

template <int S, bool TAME>
MT_HD Weather weather_at(const mt_params& p, const Frame& F, const Tex<S>& tx, f3 pos, f3 ec) {
    Weather w;
    w.hgrad = 1.0f;
    if (p.coverage_mode == 0) {
        w.lo = p.coverage;
        w.mul = p.coverage;
        w.type = 0.0f;
    } else {
        const float2 wuv = rdiv2_step<TAME>(pos.x - ec.x, pos.z - ec.z, F.r_weather);
        f4v wd = Vol<S>::template tex2<MT_WEATHER_N>(tx.weather, wuv.x, wuv.y);
        w.lo = 1.0f - wd.x;
        w.mul = wd.x;
        w.type = wd.z;
    }
    w.r_lo = Rcp{1.0f - w.lo, kExact<S, TAME> ? rcp_approx(1.0f - w.lo) : __fdividef(1.0f, 1.0f - w.lo)};
    return w;
}

// cloudRayMarch.comp:499-540
template <int S, bool TAME>
MT_HD float sample_low_frequency(const mt_params& p, const Tex<S>& tx, f3 point, float relH, const Weather& wt) {
    f4v n = Vol<S>::template tex3<MT_BASE_N>(tx.base, point);
    if (kExact<S, TAME>) {
        const float fbm = __saturatef((n.y * 0.625f) + (n.z * 0.25f) + (n.w * 0.125f));
        const float lo = fbm - 0.9f;
        float shape = __saturatef(div_core(n.x - lo, 1.0f - lo));
        if (p.height_gradient) shape = shape * wt.hgrad;
        // 0 / 0, where the threshold is 1, saturates to 0: as empty as its NaN
        return __saturatef(div_core(fminf(fmaxf(shape, wt.lo), 1.0f) - wt.lo, wt.r_lo.b)) * wt.mul;
    }
    float fbm = (n.y * 0.625f) + (n.z * 0.25f) + (n.w * 0.125f);
    fbm = gclamp(fbm, 0.0f, 1.0f);
    float baseCloud = remap_clamped(n.x, (fbm - 0.9f), 1.0f, 0.0f, 1.0f);
    // getDensityHeightGradientForPoint(relH, type): every call of a step passes
    // the primary sample's height and weather, so it is evaluated once per step
    // (Weather::hgrad).
    if (p.height_gradient) baseCloud = baseCloud * wt.hgrad;
    // remapClampedBeforeAndAfter(baseCloud, lo, 1, 0, 1), its width 1 - lo
    // computed once per step
    float v = gclamp(baseCloud, wt.lo, 1.0f);
    float bc = gclamp(0.0f + (((v - wt.lo) / wt.r_lo.b) * (1.0f - 0.0f)), 0.0f, 1.0f);
    return bc * wt.mul;
}

// sample_low_frequency for a cone-light sample (cloudRayMarch.comp:659-666).
// Light samples reach colour only: fused lerps, the quotients as products with
// the reciprocal (the remap's varying one by the fast division) and min/max
// clamps, a few ulp from the exact sequence above.
template <int S>
MT_HD float sample_light(const mt_params& p, const Tex<S>& tx, f3 point, const Weather& wt) {
    const f4v n = Vol<S>::template tex3_light<MT_BASE_N>(tx.base, point);
    const float fbm = __saturatef(fmaf(n.w, 0.125f, fmaf(n.z, 0.25f, n.y * 0.625f)));
    const float lo = fbm - 0.9f;
    float baseCloud = __saturatef((n.x - lo) * rcp_approx(1.0f - lo));
    if (p.height_gradient) baseCloud = baseCloud * wt.hgrad;
    const float v = fminf(fmaxf(baseCloud, wt.lo), 1.0f);
    const float bc = __saturatef((v - wt.lo) * wt.r_lo.y);
    return bc * wt.mul;
}

// Two cone-light samples at once in the pair type (FP16 storage): sample i in
// the low half, sample i + 1 in the high half.  Each sample's filtered texel,
// FBM, base-shape remap, height gradient and coverage remap --
// sample_light's steps, with the division by a reciprocal -- run as half2
// arithmetic; the results return to FP32 for the erosion and the accumulation
// of the light density.  (bfloat16's 8-bit mantissa is too coarse for this:
// the bfloat16 form does its cone-light samples in FP32.)
template <class P>
MT_HD float2 sample_light_pair(const mt_params& p, const uint4* base, f3 s0, f3 s1, const Weather& wt) {
    using Q = Pair<P>;
    const PairTexel<P> n0 = tex3_p16q_pairs<MT_BASE_N, P>(base, s0);
    const PairTexel<P> n1 = tex3_p16q_pairs<MT_BASE_N, P>(base, s1);
    const P x = Q::lows(n0.rg, n1.rg), y = Q::highs(n0.rg, n1.rg);
    const P z = Q::lows(n0.ba, n1.ba), w = Q::highs(n0.ba, n1.ba);
    const P zero = Q::splat(0.0f), one = Q::splat(1.0f);
    P fbm = __hfma2(w, Q::splat(0.125f), __hfma2(z, Q::splat(0.25f), __hmul2(y, Q::splat(0.625f))));
    fbm = __hmin2(__hmax2(fbm, zero), one);
    const P lo = __hsub2(fbm, Q::splat(0.9f));
    P bc = __hmin2(__hmax2(__hmul2(__hsub2(x, lo), h2rcp(__hsub2(one, lo))), zero), one);
    if (p.height_gradient) bc = __hmul2(bc, Q::splat(wt.hgrad));
    const P wlo = Q::splat(wt.lo);
    const P v = __hmin2(__hmax2(bc, wlo), one);
    bc = __hmin2(__hmax2(__hmul2(__hsub2(v, wlo), Q::splat(wt.r_lo.y)), zero), one);
    return Q::to_float2(__hmul2(bc, Q::splat(wt.mul)));
}

// cloudRayMarch.comp:542-563.  The texture part is the same for the primary
// erosion (:645) and the six cone-light erosions (:665): all are evaluated at
// the primary sample point with the primary height, so it is computed once.
template <int S, bool EXACT> MT_HD float erosion_modifier(const Tex<S>& tx, f3 point, float h) {
    f4v curl = Vol<S>::template tex2<MT_CURL_N>(tx.curl, point.x, point.y);
    point.x = point.x + (curl.x * (1.0f - h)) * 0.5f;
    point.y = point.y + (curl.y * (1.0f - h)) * 0.5f;
    f4v hf = Vol<S>::template tex3<MT_DETAIL_N>(tx.detail, point);
    float hfbm = (hf.x * 0.625f) + (hf.y * 0.25f) + (hf.z * 0.125f);
    if (EXACT) return __saturatef(gmix(hfbm, 1.0f - hfbm, __saturatef(h * 2.0f)));
    return gclamp(gmix(hfbm, 1.0f - hfbm, gclamp(h * 2.0f, 0.0f, 1.0f)), 0.0f, 1.0f);
}
// Per-ray constants of cloudRayMarch.comp:565-624, shared by every step (the
// per-frame ones are in Frame).
struct RayConsts {
    f3 dir, startPos;
    f3 koff[6];  // cone-light offsets ((stepSize * kernel[i]) * i) / thickness
    float stepSize, cos_angle, cos_q, HG_light, lenInner;
};

MT_HD void ray_consts(const mt_params& p, const Frame& F, f3 dir, f3 startPos, float stepSize, RayConsts& rc) {
    rc.dir = dir;
    rc.startPos = startPos;
    rc.stepSize = stepSize;
    // the sun direction and the cone-light kernel are the frame's (Frame::light_dir, cone)
    const f3 lightDir = ld3(F.light_dir);
    rc.cos_angle = dot3(normalize3_r(dir), lightDir);
    rc.cos_q = rdiv(rc.cos_angle - 0.7f, MT_RCP(0.7f, 1.0f));
    rc.HG_light = gmax(henyey_greenstein(rc.cos_angle, 0.6f), 0.7f * henyey_greenstein(rc.cos_angle, 0.99f - 0.1f));
    // the step-independent part of the light sample position
    // pos + ((stepSize * kernel[i]) * i) (cloudRayMarch.comp:656)
    // in units of the layer thickness, as the light samples' positions are used
    for (int i = 0; i < 6; ++i) rc.koff[i] = ((stepSize * ld3(F.cone[i])) * (float)i) * F.r_thick.y;
    rc.lenInner = length3(startPos - ld3(F.eye));
}

struct StepOut {
    // bit 4: baseDensity > 0 (cloudRayMarch.comp:642).  Traced marches (TR)
    // also carry the step's jitter index in bits 0-3 and its light samples'
    // cbl > 0 in bits 5-10: the step's part of the control-flow signature.
    int code;
    float hfd;  // eroded density (:645)
    float E;    // light energy (:673)
};
constexpr int kInCloud = 16;

// How a march is compiled: for tame frames (Frame::tame: no range checks on the
// steps' quotients), for every frame, and for every frame with the per-ray trace.
// kBatch is kTame as the batch kernel takes it: its views' constants come from
// memory and press on the registers, so the library's square root and the light
// samples three a turn do better there (20-view batch 9.54 / 8.05 -> 9.31 / 7.86 ms by
// view, 24 sessions 1.59 / 1.38 -> 1.55 / 1.34; frames lose 1 %).
constexpr int kTame = 0, kGeneral = 1, kTraced = 2, kBatch = 3;
template <int MODE> constexpr bool kIsTame = MODE == kTame || MODE == kBatch;

// One iteration of the march loop body (cloudRayMarch.comp:629-678) at
// parameter t, up to the accumulation: everything that does not depend on the
// running accumDensity / transmittance.
template <int S, int MODE>
MT_HD StepOut eval_step(const mt_params& p, const Frame& F, const Tex<S>& tx, const mt_time_ubo& tm,
                        const float (*jitter)[3], const RayConsts& rc, float t) {
    constexpr bool TAME = kIsTame<MODE>, TR = MODE == kTraced, EXACT = kExact<S, TAME>;
    StepOut o{0, 0.0f, 0.0f};
    // int(mod(float(frame + int(t)), 16)), 0..15 for every finite t; in a tame
    // frame (t below 2^24 - 16) the low four bits of the whole number
    const int step = tm.frame_count_mod16 + f2i(t);
    const int _index = (TAME ? step : f2i(gmod((float)step, 16.0f))) & 15;
    if (TR) o.code = _index;
    const float* j = jitter[_index];
    f3 jd = rc.dir + f3{j[0], j[1], j[2]};
    f3 pos = ld3(F.eye) + t * jd;
    const float relH = relative_height<TAME, EXACT, EXACT && MODE == kTame>(F, pos, ld3(F.ec), rc.lenInner, rc.dir, ld3(F.eye));
    // Empty steps, found before anything is fetched for them (results unchanged;
    // of the benchmark views' executed steps 12 % are too high, 6 % have no
    // gradient otherwise and 25 % only a gradient below the threshold.  960x540
    // full frames 518 / 418 / 726 -> 504 / 385 / 690 us by view).  At heights from
    // 0.65 both gradients are 0, whatever the cloud type ...
    if (p.height_gradient && relH >= 0.65f) return o;
    Weather wt = weather_at<S, TAME>(p, F, tx, pos, ld3(F.ec));
    // (the 16-bit forms keep its check: without it their compiler settings
    // contract its blends another way, which moves their results by roundings)
    if (p.height_gradient) wt.hgrad = height_gradient<EXACT>(relH, wt.type);
    // ... a zero height gradient or zero coverage makes the density 0 (or NaN
    // when the coverage is 0), never > 0 ...
    if ((p.height_gradient && wt.hgrad == 0.0f) || wt.mul == 0.0f) return o;
    // ... and so does a gradient that does not exceed the coverage threshold:
    // the base shape is in [0, 1], so shape * gradient <= gradient <= lo (a
    // product's rounding is monotone), the coverage remap clamps it to lo and
    // its numerator lo - lo is 0 (0 / 0 = NaN when lo = 1, not > 0 either).
    if (wt.hgrad <= wt.lo && wt.lo <= 1.0f) return o;
    f3 sp = relative_position<TAME>(F, pos, ld3(F.ec));
    sp = rdiv3_step<TAME>(sp, F.r_period);
    sp = sp + ((relH * ld3(F.skew)) * p.cloud_top_offset) * 0.009f;
    sp = sp + ld3(F.wind_t);
    float baseDensity = sample_low_frequency<S, TAME>(p, tx, sp, relH, wt) * 0.380f;
    if (baseDensity > 0.0f) {
        const Erosion ero = make_erosion<EXACT>(erosion_modifier<S, EXACT>(tx, sp, relH));
        o.code |= kInCloud;
        o.hfd = erode<EXACT>(baseDensity * 1.4f, ero);
        float dl = 0.0f;
        // The six cone-light samples (colour only: see sample_light), unrolled in
        // the FP32-filtered forms: the offsets koff[i] stay in registers instead
        // of an indexed local array, and the samples' loads overlap (rolled ->
        // unrolled: 960x540 full frames 497 / 376 -> 492 / 366 us by view, 4K 5.45 /
        // 3.59 -> 5.39 / 3.56 ms, 20-view batch 12.0 / 9.92 -> 11.6 / 9.57 ms,
        // bfloat16 1603x901 1.21 -> 1.17 ms).
        // relative_position(pos + offset) = (pos - base) / thickness + offset / thickness.
        // Explicit roundings and fmas: the same bits in every kernel that
        // inlines this, whatever the compiler's contraction setting.
        const f3 pb = pos - f3{F.ec[0], F.inner_alt, F.ec[2]};
        const f3 prel{__fmul_rn(pb.x, F.r_thick.y), __fmul_rn(pb.y, F.r_thick.y), __fmul_rn(pb.z, F.r_thick.y)};
        auto light_point = [&](int i) {
            if (i == 0) return prel;  // its offset is 0
            const f3 k = rc.koff[i];
            return f3{__fadd_rn(prel.x, k.x), __fadd_rn(prel.y, k.y), __fadd_rn(prel.z, k.z)};
        };
        if constexpr (S != MT_STORAGE_F16) {
            constexpr int kTurn = MODE == kBatch ? 3 : 6;
#pragma unroll kTurn
            for (int i = 0; i < 6; ++i) {
                const float cbl = sample_light<S>(p, tx, light_point(i), wt);
                if (cbl > 0.0f) {
                    dl = fmaf(fmaf(1.5f, cbl, -ero.lo), ero.r.y, dl);  // erode(1.5 * cbl)
                    if (TR) o.code |= 32 << i;
                }
            }
        } else {
            // FP16 storage: two samples at a time, density math in half2; rolled
            // (unrolled, the 4K frame takes 5.09 ms for 4.94)
#pragma unroll 1
            for (int i = 0; i < 6; i += 2) {
                const float2 cbl = sample_light_pair<__half2>(p, tx.base, light_point(i), light_point(i + 1), wt);
                if (cbl.x > 0.0f) {
                    dl = fmaf(fmaf(1.5f, cbl.x, -ero.lo), ero.r.y, dl);
                    if (TR) o.code |= 32 << i;
                }
                if (cbl.y > 0.0f) {
                    dl = fmaf(fmaf(1.5f, cbl.y, -ero.lo), ero.r.y, dl);
                    if (TR) o.code |= 32 << (i + 1);
                }
            }
        }
        o.E = light_energy<TAME, EXACT>(relH, dl, baseDensity, rc.HG_light, rc.cos_q, 5.0f);
    }
    return o;
}

// cloudRayMarch.comp:565-688, step-parallel.  A group of G lanes marches one
// ray: lane j evaluates step c*G + j of chunk c, with t rebuilt by the same
// serial `t += stepSize` additions as the reference's loop, so every lane sees
// bit-identical t.  The loop-carried part (accumDensity, transmittance,
// colour, the early exit) is then applied in step order by an in-group scan;
// steps past the exit are discarded.  Result, counters and control flow equal
// the sequential loop's.  Three forms of the scan: one lane applies its own step
// (a scan over one lane still shuffled five times a step: 4K full frames 5.04 /
// 3.34 -> 4.69 / 3.16 ms by view, FP16 4.74 / 3.11 -> 4.12 / 2.81, 20-view batch
// 10.8 / 8.89 -> 9.85 / 8.28 ms); 2 and 4 lanes take the steps one by one,
// unrolled; longer groups loop over the in-cloud steps (640x360 frames at 16
// lanes 59.5 / 55.7 -> 52.6 / 45.1 us; at 4 lanes 219 -> 223 us for the 1080p
// frame, so not there).
template <int G, int S, int MODE>
MT_HD f3 ray_march_group(const mt_params& p, const Frame& F, const Tex<S>& tx, const mt_time_ubo& tm,
                         const float (*jitter)[3], f3 dir, f3 startPos, float start_t, float end_t, float& accum,
                         Counts& cnt, unsigned gmask, int lane) {
    float _dot = dot3(dir, f3{0.0f, 1.0f, 0.0f});
    float maxSteps;
    if (p.steps_min == p.steps_max)
        maxSteps = (float)p.steps_min;
    else
        maxSteps = floorf(gmix((float)p.steps_min, (float)p.steps_max, 1.0f - _dot));
    const float thick = end_t - start_t;
    const float stepSize = thick / maxSteps;
    RayConsts rc;
    ray_consts(p, F, dir, startPos, stepSize, rc);
    float transmittance = 1.0f;
    f3 color{0.0f, 0.0f, 0.0f};
    // Iteration guard (not in the reference): a step below the ulp of t would
    // never advance.  A valid ray runs steps or steps+1 iterations.
    const int cap = 2 * f2i(maxSteps) + 8;
    if (lane == 0) cnt.rays++;
    constexpr unsigned kGroup = G == 32 ? 0xffffffffu : (1u << G) - 1u;
    const int shift = (int)(threadIdx.x & 31u) & ~(G - 1);  // the group's first lane
    float t_base = start_t;
    int s_base = 0;
    // A ray that ends before it begins (the two are distances from the origin, so a
    // ray toward it from far away does) marches no step.  Without this its negative
    // steps would bring later lanes of a long chunk below the end.
    bool done = G > 4 && !(start_t < end_t);
    while (!done) {
        float t = t_base;
        for (int k = 0; k < lane; ++k) t += stepSize;
        const int valid = (t < end_t) && (s_base + lane < cap);
        StepOut o{0, 0.0f, 0.0f};
        if (valid) o = eval_step<S, MODE>(p, F, tx, tm, jitter, rc, t);
        auto apply = [&](float hfd, float E) {
            accum = accum + hfd * 0.5f;
            const float k = 1.0f - accum;
            // mix(transmittance, E, k); the 16-bit forms' compiler settings would
            // contract it, so they state their contraction
            transmittance = S == MT_STORAGE_U8 ? gmix(transmittance, E, k)
                                               : __fmaf_rn(E, k, __fmul_rn(transmittance, 1.0f - k));
            color = color + f3{transmittance, transmittance, transmittance};
            if (lane == 0) cnt.light += 6;
        };
        if constexpr (G == 1) {
            if (!valid) break;
            cnt.primary++;
            if (MODE == kTraced) cnt.sig = (cnt.sig ^ (unsigned)o.code) * 16777619u;  // FNV-1a step
            if (o.code & kInCloud) apply(o.hfd, o.E);
            if (accum >= p.accum_limit) {
                accum = 1.0f;
                break;
            }
            t_base = t + stepSize;
            s_base++;
        } else if constexpr (G <= 4) {
#pragma unroll
            for (int k = 0; k < G; ++k) {
                // one shuffle for whether the step exists and what it is; its two
                // values only where it applies them (1080p frame 202 / 167 ->
                // 201 / 165 us by view, 480x270 full frame 140 / 94 -> 139 / 89)
                const int code = __shfl_sync(gmask, valid ? o.code : -1, k, G);
                if (code < 0) {  // past the end of the ray
                    done = true;
                    break;
                }
                if (lane == 0) cnt.primary++;
                if (MODE == kTraced && lane == 0) cnt.sig = (cnt.sig ^ (unsigned)code) * 16777619u;
                if (code & kInCloud) {
                    const float hfd = __shfl_sync(gmask, o.hfd, k, G);
                    const float E = __shfl_sync(gmask, o.E, k, G);
                    apply(hfd, E);
                }
                if (accum >= p.accum_limit) {
                    accum = 1.0f;
                    done = true;
                    break;
                }
            }
        } else {
            // Only in-cloud steps move the accumulated density, so only after
            // them can the ray end early (and after its first step, should the
            // limit not lie above 0): a loop over those, where the steps of a
            // long chunk one by one take four shuffles each.
            static_assert(G <= 4 || MODE != kTraced, "traced marches use 1 or 4 lanes");
            const unsigned in_chunk = __ballot_sync(gmask, valid) >> shift & kGroup;  // the first steps: t grows
            const unsigned cloud = __ballot_sync(gmask, (o.code & kInCloud) != 0) >> shift & kGroup;
            int executed = __popc(in_chunk);
            done = executed < G;
            unsigned events = (cloud | (accum >= p.accum_limit ? 1u : 0u)) & in_chunk;
            while (events) {
                const int k = __ffs((int)events) - 1;
                events &= events - 1u;
                const float hfd = __shfl_sync(gmask, o.hfd, k, G);
                const float E = __shfl_sync(gmask, o.E, k, G);
                if (cloud >> k & 1u) apply(hfd, E);
                if (accum >= p.accum_limit) {
                    accum = 1.0f;
                    done = true;
                    executed = k + 1;
                    break;
                }
            }
            if (lane == 0) cnt.primary += executed;
        }
        if (G > 1 && !done) {
            t_base = __shfl_sync(gmask, t, G - 1, G) + stepSize;
            s_base += G;
        }
    }
    return color;
}

// cloudRayMarch.comp:690-826 for one pixel, marched by a group of G lanes;
// lane 0 stores.  `jitter`: the view's per-step jitter table (a.jitter, or a
// copy of it in shared memory).
template <int G, int S, int MODE>
MT_HD void march_pixel(const MarchArgs& a, const Frame& F, const Tex<S>& tx, int px, int py, Counts& cnt,
                       unsigned gmask, int lane, const float (*jitter)[3]) {
    constexpr bool TR = MODE == kTraced;
    const mt_params& p = a.params;
    const int W = a.width;
    // this frame's camera basis and cloudRayMarch.comp's jitter: the TXAA
    // geometry constants (the same camera, slot and image size)
    const ViewConsts& vc = a.vc_txaa;
    float ux = rdiv((float)px, Rcp{vc.r_w[0], vc.r_w[1]}), uy = rdiv((float)py, Rcp{vc.r_h[0], vc.r_h[1]});
    uy = 1.0f - uy;
    const Ray ray = cast_ray(vc, ld3(F.eye), ux, uy);
    float _dot = dot3(f3{0.0f, 1.0f, 0.0f}, ray.direction);
    const float bgMul = gmax(0.620f, _dot);
    const float fade = 0.06f;
    const size_t o = (size_t)py * (size_t)W + (size_t)px;
    f3 bg;
    if (_dot < 0.0f) {
        f3 cNear = f3{0.0f, 0.16f, 0.51f} * 0.4f;
        f3 c2 = f3{0.0f, 0.73f, 0.95f} * 0.5f;
        bg = mix3(cNear, c2, -ray.direction.y * 5.5f);
        if (lane == 0) {
            a.cur[o] = make_float4(bg.x, bg.y, bg.z, 1.0f);
            if (a.mask) a.mask[o] = 0.0f;
            if (TR) a.trace[o] = make_uint4(0u, 0u, 0u, 0u);
        }
        return;
    }
    bg = atmosphere_color(F, ray.direction);  // sunIntensity 0.780 is in F.sky_sunE
    bg = bg * bgMul;
    if (_dot < fade) {
        if (lane == 0) {
            a.cur[o] = make_float4(bg.x, bg.y, bg.z, 1.0f);
            if (a.mask) a.mask[o] = 0.0f;
            if (TR) a.trace[o] = make_uint4(0u, 0u, 0u, 0u);
        }
        return;
    }
    const f3 ec = ld3(F.ec);
    Isect in, out;
    if (p.fp64_shells) {
        // ray.origin is the eye: the origin terms are the frame's
        in = ray_sphere_fp64(F.sh_o[0], F.sh_c[0], ray.direction, ec, F.Rin);
        out = ray_sphere_fp64(F.sh_o[1], F.sh_c[1], ray.direction, ec, F.Rout);
    } else {
        in = ray_sphere(F.sh32_o[0], F.sh32_c[0], ray.direction, ec, F.Rin);
        out = ray_sphere(F.sh32_o[1], F.sh32_c[1], ray.direction, ec, F.Rout);
    }
    float accum = 0.0f;
    if (TR) cnt.sig = 2166136261u;
    f3 res = ray_march_group<G, S, MODE>(p, F, tx, a.time, jitter, ray.direction, in.point, in.t, out.t, accum, cnt,
                                       gmask, lane);
    if (lane != 0) return;
    float godAccum = accum;
    accum = accum * gsmoothstep(0.0f, 1.0f, gmin(1.0f, remap(ray.direction.y, fade, 0.2f, 0.0f, 1.0f)));
    f3 fc = mix3(bg, res, accum);
    a.cur[o] = make_float4(fc.x, fc.y, fc.z, 1.0f);
    if (a.mask) a.mask[o] = godray_value(25.0f * gmin(0.05f, 1.0f - godAccum), ray.direction.y);
    // one ray per thread in march_kernel: lane 0's counters are this ray's
    if (TR) a.trace[o] = make_uint4(cnt.primary, cnt.light / 6u, cnt.primary ? cnt.sig : 0u, 0u);
}

// Ray -> marched pixel.  Checkerboard: the reference's group grid covers
// groups_x x groups_y blocks of 4x4 (Renderer.cpp:713-716); each ray is one
// block's slot pixel.  Full: one ray per pixel.  G consecutive lanes (an
// aligned segment of a warp) march one ray.  BS threads per CTA (256 by
// default, 128 or 32 selectable; 128 at most for one and two lanes per ray, whose
// rays end furthest apart: 960x540 full frames 357 / 234 -> 344 / 230 us by view, FP16
// 4K 3.76 / 2.58 -> 3.70 / 2.54 ms, 640x360 full frame 205 / 140 -> 196 / 139).
// Resident threads per SM: 1024, 64 registers a thread.  (1280 for one lane per ray,
// at 48 registers with some 200 B of spills: RGBA8 4K 4.69 ms for 4.62, bfloat16
// 1603x901 1.06 for 1.01; FP16, us by view, 680x680 417 / 403 / 365 for 375 / 348 /
// 317, 4K 4775 / 3748 / 3241 for 4641 / 3647 / 3138.)
// Every step reads its jitter vector at an index taken from int(t), which
// differs from lane to lane: from the parameter space a warp's reads at up to
// 16 different words are served one word at a time, from shared memory in one
// pass (48 words, 3 apart: distinct banks), so the table is copied there.
constexpr int march_min_blocks(int BS) {
    return 1024 / BS < 32 ? 1024 / BS : 32;  // at most 32 CTAs an SM
}
// The rays of a warp.  One lane per ray: 8x4 rays, which fetch nearer cells and end
// nearer one another than 32 in a row (960x540 full frames 387 / 235 -> 357 / 234 us by
// view, bfloat16 1603x901 976 / 604 -> 892 / 589, 3840x2160 frame 628 / 523 ->
// 607 / 518).  More lanes: a row of rays (2 lanes on 4x4 rays: 640x360 full frame
// 196 / 139 -> 190 / 138, but 2560x1440 frame 307 / 267 -> 304 / 277).
template <int G> struct WarpTile {
    static constexpr int R = 32 / G, W = R >= 32 ? 8 : R, H = R / W;
    // the launch's rays in whole tiles
    static long long rays(const MarchArgs& a) {
        const bool full = (a.flags & MT_RENDER_FULL) != 0;
        const long long nx = full ? a.width : a.groups_x, ny = full ? a.height : a.groups_y;
        return (nx + W - 1) / W * ((ny + H - 1) / H) * R;
    }
};
template <int G, int S, int BS, int MODE>
__global__ void __launch_bounds__(BS, march_min_blocks(BS))
    march_kernel(const __grid_constant__ MarchArgs a) {
    static_assert(G >= 1 && G <= 32 && (32 % G) == 0, "G must divide the warp");
    const Frame& F = a.frame;
    const Tex<S> tx = make_tex<S>(a);
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned idx = (unsigned)(tid / G);  // rays < 2^31 (images are at most 16384^2)
    const int lane = (int)(threadIdx.x % G);
    const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
    __shared__ float s_jitter[16][3];
    for (int i = threadIdx.x; i < 48; i += BS) (&s_jitter[0][0])[i] = (&a.jitter[0][0])[i];
    __syncthreads();
    Counts cnt{0u, 0u, 0u};
    unsigned pixels = 0;
    int px = 0, py = 0;
    bool active;
    using T = WarpTile<G>;
    const bool full = (a.flags & MT_RENDER_FULL) != 0;
    const int nx = full ? a.width : a.groups_x, ny = full ? a.height : a.groups_y;
    const unsigned cols = (unsigned)(nx + T::W - 1) / T::W, rows = (unsigned)(ny + T::H - 1) / T::H;
    const unsigned tile = idx / T::R, sub = idx % T::R;
    const int rx = (int)(tile % cols * T::W + sub % T::W);
    const int ry = march_row((int)(tile / cols), (int)rows, a.bottom_up) * T::H + (int)(sub / T::W);
    active = tile / cols < rows && rx < nx && ry < ny;
    if (full) {
        px = rx;
        py = ry;
    } else {
        const int id = a.time.frame_count_mod16;
        px = rx * 4 + a.params.slot_x[id];
        py = ry * 4 + a.params.slot_y[id];
        active = active && px < a.width && py < a.height;
    }
    if (active) {
        march_pixel<G, S, MODE>(a, F, tx, px, py, cnt, gmask, lane, s_jitter);
        pixels = lane == 0 ? 1u : 0u;
    }
    if (a.stats) flush_counts(a.stats, cnt, pixels);
}


// Batched form (config 3): one persistent launch over many views of uneven
// size.  Each CTA repeatedly takes the next tile from the batch's counter and
// marches its rays, 128/G rays per pass; per-view arguments come from the
// view table in global memory.  Per-pixel results equal those of separate
// march_kernel launches (the same march_pixel runs on the same inputs).
template <int G, int S, int MODE>
__global__ void __launch_bounds__(128, 8) march_batch_kernel(const __grid_constant__ BatchArgs b) {
    __shared__ int s_tile;
    const int lane = (int)(threadIdx.x % G);
    const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
    constexpr int kRaysPerPass = 128 / G;
    Counts cnt{0u, 0u, 0u};
    unsigned pixels = 0;
    for (;;) {
        if (threadIdx.x == 0) s_tile = (int)atomicAdd(b.counter, 1u);
        __syncthreads();
        const int t = s_tile;
        __syncthreads();
        if (t >= b.n_tiles) break;
        const BatchTile tile = b.tiles[t];
        const MarchArgs& a = b.views[tile.view];
        const Frame& F = a.frame;
        const Tex<S> tx = make_tex<S>(a);
        const bool full = (a.flags & MT_RENDER_FULL) != 0;
        const int id = a.time.frame_count_mod16;
        const int sx = full ? 0 : a.params.slot_x[id], sy = full ? 0 : a.params.slot_y[id];
        const int step = full ? 1 : 4;
        const int tile_rays = b.tile_w * b.tile_h;
        for (int r0 = 0; r0 < tile_rays; r0 += kRaysPerPass) {
            const int r = r0 + (int)(threadIdx.x / G);
            const int rx = tile.rx0 + r % b.tile_w, ry = tile.ry0 + r / b.tile_w;
            const int px = rx * step + sx, py = ry * step + sy;
            const bool active = r < tile_rays && rx < tile.nrx && ry < tile.nry && px < a.width && py < a.height;
            if (active) {
                march_pixel<G, S, MODE>(a, F, tx, px, py, cnt, gmask, lane, a.jitter);
                pixels += lane == 0 ? 1u : 0u;
            }
        }
    }
    if (b.stats) flush_counts(b.stats, cnt, pixels);
}

// The batch kernel for `lanes` per ray, with or without the special cases of
// frames that are not tame.  Both at every lane count: the tiles are made for the
// batch's lanes (general kernels at one lane, on a 200x180 full frame's tiles for 8
// lanes: 205 / 261 us by view, at 8 lanes 89 / 92; the frame alone at 4 | 8 lanes
// 87 / 96 | 65 / 64).
using BatchKernel = void (*)(BatchArgs);
template <int S, int MODE> BatchKernel batch_kernel(int lanes) {
    switch (lanes) {
        case 1: return march_batch_kernel<1, S, MODE>;
        case 2: return march_batch_kernel<2, S, MODE>;
        case 4: return march_batch_kernel<4, S, MODE>;
        case 16: return march_batch_kernel<16, S, MODE>;
        case 32: return march_batch_kernel<32, S, MODE>;
        default: return march_batch_kernel<8, S, MODE>;
    }
}
template <int S> BatchKernel batch_kernel(int lanes, bool tame) {
    return tame ? batch_kernel<S, kBatch>(lanes) : batch_kernel<S, kGeneral>(lanes);
}

template <int S> cudaError_t launch_batch_storage(const BatchArgs& b, int lanes, int blocks, cudaStream_t s) {
    batch_kernel<S>(lanes, b.tame != 0)<<<blocks, 128, 0, s>>>(b);
    return cudaGetLastError();
}

template <int S> int batch_blocks_storage(int device, int lanes, bool tame) {
    int per_sm = 0, sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_kernel<S>(lanes, tame), 128, 0);
    return (per_sm > 0 ? per_sm : 1) * (sms > 0 ? sms : 1);
}

template <int G, int S, int BS, int MODE> void launch_march_kernel(const MarchArgs& a, cudaStream_t s) {
    const unsigned blocks = (unsigned)((WarpTile<G>::rays(a) * G + BS - 1) / BS);
    march_kernel<G, S, BS, MODE><<<blocks, BS, 0, s>>>(a);
}

// The CTA size asked for, 128 threads at most for one and two lanes per ray.
template <int S, int BS, int MODE> void launch_march_bs(const MarchArgs& a, cudaStream_t s) {
    constexpr int BS2 = BS < 128 ? BS : 128;
    switch (a.lanes) {
        case 1: launch_march_kernel<1, S, BS2, MODE>(a, s); break;
        case 2: launch_march_kernel<2, S, BS2, MODE>(a, s); break;
        case 4: launch_march_kernel<4, S, BS, MODE>(a, s); break;
        case 16: launch_march_kernel<16, S, BS, MODE>(a, s); break;
        case 32: launch_march_kernel<32, S, BS, MODE>(a, s); break;
        default: launch_march_kernel<8, S, BS, MODE>(a, s); break;
    }
}

template <int S> cudaError_t launch_march_storage(const MarchArgs& a, cudaStream_t s) {
    if (a.trace) {  // 256-thread CTAs, 1 or 4 lanes
        if (a.lanes == 1)
            launch_march_kernel<1, S, 256, kTraced>(a, s);
        else
            launch_march_kernel<4, S, 256, kTraced>(a, s);
    } else if (!a.frame.tame) {  // the default CTA size only
        launch_march_bs<S, 256, kGeneral>(a, s);
    } else if (a.block == 256) {
        launch_march_bs<S, 256, kTame>(a, s);
    } else if (a.block == 128) {
        launch_march_bs<S, 128, kTame>(a, s);
    } else {
        launch_march_bs<S, 32, kTame>(a, s);
    }
    return cudaGetLastError();
}

}  // namespace mt
