// The two downstream full-screen passes that consume the compute stage's
// outputs:
//
//   godrays_kernel  <- shaders/postProcess_GodRays.frag:66-149 (100-sample
//                      radial blur of the god-ray mask, added to the HDR image)
//   tonemap_kernel  <- shaders/postProcess_ToneMap.frag:68-84 (Uncharted-2
//                      filmic curve + WangHash dither)
//
// Both shaders run one fragment per pixel (in_uv at the pixel centre) and
// store with imageStore at pixelPos = clamp(round(dim * in_uv)), which is the
// fragment's own pixel or the next one.  The fragment whose store lands on a
// pixel p: along each axis the candidates are fragments p and p - 1, and where
// both map to p the later one in raster order (the larger index) wins.  The tone
// map's threads own pixels and find their fragments; the blur's own fragments and
// write the pixels they win, and a pixel that no fragment stores to is copied by
// the thread of its own index.  Each output pixel is read and written by exactly
// one thread, so the result is defined (in the reference, colliding stores race),
// and the blur's out may alias in.
//
// Compiled with -fmad=false and IEEE division: the operation order follows
// the shaders' so the results equal the CPU restatement bit for bit except
// through powf (tone map).
#include <cuda_runtime.h>

#include "mt_kernels.h"
#include "mt_device.cuh"

namespace mt {

namespace {

// pixelPos of the fragment at index f along an axis of size n
// (postProcess_GodRays.frag:69, postProcess_ToneMap.frag:71).
MT_HD float frag_uv(int f, int n) { return ((float)f + 0.5f) / (float)n; }
MT_HD int frag_pixel(int f, int n) { return imin(imax(f2i(roundf((float)n * frag_uv(f, n))), 0), n - 1); }

// The fragment whose store lands on pixel p (the last one in raster order),
// or -1 when none does.
MT_HD int winner_fragment(int p, int n) {
    if (frag_pixel(p, n) == p) return p;
    if (p > 0 && frag_pixel(p - 1, n) == p) return p - 1;
    return -1;
}

// 1 / 16581375 as the shader's bitDec.w (postProcess_GodRays.frag:36-37).
__device__ __forceinline__ float bit_dec_w() { return 1.0f / 16581375.0f; }

constexpr float kFloorMagic = 12582912.0f;  // 1.5 * 2^23

// A tap's coordinate along one axis of the mask: texel index and weight.  The
// floor is one addition rounded down: the image is at most 16384 texels wide and
// a tap at most a texel outside it, so floor(v) + 1.5 * 2^23 is exact.
struct AxisTap {
    float w;
    int i;
};
MT_HD AxisTap axis_tap(float u, float n) {
    const float v = u * n - 0.5f, t = __fadd_rd(v, kFloorMagic);
    return AxisTap{v - (t - kFloorMagic), __float_as_int(t) - __float_as_int(kFloorMagic)};
}

// extract32fFromRGBA8f (postProcess_GodRays.frag:39-43) over the R32F mask:
// the texel (m, 0, 0, 0) decodes to m, the opaque-black border (0, 0, 0, 1)
// to bitDec.w.  LINEAR filter with exact FP32 weights, like every sampler
// here: the value channel and the border channel are interpolated x then y,
// then decoded as dot(texel, bitDec) in the shader's order.  INSIDE: all four
// texels are in the image, where the border channel is 0.  FLAT: no branch at the
// border, the texels' indices clamped instead, so that several taps' loads are in
// flight together.
template <bool INSIDE, bool FLAT> MT_HD float mask_decode(const GodrayArgs& a, AxisTap x, AxisTap y) {
    if (INSIDE || (!FLAT && (unsigned)x.i < (unsigned)(a.width - 1) && (unsigned)y.i < (unsigned)(a.height - 1))) {
        const float* r = a.mask + (y.i * a.width + x.i);
        const float* r1 = r + a.width;
        const float2 p = make_float2(__ldg(r), __ldg(r1)), q = make_float2(__ldg(r + 1), __ldg(r1 + 1));
        const float2 rows = lerp2(p, q, splat2(x.w));
        return lerp1(rows.x, rows.y, y.w);
    }
    float val[4], brd[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int i = x.i + (k & 1), j = y.i + (k >> 1);
        const int ic = FLAT ? imin(imax(i, 0), a.width - 1) : i, jc = FLAT ? imin(imax(j, 0), a.height - 1) : j;
        const bool out = i < 0 || j < 0 || i >= a.width || j >= a.height;
        const float t = FLAT || !out ? __ldg(a.mask + (jc * a.width + ic)) : 0.0f;
        val[k] = out ? 0.0f : t;
        brd[k] = out ? 1.0f : 0.0f;
    }
    const float v = lerp1(lerp1(val[0], val[1], x.w), lerp1(val[2], val[3], x.w), y.w);
    const float o = lerp1(lerp1(brd[0], brd[1], x.w), lerp1(brd[2], brd[3], x.w), y.w);
    // dot(texel, bitDec) = v*1 + 0*bitDec.y + 0*bitDec.z + o*bitDec.w, left to right
    return ((v * 1.0f + 0.0f) + 0.0f) + o * bit_dec_w();
}

struct GodrayFrame {
    float blend;   // dot(cam_to_sun, camForward)
    float ssx, ssy;
    bool outside;  // sun outside [0,1]^2 in screen space (never, after the clamp)
};

// The per-frame quantities of postProcess_GodRays.frag:74-93.  Evaluated on
// the device by every thread (a few dozen flops): host compilers may contract
// these into fused multiply-adds.
MT_HD GodrayFrame godray_frame(const mt_camera_ubo& cam) {
    GodrayFrame g;
    const f3 sun{0.0f, 1.0f, 0.0f};
    const f3 cam_to_sun = normalize3(sun - ld3(cam.eye));
    const f3 fwd = -normalize3(f3{cam.view[2], cam.view[6], cam.view[10]});
    g.blend = dot3(cam_to_sun, fwd);
    // camera.proj * camera.view * vec4(sun, 1): the matrix product first,
    // column j = proj * view[j], then that times the vector.
    float M[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i)
            M[j][i] = cam.proj[0 * 4 + i] * cam.view[j * 4 + 0] + cam.proj[1 * 4 + i] * cam.view[j * 4 + 1] +
                      cam.proj[2 * 4 + i] * cam.view[j * 4 + 2] + cam.proj[3 * 4 + i] * cam.view[j * 4 + 3];
    const float nx = M[0][0] * 0.0f + M[1][0] * 1.0f + M[2][0] * 0.0f + M[3][0] * 1.0f;
    const float ny = M[0][1] * 0.0f + M[1][1] * 1.0f + M[2][1] * 0.0f + M[3][1] * 1.0f;
    g.ssx = gclamp((nx + 1.0f) / 2.0f, 0.0f, 1.0f);
    g.ssy = gclamp((ny + 1.0f) / 2.0f, 0.0f, 1.0f);
    g.outside = g.ssx < 0.0f || g.ssx > 1.0f || g.ssy < 0.0f || g.ssy > 1.0f;
    return g;
}

// The blur.  Bound by instruction issue and texel latency: 100 bilinear taps a
// fragment, each with its coordinates, loads, nine interpolation operations and the
// channels' weighted sums.  A fragment's taps step along a line, ux -= dx and
// uy -= dy on every tap, so their columns depend on its column alone and their rows
// on its row.  A thread takes ROWS fragments of one column and computes each tap's
// column once for all of them; a CTA's first threads step through the taps' rows,
// whose texels and weights all of them then tabulate in shared memory (small images,
// where the steps' serial chain would be the time: one fragment a thread, its rows
// its own).  A CTA whose taps all lie inside the image (coordinates move
// monotonically, so the ends decide) takes the loop without border checks, where
// neighbouring rows share filtered texels (god_blur), and one sum serves red and
// green where the light's are equal, as the reference's are.
// One pixel a thread with its own taps and border checks took 409 us at 1080p and
// 1.58 ms at 4K (430 M warp instructions at 1080p); rows and columns looked up apart
// 237 us and 0.79 ms (173 M); threads over fragments, whose rows are one apart where
// pixels' fragments repeat and skip, sharing filtered texels 222 us and 0.71 ms
// (unrolled by 2, 224 us).
constexpr int kGodTaps = 100, kGodWarps = 4;
// Rows a thread, by pixels: more share more of a tap, fewer leave more CTAs
// (1 | 2 | 4 rows, us: 320x180 25 | 42 | -, 640x360 54 | 44 | -, 1280x720 141 | 121 | -,
// 1920x1080 283 | 229 | 222; 8 rows 268).
constexpr long long kRows2 = 200000, kRows4 = 1800000;
// Small images are latency: up to here the taps take no branch at the border and are
// unrolled by 20 (branch, by 4 | flat, us, sun in the image and at its edge: 160x90
// 25 / 33 | 17 / 17, 256x144 25 / 35 | 19 / 19, 320x180 25 / 39 | 25 / 23, 400x225 28 / 41 |
// 33 / 33, 640x360 43 / 64 | 62 / 64).
constexpr long long kFlat = 72000;

// One axis of a fragment: its first tap, its step and whether all its taps keep a
// texel and a half from the ends (the recurrence's roundings move a tap by less
// than a tenth of one); the pixel it stores to (negative: a later fragment stores
// there too); and whether any fragment stores to the pixel of its own index, which
// keeps its input otherwise.
struct GodAxis {
    float u, d;
    int pixel;
    bool covered, inside;
};
MT_HD GodAxis god_axis(int f, int n, float ss) {
    GodAxis x;
    f = imin(f, n - 1);
    const int p = frag_pixel(f, n);
    x.pixel = winner_fragment(p, n) == f ? p : -1;
    x.covered = winner_fragment(f, n) >= 0;
    x.u = frag_uv(f, n);
    x.d = ((x.u - ss) / 100.0f) * 1.0f;
    const float lo = 1.5f / (float)n, hi = 1.0f - 2.5f / (float)n, last = x.u + (ss - x.u) * 0.99f;
    x.inside = x.u >= lo && x.u <= hi && last >= lo && last <= hi;
    return x;
}

// The sums of a thread's fragments, ROWS rows of one column from the table's row on.
// INSIDE: no tap touches the border; and, for several rows, from the second tap on
// each row taps the texel row of the row above it or the next, as fragments
// close in on the sun together.  Then the rows' filtered texels chain: a row's
// upper texels are its upper neighbour's, upper or lower, and it loads and filters
// its lower two, in packed pairs of rows.
template <int ROWS, bool INSIDE, bool FLAT, bool SHARED_RG>
MT_HD void god_blur(const GodrayArgs& a, const AxisTap* rows, GodAxis col, GodAxis row, float2 (&ax)[(ROWS + 1) / 2],
                    float2 (&ay)[(ROWS + 1) / 2], float2 (&az)[(ROWS + 1) / 2]) {
    constexpr int TH = kGodWarps * ROWS, PAIRS = (ROWS + 1) / 2;
    const float w = 1.0f * 0.001f;  // illuminationDecay * WEIGHT_FOR_SAMPLE, DECAY = 1
    const float fw = (float)a.width, fh = (float)a.height;
    auto add = [&](int k, float2 s) {
        if (ROWS == 1) {  // no pair to fill
            ax[0].x = ax[0].x + (a.light[0] * s.x) * w;
            if (!SHARED_RG) ay[0].x = ay[0].x + (a.light[1] * s.x) * w;
            az[0].x = az[0].x + (a.light[2] * s.x) * w;
            return;
        }
        auto weighted = [&](float light) { return mul2(mul2(splat2(light), s), splat2(w)); };
        ax[k] = add2(ax[k], weighted(a.light[0]));
        if (!SHARED_RG) ay[k] = add2(ay[k], weighted(a.light[1]));
        az[k] = add2(az[k], weighted(a.light[2]));
    };
    auto single = [&](int i) {
        const AxisTap x = axis_tap(col.u, fw);
#pragma unroll
        for (int k = 0; k < PAIRS; ++k) {
            float s[2] = {0.0f, 0.0f};
#pragma unroll
            for (int h = 0; h < 2 && 2 * k + h < ROWS; ++h) {
                const AxisTap y = ROWS == 1 ? axis_tap(row.u, fh) : rows[i * TH + 2 * k + h];
                s[h] = mask_decode<INSIDE, FLAT>(a, x, y);
            }
            add(k, make_float2(s[0], s[1]));
        }
        col.u -= col.d;
        if (ROWS == 1) row.u -= row.d;
    };
    if (INSIDE && ROWS > 1) {
        single(0);
#pragma unroll 1
        for (int i = 1; i < kGodTaps; ++i) {
            const AxisTap x = axis_tap(col.u, fw);
            const int lower = x.i + a.width;
            int last = 0;
            float up = 0.0f, down = 0.0f;  // the last row's filtered texels
#pragma unroll
            for (int k = 0; k < PAIRS; ++k) {
                const float4 t = *reinterpret_cast<const float4*>(rows + i * TH + 2 * k);
                const int j0 = __float_as_int(t.y), j1 = __float_as_int(t.w);
                const float *r0 = a.mask + (j0 * a.width + lower), *r1 = a.mask + (j1 * a.width + lower);
                const float2 d = lerp2(make_float2(__ldg(r0), __ldg(r1)), make_float2(__ldg(r0 + 1), __ldg(r1 + 1)),
                                       splat2(x.w));
                float2 u;
                if (k == 0) {
                    const float* r = a.mask + (j0 * a.width + x.i);
                    u.x = lerp1(__ldg(r), __ldg(r + 1), x.w);
                } else {
                    u.x = j0 != last ? down : up;
                }
                u.y = j1 != j0 ? d.x : u.x;
                add(k, lerp2(u, d, make_float2(t.x, t.z)));
                last = j1;
                up = u.y;
                down = d.y;
            }
            col.u -= col.d;
        }
    } else {
        constexpr int kUnroll = FLAT ? 20 : ROWS == 1 ? 4 : 2;
#pragma unroll kUnroll
        for (int i = 0; i < kGodTaps; ++i) single(i);
    }
    if (SHARED_RG) {
#pragma unroll
        for (int k = 0; k < PAIRS; ++k) ay[k] = ax[k];
    }
}

template <int ROWS, bool FLAT>
__global__ void __launch_bounds__(32 * kGodWarps) godrays_kernel(const __grid_constant__ GodrayArgs a) {
    constexpr int TH = kGodWarps * ROWS;
    __shared__ __align__(16) AxisTap taps[ROWS == 1 ? 1 : kGodTaps * TH];
    __shared__ GodrayFrame frame;
    __shared__ int pixel_y[TH];
    __shared__ bool covered_y[TH];
    const int W = a.width, H = a.height;
    const int first = ((int)threadIdx.x >> 5) * ROWS;  // the thread's first row in the tile
    const int px = (int)blockIdx.x * 32 + ((int)threadIdx.x & 31), y0 = (int)blockIdx.y * TH;
    if (ROWS > 1) {
        if (threadIdx.x == 0) frame = godray_frame(a.camera);
        __syncthreads();
    }
    const GodrayFrame g = ROWS > 1 ? frame : godray_frame(a.camera);
    const bool blurs = !(g.blend < 0.0f) && !g.outside;  // else the image passes as it is, and needs no taps
    const GodAxis col = god_axis(px, W, g.ssx);
    // one row a thread: its own; else the row that this thread tabulates
    GodAxis row = god_axis(y0 + (ROWS == 1 ? first : (int)threadIdx.x & (TH - 1)), H, g.ssy);
    bool inside = col.inside && row.inside;
    inside = ROWS == 1 ? __all_sync(0xffffffffu, inside) != 0 : __syncthreads_and(inside) != 0;
    if (ROWS > 1) {
        bool chain = true;
        if (threadIdx.x < TH) {
            pixel_y[threadIdx.x] = row.pixel;
            covered_y[threadIdx.x] = row.covered;
#pragma unroll 10
            for (int i = 0; blurs && i < kGodTaps; ++i) {
                taps[i * TH + threadIdx.x].w = row.u;
                row.u -= row.d;
            }
        }
        __syncthreads();
        for (int e = (int)threadIdx.x; blurs && e < kGodTaps * TH; e += 32 * kGodWarps) {  // whole warps
            const AxisTap y = axis_tap(taps[e].w, (float)H);
            const int below = __shfl_down_sync(0xffffffffu, y.i, 1, TH);
            chain = chain && (e < TH || (unsigned)below - (unsigned)y.i <= 1u);
            taps[e] = y;
        }
        inside = __syncthreads_and(chain) != 0 && inside;
    }
    constexpr int PAIRS = (ROWS + 1) / 2;
    float2 ax[PAIRS], ay[PAIRS], az[PAIRS];
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) ax[k] = ay[k] = az[k] = make_float2(0.0f, 0.0f);
    if (blurs) {
        if (inside && a.light[0] == a.light[1])
            god_blur<ROWS, true, FLAT, true>(a, taps + first, col, row, ax, ay, az);
        else if (inside)
            god_blur<ROWS, true, FLAT, false>(a, taps + first, col, row, ax, ay, az);
        else
            god_blur<ROWS, false, FLAT, false>(a, taps + first, col, row, ax, ay, az);
    }
    if (px >= W) return;
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
        const int py = y0 + first + k;
        if (py >= H) return;
        if (!(col.covered && (ROWS == 1 ? row.covered : covered_y[first + k]))) {  // the pixel of this index
            const size_t own = (size_t)py * (size_t)W + (size_t)px;
            a.out[own] = a.in[own];
        }
        const int y = ROWS == 1 ? row.pixel : pixel_y[first + k];
        if (col.pixel < 0 || y < 0) continue;
        const size_t idx = (size_t)y * (size_t)W + (size_t)col.pixel;
        float4 v = a.in[idx];
        if (!(g.blend < 0.0f)) {
            // the out-of-frustum branch discards what it accumulated (:126)
            auto of = [&](const float2(&sums)[PAIRS]) { return k & 1 ? sums[k / 2].y : sums[k / 2].x; };
            v.x += (of(ax) * 1.0f) * g.blend;
            v.y += (of(ay) * 1.0f) * g.blend;
            v.z += (of(az) * 1.0f) * g.blend;
            v.w += 1.0f * g.blend;
        }
        a.out[idx] = v;
    }
}

// Uncharted2Tonemap (postProcess_ToneMap.frag:32-35) with A..F = .15 .5 .1 .2 .02 .3
MT_HD float uncharted2(float x) {
    const float A = 0.15f, B = 0.50f, C = 0.10f, D = 0.20f, E = 0.02f, F = 0.30f;
    return ((x * (A * x + C * B) + D * E) / (x * (A * x + B) + D * F)) - E / F;
}

// WangHashNoise (postProcess_ToneMap.frag:52-66)
MT_HD float wang_hash_noise(uint32_t u, uint32_t v, uint32_t s) {
    uint32_t seed = (u * 1664525u + v) + s;
    seed = (seed ^ 61u) ^ (seed >> 16u);
    seed *= 9u;
    seed = seed ^ (seed >> 4u);
    seed *= 0x27d4eb2du;
    seed = seed ^ (seed >> 15u);
    return __uint2float_rn(seed) * (1.0f / 4294967296.0f);
}

// uint(time.y): truncation; negative and NaN give 0, beyond the range saturates.
MT_HD uint32_t f2u(float t) { return __float2uint_rz(t); }

// tonemap(x, 100) of postProcess_ToneMap.frag:37-46
MT_HD float tonemap1(float x) {
    const float color = uncharted2(2.5f * x);
    const float whitemap = 1.0f / uncharted2(100.0f);
    return powf(color * whitemap, 1.0f / 2.2f);
}

// Vulkan float -> UNORM8: clamp to [0, 1], scale, round to nearest even.
MT_HD uint32_t unorm8(float f) {
    const float c = (f > 0.0f) ? (f < 1.0f ? f : 1.0f) : 0.0f;  // NaN -> 0
    return (uint32_t)__float2uint_rn(c * 255.0f);
}

// One axis of a pixel's filtered fetch: the fragment that stores to it (negative:
// none) and where that fragment samples.
struct ToneAxis {
    int fragment, i;
    float w;
};
MT_HD ToneAxis tone_axis(int p, int n) {
    ToneAxis t;
    t.fragment = winner_fragment(p, n);
    const float u = frag_uv(t.fragment, n) * (float)n - 0.5f, fu = floorf(u);
    t.i = f2i(fu);
    t.w = u - fu;
    return t;
}

// The tone map.  Bound by instruction issue (three powf and three divisions a
// pixel), with 24 bytes a pixel far below it.  As in the blur, a pixel's column and
// row are each looked up along one axis: a thread takes ROWS pixels of a column and
// finds it once, a CTA's first threads find its rows once for the 32 columns.  The
// blur's size lines hold here too (every pixel alone | 2 | 4 rows a thread, us:
// 800x450 9 | 9 | 11, 1280x720 17 | 15 | 17, 1920x1080 34 | 29 | 29, 3840x2160
// 122 | 101 | 97).
constexpr int kToneWarps = 8;

template <int ROWS, bool RGBA8>
__global__ void __launch_bounds__(32 * kToneWarps) tonemap_kernel(const __grid_constant__ TonemapArgs a) {
    constexpr int TH = kToneWarps * ROWS;
    __shared__ ToneAxis rows[ROWS == 1 ? 1 : TH];
    const int first = ((int)threadIdx.x >> 5) * ROWS;  // the thread's first row in the tile
    const int px = (int)blockIdx.x * 32 + ((int)threadIdx.x & 31), y0 = (int)blockIdx.y * TH;
    if (ROWS > 1) {
        if (threadIdx.x < TH) rows[threadIdx.x] = tone_axis(y0 + (int)threadIdx.x, a.height);
        __syncthreads();
    }
    if (px >= a.width) return;
    const ToneAxis col = tone_axis(px, a.width);
    if (col.fragment < 0) return;  // no fragment stores here: the pixel keeps its contents
    const uint32_t time = f2u(a.time_y);
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
        const int py = y0 + first + k;
        if (py >= a.height) return;
        const ToneAxis row = ROWS == 1 ? tone_axis(py, a.height) : rows[first + k];
        if (row.fragment < 0) continue;
        const f4v c = tex2_border_at(a.in, a.width, a.height, col.i, col.w, row.i, row.w);
        const float noise = wang_hash_noise((uint32_t)px, (uint32_t)py, time) * 0.01f;
        const float r = tonemap1(c.x) + noise, g = tonemap1(c.y) + noise, b = tonemap1(c.z) + noise;
        const size_t idx = (size_t)py * (size_t)a.width + (size_t)px;
        if (RGBA8)
            static_cast<uint32_t*>(a.out)[idx] = unorm8(r) | (unorm8(g) << 8) | (unorm8(b) << 16) | (255u << 24);
        else
            static_cast<float4*>(a.out)[idx] = make_float4(r, g, b, 1.0f);
    }
}

}  // namespace

cudaError_t launch_godrays(const GodrayArgs& a, cudaStream_t s) {
    const unsigned gx = (unsigned)((a.width + 31) / 32);
    const long long pixels = (long long)a.width * a.height;
    if (pixels >= kRows4)
        godrays_kernel<4, false><<<dim3(gx, (unsigned)((a.height + 15) / 16)), 128, 0, s>>>(a);
    else if (pixels >= kRows2)
        godrays_kernel<2, false><<<dim3(gx, (unsigned)((a.height + 7) / 8)), 128, 0, s>>>(a);
    else if (pixels > kFlat)
        godrays_kernel<1, false><<<dim3(gx, (unsigned)((a.height + 3) / 4)), 128, 0, s>>>(a);
    else
        godrays_kernel<1, true><<<dim3(gx, (unsigned)((a.height + 3) / 4)), 128, 0, s>>>(a);
    return cudaGetLastError();
}

namespace {
template <int ROWS> void launch_tonemap_rows(const TonemapArgs& a, cudaStream_t s) {
    const dim3 grid((unsigned)((a.width + 31) / 32), (unsigned)((a.height + kToneWarps * ROWS - 1) / (kToneWarps * ROWS)));
    if (a.format == MT_LDR_RGBA8)
        tonemap_kernel<ROWS, true><<<grid, 32 * kToneWarps, 0, s>>>(a);
    else
        tonemap_kernel<ROWS, false><<<grid, 32 * kToneWarps, 0, s>>>(a);
}
}  // namespace

cudaError_t launch_tonemap(const TonemapArgs& a, cudaStream_t s) {
    const long long pixels = (long long)a.width * a.height;
    if (pixels >= kRows4)
        launch_tonemap_rows<4>(a, s);
    else if (pixels >= kRows2)
        launch_tonemap_rows<2>(a, s);
    else
        launch_tonemap_rows<1>(a, s);
    return cudaGetLastError();
}

}  // namespace mt
