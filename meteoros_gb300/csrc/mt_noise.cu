// Seeded noise-volume generation on the GPU.
//
// The reference loads pre-baked Nubis textures (Sky.cpp:25-58); these kernels
// generate the same four volumes from a seed instead.  Lattice hashing is
// built on the integer core of the reference's WangHashNoise
// (shaders/postProcess_ToneMap.frag:52-66).  Noise families: tileable Worley
// (cellular) noise, Perlin's improved gradient noise (Perlin 2002) and fBm
// sums, arranged as the Nubis cloud textures describe them (R = Perlin-Worley,
// GBA = Worley fBm at rising frequencies).  Every step is an IEEE FP32
// +, -, *, / or sqrt in a fixed order (this file is compiled with
// -fmad=false), so the output is bit-identical to the CPU generator that the
// tests hold it against.
//
// One thread per texel; the base volume, 27 cells in each of nine Worley
// octaves a texel, takes 2x2x2 texels a thread.  Outputs: RGBA8 words plus IEEE half and bfloat16
// copies for the precision form, all in create3DTextureFromMany2DTextures
// layout (x fastest, then y, then slice z).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "mt_kernels.h"

namespace mt {
namespace {

__device__ __forceinline__ uint32_t wang(uint32_t u, uint32_t v, uint32_t s) {
    uint32_t seed = (u * 1664525u + v) + s;
    seed = (seed ^ 61u) ^ (seed >> 16u);
    seed *= 9u;
    seed = seed ^ (seed >> 4u);
    seed *= 0x27d4eb2du;
    seed = seed ^ (seed >> 15u);
    return seed;
}
__device__ __forceinline__ uint32_t hash3(uint32_t x, uint32_t y, uint32_t z, uint32_t s) {
    return wang(wang(x, y, s), z, s);
}
__device__ __forceinline__ uint32_t salt(uint32_t s, uint32_t k) { return s + k * 0x9E3779B9u; }
__device__ __forceinline__ float clamp01(float x) {
    x = x < 0.0f ? 0.0f : x;
    return 1.0f < x ? 1.0f : x;
}
__device__ __forceinline__ float lerpf(float a, float b, float t) { return a + t * (b - a); }
__device__ __forceinline__ float fade(float t) { return ((t * t) * t) * ((t * ((t * 6.0f) - 15.0f)) + 10.0f); }

// Inverted Worley noise with period F cells; p in cell units.
__device__ float worley3(float px, float py, float pz, int F, uint32_t s) {
    const uint32_t m = (uint32_t)F - 1u;
    float fx = floorf(px), fy = floorf(py), fz = floorf(pz);
    int cx = (int)fx, cy = (int)fy, cz = (int)fz;
    float rx = px - fx, ry = py - fy, rz = pz - fz;
    float best = 100.0f;
    for (int dz = -1; dz <= 1; ++dz) {
        const uint32_t wz = (uint32_t)(cz + dz) & m;
        for (int dy = -1; dy <= 1; ++dy) {
            const uint32_t wy = (uint32_t)(cy + dy) & m;
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                const uint32_t wx = (uint32_t)(cx + dx) & m;
                const uint32_t h = hash3(wx, wy, wz, s);
                float ox = (float)(h & 1023u) * (1.0f / 1024.0f);
                float oy = (float)((h >> 10) & 1023u) * (1.0f / 1024.0f);
                float oz = (float)((h >> 20) & 1023u) * (1.0f / 1024.0f);
                float vx = ((float)dx + ox) - rx;
                float vy = ((float)dy + oy) - ry;
                float vz = ((float)dz + oz) - rz;
                float d2 = vx * vx + vy * vy + vz * vz;
                best = d2 < best ? d2 : best;
            }
        }
    }
    float d = sqrtf(best);
    return 1.0f - (d < 1.0f ? d : 1.0f);
}

__device__ __forceinline__ float grad2(uint32_t h, float x, float y) {
    switch (h & 7u) {
        case 0: return x + y;
        case 1: return -x + y;
        case 2: return x - y;
        case 3: return -x - y;
        case 4: return x;
        case 5: return -x;
        case 6: return y;
        default: return -y;
    }
}

__device__ float perlin2(float px, float py, int F, uint32_t s) {
    const uint32_t m = (uint32_t)F - 1u;
    float fx = floorf(px), fy = floorf(py);
    int ix = (int)fx, iy = (int)fy;
    float x = px - fx, y = py - fy;
    float u = fade(x), v = fade(y);
    uint32_t x0 = (uint32_t)ix & m, x1 = (uint32_t)(ix + 1) & m;
    uint32_t y0 = (uint32_t)iy & m, y1 = (uint32_t)(iy + 1) & m;
    float g00 = grad2(wang(x0, y0, s), x, y);
    float g10 = grad2(wang(x1, y0, s), x - 1.0f, y);
    float g01 = grad2(wang(x0, y1, s), x, y - 1.0f);
    float g11 = grad2(wang(x1, y1, s), x - 1.0f, y - 1.0f);
    return lerpf(lerpf(g00, g10, u), lerpf(g01, g11, u), v);
}

__device__ float perlin_fbm2(float x, float y, int F, int octaves, uint32_t s) {
    float sum = 0.0f, amp = 1.0f, tot = 0.0f;
    int f = F;
    for (int o = 0; o < octaves; ++o) {
        float ff = (float)f;
        sum = sum + amp * perlin2(x * ff, y * ff, f, s + (uint32_t)o);
        tot = tot + amp;
        amp = amp * 0.5f;
        f *= 2;
    }
    return sum / tot;
}

__device__ __forceinline__ uint32_t q8(float v) { return (uint32_t)(int)floorf(clamp01(v) * 255.0f + 0.5f); }

// A texel in its three storages; channels clamped to [0, 1].
struct Texel {
    uint32_t u8;
    uint2 h16, b16;
};
__device__ __forceinline__ Texel make_texel(float r, float g, float b, float a) {
    r = clamp01(r);
    g = clamp01(g);
    b = clamp01(b);
    a = clamp01(a);
    Texel t;
    t.u8 = q8(r) | (q8(g) << 8) | (q8(b) << 16) | (q8(a) << 24);
    const __half2 hl = __floats2half2_rn(r, g), hh = __floats2half2_rn(b, a);
    t.h16 = make_uint2(*reinterpret_cast<const uint32_t*>(&hl), *reinterpret_cast<const uint32_t*>(&hh));
    const __nv_bfloat162 bl = __floats2bfloat162_rn(r, g), bh = __floats2bfloat162_rn(b, a);
    t.b16 = make_uint2(*reinterpret_cast<const uint32_t*>(&bl), *reinterpret_cast<const uint32_t*>(&bh));
    return t;
}
__device__ __forceinline__ void put(const NoiseOut& o, size_t i, float r, float g, float b, float a) {
    const Texel t = make_texel(r, g, b, a);
    o.u8[i] = t.u8;
    o.h16[i] = t.h16;
    o.b16[i] = t.b16;
}

// ---------------------------------------------------------------------------
// 128^3: R Perlin-Worley, G/B/A Worley fBm at base frequencies 4/8/16 (octaves
// F, 2F, 4F).  ALU-bound: every texel looks at 27 feature points in each of
// nine Worley octaves and at 8 corners in each of four Perlin octaves.
//
// A thread owns the 2x2x2 texels at even coordinates: in every octave (at most
// 64 cells over 128 texels) they lie in one cell, so they share each feature
// point's unpacking, its three pairs of offsets and squares, and the Perlin
// corners' gradients.  A block owns 32x8x8 texels and hashes the feature points
// of its cells and their neighbours once, into shared memory (1229 words).
//
// The Worley part is exact whatever the order of its operations: in units of
// 1/1024 cell a feature point is a whole number below 1024 and so is a texel
// centre's position in its cell ((2x + 1) F / 256 cells, F at least 4), so
// offsets are whole numbers below 2048 and a squared distance is one below
// 2^24.  Offsets come from the hash's 10-bit fields dropped into the mantissa
// of a power of two.  The Perlin part's corner dot products are sums of
// multiples of 1/256 below 4, exact too; its fades and lerps keep their order.
//
// One thread per texel, hashing as it went, the kernel took 766 us (ncu, cold
// caches); now 131 us with the small outputs beside it.  All of mt_generate_volumes:
// 864 -> 164 us.
// ---------------------------------------------------------------------------
constexpr int kTileX = 32, kTileY = 8, kTileZ = 8;

// The cells of frequency F a tile touches, with a neighbour on either side.
template <int F> struct TileCells {
    static constexpr int along(int texels) { return (texels * F / MT_BASE_N > 1 ? texels * F / MT_BASE_N : 1) + 2; }
    static constexpr int NX = along(kTileX), NY = along(kTileY), NZ = along(kTileZ), COUNT = NX * NY * NZ;
};

template <int F> __device__ __forceinline__ void hash_cells(uint32_t* cells, int x0, int y0, int z0, uint32_t s) {
    using T = TileCells<F>;
    const int cx = x0 * F / MT_BASE_N - 1, cy = y0 * F / MT_BASE_N - 1, cz = z0 * F / MT_BASE_N - 1;
    for (int i = threadIdx.x; i < T::COUNT; i += blockDim.x) {
        const int ix = i % T::NX, iy = (i / T::NX) % T::NY, iz = i / (T::NX * T::NY);
        cells[i] = hash3((uint32_t)(cx + ix) & (F - 1u), (uint32_t)(cy + iy) & (F - 1u),
                         (uint32_t)(cz + iz) & (F - 1u), s);
    }
}

// Inverted Worley noise at frequency F of the texels (x, y, z) + {0, 1}^3 (x
// fastest); (x, y, z) even, inside the tile at (x0, y0, z0).
template <int F>
__device__ __forceinline__ void worley8(float w[8], const uint32_t* cells, int x0, int y0, int z0, int x, int y,
                                        int z) {
    using T = TileCells<F>;
    const int cx = x * F / MT_BASE_N - x0 * F / MT_BASE_N, cy = y * F / MT_BASE_N - y0 * F / MT_BASE_N,
              cz = z * F / MT_BASE_N - z0 * F / MT_BASE_N;
    const uint32_t* base = cells + (cz * T::NY + cy) * T::NX + cx;
    // a texel centre's offset in its cell, in 1/1024 cell; the next texel's is 8F on
    const float rx = (float)(((2 * x + 1) * F * 4) & 1023), ry = (float)(((2 * y + 1) * F * 4) & 1023),
                rz = (float)(((2 * z + 1) * F * 4) & 1023);
    // squared distances as their bits (non-negative floats order like integers),
    // for the three-input integer minimum
    int best[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) best[i] = __float_as_int(100.0f * 1048576.0f);
#pragma unroll 1
    for (int dz = 0; dz < 3; ++dz) {
        const float bz = 8192.0f + (rz - (float)(1024 * (dz - 1)));
#pragma unroll 1
        for (int dy = 0; dy < 3; ++dy) {
            const float by = 8192.0f + (ry - (float)(1024 * (dy - 1)));
            const uint32_t* row = base + (dz * T::NY + dy) * T::NX;
            int d2[3][8];
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
                const uint32_t h = row[dx];
                const float bx = 8388608.0f + (rx - (float)(1024 * (dx - 1)));
                // 2^23 + the field at bit 0, 2^13 + the field at bit 10
                const float X = __uint_as_float((h & 1023u) | 0x4B000000u) - bx;
                const float Y = __uint_as_float((h & 0xFFC00u) | 0x46000000u) - by;
                const float Z = __uint_as_float(((h >> 10) & 0xFFC00u) | 0x46000000u) - bz;
                const float X1 = X - 8.0f * F, Y1 = Y - 8.0f * F, Z1 = Z - 8.0f * F;
                const float xx[2] = {X * X, X1 * X1};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float yv = (i & 2) ? Y1 : Y, xy = fmaf(yv, yv, xx[i & 1]);
                    d2[dx][i] = __float_as_int(fmaf(Z, Z, xy));
                    d2[dx][i + 4] = __float_as_int(fmaf(Z1, Z1, xy));
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) best[i] = min(__vimin3_s32(best[i], d2[0][i], d2[1][i]), d2[2][i]);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float d = sqrtf(__int_as_float(best[i]) * (1.0f / 1048576.0f));
        w[i] = 1.0f - (d < 1.0f ? d : 1.0f);
    }
}

// The three octaves F, 2F, 4F over the cells at c, summed into out as they come.
template <int F>
__device__ __forceinline__ void worley_fbm8(float out[8], const uint32_t* c, int x0, int y0, int z0, int x, int y,
                                            int z) {
    float w[8];
    worley8<F>(w, c, x0, y0, z0, x, y, z);
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = w[i] * 0.625f;
    c += TileCells<F>::COUNT;
    worley8<2 * F>(w, c, x0, y0, z0, x, y, z);
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = out[i] + w[i] * 0.25f;
    c += TileCells<2 * F>::COUNT;
    worley8<4 * F>(w, c, x0, y0, z0, x, y, z);
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = out[i] + w[i] * 0.125f;
}
template <int F> __device__ __forceinline__ void hash_fbm(uint32_t* c, int x0, int y0, int z0, uint32_t s) {
    hash_cells<F>(c, x0, y0, z0, s);
    hash_cells<2 * F>(c + TileCells<F>::COUNT, x0, y0, z0, s + 1u);
    hash_cells<4 * F>(c + TileCells<F>::COUNT + TileCells<2 * F>::COUNT, x0, y0, z0, s + 2u);
}
template <int F> constexpr int kFbmCells = TileCells<F>::COUNT + TileCells<2 * F>::COUNT + TileCells<4 * F>::COUNT;

// Perlin's gradient of a corner's hash as a vector of -1, 0, 1: the dot product
// is one of x, y plus or minus one of y, x, z.
__device__ __forceinline__ void grad3(uint32_t h, float& gx, float& gy, float& gz) {
    h &= 15u;
    const float su = (h & 1u) ? -1.0f : 1.0f, sv = (h & 2u) ? -1.0f : 1.0f;
    const bool u_is_x = h < 8u, v_is_y = h < 4u, v_is_x = h == 12u || h == 14u;
    gx = u_is_x ? su : (v_is_x ? sv : 0.0f);
    gy = u_is_x ? (v_is_y ? sv : 0.0f) : su;
    gz = (v_is_y || v_is_x) ? 0.0f : sv;
}

// Perlin noise at frequency F of the eight texels.
__device__ __forceinline__ void perlin8(float out[8], int x, int y, int z, int F, uint32_t s) {
    const uint32_t m = (uint32_t)F - 1u;
    const uint32_t cx = (uint32_t)(x * F / MT_BASE_N), cy = (uint32_t)(y * F / MT_BASE_N),
                   cz = (uint32_t)(z * F / MT_BASE_N);
    float px[2], py[2], pz[2], u[2], v[2], w[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        px[i] = (float)(((2 * (x + i) + 1) * F) & 255) * (1.0f / 256.0f);
        py[i] = (float)(((2 * (y + i) + 1) * F) & 255) * (1.0f / 256.0f);
        pz[i] = (float)(((2 * (z + i) + 1) * F) & 255) * (1.0f / 256.0f);
        u[i] = fade(px[i]);
        v[i] = fade(py[i]);
        w[i] = fade(pz[i]);
    }
    float plane[2][8];  // the bilinear blend of each z plane's corners, per texel
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        float a[2][8];  // the blend along x of each row's corners
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            float g[2][8];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                float gx, gy, gz;
                grad3(hash3((cx + (uint32_t)k) & m, (cy + (uint32_t)b) & m, (cz + (uint32_t)c) & m, s), gx, gy, gz);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    g[k][i] = gx * (px[i & 1] - (float)k) + gy * (py[(i >> 1) & 1] - (float)b) +
                              gz * (pz[i >> 2] - (float)c);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) a[b][i] = lerpf(g[0][i], g[1][i], u[i & 1]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) plane[c][i] = lerpf(a[0][i], a[1][i], v[(i >> 1) & 1]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = lerpf(plane[0][i], plane[1][i], w[i >> 2]);
}

__device__ __forceinline__ void gen_base_tile(uint32_t s, const NoiseOut& o, int tile) {
    constexpr int N = MT_BASE_N, TX = N / kTileX, TY = N / kTileY;
    __shared__ uint32_t cells[kFbmCells<4> + kFbmCells<8> + kFbmCells<16>];
    const int x0 = tile % TX * kTileX, y0 = tile / TX % TY * kTileY, z0 = tile / (TX * TY) * kTileZ;
    hash_fbm<4>(cells, x0, y0, z0, salt(s, 2));
    hash_fbm<8>(cells + kFbmCells<4>, x0, y0, z0, salt(s, 3));
    hash_fbm<16>(cells + kFbmCells<4> + kFbmCells<8>, x0, y0, z0, salt(s, 4));
    __syncthreads();
    const int tid = (int)threadIdx.x;
    const int x = x0 + 2 * (tid & 15), y = y0 + 2 * ((tid >> 4) & 3), z = z0 + 2 * (tid >> 6);
    float r[8], g[8], b[8], a[8];
    {
        // perlin_fbm: octaves 4, 8, 16, 32 at amplitudes 1, 1/2, 1/4, 1/8
        float amp = 1.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = 0.0f;
#pragma unroll 1
        for (int oct = 0; oct < 4; ++oct) {
            float p[8];
            perlin8(p, x, y, z, 4 << oct, salt(s, 1) + (uint32_t)oct);
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = r[i] + amp * p[i];
            amp = amp * 0.5f;
        }
    }
    worley_fbm8<4>(g, cells, x0, y0, z0, x, y, z);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float p01 = clamp01((r[i] / 1.875f) * 0.5f + 0.5f);
        r[i] = (p01 - (g[i] - 1.0f)) / (1.0f - (g[i] - 1.0f));
    }
    worley_fbm8<8>(b, cells + kFbmCells<4>, x0, y0, z0, x, y, z);
    worley_fbm8<16>(a, cells + kFbmCells<4> + kFbmCells<8>, x0, y0, z0, x, y, z);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {  // the two texels of a row as one store per storage
        const size_t at = (((size_t)(z + (i >> 2)) * N + (size_t)(y + ((i >> 1) & 1))) * N + (size_t)x) / 2;
        const Texel t0 = make_texel(r[i], g[i], b[i], a[i]), t1 = make_texel(r[i + 1], g[i + 1], b[i + 1], a[i + 1]);
        reinterpret_cast<uint2*>(o.u8)[at] = make_uint2(t0.u8, t1.u8);
        reinterpret_cast<uint4*>(o.h16)[at] = make_uint4(t0.h16.x, t0.h16.y, t1.h16.x, t1.h16.y);
        reinterpret_cast<uint4*>(o.b16)[at] = make_uint4(t0.b16.x, t0.b16.y, t1.b16.x, t1.b16.y);
    }
}

// 32^3: Worley at frequencies 8/16/32 in R/G/B.
__device__ __forceinline__ void gen_detail_texel(uint32_t s, const NoiseOut& o, uint32_t i) {
    const int N = MT_DETAIL_N;
    const int x = (int)(i % N), y = (int)((i / N) % N), z = (int)(i / (N * N));
    const float inv = 1.0f / (float)N;
    float px = ((float)x + 0.5f) * inv, py = ((float)y + 0.5f) * inv, pz = ((float)z + 0.5f) * inv;
    float r = worley3(px * 8.0f, py * 8.0f, pz * 8.0f, 8, salt(s, 5));
    float g = worley3(px * 16.0f, py * 16.0f, pz * 16.0f, 16, salt(s, 6));
    float b = worley3(px * 32.0f, py * 32.0f, pz * 32.0f, 32, salt(s, 7));
    put(o, i, r, g, b, 1.0f);
}

// 128^2 curl of a tileable Perlin fBm potential (central differences).
__device__ __forceinline__ void gen_curl_texel(uint32_t s, const NoiseOut& o, uint32_t i) {
    const int N = MT_CURL_N;
    const int x = (int)(i % N), y = (int)(i / N);
    const float inv = 1.0f / (float)N;
    float px = ((float)x + 0.5f) * inv, py = ((float)y + 0.5f) * inv;
    const uint32_t sp = salt(s, 8);
    float dy = perlin_fbm2(px, py + inv, 4, 3, sp) - perlin_fbm2(px, py - inv, 4, 3, sp);
    float dx = perlin_fbm2(px + inv, py, 4, 3, sp) - perlin_fbm2(px - inv, py, 4, 3, sp);
    float cx = dy * 4.0f;
    float cy = -(dx * 4.0f);
    float mag = sqrtf(cx * cx + cy * cy);
    put(o, i, cx * 0.5f + 0.5f, cy * 0.5f + 0.5f, mag, 1.0f);
}

// 512^2 weather: R coverage, G precipitation, B cloud type, A = 1.
__device__ __forceinline__ void gen_weather_texel(uint32_t s, const NoiseOut& o, uint32_t i) {
    const int N = MT_WEATHER_N;
    const int x = (int)(i % N), y = (int)(i / N);
    const float inv = 1.0f / (float)N;
    float px = ((float)x + 0.5f) * inv, py = ((float)y + 0.5f) * inv;
    float f = perlin_fbm2(px, py, 4, 6, salt(s, 9)) * 0.5f + 0.5f;
    float cov = clamp01(f * 1.2f - 0.2f);
    float precip = (float)(wang((uint32_t)x, (uint32_t)y, salt(s, 10)) >> 8) * (1.0f / 16777216.0f);
    uint32_t t = wang((uint32_t)(x >> 6), (uint32_t)(y >> 6), salt(s, 11)) % 3u;
    float type = t == 0u ? 0.0f : (t == 1u ? 0.5f : 1.0f);
    put(o, i, cov, precip, type, 1.0f);
}

// One launch for the four outputs: the base volume's tiles first, then the small
// ones, whose blocks fill its last wave (29 us as three launches of their own).
constexpr int kGenThreads = 256;
constexpr int kBaseTiles = (MT_BASE_N / kTileX) * (MT_BASE_N / kTileY) * (MT_BASE_N / kTileZ);
constexpr int kDetailBlocks = MT_DETAIL_N * MT_DETAIL_N * MT_DETAIL_N / kGenThreads;
constexpr int kCurlBlocks = MT_CURL_N * MT_CURL_N / kGenThreads;
constexpr int kWeatherBlocks = MT_WEATHER_N * MT_WEATHER_N / kGenThreads;
static_assert((kTileX / 2) * (kTileY / 2) * (kTileZ / 2) == kGenThreads, "a thread owns 2x2x2 texels of the tile");

__global__ void __launch_bounds__(kGenThreads, 3) gen_volumes_kernel(uint32_t s, NoiseOut base, NoiseOut detail,
                                                                     NoiseOut curl, NoiseOut weather) {
    int block = (int)blockIdx.x;
    if (block < kBaseTiles) {
        gen_base_tile(s, base, block);
        return;
    }
    block -= kBaseTiles;
    if (block < kWeatherBlocks) {
        gen_weather_texel(s, weather, (uint32_t)(block * kGenThreads) + threadIdx.x);
        return;
    }
    block -= kWeatherBlocks;
    if (block < kDetailBlocks)
        gen_detail_texel(s, detail, (uint32_t)(block * kGenThreads) + threadIdx.x);
    else
        gen_curl_texel(s, curl, (uint32_t)((block - kDetailBlocks) * kGenThreads) + threadIdx.x);
}

__global__ void __launch_bounds__(kGenThreads) gen_weather_kernel(uint32_t s, NoiseOut o) {
    gen_weather_texel(s, o, blockIdx.x * kGenThreads + threadIdx.x);
}

// ---------------------------------------------------------------------------
// The layouts the samplers read, from a volume's texels, in one pass over every
// volume that changed (LayoutJob):
//   * RGBA8 plane quads of a volume, bilinear cells of an image: entry (x, y[,
//     z]) holds the four texels a fetch at that cell interpolates in plane z,
//     {(x0,y0), (x1,y0), (x0,y1), (x1,y1)} with x1 = (x + 1) mod N, y1 likewise
//     (REPEAT), as one 16-byte word;
//   * the same of a volume's IEEE half and bfloat16 texels, a 32-byte entry
//     {(x0,y0), (x1,y0)}, {(x0,y1), (x1,y1)} each;
//   * FROM_U8 (uploaded and decoded volumes): the 16-bit texels themselves,
//     c / 255 rounded to nearest even.  c * (1 / 255) rounds to the same half and
//     the same bfloat16 for each of the 256 bytes.
// Bound by its stores: 96 bytes a texel of the base volume (112 with the 16-bit
// texels), 32 bytes an instruction.  The four outputs of the generator take
// 32 us (ncu, cold caches; 201 MB written); one kernel per layout and volume,
// each reading its input again, took 65, and twelve launches of an upload 98.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void store32(uint4* p, uint2 a, uint2 b, uint2 c, uint2 d) {
    asm volatile("st.global.v8.u32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(b.x),
                 "r"(b.y), "r"(c.x), "r"(c.y), "r"(d.x), "r"(d.y)
                 : "memory");
}
__device__ __forceinline__ void u8_to_16(uint32_t v, uint2& h, uint2& b) {
    const float k = 1.0f / 255.0f;
    const float c0 = (float)(v & 0xffu) * k, c1 = (float)((v >> 8) & 0xffu) * k, c2 = (float)((v >> 16) & 0xffu) * k,
                c3 = (float)(v >> 24) * k;
    const __half2 hl = __floats2half2_rn(c0, c1), hh = __floats2half2_rn(c2, c3);
    h = make_uint2(*reinterpret_cast<const uint32_t*>(&hl), *reinterpret_cast<const uint32_t*>(&hh));
    const __nv_bfloat162 bl = __floats2bfloat162_rn(c0, c1), bh = __floats2bfloat162_rn(c2, c3);
    b = make_uint2(*reinterpret_cast<const uint32_t*>(&bl), *reinterpret_cast<const uint32_t*>(&bh));
}

struct LayoutArgs {
    LayoutJob job[kMaxLayoutJobs];
    unsigned first_block[kMaxLayoutJobs + 1];
    int n_jobs;
};

template <bool FROM_U8> __global__ void __launch_bounds__(256) layouts_kernel(const __grid_constant__ LayoutArgs a) {
    int k = 0;
    while (k + 1 < a.n_jobs && blockIdx.x >= a.first_block[k + 1]) ++k;
    const LayoutJob& j = a.job[k];
    const unsigned i = (blockIdx.x - a.first_block[k]) * 256u + threadIdx.x;
    const unsigned n = (unsigned)j.n, m = n - 1u;
    const unsigned x = i & m, row = i & ~m, y = (i / n) & m, plane = row - y * n;
    const unsigned x1 = (x + 1u) & m, row1 = plane + ((y + 1u) & m) * n;
    const unsigned at[4] = {row + x, row + x1, row1 + x, row1 + x1};
    uint32_t t[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) t[c] = j.u8[at[c]];
    j.quads[i] = make_uint4(t[0], t[1], t[2], t[3]);
    uint2 h[4], b[4];
    if (FROM_U8) {
#pragma unroll
        for (int c = 0; c < 4; ++c) u8_to_16(t[c], h[c], b[c]);
        j.h16[i] = h[0];
        j.b16[i] = b[0];
    }
    if (!j.quads_h16) return;  // an image
    if (!FROM_U8) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            h[c] = j.h16[at[c]];
            b[c] = j.b16[at[c]];
        }
    }
    store32(j.quads_h16 + 2u * i, h[0], h[1], h[2], h[3]);
    store32(j.quads_b16 + 2u * i, b[0], b[1], b[2], b[3]);
}

}  // namespace

cudaError_t launch_layouts(const LayoutJob* jobs, int n_jobs, bool from_u8, cudaStream_t s) {
    if (n_jobs <= 0) return cudaSuccess;
    LayoutArgs a = {};
    a.n_jobs = n_jobs;
    unsigned blocks = 0;
    for (int k = 0; k < n_jobs; ++k) {
        const unsigned n = (unsigned)jobs[k].n;
        a.job[k] = jobs[k];
        a.first_block[k] = blocks;
        blocks += n * n * (jobs[k].quads_h16 ? n : 1u) / 256u;  // n is a power of two, at least 32
    }
    a.first_block[n_jobs] = blocks;
    if (from_u8)
        layouts_kernel<true><<<blocks, 256, 0, s>>>(a);
    else
        layouts_kernel<false><<<blocks, 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_generate_volumes(uint32_t seed, NoiseOut base, NoiseOut detail, NoiseOut curl, NoiseOut weather,
                                    cudaStream_t s) {
    gen_volumes_kernel<<<kBaseTiles + kWeatherBlocks + kDetailBlocks + kCurlBlocks, kGenThreads, 0, s>>>(
        seed, base, detail, curl, weather);
    return cudaGetLastError();
}
cudaError_t launch_generate_weather(uint32_t seed, NoiseOut o, cudaStream_t s) {
    gen_weather_kernel<<<kWeatherBlocks, kGenThreads, 0, s>>>(seed, o);
    return cudaGetLastError();
}

}  // namespace mt
