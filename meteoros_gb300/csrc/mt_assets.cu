// Noise-volume assets: a 3D volume from its stack of TGA slices, decoded on the
// device.  The reference loads slice z from the file "<name>(z+1).tga" with
// stb_image (forced to 4 components) and copies it to depth z of an RGBA8
// volume (ImageLoadingUtility.cpp:75-139); its assets are run-length encoded
// 32-bit TGAs (image type 10) with the bottom-left origin.
//
// TGA decoding, as the reference's decoder does it:
//   * header: id length (byte 0), colour-map type (1, must be 0), image type
//     (2: raw, 10: run-length), width (12-13), height (14-15), bits per pixel
//     (16: 24 or 32), descriptor (17: bit 5 set = top-left origin); the pixel
//     data follow the image id;
//   * run-length packets: a count byte c (1 + (c & 127) pixels), a run of one
//     pixel value when c & 128, else that many literal pixels; packets run on
//     across scanlines; bytes past the end of the file read as 0;
//   * pixels are B, G, R[, A]; 24-bit pixels get A = 255; rows are flipped to
//     top-first unless the origin is top-left.
//
// One CTA per slice: the file is staged in shared memory, 16 bytes a load (the
// host packs slices at 16-byte offsets), one thread walks the packet headers (a
// serial dependency chain, cheap from shared memory) in rounds, and the CTA's
// threads take the round's pixels in raster order, each finding its packet by
// bisection: stores coalesce and long and short packets cost alike.  The base
// volume's 128 slices take 28 us (ncu, cold caches); with byte loads and a thread
// per packet, storing its pixels one by one across rows, they took 63.
#include <cuda_runtime.h>

#include "mt_kernels.h"

namespace mt {

namespace {

constexpr int kRound = 1024;  // packets per walk/expand round
constexpr int kTgaThreads = 512;

struct File {
    const unsigned char* bytes;  // in shared memory, readable to 8 past the end
    int size;
    // a byte; 0 past the end
    __device__ __forceinline__ unsigned at(int p) const { return p < size ? (unsigned)bytes[p] : 0u; }
    // the pixel at p as an RGBA word
    __device__ __forceinline__ uint32_t pixel(int p, int bytes_pp) const {
        uint32_t w;
        if (p + bytes_pp <= size) {  // four bytes from two aligned words
            const uint32_t* q = reinterpret_cast<const uint32_t*>(bytes) + (p >> 2);
            w = __funnelshift_r(q[0], q[1], 8 * (p & 3));
        } else {
            w = at(p) | (at(p + 1) << 8) | (at(p + 2) << 16) | (at(p + 3) << 24);
        }
        if (bytes_pp == 3) w |= 0xff000000u;
        return __byte_perm(w, 0u, 0x3012u);  // B, G, R, A -> R, G, B, A
    }
};

__global__ void __launch_bounds__(kTgaThreads) tga_decode_kernel(const unsigned char* __restrict__ blob,
                                                                 const TgaSlice* __restrict__ slices, uint32_t* vol,
                                                                 int log2n) {
    extern __shared__ uint4 sm[];
    __shared__ int p_first[kRound], p_pos[kRound];  // a run of one value has the complement of its position
    __shared__ int s_n, s_pos, s_pix;
    const TgaSlice sl = slices[blockIdx.x];
    const File f{reinterpret_cast<const unsigned char*>(sm), (int)sl.size};
    const uint4* src = reinterpret_cast<const uint4*>(blob + sl.offset);
    for (int i = threadIdx.x; i < (f.size + 15) / 16; i += kTgaThreads) sm[i] = __ldg(src + i);
    if (threadIdx.x == 0) s_pix = 0;
    __syncthreads();
    const int bpp = (int)f.at(16) / 8;
    // colour-map type 0 (checked on the host): the pixels follow the image id
    const int data = 18 + (int)f.at(0);
    const bool rle = f.at(2) == 10;
    const bool flip = !(f.at(17) & 32u);
    const int n = 1 << log2n, N = n * n;
    uint32_t* out = vol + (size_t)blockIdx.x * (size_t)N;
    auto store = [&](int i, uint32_t v) {
        const int x = i & (n - 1), y = i >> log2n;
        out[(flip ? n - 1 - y : y) * n + x] = v;
    };
    if (!rle) {
        for (int i = threadIdx.x; i < N; i += kTgaThreads) store(i, f.pixel(data + i * bpp, bpp));
        return;
    }
    if (threadIdx.x == 0) s_pos = data;
    // every round covers at least one pixel, so at most N rounds
    for (int round = 0; round <= N; ++round) {
        const int begin = s_pix;
        __syncthreads();  // every thread has read s_pix before thread 0 moves it
        if (begin >= N) break;
        if (threadIdx.x == 0) {
            int pos = s_pos, pix = begin, k = 0;
            while (k < kRound && pix < N) {
                const unsigned c = f.at(pos);
                const int count = 1 + (int)(c & 127u);
                const bool run = (c & 128u) != 0;
                p_first[k] = pix;
                p_pos[k] = run ? ~(pos + 1) : pos + 1;
                pos += 1 + (run ? bpp : count * bpp);
                pix += count;
                ++k;
            }
            s_n = k;
            s_pos = pos;
            s_pix = pix;
        }
        __syncthreads();
        const int end = s_pix < N ? s_pix : N;
        for (int i = begin + (int)threadIdx.x; i < end; i += kTgaThreads) {
            int lo = 0, hi = s_n - 1;  // the last packet that begins at or before i
            while (lo < hi) {
                const int mid = (lo + hi + 1) / 2;
                if (p_first[mid] <= i)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            const int pos = p_pos[lo];
            store(i, f.pixel(pos < 0 ? ~pos : pos + (i - p_first[lo]) * bpp, bpp));
        }
        __syncthreads();
    }
}

}  // namespace

cudaError_t launch_tga_decode(const unsigned char* blob, const TgaSlice* slices, int n_slices, size_t max_size,
                              uint32_t* vol, int log2n, cudaStream_t s) {
    const size_t shared = (max_size + 15) / 16 * 16 + 16;
    cudaError_t e = cudaFuncSetAttribute(tga_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
    if (e != cudaSuccess) return e;
    tga_decode_kernel<<<n_slices, kTgaThreads, shared, s>>>(blob, slices, vol, log2n);
    return cudaGetLastError();
}

}  // namespace mt
