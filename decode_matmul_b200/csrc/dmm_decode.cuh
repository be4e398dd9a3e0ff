// Decode-only kernel: tiled codes -> logical [N, K] weights, through the same table and
// XOR decode core that the matmul kernels use, so a bit-exact check of its output is a
// check of the decode stage itself.
#pragma once
#include "dmm_common.cuh"
#include "dmm_launch.h"

namespace dmm {

constexpr int kDecodeThreads = 1024;
constexpr int kDecodeTiles = 4;  // k-tiles per work item of decode_kernel

// Re-tiles codes from the layout of fast_decode_matmul_cuda -- flat uint32 [N/32][K/16][lane:32],
// word = code(n = 32*nb + lane, j = 2*kp) | code(j = 2*kp + 1) << 16, the completion this library
// defines for the reference's lane-per-column reads (fast_decode_matmul_cuda.cu:106,110-113,130) --
// into the tile layout [N/16][K/32][g:8][t:4][h:2] that every kernel of this library streams.
// One warp per (32-row block, k-tile): 256 contiguous bytes in, 256 contiguous bytes out; lane l
// holds the four codes of row 32*nb + l and trades two of them with lane l ^ 8 (rows g and g + 8
// of a strip share a 32-bit word of the tile layout).
__global__ void __launch_bounds__(256) retile_fast_kernel(const uint32_t *__restrict__ fast, uint32_t *__restrict__ tiled,
                                                          long long N, long long K) {
    const long long KT = K / 32;
    const long long warp = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= (N / 32) * KT) return;
    const long long nb = warp / KT, kt = warp - nb * KT;
    const uint32_t *src = fast + (nb * (K / 16) + 2 * kt) * 32;
    const uint32_t w0 = __ldg(src + lane), w1 = __ldg(src + 32 + lane);  // codes j = 4kt, 4kt+1 | 4kt+2, 4kt+3
    const uint32_t p0 = __shfl_xor_sync(0xffffffffu, w0, 8), p1 = __shfl_xor_sync(0xffffffffu, w1, 8);
    const int strip = lane >> 4, h = (lane >> 3) & 1, g = lane & 7;
    // word (g, t) of the tile layout = code of row g (low half) | code of row g + 8 (high half)
    uint2 out;
    if (h == 0) {  // this lane is row g: writes t = 0, 1 from its w0 and the partner's w0
        out.x = (w0 & 0xFFFFu) | (p0 << 16);
        out.y = (w0 >> 16) | (p0 & 0xFFFF0000u);
    } else {       // this lane is row g + 8: writes t = 2, 3 from the partner's w1 and its own
        out.x = (p1 & 0xFFFFu) | (w1 << 16);
        out.y = (p1 >> 16) | (w1 & 0xFFFF0000u);
    }
    uint32_t *dst = tiled + ((2 * nb + strip) * KT + kt) * 32 + g * 4 + h * 2;
    *reinterpret_cast<uint2 *>(dst) = out;
}

inline int launch_retile_fast(const void *fast, void *tiled, long long N, long long K, cudaStream_t stream) {
    const long long warps = (N / 32) * (K / 32);
    const unsigned blocks = static_cast<unsigned>((warps + 7) / 8);
    retile_fast_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const uint32_t *>(fast),
                                                   reinterpret_cast<uint32_t *>(tiled), N, K);
    return cudaGetLastError();
}


// What bounds it: the stores (eight times the bytes of the codes for fp16).  A warp therefore takes items of
// kDecodeTiles k-tiles of one strip and maps its lanes so that one 16-byte store instruction covers four rows x
// 128 bytes, whole cache lines: lane = (row g mod 4, k-tile parity, code column t).  The words of the next item
// are loaded before the current one is decoded (a warp has four loads in flight while it works on four others),
// and the position of an item costs one 32-bit division.  11008 x 4096 to fp16 (101 MB in and out): 22.6 us, 4.5 TB/s;
// one word per thread and iteration, with one load in flight, 64-byte runs and 64-bit divisions, took 38.9 us.
template <bool kF16>
__global__ void __launch_bounds__(kDecodeThreads) decode_kernel(const uint32_t *__restrict__ words,
                                                               const void *__restrict__ cb, int cb_is_f16,
                                                               void *__restrict__ w_out, long long K, unsigned kt_count,
                                                               unsigned items_per_strip, unsigned items,
                                                               int sign_convention, unsigned dyn_smem_bytes) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t base = smem_u32(smem_raw);
    const uint32_t lut_addr = (base + 0xFFFFu) & ~0xFFFFu;
    if (lut_addr + kLutBytes > base + dyn_smem_bytes) {
        if (threadIdx.x == 0) raise_status(DMM_STATUS_BAD_SMEM);
        return;
    }
    constexpr int P = kDecodeTiles / 2;  // pairs of k-tiles per item
    const int lane = threadIdx.x & 31, t = lane & 3, kp = (lane >> 2) & 1, g4 = lane >> 3;
    const unsigned step = gridDim.x * (kDecodeThreads / 32);
    unsigned item = blockIdx.x * (kDecodeThreads / 32) + (threadIdx.x >> 5);
    // words of an item: pair p of k-tiles, rows g4 and g4 + 4 of the strip's first eight
    uint32_t w[P][2];
    auto load = [&](unsigned it) {
        const unsigned strip = it / items_per_strip, kt0 = (it - strip * items_per_strip) * kDecodeTiles + kp;
        const uint32_t *src = words + static_cast<size_t>(strip) * kt_count * 32 + g4 * 4 + t;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const unsigned kt = kt0 + 2 * p;
#pragma unroll
            for (int h = 0; h < 2; ++h) w[p][h] = kt < kt_count ? __ldg(src + static_cast<size_t>(kt) * 32 + h * 16) : 0u;
        }
    };
    if (item < items) load(item);  // (in flight while the table is built)

    const bool bad = lut_fill(lut_addr, cb, cb_is_f16, sign_convention, kF16 ? kFmtOffset : kFmtTwos, threadIdx.x,
                              kDecodeThreads);
    if (bad) raise_status(DMM_STATUS_BAD_CODEBOOK);
    __syncthreads();
    const LutLane ll = lut_lane(lut_addr, lane);

    for (; item < items; item += step) {
        uint32_t cur[P][2];
#pragma unroll
        for (int p = 0; p < P; ++p) {
            cur[p][0] = w[p][0];
            cur[p][1] = w[p][1];
        }
        if (item + step < items) load(item + step);
        const unsigned strip = item / items_per_strip, kt0 = (item - strip * items_per_strip) * kDecodeTiles + kp;
        const long long n0 = static_cast<long long>(strip) * 16 + g4;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const unsigned kt = kt0 + 2 * p;
            if (kt >= kt_count) continue;
            const long long at = n0 * K + 32ll * kt + 8 * t;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint2 d[2] = {decode8<0>(cur[p][h], ll), decode8<1>(cur[p][h], ll)};  // rows g and g + 8
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const long long o = at + (4 * h + 8 * e) * K;
                    if constexpr (kF16) {
                        uint32_t r[4];
                        bytes_to_quarters(d[e], r);
                        *reinterpret_cast<uint4 *>(reinterpret_cast<__half *>(w_out) + o) = make_uint4(r[0], r[1], r[2], r[3]);
                    } else {
                        *reinterpret_cast<uint2 *>(reinterpret_cast<int8_t *>(w_out) + o) = d[e];
                    }
                }
            }
        }
    }
}

inline int launch_decode(const void *codes, const void *cb, int cb_is_f16, void *w_out, long long N, long long K,
                         int sign_convention, int num_sms, cudaStream_t stream) {
    constexpr unsigned kDyn = 0xFFFFu + kLutBytes + 1;
    const long long kt = K / 32, per_strip = (kt + kDecodeTiles - 1) / kDecodeTiles, items = N / 16 * per_strip;
    if (items >= (1ll << 31)) return DMM_ERR_SHAPE;  // (a terabyte of codes)
    long long blocks = (items + kDecodeThreads / 32 - 1) / (kDecodeThreads / 32);
    if (blocks > num_sms) blocks = num_sms;
    cudaError_t err;
    if (cb_is_f16) {
        err = cudaFuncSetAttribute(decode_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDyn);
        if (err != cudaSuccess) return err;
        decode_kernel<true><<<(unsigned)blocks, kDecodeThreads, kDyn, stream>>>(
            reinterpret_cast<const uint32_t *>(codes), cb, 1, w_out, K, static_cast<unsigned>(kt),
            static_cast<unsigned>(per_strip), static_cast<unsigned>(items), sign_convention, kDyn);
    } else {
        err = cudaFuncSetAttribute(decode_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDyn);
        if (err != cudaSuccess) return err;
        decode_kernel<false><<<(unsigned)blocks, kDecodeThreads, kDyn, stream>>>(
            reinterpret_cast<const uint32_t *>(codes), cb, 0, w_out, K, static_cast<unsigned>(kt),
            static_cast<unsigned>(per_strip), static_cast<unsigned>(items), sign_convention, kDyn);
    }
    return cudaGetLastError();
}

}  // namespace dmm
