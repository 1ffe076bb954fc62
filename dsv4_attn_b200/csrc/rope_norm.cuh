// Pre- and post-pass of the attention path: partial RoPE on the last n_rope
// dimensions of a vector (split-halves pairing: element i rotates with element
// i + n_rope/2), optionally followed by an RMS norm over the whole vector.  One
// kernel covers the three uses: queries before decode (RoPE by +position, then
// norm), new cache rows before they are quantised (the same with one vector per
// position) and the attention output afterwards (RoPE by -position, no norm).
//
// A warp takes G vectors of one row (they share the position, hence the sine and cosine); all of
// their loads are in flight before the first is used (16-byte loads for the part that is only
// normalised, one rotated pair per lane), and each vector is written once from registers.
// HBM-bound when there are enough vectors; below that the time is one load latency, so the launch takes G = 2 only where
// that still gives every SM eight warps.  The frequencies come with the arguments (a double pow per thread took longer than
// the loads).  Cold memory: 65,536 x 16 vectors of 576 457 -> 418 us, 64 x 128 14.3 -> 10.2 us (with one vector in flight per warp);
// G = 4 at 86 registers leaves 16 warps an SM: 483 us.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "ptx.cuh"
#include "compress_reduce.cuh"   // unpack8

namespace dsv4 {

struct RopeNormArgs {
    int64_t n_rows;            // positions
    int vecs_per_row;          // vectors that share a position (heads)
    int c;                     // vector width; c - n_rope is a multiple of 8 and at most 512
    int n_rope;                // 64
    int inverse;               // rotate by -position
    float eps, theta;
    const __nv_bfloat16* x;
    __nv_bfloat16* out;        // may alias x
    const int32_t* positions;  // [n_rows]
    const __nv_bfloat16* weight;   // [c] or null: no norm
    float freq[32];            // 1 / theta^(2 i / n_rope): the angle of pair i per position
};

constexpr int kRopeNormThreads = 256;

template <int G>
__global__ void __launch_bounds__(kRopeNormThreads, 4) rope_norm_kernel(const __grid_constant__ RopeNormArgs a) {
    ptx::pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int nope = a.c - a.n_rope;
    constexpr int kHalf = 32;               // one rotated pair per lane
    const float freq = a.freq[lane];
    const int groups_per_row = (a.vecs_per_row + G - 1) / G;
    const int64_t n_items = a.n_rows * groups_per_row;
    bool have[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) have[h] = 16 * lane + 8 * h < nope;
    ptx::pdl_wait();
    for (int64_t item = int64_t(blockIdx.x) * (kRopeNormThreads / 32) + (threadIdx.x >> 5); item < n_items;
         item += int64_t(gridDim.x) * (kRopeNormThreads / 32)) {
        const int64_t row = item / groups_per_row;
        const int vec0 = int(item - row * groups_per_row) * G;
        const int n = min(G, a.vecs_per_row - vec0);
        const int64_t at = (row * a.vecs_per_row + vec0) * a.c;
        const __nv_bfloat16* src = a.x + at;
        __nv_bfloat16* dst = a.out + at;
        // elements [16 lane, 16 lane + 16) of the part that is not rotated, in two 16-byte halves, and the pair (lane, lane + 32) of the rest
        uint4 raw[G][2];
        __nv_bfloat16 e1[G], e2[G];
        const int32_t position = ptx::ld(a.positions + row);
#pragma unroll
        for (int j = 0; j < G; ++j) {
            if (j >= n) continue;
            const __nv_bfloat16* v = src + int64_t(j) * a.c;
#pragma unroll
            for (int h = 0; h < 2; ++h) raw[j][h] = have[h] ? ptx::ldg_stream_v4(v + 16 * lane + 8 * h) : make_uint4(0, 0, 0, 0);
            e1[j] = v[nope + lane];
            e2[j] = v[nope + kHalf + lane];
        }
        float sn, cs;
        // the angle in FP32 as the reference forms it
        sincosf((a.inverse ? -float(position) : float(position)) * freq, &sn, &cs);
#pragma unroll
        for (int j = 0; j < G; ++j) {
            if (j >= n) continue;
            __nv_bfloat16* v = dst + int64_t(j) * a.c;
            const float y1 = __bfloat162float(e1[j]), y2 = __bfloat162float(e2[j]);
            float x1 = y1 * cs - y2 * sn, x2 = y1 * sn + y2 * cs;
            if (a.weight != nullptr) {
                float f[16];
                {
                    float lo[8], hi[8];
                    unpack8(raw[j][0], lo);
                    unpack8(raw[j][1], hi);
#pragma unroll
                    for (int k = 0; k < 8; ++k) { f[k] = lo[k];  f[8 + k] = hi[k]; }
                }
                float ss = x1 * x1 + x2 * x2;
#pragma unroll
                for (int k = 0; k < 16; ++k) ss = fmaf(f[k], f[k], ss);
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, d);
                // x / rms * w as x * (1 / rms) * w: the difference is far below the BF16 rounding of the result
                const float inv_rms = 1.f / sqrtf(ss / float(a.c) + a.eps);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (!have[h]) continue;
                    float w[8];
                    unpack8(ptx::ld(reinterpret_cast<const uint4*>(a.weight + 16 * lane + 8 * h)), w);
                    float* g = f + 8 * h;
#pragma unroll
                    for (int k = 0; k < 8; ++k) g[k] = g[k] * inv_rms * w[k];
                    raw[j][h].x = ptx::pack_bf16x2(g[0], g[1]);  raw[j][h].y = ptx::pack_bf16x2(g[2], g[3]);
                    raw[j][h].z = ptx::pack_bf16x2(g[4], g[5]);  raw[j][h].w = ptx::pack_bf16x2(g[6], g[7]);
                }
                x1 = x1 * inv_rms * __bfloat162float(a.weight[nope + lane]);
                x2 = x2 * inv_rms * __bfloat162float(a.weight[nope + kHalf + lane]);
            }
            // without a norm the part that is not rotated is unchanged: written only when out is another buffer
            if (a.weight != nullptr || dst != src) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (have[h]) *reinterpret_cast<uint4*>(v + 16 * lane + 8 * h) = raw[j][h];
            }
            v[nope + lane] = __float2bfloat16_rn(x1);
            v[nope + kHalf + lane] = __float2bfloat16_rn(x2);
        }
    }
}

}  // namespace dsv4
