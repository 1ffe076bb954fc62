// CSA compressor, second pass: per output block and channel, a softmax over the
// 2m gating logits (m of the block's own rows on the a-side, m rows of the
// previous block on the b-side, each plus a per-position bias) weights the 2m
// value rows.  A pure streaming kernel: every input element is read once with
// vector loads, one thread owns 4 consecutive channels of one output block (8-byte loads: a
// thread then holds 16 vectors = 32 registers of raw data).  Bound by HBM and, close behind, by instruction issue: the
// arithmetic is done two channels at a time (packed BF16 for the reference maximum, packed FP32 for the rest), 230
// instructions a thread instead of 420, and three blocks fit an SM at 80 registers (at four and 64 registers it
// spills).  32k rows of 576, back to back on rotating inputs: 30.8 -> 28.5 us, 5.6 TB/s (28.1 without the bound on
// the reference maximum below).  The grid is sized so that all SMs hold two waves
// of resident blocks.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <math_constants.h>
#include <stdint.h>

#include "ptx.cuh"

namespace dsv4 {

struct CompressReduceArgs {
    int B, n, n_blocks, c_out, m;
    const __nv_bfloat16* C_a;  const __nv_bfloat16* C_b;
    const __nv_bfloat16* Z_a;  const __nv_bfloat16* Z_b;
    const __nv_bfloat16* B_a;  const __nv_bfloat16* B_b;
    __nv_bfloat16* out;
    int64_t stride_c_b, stride_c_n;        // element strides of the four input streams
    int64_t stride_out_b, stride_out_blk;
};

constexpr int kCompressThreads = 256;

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
}

// Four BF16 values and their FP32 unpacking.
__device__ __forceinline__ uint2 load_stream4(const __nv_bfloat16* p) {
    uint2 v;
    asm volatile("ld.global.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ void unpack4(const uint2& v, float (&f)[4]) {
    f[0] = __uint_as_float(v.x << 16);  f[1] = __uint_as_float(v.x & 0xFFFF0000u);
    f[2] = __uint_as_float(v.y << 16);  f[3] = __uint_as_float(v.y & 0xFFFF0000u);
}

// VEC = 4: 8-byte vectors (c_out % 4 == 0 and rows aligned to the vector); VEC = 1: any c_out.
template <int M, int VEC>
__global__ void __launch_bounds__(kCompressThreads, VEC == 4 ? 3 : 2) compress_reduce_kernel(const CompressReduceArgs a) {
    ptx::pdl_trigger();
    ptx::pdl_wait();
    const int vecs = a.c_out / VEC;
    const int64_t total = int64_t(a.B) * a.n_blocks * vecs;
    for (int64_t idx = int64_t(blockIdx.x) * kCompressThreads + threadIdx.x; idx < total;
         idx += int64_t(gridDim.x) * kCompressThreads) {
        const int v = int(idx % vecs);
        const int64_t bb = idx / vecs;
        const int blk = int(bb % a.n_blocks);
        const int b = int(bb / a.n_blocks);
        const int ch = v * VEC;
        const int64_t row_a = int64_t(b) * a.stride_c_b + int64_t(blk) * M * a.stride_c_n + ch;
        const int64_t row_b = row_a - int64_t(M) * a.stride_c_n;      // previous block (blk > 0 only)
        float o[VEC];
        if constexpr (VEC == 4) {
            using V = uint2;
            // all 4m data vectors in flight first; the biases are small and cached, they are
            // re-read where needed so that the raw data can stay in registers
            V za[M], ca[M], zb[M], cb[M];
#pragma unroll
            for (int j = 0; j < M; ++j) {
                za[j] = load_stream4(a.Z_a + row_a + j * a.stride_c_n);
                ca[j] = load_stream4(a.C_a + row_a + j * a.stride_c_n);
            }
            const bool has_b = blk > 0;
            if (has_b) {
#pragma unroll
                for (int j = 0; j < M; ++j) {
                    zb[j] = load_stream4(a.Z_b + row_b + j * a.stride_c_n);
                    cb[j] = load_stream4(a.C_b + row_b + j * a.stride_c_n);
                }
            }
            auto bias = [&](int j, bool bside) { return ptx::ld(reinterpret_cast<const V*>((bside ? a.B_b : a.B_a) + int64_t(j) * a.c_out + ch)); };
            // The reference maximum is found in packed BF16 arithmetic.  A BF16 sum is within 2^-8 of the FP32 one; raised by that much the
            // reference is no lower than the true maximum, so that no weight exceeds 1, and while it is small (kNear) the weight of
            // the true maximum is no smaller than 2^-1.5.  Larger logits (and infinities) take the exact maximum and differences formed
            // before the factor log2(e): from 2^15 up the weights of finite logits would overflow or all vanish otherwise.
            constexpr int P = VEC / 2;
            constexpr float kLog2e = 1.4426950408889634f, kNear = 128.f;
            __nv_bfloat162 pm[P];
#pragma unroll
            for (int k = 0; k < P; ++k) pm[k] = __float2bfloat162_rn(-CUDART_INF_F);
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                if (side == 1 && !has_b) break;
#pragma unroll
                for (int j = 0; j < M; ++j) {
                    const V z = side ? zb[j] : za[j], u = bias(j, side == 1);
                    const __nv_bfloat162 *z2 = reinterpret_cast<const __nv_bfloat162*>(&z), *u2 = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
                    for (int k = 0; k < P; ++k) pm[k] = __hmax2(pm[k], __hadd2(z2[k], u2[k]));
                }
            }
            __nv_bfloat162 size = __habs2(pm[0]);
#pragma unroll
            for (int k = 1; k < P; ++k) size = __hmax2(size, __habs2(pm[k]));
            if (__hble2(size, __float2bfloat162_rn(kNear))) {
                // the logits are formed in FP32, two channels an instruction
                const uint64_t log2e2 = ptx::pack_f32x2(kLog2e, kLog2e);
                uint64_t nref[P], sum2[P], acc2[P];         // nref: -(reference maximum) * log2(e)
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    const float lo = __low2float(pm[k]), hi = __high2float(pm[k]);
                    nref[k] = ptx::pack_f32x2(fmaf(fabsf(lo), -kLog2e / 256.f, -lo * kLog2e), fmaf(fabsf(hi), -kLog2e / 256.f, -hi * kLog2e));
                    sum2[k] = 0ull;  acc2[k] = 0ull;
                }
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                    if (side == 1 && !has_b) break;
#pragma unroll
                    for (int j = 0; j < M; ++j) {
                        float z[VEC], u[VEC], c[VEC];
                        unpack4(side ? zb[j] : za[j], z);
                        unpack4(bias(j, side == 1), u);
                        unpack4(side ? cb[j] : ca[j], c);
#pragma unroll
                        for (int k = 0; k < P; ++k) {
                            const uint64_t t = ptx::add_f32x2(ptx::pack_f32x2(z[2 * k], z[2 * k + 1]), ptx::pack_f32x2(u[2 * k], u[2 * k + 1]));
                            float e0, e1;
                            ptx::unpack_f32x2(ptx::fma_f32x2(t, log2e2, nref[k]), e0, e1);
                            const uint64_t e = ptx::pack_f32x2(ptx::ex2(e0), ptx::ex2(e1));
                            sum2[k] = ptx::add_f32x2(sum2[k], e);
                            acc2[k] = ptx::fma_f32x2(e, ptx::pack_f32x2(c[2 * k], c[2 * k + 1]), acc2[k]);
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    float s0, s1, a0, a1;
                    ptx::unpack_f32x2(sum2[k], s0, s1);
                    ptx::unpack_f32x2(acc2[k], a0, a1);
                    o[2 * k] = a0 / s0;
                    o[2 * k + 1] = a1 / s1;
                }
            } else {
                float zmax[VEC], sum[VEC], acc[VEC];
#pragma unroll
                for (int k = 0; k < VEC; ++k) { zmax[k] = -CUDART_INF_F;  sum[k] = 0.f;  acc[k] = 0.f; }
#pragma unroll
                for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
                    for (int side = 0; side < 2; ++side) {
                        if (side == 1 && !has_b) break;
#pragma unroll
                        for (int j = 0; j < M; ++j) {
                            float z[VEC], u[VEC], c[VEC];
                            unpack4(side ? zb[j] : za[j], z);
                            unpack4(bias(j, side == 1), u);
                            unpack4(side ? cb[j] : ca[j], c);
#pragma unroll
                            for (int k = 0; k < VEC; ++k) {
                                if (pass == 0) {
                                    zmax[k] = fmaxf(zmax[k], z[k] + u[k]);
                                } else {
                                    const float e = ptx::ex2((z[k] + u[k] - zmax[k]) * kLog2e);
                                    sum[k] += e;
                                    acc[k] = fmaf(e, c[k], acc[k]);
                                }
                            }
                        }
                    }
#pragma unroll
                    for (int k = 0; k < VEC; ++k)
                        if (pass == 0 && !(fabsf(zmax[k]) < CUDART_INF_F)) zmax[k] = 0.f;      // all -inf (or NaN): avoid inf - inf
                }
#pragma unroll
                for (int k = 0; k < VEC; ++k) o[k] = acc[k] / sum[k];
            }
        } else {
            float z[2 * M], c[2 * M];
#pragma unroll
            for (int j = 0; j < M; ++j) {
                z[j] = __bfloat162float(a.Z_a[row_a + j * a.stride_c_n]) + __bfloat162float(a.B_a[int64_t(j) * a.c_out + ch]);
                c[j] = __bfloat162float(a.C_a[row_a + j * a.stride_c_n]);
                if (blk > 0) {
                    z[M + j] = __bfloat162float(a.Z_b[row_b + j * a.stride_c_n]) + __bfloat162float(a.B_b[int64_t(j) * a.c_out + ch]);
                    c[M + j] = __bfloat162float(a.C_b[row_b + j * a.stride_c_n]);
                } else {
                    z[M + j] = -CUDART_INF_F;
                    c[M + j] = 0.f;
                }
            }
            float zmax = z[0];
#pragma unroll
            for (int j = 1; j < 2 * M; ++j) zmax = fmaxf(zmax, z[j]);
            if (!(zmax > -CUDART_INF_F) || !(zmax < CUDART_INF_F)) zmax = 0.f;
            float sum = 0.f, acc = 0.f;
#pragma unroll
            for (int j = 0; j < 2 * M; ++j) {
                const float e = ptx::ex2((z[j] - zmax) * 1.4426950408889634f);
                sum += e;
                acc = fmaf(e, c[j], acc);
            }
            o[0] = acc / sum;
        }
        __nv_bfloat16* dst = a.out + int64_t(b) * a.stride_out_b + int64_t(blk) * a.stride_out_blk + ch;
        if constexpr (VEC == 4) {
            uint2 w;
            w.x = ptx::pack_bf16x2(o[0], o[1]);  w.y = ptx::pack_bf16x2(o[2], o[3]);
            *reinterpret_cast<uint2*>(dst) = w;
        } else {
            dst[0] = __float2bfloat16_rn(o[0]);
        }
    }
}

}  // namespace dsv4
