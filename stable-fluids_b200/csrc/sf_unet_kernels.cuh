// sf_unet_kernels.cuh -- kernels of the warm-start network besides the
// convolution (sf_unet_tc.cuh) and its weight gradient (sf_unet_wgrad.cuh): 2x
// average pooling, 2x nearest upsampling, and the element-wise pieces of
// training.
//
// Activations are channels-last BF16: element (voxel v, channel c) at
// v * C + c, v = x + nx (y + ny z), C a multiple of 16 (padded with zeros).
// Weights are BF16 [tap][cout][cin] with tap = (dz+1)*9 + (dy+1)*3 + (dx+1),
// plus an FP32 master copy for the optimizer. Zero padding at the grid edge.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "sf_types.h"

namespace sfb::net {

// ------------------------------------------------------ element-wise pieces --

// Network input: channel 0 = b * scale, channel 1 = p_prev * scale, the
// other 14 channels zero (16-channel padded tensor). scale = 1 / rms(b) is
// read from *scale.
__global__ void k_pack_input(const float* __restrict__ b, const float* __restrict__ p_prev, const float* __restrict__ scale, float b_factor, __nv_bfloat16* __restrict__ out, size_t n) {
    const float s = *scale;
    for (size_t v = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; v < n; v += static_cast<size_t>(gridDim.x) * blockDim.x) {
        __nv_bfloat162 pair = __floats2bfloat162_rn(b[v] * b_factor * s, p_prev ? p_prev[v] * s : 0.0f);
        uint4 z4 = make_uint4(0, 0, 0, 0);
        uint4 first = z4;
        first.x = *reinterpret_cast<uint32_t*>(&pair);
        reinterpret_cast<uint4*>(out + v * 16)[0] = first;
        reinterpret_cast<uint4*>(out + v * 16)[1] = z4;
    }
}

// scale = 1 / rms(b_factor * b) from the FP64 sum of squares in *sumsq.
__global__ void k_finish_scale(const double* __restrict__ sumsq, double n, float* __restrict__ scale) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        const double rms = sqrt(*sumsq / n);
        *scale = rms > 0.0 ? static_cast<float>(1.0 / rms) : 1.0f;
    }
}

// Adds the block's sum of acc to *out: one atomic a block. (One a warp, of 4736
// blocks, made the sum over 128^3 voxels wait 62 us for its atomics; now it takes 8.)
// 256 threads, all of them.
__device__ __forceinline__ void add_block_sum(double acc, double* out) {
    __shared__ double part[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) acc += part[k];
        atomicAdd(out, acc);
    }
}

__global__ void __launch_bounds__(256) k_sum_squares(const float* __restrict__ b, float b_factor, size_t n, double* __restrict__ out) {
    double acc = 0.0;
    for (size_t v = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; v < n; v += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const double x = static_cast<double>(b[v]) * b_factor;
        acc += x * x;
    }
    add_block_sum(acc, out);
}

// p0 = p_prev + delta / scale (the network predicts the scaled correction).
// p_prev may alias p0 (element-wise, each thread reads before it writes).
__global__ void k_unpack_output(const float* __restrict__ delta, const float* p_prev, const float* __restrict__ scale, float* p0, size_t n) {
    const float inv = 1.0f / *scale;
    for (size_t v = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; v < n; v += static_cast<size_t>(gridDim.x) * blockDim.x) p0[v] = (p_prev ? p_prev[v] : 0.0f) + delta[v] * inv;
}

// The pooling and upsampling kernels below move 8 channels (16 bytes)
// per thread; channel counts, strides and offsets are multiples of 8. The
// 2-D launches give blockIdx.y = y and blockIdx.z = z of the output grid and
// threads over (x, 8-channel chunk) of one row.
struct Bf8 {
    float v[8];
};
__device__ __forceinline__ Bf8 load8(const __nv_bfloat16* p) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
    Bf8 r;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 f = __bfloat1622float2(h[k]);
        r.v[2 * k] = f.x;
        r.v[2 * k + 1] = f.y;
    }
    return r;
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const Bf8& r) {
    uint4 u;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(r.v[2 * k], r.v[2 * k + 1]);
    *reinterpret_cast<uint4*>(p) = u;
}

inline dim3 row_grid(int nx, int chunks_per_voxel, int ny, int nz) { return dim3(static_cast<unsigned>((nx * chunks_per_voxel + 255) / 256), static_cast<unsigned>(ny), static_cast<unsigned>(nz)); }

// 2x2x2 average pooling (even dims of the fine grid); channel stride in_ch.
// Launch: row_grid(coarse.nx, C / 8, coarse.ny, coarse.nz), 256 threads.
__global__ void k_pool2(const __nv_bfloat16* __restrict__ in, int in_ch, int in_off, __nv_bfloat16* __restrict__ out, int C, Dims coarse) {
    const int c8n = C / 8;
    const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= coarse.nx * c8n) return;
    const int x = i / c8n, c = (i % c8n) * 8, y = static_cast<int>(blockIdx.y), z = static_cast<int>(blockIdx.z);
    const int fnx = coarse.nx * 2, fny = coarse.ny * 2;
    Bf8 s{};
    for (int k = 0; k < 8; ++k) {
        const size_t fv = static_cast<size_t>(2 * x + (k & 1)) + static_cast<size_t>(fnx) * (2 * y + ((k >> 1) & 1) + static_cast<size_t>(fny) * (2 * z + (k >> 2)));
        const Bf8 a = load8(in + fv * in_ch + in_off + c);
#pragma unroll
        for (int j = 0; j < 8; ++j) s.v[j] += a.v[j];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s.v[j] *= 0.125f;
    const size_t v = static_cast<size_t>(x) + static_cast<size_t>(coarse.nx) * (y + static_cast<size_t>(coarse.ny) * z);
    store8(out + v * C + c, s);
}

// The gradient through a ReLU whose output is act.
__device__ __forceinline__ void relu_mask(Bf8& g, const Bf8& act) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (!(act.v[j] > 0.0f)) g.v[j] = 0.0f;
}

// Gradient of an encoder level's output, which feeds the skip connection and
// the pooling: channels [off, off + C) of the concatenation's gradient plus 1/8
// of the coarse parent's, rounded to BF16, through the ReLU whose output is act
// (C channels). Launch: row_grid(fine nx, C / 8, fine ny, fine nz). Bound by
// memory: a copy, an addition and a mask in passes of their own took 86 us at
// 128^3 with 16 channels, this one pass 48.
__global__ void k_skip_backward(const __nv_bfloat16* __restrict__ gcat, int cat_ch, int off, const __nv_bfloat16* __restrict__ act, const __nv_bfloat16* __restrict__ gcoarse, int C, Dims coarse, __nv_bfloat16* __restrict__ gfine) {
    const int c8n = C / 8, fnx = coarse.nx * 2, fny = coarse.ny * 2;
    const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= fnx * c8n) return;
    const int x = i / c8n, c = (i % c8n) * 8, y = static_cast<int>(blockIdx.y), z = static_cast<int>(blockIdx.z);
    const size_t cv = static_cast<size_t>(x / 2) + static_cast<size_t>(coarse.nx) * (y / 2 + static_cast<size_t>(coarse.ny) * (z / 2));
    const size_t fv = static_cast<size_t>(x) + static_cast<size_t>(fnx) * (y + static_cast<size_t>(fny) * z);
    const Bf8 skip = load8(gcat + fv * cat_ch + off + c), a = load8(act + fv * C + c);
    Bf8 g = load8(gcoarse + cv * C + c);
#pragma unroll
    for (int j = 0; j < 8; ++j) g.v[j] = __fmaf_rn(0.125f, g.v[j], skip.v[j]);
    relu_mask(g, a);
    store8(gfine + fv * C + c, g);
}

// The input of a decoder level: the coarse tensor upsampled 2x (nearest) in
// channels [0, C), the skip connection in the S after them. Launch:
// row_grid(fine nx, (C + S) / 8, fine ny, fine nz). Bound by its writes (61 us
// for 272 MB at the finest level of 128^3, as long as the two parts in passes of
// their own took; one launch less). Convolutions that wrote their channels of
// the concatenation themselves lost as much as the copy took: 32 bytes of every
// 96, and the pooling and the backward pass read them so too.
__global__ void k_upsample2_concat(const __nv_bfloat16* __restrict__ in, int C, Dims coarse, const __nv_bfloat16* __restrict__ skip, int S, __nv_bfloat16* __restrict__ out) {
    const int c8n = (C + S) / 8, fnx = coarse.nx * 2, fny = coarse.ny * 2;
    const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= fnx * c8n) return;
    const int x = i / c8n, c = (i % c8n) * 8, y = static_cast<int>(blockIdx.y), z = static_cast<int>(blockIdx.z);
    const size_t cv = static_cast<size_t>(x / 2) + static_cast<size_t>(coarse.nx) * (y / 2 + static_cast<size_t>(coarse.ny) * (z / 2));
    const size_t fv = static_cast<size_t>(x) + static_cast<size_t>(fnx) * (y + static_cast<size_t>(fny) * z);
    const __nv_bfloat16* const from = c < C ? in + cv * C + c : skip + fv * S + (c - C);
    *reinterpret_cast<uint4*>(out + fv * (C + S) + c) = *reinterpret_cast<const uint4*>(from);
}

// Backward of the upsampling and of the ReLU before it (its output act): the
// coarse gradient is the sum over its 8 children of channels [off, off + C) of
// the fine gradient. Launch: row_grid(coarse.nx, C / 8, coarse.ny, coarse.nz).
__global__ void k_upsample2_backward(const __nv_bfloat16* __restrict__ gfine, int fine_ch, int off, int C, Dims coarse, const __nv_bfloat16* __restrict__ act, __nv_bfloat16* __restrict__ gcoarse) {
    const int c8n = C / 8, fnx = coarse.nx * 2, fny = coarse.ny * 2;
    const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= coarse.nx * c8n) return;
    const int x = i / c8n, c = (i % c8n) * 8, y = static_cast<int>(blockIdx.y), z = static_cast<int>(blockIdx.z);
    Bf8 s{};
    for (int k = 0; k < 8; ++k) {
        const size_t fv = static_cast<size_t>(2 * x + (k & 1)) + static_cast<size_t>(fnx) * (2 * y + ((k >> 1) & 1) + static_cast<size_t>(fny) * (2 * z + (k >> 2)));
        const Bf8 a = load8(gfine + fv * fine_ch + off + c);
#pragma unroll
        for (int j = 0; j < 8; ++j) s.v[j] += a.v[j];
    }
    const size_t v = static_cast<size_t>(x) + static_cast<size_t>(coarse.nx) * (y + static_cast<size_t>(coarse.ny) * z);
    relu_mask(s, load8(act + v * C + c));
    store8(gcoarse + v * C + c, s);
}

// g *= (act > 0): the gradient through a ReLU whose output is act; n is a
// multiple of 8.
__global__ void k_relu_backward(__nv_bfloat16* __restrict__ g, const __nv_bfloat16* __restrict__ act, size_t n) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n / 8; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        Bf8 v = load8(g + 8 * i);
        relu_mask(v, load8(act + 8 * i));
        store8(g + 8 * i, v);
    }
}

// Mean squared error of the FP32 output against the target; writes the
// gradient (channel 0 of a 16-channel BF16 tensor) and adds the loss sum.
__global__ void __launch_bounds__(256) k_mse(const float* __restrict__ out, const float* __restrict__ target, size_t n, __nv_bfloat16* __restrict__ grad16, double* __restrict__ loss_sum) {
    double acc = 0.0;
    const float k = 2.0f / static_cast<float>(n);
    for (size_t v = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; v < n; v += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const float e = out[v] - target[v];
        acc += static_cast<double>(e) * e;
        uint4 z4 = make_uint4(0, 0, 0, 0);
        __nv_bfloat162 first = __floats2bfloat162_rn(k * e, 0.0f);
        uint4 f = z4;
        f.x = *reinterpret_cast<uint32_t*>(&first);
        reinterpret_cast<uint4*>(grad16 + v * 16)[0] = f;
        reinterpret_cast<uint4*>(grad16 + v * 16)[1] = z4;
    }
    add_block_sum(acc, loss_sum);
}

// Adam on FP32 master weights; refreshes the BF16 copy and the transposed,
// tap-flipped BF16 copy used by the data-gradient convolution.
__global__ void k_adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v, __nv_bfloat16* __restrict__ w16, __nv_bfloat16* __restrict__ w16t, int cout, int cin, size_t n, float lr, float b1, float b2, float eps, float bc1, float bc2) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float wi = w[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
        w[i] = wi;
        if (w16) {
            w16[i] = __float2bfloat16(wi);
            const int tap = static_cast<int>(i / (static_cast<size_t>(cout) * cin));
            const int co = static_cast<int>((i / cin) % cout), ci = static_cast<int>(i % cin);
            w16t[(static_cast<size_t>(26 - tap) * cin + ci) * cout + co] = __float2bfloat16(wi);
        }
    }
}

}  // namespace sfb::net
