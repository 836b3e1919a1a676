// The row kernels of decoder_rows.cuh for a step of one token per sequence: a block per row, four values per thread, in bf16 models.
//
// Such a kernel is a link of a chain of launches a few microseconds long, bound by latencies: launch, one round trip for its operands,
// block-wide sums.  These forms keep the row in registers, meet once per norm (the warps' means and squared distances are put together
// instead of two sums one after the other), and load everything but their predecessor's result before griddepcontrol.wait: every kernel
// of a bf16 step lets its successor start only after its own wait has returned, so what the kernels before the predecessor wrote is complete by then.
#pragma once

#include "decoder_rows.cuh"

namespace gptb200 {
namespace dec {

__device__ __forceinline__ float warp_total(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the block with one barrier; `part` (32 floats of shared memory) belongs to this call alone.
__device__ __forceinline__ float block_total(float v, float *part)
{
    v = warp_total(v);
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    if (lane == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    return warp_total(lane < warps ? part[lane] : 0.0f);
}

// Layer norm of a row spread over the block, columns d .. d + 3 per thread; columns from `width` on do not count.  One barrier.
__device__ __forceinline__ void row_moments(float4 v, int d, int width, float eps, float2 *part, float &mean, float &rstd)
{
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const float in[4] = {d < width ? v.x : 0.0f, d + 1 < width ? v.y : 0.0f, d + 2 < width ? v.z : 0.0f, d + 3 < width ? v.w : 0.0f};
    const auto count = [&](int warp) { return static_cast<float>(min(max(width - warp * 128, 0), 128)); };
    const float n = count(threadIdx.x >> 5);
    const float own = n > 0.0f ? warp_total((in[0] + in[1]) + (in[2] + in[3])) / n : 0.0f;
    float var = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (d + k < width) var = fmaf(in[k] - own, in[k] - own, var);
    var = warp_total(var);
    if (lane == 0) part[threadIdx.x >> 5] = make_float2(own, var);
    __syncthreads();
    const float2 other = lane < warps ? part[lane] : make_float2(0.0f, 0.0f);
    const float m = lane < warps ? count(lane) : 0.0f;
    mean = warp_total(m * other.x) / width;
    rstd = rsqrtf(warp_total(fmaf(m * (other.x - mean), other.x - mean, other.y)) / width + eps);
}

__device__ __forceinline__ float4 normed4(float4 v, float mean, float rstd, float4 w, float4 b)
{
    return make_float4((v.x - mean) * rstd * w.x + b.x, (v.y - mean) * rstd * w.y + b.y, (v.z - mean) * rstd * w.z + b.z, (v.w - mean) * rstd * w.w + b.w);
}

// layer_begin_kernel for one token per sequence, behind the token input's projection (p.side_y): the residual, the earlier states and
// the parameters come before the wait.  768 columns, 12 states, in a step: 5.5 -> 2.9 us from the predecessor's end to its own.
template <typename T>
__global__ void __launch_bounds__(1024)
layer_begin_row_kernel(const LayerBegin<T> p)
{
    __shared__ float squares[32];
    __shared__ float2 moments[32];
    const int d = 4 * threadIdx.x, row = p.row_list ? p.row_list[blockIdx.x] : blockIdx.x;
    const bool live = d < p.pitch;
    const long long at = static_cast<long long>(row) * p.pitch + d;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const StepEntry e = p.entries[p.row_entry[row]];
    float4 v = zero, side_w = zero, sum = zero, w = zero, b = zero, before = zero, share = zero;
    float own = 1.0f;
    if (live) {
        v = load4(p.x_in + at);
        side_w = load4(p.side_w + d);
        w = load4(p.norm_w + d);
        b = load4(p.norm_b + d);
        if (p.shift) {
            share = load4(p.shift + d);
            before = load4(reinterpret_cast<const float *>(e.slot + p.shift_state) + e.parity * p.pitch + d);
        }
        const float *s = p.states + at;
#pragma unroll 4
        for (int j = 0; j < p.n_states - 1; ++j, s += p.state_stride) {
            const float4 u = load4(s);
            const float c = __ldg(p.coef + j);
            sum.x = fmaf(c, u.x, sum.x); sum.y = fmaf(c, u.y, sum.y); sum.z = fmaf(c, u.z, sum.z); sum.w = fmaf(c, u.w, sum.w);
        }
        if (p.n_states > 0) own = __ldg(p.coef + p.n_states - 1);
    }
    grid_dependency_wait();
    grid_dependency_launch();
    const float4 y = live ? load4(p.side_y + at) : zero;
    const float inv = rsqrtf(block_total(fmaf(y.x, y.x, y.y * y.y) + fmaf(y.z, y.z, y.w * y.w), squares) / p.width + p.eps);
    v.x += y.x * inv * side_w.x; v.y += y.y * inv * side_w.y; v.z += y.z * inv * side_w.z; v.w += y.w * inv * side_w.w;
    if (p.n_states > 0) {
        if (live) store4(p.states + (p.n_states - 1) * p.state_stride + at, v);
        v = make_float4(fmaf(own, v.x, sum.x), fmaf(own, v.y, sum.y), fmaf(own, v.z, sum.z), fmaf(own, v.w, sum.w));
    }
    float mean, rstd;
    row_moments(v, d, p.width, p.eps, moments, mean, rstd);
    if (!live) return;
    if (p.x_out) store4(p.x_out + at, v);
    const float4 n = normed4(v, mean, rstd, w, b);
    T *h = p.h + static_cast<long long>(blockIdx.x) * p.pitch + d;
    if (!p.shift) {
        store4(h, n);
        return;
    }
    store4(h, make_float4(n.x + (before.x - n.x) * share.x, n.y + (before.y - n.y) * share.y, n.z + (before.z - n.z) * share.z, n.w + (before.w - n.w) * share.w));
    store4(reinterpret_cast<float *>(e.slot + p.shift_state) + (e.parity ^ 1) * p.pitch + d, n);
}

// sublayer_end_kernel, a row in registers; the residual row is older than the predecessor (the product that writes y).  768 columns: 2.9 -> 1.9 us.
template <typename T>
__global__ void __launch_bounds__(1024)
sublayer_end_row_kernel(float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ norm1_w, const float *__restrict__ norm1_b,
                        const float *__restrict__ norm2_w, const float *__restrict__ norm2_b, T *__restrict__ out, int width, int pitch, float eps)
{
    __shared__ float2 first[32], second[32];
    const int d = 4 * threadIdx.x;
    const bool live = d < pitch;
    const long long at = static_cast<long long>(blockIdx.x) * pitch + d;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 r = zero, w1 = zero, b1 = zero, w2 = zero, b2 = zero;
    if (live) {
        r = load4(x + at);
        w1 = load4(norm1_w + d);
        b1 = load4(norm1_b + d);
        if (norm2_w) {
            w2 = load4(norm2_w + d);
            b2 = load4(norm2_b + d);
        }
    }
    grid_dependency_wait();
    grid_dependency_launch();
    const float4 v = live ? load4(y + at) : zero;
    float mean, rstd;
    row_moments(v, d, width, eps, first, mean, rstd);
    const float4 n = normed4(v, mean, rstd, w1, b1);
    r.x += n.x; r.y += n.y; r.z += n.z; r.w += n.w;
    if (live) store4(x + at, r);
    if (norm2_w) {
        row_moments(r, d, width, eps, second, mean, rstd);
        r = normed4(r, mean, rstd, w2, b2);
    }
    if (live) store4(out + at, r);
}

// residual_norm_kernel for one token per sequence, behind a product (p.y).  Eight rows of 2048: 3.0 -> 2.2 us.
template <typename T>
__global__ void __launch_bounds__(1024)
residual_norm_row_kernel(const ResidualNorm<T> p)
{
    __shared__ float squares[32];
    const int d = 4 * threadIdx.x, row = p.row_list ? p.row_list[blockIdx.x] : blockIdx.x;
    const bool live = d < p.pitch;
    const long long at = static_cast<long long>(row) * p.pitch + d;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const StepEntry e = p.entries[p.row_entry[row]];
    float4 v = zero, w = zero, before = zero;
    if (live) {
        v = load4(p.x_in + at);
        w = load4(p.norm_w + d);
        if (p.mixes) before = load4(reinterpret_cast<const float *>(e.slot + p.shift_state) + e.parity * p.pitch + d);
    }
    grid_dependency_wait();
    grid_dependency_launch();
    const float4 y = live ? load4(p.y + at) : zero;
    v.x = fmaf(p.mult, y.x, v.x); v.y = fmaf(p.mult, y.y, v.y); v.z = fmaf(p.mult, y.z, v.z); v.w = fmaf(p.mult, y.w, v.w);
    const float inv = rsqrtf(block_total(fmaf(v.x, v.x, v.y * v.y) + fmaf(v.z, v.z, v.w * v.w), squares) / p.width + p.eps);
    if (!live) return;
    if (p.x_out) store4(p.x_out + at, v);
    const float4 n = make_float4(v.x * inv * w.x, v.y * inv * w.y, v.z * inv * w.z, v.w * inv * w.w);
    T *h = p.h + static_cast<long long>(blockIdx.x) * p.pitch + d;
    if (!p.mixes) {
        store4(h, n);
        return;
    }
    for (int k = 0; k < p.mixes; ++k) {
        const float4 m = load4(p.mix + k * p.pitch + d);
        store4(h + k * p.mix_stride, make_float4(n.x + (before.x - n.x) * m.x, n.y + (before.y - n.y) * m.y, n.z + (before.z - n.z) * m.z, n.w + (before.w - n.w) * m.w));
    }
    store4(reinterpret_cast<float *>(e.slot + p.shift_state) + (e.parity ^ 1) * p.pitch + d, n);
}

}  // namespace dec
}  // namespace gptb200
