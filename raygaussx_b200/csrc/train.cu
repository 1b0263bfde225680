// What a training iteration does around the operator, on the device: the parameterisation of the Gaussians
// (scripts/train.py:123 through classes/point_cloud.py:509-559), the image loss
// (1 - l) L1 + l (1 - SSIM) with its gradient (scripts/train.py:128-137, utils/loss_utils.py:17-62),
// the densification statistics (classes/point_cloud.py:468-479) and Adam.
//
// All of it is bound by memory on a large scene and by launches on a small one: written with framework
// operators an iteration is some 250 launches, and every intermediate (five blurred images, the squared moments,
// the concatenated colours' gradient ...) makes a round trip through memory.
#include "rgx_internal.cuh"
#include "device_math.cuh"

namespace rgx {

namespace {

// ---------------------------------------------------------------- parameterisation
__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// One thread per colour coefficient (per four of them at degree 3), the first n also take a Gaussian's geometry, the first
// n * lobes a lobe.
// Bound by memory: reads and writes every value once (3 M Gaussians, degree 3: 1.4 GB each way in 0.23 ms, 6 TB/s; one value per thread 0.52).
template <int K>                     // coefficients per channel; 0: any number
__global__ void __launch_bounds__(256) activate_kernel(rgx_activation a) {
    after_previous();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int k_all = K ? K : a.sh_coeffs;
    if (K == 16) {                       // four values per thread, written 16 bytes at a time
        if (i < (size_t)a.n * 12) {
            const size_t row = i >> 2;
            const int k = (int)(i & 3) * 4;
            const float* sh = a.sh + row * 15 + k - 1;
            const float first = k == 0 ? load_streaming(a.rgb + row) : load_streaming(sh);
            reinterpret_cast<float4*>(a.color)[i] = make_float4(first, load_streaming(sh + 1), load_streaming(sh + 2), load_streaming(sh + 3));
        }
    } else if (i < (size_t)a.n * 3 * k_all) {
        const size_t row = i / k_all;
        const int k = (int)(i - row * k_all);
        a.color[i] = k == 0 ? a.rgb[row] : a.sh[row * (k_all - 1) + (k - 1)];
    }
    if (i < (size_t)a.n) {
#pragma unroll
        for (int c = 0; c < 3; ++c) a.scales[3 * i + c] = expf(a.log_scales[3 * i + c]);
        if (a.quaternions) {
            const float q0 = a.raw_quaternions[4 * i], q1 = a.raw_quaternions[4 * i + 1], q2 = a.raw_quaternions[4 * i + 2], q3 = a.raw_quaternions[4 * i + 3];
            const float len = sqrtf((q0 * q0 + q2 * q2) + (q1 * q1 + q3 * q3));      // the order of torch.norm: same bits
            reinterpret_cast<float4*>(a.quaternions)[i] = make_float4(q0 / len, q1 / len, q2 / len, q3 / len);
        }
    }
    if (i < (size_t)a.n * a.num_lobes) {
        a.sharpness[i] = softplus(a.raw_sharpness[i]);
        if (a.lobe_axis) {
            const float x = a.raw_axis[3 * i], y = a.raw_axis[3 * i + 1], z = a.raw_axis[3 * i + 2];
            const float len = sqrtf(x * x + y * y + z * z);
            a.lobe_axis[3 * i] = x / len; a.lobe_axis[3 * i + 1] = y / len; a.lobe_axis[3 * i + 2] = z / len;
        }
    }
}

// The same with the arrows reversed: a.scales ... a.lobe_axis hold the gradients of the activated values, and the gradients of
// the parameters are written to g_*.
template <int K>
__global__ void __launch_bounds__(256) activate_backward_kernel(rgx_activation a, rgx_activation_grads g) {
    after_previous();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int k_all = K ? K : a.sh_coeffs;
    if (K == 16) {
        if (g.color && i < (size_t)a.n * 12) {
            const size_t row = i >> 2;
            const int k = (int)(i & 3) * 4;
            const float4 v = load_streaming(reinterpret_cast<const float4*>(g.color) + i);
            if (k != 0) { if (g.sh) g.sh[row * 15 + k - 1] = v.x; }
            else if (g.rgb) g.rgb[row] = v.x;
            if (g.sh) {
                float* sh = g.sh + row * 15 + k;
                sh[0] = v.y; sh[1] = v.z; sh[2] = v.w;
            }
        }
    } else if (g.color && i < (size_t)a.n * 3 * k_all) {
        const size_t row = i / k_all;
        const int k = (int)(i - row * k_all);
        const float v = g.color[i];
        if (k == 0) { if (g.rgb) g.rgb[row] = v; }
        else if (g.sh) g.sh[row * (k_all - 1) + (k - 1)] = v;
    }
    if (i < (size_t)a.n) {
        if (g.scales && g.log_scales)
#pragma unroll
            for (int c = 0; c < 3; ++c) g.log_scales[3 * i + c] = g.scales[3 * i + c] * a.scales[3 * i + c];
        if (g.quaternions && g.raw_quaternions) {
            // d(q / |q|): the part of the gradient across q, over |q|
            float q[4], d[4], dot = 0.f, len2 = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) { q[c] = a.raw_quaternions[4 * i + c]; d[c] = g.quaternions[4 * i + c]; len2 += q[c] * q[c]; }
            const float inv = 1.0f / sqrtf(len2);
#pragma unroll
            for (int c = 0; c < 4; ++c) dot += q[c] * inv * d[c];
#pragma unroll
            for (int c = 0; c < 4; ++c) g.raw_quaternions[4 * i + c] = (d[c] - q[c] * inv * dot) * inv;
        }
    }
    if (i < (size_t)a.n * a.num_lobes) {
        if (g.sharpness && g.raw_sharpness) {
            const float x = a.raw_sharpness[i];
            g.raw_sharpness[i] = g.sharpness[i] * (x > 20.f ? 1.0f : 1.0f / (1.0f + expf(-x)));
        }
        if (g.lobe_axis && g.raw_axis) {
            float v[3], d[3], dot = 0.f, len2 = 0.f;
#pragma unroll
            for (int c = 0; c < 3; ++c) { v[c] = a.raw_axis[3 * i + c]; d[c] = g.lobe_axis[3 * i + c]; len2 += v[c] * v[c]; }
            const float inv = 1.0f / sqrtf(len2);
#pragma unroll
            for (int c = 0; c < 3; ++c) dot += v[c] * inv * d[c];
#pragma unroll
            for (int c = 0; c < 3; ++c) g.raw_axis[3 * i + c] = (d[c] - v[c] * inv * dot) * inv;
        }
    }
}

// ---------------------------------------------------------------- image loss
constexpr int kRad = 5, kTaps = 2 * kRad + 1;      // 11-tap window, sigma 1.5 (utils/loss_utils.py:22-31)
constexpr int kTile = 32, kSpan = kTile + 2 * kRad, kRows = 8;
constexpr float kSsimC1 = 0.01f * 0.01f, kSsimC2 = 0.03f * 0.03f;

struct Taps {
    float w[kTaps];
};

struct LossArgs {
    const float* rays;       // [h * fy, w * fx, 3]
    const float* target;     // [3, h, w]
    int w, h, fx, fy;
    float lambda;
    Taps taps;
};

// pixel (x, y) of channel c: the mean of its rays; zero outside, as the blur's padding
__device__ __forceinline__ float pixel_of(const LossArgs& a, int c, int x, int y) {
    const size_t W = (size_t)a.w * a.fx;
    if (a.fx == 1 && a.fy == 1) return a.rays[((size_t)y * W + x) * 3 + c];
    float sum = 0.f;
    for (int j = 0; j < a.fy; ++j)
        for (int i = 0; i < a.fx; ++i) sum += a.rays[(((size_t)y * a.fy + j) * W + (size_t)x * a.fx + i) * 3 + c];
    return sum / (float)(a.fx * a.fy);
}

__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int t = threadIdx.y * kTile + threadIdx.x;
    __syncthreads();
    if ((t & 31) == 0) red[t >> 5] = v;
    __syncthreads();
    float s = 0.f;
    for (int i = 0; i < kRows; ++i) s += red[i];
    return s;
}

// A block takes a tile of 32x32 pixels of one channel: both images with a rim of five pixels into shared memory, the five blurred
// moments along x, then along y, all without leaving the SM.  Per pixel the derivative of SSIM with respect to the blurred
// image, its blurred square and the blurred product (maps, three planes), which is what the backward needs to blur.
// About 190 arithmetic instructions per pixel and channel; 1256x828: 63 us and 50 us for the backward, where framework operators took 1.9 ms for both.
template <bool SSIM>
__global__ void __launch_bounds__(kTile * kRows) image_loss_kernel(LossArgs a, float* maps, float2* partial) {
    after_previous();
    __shared__ float s_x[SSIM ? kSpan : 1][kSpan + 1], s_y[SSIM ? kSpan : 1][kSpan + 1];
    __shared__ float s_h[5][SSIM ? kSpan : 1][kTile];
    __shared__ float red[kRows];
    const int c = blockIdx.z, x0 = blockIdx.x * kTile, y0 = blockIdx.y * kTile, tx = threadIdx.x, ty = threadIdx.y;
    const size_t plane = (size_t)a.w * a.h;
    float l1 = 0.f, ss = 0.f;
    if (SSIM) {
        for (int j = ty; j < kSpan; j += 2 * kRows)
#pragma unroll
            for (int i = tx; i < kSpan; i += kTile) {
                // two rows at a time, or each pair of loads would wait for the stores of the one before
                float u[2], v[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int x = x0 + i - kRad, y = y0 + j + k * kRows - kRad;
                    const bool in = j + k * kRows < kSpan && x >= 0 && y >= 0 && x < a.w && y < a.h;
                    u[k] = in ? pixel_of(a, c, x, y) : 0.f;
                    v[k] = in ? a.target[c * plane + (size_t)y * a.w + x] : 0.f;
                }
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    if (j + k * kRows < kSpan) { s_x[j + k * kRows][i] = u[k]; s_y[j + k * kRows][i] = v[k]; }
            }
        __syncthreads();
        for (int j = ty; j < kSpan; j += kRows) {
            float m1 = 0.f, m2 = 0.f, xx = 0.f, yy = 0.f, xy = 0.f;
#pragma unroll
            for (int k = 0; k < kTaps; ++k) {
                const float u = s_x[j][tx + k], v = s_y[j][tx + k], w = a.taps.w[k];
                m1 = fmaf(w, u, m1); m2 = fmaf(w, v, m2);
                xx = fmaf(w, u * u, xx); yy = fmaf(w, v * v, yy); xy = fmaf(w, u * v, xy);
            }
            s_h[0][j][tx] = m1; s_h[1][j][tx] = m2; s_h[2][j][tx] = xx; s_h[3][j][tx] = yy; s_h[4][j][tx] = xy;
        }
        __syncthreads();
    }
    for (int j = ty; j < kTile; j += kRows) {
        const int x = x0 + tx, y = y0 + j;
        if (x >= a.w || y >= a.h) continue;
        if (!SSIM) {
            l1 += fabsf(pixel_of(a, c, x, y) - a.target[c * plane + (size_t)y * a.w + x]);
            continue;
        }
        l1 += fabsf(s_x[j + kRad][tx + kRad] - s_y[j + kRad][tx + kRad]);
        float v[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < kTaps; ++k)
#pragma unroll
            for (int q = 0; q < 5; ++q) v[q] = fmaf(a.taps.w[k], s_h[q][j + k][tx], v[q]);
        const float m1 = v[0], m2 = v[1], m11 = m1 * m1, m22 = m2 * m2, m12 = m1 * m2;
        const float s1 = v[2] - m11, s2 = v[3] - m22, s12 = v[4] - m12;
        const float A = 2.f * m12 + kSsimC1, B = 2.f * s12 + kSsimC2, C = m11 + m22 + kSsimC1, D = s1 + s2 + kSsimC2;
        const float inv = 1.0f / (C * D), S = A * B * inv;
        ss += S;
        if (maps) {
            const float d_s1 = -S / D, d_s12 = 2.f * A * inv;
            const size_t at = c * plane + (size_t)y * a.w + x;
            maps[at] = 2.f * m2 * B * inv - 2.f * m1 * S / C - 2.f * m1 * d_s1 - m2 * d_s12;
            maps[3 * plane + at] = d_s1;
            maps[6 * plane + at] = d_s12;
        }
    }
    l1 = block_sum(l1, red);
    if (SSIM) ss = block_sum(ss, red);
    if (tx == 0 && ty == 0) partial[(blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = make_float2(l1, ss);
}

// The partial sums in a fixed order, in double: (1 - l) L1 + l (1 - SSIM).
__global__ void __launch_bounds__(256) image_loss_sum_kernel(const float2* partial, int count, double values, float lambda, float* loss) {
    after_previous();
    __shared__ double s_a[256], s_b[256];
    double l1 = 0., ss = 0.;
    for (int i = threadIdx.x; i < count; i += 256) { l1 += partial[i].x; ss += partial[i].y; }
    s_a[threadIdx.x] = l1; s_b[threadIdx.x] = ss;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) { s_a[threadIdx.x] += s_a[threadIdx.x + o]; s_b[threadIdx.x] += s_b[threadIdx.x + o]; }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        float out = (1.0f - lambda) * (float)(s_a[0] / values);
        if (lambda != 0.f) out += lambda * (1.0f - (float)(s_b[0] / values));
        *loss = out;
    }
}

// Gradient of the loss with respect to the rays: the three maps blurred, and the sign of the difference.
template <bool SSIM>
__global__ void __launch_bounds__(kTile * kRows) image_loss_backward_kernel(LossArgs a, const float* maps, const float* grad_loss, float* out) {
    after_previous();
    __shared__ float s_m[3][SSIM ? kSpan : 1][kSpan + 1];
    __shared__ float s_h[3][SSIM ? kSpan : 1][kTile];
    const int c = blockIdx.z, x0 = blockIdx.x * kTile, y0 = blockIdx.y * kTile, tx = threadIdx.x, ty = threadIdx.y;
    const size_t plane = (size_t)a.w * a.h;
    if (SSIM) {
        for (int j = ty; j < kSpan; j += kRows)
            for (int i = tx; i < kSpan; i += kTile) {
                const int x = x0 + i - kRad, y = y0 + j - kRad;
                const bool in = x >= 0 && y >= 0 && x < a.w && y < a.h;
#pragma unroll
                for (int q = 0; q < 3; ++q) s_m[q][j][i] = in ? maps[(size_t)(3 * q + c) * plane + (size_t)y * a.w + x] : 0.f;
            }
        __syncthreads();
        for (int j = ty; j < kSpan; j += kRows) {
            float v[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < kTaps; ++k)
#pragma unroll
                for (int q = 0; q < 3; ++q) v[q] = fmaf(a.taps.w[k], s_m[q][j][tx + k], v[q]);
#pragma unroll
            for (int q = 0; q < 3; ++q) s_h[q][j][tx] = v[q];
        }
        __syncthreads();
    }
    const float per_value = (grad_loss ? *grad_loss : 1.0f) / (float)(3 * plane) / (float)(a.fx * a.fy);
    for (int j = ty; j < kTile; j += kRows) {
        const int x = x0 + tx, y = y0 + j;
        if (x >= a.w || y >= a.h) continue;
        const float u = pixel_of(a, c, x, y), t = a.target[c * plane + (size_t)y * a.w + x];
        float g = (1.0f - a.lambda) * (u > t ? 1.0f : u < t ? -1.0f : 0.0f);
        if (SSIM) {
            float v[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < kTaps; ++k)
#pragma unroll
                for (int q = 0; q < 3; ++q) v[q] = fmaf(a.taps.w[k], s_h[q][j + k][tx], v[q]);
            g -= a.lambda * (v[0] + 2.f * u * v[1] + t * v[2]);
        }
        g *= per_value;
        const size_t W = (size_t)a.w * a.fx;
        for (int jj = 0; jj < a.fy; ++jj)
            for (int i = 0; i < a.fx; ++i) out[(((size_t)y * a.fy + jj) * W + (size_t)x * a.fx + i) * 3 + c] = g;
    }
}

LossArgs loss_args(const float* rays, const float* target, int w, int h, int fx, int fy, float lambda) {
    LossArgs a{rays, target, w, h, fx, fy, lambda, {}};
    double sum = 0., v[kTaps];
    for (int k = 0; k < kTaps; ++k) sum += v[k] = exp(-(double)((k - kRad) * (k - kRad)) / (2.0 * 1.5 * 1.5));
    for (int k = 0; k < kTaps; ++k) a.taps.w[k] = (float)(v[k] / sum);
    return a;
}
dim3 loss_grid(int w, int h) { return dim3((w + kTile - 1) / kTile, (h + kTile - 1) / kTile, 3); }

// ---------------------------------------------------------------- statistics, Adam
// classes/point_cloud.py:468-485; a null norm_sum counts only (gradients of Gaussians not visible).
__global__ void __launch_bounds__(256) gradient_stats_kernel(int n, const float* pos, const float* grad, const float* eye, float* norm_sum, float* count,
                                                             float* also) {
    after_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gx = grad[3 * (size_t)i], gy = grad[3 * (size_t)i + 1], gz = grad[3 * (size_t)i + 2];
    const float norm = sqrtf(gx * gx + gy * gy + gz * gz);
    if (norm_sum) {
        const float dx = pos[3 * (size_t)i] - eye[0], dy = pos[3 * (size_t)i + 1] - eye[1], dz = pos[3 * (size_t)i + 2] - eye[2];
        norm_sum[i] += norm * fmaxf(sqrtf(dx * dx + dy * dy + dz * dz), 1.0f);
    }
    if (norm > 0.f) {
        count[i] += 1.0f;
        if (also) also[i] += 1.0f;
    }
}

constexpr int kAdamChunk = 4096;     // values per block: sixteen per thread

struct AdamTable {
    rgx_adam_tensor t[RGX_ADAM_MAX];
    unsigned first[RGX_ADAM_MAX + 1];   // first block of each tensor
    int count;
    float rest1, beta2, rest2, eps;     // rest = 1 - beta, rounded once
};

__device__ __forceinline__ void adam_value(float& p, float g, float& m, float& v, float rest1, float beta2, float rest2, float step, float inv_root,
                                           float eps) {
    m = fmaf(rest1, g - m, m);
    v = fmaf(v, beta2, rest2 * g * g);
    p -= step * (m / fmaf(sqrtf(v), inv_root, eps));
}

// All tensors of a step in one launch.  Bound by memory: 16 bytes read and 12 written per value; 177 M values: 0.76 ms, 6.5 TB/s (foreach
// operators, a launch and a round trip per term of the formula: 3.0 ms).
__global__ void __launch_bounds__(256) adam_kernel(const __grid_constant__ AdamTable a) {
    after_previous();
    int k = 0;
    while (k + 1 < a.count && blockIdx.x >= a.first[k + 1]) ++k;
    const rgx_adam_tensor& t = a.t[k];
    const size_t begin = (size_t)(blockIdx.x - a.first[k]) * kAdamChunk, end = min(begin + kAdamChunk, (size_t)t.n);
    const bool wide = ((reinterpret_cast<uintptr_t>(t.param) | reinterpret_cast<uintptr_t>(t.grad) | reinterpret_cast<uintptr_t>(t.exp_avg) |
                        reinterpret_cast<uintptr_t>(t.exp_avg_sq)) & 15u) == 0;
    if (wide) {
        const size_t whole = begin + ((end - begin) & ~(size_t)3);
#pragma unroll 2
        for (size_t i = begin + 4 * threadIdx.x; i < whole; i += 4 * 256) {
            float4 p = *reinterpret_cast<float4*>(t.param + i), m = *reinterpret_cast<float4*>(t.exp_avg + i), v = *reinterpret_cast<float4*>(t.exp_avg_sq + i);
            const float4 g = load_streaming(reinterpret_cast<const float4*>(t.grad + i));
            adam_value(p.x, g.x, m.x, v.x, a.rest1, a.beta2, a.rest2, t.step_size, t.inv_root, a.eps);
            adam_value(p.y, g.y, m.y, v.y, a.rest1, a.beta2, a.rest2, t.step_size, t.inv_root, a.eps);
            adam_value(p.z, g.z, m.z, v.z, a.rest1, a.beta2, a.rest2, t.step_size, t.inv_root, a.eps);
            adam_value(p.w, g.w, m.w, v.w, a.rest1, a.beta2, a.rest2, t.step_size, t.inv_root, a.eps);
            *reinterpret_cast<float4*>(t.param + i) = p;
            __stcs(reinterpret_cast<float4*>(t.exp_avg + i), m);
            __stcs(reinterpret_cast<float4*>(t.exp_avg_sq + i), v);
        }
    }
    for (size_t i = (wide ? begin + ((end - begin) & ~(size_t)3) : begin) + threadIdx.x; i < end; i += 256)
        adam_value(t.param[i], t.grad[i], t.exp_avg[i], t.exp_avg_sq[i], a.rest1, a.beta2, a.rest2, t.step_size, t.inv_root, a.eps);
}

int done(cudaError_t e) {
    if (e == cudaSuccess) return RGX_OK;
    (void)cudaGetLastError();
    return RGX_E_CUDA;
}

}  // namespace

}  // namespace rgx

using namespace rgx;

static size_t activation_threads(const rgx_activation* a) {
    const int colors = a->sh_coeffs == 16 ? 12 : 3 * a->sh_coeffs;
    return (size_t)a->n * (size_t)(colors > a->num_lobes ? colors : a->num_lobes);
}

extern "C" RGX_API int rgx_activate(int device, const rgx_activation* a, rgx_stream stream) {
    if (!a || a->n < 0 || a->sh_coeffs < 1 || a->num_lobes < 0) return RGX_E_INVALID;
    if (a->n == 0) return RGX_OK;
    if (!a->log_scales || !a->rgb || (a->sh_coeffs > 1 && !a->sh) || !a->scales || !a->color || (a->sh_coeffs == 16 && !aligned16(a->color)) || (a->quaternions && (!a->raw_quaternions || !aligned16(a->quaternions))) ||
        (a->num_lobes > 0 && (!a->raw_sharpness || !a->sharpness || (a->lobe_axis && !a->raw_axis))))
        return RGX_E_INVALID;
    DeviceGuard guard(device);
    if (!guard.ok) return done(cudaErrorInvalidDevice);
    const unsigned blocks = (unsigned)((activation_threads(a) + 255) / 256);
    cudaStream_t s = (cudaStream_t)stream;
    switch (a->sh_coeffs) {
        case 4: launch_after(activate_kernel<4>, blocks, 256, 0, s, *a); break;
        case 9: launch_after(activate_kernel<9>, blocks, 256, 0, s, *a); break;
        case 16: launch_after(activate_kernel<16>, blocks, 256, 0, s, *a); break;
        default: launch_after(activate_kernel<0>, blocks, 256, 0, s, *a);
    }
    return done(cudaGetLastError());
}

extern "C" RGX_API int rgx_activate_backward(int device, const rgx_activation* a, const rgx_activation_grads* g, rgx_stream stream) {
    if (!a || !g || a->n < 0 || a->sh_coeffs < 1 || a->num_lobes < 0) return RGX_E_INVALID;
    if (a->n == 0) return RGX_OK;
    if ((a->sh_coeffs == 16 && !aligned16(g->color)) || (g->log_scales && (!g->scales || !a->scales)) || (g->raw_quaternions && (!g->quaternions || !a->raw_quaternions)) ||
        (g->raw_sharpness && (!g->sharpness || !a->raw_sharpness)) || (g->raw_axis && (!g->lobe_axis || !a->raw_axis)))
        return RGX_E_INVALID;
    DeviceGuard guard(device);
    if (!guard.ok) return done(cudaErrorInvalidDevice);
    const unsigned blocks = (unsigned)((activation_threads(a) + 255) / 256);
    cudaStream_t s = (cudaStream_t)stream;
    switch (a->sh_coeffs) {
        case 4: launch_after(activate_backward_kernel<4>, blocks, 256, 0, s, *a, *g); break;
        case 9: launch_after(activate_backward_kernel<9>, blocks, 256, 0, s, *a, *g); break;
        case 16: launch_after(activate_backward_kernel<16>, blocks, 256, 0, s, *a, *g); break;
        default: launch_after(activate_backward_kernel<0>, blocks, 256, 0, s, *a, *g);
    }
    return done(cudaGetLastError());
}

static bool bad_image(const float* rays, const float* target, int w, int h, int fx, int fy) {
    return !rays || !target || w <= 0 || h <= 0 || fx <= 0 || fy <= 0 || (long long)w * h * fx * fy > (1ll << 30) || h > 65535 * kTile;
}

extern "C" RGX_API size_t rgx_image_loss_scratch_floats(int w, int h) {
    const dim3 g = loss_grid(w, h);
    return w > 0 && h > 0 ? 2 * (size_t)g.x * g.y * g.z : 0;
}

extern "C" RGX_API int rgx_image_loss(int device, const float* rays, const float* target, int w, int h, int fx, int fy, float lambda_ssim,
                                      float* maps, float* scratch, float* loss, rgx_stream stream) {
    if (bad_image(rays, target, w, h, fx, fy) || !scratch || (reinterpret_cast<uintptr_t>(scratch) & 7u) || !loss) return RGX_E_INVALID;
    DeviceGuard guard(device);
    if (!guard.ok) return done(cudaErrorInvalidDevice);
    cudaStream_t s = (cudaStream_t)stream;
    const LossArgs a = loss_args(rays, target, w, h, fx, fy, lambda_ssim);
    const dim3 grid = loss_grid(w, h), block(kTile, kRows);
    float2* partial = reinterpret_cast<float2*>(scratch);
    if (lambda_ssim != 0.f) launch_after(image_loss_kernel<true>, grid, block, 0, s, a, maps, partial);
    else launch_after(image_loss_kernel<false>, grid, block, 0, s, a, nullptr, partial);
    launch_after(image_loss_sum_kernel, 1, 256, 0, s, partial, (int)(grid.x * grid.y * grid.z), 3.0 * (double)w * (double)h, lambda_ssim, loss);
    return done(cudaGetLastError());
}

extern "C" RGX_API int rgx_image_loss_backward(int device, const float* rays, const float* target, int w, int h, int fx, int fy,
                                               float lambda_ssim, const float* maps, const float* grad_loss, float* grad_rays, rgx_stream stream) {
    if (bad_image(rays, target, w, h, fx, fy) || !grad_rays || (lambda_ssim != 0.f && !maps)) return RGX_E_INVALID;
    DeviceGuard guard(device);
    if (!guard.ok) return done(cudaErrorInvalidDevice);
    cudaStream_t s = (cudaStream_t)stream;
    const LossArgs a = loss_args(rays, target, w, h, fx, fy, lambda_ssim);
    const dim3 grid = loss_grid(w, h), block(kTile, kRows);
    if (lambda_ssim != 0.f) launch_after(image_loss_backward_kernel<true>, grid, block, 0, s, a, maps, grad_loss, grad_rays);
    else launch_after(image_loss_backward_kernel<false>, grid, block, 0, s, a, nullptr, grad_loss, grad_rays);
    return done(cudaGetLastError());
}

extern "C" RGX_API int rgx_gradient_stats(int device, int n, const float* positions, const float* grad, const float* eye, float* norm_sum,
                                          float* count, float* also, rgx_stream stream) {
    if (n < 0 || (n > 0 && (!grad || !count || (norm_sum && (!positions || !eye))))) return RGX_E_INVALID;
    if (n == 0) return RGX_OK;
    DeviceGuard guard(device);
    if (!guard.ok) return done(cudaErrorInvalidDevice);
    launch_after(gradient_stats_kernel, (n + 255) / 256, 256, 0, (cudaStream_t)stream, n, positions, grad, eye, norm_sum, count, also);
    return done(cudaGetLastError());
}

extern "C" RGX_API int rgx_adam_step(int device, const rgx_adam_tensor* tensors, int count, double beta1, double beta2, double eps, rgx_stream stream) {
    if (count < 0 || count > RGX_ADAM_MAX || (count > 0 && !tensors)) return RGX_E_INVALID;
    AdamTable a{};
    a.rest1 = (float)(1.0 - beta1); a.beta2 = (float)beta2; a.rest2 = (float)(1.0 - beta2); a.eps = (float)eps;
    unsigned long long blocks = 0;
    for (int k = 0; k < count; ++k) {
        const rgx_adam_tensor& t = tensors[k];
        if (t.n < 0 || (t.n > 0 && (!t.param || !t.grad || !t.exp_avg || !t.exp_avg_sq))) return RGX_E_INVALID;
        if (t.n == 0) continue;
        a.t[a.count] = t;
        a.first[a.count++] = (unsigned)blocks;
        blocks += ((unsigned long long)t.n + kAdamChunk - 1) / kAdamChunk;
    }
    if (blocks > 0x7fffffffull) return RGX_E_TOO_LARGE;
    if (a.count == 0) return RGX_OK;
    DeviceGuard guard(device);
    if (!guard.ok) return done(cudaErrorInvalidDevice);
    launch_after(adam_kernel, (unsigned)blocks, 256, 0, (cudaStream_t)stream, a);
    return done(cudaGetLastError());
}
