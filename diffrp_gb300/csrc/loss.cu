// loss.cu -- fused mean-absolute-error loss for image fitting: one pass reads
// prediction and target, keeps the per-element gradient sign(p - t) * scale
// (as floats, or as two bits that the backward scales) and per-block partial
// sums (compensated float sums over a grid of a few blocks per SM); a second
// single-block pass adds the partials in a fixed order with compensated
// float-pair sums (reproducible loss).
#include "drp_common.cuh"
#include "drp_internal.h"

namespace drp {

constexpr int kLossThreads = 256;
constexpr int kLossBlocksPerSM = 8;

__device__ inline float l1_grad(float d, float scale) { return d > 0.0f ? scale : (d < 0.0f ? -scale : 0.0f); }

// Block sum of the threads' partial sums (block of kLossThreads).
__device__ inline void l1_block_partial(float s, float* partial) {
    __shared__ float warp_sum[kLossThreads / 32];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        float v = threadIdx.x < kLossThreads / 32 ? warp_sum[threadIdx.x] : 0.0f;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (threadIdx.x == 0) partial[blockIdx.x] = v;
    }
}

// Grid-stride pass over float4 groups (scalar head/tail when the three
// pointers are not 16-byte aligned alike); one partial per block.  The grid is
// fixed per device, so the summation order -- and the loss -- is reproducible.
__global__ void __launch_bounds__(kLossThreads) l1_partial_kernel(const float* p, const float* t, long long n,
                                                                  float scale, float* grad, float* partial) {
    const long long stride = (long long)gridDim.x * kLossThreads;
    const long long tid = (long long)blockIdx.x * kLossThreads + threadIdx.x;
    float s = 0.0f, c = 0.0f;
    const bool vec = ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(t) |
                       reinterpret_cast<uintptr_t>(grad)) & 15) == 0;
    long long done = 0;
    if (vec) {
        const long long n4 = n >> 2;
        const float4* p4 = reinterpret_cast<const float4*>(p);
        const float4* t4 = reinterpret_cast<const float4*>(t);
        float4* g4 = reinterpret_cast<float4*>(grad);
        for (long long i = tid; i < n4; i += stride) {
            const float4 a = p4[i], b = t4[i];
            const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z, dw = a.w - b.w;
            kahan_add(s, c, (fabsf(dx) + fabsf(dy)) + (fabsf(dz) + fabsf(dw)));
            g4[i] = make_float4(l1_grad(dx, scale), l1_grad(dy, scale), l1_grad(dz, scale), l1_grad(dw, scale));
        }
        done = n4 << 2;
    }
    for (long long i = done + tid; i < n; i += stride) {
        const float d = p[i] - t[i];
        kahan_add(s, c, fabsf(d));
        grad[i] = l1_grad(d, scale);
    }
    l1_block_partial(s, partial);
}

// l1_partial_kernel for 16-byte aligned p and t that keeps the signs instead of
// writing the gradient: byte i has bit k set where element 4 i + k is above its
// target and bit 4 + k where it is below.  The sums are formed in the same
// order.  What bounds it: reading p and t; with the gradient written here (a
// third array, read again by its scaling) the loss of 4.8M pixels x 8 channels
// and its backward took 75 + 97 us, this way 59 + 28.
__global__ void __launch_bounds__(kLossThreads) l1_sign_kernel(const float* p, const float* t, long long n,
                                                               unsigned char* signs, float* partial) {
    const long long stride = (long long)gridDim.x * kLossThreads;
    const long long tid = (long long)blockIdx.x * kLossThreads + threadIdx.x;
    float s = 0.0f, c = 0.0f;
    const long long n4 = n >> 2;
    const float4* p4 = reinterpret_cast<const float4*>(p);
    const float4* t4 = reinterpret_cast<const float4*>(t);
    const auto code = [](float d, int k) { return d > 0.0f ? 1u << k : (d < 0.0f ? 16u << k : 0u); };
#pragma unroll 4
    for (long long i = tid; i < n4; i += stride) {
        const float4 a = p4[i], b = t4[i];
        const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z, dw = a.w - b.w;
        kahan_add(s, c, (fabsf(dx) + fabsf(dy)) + (fabsf(dz) + fabsf(dw)));
        signs[i] = (unsigned char)(code(dx, 0) | code(dy, 1) | code(dz, 2) | code(dw, 3));
    }
    for (long long i = 4 * n4 + tid; i < n; i += stride) kahan_add(s, c, fabsf(p[i] - t[i]));
    if (tid == 0 && (n & 3)) {
        unsigned m = 0u;
        for (int k = 0; k < (int)(n & 3); ++k) m |= code(p[4 * n4 + k] - t[4 * n4 + k], k);
        signs[n4] = (unsigned char)m;
    }
    l1_block_partial(s, partial);
}

// grad[i] = (sign * scale) * upstream[0] from l1_sign_kernel's bytes; grad
// 16-byte aligned.  Bound by the writes.
__global__ void __launch_bounds__(kLossThreads) l1_grad_kernel(const unsigned char* signs, long long n, float scale,
                                                               const float* upstream, float* grad) {
    const long long stride = (long long)gridDim.x * kLossThreads;
    const long long tid = (long long)blockIdx.x * kLossThreads + threadIdx.x;
    const float g = *upstream;
    const float up = scale * g, down = -scale * g, tie = 0.0f * g;  // (a tie's gradient follows inf and nan too)
    const auto value = [&](unsigned m, int k) { return (m >> k) & 1u ? up : ((m >> (k + 4)) & 1u ? down : tie); };
    const long long n4 = n >> 2;
    float4* g4 = reinterpret_cast<float4*>(grad);
#pragma unroll 4
    for (long long i = tid; i < n4; i += stride) {
        const unsigned m = signs[i];
        g4[i] = make_float4(value(m, 0), value(m, 1), value(m, 2), value(m, 3));
    }
    if (tid < (n & 3)) grad[4 * n4 + tid] = value(signs[n4], (int)tid);
}

// Fixed-order compensated sum of the partials (l1_final_block,
// drp_common.cuh) in one block.
__global__ void __launch_bounds__(kFinalThreads) l1_final_kernel(const float* partial, long long nblocks, float scale,
                                                                 float* loss) {
    pdl_wait();
    pdl_launch_dependents();
    l1_final_block<kFinalThreads>(partial, nblocks, scale, loss);
}

void launch_l1_final(const float* partial, long long nblocks, float scale, float* loss, cudaStream_t s) {
    launch_pdl(l1_final_kernel, dim3(1), dim3(kFinalThreads), s, partial, nblocks, scale, loss);
    drp_note_launch();
}

// dst = src * scale[0]: 16-byte groups from the first aligned float, scalar
// head and tail (grid-stride).
__global__ void __launch_bounds__(256) scale_floats_kernel(float* dst, const float* src, long long n,
                                                           const float* scale) {
    pdl_wait();
    pdl_launch_dependents();
    const float k = *scale;
    const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const bool same_phase = ((reinterpret_cast<uintptr_t>(dst) ^ reinterpret_cast<uintptr_t>(src)) & 15) == 0;
    long long h = same_phase ? (long long)(((16 - (reinterpret_cast<uintptr_t>(dst) & 15)) & 15) >> 2) : n;
    if (h > n) h = n;
    for (long long i = i0; i < h; i += stride) dst[i] = src[i] * k;
    const long long n4 = (n - h) >> 2;
    float4* d4 = reinterpret_cast<float4*>(dst + h);
    const float4* s4 = reinterpret_cast<const float4*>(src + h);
    for (long long i = i0; i < n4; i += stride) {
        const float4 v = s4[i];
        d4[i] = make_float4(v.x * k, v.y * k, v.z * k, v.w * k);
    }
    const long long t0 = h + 4 * n4;
    if (i0 < n - t0) dst[t0 + i0] = src[t0 + i0] * k;
}

// Blocks for n elements: enough to fill every SM, never more than one
// float4 group per thread.
static long long l1_blocks(long long n) {
    const int sms = drp_current_sm_count();
    if (sms <= 0) return 1;  // no device: callers fail at launch
    const long long max_blocks = (long long)sms * kLossBlocksPerSM;
    const long long need = ((n + 3) / 4 + kLossThreads - 1) / kLossThreads;
    return need < max_blocks ? (need > 0 ? need : 1) : max_blocks;
}

}  // namespace drp

extern "C" __attribute__((visibility("default"))) int drp_l1_loss_workspace_size(long long n, size_t* bytes) {
    if (!bytes || n < 0) {
        drp_set_last_error("drp_l1_loss_workspace_size: bad arguments");
        return 1;
    }
    // the most blocks any device uses: one float4 group per thread (the grid
    // is capped below that by the SM count), so the size is device-independent
    const long long most = ((n + 3) / 4 + drp::kLossThreads - 1) / drp::kLossThreads;
    *bytes = (size_t)(most > 0 ? most : 1) * sizeof(float) + 256;
    return 0;
}

extern "C" __attribute__((visibility("default"))) int drp_l1_loss_fwd(void* workspace, size_t workspace_bytes,
                                                                      const float* pred, const float* target,
                                                                      long long n, float scale, float* loss,
                                                                      float* grad, void* stream) {
    const long long nblocks = drp::l1_blocks(n);
    if (n <= 0 || !pred || !target || !loss || !grad || !workspace ||
        workspace_bytes < (size_t)nblocks * sizeof(float) || nblocks > 0x7fffffffll) {
        drp_set_last_error("drp_l1_loss_fwd: bad arguments or workspace too small");
        return 1;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float* partial = static_cast<float*>(workspace);
    drp::l1_partial_kernel<<<(unsigned)nblocks, drp::kLossThreads, 0, s>>>(pred, target, n, scale, grad, partial);
    drp_note_launch();
    drp::launch_l1_final(partial, nblocks, scale, loss, s);
    return drp_check_launch("drp_l1_loss_fwd");
}

extern "C" __attribute__((visibility("default"))) int drp_l1_loss_sign_fwd(void* workspace, size_t workspace_bytes,
                                                                           const float* pred, const float* target,
                                                                           long long n, float scale, float* loss,
                                                                           void* signs, void* stream) {
    const long long nblocks = drp::l1_blocks(n);
    if (n <= 0 || !pred || !target || !loss || !signs || !workspace ||
        ((reinterpret_cast<uintptr_t>(pred) | reinterpret_cast<uintptr_t>(target)) & 15) ||
        workspace_bytes < (size_t)nblocks * sizeof(float) || nblocks > 0x7fffffffll) {
        drp_set_last_error("drp_l1_loss_sign_fwd: bad arguments or workspace too small");
        return 1;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float* partial = static_cast<float*>(workspace);
    drp::l1_sign_kernel<<<(unsigned)nblocks, drp::kLossThreads, 0, s>>>(pred, target, n,
                                                                       static_cast<unsigned char*>(signs), partial);
    drp_note_launch();
    drp::launch_l1_final(partial, nblocks, scale, loss, s);
    return drp_check_launch("drp_l1_loss_sign_fwd");
}

extern "C" __attribute__((visibility("default"))) int drp_l1_loss_bwd(const void* signs, long long n, float scale,
                                                                      const float* upstream, float* grad,
                                                                      void* stream) {
    if (n <= 0 || !signs || !upstream || !grad || (reinterpret_cast<uintptr_t>(grad) & 15)) {
        drp_set_last_error("drp_l1_loss_bwd: bad arguments");
        return 1;
    }
    drp::l1_grad_kernel<<<(unsigned)drp::l1_blocks(n), drp::kLossThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const unsigned char*>(signs), n, scale, upstream, grad);
    drp_note_launch();
    return drp_check_launch("drp_l1_loss_bwd");
}

extern "C" __attribute__((visibility("default"))) int drp_scale_floats(float* dst, const float* src, long long n,
                                                                      const float* scale, void* stream) {
    if (n < 0 || (n > 0 && (!dst || !src || !scale)) || ((reinterpret_cast<uintptr_t>(dst) |
                                                        reinterpret_cast<uintptr_t>(src)) & 3)) {
        drp_set_last_error("drp_scale_floats: bad arguments");
        return 1;
    }
    if (n == 0) return 0;
    const int sms = drp_current_sm_count();
    long long blocks = (n / 4 + 255) / 256;
    const long long cap = (long long)(sms > 0 ? sms : 1) * 8;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    drp::launch_pdl(drp::scale_floats_kernel, dim3((unsigned)blocks), dim3(256), static_cast<cudaStream_t>(stream),
                    dst, src, n, scale);
    drp_note_launch();
    return drp_check_launch("drp_scale_floats");
}
