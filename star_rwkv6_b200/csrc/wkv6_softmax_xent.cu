// Next-token loss of the language-model head in one pass over the logits: for every row (token) the softmax
// cross-entropy against its target id and, in the same kernel, the gradient with respect to the logits, written over
// the logits themselves:   loss[row] = logsumexp(z) - z[target];   z <- (softmax(z) - onehot(target)) * scale.
// bf16 logits [rows, V], fp32 arithmetic.  A training step of the 1.6B-shape model has 32768 x 65536 logits (4.3 GB in
// bf16): the framework path copies them to fp32, writes fp32 log-probabilities, reads them back in the backward and
// converts the gradient to bf16 again (about 65 GB of traffic, 20 ms); this kernel reads a row once and writes the gradient
// once (8.6 GB).
// The reference has no trainer (its trainer files are empty); this belongs to the training step built around the op.
#include <cuda_bf16.h>

#include <cstdint>

#include "wkv6_internal.h"

namespace wkv6 {

__device__ __forceinline__ float exp2f_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// exp(z - mx) of two logits.  The difference is formed before it is scaled: it is exact for logits near the maximum, where one
// fused multiply-add z log2(e) - mx log2(e) is off by the rounding of its second term (3e-4 of the result at mx = 1e4), and no
// term overflows for logits at the end of the type's range.  The packed instructions do both steps at the cost of that one.
__device__ __forceinline__ float2 exp_pair(float2 z, float2 neg_mx) {
    constexpr float kLog2e = 1.4426950408889634f;
    unsigned long long d, m, c;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(z.x), "f"(z.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(m) : "f"(neg_mx.x), "f"(neg_mx.y));
    asm("mov.b64 %0, {%1, %1};" : "=l"(c) : "f"(kLog2e));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(m));
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(c));
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(d));
    return make_float2(exp2f_fast(r.x), exp2f_fast(r.y));
}

constexpr int kXentThreads = 512;
constexpr int kXentMaxVecs = 16;  // 16-byte vectors per thread: V <= 512 * 16 * 8 = 65536

__device__ __forceinline__ float xent_block_reduce(float x, bool is_max, float *scratch) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float y = __shfl_xor_sync(0xffffffffu, x, o);
        x = is_max ? fmaxf(x, y) : x + y;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) scratch[warp] = x;
    __syncthreads();
    float t = scratch[0];
#pragma unroll
    for (int i = 1; i < kXentThreads / 32; ++i) t = is_max ? fmaxf(t, scratch[i]) : t + scratch[i];
    return t;
}

__device__ __forceinline__ void xent_copy16(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}

// What bounds it: 4 B of traffic per logit against two exponentials and about twenty other instructions per logit, which
// take about as long (at V = 65536 the special-function pipe alone needs 0.7 of the time the bytes need).  One CTA per row
// ran the three one after the other - load, compute, store: a row fills the registers of an SM, so no second row was in
// flight (4096 x 65536: 325 us, 3.3 TB/s).  Now a CTA walks rows, and while it computes on one (in registers) the next one
// travels into shared memory.  A thread reads back only the vectors it copied itself, so the hand-over needs no barrier.
template <int VECS>
__global__ void __launch_bounds__(kXentThreads, VECS == 16 ? 1 : VECS == 4 ? 2 : 3)
softmax_xent_kernel(int64_t rows, int V, __nv_bfloat16 *__restrict__ logits, const int64_t *__restrict__ targets, float scale,
                    float *__restrict__ loss) {
    extern __shared__ uint4 next_row[];  // [VECS][kXentThreads]
    __shared__ float scratch[kXentThreads / 32];
    const int nvec = V >> 3, tid = threadIdx.x;
    auto request = [&](int64_t row) {
        if (row < rows) {
            const uint4 *zrow = reinterpret_cast<const uint4 *>(logits + row * (int64_t)V);
#pragma unroll
            for (int j = 0; j < VECS; ++j) {
                const int i = tid + j * kXentThreads;
                if (i < nvec) xent_copy16(next_row + j * kXentThreads + tid, zrow + i);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    request(blockIdx.x);
    for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
        uint4 *zrow = reinterpret_cast<uint4 *>(logits + row * (int64_t)V);
        const int64_t tgt = targets[row];
        const bool ignore = tgt < 0 || tgt >= V;  // such rows contribute neither loss nor gradient
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        uint4 z[VECS];
#pragma unroll
        for (int j = 0; j < VECS; ++j)
            if (tid + j * kXentThreads < nvec) z[j] = next_row[j * kXentThreads + tid];
        request(row + gridDim.x);
        // read before the barriers below, behind which the row is overwritten
        float target_logit = 0.f;
        if (tid == 0) target_logit = ignore ? 0.f : __bfloat162float(logits[row * (int64_t)V + tgt]);
        float mx = -3.0e38f;
#pragma unroll
        for (int j = 0; j < VECS; ++j) {
            if (tid + j * kXentThreads < nvec) {
                const __nv_bfloat162 *p = reinterpret_cast<const __nv_bfloat162 *>(&z[j]);
                __nv_bfloat162 m = __hmax2(__hmax2(p[0], p[1]), __hmax2(p[2], p[3]));   // exact: a maximum of bf16 values
                const float2 f = __bfloat1622float2(m);
                mx = fmaxf(mx, fmaxf(f.x, f.y));
            }
        }
        mx = xent_block_reduce(mx, true, scratch);
        const float2 neg_mx = make_float2(-mx, -mx);
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < VECS; ++j) {
            if (tid + j * kXentThreads < nvec) {
                const __nv_bfloat162 *p = reinterpret_cast<const __nv_bfloat162 *>(&z[j]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 x = exp_pair(__bfloat1622float2(p[e]), neg_mx);
                    sum += x.x + x.y;
                }
            }
        }
        sum = xent_block_reduce(sum, false, scratch);
        if (tid == 0) loss[row] = ignore ? 0.f : (mx + logf(sum)) - target_logit;
        const float sc = ignore ? 0.f : scale, inv = 1.f / sum;
        const int tvec = ignore ? -1 : (int)(tgt >> 3), telem = (int)(tgt & 7);
#pragma unroll
        for (int j = 0; j < VECS; ++j) {
            const int i = tid + j * kXentThreads;
            if (i < nvec) {
                __nv_bfloat162 *p = reinterpret_cast<__nv_bfloat162 *>(&z[j]);
                float g[8];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 x = exp_pair(__bfloat1622float2(p[e]), neg_mx);
                    g[2 * e] = x.x * inv;
                    g[2 * e + 1] = x.y * inv;
                }
                if (i == tvec) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) g[e] -= e == telem ? 1.f : 0.f;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) p[e] = __floats2bfloat162_rn(g[2 * e] * sc, g[2 * e + 1] * sc);
                zrow[i] = z[j];
            }
        }
    }
}

template <int VECS>
static int xent_launch(int64_t rows, int V, __nv_bfloat16 *z, const int64_t *targets, float scale, float *loss, cudaStream_t st) {
    constexpr int smem = VECS * kXentThreads * 16, per_sm = VECS == 16 ? 1 : VECS == 4 ? 2 : 3;
    cudaError_t e = cudaFuncSetAttribute(softmax_xent_kernel<VECS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(softmax_xent_kernel)");
    const int64_t most = (int64_t)sm_count() * per_sm;
    softmax_xent_kernel<VECS><<<(unsigned)(rows < most ? rows : most), kXentThreads, smem, st>>>(rows, V, z, targets, scale, loss);
    e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "softmax_xent_kernel launch");
}

// g <- g * (*scale): the chain rule of the loss, whose gradient the forward has already left in g.  A loss that is itself the
// end of the graph arrives with a gradient of exactly 1, for which nothing has to be touched.
__global__ void __launch_bounds__(256) scale_rows_kernel(size_t nvec, __nv_bfloat16 *__restrict__ g, const float *__restrict__ scale) {
    const float s = __bfloat162float(__float2bfloat16_rn(*scale));   // the factor in the gradient's own dtype
    if (s == 1.f) return;
    uint4 *v = reinterpret_cast<uint4 *>(g);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += (size_t)gridDim.x * blockDim.x) {
        uint4 q = v[i];
        __nv_bfloat162 *p = reinterpret_cast<__nv_bfloat162 *>(&q);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(p[e]);
            p[e] = __floats2bfloat162_rn(f.x * s, f.y * s);
        }
        v[i] = q;
    }
}

}  // namespace wkv6

using namespace wkv6;

extern "C" int wkv6_softmax_xent_bf16(int64_t rows, int32_t V, void *logits_inout, const int64_t *targets, float scale,
                                      float *loss, void *stream) {
    if (rows < 0 || V < 8 || V % 8 || V > kXentThreads * kXentMaxVecs * 8)
        return fail(WKV6_ERR_UNSUPPORTED, "wkv6_softmax_xent_bf16: rows=%lld V=%d (V a multiple of 8, at most %d)", (long long)rows, V,
                    kXentThreads * kXentMaxVecs * 8);
    if (rows == 0) return WKV6_OK;
    if (rows > 2147483647LL) return fail(WKV6_ERR_UNSUPPORTED, "wkv6_softmax_xent_bf16: too many rows");
    if (!logits_inout || !targets || !loss) return fail(WKV6_ERR_INVALID, "wkv6_softmax_xent_bf16: NULL argument");
    if (reinterpret_cast<uintptr_t>(logits_inout) % 16) return fail(WKV6_ERR_INVALID, "wkv6_softmax_xent_bf16: logits must be 16-byte aligned");
    __nv_bfloat16 *z = static_cast<__nv_bfloat16 *>(logits_inout);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (V <= kXentThreads * 8) return xent_launch<1>(rows, V, z, targets, scale, loss, st);
    if (V <= kXentThreads * 32) return xent_launch<4>(rows, V, z, targets, scale, loss, st);
    return xent_launch<16>(rows, V, z, targets, scale, loss, st);
}

extern "C" int wkv6_scale_bf16(int64_t n, void *g, const float *scale, void *stream) {
    if (n < 0 || n % 8) return fail(WKV6_ERR_INVALID, "wkv6_scale_bf16: n=%lld is not a multiple of 8", (long long)n);
    if (n == 0) return WKV6_OK;
    if (!g || !scale || reinterpret_cast<uintptr_t>(g) % 16) return fail(WKV6_ERR_INVALID, "wkv6_scale_bf16: NULL or misaligned argument");
    const int64_t blocks = (n / 8 + 255) / 256, most = 8LL * sm_count();
    scale_rows_kernel<<<(unsigned)(blocks < most ? blocks : most), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        (size_t)(n / 8), static_cast<__nv_bfloat16 *>(g), scale);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "scale_rows_kernel launch");
}
