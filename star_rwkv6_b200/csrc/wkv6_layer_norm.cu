// LayerNorm over the channels of every token, with the residual addition in front of it:
//   s = x + o  (optional),   y = (s - mean) rstd gamma + beta,
// and its backward, gx = gs + LN'(gy) (gs: the gradient that reaches s past the norm, optional), gamma and beta gradients
// (the two norms of a block, rwkv6_model.py:197-215, with x + TimeMix(LN(x)) in front of the second).
//
// Both directions are bound by HBM: a thread owns eight channels of many rows, so that a row is read once, the parameters and
// (backward) their gradients stay in registers, and the block reductions of one group of rows run under the loads of the next.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "wkv6_internal.h"

namespace wkv6 {

constexpr int kLnMaxD = 8192;

__device__ __forceinline__ float warp_total(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

__device__ __forceinline__ void un8(const uint4 &v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

__device__ __forceinline__ uint4 pk8(const float (&f)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t *>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ uint4 ld16(const __nv_bfloat16 *p) { return *reinterpret_cast<const uint4 *>(p); }

__host__ __device__ constexpr int ln_blocks(int threads) { return threads == 256 ? 4 : threads == 512 ? 2 : 1; }   // per SM, forward

// Block of D / 8 threads (rounded up to warps, at most THREADS), eight channels a thread, over groups of ROWS rows blockIdx.x +
// gridDim.x n; the next group's rows are requested before this one is reduced.  (A warp per row, the whole row in its registers,
// took 25 us at 4004 x 4096 and 11.7 us at 16 x 4096, the latter a chain of 16 loads' worth of arithmetic in one warp.)
template <int THREADS, int ROWS>
__global__ void __launch_bounds__(THREADS, ln_blocks(THREADS)) ln_fwd_kernel(long long rows, int D, float eps, const __nv_bfloat16 *__restrict__ x,
                                                                             const __nv_bfloat16 *__restrict__ o,
                                                                             const __nv_bfloat16 *__restrict__ gamma,
                                                                             const __nv_bfloat16 *__restrict__ beta,
                                                                             __nv_bfloat16 *__restrict__ s_out, __nv_bfloat16 *__restrict__ y,
                                                                             float *__restrict__ stat) {
    __shared__ float red[2][ROWS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, c = threadIdx.x * 8;
    const bool act = c < D;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 xv[ROWS], ov[ROWS];
    auto fetch = [&](long long r0) {
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const bool ok = act && r0 + i < rows;
            xv[i] = ok ? ld16(x + (size_t)(r0 + i) * D + c) : zero;
            ov[i] = ok && o != nullptr ? ld16(o + (size_t)(r0 + i) * D + c) : zero;
        }
    };
    const long long step = (long long)gridDim.x * ROWS;
    long long r0 = (long long)blockIdx.x * ROWS;
    fetch(r0);
    const uint4 gv = act ? ld16(gamma + c) : zero, bv = act ? ld16(beta + c) : zero;
    for (; r0 < rows; r0 += step) {
        float v[ROWS][8], sum[ROWS];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            un8(xv[i], v[i]);
            if (o != nullptr) {
                float b[8];
                un8(ov[i], b);
#pragma unroll
                for (int e = 0; e < 8; ++e) v[i][e] += b[e];
                const uint4 r = pk8(v[i]);               // the sum as it is stored, rounded
                un8(r, v[i]);
                if (act && r0 + i < rows) *reinterpret_cast<uint4 *>(s_out + (size_t)(r0 + i) * D + c) = r;
            }
            sum[i] = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) sum[i] += v[i][e];
        }
        if (r0 + step < rows) fetch(r0 + step);
        float mean[ROWS];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            sum[i] = warp_total(sum[i]);
            if (lane == 0) red[0][i][warp] = sum[i];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            mean[i] = warp_total(lane < warps ? red[0][i][lane] : 0.f) / D;
            float q = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) q = fmaf(v[i][e] - mean[i], v[i][e] - mean[i], q);
            q = warp_total(act ? q : 0.f);
            if (lane == 0) red[1][i][warp] = q;
        }
        __syncthreads();     // also keeps red[0] until everyone has read it
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const float rstd = rsqrtf(warp_total(lane < warps ? red[1][i][lane] : 0.f) / D + eps);
            if (r0 + i < rows) {
                if (stat != nullptr && threadIdx.x == 0) *reinterpret_cast<float2 *>(stat + 2 * (r0 + i)) = make_float2(mean[i], rstd);
                if (act) {
                    float g[8], b[8];
                    un8(gv, g); un8(bv, b);
#pragma unroll
                    for (int e = 0; e < 8; ++e) g[e] = fmaf((v[i][e] - mean[i]) * rstd, g[e], b[e]);
                    *reinterpret_cast<uint4 *>(y + (size_t)(r0 + i) * D + c) = pk8(g);
                }
            }
        }
    }
}

// The same shape; partial [grid][2][D]: sums of gy xhat and of gy over the block's rows.
__host__ __device__ constexpr int ln_rows(int threads) { return threads > 512 ? 1 : 2; }   // rows in flight (and as many requested)
template <int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 2 : 1) ln_bwd_kernel(long long rows, int D, const __nv_bfloat16 *__restrict__ s,
                                                                             const float *__restrict__ stat, const __nv_bfloat16 *__restrict__ gamma,
                                                                             const __nv_bfloat16 *__restrict__ gy,
                                                                             const __nv_bfloat16 *__restrict__ gs, __nv_bfloat16 *__restrict__ gx,
                                                                             float *__restrict__ partial) {
    constexpr int ROWS = ln_rows(THREADS);
    __shared__ float red[2][2 * ROWS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, c = threadIdx.x * 8;
    const bool act = c < D;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    float dg[8] = {}, db[8] = {};
    uint4 xn[ROWS], gn[ROWS], rn[ROWS];
    float2 sn[ROWS];
    auto fetch = [&](long long r0) {
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const bool ok = act && r0 + i < rows;
            const size_t p = (size_t)(r0 + i) * D + c;
            xn[i] = ok ? ld16(s + p) : zero;
            gn[i] = ok ? ld16(gy + p) : zero;
            rn[i] = ok && gs != nullptr ? ld16(gs + p) : zero;
            sn[i] = r0 + i < rows ? *reinterpret_cast<const float2 *>(stat + 2 * (r0 + i)) : make_float2(0.f, 0.f);
        }
    };
    const long long step = (long long)gridDim.x * ROWS;
    long long r0 = (long long)blockIdx.x * ROWS;
    fetch(r0);
    const uint4 gmv = act ? ld16(gamma + c) : zero;
    int buf = 0;
    for (; r0 < rows; r0 += step) {
        uint4 xv[ROWS], gv[ROWS], rv[ROWS];
        float2 st[ROWS];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) { xv[i] = xn[i]; gv[i] = gn[i]; rv[i] = rn[i]; st[i] = sn[i]; }
        if (r0 + step < rows) fetch(r0 + step);
        float sum[2 * ROWS], gm[8];
        un8(gmv, gm);
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            float xf[8], g[8], s1 = 0.f, s2 = 0.f;
            un8(xv[i], xf); un8(gv[i], g);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float xh = act ? (xf[e] - st[i].x) * st[i].y : 0.f;
                const float gg = g[e] * gm[e];
                s1 += gg;
                s2 = fmaf(gg, xh, s2);
                dg[e] = fmaf(g[e], xh, dg[e]);
                db[e] += g[e];
            }
            sum[2 * i] = s1; sum[2 * i + 1] = s2;
        }
#pragma unroll
        for (int k = 0; k < 2 * ROWS; ++k) {
            sum[k] = warp_total(sum[k]);
            if (lane == 0) red[buf][k][warp] = sum[k];
        }
        __syncthreads();      // the other buffer's readers are past it by the next one
#pragma unroll
        for (int k = 0; k < 2 * ROWS; ++k) sum[k] = warp_total(lane < warps ? red[buf][k][lane] : 0.f) / D;
        buf ^= 1;
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
            if (act && r0 + i < rows) {
                float xf[8], g[8], a[8];
                un8(xv[i], xf); un8(gv[i], g); un8(rv[i], a);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float xh = (xf[e] - st[i].x) * st[i].y;
                    a[e] += st[i].y * (fmaf(g[e], gm[e], -sum[2 * i]) - xh * sum[2 * i + 1]);
                }
                *reinterpret_cast<uint4 *>(gx + (size_t)(r0 + i) * D + c) = pk8(a);
            }
    }
    if (act) {
        float *p = partial + (size_t)blockIdx.x * 2 * D + c;
        *reinterpret_cast<float4 *>(p) = make_float4(dg[0], dg[1], dg[2], dg[3]);
        *reinterpret_cast<float4 *>(p + 4) = make_float4(dg[4], dg[5], dg[6], dg[7]);
        *reinterpret_cast<float4 *>(p + D) = make_float4(db[0], db[1], db[2], db[3]);
        *reinterpret_cast<float4 *>(p + D + 4) = make_float4(db[4], db[5], db[6], db[7]);
    }
}

// column sums of partial [parts][2 D] in a fixed order, rounded to bf16: 32 columns x 8 groups of parts per block
__global__ void __launch_bounds__(256) ln_param_kernel(int parts, int D, const float *__restrict__ partial, __nv_bfloat16 *__restrict__ ggamma,
                                                       __nv_bfloat16 *__restrict__ gbeta) {
    __shared__ float red[8][33];
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
    float t = 0.f;
    if (c < 2 * D) {
#pragma unroll 8
        for (int p = grp; p < parts; p += 8) t += partial[(size_t)p * 2 * D + c];
    }
    red[grp][lane] = t;
    __syncthreads();
    if (grp == 0 && c < 2 * D) {
#pragma unroll
        for (int k = 1; k < 8; ++k) t += red[k][lane];
        if (c < D) ggamma[c] = __float2bfloat16_rn(t); else gbeta[c - D] = __float2bfloat16_rn(t);
    }
}

static int ln_threads(int D) { return D <= 2048 ? 256 : D <= 4096 ? 512 : 1024; }

// 512 threads per SM (1024 for the widest rows): what the registers allow; no more blocks than groups of rows
static int ln_grid(long long rows, int D) {
    const int t = ln_threads(D), rows_each = ln_rows(t);
    const long long want = (long long)sm_count() * (t == 256 ? 2 : 1), most = (rows + rows_each - 1) / rows_each;
    return (int)(want < most ? want : most);
}

static int ln_check(long long rows, int D, const char *what) {
    if (rows < 0 || D < 8 || D % 8 || D > kLnMaxD) return fail(WKV6_ERR_UNSUPPORTED, "%s: rows=%lld D=%d (D a multiple of 8, at most %d)", what, rows, D, kLnMaxD);
    return WKV6_OK;
}

}  // namespace wkv6

using namespace wkv6;

#define LN_PTR(p) \
    if ((p) == nullptr || reinterpret_cast<uintptr_t>(p) % 16) return fail(WKV6_ERR_INVALID, #p " is NULL or not 16-byte aligned")

extern "C" {

__attribute__((visibility("default")))
int wkv6_layer_norm_forward(int64_t rows, int32_t D, float eps, const void *x, const void *o, const void *gamma, const void *beta,
                            void *s_out, void *y, float *stat, void *stream) {
    if (int rc = ln_check(rows, D, "wkv6_layer_norm_forward")) return rc;
    if (rows == 0) return WKV6_OK;
    LN_PTR(x); LN_PTR(gamma); LN_PTR(beta); LN_PTR(y);
    if (o != nullptr) { LN_PTR(o); LN_PTR(s_out); }
    if (stat != nullptr) LN_PTR(stat);
    using bf = __nv_bfloat16;
    const int threads = ln_threads(D), block = (D / 8 + 31) / 32 * 32;
    const long long most = (long long)sm_count() * ln_blocks(threads);     // blocks at a time
    cudaStream_t st = static_cast<cudaStream_t>(stream);
#define LN_FWD(THREADS, ROWS)                                                                                                          \
    ln_fwd_kernel<THREADS, ROWS><<<(unsigned)((rows + ROWS - 1) / ROWS < most ? (rows + ROWS - 1) / ROWS : most), block, 0, st>>>(        \
        rows, D, eps, static_cast<const bf *>(x), static_cast<const bf *>(o), static_cast<const bf *>(gamma), static_cast<const bf *>(beta), \
        static_cast<bf *>(s_out), static_cast<bf *>(y), stat)
    if (threads == 1024) LN_FWD(1024, 1);
    else if (rows <= most) { if (threads == 256) LN_FWD(256, 1); else LN_FWD(512, 1); }      // one row per block: the shortest chain
    else if (threads == 256) LN_FWD(256, 2);
    else LN_FWD(512, 2);
#undef LN_FWD
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "ln_fwd_kernel launch");
}

__attribute__((visibility("default")))
size_t wkv6_layer_norm_workspace_bytes(int64_t rows, int32_t D) {
    return rows <= 0 || D <= 0 ? 0 : (size_t)ln_grid(rows, D) * 2 * D * sizeof(float);
}

__attribute__((visibility("default")))
int wkv6_layer_norm_backward(int64_t rows, int32_t D, const void *s, const float *stat, const void *gamma, const void *gy, const void *gs,
                             void *gx, void *ggamma, void *gbeta, void *workspace, size_t workspace_bytes, void *stream) {
    if (int rc = ln_check(rows, D, "wkv6_layer_norm_backward")) return rc;
    LN_PTR(ggamma); LN_PTR(gbeta);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int parts = 0;
    if (rows > 0) {
        LN_PTR(s); LN_PTR(stat); LN_PTR(gamma); LN_PTR(gy); LN_PTR(gx); LN_PTR(workspace);
        if (gs != nullptr) LN_PTR(gs);
        const size_t need = wkv6_layer_norm_workspace_bytes(rows, D);
        if (workspace_bytes < need) return fail(WKV6_ERR_WORKSPACE, "layer norm backward workspace: need %zu bytes, got %zu", need, workspace_bytes);
        using bf = __nv_bfloat16;
        parts = ln_grid(rows, D);
        const int threads = ln_threads(D), block = (D / 8 + 31) / 32 * 32;
        auto kernel = threads == 256 ? ln_bwd_kernel<256> : threads == 512 ? ln_bwd_kernel<512> : ln_bwd_kernel<1024>;
        kernel<<<parts, block, 0, st>>>(rows, D, static_cast<const bf *>(s), stat, static_cast<const bf *>(gamma), static_cast<const bf *>(gy),
                                        static_cast<const bf *>(gs), static_cast<bf *>(gx), static_cast<float *>(workspace));
    }
    ln_param_kernel<<<(2 * D + 31) / 32, 256, 0, st>>>(parts, D, static_cast<const float *>(workspace), static_cast<__nv_bfloat16 *>(ggamma),
                                                     static_cast<__nv_bfloat16 *>(gbeta));
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "layer norm backward launch");
}

}  // extern "C"
