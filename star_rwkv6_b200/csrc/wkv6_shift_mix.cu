// Input stage of the time-mix block: the token-shift interpolations
//   out_j[b,t,c] = x[b,t,c] + (x[b,t-1,c] - x[b,t,c]) * m_j[b,t,c],      x[b,-1,:] = 0,
// for j = 0..nmix-1, where m_j is either one vector per channel (time_mix_x: TimeMix.call, rwkv6_model.py:135-138,
// with TimeShift = pad-and-subtract, :37-44) or a full tensor (the five data-dependent mixes built from the low-rank
// projections, rwkv6_model.py:141-146).  The reference runs them as separate framework ops (a padded copy, a
// subtraction, and per mix a multiply and an add); here one kernel per direction reads x once and every m_j once.
//
// A thread owns eight adjacent channels and walks a run of consecutive tokens of one batch row, carrying the
// neighbouring token in registers: the forward walks up (carrying x[t-1]), the backward walks down (carrying
// gs[t+1] = sum_j gout_j[t+1] m_j[t+1], the gradient that reaches x[t] through the shift).  Bytes per (token,
// channel) in bf16: vector mix 4 forward / 6 backward; five tensor mixes 22 forward / 34 backward.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "wkv6_internal.h"

namespace wkv6 {

constexpr int kRun = 32;  // tokens a thread walks; the carried neighbour is re-read once per run

template <typename T> struct V8;
template <> struct V8<__nv_bfloat16> {
    using Raw = uint4;
    static __device__ __forceinline__ void get(const void *p, size_t i, Raw &q) {
        q = *reinterpret_cast<const uint4 *>(static_cast<const __nv_bfloat16 *>(p) + i);
    }
    static __device__ __forceinline__ void ld(const void *p, size_t i, float (&f)[8]) {
        Raw q;
        get(p, i, q);
        unpack(q, f);
    }
    static __device__ __forceinline__ void unpack(const Raw &q, float (&f)[8]) {
        const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&q);
#pragma unroll
        for (int e = 0; e < 4; ++e) { const float2 t = __bfloat1622float2(h[e]); f[2 * e] = t.x; f[2 * e + 1] = t.y; }
    }
    static __device__ __forceinline__ void st(void *p, size_t i, const float (&f)[8]) {
        uint4 q;
        __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&q);
#pragma unroll
        for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
        *reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(p) + i) = q;
    }
};
template <> struct V8<__half> {
    using Raw = uint4;
    static __device__ __forceinline__ void get(const void *p, size_t i, Raw &q) {
        q = *reinterpret_cast<const uint4 *>(static_cast<const __half *>(p) + i);
    }
    static __device__ __forceinline__ void ld(const void *p, size_t i, float (&f)[8]) {
        Raw q;
        get(p, i, q);
        unpack(q, f);
    }
    static __device__ __forceinline__ void unpack(const Raw &q, float (&f)[8]) {
        const __half2 *h = reinterpret_cast<const __half2 *>(&q);
#pragma unroll
        for (int e = 0; e < 4; ++e) { const float2 t = __half22float2(h[e]); f[2 * e] = t.x; f[2 * e + 1] = t.y; }
    }
    static __device__ __forceinline__ void st(void *p, size_t i, const float (&f)[8]) {
        uint4 q;
        __half2 *h = reinterpret_cast<__half2 *>(&q);
#pragma unroll
        for (int e = 0; e < 4; ++e) h[e] = __floats2half2_rn(f[2 * e], f[2 * e + 1]);
        *reinterpret_cast<uint4 *>(static_cast<__half *>(p) + i) = q;
    }
};
template <> struct V8<float> {
    struct Raw { float4 a, b; };
    static __device__ __forceinline__ void get(const void *p, size_t i, Raw &q) {
        q.a = *reinterpret_cast<const float4 *>(static_cast<const float *>(p) + i);
        q.b = *reinterpret_cast<const float4 *>(static_cast<const float *>(p) + i + 4);
    }
    static __device__ __forceinline__ void ld(const void *p, size_t i, float (&f)[8]) {
        Raw q;
        get(p, i, q);
        unpack(q, f);
    }
    static __device__ __forceinline__ void unpack(const Raw &q, float (&f)[8]) {
        const float4 a = q.a, b = q.b;
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }
    static __device__ __forceinline__ void st(void *p, size_t i, const float (&f)[8]) {
        *reinterpret_cast<float4 *>(static_cast<float *>(p) + i) = make_float4(f[0], f[1], f[2], f[3]);
        *reinterpret_cast<float4 *>(static_cast<float *>(p) + i + 4) = make_float4(f[4], f[5], f[6], f[7]);
    }
};

// Work item = (batch row b, run of kRun tokens, channel octet).  Items are laid out octet-fastest so that a warp
// reads 512 contiguous bytes of a token.
struct ShiftGeom {
    int B, T, C, runs, octets;
    size_t items;
};
__host__ __device__ inline ShiftGeom shift_geom(int B, int T, int C) {
    ShiftGeom g;
    g.B = B; g.T = T; g.C = C; g.runs = (T + kRun - 1) / kRun; g.octets = C / 8;
    g.items = (size_t)B * g.runs * g.octets;
    return g;
}

// m and out are dense [nmix][B][T][C] of the activation dtype
template <typename T, int NMIX>
__global__ void __launch_bounds__(256) shift_mix_fwd_kernel(ShiftGeom g, const void *__restrict__ x, const void *__restrict__ m,
                                                            void *__restrict__ out) {
    const size_t item = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= g.items) return;
    const int oct = (int)(item % g.octets);
    const int run = (int)((item / g.octets) % g.runs);
    const int b = (int)(item / ((size_t)g.octets * g.runs));
    const int t0 = run * kRun, t1 = min(t0 + kRun, g.T);
    const size_t plane = (size_t)g.B * g.T * g.C;
    float prev[8] = {};
    if (t0 > 0) V8<T>::ld(x, ((size_t)b * g.T + t0 - 1) * g.C + oct * 8, prev);
    for (int t = t0; t < t1; ++t) {
        const size_t i = ((size_t)b * g.T + t) * g.C + oct * 8;
        float xv[8];
        V8<T>::ld(x, i, xv);
#pragma unroll
        for (int j = 0; j < NMIX; ++j) {
            float o[8], mv[8];
            V8<T>::ld(m, (size_t)j * plane + i, mv);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = fmaf(prev[e] - xv[e], mv[e], xv[e]);
            V8<T>::st(out, (size_t)j * plane + i, o);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) prev[e] = xv[e];
    }
}

// gx[t] = sum_j gout_j[t] (1 - m_j[t]) + gs[t+1],  gs[t] = sum_j gout_j[t] m_j[t]  (gs beyond the last token is 0);
// gm_j[t] = gout_j[t] (x[t-1] - x[t])
template <typename T, int NMIX>
__global__ void __launch_bounds__(256) shift_mix_bwd_kernel(ShiftGeom g, const void *__restrict__ x, const void *__restrict__ m,
                                                            const void *__restrict__ gout, void *__restrict__ gx,
                                                            void *__restrict__ gm) {
    const size_t item = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= g.items) return;
    const int oct = (int)(item % g.octets);
    const int run = (int)((item / g.octets) % g.runs);
    const int b = (int)(item / ((size_t)g.octets * g.runs));
    const int t0 = run * kRun, t1 = min(t0 + kRun, g.T);
    const size_t plane = (size_t)g.B * g.T * g.C;
    // gs of the token after this run
    float gs_next[8] = {};
    if (t1 < g.T) {
        const size_t i = ((size_t)b * g.T + t1) * g.C + oct * 8;
#pragma unroll
        for (int j = 0; j < NMIX; ++j) {
            float go[8], mv[8];
            V8<T>::ld(gout, (size_t)j * plane + i, go);
            V8<T>::ld(m, (size_t)j * plane + i, mv);
#pragma unroll
            for (int e = 0; e < 8; ++e) gs_next[e] = fmaf(go[e], mv[e], gs_next[e]);
        }
    }
    float xcur[8];
    V8<T>::ld(x, ((size_t)b * g.T + t1 - 1) * g.C + oct * 8, xcur);
    for (int t = t1 - 1; t >= t0; --t) {
        const size_t i = ((size_t)b * g.T + t) * g.C + oct * 8;
        float xprev[8] = {};
        if (t > 0) V8<T>::ld(x, i - g.C, xprev);
        float acc[8], gs[8] = {};
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = gs_next[e];
#pragma unroll
        for (int j = 0; j < NMIX; ++j) {
            float go[8], mv[8];
            V8<T>::ld(gout, (size_t)j * plane + i, go);
            V8<T>::ld(m, (size_t)j * plane + i, mv);
            float gmj[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float gom = go[e] * mv[e];
                gs[e] += gom;
                acc[e] += go[e] - gom;
                gmj[e] = go[e] * (xprev[e] - xcur[e]);
            }
            V8<T>::st(gm, (size_t)j * plane + i, gmj);
        }
        V8<T>::st(gx, i, acc);
#pragma unroll
        for (int e = 0; e < 8; ++e) { gs_next[e] = gs[e]; xcur[e] = xprev[e]; }
    }
}

// Vector mixes (one fp32 value per channel): NV of them share one read of x and, backward, one gx.  A thread holds eight
// channels of a short run of tokens, all of whose loads are in flight at once (with runs of 32 and one token in flight the
// backward of 4 x 1024 tokens x 2048 channels ran at 1.7 TB/s: 30 us).  Block = 32 channel octets x 8 consecutive runs.
constexpr int kVecGroups = 8;
__host__ __device__ constexpr int vec_run(int nv) { return nv == 1 ? 8 : 4; }
struct VecMix { const float *mu[2]; void *out[2]; };                 // forward
struct VecGrad { const float *mu[2]; const void *gout[2]; };         // backward

template <typename T, int NV>
__global__ void __launch_bounds__(256) shift_mix_vec_fwd_kernel(int T_, int C, int blocks_per_row, const void *__restrict__ x, VecMix a) {
    constexpr int RUN = vec_run(NV);
    const int oct = blockIdx.y * 32 + (threadIdx.x & 31);
    const int b = blockIdx.x / blocks_per_row, t0 = ((blockIdx.x % blocks_per_row) * kVecGroups + (threadIdx.x >> 5)) * RUN;
    if (oct >= C / 8 || t0 >= T_) return;
    const size_t i0 = ((size_t)b * T_ + t0) * C + oct * 8;
    typename V8<T>::Raw xr[RUN + 1];
    float mu[NV][8];
    if (t0 > 0) V8<T>::get(x, i0 - C, xr[0]);
#pragma unroll
    for (int e = 0; e < RUN; ++e)
        if (t0 + e < T_) V8<T>::get(x, i0 + (size_t)e * C, xr[e + 1]);
#pragma unroll
    for (int v = 0; v < NV; ++v) V8<float>::ld(a.mu[v], (size_t)oct * 8, mu[v]);
    float prev[8] = {};
    if (t0 > 0) V8<T>::unpack(xr[0], prev);
#pragma unroll
    for (int e = 0; e < RUN; ++e)
        if (t0 + e < T_) {
            float xv[8];
            V8<T>::unpack(xr[e + 1], xv);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                float o[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) o[c] = fmaf(prev[c] - xv[c], mu[v][c], xv[c]);
                V8<T>::st(a.out[v], i0 + (size_t)e * C, o);
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) prev[c] = xv[c];
        }
}

// gx as above with m_v one vector each; gmu_v[c] = sum_t gout_v[t] (x[t-1] - x[t]), summed over this block's tokens into
// partial[v][blockIdx.x][C]
template <typename T, int NV>
__global__ void __launch_bounds__(256) shift_mix_vec_bwd_kernel(int T_, int C, int blocks_per_row, const void *__restrict__ x, VecGrad a,
                                                                void *__restrict__ gx, float *__restrict__ partial) {
    constexpr int RUN = vec_run(NV);
    __shared__ float red[kVecGroups][32 * 8];
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5, oct = blockIdx.y * 32 + lane;
    const int b = blockIdx.x / blocks_per_row, t0 = ((blockIdx.x % blocks_per_row) * kVecGroups + grp) * RUN;
    float gmu[NV][8] = {};
    if (oct < C / 8 && t0 < T_) {
        const size_t i0 = ((size_t)b * T_ + t0) * C + oct * 8;
        typename V8<T>::Raw xr[RUN + 1], gr[NV][RUN + 1];
        float mu[NV][8];
        if (t0 > 0) V8<T>::get(x, i0 - C, xr[0]);
#pragma unroll
        for (int e = 0; e <= RUN; ++e)
            if (t0 + e < T_) {
                if (e < RUN) V8<T>::get(x, i0 + (size_t)e * C, xr[e + 1]);
#pragma unroll
                for (int v = 0; v < NV; ++v) V8<T>::get(a.gout[v], i0 + (size_t)e * C, gr[v][e]);
            }
#pragma unroll
        for (int v = 0; v < NV; ++v) V8<float>::ld(a.mu[v], (size_t)oct * 8, mu[v]);
        float prev[8] = {}, pend[8];     // pend: gx[t-1] without the part that comes back through the shift at t
        if (t0 > 0) V8<T>::unpack(xr[0], prev);
#pragma unroll
        for (int e = 0; e <= RUN; ++e) {
            float gs[8] = {}, own[8] = {};
            if (t0 + e < T_) {
                float xv[8];
                if (e < RUN) V8<T>::unpack(xr[e + 1], xv);
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    float go[8];
                    V8<T>::unpack(gr[v][e], go);
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const float gom = go[c] * mu[v][c];
                        gs[c] += gom;
                        own[c] += go[c] - gom;
                        if (e < RUN) gmu[v][c] = fmaf(go[c], prev[c] - xv[c], gmu[v][c]);
                    }
                }
                if (e < RUN) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) prev[c] = xv[c];
                }
            }
            if (e > 0 && t0 + e - 1 < T_) {
#pragma unroll
                for (int c = 0; c < 8; ++c) pend[c] += gs[c];
                V8<T>::st(gx, i0 + (size_t)(e - 1) * C, pend);
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) pend[c] = own[c];
        }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        __syncthreads();
#pragma unroll
        for (int c = 0; c < 8; ++c) red[grp][c * 32 + lane] = gmu[v][c];
        __syncthreads();
        const int c = threadIdx.x & 7, o = threadIdx.x >> 3;    // channel of the block = thread
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < kVecGroups; ++k) s += red[k][c * 32 + o];
        const int ch = blockIdx.y * 256 + threadIdx.x;
        if (ch < C) partial[((size_t)v * gridDim.x + blockIdx.x) * C + ch] = s;
    }
}

// gmu[c] = sum of the per-block partial sums in a fixed order (blockIdx.y: which mix): 32 columns x 8 row groups per block, group g
// adds the partial sums g, g + 8, ... and the eight group sums are added in group order.
__global__ void __launch_bounds__(256) shift_mix_reduce_kernel(int nparts, int C, const float *__restrict__ partial,
                                                               float *__restrict__ gmu0, float *__restrict__ gmu1) {
    __shared__ float sred[8][33];
    const int cx = threadIdx.x & 31, grp = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + cx;
    float s = 0.f;
    partial += (size_t)blockIdx.y * nparts * C;
    if (c < C) {
#pragma unroll 8
        for (int p = grp; p < nparts; p += 8) s += partial[(size_t)p * C + c];
    }
    sred[grp][cx] = s;
    __syncthreads();
    if (grp == 0 && c < C) {
        float t = sred[0][cx];
#pragma unroll
        for (int g2 = 1; g2 < 8; ++g2) t += sred[g2][cx];
        (blockIdx.y ? gmu1 : gmu0)[c] = t;
    }
}

static int shift_check(int B, int T, int C, int dtype, int nmix, const char *what) {
    if (B < 0 || T < 0 || C < 8 || C % 8) return fail(WKV6_ERR_INVALID, "%s: B=%d T=%d C=%d (C must be a positive multiple of 8)", what, B, T, C);
    if (nmix != 1 && nmix != 5) return fail(WKV6_ERR_UNSUPPORTED, "%s: nmix must be 1 or 5, got %d", what, nmix);
    if (dtype != WKV6_BF16 && dtype != WKV6_F16 && dtype != WKV6_F32) return fail(WKV6_ERR_INVALID, "%s: bad dtype %d", what, dtype);
    return WKV6_OK;
}

}  // namespace wkv6

using namespace wkv6;

#define SM_PTR(p) \
    if ((p) == nullptr || reinterpret_cast<uintptr_t>(p) % 16) return fail(WKV6_ERR_INVALID, #p " is NULL or not 16-byte aligned")

#define SM_DISPATCH(KERNEL, NMIX, ...)                                                                       \
    do {                                                                                                      \
        if (dtype == WKV6_BF16) KERNEL<__nv_bfloat16, NMIX><<<grid, 256, 0, st>>>(__VA_ARGS__);                \
        else if (dtype == WKV6_F16) KERNEL<__half, NMIX><<<grid, 256, 0, st>>>(__VA_ARGS__);                   \
        else KERNEL<float, NMIX><<<grid, 256, 0, st>>>(__VA_ARGS__);                                           \
    } while (0)

static int vec_blocks(int T, int nv) { return (T + kVecGroups * vec_run(nv) - 1) / (kVecGroups * vec_run(nv)); }   // per batch row

template <int NV>
static int vec_forward(int B, int T, int C, int dtype, const void *x, const VecMix &a, cudaStream_t st) {
    const int per_row = vec_blocks(T, NV);
    const dim3 grid((unsigned)(B * per_row), (C / 8 + 31) / 32);
    SM_DISPATCH(shift_mix_vec_fwd_kernel, NV, T, C, per_row, x, a);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "shift_mix_vec_fwd_kernel launch");
}

template <int NV>
static int vec_backward(int B, int T, int C, int dtype, const void *x, const VecGrad &a, void *gx, float *gmu0, float *gmu1,
                        void *workspace, size_t workspace_bytes, cudaStream_t st) {
    const int per_row = vec_blocks(T, NV);
    const size_t need = (size_t)NV * B * per_row * C * sizeof(float);
    if (workspace == nullptr || workspace_bytes < need || reinterpret_cast<uintptr_t>(workspace) % 16)
        return fail(WKV6_ERR_WORKSPACE, "shift_mix backward workspace: need %zu bytes (16-byte aligned), got %zu", need,
                    workspace ? workspace_bytes : (size_t)0);
    float *partial = static_cast<float *>(workspace);
    const dim3 grid((unsigned)(B * per_row), (C / 8 + 31) / 32);
    SM_DISPATCH(shift_mix_vec_bwd_kernel, NV, T, C, per_row, x, a, gx, partial);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "shift_mix_vec_bwd_kernel launch");
    shift_mix_reduce_kernel<<<dim3((C + 31) / 32, NV), 256, 0, st>>>(B * per_row, C, partial, gmu0, gmu1);
    e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "shift_mix_reduce_kernel launch");
}

extern "C" {

__attribute__((visibility("default")))
int wkv6_shift_mix_forward(int32_t B, int32_t T, int32_t C, int32_t dtype, int32_t nmix, int32_t m_is_vector, const void *x,
                           const void *m, void *out, void *stream) {
    int rc = shift_check(B, T, C, dtype, nmix, "wkv6_shift_mix_forward");
    if (rc) return rc;
    if (m_is_vector && nmix != 1) return fail(WKV6_ERR_INVALID, "a vector mix has nmix == 1");
    if (B == 0 || T == 0) return WKV6_OK;
    SM_PTR(x); SM_PTR(m); SM_PTR(out);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (m_is_vector) return vec_forward<1>(B, T, C, dtype, x, VecMix{{static_cast<const float *>(m), nullptr}, {out, nullptr}}, st);
    const ShiftGeom g = shift_geom(B, T, C);
    const unsigned grid = (unsigned)((g.items + 255) / 256);
    if (nmix == 1) SM_DISPATCH(shift_mix_fwd_kernel, 1, g, x, m, out);
    else SM_DISPATCH(shift_mix_fwd_kernel, 5, g, x, m, out);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "shift_mix_fwd_kernel launch");
}

__attribute__((visibility("default")))
size_t wkv6_shift_mix_workspace_bytes(int32_t B, int32_t T, int32_t C, int32_t m_is_vector) {
    if (!m_is_vector || B <= 0 || T <= 0 || C <= 0) return 0;
    const int nv = m_is_vector == 2 ? 2 : 1;     // any other value is a truth value
    return (size_t)nv * B * vec_blocks(T, nv) * C * sizeof(float);
}

__attribute__((visibility("default")))
int wkv6_shift_mix_pair_forward(int32_t B, int32_t T, int32_t C, int32_t dtype, const void *x, const float *mu0, const float *mu1,
                                void *out0, void *out1, void *stream) {
    int rc = shift_check(B, T, C, dtype, 1, "wkv6_shift_mix_pair_forward");
    if (rc) return rc;
    if (B == 0 || T == 0) return WKV6_OK;
    SM_PTR(x); SM_PTR(mu0); SM_PTR(mu1); SM_PTR(out0); SM_PTR(out1);
    return vec_forward<2>(B, T, C, dtype, x, VecMix{{mu0, mu1}, {out0, out1}}, static_cast<cudaStream_t>(stream));
}

__attribute__((visibility("default")))
int wkv6_shift_mix_pair_backward(int32_t B, int32_t T, int32_t C, int32_t dtype, const void *x, const float *mu0, const float *mu1,
                                 const void *gout0, const void *gout1, void *gx, float *gmu0, float *gmu1, void *workspace,
                                 size_t workspace_bytes, void *stream) {
    int rc = shift_check(B, T, C, dtype, 1, "wkv6_shift_mix_pair_backward");
    if (rc) return rc;
    SM_PTR(gmu0); SM_PTR(gmu1);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (B == 0 || T == 0) {
        cudaError_t e = cudaMemsetAsync(gmu0, 0, (size_t)C * sizeof(float), st);
        if (e == cudaSuccess) e = cudaMemsetAsync(gmu1, 0, (size_t)C * sizeof(float), st);
        return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "cudaMemsetAsync(gmu)");
    }
    SM_PTR(x); SM_PTR(mu0); SM_PTR(mu1); SM_PTR(gout0); SM_PTR(gout1); SM_PTR(gx);
    return vec_backward<2>(B, T, C, dtype, x, VecGrad{{mu0, mu1}, {gout0, gout1}}, gx, gmu0, gmu1, workspace, workspace_bytes, st);
}

__attribute__((visibility("default")))
int wkv6_shift_mix_backward(int32_t B, int32_t T, int32_t C, int32_t dtype, int32_t nmix, int32_t m_is_vector, const void *x,
                            const void *m, const void *gout, void *gx, void *gm, void *workspace, size_t workspace_bytes,
                            void *stream) {
    int rc = shift_check(B, T, C, dtype, nmix, "wkv6_shift_mix_backward");
    if (rc) return rc;
    if (m_is_vector && nmix != 1) return fail(WKV6_ERR_INVALID, "a vector mix has nmix == 1");
    SM_PTR(gm);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (B == 0 || T == 0) {
        if (m_is_vector) {
            cudaError_t e0 = cudaMemsetAsync(gm, 0, (size_t)C * sizeof(float), st);
            if (e0 != cudaSuccess) return cuda_fail(e0, "cudaMemsetAsync(gmu)");
        }
        return WKV6_OK;
    }
    SM_PTR(x); SM_PTR(m); SM_PTR(gout); SM_PTR(gx);
    if (m_is_vector)
        return vec_backward<1>(B, T, C, dtype, x, VecGrad{{static_cast<const float *>(m), nullptr}, {gout, nullptr}}, gx,
                               static_cast<float *>(gm), nullptr, workspace, workspace_bytes, st);
    const ShiftGeom g = shift_geom(B, T, C);
    const unsigned grid = (unsigned)((g.items + 255) / 256);
    if (nmix == 1) SM_DISPATCH(shift_mix_bwd_kernel, 1, g, x, m, gout, gx, gm);
    else SM_DISPATCH(shift_mix_bwd_kernel, 5, g, x, m, gout, gx, gm);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "shift_mix_bwd_kernel launch");
}

}  // extern "C"
