// Data-dependent token-shift interpolations with their low-rank products inside (TimeMix.call, rwkv6_model.py:128-146):
//   l_j[t,c]   = bias_j[c] + sum_k h_j[t,k] B_j[k,c]                                j = 0..4, k < 32
//   out_j[t,c] = x[t,c] + (x[t-1,c] - x[t,c]) l_j[t,c]                              x[-1] = 0
// and the backward to x and l.  h holds the five tanh(x_mix A_j) side by side ([rows][160]).
//
// As separate steps (bias broadcast into the result, batched product onto it, element-wise kernel) the five l tensors crossed
// HBM four times and the broadcast ran at 1 TB/s (about 300 us forward at 4004 x 4096 in all).  Here l lives in accumulators only; what is
// left is x in and five results out (12 bytes per token and channel), backward x and five gradients in, gx and five gradients out
// (24).  Measured with a cold L2 at 4004 x 4096: forward 73 us, backward 150 us (forward L1 at 87 %, mostly the weight fragments each
// tile re-reads); at 4096 x 2048 49 us and 83 us.
//
// A product over k = 32 is two mma.m16n8k16 steps: the tensor work is a tenth of the transfer time, so the warp-level
// instruction is enough, and its fragments can be arranged so that nothing is staged:
//   * column n of the four n8 tiles j of a 32-channel group stands for channel 8 (n / 2) + 2 j + n % 2, so that the accumulators
//     of a thread are eight neighbouring channels (16-byte accesses to x, gout and the results);
//   * reduction index (step s, register half hh, quad lane q, element e) stands for k = 16 s + 4 q + 2 hh + e, so that a thread's
//     share of a row of h_j is one 8-byte load per step.
// l has the bits of the general path (the library's batched product with the bias added onto it, then shift_mix_*_kernel): each
// step sums the same 16 k, and product and sum are rounded where that path stores them.  The gradients of a training step are not
// determined to better than that: behind a token whose WKV output is nearly zero the per-head norm magnifies single rounding
// steps of bf16, so that 8 elements of l in a million one step off (another order of the k) move gradients by percents.
// One CTA: 128 channels, B_j in shared memory in fragment order (40 KB), eight warps = four groups of 32 channels x two runs
// of rows.  A warp walks tiles of 16 rows; the backward walks down, because gx[t] needs sum_j gout_j l_j of token t + 1.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "wkv6_internal.h"

namespace wkv6 {

constexpr int kMixes = 5, kRank = 32, kMixCols = 128, kMixThreads = 256, kMixLanes = 2;  // kMixLanes: runs of rows per CTA
constexpr int kMixWords = kMixes * 4 * 4 * 32 * 4;                                       // [mix][group][tile][lane][step, half]
constexpr int kMixSmem = kMixWords * 4 + kMixes * kMixCols * 4;
constexpr int kMixBwdSmem = kMixSmem + kMixes * 2 * kMixThreads * 16;                     // and a tile's l, [mix][row half][thread]

struct MixOut { __nv_bfloat16 *p[5]; };
struct MixGrad { const __nv_bfloat16 *p[5]; };

struct LoraGeom {
    int T, C;
    int rows;             // B * T
    int tiles;            // of 16 rows
    int run;              // tiles per run
};

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// a lane's share of a row of h_j: k = 4 q .. 4 q + 3 and 16 + 4 q .. 16 + 4 q + 3 (p points at its first element)
__device__ __forceinline__ uint4 ld_h(const __nv_bfloat16 *p, bool ok) {
    const uint2 zero = make_uint2(0u, 0u);
    const uint2 a = ok ? __ldg(reinterpret_cast<const uint2 *>(p)) : zero, b = ok ? __ldg(reinterpret_cast<const uint2 *>(p + 16)) : zero;
    return make_uint4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ uint4 ld_row(const __nv_bfloat16 *p, bool ok) {
    return ok ? __ldg(reinterpret_cast<const uint4 *>(p)) : make_uint4(0u, 0u, 0u, 0u);
}

__device__ __forceinline__ void unpack8(const uint4 &v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t *>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// B_j and the biases of this CTA's channels into shared memory; channels beyond C are zero.
__device__ __forceinline__ void stage_weights(const __nv_bfloat16 *wb, const __nv_bfloat16 *bias, int C, int ch0, uint32_t *sB, float *sBias) {
    // all loads first: one round trip to memory in front of the first tile instead of twenty
    constexpr int kEach = kMixes * (kRank / 2) * (kMixCols / 2) / kMixThreads;
    uint32_t lo[kEach], hi[kEach];   // rows k and k + 1, channels c and c + 1
    float b[(kMixes * kMixCols + kMixThreads - 1) / kMixThreads];
#pragma unroll
    for (int e = 0; e < kEach; ++e) {
        const int i = threadIdx.x + e * kMixThreads, cp = i % (kMixCols / 2), kp = i / (kMixCols / 2) % (kRank / 2), m = i / (kMixCols / 2 * (kRank / 2));
        const bool ok = ch0 + 2 * cp < C;
        const __nv_bfloat16 *p = wb + ((size_t)m * kRank + 2 * kp) * C + ch0 + 2 * cp;
        lo[e] = ok ? __ldg(reinterpret_cast<const uint32_t *>(p)) : 0u;
        hi[e] = ok ? __ldg(reinterpret_cast<const uint32_t *>(p + C)) : 0u;
    }
#pragma unroll
    for (int e = 0; e * kMixThreads < kMixes * kMixCols; ++e) {
        const int i = threadIdx.x + e * kMixThreads, m = i / kMixCols, c = i % kMixCols;
        b[e] = i < kMixes * kMixCols && ch0 + c < C ? __bfloat162float(bias[(size_t)m * C + ch0 + c]) : 0.f;
    }
#pragma unroll
    for (int e = 0; e < kEach; ++e) {
        const int i = threadIdx.x + e * kMixThreads, cp = i % (kMixCols / 2), kp = i / (kMixCols / 2) % (kRank / 2), m = i / (kMixCols / 2 * (kRank / 2));
        const int c = 2 * cp, k = 2 * kp, grp = c >> 5, cc = c & 31, n = 2 * (cc >> 3), tile = (cc & 7) >> 1;
        const int q = (k >> 2) & 3, w = 2 * (k >> 4) + ((k >> 1) & 1);
        uint32_t *d = sB + ((((m * 4 + grp) * 4 + tile) * 32) + 4 * n + q) * 4 + w;
        d[0] = __byte_perm(lo[e], hi[e], 0x5410);    // channel c:     n
        d[16] = __byte_perm(lo[e], hi[e], 0x7632);   // channel c + 1: n + 1, four lanes further
    }
#pragma unroll
    for (int e = 0; e * kMixThreads < kMixes * kMixCols; ++e)
        if (threadIdx.x + e * kMixThreads < kMixes * kMixCols) sBias[threadIdx.x + e * kMixThreads] = b[e];
    __syncthreads();
}

// product rounded, then the sum with the bias rounded, as the general path leaves them
__device__ __forceinline__ float2 biased(float x, float y, float2 bias) {
    const float2 p = __bfloat1622float2(__floats2bfloat162_rn(x, y));
    return __bfloat1622float2(__floats2bfloat162_rn(p.x + bias.x, p.y + bias.y));
}

// l of one mix for this thread's two rows (g, g + 8) and eight channels
__device__ __forceinline__ void mix_product(const uint4 &ha, const uint4 &hb, const uint32_t *sB, const float *sBias, float (&la)[8], float (&lb)[8]) {
    const uint32_t a0[4] = {ha.x, hb.x, ha.y, hb.y}, a1[4] = {ha.z, hb.z, ha.w, hb.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint4 b = *reinterpret_cast<const uint4 *>(sB + j * 128);
        const float2 bi = *reinterpret_cast<const float2 *>(sBias + 2 * j);
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        mma_16816(d, a0, b.x, b.y);
        mma_16816(d, a1, b.z, b.w);
        const float2 a = biased(d[0], d[1], bi), c = biased(d[2], d[3], bi);
        la[2 * j] = a.x; la[2 * j + 1] = a.y;
        lb[2 * j] = c.x; lb[2 * j + 1] = c.y;
    }
}

__global__ void __launch_bounds__(kMixThreads, 2) lora_mix_fwd_kernel(LoraGeom G, const __nv_bfloat16 *__restrict__ x,
                                                                      const __nv_bfloat16 *__restrict__ h,
                                                                      const __nv_bfloat16 *__restrict__ wb,
                                                                      const __nv_bfloat16 *__restrict__ bias,
                                                                      MixOut out) {
    extern __shared__ __align__(16) uint32_t sB[];
    float *sBias = reinterpret_cast<float *>(sB + kMixWords);
    const int ch0 = blockIdx.x * kMixCols;
    stage_weights(wb, bias, G.C, ch0, sB, sBias);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = warp & 3, g = lane >> 2, q = lane & 3;
    const int ch = ch0 + 32 * grp + 8 * q;
    const bool chan = ch < G.C;
    const int t0 = ((int)blockIdx.y * kMixLanes + (warp >> 2)) * G.run, t1 = min(t0 + G.run, G.tiles);
    const uint32_t *myB = sB + (grp * 4 * 32 + lane) * 4;
    const float *myBias = sBias + 32 * grp + 8 * q;
    // what the next tile reads is requested while this one is computed: every register of h as soon as its product is done
    uint4 ha[kMixes], hb[kMixes], xa4, xb4, pa4, pb4;
    auto fetch_h = [&](int t, int m) {
        const int ra = 16 * t + g, rb = ra + 8;
        ha[m] = ld_h(h + (size_t)ra * (kMixes * kRank) + m * kRank + 4 * q, ra < G.rows);
        hb[m] = ld_h(h + (size_t)rb * (kMixes * kRank) + m * kRank + 4 * q, rb < G.rows);
    };
    auto fetch_x = [&](int t) {
        const int ra = 16 * t + g, rb = ra + 8;
        const bool oka = ra < G.rows && chan, okb = rb < G.rows && chan;
        const __nv_bfloat16 *px = x + (size_t)ra * G.C + ch;
        xa4 = ld_row(px, oka); xb4 = ld_row(px + (size_t)8 * G.C, okb);
        pa4 = ld_row(px - G.C, oka && ra % G.T != 0); pb4 = ld_row(px + (size_t)7 * G.C, okb && rb % G.T != 0);
    };
    if (t0 < t1) {
        fetch_x(t0);
#pragma unroll
        for (int m = 0; m < kMixes; ++m) fetch_h(t0, m);
    }
    for (int t = t0; t < t1; ++t) {
        const int ra = 16 * t + g;
        const bool oka = ra < G.rows && chan, okb = ra + 8 < G.rows && chan, more = t + 1 < t1;
        float xa[8], xb[8], da[8], db[8];
        unpack8(xa4, xa); unpack8(xb4, xb); unpack8(pa4, da); unpack8(pb4, db);
        if (more) fetch_x(t + 1);
#pragma unroll
        for (int e = 0; e < 8; ++e) { da[e] -= xa[e]; db[e] -= xb[e]; }
        const size_t i = (size_t)ra * G.C + ch;
#pragma unroll
        for (int m = 0; m < kMixes; ++m) {
            float la[8], lb[8];
            mix_product(ha[m], hb[m], myB + m * (4 * 4 * 128), myBias + m * kMixCols, la, lb);
            if (more) fetch_h(t + 1, m);
#pragma unroll
            for (int e = 0; e < 8; ++e) { la[e] = fmaf(da[e], la[e], xa[e]); lb[e] = fmaf(db[e], lb[e], xb[e]); }
            if (oka) *reinterpret_cast<uint4 *>(out.p[m] + i) = pack8(la);
            if (okb) *reinterpret_cast<uint4 *>(out.p[m] + i + (size_t)8 * G.C) = pack8(lb);
        }
    }
}

// gl_j[t] = gout_j[t] (x[t-1] - x[t]);  gx[t] = sum_j gout_j[t] (1 - l_j[t]) + s[t+1],  s[t] = sum_j gout_j[t] l_j[t]
// (s[t+1] = 0 at the last token of a batch row).  Inside a tile s[t+1] comes from the lane four further (the second rows for
// the last of the first eight), across tiles it is carried; a run starts with the s of the row behind it.  gx is summed in the
// order of shift_mix_bwd_kernel, s[t+1] first and then mix by mix, so that it has that kernel's bits: each thread keeps its l in
// shared memory until the s of the tile are known (4096 x 2048: 83 us; 71 us with s[t+1] added last, 87 us with l kept in registers).
__global__ void __launch_bounds__(kMixThreads) lora_mix_bwd_kernel(LoraGeom G, const __nv_bfloat16 *__restrict__ x,
                                                                   const __nv_bfloat16 *__restrict__ h,
                                                                   const __nv_bfloat16 *__restrict__ wb,
                                                                   const __nv_bfloat16 *__restrict__ bias,
                                                                   MixGrad gout, __nv_bfloat16 *__restrict__ gx,
                                                                   __nv_bfloat16 *__restrict__ gl) {
    extern __shared__ __align__(16) uint32_t sB[];
    float *sBias = reinterpret_cast<float *>(sB + kMixWords);
    const int ch0 = blockIdx.x * kMixCols;
    stage_weights(wb, bias, G.C, ch0, sB, sBias);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = warp & 3, g = lane >> 2, q = lane & 3;
    const int ch = ch0 + 32 * grp + 8 * q;
    const bool chan = ch < G.C;
    const int t0 = ((int)blockIdx.y * kMixLanes + (warp >> 2)) * G.run, t1 = min(t0 + G.run, G.tiles);
    if (t0 >= t1) return;
    const size_t plane = (size_t)G.rows * G.C;
    const uint32_t *myB = sB + (grp * 4 * 32 + lane) * 4;
    const float *myBias = sBias + 32 * grp + 8 * q;
    uint4 *sL = reinterpret_cast<uint4 *>(sBias + kMixes * kMixCols) + threadIdx.x;
    float carry[8];   // lanes g = 0: s of the first row of the tile behind
#pragma unroll
    for (int e = 0; e < 8; ++e) carry[e] = 0.f;
    // what the next tile reads is requested while this one is computed (see the forward)
    uint4 ha[kMixes], hb[kMixes], goa4[kMixes], gob4[kMixes], xa4, xb4, pa4, pb4;
    auto fetch_h = [&](int t, int m) {
        const int ra = 16 * t + g, rb = ra + 8;
        const bool oka = ra < G.rows && (t != t1 || g == 0), okb = rb < G.rows && t != t1;
        ha[m] = ld_h(h + (size_t)ra * (kMixes * kRank) + m * kRank + 4 * q, oka);
        hb[m] = ld_h(h + (size_t)rb * (kMixes * kRank) + m * kRank + 4 * q, okb);
    };
    auto fetch_g = [&](int t, int m) {
        const int ra = 16 * t + g, rb = ra + 8;
        const bool oka = ra < G.rows && (t != t1 || g == 0), okb = rb < G.rows && t != t1;
        const __nv_bfloat16 *pg = gout.p[m] + (size_t)ra * G.C + ch;
        goa4[m] = ld_row(pg, oka && chan);
        gob4[m] = ld_row(pg + (size_t)8 * G.C, okb && chan);
    };
    auto fetch_x = [&](int t) {
        const int ra = 16 * t + g, rb = ra + 8;
        const bool oka = ra < G.rows && chan && t != t1, okb = rb < G.rows && chan && t != t1;
        const __nv_bfloat16 *px = x + (size_t)ra * G.C + ch;
        xa4 = ld_row(px, oka); xb4 = ld_row(px + (size_t)8 * G.C, okb);
        pa4 = ld_row(px - G.C, oka && ra % G.T != 0); pb4 = ld_row(px + (size_t)7 * G.C, okb && rb % G.T != 0);
    };
    const int first = t1 < G.tiles ? t1 : t1 - 1;
    fetch_x(first);
#pragma unroll
    for (int m = 0; m < kMixes; ++m) { fetch_h(first, m); fetch_g(first, m); }
    for (int t = first; t >= t0; --t) {
        const bool ahead = t == t1, more = t > t0;    // ahead: only s of its first row is wanted
        const int ra = 16 * t + g, rb = ra + 8;
        const bool oka = ra < G.rows && chan && !ahead, okb = rb < G.rows && chan && !ahead;
        const size_t i = (size_t)ra * G.C + ch;
        float da[8], db[8];
        {
            float xa[8], xb[8];
            unpack8(xa4, xa); unpack8(xb4, xb); unpack8(pa4, da); unpack8(pb4, db);
#pragma unroll
            for (int e = 0; e < 8; ++e) { da[e] -= xa[e]; db[e] -= xb[e]; }
        }
        if (more) fetch_x(t - 1);
        float sa[8], sb[8], aa[8], ab[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) sa[e] = sb[e] = 0.f;
#pragma unroll
        for (int m = 0; m < kMixes; ++m) {
            float la[8], lb[8], ga[8], gb[8];
            mix_product(ha[m], hb[m], myB + m * (4 * 4 * 128), myBias + m * kMixCols, la, lb);
            unpack8(goa4[m], ga); unpack8(gob4[m], gb);
#pragma unroll
            for (int e = 0; e < 8; ++e) { sa[e] = fmaf(ga[e], la[e], sa[e]); sb[e] = fmaf(gb[e], lb[e], sb[e]); }
            sL[(2 * m) * kMixThreads] = pack8(la); sL[(2 * m + 1) * kMixThreads] = pack8(lb);
            if (more) fetch_h(t - 1, m);
        }
        const bool enda = (ra + 1) % G.T == 0, endb = (rb + 1) % G.T == 0;   // last token of a batch row: nothing comes back
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float na = __shfl_sync(0xffffffffu, g == 0 ? sb[e] : sa[e], (lane + 4) & 31);
            const float nb = __shfl_sync(0xffffffffu, g == 0 ? carry[e] : sb[e], (lane + 4) & 31);
            aa[e] = enda ? 0.f : na;
            ab[e] = endb ? 0.f : nb;
            carry[e] = sa[e];
        }
#pragma unroll
        for (int m = 0; m < kMixes; ++m) {
            float la[8], lb[8], ga[8], gb[8];
            unpack8(sL[(2 * m) * kMixThreads], la); unpack8(sL[(2 * m + 1) * kMixThreads], lb);
            unpack8(goa4[m], ga); unpack8(gob4[m], gb);
            if (more) fetch_g(t - 1, m);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                aa[e] += fmaf(-ga[e], la[e], ga[e]); ab[e] += fmaf(-gb[e], lb[e], gb[e]);
                ga[e] *= da[e]; gb[e] *= db[e];
            }
            __nv_bfloat16 *po = gl + m * plane + i;
            if (oka) *reinterpret_cast<uint4 *>(po) = pack8(ga);
            if (okb) *reinterpret_cast<uint4 *>(po + (size_t)8 * G.C) = pack8(gb);
        }
        if (oka) *reinterpret_cast<uint4 *>(gx + i) = pack8(aa);
        if (okb) *reinterpret_cast<uint4 *>(gx + i + (size_t)8 * G.C) = pack8(ab);
    }
}

// Runs of rows: as many as give every SM `per_sm` CTAs, no shorter than `shortest` tiles (the backward reads one row more per run).
static LoraGeom lora_geom(int B, int T, int C, int per_sm, int shortest, dim3 *grid) {
    LoraGeom G;
    G.T = T; G.C = C; G.rows = B * T; G.tiles = (G.rows + 15) / 16;
    const int cols = (C + kMixCols - 1) / kMixCols;
    const int splits = per_sm * sm_count() / cols > 1 ? per_sm * sm_count() / cols : 1;
    G.run = (G.tiles + splits * kMixLanes - 1) / (splits * kMixLanes);
    if (G.run < shortest) G.run = shortest;
    *grid = dim3((unsigned)cols, (unsigned)((G.tiles + G.run * kMixLanes - 1) / (G.run * kMixLanes)));
    return G;
}

static int lora_check(int B, int T, int C, const char *what) {
    if (B < 0 || T < 0 || C < 8 || C % 8) return fail(WKV6_ERR_INVALID, "%s: B=%d T=%d C=%d (C must be a positive multiple of 8)", what, B, T, C);
    if ((int64_t)B * T > (1 << 30)) return fail(WKV6_ERR_UNSUPPORTED, "%s: B=%d T=%d: more than 2^30 tokens", what, B, T);
    return WKV6_OK;
}

}  // namespace wkv6

using namespace wkv6;

#define LM_PTR(p) \
    if ((p) == nullptr || reinterpret_cast<uintptr_t>(p) % 16) return fail(WKV6_ERR_INVALID, #p " is NULL or not 16-byte aligned")

extern "C" {

__attribute__((visibility("default")))
int wkv6_lora_mix_forward(int32_t B, int32_t T, int32_t C, const void *x, const void *h, const void *wb, const void *bias,
                          void *const *out, void *stream) {
    if (int rc = lora_check(B, T, C, "wkv6_lora_mix_forward")) return rc;
    if (B == 0 || T == 0) return WKV6_OK;
    LM_PTR(x); LM_PTR(h); LM_PTR(wb); LM_PTR(bias);
    if (out == nullptr) return fail(WKV6_ERR_INVALID, "out is NULL");
    MixOut o;
    for (int m = 0; m < kMixes; ++m) { LM_PTR(out[m]); o.p[m] = static_cast<__nv_bfloat16 *>(out[m]); }
    dim3 grid;
    const LoraGeom G = lora_geom(B, T, C, 2, 1, &grid);
    using bf = __nv_bfloat16;
    lora_mix_fwd_kernel<<<grid, kMixThreads, kMixSmem, static_cast<cudaStream_t>(stream)>>>(
        G, static_cast<const bf *>(x), static_cast<const bf *>(h), static_cast<const bf *>(wb), static_cast<const bf *>(bias), o);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "lora_mix_fwd_kernel launch");
}

__attribute__((visibility("default")))
int wkv6_lora_mix_backward(int32_t B, int32_t T, int32_t C, const void *x, const void *h, const void *wb, const void *bias, const void *const *gout,
                           void *gx, void *gl, void *stream) {
    if (int rc = lora_check(B, T, C, "wkv6_lora_mix_backward")) return rc;
    if (B == 0 || T == 0) return WKV6_OK;
    LM_PTR(x); LM_PTR(h); LM_PTR(wb); LM_PTR(bias); LM_PTR(gx); LM_PTR(gl);
    if (gout == nullptr) return fail(WKV6_ERR_INVALID, "gout is NULL");
    MixGrad go;
    for (int m = 0; m < kMixes; ++m) { LM_PTR(gout[m]); go.p[m] = static_cast<const __nv_bfloat16 *>(gout[m]); }
    dim3 grid;
    const LoraGeom G = lora_geom(B, T, C, 1, 4, &grid);
    using bf = __nv_bfloat16;
    cudaError_t e = cudaFuncSetAttribute(lora_mix_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMixBwdSmem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(lora_mix_bwd_kernel)");
    lora_mix_bwd_kernel<<<grid, kMixThreads, kMixBwdSmem, static_cast<cudaStream_t>(stream)>>>(
        G, static_cast<const bf *>(x), static_cast<const bf *>(h), static_cast<const bf *>(wb), static_cast<const bf *>(bias),
        go, static_cast<bf *>(gx), static_cast<bf *>(gl));
    e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "lora_mix_bwd_kernel launch");
}

}  // extern "C"
