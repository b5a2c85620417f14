// Step-by-step (register-state) WKV6 kernels for head size 64: fp32 arithmetic for any input type.
//
// One CTA of 64 threads per (batch, head, segment of the sequence); a thread keeps an 8 x 8 tile of the 64 x 64 state, as
// 32 pairs of adjacent key channels for the packed fp32 instructions (fma.rn.f32x2), and walks the segment step by step.
//
// Why this tile: a step costs three multiply-adds per state element, and what they read from shared memory must not cost
// more than they do.  With one state column x 16 rows per thread (wkv6_seq.cuh) every 12 FMAs need three 128-bit shared
// loads, four times what the load pipe delivers in that time; an 8 x 8 tile needs eight for 96 packed FMAs.  The sum over
// the eight threads that share a column (row) is a reduce-scatter of eight values: 7 shuffles.
//
// Why segments: the steps of a sequence are a chain, so B*H sequences on 148 SMs leave the chip mostly idle (64 sequences
// of 1024 steps: 1.26 ms for forward + backward, 330 us per sweep).  A segment's effect on the state is affine,
// S -> D S + b with D = exp(-sum exp(w)), so a sequence is cut into pieces that are summarised side by side (b, D), scanned
// (state_scan_kernel), and then walked side by side from their entering states.  The summary is two of the forward's three
// multiply-adds; split_segments() (wkv6_seq.cu) cuts only where the chip would otherwise idle.
//
// Measured at B2 T1024 H32 fp32 (9 segments): forward + backward 1262 -> 271 us.  The packed FMAs keep their pipe busy for
// 40-60 % of the time, the rest is issue latency with two warps per scheduler.  Capping the registers (155-248 a thread, no
// spill) for more CTAs per SM measured slower (315-424 us), as did 6 or 8 CTAs per SM by shorter segments (301-304 us) and
// no unrolling (281 us).
//
// Sweeps (S forward state, A reverse state, Z_t[i] = sum_j S_t[i][j] A_t[i][j]; gradients as in wkv6_seq.cuh):
//   step_fwd_kernel   ascending : y            (or, without an output, the summary of either direction)
//   step_gr_kernel    ascending : gr, gu, x = r * gr
//   step_gkvw_kernel  descending: gk, gv, gw from one walk of A (two separate walks in wkv6_seq.cuh)
#pragma once

#include "wkv6_seq.cuh"

namespace wkv6 {

constexpr int kStepTile = 8;        // time steps staged per tile
constexpr int kStepThreads = 64;

// ---- packed fp32 pairs ----------------------------------------------------------------------------------------------
using f2 = unsigned long long;
__device__ __forceinline__ f2 f2_pack(float lo, float hi) { f2 d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi)); return d; }
__device__ __forceinline__ float2 f2_unpack(f2 v) { float2 d; asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v)); return d; }
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) { f2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) { f2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

// Eight raw elements of a row as loaded, converted when they are staged (a half type then costs four registers in flight)
template <typename T> struct Raw8 {
    uint4 v[sizeof(T) / 2];
    __device__ __forceinline__ void load(const T *p) {
#pragma unroll
        for (int e = 0; e < (int)(sizeof(T) / 2); ++e) v[e] = __ldg(reinterpret_cast<const uint4 *>(p) + e);
    }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int e = 0; e < (int)(sizeof(T) / 2); ++e) v[e] = make_uint4(0, 0, 0, 0);
    }
    __device__ __forceinline__ void get(float (&f)[8]) const {
        const T *h = reinterpret_cast<const T *>(v);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = static_cast<float>(h[e]);
    }
};

__device__ __forceinline__ void put8(float *row, int chunk, const float (&f)[8]) {
    reinterpret_cast<float4 *>(row)[2 * chunk] = make_float4(f[0], f[1], f[2], f[3]);
    reinterpret_cast<float4 *>(row)[2 * chunk + 1] = make_float4(f[4], f[5], f[6], f[7]);
}

// sum over the eight threads that stage one row (lanes differing in their low three bits)
__device__ __forceinline__ float row_sum8(float x) {
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 4);
    return x;
}

// The eight indices of a thread's tile along one axis: 4 t .. 4 t + 3 and 32 + 4 t .. 32 + 4 t + 3 (t = 0..7), so that the
// 128-bit reads of eight neighbouring t are one contiguous 128-byte line.
__device__ __forceinline__ int tile_index(int t, int e) { return 4 * t + (e & 3) + ((e & 4) << 3); }

struct Octet { f2 p[4]; };   // elements (0,1) (2,3) (4,5) (6,7) of a tile axis
__device__ __forceinline__ Octet read_octet(const float *row, int t) {
    const ulonglong2 lo = *reinterpret_cast<const ulonglong2 *>(row + 4 * t);
    const ulonglong2 hi = *reinterpret_cast<const ulonglong2 *>(row + 32 + 4 * t);
    return Octet{{lo.x, lo.y, hi.x, hi.y}};
}
__device__ __forceinline__ void read_dup8(const float *row, int t, f2 (&d)[8]) {   // the eight values, each as a pair (x, x)
    const float4 lo = *reinterpret_cast<const float4 *>(row + 4 * t);
    const float4 hi = *reinterpret_cast<const float4 *>(row + 32 + 4 * t);
    d[0] = f2_pack(lo.x, lo.x); d[1] = f2_pack(lo.y, lo.y); d[2] = f2_pack(lo.z, lo.z); d[3] = f2_pack(lo.w, lo.w);
    d[4] = f2_pack(hi.x, hi.x); d[5] = f2_pack(hi.y, hi.y); d[6] = f2_pack(hi.z, hi.z); d[7] = f2_pack(hi.w, hi.w);
}

// Reduce-scatter of eight values over the lanes that differ in bits 2..4: the lane with t = lane >> 2 gets the sum of a[t].
__device__ __forceinline__ float scatter_sum8(const float (&a)[8], int lane) {
    float b[4], c[2];
    const bool h4 = lane & 16, h2 = lane & 8, h1 = lane & 4;
#pragma unroll
    for (int e = 0; e < 4; ++e) b[e] = (h4 ? a[e + 4] : a[e]) + __shfl_xor_sync(0xffffffffu, h4 ? a[e] : a[e + 4], 16);
#pragma unroll
    for (int e = 0; e < 2; ++e) c[e] = (h2 ? b[e + 2] : b[e]) + __shfl_xor_sync(0xffffffffu, h2 ? b[e] : b[e + 2], 8);
    return (h1 ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, h1 ? c[0] : c[1], 4);
}

// ---- geometry -------------------------------------------------------------------------------------------------------
struct StepGeom {
    int B, T, H, G, L;       // G segments of L steps (the last one shorter), L a multiple of kStepTile when G > 1
    int64_t ld, bs;
};
struct StepSeg {
    int b, h, t0, cnt;       // first step and number of steps
    size_t seq;              // (b*G + g)*H + h: row of the per-segment arrays
    int g;
    size_t base;             // element offset of (b, t0, h, 0)
};
__device__ __forceinline__ StepSeg step_segment(const StepGeom &q, int block) {
    StepSeg s;
    s.h = block % q.H;
    const int bg = block / q.H;
    s.g = bg % q.G;
    s.b = bg / q.G;
    s.t0 = s.g * q.L;
    s.cnt = min(q.L, q.T - s.t0);
    s.seq = (size_t)block;
    s.base = (size_t)s.b * q.bs + (size_t)s.t0 * q.ld + (size_t)s.h * 64;
    return s;
}

template <typename T> __device__ __forceinline__ T cast_out(float x);
template <> __device__ __forceinline__ float cast_out<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 cast_out<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

// Loads the thread's state tile from a row-major 64 x 64 fp32 matrix.
__device__ __forceinline__ void load_tile(const float *m, int ti, int tj, f2 (&S)[4][8]) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const float *r0 = m + tile_index(ti, 2 * p) * 64, *r1 = r0 + 64;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const float4 a = *reinterpret_cast<const float4 *>(r0 + 32 * half + 4 * tj);
            const float4 c = *reinterpret_cast<const float4 *>(r1 + 32 * half + 4 * tj);
            S[p][4 * half + 0] = f2_pack(a.x, c.x); S[p][4 * half + 1] = f2_pack(a.y, c.y);
            S[p][4 * half + 2] = f2_pack(a.z, c.z); S[p][4 * half + 3] = f2_pack(a.w, c.w);
        }
    }
}
__device__ __forceinline__ void zero_tile(f2 (&S)[4][8]) {
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int b = 0; b < 8; ++b) S[p][b] = 0ull;
}

struct StepFwdArgs {
    const void *P, *Q, *W, *X;   // forward: r, k, w, v; reverse summary: -, r, w, gy
    const void *u;
    void *out;                   // y
    const float *seg_in;         // G > 1: entering states [B*G,H,64,64]
    const void *s_in;            // G == 1: optional initial state [kinds,H,64,64] of s_dtype
    const int64_t *s_map;
    int s_kinds, s_dtype, u_dtype;
    void *s_out;                 // G == 1: optional final state
    float *b_out, *dec_out;      // summary: state built from zero [B*G,H,64,64], log2 of the total decay [B*G,H,64]
    int skip_g;                  // summary: the segment no scan reads (-1: none)
    bool vec_in, vec_out;        // s_in / s_out are fp32 at a 16-byte boundary: 128-bit accesses (callers' states may lie anywhere)
    StepGeom q;
};

// out_t[j] = sum_i P_t[i] S[i][j] + X_t[j] sum_i u_i P_t[i] Q_t[i],  then S[i][j] = d_t[i] S[i][j] + Q_t[i] X_t[j].
// 96 packed FMAs, 28 instructions of the reduce-scatter and 8 shared loads per step and warp.
template <typename Tx, typename TX, typename Ty, bool SUMMARY, bool REVERSE>
__global__ void __launch_bounds__(kStepThreads) step_fwd_kernel(const StepFwdArgs a) {
    constexpr int TT = kStepTile;
    __shared__ __align__(16) float sP[SUMMARY ? 1 : 2][SUMMARY ? 1 : TT][64];
    __shared__ __align__(16) float sQ[2][TT][64];
    __shared__ __align__(16) float sD[2][TT][64];
    __shared__ __align__(16) float sX[2][TT][64];
    __shared__ float sC[2][TT];

    const StepSeg s = step_segment(a.q, blockIdx.x);
    if (SUMMARY && s.g == a.skip_g) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ti = lane >> 2, tj = warp * 4 + (lane & 3);
    const int row = tid >> 3, chunk = tid & 7;
    const Tx *gP = static_cast<const Tx *>(a.P) + s.base + chunk * 8;
    const Tx *gQ = static_cast<const Tx *>(a.Q) + s.base + chunk * 8;
    const Tx *gW = static_cast<const Tx *>(a.W) + s.base + chunk * 8;
    const TX *gX = static_cast<const TX *>(a.X) + s.base + chunk * 8;

    float u8[8], dsum[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        u8[e] = SUMMARY ? 0.f : load_any(a.u, a.u_dtype, (size_t)s.h * 64 + chunk * 8 + e);
        dsum[e] = 0.f;
    }

    f2 S[4][8];
    if (SUMMARY) {
        zero_tile(S);
    } else if (a.seg_in != nullptr) {
        load_tile(a.seg_in + s.seq * 4096, ti, tj, S);
    } else if (a.s_in != nullptr) {
        int64_t kind = a.s_map ? a.s_map[s.b] : (a.s_kinds == 1 ? 0 : s.b);
        kind = kind < 0 ? 0 : (kind >= a.s_kinds ? a.s_kinds - 1 : kind);
        const size_t so = ((size_t)kind * a.q.H + s.h) * 4096;
        if (a.vec_in) {
            load_tile(static_cast<const float *>(a.s_in) + so, ti, tj, S);
        } else {
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int b = 0; b < 8; ++b) {
                    const size_t o = so + (size_t)tile_index(ti, 2 * p) * 64 + tile_index(tj, b);
                    S[p][b] = f2_pack(load_any(a.s_in, a.s_dtype, o), load_any(a.s_in, a.s_dtype, o + 64));
                }
        }
    } else {
        zero_tile(S);
    }

    Raw8<Tx> fP, fQ, fW;
    Raw8<TX> fX;
    auto fetch = [&](int tile) {
        const int t = tile * TT + row;
        if (t < s.cnt) {
            const size_t o = (size_t)t * a.q.ld;
            if (!SUMMARY) fP.load(gP + o);
            fQ.load(gQ + o); fW.load(gW + o); fX.load(gX + o);
        } else {
            if (!SUMMARY) fP.zero();
            fQ.zero(); fW.zero(); fX.zero();
        }
    };
    const int ntiles = (s.cnt + TT - 1) / TT;
    fetch(REVERSE ? ntiles - 1 : 0);
    const int jout = tile_index(tj, ti);
    Ty *gO = SUMMARY ? nullptr : static_cast<Ty *>(a.out) + s.base + jout;

    for (int it = 0; it < ntiles; ++it) {
        const int tile = REVERSE ? ntiles - 1 - it : it, buf = it & 1;
        const int n = min(TT, s.cnt - tile * TT);
        {
            float q8[8], x8[8], w8[8];
            fQ.get(q8); fX.get(x8); fW.get(w8);
            put8(sQ[buf][row], chunk, q8);
            put8(sX[buf][row], chunk, x8);
            const bool live = row < n;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float ew = expf(w8[e]);
                if (SUMMARY && live) dsum[e] += ew;
                w8[e] = expf(-ew);
            }
            put8(sD[buf][row], chunk, w8);
            if constexpr (!SUMMARY) {
                float p8[8], c = 0.f;
                fP.get(p8);
                put8(sP[buf][row], chunk, p8);
#pragma unroll
                for (int e = 0; e < 8; ++e) c = fmaf(u8[e] * p8[e], q8[e], c);
                c = row_sum8(c);
                if (chunk == 0) sC[buf][row] = c;
            }
        }
        __syncthreads();   // two buffers: whoever writes this one next has passed the barrier of the tile in between
        if (it + 1 < ntiles) fetch(REVERSE ? tile - 1 : tile + 1);
#pragma unroll 2
        for (int e = 0; e < n; ++e) {
            const int t = REVERSE ? n - 1 - e : e;
            const Octet q = read_octet(sQ[buf][t], ti), d = read_octet(sD[buf][t], ti);
            f2 x[8];
            read_dup8(sX[buf][t], tj, x);
            if constexpr (!SUMMARY) {
                const Octet p = read_octet(sP[buf][t], ti);
                float acc[8];
#pragma unroll
                for (int b = 0; b < 8; ++b) {
                    f2 y2 = f2_mul(p.p[0], S[0][b]);
                    y2 = f2_fma(p.p[1], S[1][b], y2);
                    y2 = f2_fma(p.p[2], S[2][b], y2);
                    y2 = f2_fma(p.p[3], S[3][b], y2);
                    const float2 y = f2_unpack(y2);
                    acc[b] = y.x + y.y;
                }
                const float y = scatter_sum8(acc, lane);
                gO[(size_t)(tile * TT + t) * a.q.ld] = cast_out<Ty>(fmaf(sX[buf][t][jout], sC[buf][t], y));
            }
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int b = 0; b < 8; ++b) S[p][b] = f2_fma(S[p][b], d.p[p], f2_mul(q.p[p], x[b]));
        }
    }

    if (SUMMARY) {
        // decays: eight threads per channel chunk (one per staged row) hold partial sums of exp(w)
        __syncthreads();
        put8(sD[0][row], chunk, dsum);
        __syncthreads();
        float t = 0.f;
#pragma unroll
        for (int e = 0; e < TT; ++e) t += sD[0][e][tid];
        a.dec_out[s.seq * 64 + tid] = -t * 1.4426950408889634f;
    }
    void *so = SUMMARY ? (void *)a.b_out : a.s_out;
    if (so != nullptr) {
        const int dt = SUMMARY ? (int)WKV6_F32 : a.s_dtype;
        const bool vec = SUMMARY || a.vec_out;
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const float2 v0 = f2_unpack(S[p][4 * half]), v1 = f2_unpack(S[p][4 * half + 1]);
                const float2 v2 = f2_unpack(S[p][4 * half + 2]), v3 = f2_unpack(S[p][4 * half + 3]);
                const size_t o = s.seq * 4096 + (size_t)tile_index(ti, 2 * p) * 64 + 32 * half + 4 * tj;
                if (vec) {
                    float *f = static_cast<float *>(so) + o;
                    *reinterpret_cast<float4 *>(f) = make_float4(v0.x, v1.x, v2.x, v3.x);
                    *reinterpret_cast<float4 *>(f + 64) = make_float4(v0.y, v1.y, v2.y, v3.y);
                } else {
                    store_any(so, dt, o, v0.x); store_any(so, dt, o + 1, v1.x); store_any(so, dt, o + 2, v2.x); store_any(so, dt, o + 3, v3.x);
                    store_any(so, dt, o + 64, v0.y); store_any(so, dt, o + 65, v1.y); store_any(so, dt, o + 66, v2.y); store_any(so, dt, o + 67, v3.y);
                }
            }
    }
}

struct StepBwdArgs {
    const void *r, *k, *v, *w, *gy, *u;
    void *gr, *gk, *gv, *gw;
    void *gu;                    // [B*G,H,64] of gu_dtype
    float *x;                    // fp32 [B,T,H*64] dense: r * gr, written by the gr sweep, read by the other one
    const float *s_in, *a_in;    // G > 1: entering states [B*G,H,64,64] of the forward and the reverse walk
    int u_dtype, gu_dtype;
    StepGeom q;
};

// gr_t[i] = sum_j S[i][j] gy_t[j] + u_i k_t[i] (v_t . gy_t),  then S[i][j] = d_t[i] S[i][j] + k_t[i] v_t[j].
template <typename Tx, typename Ty>
__global__ void __launch_bounds__(kStepThreads) step_gr_kernel(const StepBwdArgs a) {
    constexpr int TT = kStepTile;
    __shared__ __align__(16) float sR[2][TT][64];
    __shared__ __align__(16) float sK[2][TT][64];
    __shared__ __align__(16) float sD[2][TT][64];
    __shared__ __align__(16) float sV[2][TT][64];
    __shared__ __align__(16) float sG[2][TT][64];
    __shared__ float sVG[2][TT];

    const StepSeg s = step_segment(a.q, blockIdx.x);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ti = warp * 4 + (lane & 3), tj = lane >> 2;   // the sum over j stays inside a warp
    const int row = tid >> 3, chunk = tid & 7;
    const Tx *gR = static_cast<const Tx *>(a.r) + s.base + chunk * 8;
    const Tx *gK = static_cast<const Tx *>(a.k) + s.base + chunk * 8;
    const Tx *gV = static_cast<const Tx *>(a.v) + s.base + chunk * 8;
    const Tx *gW = static_cast<const Tx *>(a.w) + s.base + chunk * 8;
    const Ty *gG = static_cast<const Ty *>(a.gy) + s.base + chunk * 8;
    const int iout = tile_index(ti, tj);
    const float ui = load_any(a.u, a.u_dtype, (size_t)s.h * 64 + iout);
    Ty *gO = static_cast<Ty *>(a.gr) + s.base + iout;
    const size_t xld = (size_t)a.q.H * 64;
    float *gX = a.x + ((size_t)s.b * a.q.T + s.t0) * xld + (size_t)s.h * 64 + iout;

    f2 S[4][8];
    if (a.s_in != nullptr) load_tile(a.s_in + s.seq * 4096, ti, tj, S);
    else zero_tile(S);
    float gu = 0.f;

    Raw8<Tx> fR, fK, fV, fW;
    Raw8<Ty> fG;
    auto fetch = [&](int tile) {
        const int t = tile * TT + row;
        if (t < s.cnt) {
            const size_t o = (size_t)t * a.q.ld;
            fR.load(gR + o); fK.load(gK + o); fV.load(gV + o); fW.load(gW + o); fG.load(gG + o);
        } else {
            fR.zero(); fK.zero(); fV.zero(); fW.zero(); fG.zero();
        }
    };
    const int ntiles = (s.cnt + TT - 1) / TT;
    fetch(0);
    for (int it = 0; it < ntiles; ++it) {
        const int buf = it & 1, n = min(TT, s.cnt - it * TT);
        {
            float f[8], g[8], c = 0.f;
            fR.get(f); put8(sR[buf][row], chunk, f);
            fK.get(f); put8(sK[buf][row], chunk, f);
            fW.get(f);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = expf(-expf(f[e]));
            put8(sD[buf][row], chunk, f);
            fV.get(f); put8(sV[buf][row], chunk, f);
            fG.get(g); put8(sG[buf][row], chunk, g);
#pragma unroll
            for (int e = 0; e < 8; ++e) c = fmaf(f[e], g[e], c);
            c = row_sum8(c);
            if (chunk == 0) sVG[buf][row] = c;
        }
        __syncthreads();
        if (it + 1 < ntiles) fetch(it + 1);
#pragma unroll 2
        for (int t = 0; t < n; ++t) {
            const Octet k = read_octet(sK[buf][t], ti), d = read_octet(sD[buf][t], ti);
            f2 x[8], g[8], o2[4];
            read_dup8(sV[buf][t], tj, x);
            read_dup8(sG[buf][t], tj, g);
            float acc[8];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                o2[p] = f2_mul(S[p][0], g[0]);
#pragma unroll
                for (int b = 1; b < 8; ++b) o2[p] = f2_fma(S[p][b], g[b], o2[p]);
                const float2 o = f2_unpack(o2[p]);
                acc[2 * p] = o.x; acc[2 * p + 1] = o.y;
            }
            const float sum = scatter_sum8(acc, lane);
            const float vg = sVG[buf][t], ki = sK[buf][t][iout], ri = sR[buf][t][iout];
            const float gr = fmaf(ui * ki, vg, sum);
            const size_t tt = (size_t)(it * TT + t);
            gO[tt * a.q.ld] = cast_out<Ty>(gr);
            gX[tt * xld] = ri * gr;
            gu = fmaf(ri * ki, vg, gu);
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int b = 0; b < 8; ++b) S[p][b] = f2_fma(S[p][b], d.p[p], f2_mul(k.p[p], x[b]));
        }
    }
    store_any(a.gu, a.gu_dtype, s.seq * 64 + iout, gu);
}

// gk_t[i] = sum_j A[i][j] v_t[j] + u_i r_t[i] (v_t . gy_t),  gv_t[j] = sum_i A[i][j] k_t[i] + gy_t[j] sum_i u_i r_t[i] k_t[i],
// gw_t[i] = -exp(w_t[i]) (Z_t[i] - k_t[i] sum_j A[i][j] v_t[j]),  then A[i][j] = d_t[i] A[i][j] + r_t[i] gy_t[j].
// Z runs in double along the segment (Z_{t-1} = Z_t + r_t gr_t - k_t gk_t) and starts at sum_j S A of the segment's end.
template <typename Tx, typename Ty>
__global__ void __launch_bounds__(kStepThreads) step_gkvw_kernel(const StepBwdArgs a) {
    constexpr int TT = kStepTile;
    __shared__ __align__(16) float sR[2][TT][64];
    __shared__ __align__(16) float sK[2][TT][64];
    __shared__ __align__(16) float sD[2][TT][64];
    __shared__ __align__(16) float sE[2][TT][64];
    __shared__ __align__(16) float sV[2][TT][64];
    __shared__ __align__(16) float sG[2][TT][64];
    __shared__ __align__(16) float sX[2][TT][64];
    __shared__ __align__(16) float sO[2][TT][64];    // [warp][step][i]: the two warps' halves of sum_j A v
    __shared__ float sVG[2][TT], sC[2][TT];

    const StepSeg s = step_segment(a.q, blockIdx.x);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ti = lane >> 2, tj = warp * 4 + (lane & 3);
    const int row = tid >> 3, chunk = tid & 7;
    const Tx *gR = static_cast<const Tx *>(a.r) + s.base + chunk * 8;
    const Tx *gK = static_cast<const Tx *>(a.k) + s.base + chunk * 8;
    const Tx *gV = static_cast<const Tx *>(a.v) + s.base + chunk * 8;
    const Tx *gW = static_cast<const Tx *>(a.w) + s.base + chunk * 8;
    const Ty *gG = static_cast<const Ty *>(a.gy) + s.base + chunk * 8;
    const int jout = tile_index(tj, ti);
    Ty *oV = static_cast<Ty *>(a.gv) + s.base + jout;
    Ty *oK = static_cast<Ty *>(a.gk) + s.base + tid;
    Ty *oW = static_cast<Ty *>(a.gw) + s.base + tid;
    const size_t xld = (size_t)a.q.H * 64;
    const float *gX = a.x + ((size_t)s.b * a.q.T + s.t0) * xld + (size_t)s.h * 64 + chunk * 8;

    float u8[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) u8[e] = load_any(a.u, a.u_dtype, (size_t)s.h * 64 + chunk * 8 + e);
    const float ui = load_any(a.u, a.u_dtype, (size_t)s.h * 64 + tid);

    f2 A[4][8];
    double z = 0.0;
    if (a.a_in != nullptr) {
        load_tile(a.a_in + s.seq * 4096, ti, tj, A);
        if (s.g + 1 < a.q.G) {
            const float4 *sr = reinterpret_cast<const float4 *>(a.s_in + (s.seq + a.q.H) * 4096 + (size_t)tid * 64);
            const float4 *ar = reinterpret_cast<const float4 *>(a.a_in + s.seq * 4096 + (size_t)tid * 64);
#pragma unroll 4
            for (int e = 0; e < 16; ++e) {
                const float4 p = sr[e], q = ar[e];
                z += (double)p.x * (double)q.x + (double)p.y * (double)q.y + (double)p.z * (double)q.z + (double)p.w * (double)q.w;
            }
        }
    } else {
        zero_tile(A);
    }

    Raw8<Tx> fR, fK, fV, fW;
    Raw8<Ty> fG;
    float4 fX[2];
    auto fetch = [&](int tile) {
        const int t = tile * TT + row;
        if (t < s.cnt) {
            const size_t o = (size_t)t * a.q.ld;
            fR.load(gR + o); fK.load(gK + o); fV.load(gV + o); fW.load(gW + o); fG.load(gG + o);
            // x may lie in the gw buffer (fp32, dense), which this CTA overwrites a tile after reading it: ordinary loads
            fX[0] = *reinterpret_cast<const float4 *>(gX + (size_t)t * xld);
            fX[1] = *reinterpret_cast<const float4 *>(gX + (size_t)t * xld + 4);
        } else {
            fR.zero(); fK.zero(); fV.zero(); fW.zero(); fG.zero();
            fX[0] = fX[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    const int ntiles = (s.cnt + TT - 1) / TT;
    fetch(ntiles - 1);
    for (int it = 0; it < ntiles; ++it) {
        const int tile = ntiles - 1 - it, buf = it & 1, n = min(TT, s.cnt - tile * TT);
        {
            float f[8], g[8], c = 0.f, vg = 0.f;
            fR.get(f); put8(sR[buf][row], chunk, f);
            fK.get(g); put8(sK[buf][row], chunk, g);
#pragma unroll
            for (int e = 0; e < 8; ++e) c = fmaf(u8[e] * f[e], g[e], c);
            fW.get(f);
#pragma unroll
            for (int e = 0; e < 8; ++e) { f[e] = expf(f[e]); g[e] = expf(-f[e]); }
            put8(sE[buf][row], chunk, f);
            put8(sD[buf][row], chunk, g);
            fV.get(f); put8(sV[buf][row], chunk, f);
            fG.get(g); put8(sG[buf][row], chunk, g);
            reinterpret_cast<float4 *>(sX[buf][row])[2 * chunk] = fX[0];
            reinterpret_cast<float4 *>(sX[buf][row])[2 * chunk + 1] = fX[1];
#pragma unroll
            for (int e = 0; e < 8; ++e) vg = fmaf(f[e], g[e], vg);
            c = row_sum8(c);
            vg = row_sum8(vg);
            if (chunk == 0) { sC[buf][row] = c; sVG[buf][row] = vg; }
        }
        __syncthreads();
        if (it + 1 < ntiles) fetch(tile - 1);
#pragma unroll 2
        for (int e = 0; e < n; ++e) {
            const int t = n - 1 - e;
            const Octet r = read_octet(sR[buf][t], ti), k = read_octet(sK[buf][t], ti), d = read_octet(sD[buf][t], ti);
            f2 v[8], g[8];
            read_dup8(sV[buf][t], tj, v);
            read_dup8(sG[buf][t], tj, g);
            float acc[8], ok[8];
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                f2 y2 = f2_mul(k.p[0], A[0][b]);
                y2 = f2_fma(k.p[1], A[1][b], y2);
                y2 = f2_fma(k.p[2], A[2][b], y2);
                y2 = f2_fma(k.p[3], A[3][b], y2);
                const float2 y = f2_unpack(y2);
                acc[b] = y.x + y.y;
            }
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                f2 o2 = f2_mul(A[p][0], v[0]);
#pragma unroll
                for (int b = 1; b < 8; ++b) o2 = f2_fma(A[p][b], v[b], o2);
                const float2 o = f2_unpack(o2);
                ok[2 * p] = o.x; ok[2 * p + 1] = o.y;
#pragma unroll
                for (int b = 0; b < 8; ++b) A[p][b] = f2_fma(A[p][b], d.p[p], f2_mul(r.p[p], g[b]));
            }
            const float gv = scatter_sum8(acc, lane);
            oV[(size_t)(tile * TT + t) * a.q.ld] = cast_out<Ty>(fmaf(sG[buf][t][jout], sC[buf][t], gv));
            // sum over the four lanes with this ti (the other half of j is in the other warp): two values per lane
            const bool h2 = lane & 2, h1 = lane & 1;
            float b4[4], c2[2];
#pragma unroll
            for (int m = 0; m < 4; ++m) b4[m] = (h2 ? ok[m + 4] : ok[m]) + __shfl_xor_sync(0xffffffffu, h2 ? ok[m] : ok[m + 4], 2);
#pragma unroll
            for (int m = 0; m < 2; ++m) c2[m] = (h1 ? b4[m + 2] : b4[m]) + __shfl_xor_sync(0xffffffffu, h1 ? b4[m] : b4[m + 2], 1);
            *reinterpret_cast<float2 *>(&sO[warp][t][tile_index(ti, 2 * (lane & 1) + 4 * ((lane >> 1) & 1))]) = make_float2(c2[0], c2[1]);
        }
        __syncthreads();
#pragma unroll
        for (int t = TT - 1; t >= 0; --t) {
            if (t < n) {
                const float acc = sO[0][t][tid] + sO[1][t][tid], ki = sK[buf][t][tid];
                const float gk = fmaf(ui * sR[buf][t][tid], sVG[buf][t], acc);
                const float core = (float)(z - (double)ki * (double)acc);
                const size_t o = (size_t)(tile * TT + t) * a.q.ld;
                oK[o] = cast_out<Ty>(gk);
                // the state before the first step of the sequence is zero: its gw is exactly 0
                oW[o] = cast_out<Ty>((s.t0 + tile * TT + t == 0) ? 0.f : -sE[buf][t][tid] * core);
                z += (double)sX[buf][t][tid] - (double)ki * (double)gk;
            }
        }
    }
}

}  // namespace wkv6
