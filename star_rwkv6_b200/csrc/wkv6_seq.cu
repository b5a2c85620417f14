// Host side of the sequential variant: argument packing, dtype / head-size dispatch, launches.
// Head size 64 runs the register-tile kernels of wkv6_step.cuh, smaller heads those of wkv6_seq.cuh.  So does the backward of
// fp16 inputs at any head size: its results are rounded to fp16 by the operator, where another order of the same fp32 sums
// moves one value in a few hundred by a last bit (2^-10), ten times what the fp32 results differ by anywhere; callers keep
// the bits they have.
#include "wkv6_internal.h"
#include "wkv6_seq.cuh"
#include "wkv6_step.cuh"

namespace wkv6 {

// ---- sequential variant -------------------------------------------------------------------------

template <typename Tx, typename TX, typename Ty, int N, bool REV>
static int launch_col(const SeqColArgs &a, cudaStream_t st) {
    seq_col_kernel<Tx, TX, Ty, N, REV><<<a.B * a.H, 4 * N, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "seq_col_kernel launch");
}

template <typename Tx, typename Ty, int N, int MODE>
static int launch_row(const SeqRowArgs &a, cudaStream_t st) {
    constexpr int smem = seq_row_smem_bytes<N>();
    auto kern = seq_row_kernel<Tx, Ty, N, MODE>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(seq_row_kernel)");
    }
    kern<<<a.B * a.H, 4 * N, smem, st>>>(a);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, "seq_row_kernel launch");
}

template <typename Tx, typename Ty, int N>
static int seq_forward_t(const SeqColArgs &a, cudaStream_t st) {
    return launch_col<Tx, Tx, Ty, N, false>(a, st);
}

template <typename Tx, typename Ty, int N>
static int seq_backward_t(const SeqRowArgs &ra, const SeqColArgs &ca, void *gk, cudaStream_t st) {
    int rc = launch_row<Tx, Ty, N, 0>(ra, st);  // gr, gu, x
    if (rc) return rc;
    SeqRowArgs rb = ra;
    rb.out = gk;
    rc = launch_row<Tx, Ty, N, 1>(rb, st);      // gk, gw
    if (rc) return rc;
    return launch_col<Tx, Ty, Ty, N, true>(ca, st);
}

#define WKV6_DISPATCH_N(N_, Tx, Ty, CALL)                    \
    switch (N_) {                                            \
        case 8: { constexpr int kN = 8; return CALL(Tx, Ty, kN); }   \
        case 16: { constexpr int kN = 16; return CALL(Tx, Ty, kN); } \
        default: { constexpr int kN = 32; return CALL(Tx, Ty, kN); } \
    }
static bool register_tiles(const wkv6_problem *p, bool backward) { return p->N == 64 && !(backward && p->x_dtype == WKV6_F16); }

#define WKV6_DISPATCH(p, CALL)                                                                   \
    do {                                                                                         \
        if ((p)->x_dtype == WKV6_F32) { WKV6_DISPATCH_N((p)->N, float, float, CALL) }            \
        else if ((p)->x_dtype == WKV6_F16) { WKV6_DISPATCH_N((p)->N, __half, float, CALL) }      \
        else if ((p)->y_dtype == WKV6_BF16) { WKV6_DISPATCH_N((p)->N, __nv_bfloat16, __nv_bfloat16, CALL) } \
        else { WKV6_DISPATCH_N((p)->N, __nv_bfloat16, float, CALL) }                             \
    } while (0)

// ---- head size 64: register tiles, optionally split along T ---------------------------------------------------------

#define WKV6_DISPATCH_TYPES(p, CALL)                                                 \
    do {                                                                             \
        if ((p)->x_dtype == WKV6_F32) CALL(float, float);                            \
        else if ((p)->x_dtype == WKV6_F16) CALL(__half, float);                      \
        else if ((p)->y_dtype == WKV6_BF16) CALL(__nv_bfloat16, __nv_bfloat16);      \
        else CALL(__nv_bfloat16, float);                                             \
    } while (0)

#define WKV6_DISPATCH_TYPES_NO_F16(p, CALL)                                          \
    do {                                                                             \
        if ((p)->x_dtype == WKV6_F32) CALL(float, float);                            \
        else if ((p)->y_dtype == WKV6_BF16) CALL(__nv_bfloat16, __nv_bfloat16);      \
        else CALL(__nv_bfloat16, float);                                             \
    } while (0)

static StepGeom step_geom(const wkv6_problem *p, const Dims &d, int G, int L) {
    return StepGeom{p->B, p->T, p->H, G, L, d.ld, d.bs};
}

static int launched(const char *what) {
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WKV6_OK : cuda_fail(e, what);
}

static StepFwdArgs step_fwd_args(const wkv6_problem *p, const StepGeom &q) {
    StepFwdArgs a{};
    a.u_dtype = p->u_dtype; a.s_dtype = p->s_dtype; a.q = q; a.skip_g = -1;
    return a;
}

static int step_forward(const wkv6_problem *p, const StepFwdArgs &a, cudaStream_t st) {
    const unsigned grid = (unsigned)(p->B * a.q.G * p->H);
#define CALL_FWD(Tx, Ty) step_fwd_kernel<Tx, Tx, Ty, false, false><<<grid, kStepThreads, 0, st>>>(a)
    WKV6_DISPATCH_TYPES(p, CALL_FWD);
#undef CALL_FWD
    return launched("step_fwd_kernel launch");
}

static int step_summary(const wkv6_problem *p, const StepFwdArgs &a, bool reverse, cudaStream_t st) {
    const unsigned grid = (unsigned)(p->B * a.q.G * p->H);
    if (reverse) {
#define CALL_SUM(Tx, Ty) step_fwd_kernel<Tx, Ty, Ty, true, true><<<grid, kStepThreads, 0, st>>>(a)
        WKV6_DISPATCH_TYPES_NO_F16(p, CALL_SUM);
#undef CALL_SUM
    } else {
#define CALL_SUM(Tx, Ty) step_fwd_kernel<Tx, Tx, Ty, true, false><<<grid, kStepThreads, 0, st>>>(a)
        WKV6_DISPATCH_TYPES(p, CALL_SUM);
#undef CALL_SUM
    }
    return launched("step_fwd_kernel (summary) launch");
}

static int step_backward(const wkv6_problem *p, const StepBwdArgs &a, cudaStream_t st) {
    const unsigned grid = (unsigned)(p->B * a.q.G * p->H);
#define CALL_GR(Tx, Ty) step_gr_kernel<Tx, Ty><<<grid, kStepThreads, 0, st>>>(a)
    WKV6_DISPATCH_TYPES_NO_F16(p, CALL_GR);
#undef CALL_GR
    if (int rc = launched("step_gr_kernel launch")) return rc;
#define CALL_GKVW(Tx, Ty) step_gkvw_kernel<Tx, Ty><<<grid, kStepThreads, 0, st>>>(a)
    WKV6_DISPATCH_TYPES_NO_F16(p, CALL_GKVW);
#undef CALL_GKVW
    return launched("step_gkvw_kernel launch");
}

static StepBwdArgs step_bwd_args(const wkv6_problem *p, const StepGeom &q, const void *r, const void *k, const void *v,
                                 const void *w, const void *u, const void *gy, void *gr, void *gk, void *gv, void *gw, void *gu,
                                 float *x) {
    StepBwdArgs a{};
    a.r = r; a.k = k; a.v = v; a.w = w; a.gy = gy; a.u = u; a.gr = gr; a.gk = gk; a.gv = gv; a.gw = gw; a.gu = gu; a.x = x;
    a.u_dtype = p->u_dtype; a.gu_dtype = p->gu_dtype; a.q = q;
    return a;
}

// Segments of the split path.  A CTA of the register-tile kernels is two warps and four of them fill an SM's issue slots
// (six or eight measured slower); the count is rounded down so that every SM gets the same number.  Above one and a half CTAs
// per SM the chip idles less than the summaries (two of the forward's three multiply-adds) would cost.  A segment keeps at
// least 32 steps: shorter ones move more state than input.  Below 96 steps the chain saved (0.25 us a step and sweep) is no
// more than the summary and scan launches (B2 T64 H2: 92 us in one piece, 111 us in two).
int seq_split_segments(const wkv6_problem *p) {
    constexpr int kMinSteps = 32;
    const int64_t seqs = (int64_t)p->B * p->H;
    const int sms = sm_count();
    if (p->N != 64 || seqs == 0 || 2 * seqs > 3 * sms || p->T < 3 * kMinSteps) return 1;
    const int64_t want = 4 * sms / seqs, most = p->T / kMinSteps;
    const int64_t n = want < most ? want : most;
    const int L = seq_segment_length(p->T, (int)n);
    return (p->T + L - 1) / L;
}

int seq_segment_length(int T, int G) {   // multiple of the staging tile, equal pieces but for the last
    const int L = (T + G - 1) / G;
    return (L + kStepTile - 1) / kStepTile * kStepTile;
}

static size_t seg_states(const wkv6_problem *p, int G) { return (size_t)p->B * G * p->H * 4096; }

size_t seq_split_state_bytes(const wkv6_problem *p, int G) { return seg_states(p, G) * sizeof(float); }

// forward: b, dec; backward: b, dec, reverse entering states and, where gw cannot hold it, x
size_t seq_split_workspace(const wkv6_problem *p, const Dims &d, int G, bool backward) {
    const size_t n = seg_states(p, G);
    return sizeof(float) * (n + n / 64 + (backward ? n : 0)) + (backward ? seq_backward_workspace(p, d) : 0);
}

int seq_forward_split(const wkv6_problem *p, const Dims &d, int G, const void *r, const void *k, const void *v, const void *w,
                      const void *u, void *y, const void *s_in, const int64_t *s_map, int s_kinds, void *s_out, float *states,
                      float *ws, cudaStream_t st) {
    const size_t n = seg_states(p, G);
    const StepGeom q = step_geom(p, d, G, seq_segment_length(p->T, G));
    StepFwdArgs a = step_fwd_args(p, q);
    a.Q = k; a.W = w; a.X = v; a.b_out = ws; a.dec_out = ws + n; a.skip_g = s_out == nullptr ? G - 1 : -1;
    int rc = step_summary(p, a, false, st);
    if (rc) return rc;
    rc = state_scan(p->B, p->H, G, a.dec_out, a.b_out, s_in, s_map, s_kinds, p->s_dtype, states, s_out, p->s_dtype, false, st);
    if (rc) return rc;
    a = step_fwd_args(p, q);
    a.P = r; a.Q = k; a.W = w; a.X = v; a.u = u; a.out = y; a.seg_in = states;
    return step_forward(p, a, st);
}

int seq_backward_split(const wkv6_problem *p, const Dims &d, int G, const void *r, const void *k, const void *v, const void *w,
                       const void *u, const void *gy, void *gr, void *gk, void *gv, void *gw, float *gu, const float *states,
                       float *ws, cudaStream_t st) {
    if (!register_tiles(p, true)) return fail(WKV6_ERR_UNSUPPORTED, "the backward of fp16 inputs is not split");
    const size_t n = seg_states(p, G);
    const StepGeom q = step_geom(p, d, G, seq_segment_length(p->T, G));
    float *a_in = ws + n + n / 64;
    StepFwdArgs s = step_fwd_args(p, q);
    s.Q = r; s.W = w; s.X = gy; s.b_out = ws; s.dec_out = ws + n; s.skip_g = 0;
    int rc = step_summary(p, s, true, st);
    if (rc) return rc;
    rc = state_scan(p->B, p->H, G, s.dec_out, s.b_out, nullptr, nullptr, 0, WKV6_F32, a_in, nullptr, WKV6_F32, true, st);
    if (rc) return rc;
    float *x = seq_backward_workspace(p, d) ? a_in + n : static_cast<float *>(gw);
    StepBwdArgs a = step_bwd_args(p, q, r, k, v, w, u, gy, gr, gk, gv, gw, gu, x);
    a.s_in = states; a.a_in = a_in;
    return step_backward(p, a, st);
}

int seq_forward(const wkv6_problem *p, const Dims &d, const void *r, const void *k, const void *v,
                       const void *w, const void *u, void *y, const void *s_in, const int64_t *s_map,
                       int s_kinds, void *s_out, cudaStream_t st) {
    if (register_tiles(p, false)) {
        StepFwdArgs a = step_fwd_args(p, step_geom(p, d, 1, p->T));
        a.P = r; a.Q = k; a.W = w; a.X = v; a.u = u; a.out = y;
        a.s_in = s_in; a.s_map = s_map; a.s_kinds = s_kinds; a.s_out = s_out;
        a.vec_in = p->s_dtype == WKV6_F32 && aligned16(s_in);
        a.vec_out = p->s_dtype == WKV6_F32 && aligned16(s_out);
        return step_forward(p, a, st);
    }
    SeqColArgs a{};
    a.P = r; a.Q = k; a.W = w; a.X = v; a.u = u; a.out = y;
    a.s_in = s_in; a.s_map = s_map; a.s_out = s_out; a.s_kinds = s_kinds; a.s_dtype = p->s_dtype;
    a.u_dtype = p->u_dtype; a.B = p->B; a.T = p->T; a.H = p->H; a.ld = d.ld; a.bs = d.bs;
#define CALL_FWD(Tx, Ty, kN) seq_forward_t<Tx, Ty, kN>(a, st)
    WKV6_DISPATCH(p, CALL_FWD);
#undef CALL_FWD
}

size_t seq_backward_workspace(const wkv6_problem *p, const Dims &d) {
    if (p->y_dtype == WKV6_F32 && d.dense) return 0;  // x = r*gr is staged in the gw buffer itself
    return (size_t)p->B * p->T * d.C * sizeof(float);
}

int seq_backward(const wkv6_problem *p, const Dims &d, const void *r, const void *k, const void *v,
                        const void *w, const void *u, const void *gy, void *gr, void *gk, void *gv, void *gw,
                        void *gu, void *ws, size_t ws_bytes, cudaStream_t st) {
    const size_t need = seq_backward_workspace(p, d);
    if (need > 0 && (ws == nullptr || ws_bytes < need))
        return fail(WKV6_ERR_WORKSPACE, "backward workspace: need %zu bytes, got %zu", need, ws ? ws_bytes : (size_t)0);
    if (register_tiles(p, true))
        return step_backward(p, step_bwd_args(p, step_geom(p, d, 1, p->T), r, k, v, w, u, gy, gr, gk, gv, gw, gu,
                                              need ? static_cast<float *>(ws) : static_cast<float *>(gw)), st);
    SeqRowArgs ra{};
    ra.r = r; ra.k = k; ra.w = w; ra.v = v; ra.gy = gy; ra.u = u; ra.out = gr; ra.gw = gw; ra.gu = gu;
    ra.x = need ? static_cast<float *>(ws) : static_cast<float *>(gw);
    ra.u_dtype = p->u_dtype; ra.gu_dtype = p->gu_dtype; ra.B = p->B; ra.T = p->T; ra.H = p->H; ra.ld = d.ld; ra.bs = d.bs;
    SeqColArgs ca{};
    ca.P = k; ca.Q = r; ca.W = w; ca.X = gy; ca.u = u; ca.out = gv; ca.u_dtype = p->u_dtype;
    ca.s_dtype = WKV6_F32; ca.B = p->B; ca.T = p->T; ca.H = p->H; ca.ld = d.ld; ca.bs = d.bs;
#define CALL_BWD(Tx, Ty, kN) seq_backward_t<Tx, Ty, kN>(ra, ca, gk, st)
    if (p->N == 64) return CALL_BWD(__half, float, 64);
    WKV6_DISPATCH(p, CALL_BWD);
#undef CALL_BWD
}

}  // namespace wkv6
