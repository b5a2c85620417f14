// Declarations shared by the translation units of the library (not part of the public ABI).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/wkv6_b200.h"

namespace wkv6 {

struct Dims {
    int64_t C;    // H*N
    int64_t ld;   // resolved row stride (elements)
    int64_t bs;   // resolved batch stride (elements)
    bool dense;   // ld == C and bs == T*C
};

int sm_count();   // of the current device
inline bool aligned16(const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }
int fail(int code, const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *what);
size_t dtype_size(int dt);
int validate(const wkv6_problem *p, Dims *d);

// sequential variant (wkv6_seq.cu)
int seq_forward(const wkv6_problem *p, const Dims &d, const void *r, const void *k, const void *v, const void *w,
                const void *u, void *y, const void *s_in, const int64_t *s_map, int s_kinds, void *s_out,
                cudaStream_t st);
size_t seq_backward_workspace(const wkv6_problem *p, const Dims &d);
int seq_backward(const wkv6_problem *p, const Dims &d, const void *r, const void *k, const void *v, const void *w,
                 const void *u, const void *gy, void *gr, void *gk, void *gv, void *gw, void *gu, void *ws,
                 size_t ws_bytes, cudaStream_t st);
// the same split along T into G segments (head size 64): entering states left by the forward for the backward in `states`
int seq_split_segments(const wkv6_problem *p);
int seq_segment_length(int T, int G);
size_t seq_split_state_bytes(const wkv6_problem *p, int G);
size_t seq_split_workspace(const wkv6_problem *p, const Dims &d, int G, bool backward);
int seq_forward_split(const wkv6_problem *p, const Dims &d, int G, const void *r, const void *k, const void *v, const void *w,
                      const void *u, void *y, const void *s_in, const int64_t *s_map, int s_kinds, void *s_out, float *states,
                      float *ws, cudaStream_t st);
int seq_backward_split(const wkv6_problem *p, const Dims &d, int G, const void *r, const void *k, const void *v, const void *w,
                       const void *u, const void *gy, void *gr, void *gk, void *gv, void *gw, float *gu, const float *states,
                       float *ws, cudaStream_t st);

// chunked tensor-core variant (wkv6_chunk.cu)
bool chunk_supported(const wkv6_problem *p);
int chunk_status();
int chunk_debug_inject(int skip_load_chunk, long long wait_limit_ms);
size_t chunk_ckpt_bytes(const wkv6_problem *p);
int chunk_sum_rows(const float *in, int64_t rows, int64_t n, float *out, cudaStream_t st);
size_t chunk_backward_workspace(const wkv6_problem *p, const Dims &d, int have_ckpt);
int chunk_forward(const wkv6_problem *p, const Dims &d, const void *r, const void *k, const void *v, const void *w,
                  const void *u, void *y, const void *s_in, const int64_t *s_map, int s_kinds, void *s_out,
                  void *ckpt, cudaStream_t st);
int chunk_backward(const wkv6_problem *p, const Dims &d, const void *r, const void *k, const void *v, const void *w,
                   const void *u, const void *gy, void *gr, void *gk, void *gv, void *gw, void *gu, const void *ckpt,
                   void *ws, size_t ws_bytes, cudaStream_t st);

int chunk_backward_seeded(const wkv6_problem *p, const Dims &d, const void *r, const void *k, const void *v,
                          const void *w, const void *u, const void *gy, void *gr, void *gk, void *gv, void *gw,
                          void *gu, const void *ckpt, const float *ab_in, void *ws, size_t ws_bytes, cudaStream_t st);
int chunk_segment_summary(const wkv6_problem *p, const Dims &d, const void *x1, const void *x2, const void *w,
                          bool reverse, float *b_out, float *dec_log2_out, int skip_mod, int skip_rem, cudaStream_t st);
int state_scan(int B, int H, int G, const float *dec, const float *bsum, const void *s0, const int64_t *s_map, int s_kinds,
               int s_dtype, float *out, void *last, int last_dtype, bool reverse, cudaStream_t st);
// Sequences cut along T into G segments, for problems that leave SMs idle otherwise (1: not cut).
int chunk_split_segments(const wkv6_problem *p);
size_t chunk_split_workspace(const wkv6_problem *p, bool backward);
int chunk_forward_split(const wkv6_problem *p, const Dims &d, const void *r, const void *k, const void *v, const void *w,
                        const void *u, void *y, const void *s_in, const int64_t *s_map, int s_kinds, void *s_out, void *ckpt,
                        float *ws, cudaStream_t st);
int chunk_backward_split(const wkv6_problem *p, const Dims &d, const void *r, const void *k, const void *v, const void *w,
                         const void *u, const void *gy, void *gr, void *gk, void *gv, void *gw, float *gu_rows, const void *ckpt,
                         float *ws, cudaStream_t st);
int resolve_variant(const wkv6_problem *p);

}  // namespace wkv6
