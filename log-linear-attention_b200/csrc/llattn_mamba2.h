// Internal launch parameters shared by the log-linear Mamba-2 kernels.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>

#include "../../include/llattn.h"

namespace llattn {

constexpr int M2_MLOW = 3;   // a segment is 2^M2_MLOW chunks (512 tokens)
constexpr int M2_MAX_LH = 10;   // segment levels held by the per-level scans over segments (T <= 512 * 2^10)
constexpr int M2_MAX_L_TC = 20;   // lambda levels that the tcgen05 kernels' tables hold; more go to the warp-level kernels

struct Mamba2Params {
    // tensor maps (64-column panels, 128 rows) for the tcgen05 kernels; valid only when those run
    alignas(64) CUtensorMap tm_q, tm_k, tm_v, tm_do, tm_x, tm_y;
    alignas(64) CUtensorMap tm_h0;             // level states of the segments as a (B*H*NS*LH*K, V) matrix
    alignas(64) CUtensorMap tm_lo;             // level states inside the segments as a (B*H*ceil(NT/2)*K, V) matrix
    alignas(64) CUtensorMap tm_lo_a, tm_dh, tm_df;   // gradients of the pairs' and of the segments' summaries, what the readers of a segment send back
    alignas(64) CUtensorMap tm_dv;
    alignas(64) CUtensorMap tm_dq, tm_dk;      // fp32 (B*T, G, K) accumulators, 32-column boxes (reduce-add); or the bf16 gradients
    // inputs
    const __nv_bfloat16* q;      // (B,T,G,K)
    const __nv_bfloat16* k;      // (B,T,G,K)
    const __nv_bfloat16* v;      // (B,T,H,V)
    const float* g;              // (B,T,H) raw log decay
    const float* cum_in;         // (B,T,H) backward: the forward call's g_cum, for level states that are made again (null: from g)
    const __nv_bfloat16* l;      // (B,T,H,L)
    const __nv_bfloat16* d_o;    // (B,T,H,V) upstream gradient (backward only)
    // outputs
    __nv_bfloat16* o;            // (B,T,H,V)
    float* g_cum;                // (B,T,H) in-chunk inclusive cumsum of g
    float* dq_acc;               // (B,T,G,K) fp32 accumulators (backward)
    float* dk_acc;               // (B,T,G,K)
    __nv_bfloat16 *dq_out, *dk_out;   // (B,T,G,K) the gradients themselves, where a CTA has all heads of a group (null: the accumulators)
    __nv_bfloat16* dv;           // (B,T,H,V)
    float* dl;                   // (B,T,H,L)
    float* wq;                   // (B,T,H)  accumulates q.dq - k.dk per token and head (backward)
    // segment-level scratch
    float* seg_F;                // (B,H,NS,K,V)
    float* seg_D;                // (B,H,NS)
    __nv_bfloat16* seg_H0;       // (B,H,NS,LH,K,V)
    __nv_bfloat16* lo_H;         // (B,H,ceil(NT/2),K,V) level states inside the segments, in the place of the first pair of chunks that reads them (null:
                                 // not made); the place of a segment's first pair, which reads none, holds the decays over its pairs, fp32
    float* seg_dF;               // (B,H,NS,LH,K,V) reader summaries (backward)
    float* seg_dHf;              // (B,H,NS,K,V) gradient w.r.t. the segment summaries (backward)
    __nv_bfloat16* lo_A;         // (B,H,ceil(NT/2),K,V) gradient of every pair's summary (backward)
    // per-chunk scalars from which the decay gradient across chunk boundaries is assembled
    float* Zc;                   // (B,H,NT,LZ)      reader side: sum_t lambda * dlambda per level
    float* Yc;                   // (B,H,NT,MLOW+1)  contributor side: <KV_c, adjoint state> per low level, + combined high
    float* Yseg;                 // (B,H,NS,LH)      contributor side per segment and high level
    float* Xt;                   // (B,H,NT)         what reaches the end of each chunk, summed over the levels
    int LZ;                      // MLOW + LH
    int* err;                    // device status word: set to 1 when a bounded wait on the tensor core gave up
    int B, T, H, G, K, V, L;
    int NT, NS, LH;
    int o_has_high;              // warp-level chunk kernel: o holds the partial output of the high levels
    int hc;                      // heads per CTA of the output and gradient kernels
    int chunk_rounding;          // backward: a sequence of an odd number of chunks, or with K = 64, takes the chunk-by-chunk kernels
    // forward of a layer: y = o + D x takes the place of o (tensor-core kernels; res_D NULL: none)
    const __nv_bfloat16* res_x;  // (B,res_T,H,V)
    const void* res_D;           // (H), fp32 like y if res_f32, else bf16
    void* res_y;                 // (B,res_T,H,V)
    int res_T, res_f32;          // res_T: tokens of a sequence of x and y
    int res_n;                   // the first res_n <= T of them are written
    int res_round;               // bf16 y: D x is rounded to bf16 before the sum, as two operators would
    int warp_level;              // forward: keep to the warp-level chunk kernels, whose partial outputs take no whole pairs of chunks
    int oT;                      // tokens of a sequence of o (T, or those of the prompt whose whole chunks these are)
    float* pr_states;            // forward of the whole chunks of a prompt of T + pr_n tokens: also its level states, (B,H,pr_L,K,V)
    float* pr_part;              // (B,pr_n,H,V) scratch of the tail
    int pr_n, pr_L;
    int reuse_states;            // backward: seg_D / seg_H0 come from the forward call, do not recompute them
};

bool mamba2_uses_tc(const Mamba2Params& p);
// by what a call's sizes say alone (the workspace is carved by it)
inline bool mamba2_bwd_shape_uses_tc(const Mamba2Params& p) {
    return p.L <= M2_MAX_L_TC && !(p.chunk_rounding && (p.K != 128 || ((p.T / 64) % 2) != 0));
}
bool mamba2_bwd_uses_tc(const Mamba2Params& p);
// Whether every pair of chunks and all 128 state rows of the tensor-core tiles hold data: the kernel of one segment comes without the tests for it then.
inline bool mamba2_whole_pairs(const Mamba2Params& p) { return p.NT % 2 == 0 && p.K == 128; }
int mamba2_fwd_dispatch(Mamba2Params p, cudaStream_t stream);
int mamba2_bwd_dispatch(Mamba2Params p, cudaStream_t stream);
// segment summaries and the per-level scan over segments only (needs NS > 1)
int mamba2_fwd_states_dispatch(Mamba2Params p, cudaStream_t stream);
// outputs on tcgen05 (K = 64 or 128, V = 64): sequences of one segment, and any other
int mamba2_fwd_one_segment_tc_launch(const Mamba2Params& p, cudaStream_t stream);
int mamba2_out_tc_launch(const Mamba2Params& p, cudaStream_t stream);
int mamba2_heads_per_cta(const Mamba2Params& p, int sms);
bool mamba2_cta_has_group(const Mamba2Params& p);      // one CTA of those kernels has all heads that share q and k
// gradients on tcgen05: what the readers of the high levels send back; behind the scan over segments the gradient of every pair's summary; dq, dk, dv, d lambda
int mamba2_readers_tc_launch(const Mamba2Params& p, cudaStream_t stream);
int mamba2_adjoint_tc_launch(const Mamba2Params& p, cudaStream_t stream);
int mamba2_gradients_tc_launch(const Mamba2Params& p, cudaStream_t stream);
int mamba2_state_tc_launch(const Mamba2Params& p, cudaStream_t stream);
extern std::atomic<int> g_use_tensor_core_path;   // test hook, see llattn_testing.h
// segment summaries and decays inside the workspace of a forward call (null when it has one segment only)
int mamba2_prompt_states_check(int B, int T, int H, int G, int K, int V, int L);
int mamba2_prompt_states_launch(const __nv_bfloat16* k, const __nv_bfloat16* v, const float* g, float* states, const float* seg_F, const float* seg_D,
                                int B, int T0, int n, int H, int G, int K, int L, cudaStream_t stream);
// the tokens of a prompt behind its last whole chunk; bases of the tensors of all B (T0 + n) tokens
struct Mamba2Tail {
    const __nv_bfloat16 *q, *k, *v, *lam, *x;
    const float* g;
    const void* D;               // (H) or null
    void* y;                     // (B,T0+n,H,64)
    float* states;               // (B,H,L,K,64)
    float* part;                 // (B,n,H,64) what the tokens among themselves add to the outputs
    int T0, n, H, G, L, lam_L, d_f32;
};
int mamba2_tail_intra_launch(const Mamba2Tail& a, int B, int K, cudaStream_t stream);       // before or beside the whole chunks
int mamba2_tail_levels_launch(const Mamba2Tail& a, int B, int K, cudaStream_t stream);      // behind the states after them
int mamba2_fwd_workspace_segments(const void* ws, size_t bytes, int B, int T, int H, int G, int K, int V, const float** F, const float** D);
// clears acc_bytes (a multiple of 16) at acc and ndl floats at dl, and takes the in-chunk cumulative sum of g apart
int mamba2_bwd_init(const float* gc, float* g, long BT, int H, void* acc, size_t acc_bytes, float* dl, long ndl, cudaStream_t stream);
int mamba2_dg(const Mamba2Params& p, float* dg, cudaStream_t stream);
void cast_f32_to_bf16(const float* src, void* dst, long n, cudaStream_t stream);

}  // namespace llattn
