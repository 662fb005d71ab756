/* C ABI of the B200 (sm_100a) chunkwise log-linear attention library, libllattn.so.
 *
 * Every entry point takes raw device pointers, sizes and a CUDA stream (passed as void*), launches
 * asynchronously on that stream, never synchronises the device and never allocates: scratch
 * memory is provided by the caller (size from the matching *_workspace_bytes call; 256-byte
 * aligned).  Return value: 0 on success, a negative LLATTN_ERR_* code for rejected arguments,
 * or a positive cudaError_t value if a launch failed.
 *
 * Tensor layouts (all contiguous, "sequence first", as the reference passes them with
 * head_first=False): q,k (B,T,G,K) bf16; v,o,do,dv (B,T,H,V) bf16; g,dg (B,T,H) fp32;
 * lambda (B,T,H,L) bf16; dlambda (B,T,H,L) fp32; dq,dk (B,T,G,K) bf16.  Head h uses q/k group
 * h / (H/G).  Constraints: T % 64 == 0, T <= 524288 (the scans over 512-token segments hold ten segment
 * levels), K in {64,128}, V == 64, H % G == 0, L >= 7 + ceil(log2(T/64)), L <= 32 (the reference's
 * checks: hattention/chunkwise.py:1140-1153, 1211-1214).
 *
 * Status word.  The first 4 bytes of every workspace are a status word that the call clears and that a
 * kernel sets to 1 if one of its bounded waits (on a TMA transfer or on the tensor core) ran out; the
 * outputs of such a call are not valid.  A launch cannot report this through its return value (nothing
 * waits for the GPU), so callers that want to know read the word after synchronising:
 * llattn_workspace_status, or llattn_static_scratch_status for llattn_mamba2_fwd_static.
 */
#ifndef LLATTN_H_
#define LLATTN_H_

#include <stddef.h>

#ifdef __cplusplus
extern "C" {
#endif

#define LLATTN_ERR_UNSUPPORTED_SHAPE (-1)   /* K / V / L outside the compiled set            */
#define LLATTN_ERR_BAD_LENGTH (-2)          /* T not a multiple of the 64-token chunk        */
#define LLATTN_ERR_TOO_FEW_LEVELS (-3)      /* L < 7 + ceil(log2(T/64))                      */
#define LLATTN_ERR_BAD_GROUPS (-4)          /* H % G != 0                                    */
#define LLATTN_ERR_WORKSPACE (-5)           /* workspace NULL, misaligned or too small       */
#define LLATTN_ERR_NULL (-6)                /* a required pointer is NULL                    */
#define LLATTN_ERR_STATIC_SCRATCH (-7)      /* problem needs more than LLATTN_STATIC_SCRATCH_BYTES */
#define LLATTN_ERR_TENSOR_MAP (-8)          /* the driver refused a TMA tensor map for these pointers */
#define LLATTN_ERR_ALIGNMENT (-9)           /* a pointer that the kernels access in 16-byte words */

/* Size of the built-in scratch array used by llattn_mamba2_fwd_static (16 MiB). */
#define LLATTN_STATIC_SCRATCH_BYTES (16u << 20)

/* Library / ABI version, for the loader's sanity check. */
int llattn_version(void);
/* Number of kernels this library has launched in the process so far (all entry points, all threads). */
unsigned long long llattn_kernel_launches(void);
/* Copies the status word of `workspace` (a workspace that an earlier call on `stream` used) to *status_host
 * and returns after the stream has drained: unlike the compute entry points this one synchronises.
 * 0 = every wait completed, 1 = a kernel gave up and the call's outputs must be discarded.  (No counterpart
 * in the reference, whose Triton kernels have no bounded waits.) */
int llattn_workspace_status(const void* workspace, int* status_host, void* stream);
/* Chunk length the kernels are built for (64, as hattention/kernel.py:355-356 fixes it). */
int llattn_chunk(void);

/* Zero bytes on the stream (accumulators of the calls below). */
int llattn_clear(void* dst, size_t bytes, void* stream);

/* Log-linear Mamba-2 forward.  Replaces hattention.chunkwise.chunkwise_fwd
 * (hattention/chunkwise.py:1118-1275) with output_final_state=False: writes o and the in-chunk
 * inclusive cumulative sum of g (the reference returns both). */
size_t llattn_mamba2_fwd_workspace_bytes(int B, int T, int H, int G, int K, int V, int L);
int llattn_mamba2_fwd(const void* q, const void* k, const void* v, const float* g, const void* lambda,
                      void* o, float* g_cum, void* workspace, size_t workspace_bytes,
                      int B, int T, int H, int G, int K, int V, int L, void* stream);

/* llattn_mamba2_fwd whose output leaves as y (B,T_y,H,V) = o + D x, o rounded to bf16 first: the D residual of a Mamba-2 layer, of the first
 * T_y <= T tokens.  x is (B,T_y,H,V) bf16; y and D (H) are fp32 (y_is_f32 != 0) or bf16; x is 16-byte, y 32-byte aligned.  LLATTN_ERR_UNSUPPORTED_SHAPE
 * where the tensor-core kernels do not run (L > 20): there o and the sum are two calls (llattn_mamba2_residual). */
int llattn_mamba2_fwd_residual(const void* q, const void* k, const void* v, const float* g, const void* lambda,
                               const void* x, const void* D, void* y, int y_is_f32, int T_y, float* g_cum, void* workspace, size_t workspace_bytes,
                               int B, int T, int H, int G, int K, int V, int L, void* stream);

/* A prompt of T whole-chunk tokens and a tail of `tail` < 64 (split q .. lambda, plain x and y, see the prompts below) in one call: the
 * forward with y = o + D x (D x rounded to bf16 first where they are bf16), llattn_mamba2_prompt_states and llattn_mamba2_prompt_tail for
 * state_levels levels, the states beside the output where both leave room.  Without D (NULL) y is o, bf16.  tail_part: as there. */
int llattn_mamba2_fwd_prompt(const void* q, const void* k, const void* v, const float* g, const void* lambda,
                             const void* x, const void* D, void* y, int y_is_f32, int tail, float* tail_part, float* states, int state_levels, float* g_cum,
                             void* workspace, size_t workspace_bytes, int B, int T, int H, int G, int K, int V, int L, void* stream);

/* Forward for callers that cannot hand the library a scratch buffer.  (No counterpart in the
 * reference: its drivers allocate with torch on every call.)
 *
 * Who needs it: code that must not call cudaMalloc / cudaFree or any allocator behind them at the
 * point where the operator runs - for instance a serving loop that has handed all device memory to
 * its own pool, a host that embeds this library without torch, or a latency-critical section where
 * the device-wide synchronisation of cudaMalloc is not acceptable - and that has no spare buffer
 * of its own to pass as `workspace`.
 *
 * Same computation and results as llattn_mamba2_fwd, but the segment-level scratch lives in an
 * array compiled into the library (LLATTN_STATIC_SCRATCH_BYTES = 16 MiB of device memory on every
 * GPU that loads the library, held until the process exits).  The call allocates and frees
 * nothing.  Shapes whose scratch need (llattn_mamba2_fwd_workspace_bytes) exceeds the array are
 * rejected with LLATTN_ERR_STATIC_SCRATCH; at T = 4096, K = 128, V = 64 the need is 1.125 MiB per
 * (batch, head), so the array serves B*H <= 14 there.
 *
 * The first call on each device looks up the array's device address (cudaGetSymbolAddress) for
 * the device that is current at that moment and caches it; make that first call with the right
 * device current and before starting any stream capture.  All calls on one device share the one
 * array, and it keeps whatever the previous call left in it (the kernels overwrite every element
 * before reading it, so no clearing is needed): two calls whose kernels can overlap on the GPU
 * - different streams, or different host threads - race on it and must be serialised by the caller.
 * (Two host threads that make the FIRST call on a device at the same time both store the same looked-up
 * address into the cache; that is harmless, the race on the array itself is not.)
 * llattn_static_scratch_status reads the status word of the array on the current device (see "Status
 * word" above) after synchronising `stream`. */
size_t llattn_static_scratch_bytes(void);
int llattn_static_scratch_status(int* status_host, void* stream);
int llattn_mamba2_fwd_static(const void* q, const void* k, const void* v, const float* g, const void* lambda,
                             void* o, float* g_cum, int B, int T, int H, int G, int K, int V, int L, void* stream);

/* Log-linear Mamba-2 backward.  Replaces hattention.chunkwise.chunkwise_bwd
 * (hattention/chunkwise.py:1286-1597).  `g_cum` is the in-chunk cumulative sum that the forward
 * returned (the reference saves that tensor for backward, hattention/kernel.py:86,125); dg is the
 * gradient w.r.t. the raw per-token g.  dq and dk are already summed over the heads of each group
 * (chunkwise.py:1583-1591). */
size_t llattn_mamba2_bwd_workspace_bytes(int B, int T, int H, int G, int K, int V, int L);
int llattn_mamba2_bwd(const void* q, const void* k, const void* v, const float* g_cum, const void* lambda,
                      const void* d_o, void* dq, void* dk, void* dv, float* dg, float* dlambda,
                      void* workspace, size_t workspace_bytes,
                      int B, int T, int H, int G, int K, int V, int L, void* stream);

/* Same as llattn_mamba2_bwd, but the segment-level states of the forward pass are read from the
 * workspace that the matching llattn_mamba2_fwd call used (unmodified since), instead of being
 * recomputed from k, v, g (two launches less).  fwd_workspace == NULL behaves exactly like
 * llattn_mamba2_bwd.  No counterpart in the reference, whose autograd function keeps only the inputs
 * (hattention/kernel.py:125) and recomputes the states per level (hattention/chunkwise.py:1464-1490). */
int llattn_mamba2_bwd_saved(const void* q, const void* k, const void* v, const float* g_cum, const void* lambda,
                            const void* d_o, void* dq, void* dk, void* dv, float* dg, float* dlambda,
                            void* workspace, size_t workspace_bytes, const void* fwd_workspace, size_t fwd_workspace_bytes,
                            int B, int T, int H, int G, int K, int V, int L, void* stream);

/* llattn_mamba2_bwd_saved for the backward of a whole layer: for a sequence of an odd number of chunks, or K = 64, it keeps the chunk-by-chunk
 * kernels (everything else is as above).  The gradients of A and dt_bias are sums of dg dt over all tokens that cancel to a few per cent
 * of their terms, so their last per cents depend on where intermediate results are rounded, and these calls return the digits that they
 * always did.  Accuracy is not the reason: against fp64 the sums of the tensor-core kernels are as good or better (mamba2_bwd.cu). */
size_t llattn_mamba2_bwd_layer_workspace_bytes(int B, int T, int H, int G, int K, int V, int L);   /* at most llattn_mamba2_bwd_workspace_bytes */
int llattn_mamba2_bwd_layer(const void* q, const void* k, const void* v, const float* g_cum, const void* lambda,
                            const void* d_o, void* dq, void* dk, void* dv, float* dg, float* dlambda,
                            void* workspace, size_t workspace_bytes, const void* fwd_workspace, size_t fwd_workspace_bytes,
                            int B, int T, int H, int G, int K, int V, int L, void* stream);

/* Element-wise preparation of the log-linear Mamba-2 layer call, its backward, and the D residual.
 * Replace the torch ops around the kernel in hmamba_chunk_scan_combined (hattention/mamba_apis.py:
 * 346-366, 401-402) and compute_lambda (hattention/mamba_apis.py:70-85).  rows = B*T*H; x, v, dv, dx, dy, o, y
 * are bf16 (rows, P); dt_raw, ddt bf16 (rows); dl, lambda, ddl bf16 (rows, L); g, dg fp32 (rows); dlambda fp32
 * (rows, L); A, dt_bias (may be NULL), D (may be NULL) fp32 (H); Lp fp32 (H, L).  lambda_mode: 0 "positive"
 * softplus(Lp dl), 1 "bounded" exp(-exp(Lp) softplus(dl)), 2 none Lp dl.
 *   fwd: dt = softplus(dt_raw + dt_bias); v = x dt; g = A dt; lambda = f(Lp, dl)
 *   bwd: dx = dv dt + D dy; ddt, ddl; dA, dbias, dD (H) and dLp (H, L) are ACCUMULATED with atomics into
 *        buffers the caller has cleared
 *   residual: y = o + D x, y fp32 (y_is_f32 != 0; what torch's promotion gives for fp32 D) or bf16
 * Constraints: P % 8 == 0, P <= 256, L <= 64. */
int llattn_mamba2_prep_fwd(const void* x, const void* dt_raw, const float* dt_bias, const float* A, const void* dl, const float* Lp,
                           void* v, float* g, void* lambda, long rows, int H, int P, int L, int lambda_mode, void* stream);
int llattn_mamba2_prep_bwd(const void* x, const void* dt_raw, const float* dt_bias, const float* A, const void* dl, const float* Lp,
                           const float* D, const void* dv, const float* dg, const float* dlambda, const void* dy,
                           void* dx, void* ddt, void* ddl, float* dA, float* dbias, float* dLp, float* dD,
                           long rows, int H, int P, int L, int lambda_mode, void* stream);
/* The same passes for parameters in the dtype the model keeps them in: dt_bias, Lp, D fp32 or bf16 by their flags. */
int llattn_mamba2_layer_prep_fwd(const void* x, const void* dt_raw, const void* dt_bias, int bias_is_f32, const float* A, const void* dl,
                                 const void* Lp, int lp_is_f32, void* v, float* g, void* lambda, long rows, int H, int P, int L,
                                 int lambda_mode, void* stream);
int llattn_mamba2_layer_prep_bwd(const void* x, const void* dt_raw, const void* dt_bias, int bias_is_f32, const float* A, const void* dl,
                                 const void* Lp, int lp_is_f32, const void* D, int d_is_f32, const void* dv, const float* dg,
                                 const float* dlambda, const void* dy, void* dx, void* ddt, void* ddl, float* dA, float* dbias,
                                 float* dLp, float* dD, long rows, int H, int P, int L, int lambda_mode, void* stream);
int llattn_mamba2_residual(const void* o, const void* x, const float* D, void* y, int y_is_f32, long rows, int H, int P, void* stream);

/* What the mixer does around the scan, in place on the rows of its projection zxbcdtdl (B,T,W), W = 2 H 64 + 2 G N + H + H L:
 * [z (H 64) | x (H 64) | B (G N) | C (G N) | dt (H) | dl (H L)], bf16.  Replace the split, convolution, preparation, gated norm and
 * the gradients of all of them in hmamba_split_conv1d_scan_combined (hattention/mamba_apis.py:186-259).
 *   prep_fwd: (x, B, C) = silu(causal depthwise convolution with four taps); v = x softplus(dt + dt_bias), g = A softplus(...),
 *        lambda = f(Lp, dl); writes x, v (B,T,H,64), k = B, q = C (B,T,G,N), g, lambda
 *   prep_bwd: from dv, dq, dk, dg, dlambda of the scan and dy of the norm (for the D residual): every slice of dzx but z's, and
 *        dconv_w (channels,4), dconv_b, dA, dbias, dLp ACCUMULATED into fp32 buffers the caller has cleared (the
 *        first two, and dw below, at 16-byte boundaries)
 *   norm_fwd: out = RMSNorm((o + D x) silu(z)) w, and rstd per token; norm_bwd: dy (gradient of o and of o + D x), the z slice of dzx, and
 *        dw, dD accumulated
 * conv_w, conv_b (may be NULL), dt_bias (may be NULL), Lp, D (may be NULL), w are fp32 or bf16 by their flags.  Constraints: heads of 64,
 * N % 64 == 0, H <= 128, L <= 64. */
int llattn_mixer_prep_fwd(const void* zx, const void* conv_w, int conv_w_f32, const void* conv_b, int conv_b_f32, const void* dt_bias,
                          int bias_f32, const float* A, const void* Lp, int lp_f32, void* x, void* v, void* k, void* q, float* g,
                          void* lambda, int B, int T, int H, int G, int N, int L, int lambda_mode, void* stream);
int llattn_mixer_prep_bwd(const void* zx, const void* conv_w, int conv_w_f32, const void* conv_b, int conv_b_f32, const void* dt_bias,
                          int bias_f32, const float* A, const void* Lp, int lp_f32, const void* D, int d_f32, const void* dv, const void* dy,
                          const void* dq, const void* dk, const float* dg, const float* dlambda, void* dzx, float* dconv_w, float* dconv_b,
                          float* dA, float* dbias, float* dLp, int B, int T, int H, int G, int N, int L, int lambda_mode, void* stream);
int llattn_mixer_norm_fwd(const void* o, const void* x, const void* D, int d_f32, const void* zx, int zx_width, const void* w, int w_f32,
                          void* out, float* rstd, long rows, int H, float eps, void* stream);
int llattn_mixer_norm_bwd(const void* o, const void* x, const void* D, int d_f32, const void* zx, int zx_width, const void* w, int w_f32,
                          const void* dn, const float* rstd, void* dy, void* dzx, float* dw, float* dD, long rows, int H, void* stream);

/* Prefill hand-off: the level states after T tokens, states fp32 (B,H,K,V,L), every level written.
 * Level 0 is k_m v_m^T for the last token m = T-1; for each set bit j of m, level j+1 holds the 2^j
 * tokens that follow the buckets of the higher set bits, each decayed to token m; other levels are zero.
 * Replaces the state side of hattention_prefill (hattention/kernel.py:470-560): the final states `ht` of
 * chunk_fwd_kernel_h (hattention/chunkwise.py:171-173, 278-280) for the inter-chunk levels together with
 * postprocess_prefill_hstate_ (hattention/kernel.py:378-466) for the levels inside the last chunk and its
 * clearing of unpopulated levels.  k (B,T,G,K), v (B,T,H,V) bf16, g (B,T,H) fp32 raw log decay.  Any T >= 1;
 * K in {64,128}, V == 64, bit_length(T-1) + 1 <= L <= 32. */
int llattn_mamba2_final_state(const void* k, const void* v, const float* g, float* states,
                              int B, int T, int H, int G, int K, int V, int L, void* stream);

/* One decode step (hattention_step, hattention/kernel.py:563-633, with HState.cascade_weak / insert and
 * step_output, hattention/recurrent.py:42-54, 79-98, 134-166) for every (batch, head): levels 0..carry_level
 * are summed into level carry_level (the caller runs the cascade on the token counts, which are the same
 * for every sequence: carry_level is the first level that is not full), every level is multiplied by
 * exp(g), level 0 becomes k v^T, and o = q . sum_l lambda_l S_l.  states fp32 (B,H,K,V,L) updated in place;
 * q, k (B,G,K), v (B,H,V), lambda (B,H,L), o (B,H,V) bf16; g (B,H) fp32.  256 % V == 0, L <= 32. */
int llattn_mamba2_step(float* states, const void* q, const void* k, const void* v, const float* g, const void* lambda, void* o,
                       int B, int H, int G, int K, int V, int L, int carry_level, void* stream);

/* ---- Prompts of any length and decode steps on LEVEL-MAJOR states: fp32, stored (B,H,L,K,V), one contiguous K x V block per
 * level of a head (the tensor a caller sees can still have the shape (B,H,K,V,L)).  A step then moves only the levels that
 * hold tokens.
 *
 * llattn_mamba2_layer_step: hselective_state_update (hattention/mamba_apis.py:407-566) in one launch.  q, k (B,G,K), x (B,H,V),
 * dt (B,H), dl (B,H,L) bf16; Lp (H,L), D (H), dt_bias (H) fp32 or bf16 by their flags, the last two may be NULL; A (H) fp32.
 *     dt = softplus(dt + dt_bias), v = x dt, g = A dt, lambda = f(Lp, dl), the step of llattn_mamba2_step, y = o + D x
 * with the rounding of the reference's torch operators; y bf16, fp32 with an fp32 D.  dt == NULL: x is v and g (B,H) fp32 is
 * given; Lp == NULL: dl is lambda.  `live`: bit l is set when level l holds tokens before the step (counts > 0); levels
 * whose bit is clear are taken as zero and not read.  carry_level as in llattn_mamba2_step.  V % 16 == 0, V <= 256, K <= 1024.
 * llattn_gdn_layer_step: the one-token call of chunk_h_gated_delta_rule (hattention/gated_delta_rule_apis.py:93-132).  q, k
 * (B,G,K) raw; with l2norm != 0 they are normalised (q scaled) first; lambda_mul != 0: lambda is multiplied by it and rounded to
 * bf16.  V % 16 == 0, K <= 256.
 * Both launch on `device`, which `stream` belongs to. */
int llattn_mamba2_layer_step(float* states, const void* q, const void* k, const void* x, const void* dt, const float* g,
                             const void* dl, const void* Lp, int lp_is_f32, const void* D, int d_is_f32, const void* dt_bias,
                             int bias_is_f32, const float* A, void* y, int B, int H, int G, int K, int V, int L, unsigned live,
                             int carry_level, int lambda_mode, int dt_softplus, int device, void* stream);
int llattn_gdn_layer_step(float* states, const void* q, const void* k, const void* v, const void* beta, const float* g,
                          const void* lambda, void* o, int B, int H, int G, int K, int V, int L, unsigned live, int carry_level,
                          int l2norm, float scale, float lambda_mul, int device, void* stream);

/* Prompts of T + tail tokens, T % 64 == 0, tail < 64: the whole chunks through the chunkwise kernels, the tail behind them in kernels
 * that keep in fp32 what a decode step keeps in fp32.  Together these replace hattention_prefill (hattention/kernel.py:469-560) and
 * the torch operators of the layer around it (hattention/mamba_apis.py:346-399).  "Split" tensors hold the B x T tokens of whole
 * chunks first and the B x tail others behind them (the plain (B,T+tail,...) for B = 1 or without a tail).
 *   mamba2_prompt_prep: split v, g, lambda of plain x, dt, dl, and, where q_split and k_split are given, split copies of q and k; rounded
 *     as torch's operators on bf16 tensors round; dt_bias (may be NULL) and Lp are fp32 or bf16 by their flags
 *   mamba2_prompt_residual: y = o + D x of the whole chunks; o (B,T,H,P), plain x, y; y and D are fp32 (y_is_f32 != 0) or bf16
 *   mamba2_prompt_states: the level states after T tokens, level-major; k, v, g of the whole chunks.  With the workspace of the forward
 *     call on them (may be NULL) the levels that hold whole 512-token segments are sums of its summaries.  With a tail: as the first
 *     token of it finds them once the cascade has run, and without the levels 0 .. 6.
 *   mamba2_prompt_tail: outputs of the tail (y plain, with D its residual) and the level states after it, from those; split q .. lambda;
 *     tail_part: B tail H V floats of scratch (16-byte aligned; may be NULL for T = 0) */
int llattn_mamba2_prompt_prep(const void* x, const void* dt_raw, const void* dt_bias, int bias_is_f32, const float* A, const void* dl,
                              const void* Lp, int lp_is_f32, const void* q, const void* k, void* v, float* g, void* lambda, void* q_split,
                              void* k_split, int B, int T, int tail, int H, int G, int K, int P, int L, int lambda_mode, void* stream);
int llattn_mamba2_prompt_residual(const void* o, const void* x, const void* D, void* y, int y_is_f32, int B, int T, int tail, int H, int P,
                                  void* stream);
int llattn_mamba2_prompt_states(const void* k, const void* v, const float* g, float* states, const void* fwd_workspace,
                                size_t fwd_workspace_bytes, int B, int T, int tail, int H, int G, int K, int V, int L, void* stream);
int llattn_mamba2_prompt_tail(const void* q, const void* k, const void* v, const float* g, const void* lambda, const void* x, const void* D,
                              int y_is_f32, void* y, float* states, int state_levels, float* tail_part, int B, int T, int tail, int H, int G, int K,
                              int V, int L, void* stream);

/*   gdn_prompt_prep: a value head of V columns as `rep` heads of V / rep columns that share everything else ((B,T,H,V) is (B,T,H rep,V / rep)
 *     in memory).  Split, one row per part: l2norm of q (scaled) and k, K_out >= K columns wide (at most 128), and, each where its pointer is
 *     given, v, beta and g, lambda (times lambda_mul unless 0).  q, k have G groups of H / G heads.
 *   gdn_prompt: outputs and level states of a prompt from those: heads counts parts, V (64 or 128) the columns of one.  o_chunks
 *     (B,T,heads,V) receives the whole chunks' outputs (g_cum, Aw, Au of them as in llattn_gdn_fwd; none of these is used for T = 0), o
 *     (B,T+tail,heads,V) those of the tail (o_chunks may be o for B = 1 or without a tail); states level-major (B,heads / rep,state_levels,
 *     state_rows,rep V), every level written; scratch (16-byte aligned) for a tail only. */
int llattn_gdn_prompt_prep(const void* q, const void* k, const void* v, const void* beta, const float* g, const void* lambda,
                           void* qn, void* kn, void* v_split, void* beta_split, float* g_split, void* lambda_split,
                           int B, int T, int tail, int H, int G, int K, int K_out, int V, int rep, int L, float scale, float lambda_mul,
                           void* stream);
size_t llattn_gdn_prompt_scratch_bytes(int B, int T, int tail, int heads, int rep, int V);
int llattn_gdn_prompt(const void* q, const void* k, const void* v, const void* beta, const float* g, const void* lambda, void* o_chunks, void* o,
                      float* g_cum, void* Aw, void* Au, float* states, int state_rows, int rep, int state_levels, void* scratch,
                      size_t scratch_bytes, void* workspace, size_t workspace_bytes, int B, int T, int tail, int heads, int K, int V, int L,
                      void* stream);

/* Log-linear Gated DeltaNet forward.  Replaces hattention.chunkwise_hgdn.chunkwise_fwd
 * (hattention/chunkwise_hgdn.py:566-788) with output_final_state=False.  q and k are per head,
 * (B,T,H,K), and must already be L2-normalised (q also scaled) as the reference's autograd
 * function does before the call (hattention/kernel.py:110-111); beta is (B,T,H) bf16; g is the raw
 * log decay.  Writes o, the in-chunk cumulative g, and the two 64x64 UT-transform inverses per
 * chunk, Aw and Au, as (B,T,H,64) bf16 (the reference returns and saves them for the backward).
 * Constraints: T % 64 == 0, K == 128, V in {64,128}, 7 + ceil(log2(T/64)) <= L <= 32, T <= 16384. */
size_t llattn_gdn_fwd_workspace_bytes(int B, int T, int H, int K, int V, int L);
int llattn_gdn_fwd(const void* q, const void* k, const void* v, const void* beta, const float* g, const void* lambda,
                   void* o, float* g_cum, void* Aw, void* Au, void* workspace, size_t workspace_bytes,
                   int B, int T, int H, int K, int V, int L, void* stream);

/* Prompt pass of the log-linear Gated DeltaNet layer: llattn_gdn_fwd plus the level states a decoder continues
 * from.  `states` is fp32 (B,H,K,V,L), level innermost (the layout of the reference's HState,
 * hattention/recurrent.py:9-40); it is cleared and then, for every set bit j of NT - 1 (NT = T / 64), level
 * 7 + j receives the state of the block of 2^j chunks that the LAST chunk reads, i.e. the states as they stand
 * before the last 64 tokens.  The caller feeds those 64 tokens (and any tokens beyond T) through
 * llattn_gdn_step, which builds the levels inside the chunk.  Together the two replace hattention_prefill with
 * hstruct = GDELTA (hattention/kernel.py:469-560: chunkwise_fwd with output_final_state=True, then
 * postprocess_prefill_hstate_, :378-466).  Other arguments and constraints as llattn_gdn_fwd. */
int llattn_gdn_prefill(const void* q, const void* k, const void* v, const void* beta, const float* g, const void* lambda,
                       void* o, float* g_cum, void* Aw, void* Au, float* states, void* workspace, size_t workspace_bytes,
                       int B, int T, int H, int K, int V, int L, void* stream);

/* One decode step of the log-linear Gated DeltaNet layer for every (batch, head).  Replaces hattention_step with
 * hstruct = GDELTA (hattention/kernel.py:563-633) after its l2norm / scale of q and k, i.e. HState.cascade_weak /
 * insert with the delta-rule gate and step_output (hattention/recurrent.py:42-54, 79-98, 134-166): levels
 * 0..carry_level are summed into level carry_level (the caller runs the cascade on the token counts), every
 * level becomes exp(g) (S - beta k (k^T S)), level 0 becomes beta k v^T, and o = q . sum_l lambda_l S_l.
 * states fp32 (B,H,K,V,L) updated in place, one pass over HBM; q, k (B,H,K) already normalised (q also scaled),
 * v (B,H,V), beta (B,H), lambda (B,H,L), o (B,H,V) bf16; g (B,H) fp32 log decay.
 * K % 32 == 0, K <= 256, V % 8 == 0, L <= 32 (K / 32 in {1,2,3,4,6,8}; {2,4} when L > 16). */
int llattn_gdn_step(float* states, const void* q, const void* k, const void* v, const void* beta, const float* g,
                    const void* lambda, void* o, int B, int H, int K, int V, int L, int carry_level, void* stream);

/* Log-linear Gated DeltaNet backward, first stage: everything that involves the inter-chunk level
 * states.  Replaces, inside hattention.chunkwise_hgdn.chunkwise_bwd (hattention/chunkwise_hgdn.py:
 * 799-1010), the per-level loop over chunk_gated_delta_rule_fwd_h (state recomputation),
 * chunk_gated_delta_rule_bwd_dhu (adjoint states) and the state-dependent parts of chunk_bwd_dqkwg /
 * chunk_bwd_dv_local.  Inputs are those the reference saves for its backward: q, k (normalised, as in
 * the forward), v, beta, the in-chunk cumulative g, lambda, Aw, Au, and d_o.  Per chunk, with
 * kd = k exp(gl - G), wd = w exp(G), qd = exp(G)(q - tril(q k^T) w), u as in the forward, writes the
 * gradients with respect to those chunk matrices, fp32 (B,T,H,K): d_qd, d_wd, d_kd; bf16 (B,T,H,V):
 * d_u; the part of the gradient of each chunk's total log decay that comes from the state decay,
 * d_gl fp32 (B,T/64,H); and columns 7 .. 7+ceil(log2(T/64))-1 of dlambda, fp32 (B,T,H,L) (other
 * columns are left untouched).  Same shape constraints as llattn_gdn_fwd. */
size_t llattn_gdn_bwd_levels_workspace_bytes(int B, int T, int H, int K, int V, int L);
int llattn_gdn_bwd_levels(const void* q, const void* k, const void* v, const void* beta, const float* g_cum, const void* lambda,
                          const void* Aw, const void* Au, const void* d_o, float* d_qd, float* d_wd, float* d_kd, void* d_u,
                          float* d_gl, float* dlambda, void* workspace, size_t workspace_bytes,
                          int B, int T, int H, int K, int V, int L, void* stream);

/* Log-linear Gated DeltaNet backward, complete.  Replaces hattention.chunkwise_hgdn.chunkwise_bwd
 * (hattention/chunkwise_hgdn.py:799-1010): the stage above followed by the chunk-local part
 * (gradients through kd, wd, qd, u, the UT transform, tril(q k^T) and the intra-chunk output).
 * Inputs as saved by the reference's autograd function (hattention/kernel.py:113-120): normalised
 * q, k, then v, beta, the in-chunk cumulative g, lambda, Aw, Au, and d_o (bf16 (B,T,H,V)).
 * Outputs are fp32: dq, dk (B,T,H,K) with respect to the NORMALISED q, k (the caller applies the
 * l2norm / scale backward as hattention/kernel.py:208-221 does), dv (B,T,H,V), dbeta, dg (B,T,H)
 * with respect to the raw g, dlambda (B,T,H,L; every column is written).  Same shape constraints
 * as llattn_gdn_fwd. */
size_t llattn_gdn_bwd_workspace_bytes(int B, int T, int H, int K, int V, int L);
int llattn_gdn_bwd(const void* q, const void* k, const void* v, const void* beta, const float* g_cum, const void* lambda,
                   const void* Aw, const void* Au, const void* d_o, float* dq, float* dk, float* dv, float* dbeta, float* dg,
                   float* dlambda, void* workspace, size_t workspace_bytes,
                   int B, int T, int H, int K, int V, int L, void* stream);

/* The same forward and backward with the forward's intermediates kept between the two calls, so that
 * the backward does not recompute them (the reference recomputes w, u and the level states in its
 * backward, hattention/chunkwise_hgdn.py:820-870; keeping them trades memory for about a fifth of the
 * step).  llattn_gdn_fwd_keep is llattn_gdn_fwd with a larger workspace that, on return, holds the
 * chunk matrices and every chunk's level states; the caller leaves it untouched and hands it to
 * llattn_gdn_bwd_kept as fwd_workspace.  Results are those of llattn_gdn_fwd / llattn_gdn_bwd. */
size_t llattn_gdn_fwd_keep_workspace_bytes(int B, int T, int H, int K, int V, int L);
int llattn_gdn_fwd_keep(const void* q, const void* k, const void* v, const void* beta, const float* g, const void* lambda,
                        void* o, float* g_cum, void* Aw, void* Au, void* workspace, size_t workspace_bytes,
                        int B, int T, int H, int K, int V, int L, void* stream);
size_t llattn_gdn_bwd_kept_workspace_bytes(int B, int T, int H, int K, int V, int L);
int llattn_gdn_bwd_kept(const void* q, const void* k, const void* v, const void* beta, const float* g_cum, const void* lambda,
                        const void* Aw, const void* Au, const void* d_o, float* dq, float* dk, float* dv, float* dbeta,
                        float* dg, float* dlambda, const void* fwd_workspace, size_t fwd_workspace_bytes, void* workspace,
                        size_t workspace_bytes, int B, int T, int H, int K, int V, int L, void* stream);
/* llattn_gdn_bwd_kept with dv written in bf16 (B,T,H,V), the dtype the reference's autograd function returns for bf16 v
 * (hattention/kernel.py:226: dv.to(v)): saves the caller a conversion pass over dv.  Same workspace size. */
int llattn_gdn_bwd_kept_bf16dv(const void* q, const void* k, const void* v, const void* beta, const float* g_cum,
                               const void* lambda, const void* Aw, const void* Au, const void* d_o, float* dq, float* dk,
                               void* dv_bf16, float* dbeta, float* dg, float* dlambda, const void* fwd_workspace,
                               size_t fwd_workspace_bytes, void* workspace, size_t workspace_bytes,
                               int B, int T, int H, int K, int V, int L, void* stream);

/* llattn_gdn_bwd_kept_bf16dv that also takes the backward of the l2 normalisation (below): q = l2norm(raw_q) * scale, k = l2norm(raw_k), and gq,
 * gk (B,T,H,K) bf16 are the gradients of raw_q, raw_k.  K = 128. */
int llattn_gdn_bwd_kept_normed(const void* q, const void* k, const void* raw_q, const void* raw_k, float scale, const void* v, const void* beta,
                               const float* g_cum, const void* lambda, const void* Aw, const void* Au, const void* d_o, void* gq, void* gk,
                               void* dv_bf16, float* dbeta, float* dg, float* dlambda, const void* fwd_workspace, size_t fwd_workspace_bytes,
                               void* workspace, size_t workspace_bytes, int B, int T, int H, int K, int V, int L, void* stream);

/* Row-wise L2 normalisation of q / k and its backward, as applied around the Gated DeltaNet drivers
 * when use_qk_l2norm_in_kernel is set.  Replace fla.modules.l2norm.l2norm_fwd / l2norm_bwd with the
 * scale folded in (hattention/kernel.py:20-29: l2norm_and_scale_fwd / l2norm_and_scale_bwd).
 *   fwd: y = bf16(bf16(x rsqrt(sum x^2 + 1e-6)) * scale)        x, y bf16 (rows, D)
 *   bwd: dx = bf16((g - yhat (yhat . g)) rstd), g = dy * scale   dy fp32 (rows, D), dx bf16
 * Constraints: D % 8 == 0, D <= 256. */
int llattn_l2norm_fwd(const void* x, void* y, long rows, int D, float scale, void* stream);
int llattn_l2norm_bwd(const void* x, const float* dy, void* dx, long rows, int D, float scale, void* stream);

/* The gradients that leave a Gated DeltaNet backward, in one pass: gq, gk (rows,K) bf16 = l2norm backward of dq, dk (K_in >= K columns, at
 * most 128: padded keys) at raw q, k (q with `scale`), gbeta (rows) and glambda (rows,L) bf16; lambda_mul != 0: glambda is
 * rounded, multiplied and rounded again, as the reference's lambda / scale differentiates (gated_delta_rule_apis.py:65-70).  The fp32
 * inputs have `rep` rows for each row of the results, which are summed (parts of a wide value head); gg (rows) takes the sums of dg where
 * dg is given.  Without q (NULL) dbeta and dlambda only. */
int llattn_gdn_grad_out(const void* q, const void* k, const float* dq, const float* dk, const float* dbeta, const float* dlambda,
                        const float* dg, void* gq, void* gk, void* gbeta, void* glambda, float* gg, long rows, int rep, int K, int K_in, int L,
                        float scale, float lambda_mul, void* stream);

/* Diagnostic: one 128 x N x kred bf16 tensor-core product (tcgen05.mma, accumulator in tensor
 * memory) per operand-layout combination used by the kernels: mode 0: D = A B^T with A [128][kred],
 * B [N][kred]; mode 1: D = A B with B [kred][N]; mode 2: D = A^T B with A [kred][128], B [kred][N].
 * D is [128][N] fp32.  Modes 10, 11, 12 are the same three products issued through compile-time shaped
 * loops in a branch of one lane; modes 20..23 by a converged warp with an elected lane leading (23: D = A^T B^T with
 * A [kred][128], B [N][kred]), modes 30, 31 as 20, 21 with A in tensor memory.  *err_flag is set to 1 if the tensor core did not signal completion within
 * the kernel's bounded wait.  (No counterpart in the reference; used by the test-suite.) */
int llattn_selftest_umma(const void* A, const void* B, float* D, int N, int kred, int mode, int* err_flag, void* stream);

/* Diagnostic: SM clock cycles from the issue of `reps` back-to-back 128 x N x kred products of one layout
 * combination (operands resident in shared memory, accumulator in tensor memory; modes 0..2 as above, 3 and 4 with the
 * 256-row operand of the Gated DeltaNet scans; issued by a converged warp: 20..24 the layouts of 0..4, 30, 31 those of
 * 0, 1 with A in tensor memory) to their completion, written to *cycles (device memory); issuers = 2 lets two warps issue `reps` products each at the
 * same time into separate accumulators.  (No counterpart in the reference.) */
int llattn_selftest_umma_cycles(int N, int kred, int mode, int reps, int issuers, long long* cycles, int* err_flag, void* stream);

#ifdef __cplusplus
}
#endif
#endif /* LLATTN_H_ */
