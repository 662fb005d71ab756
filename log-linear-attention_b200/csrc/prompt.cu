// Prompts of any length: what surrounds the chunkwise kernels when a prompt is not a whole number of chunks.
//
// Reference being replaced: hattention_prefill (hattention/kernel.py:469-560), which runs the chunkwise kernels on the whole
// chunks, steps the remaining tokens one by one and rebuilds the levels inside the last chunk (postprocess_prefill_hstate_,
// :378-466), and the torch operators around it (hattention/mamba_apis.py:346-399, gated_delta_rule_apis.py:65-92).
//
// Here the whole chunks of a prompt go through the chunkwise kernels and the n < 64 tokens behind them (its tail) through one kernel that
// keeps in fp32 what a decode step keeps in fp32, for all of them at once.  The tensors that the passes read hold the B T0 tokens of whole
// chunks first and the B n tails behind them, so that each part is a plain tensor of its own; for one sequence, or without a tail,
// that is how they are stored anyway.
#include "llattn_gdn.h"
#include "rowwise.cuh"

namespace llattn {

// place of token (b, t) in those tensors
__device__ __forceinline__ long split_token(unsigned b, unsigned t, int B, int T0, int n) {
    return t < (unsigned)T0 ? (long)b * T0 + t : (long)B * T0 + (long)b * n + (t - T0);
}

// ---- log-linear Mamba-2: what torch's operators make of x, dt, A, dl and L before the scan of a prompt: dt + bias rounded to bf16 unless the
// bias is fp32, softplus and A dt in fp32, lambda rounded at every operator.  LPR lanes per (b, t, h) row; the blocks behind those of the rows
// copy q and k (16 bytes a thread) where several sequences have tails.
template <int LPR>
__global__ void __launch_bounds__(256) m2_prompt_prep_kernel(const bf16* __restrict__ x, const bf16* __restrict__ dt_raw, const void* __restrict__ dt_bias, int bias_f32,
                                                             const float* __restrict__ A, const bf16* __restrict__ dl, const void* __restrict__ Lp, int lp_f32,
                                                             const uint4* __restrict__ q, const uint4* __restrict__ k, bf16* __restrict__ v,
                                                             float* __restrict__ g, bf16* __restrict__ lam, uint4* __restrict__ qs, uint4* __restrict__ ks,
                                                             int B, int T0, int n, int H, int P, int L, int mode, int row_blocks, int qk16) {
    chain_wait();
    const unsigned T = T0 + n;
    if ((int)blockIdx.x >= row_blocks) {
        // qk16: 16-byte words of a token of q (and of k)
        const unsigned e = (blockIdx.x - row_blocks) * 256u + threadIdx.x;
        const unsigned all = (unsigned)B * T * qk16;
        if (e >= 2u * all) return;
        const bool is_k = e >= all;
        const unsigned i = is_k ? e - all : e;
        const unsigned c = i % qk16, tok = i / qk16;
        (is_k ? ks : qs)[split_token(tok / T, tok % T, B, T0, n) * qk16 + c] = (is_k ? k : q)[i];
        return;
    }
    const int lane = threadIdx.x % LPR;
    const unsigned row = (blockIdx.x * 256u + threadIdx.x) / LPR;
    if (row >= (unsigned)B * T * H) return;
    const int h = row % H;
    const unsigned tok = row / H;
    const long dst = split_token(tok / T, tok % T, B, T0, n) * H + h;
    float dt = __bfloat162float(dt_raw[row]);
    if (dt_bias) {
        dt += load_param(dt_bias, h, bias_f32);
        if (!bias_f32) dt = round_bf16(dt);
    }
    dt = softplus_torch(dt);
    if (lane == 0) g[dst] = A[h] * dt;
    if (lane * 8 < P) {
        uint4 out;
        const uint4 raw = *reinterpret_cast<const uint4*>(x + (long)row * P + lane * 8);
        const __nv_bfloat162* hx = reinterpret_cast<const __nv_bfloat162*>(&raw);
        uint32_t* o = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = pack_bf16(__bfloat162float(hx[i].x) * dt, __bfloat162float(hx[i].y) * dt);
        *reinterpret_cast<uint4*>(v + dst * P + lane * 8) = out;
    }
    for (int j = lane; j < L; j += LPR)
        lam[dst * L + j] = __float2bfloat16(lambda_torch(mode, load_param(Lp, h * L + j, lp_f32), __bfloat162float(dl[(long)row * L + j])));
}

// y = o + D x for the whole chunks: T0 tokens of each sequence of o, the first T0 of the T0 + n of those of x and y; y has the dtype of D, and
// a bf16 D x is rounded before the sum, as two operators would.  P / 8 threads a row.
template <bool F32OUT>
__global__ void __launch_bounds__(256) m2_prompt_residual_kernel(const bf16* __restrict__ o, const bf16* __restrict__ x, const void* __restrict__ D,
                                                                 void* __restrict__ y, int B, int T0, int n, int H, int P) {
    chain_wait();
    const unsigned p8 = P / 8;
    const unsigned e = blockIdx.x * 256u + threadIdx.x;
    const unsigned row = e / p8, c = (e % p8) * 8;
    if (row >= (unsigned)B * T0 * H) return;
    const unsigned h = row % H, tok = row / H, t = tok % T0, b = tok / T0;
    const long at = (((long)b * (T0 + n) + t) * H + h) * P + c;
    const uint4 ro = *reinterpret_cast<const uint4*>(o + (long)row * P + c), rx = *reinterpret_cast<const uint4*>(x + at);
    const float d = load_param(D, h, F32OUT);
    const __nv_bfloat162* ho = reinterpret_cast<const __nv_bfloat162*>(&ro);
    const __nv_bfloat162* hx = reinterpret_cast<const __nv_bfloat162*>(&rx);
    float r[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float x0 = __bfloat162float(hx[i].x) * d, x1 = __bfloat162float(hx[i].y) * d;
        r[2 * i] = __bfloat162float(ho[i].x) + (F32OUT ? x0 : round_bf16(x0));
        r[2 * i + 1] = __bfloat162float(ho[i].y) + (F32OUT ? x1 : round_bf16(x1));
    }
    if (F32OUT) {
        float* w = reinterpret_cast<float*>(y) + at;
        *reinterpret_cast<float4*>(w) = make_float4(r[0], r[1], r[2], r[3]);
        *reinterpret_cast<float4*>(w + 4) = make_float4(r[4], r[5], r[6], r[7]);
    } else {
        uint4 out;
        uint32_t* w = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = pack_bf16(r[2 * i], r[2 * i + 1]);
        *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(y) + at) = out;
    }
}

// ---- Gated DeltaNet: q, k normalised (q scaled), widened to Ko columns and expanded to one per head, lambda scaled, split into whole chunks and
// tails, in one launch.  16 lanes per (b, t, h) row.
struct GdnPrepArgs {
    const bf16 *q, *k;       // (B,T,G,K)
    const bf16 *v;           // (B,T,H,V)
    const bf16* beta;        // (B,T,H)
    const float* g;          // (B,T,H)
    const bf16* l;           // (B,T,H,L)
    // results, split, one row per part of a head: a value head of V columns is `rep` heads of V / rep columns that share q, k, beta, g, lambda
    bf16 *qn, *kn;           // (B,T,H rep,Ko)
    bf16 *vp, *bp;           // (B,T,H rep,V / rep), (B,T,H rep)
    float* gp;               // (B,T,H rep)
    bf16* lp;                // (B,T,H rep,Lo)
    int B, T0, n, H, G, K, Ko, V, rep, L;
    float scale, lam_mul;    // lam_mul = 0: lambda as it is
};

__global__ void __launch_bounds__(256) gdn_prompt_prep_kernel(const __grid_constant__ GdnPrepArgs a) {
    chain_wait();
    const int lane = threadIdx.x & 15;
    const unsigned row = blockIdx.x * 16u + (threadIdx.x >> 4);
    const unsigned heads = a.H * a.rep, T = a.T0 + a.n, rows = (unsigned)a.B * T * heads;
    const bool have = row < rows;
    const unsigned hp = row % heads, h = hp / a.rep, part = hp % a.rep, tok = row / heads;
    const long dst = split_token(tok / T, tok % T, a.B, a.T0, a.n) * heads + hp;
    const long tr = have ? tok : 0;
    const long src = tr * a.H + h, qsrc = tr * a.G + h / (a.H / a.G);
    uint4 raw[2];
    float rstd[2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        raw[w] = make_uint4(0, 0, 0, 0);
        if (have && lane * 8 < a.K) raw[w] = *reinterpret_cast<const uint4*>((w ? a.k : a.q) + qsrc * a.K + lane * 8);
        const __nv_bfloat162* f = reinterpret_cast<const __nv_bfloat162*>(&raw[w]);
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float x0 = __bfloat162float(f[i].x), x1 = __bfloat162float(f[i].y);
            ss += x0 * x0 + x1 * x1;
        }
#pragma unroll
        for (int d = 8; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
        rstd[w] = rsqrtf(ss + 1e-6f);
    }
    if (!have) return;
    if (lane * 8 < a.Ko) {
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const __nv_bfloat162* f = reinterpret_cast<const __nv_bfloat162*>(&raw[w]);
            uint4 out;
            __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                o[i] = __floats2bfloat162_rn(__bfloat162float(f[i].x) * rstd[w], __bfloat162float(f[i].y) * rstd[w]);
                if (w == 0) o[i] = __floats2bfloat162_rn(__bfloat162float(o[i].x) * a.scale, __bfloat162float(o[i].y) * a.scale);
            }
            *reinterpret_cast<uint4*>((w ? a.kn : a.qn) + dst * a.Ko + lane * 8) = out;
        }
    }
    if (a.vp) {
        const int width = a.V / a.rep;
        for (int c = lane * 8; c < width; c += 128) {
            *reinterpret_cast<uint4*>(a.vp + dst * width + c) = *reinterpret_cast<const uint4*>(a.v + src * a.V + part * width + c);
        }
    }
    if (a.lp)
        for (int j = lane; j < a.L; j += 16) {
            float x = __bfloat162float(a.l[src * a.L + j]);
            if (a.lam_mul != 0.f) x *= a.lam_mul;
            a.lp[dst * a.L + j] = __float2bfloat16(x);
        }
    if (lane == 0 && a.gp) {
        a.gp[dst] = a.g[src];
        a.bp[dst] = a.beta[src];
    }
}

// ---- Gated DeltaNet: the level states after the last token of a prompt without a tail (gdn_tail.cu has the others).  The scan over chunks leaves the
// inter-chunk levels as they stand before the last chunk; the tokens of that chunk advance them, and build the levels inside it.  Every level is
// independent of the others: level 0 is the last token alone, level j + 1 (for each set bit j of the last token's position in
// the chunk) starts from zero at the first of its 2^j tokens, takes their writes and then the transitions of the tokens behind
// them, and the levels of earlier chunks take the transitions of all.  fp32 throughout, as the decode kernel steps.
// Level-major states of value heads that are processed as `rep` parts of Vs columns.
//
// A warp holds sixteen columns of one level: a lane has two of them and 32 of the 128 state rows (four lanes a column pair), as pairs of
// rows, so that a token is 96 packed fp32 instructions and four shuffles, without a barrier.  What bounds it is that chain of at most 64
// tokens and the fp32 rate: every live level takes every token of the chunk.  (Four columns a warp with the rows over all 32 lanes
// was bound by the twenty shuffles of a token: T = 827, 59 tokens, 16 heads of 128 x 128 31 us, now 24; T = 777, 9 tokens, 12.1 and 8.6.)
// Four warps a CTA; grid (B*H, 64-column blocks, levels).
constexpr int TAIL_KD = 128, TAIL_COLS = 64;

__global__ void __launch_bounds__(128) gdn_tail_states_kernel(const bf16* __restrict__ kn, const bf16* __restrict__ v, const bf16* __restrict__ beta,
                                                              const float* __restrict__ g, float* __restrict__ states, int T, int H, int K, int Vs,
                                                              int rep, int L, unsigned live) {
    chain_wait();
    __shared__ __align__(16) bf16 sK[CH * TAIL_KD];
    __shared__ __align__(16) float sV[CH * TAIL_COLS];
    __shared__ float sB[CH], sD[CH];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // the live levels first, from the highest down (the lower ones see fewer tokens), then the dead ones, which are cleared: in the
    // order of the levels some SMs got three of the long CTAs and others none
    int lev = -1;
    {
        const unsigned nl = __popc(live), all = L < 32 ? (1u << L) - 1u : ~0u;
        unsigned left = blockIdx.z < nl ? live : all & ~live;
        const unsigned skip = blockIdx.z < nl ? blockIdx.z : blockIdx.z - nl;
        for (unsigned i = 0; i <= skip; ++i) {
            lev = 31 - __clz(left);
            left &= ~(1u << lev);
        }
    }
    const int h = blockIdx.x % H, b = blockIdx.x / H;
    const int m = T - 1, c0 = m & ~(CH - 1), n = m - c0 + 1;
    const int cols = min(TAIL_COLS, Vs - (int)blockIdx.y * TAIL_COLS);
    const int cl = warp * 16 + (lane >> 2) * 2, r = lane & 3;        // the lane's columns in the block; its rows: 8-row groups 4 j + r
    const int V = Vs * rep;                                  // H counts parts of value heads, rep of them in one
    const long bh = (long)b * H + h;
    float* S = states + (bh / rep * L + lev) * (long)K * V + bh % rep * Vs + blockIdx.y * TAIL_COLS + cl;
    // tokens [s0, s1) of the chunk write to this level; [s1, n) only advance it
    int s0 = -1, s1 = 0;
    if (lev == 0) {
        s0 = n - 1;
        s1 = n;
    } else if (lev < INTRA_LEVELS) {
        if (((m & (CH - 1)) >> (lev - 1)) & 1) {
            s0 = ((m & (CH - 1)) >> lev) << lev;
            s1 = s0 + (1 << (lev - 1));
        }
    } else if (lev - INTRA_LEVELS < 25 && ((m >> (lev - 1)) & 1)) {
        s0 = s1 = 0;
    }
    const bool mine = cl < cols;
    f32x2 s[2][16];                                          // [column][pair of rows]
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int row = ((i >> 2) * 4 + r) * 8 + (i & 3) * 2;
        float2 x[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        if (mine && s0 >= 0 && lev >= INTRA_LEVELS)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (row + e < K) x[e] = *reinterpret_cast<const float2*>(S + (long)(row + e) * V);
        s[0][i] = pack2(x[0].x, x[1].x);
        s[1][i] = pack2(x[0].y, x[1].y);
    }
    if (s0 >= 0) {
        const long t0 = (long)b * T + c0;
        for (int e = tid; e < n * (TAIL_KD / 8); e += 128) {
            const int i = e / (TAIL_KD / 8), c8 = (e % (TAIL_KD / 8)) * 8;
            *reinterpret_cast<uint4*>(sK + i * TAIL_KD + c8) = *reinterpret_cast<const uint4*>(kn + ((t0 + i) * H + h) * TAIL_KD + c8);
        }
        for (int e = tid; e < n * (TAIL_COLS / 2); e += 128) {
            const int i = e / (TAIL_COLS / 2), c = (e % (TAIL_COLS / 2)) * 2;
            float2 x = make_float2(0.f, 0.f);
            if (c < cols)
                x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(v + ((t0 + i) * H + h) * Vs + blockIdx.y * TAIL_COLS + c));
            *reinterpret_cast<float2*>(sV + i * TAIL_COLS + c) = x;
        }
        for (int i = tid; i < n; i += 128) {
            sB[i] = __bfloat162float(beta[(t0 + i) * H + h]);
            sD[i] = fexp(g[(t0 + i) * H + h]);
        }
        __syncthreads();
        for (int t = s0; t < n; ++t) {
            f32x2 k[16];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint4 raw = *reinterpret_cast<const uint4*>(sK + t * TAIL_KD + (j * 4 + r) * 8);
                const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) k[j * 4 + u] = pack2(__uint_as_float(w[u] << 16), __uint_as_float(w[u] & 0xffff0000u));
            }
            float d[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                f32x2 a0 = mul2(k[0], s[c][0]), a1 = mul2(k[1], s[c][1]);
#pragma unroll
                for (int i = 2; i < 16; i += 2) {
                    a0 = fma2(k[i], s[c][i], a0);
                    a1 = fma2(k[i + 1], s[c][i + 1], a1);
                }
                const float2 x = unpack2(a0), y = unpack2(a1);
                d[c] = (x.x + x.y) + (y.x + y.y);
            }
#pragma unroll
            for (int w = 1; w < 4; w <<= 1) {
                d[0] += __shfl_xor_sync(0xffffffffu, d[0], w);
                d[1] += __shfl_xor_sync(0xffffffffu, d[1], w);
            }
            const float dec = sD[t], be = sB[t];
            float2 w2 = make_float2(0.f, 0.f);
            if (t < s1) w2 = *reinterpret_cast<const float2*>(sV + t * TAIL_COLS + cl);
            // s' = dec (s - beta k d) + beta k w
            const float x0 = be * (w2.x - dec * d[0]), x1 = be * (w2.y - dec * d[1]);
            const f32x2 dec2 = pack2(dec, dec), x02 = pack2(x0, x0), x12 = pack2(x1, x1);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                s[0][i] = fma2(dec2, s[0][i], mul2(k[i], x02));
                s[1][i] = fma2(dec2, s[1][i], mul2(k[i], x12));
            }
        }
    }
    if (!mine) return;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int row = ((i >> 2) * 4 + r) * 8 + (i & 3) * 2;
        const float2 x = unpack2(s[0][i]), y = unpack2(s[1][i]);
        if (row < K) *reinterpret_cast<float2*>(S + (long)row * V) = make_float2(x.x, y.x);
        if (row + 1 < K) *reinterpret_cast<float2*>(S + (long)(row + 1) * V) = make_float2(x.y, y.y);
    }
}

int gdn_prompt_states_launch(const bf16* kn, const bf16* v, const bf16* beta, const float* g, float* states, int B, int T, int H, int K, int V, int rep,
                             int L, cudaStream_t stream) {
    dim3 grid(B * H, (V + TAIL_COLS - 1) / TAIL_COLS, L);
    launch_chained(gdn_tail_states_kernel, grid, 128, 0, stream, kn, v, beta, g, states, T, H, K, V, rep, L, 1u | (unsigned)(T - 1) << 1);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

}  // namespace llattn

extern "C" {

int llattn_mamba2_prompt_prep(const void* x, const void* dt_raw, const void* dt_bias, int bias_is_f32, const float* A, const void* dl, const void* Lp,
                              int lp_is_f32, const void* q, const void* k, void* v, float* g, void* lambda, void* q_split, void* k_split,
                              int B, int T, int tail, int H, int G, int K, int P, int L, int lambda_mode, void* stream) {
    if (B <= 0 || T < 0 || tail < 0 || T + tail <= 0 || H <= 0 || G <= 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (P <= 0 || P > 256 || P % 8 != 0 || (G * K) % 8 != 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (L <= 0 || L > 64 || lambda_mode < 0 || lambda_mode > 2) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (!x || !dt_raw || !A || !dl || !Lp || !v || !g || !lambda) return LLATTN_ERR_NULL;
    if ((q_split != nullptr) != (k_split != nullptr) || (q_split && (!q || !k))) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {x, v, q_split, k_split}) || (q_split && llattn::misaligned(16, {q, k}))) return LLATTN_ERR_ALIGNMENT;
    using bf = __nv_bfloat16;
    const long rows = (long)B * (T + tail) * H;
    const int lpr = P <= 64 ? 8 : (P <= 128 ? 16 : 32);
    const int qk16 = G * K / 8;
    const long copies = q_split ? 2l * B * (T + tail) * qk16 : 0;
    if (rows * lpr > 0x7fffff00l || copies > 0x7fffff00l) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    const int row_blocks = (int)((rows * lpr + 255) / 256);
    const unsigned grid = row_blocks + (unsigned)((copies + 255) / 256);
    cudaStream_t st = (cudaStream_t)stream;
#define LLATTN_PP(N) llattn::launch_chained(llattn::m2_prompt_prep_kernel<N>, grid, 256, 0, st, (const bf*)x, (const bf*)dt_raw, dt_bias, bias_is_f32, A, (const bf*)dl, Lp, lp_is_f32, (const uint4*)q, (const uint4*)k, (bf*)v, g, (bf*)lambda, (uint4*)q_split, (uint4*)k_split, B, T, tail, H, P, L, lambda_mode, row_blocks, qk16)
    if (lpr == 8) LLATTN_PP(8);
    else if (lpr == 16) LLATTN_PP(16);
    else LLATTN_PP(32);
#undef LLATTN_PP
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int llattn_mamba2_prompt_residual(const void* o, const void* x, const void* D, void* y, int y_is_f32, int B, int T, int tail, int H, int P, void* stream) {
    if (B <= 0 || T <= 0 || tail < 0 || H <= 0 || P <= 0 || P % 8 != 0 || (long)B * T * H * P > 0x7fffff00l * 8) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (!o || !y || !D || !x) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {o, x, y})) return LLATTN_ERR_ALIGNMENT;
    using bf = __nv_bfloat16;
    const unsigned grid = (unsigned)(((long)B * T * H * (P / 8) + 255) / 256);
    cudaStream_t st = (cudaStream_t)stream;
    if (y_is_f32) llattn::launch_chained(llattn::m2_prompt_residual_kernel<true>, grid, 256, 0, st, (const bf*)o, (const bf*)x, D, y, B, T, tail, H, P);
    else llattn::launch_chained(llattn::m2_prompt_residual_kernel<false>, grid, 256, 0, st, (const bf*)o, (const bf*)x, D, y, B, T, tail, H, P);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int llattn_gdn_prompt_prep(const void* q, const void* k, const void* v, const void* beta, const float* g, const void* lambda,
                           void* qn, void* kn, void* v_split, void* beta_split, float* g_split, void* lambda_split,
                           int B, int T, int tail, int H, int G, int K, int K_out, int V, int rep, int L, float scale, float lambda_mul, void* stream) {
    if (B <= 0 || T < 0 || tail < 0 || T + tail <= 0 || H <= 0 || G <= 0 || H % G != 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (K <= 0 || K % 8 != 0 || K_out < K || K_out > 128 || K_out % 8 != 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (V <= 0 || rep <= 0 || V % (8 * rep) != 0 || L <= 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if ((long)B * (T + tail) * H * rep > 0x7fffff00l) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (!q || !k || !qn || !kn || (v_split && !v) || (lambda_split && !lambda) || (g_split && (!g || !beta || !beta_split))) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {q, k, qn, kn, v_split}) || (v_split && llattn::misaligned(16, {v}))) return LLATTN_ERR_ALIGNMENT;
    using bf = __nv_bfloat16;
    llattn::GdnPrepArgs a{(const bf*)q, (const bf*)k, (const bf*)v, (const bf*)beta, g, (const bf*)lambda, (bf*)qn, (bf*)kn, (bf*)v_split,
                          (bf*)beta_split, g_split, (bf*)lambda_split, B, T, tail, H, G, K, K_out, V, rep, L, scale, lambda_mul};
    const unsigned grid = (unsigned)(((long)B * (T + tail) * H * rep + 15) / 16);
    llattn::launch_chained(llattn::gdn_prompt_prep_kernel, grid, 256, 0, (cudaStream_t)stream, a);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

}  // extern "C"
