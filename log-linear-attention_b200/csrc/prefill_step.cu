// Prefill hand-off and single-token decode step of log-linear Mamba-2 for sm_100a.
//
// Reference being replaced: the level-state side of hattention_prefill (hattention/kernel.py:470-560:
// chunk_fwd_kernel_h's final states `ht` for the inter-chunk levels plus postprocess_prefill_hstate_,
// :378-466, for the levels inside the last chunk) and hattention_step (kernel.py:563-633 with
// HState.cascade_weak / insert / step_output, hattention/recurrent.py:42-54, 79-98, 134-166).
//
// After m + 1 = T tokens the state of level 0 is k_m v_m^T, and for every set bit j of m, level j + 1
// holds the 2^j tokens that follow the buckets of the higher set bits (oldest tokens in the highest
// level):   S_l = sum_{s in bucket l} exp(sum_{r = s+1 .. m} g_r) k_s v_s^T .
//   mamba2_final_state_kernel : one CTA per (batch, head, level) sums its bucket with warp-level MMA
//       (decay folded into v), 64 tokens at a time from the end of the bucket backwards.
//   mamba2_prompt_state_kernel : the same states level-major, with the segment summaries of the forward call
//   mamba2_tail_intra_kernel, mamba2_tail_levels_kernel : the tokens of a prompt behind its last whole chunk
//   mamba2_step_kernel : one CTA per (batch, head); the host passes the carry level j of the cascade
//       (levels 0..j are summed into level j); then every level is decayed by exp(g), level 0 becomes
//       k v^T, and o = q . sum_l lambda_l S_l.  HBM-bound: reads and writes L*K*V floats per head.
#include "rowwise.cuh"
#include "llattn_mamba2.h"
#include "../../include/llattn.h"

namespace llattn {

template <int KD, int VD>
__global__ void __launch_bounds__(256, 1) mamba2_final_state_kernel(const bf16* __restrict__ k, const bf16* __restrict__ v,
                                                                    const float* __restrict__ g, float* __restrict__ states,
                                                                    int B, int T, int H, int G, int L) {
    chain_wait();
    constexpr int LDK = KD + PAD, LDV = VD + PAD;
    constexpr int MT = KD / 128;                         // 16-row tiles of the K x V result per warp (8 warps)
    static_assert(KD % 128 == 0 || KD == 64, "K rows are split over the warps");
    __shared__ __align__(16) bf16 sK[CH * LDK];
    __shared__ __align__(16) bf16 sVs[CH * LDV];
    __shared__ float sDec[CH];
    __shared__ float sRed[8];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int lev = blockIdx.y;
    const int h = blockIdx.x % H, b = blockIdx.x / H;
    const int grp = h / (H / G);
    const int m = T - 1;
    // bucket of this level
    int s0 = 0, s1 = 0;
    if (lev == 0) {
        s0 = m;
        s1 = m + 1;
    } else if (lev - 1 < 31 && ((m >> (lev - 1)) & 1)) {
        s0 = (m >> lev) << lev;                          // tokens taken by the higher set bits
        s1 = s0 + (1 << (lev - 1));
    }
    float* out = states + ((long)(b * H + h) * KD * VD) * L + lev;
    if (s1 == s0) {
        for (int e = tid; e < KD * VD; e += 256) out[(long)e * L] = 0.f;
        return;
    }
    // decay from the end of the bucket to the last token: sum_{r = s1 .. m} g_r
    float part = 0.f;
    for (int r = s1 + tid; r <= m; r += 256) part += g[((long)b * T + r) * H + h];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) part += __shfl_xor_sync(0xffffffffu, part, d);
    if (lane == 0) sRed[warp] = part;
    __syncthreads();
    float after = 0.f;
    for (int w = 0; w < 8; ++w) after += sRed[w];

    // warps split the K rows: K = 128 -> 16 rows each; K = 64 -> warps 0..3 take 16 rows each
    const bool active = (KD >= 128) || warp < 4;
    constexpr int MTW = (KD >= 128) ? MT : 1;
    float acc[MTW][VD / 8][4];
    zero_acc(acc);
    const int lr = lane >> 2, lc2 = (lane & 3) * 2;
    for (int e1 = s1; e1 > s0; e1 -= CH) {
        const int a = max(e1 - CH, s0);                  // tile [a, e1), up to 64 tokens, rows beyond are zero
        const int n = e1 - a;
        __syncthreads();                                 // previous tile consumed
        // in-tile decay: token a + i gets exp(after + sum_{r = a+i+1 .. e1-1} g_r)
        if (warp == 0) {
            const int i0 = CH - 1 - 2 * lane, i1 = CH - 2 - 2 * lane;      // reversed order
            float x0 = (i0 + 1 < n) ? g[((long)b * T + a + i0 + 1) * H + h] : 0.f;
            float x1 = (i1 + 1 < n) ? g[((long)b * T + a + i1 + 1) * H + h] : 0.f;
            warp_cumsum64(x0, x1, lane);
            sDec[i0] = (i0 < n) ? fexp(after + x0) : 0.f;
            sDec[i1] = (i1 < n) ? fexp(after + x1) : 0.f;
        }
        for (int e = tid; e < CH * (KD / 8); e += 256) {
            const int i = e / (KD / 8), c8 = (e % (KD / 8)) * 8;
            uint4 x = make_uint4(0, 0, 0, 0);
            if (i < n) x = *reinterpret_cast<const uint4*>(k + (((long)b * T + a + i) * G + grp) * KD + c8);
            *reinterpret_cast<uint4*>(sK + i * LDK + c8) = x;
        }
        __syncthreads();
        for (int e = tid; e < CH * (VD / 8); e += 256) {
            const int i = e / (VD / 8), c8 = (e % (VD / 8)) * 8;
            uint4 x = make_uint4(0, 0, 0, 0);
            if (i < n) {
                x = *reinterpret_cast<const uint4*>(v + (((long)b * T + a + i) * H + h) * VD + c8);
                const float d = sDec[i];
                uint32_t* xw = reinterpret_cast<uint32_t*>(&x);
#pragma unroll
                for (int q4 = 0; q4 < 4; ++q4) {
                    const __nv_bfloat162 t2 = *reinterpret_cast<const __nv_bfloat162*>(&xw[q4]);
                    xw[q4] = pack_bf16(__bfloat162float(t2.x) * d, __bfloat162float(t2.y) * d);
                }
            }
            *reinterpret_cast<uint4*>(sVs + i * LDV + c8) = x;
        }
        __syncthreads();
        if (active) warp_gemm<MTW, VD / 16, true, true>(acc, sK, LDK, warp * 16 * MTW, sVs, LDV, 0, CH, lane);
        // decay accumulated over this tile for the next (earlier) tile: sum_{r = a .. e1-1} g_r
        float tile = 0.f;
        if (warp == 0) {
            float x = 0.f;
            for (int i = lane; i < n; i += 32) x += g[((long)b * T + a + i) * H + h];
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
            if (lane == 0) sRed[0] = x;
        }
        __syncthreads();
        tile = sRed[0];
        after += tile;
    }
    if (active) {
#pragma unroll
        for (int mt = 0; mt < MTW; ++mt)
#pragma unroll
            for (int nt = 0; nt < VD / 8; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int row = warp * 16 * MTW + mt * 16 + lr + (e >> 1) * 8, col = nt * 8 + lc2 + (e & 1);
                    out[((long)row * VD + col) * L] = acc[mt][nt][e];
                }
    }
}

// The same states level-major (B,H,L,K,V), after T whole-chunk tokens.  One CTA per (batch, head, level).  With tokens to follow (n > 0) the
// states are the ones that the next token finds once the cascade has run: level j + 1 holds 2^j tokens for every set bit j of T, the levels
// inside a chunk are left to the kernel of those tokens.
// A bucket is walked in blocks of at most 256 tokens from its end: the decays of a block come from one scan over its 256 values of g, and
// its 64-token tiles are copied two deep, so that a tile costs one product behind one barrier.  (A tile that fetched its own decays and
// loaded k, then v, cost three dependent trips to memory: 24 us for a 1000-token prompt of 48 heads, most of it the four tiles of the level
// that holds 256 tokens.)  With the segment summaries of the forward call on the same tensors (seg_F, seg_D; null when there is one
// segment) a level of 2^j segments is an element-wise pass over 2^j summaries instead of 2^(j+3) products.
template <int KD>
struct PromptStateSmem {
    static constexpr int LDK = KD + PAD, LDV = 64 + PAD;
    static constexpr size_t k_off = 0, v_off = 2ull * CH * LDK * 2, dec_off = v_off + 2ull * CH * LDV * 2, red_off = dec_off + 256 * 4, total = red_off + 64;
};

template <int KD>
__global__ void __launch_bounds__(256) mamba2_prompt_state_kernel(const bf16* __restrict__ k, const bf16* __restrict__ v, const float* __restrict__ g,
                                                                  float* __restrict__ states, const float* __restrict__ seg_F,
                                                                  const float* __restrict__ seg_D, int T, int n, int H, int G, int L) {
    chain_wait();
    using SM = PromptStateSmem<KD>;
    constexpr int VD = 64, LDK = SM::LDK, LDV = SM::LDV, KV = KD * VD, SEG = 512;
    constexpr int MT = KD / 64, NPW = VD / 32;           // a warp: 16 MT rows x 32 columns (4 x 2 warps)
    extern __shared__ __align__(16) unsigned char smem[];
    bf16* sK = reinterpret_cast<bf16*>(smem + SM::k_off);
    bf16* sV = reinterpret_cast<bf16*>(smem + SM::v_off);
    float* sDec = reinterpret_cast<float*>(smem + SM::dec_off);
    float* sRed = reinterpret_cast<float*>(smem + SM::red_off);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int lev = blockIdx.y, h = blockIdx.x % H, b = blockIdx.x / H, grp = h / (H / G);
    const long bh = blockIdx.x;
    const int m = T - 1, bits = n > 0 ? T : m;
    if (n > 0 && lev < INTRA_LEVELS) return;
    int s0 = 0, s1 = 0;
    if (lev == 0) {
        s0 = m;
        s1 = m + 1;
    } else if (lev - 1 < 31 && ((bits >> (lev - 1)) & 1)) {
        s0 = (bits >> lev) << lev;
        s1 = s0 + (1 << (lev - 1));
    }
    float* out = states + (bh * L + lev) * KV;
    if (s1 == s0) {
        for (int e = tid * 4; e < KV; e += 1024) *reinterpret_cast<float4*>(out + e) = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    auto block_sum = [&](float x) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
        if (lane == 0) sRed[warp] = x;
        __syncthreads();
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += sRed[w];
        __syncthreads();
        return t;
    };
    const float* gb = g + (long)b * T * H + h;
    // the last segment of a sequence has no summary: its tokens are walked, and a bucket that ends with it takes the others behind that
    const int rl = m / SEG, NS = (T + SEG - 1) / SEG;
    const bool sums = seg_F != nullptr && s1 - s0 >= SEG;
    const int w0 = sums ? max(s0, rl * SEG) : s0;          // first token of the walk
    auto add_segments = [&](bool have) {
        // behind the bucket: whole segments up to the one of the last token, then that segment's tokens up to the last one
        const int r0 = s0 / SEG, r1 = min(s1 / SEG, rl);
        const float *D = seg_D + bh * NS, *F = seg_F + bh * NS * KV;
        float part = 0.f;
        for (int r = r1 + tid; r < rl; r += 256) part += D[r];
        for (int t = rl * SEG + tid; t <= m; t += 256) part += gb[(long)t * H];
        float after = block_sum(part);
        float4 acc[KV / 1024];
#pragma unroll
        for (int i = 0; i < KV / 1024; ++i)
            acc[i] = have ? *reinterpret_cast<const float4*>(out + i * 1024 + tid * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = r1 - 1; r >= r0; --r) {
            const float w = fexp(after);
#pragma unroll
            for (int i = 0; i < KV / 1024; ++i) {
                const float4 f = *reinterpret_cast<const float4*>(F + (long)r * KV + i * 1024 + tid * 4);
                acc[i].x += w * f.x; acc[i].y += w * f.y; acc[i].z += w * f.z; acc[i].w += w * f.w;
            }
            after += D[r];
        }
#pragma unroll
        for (int i = 0; i < KV / 1024; ++i) *reinterpret_cast<float4*>(out + i * 1024 + tid * 4) = acc[i];
    };
    if (sums && w0 >= s1) return add_segments(false);
    const int wr = warp & 3, wc = warp >> 2;
    float acc[MT][2 * NPW][4];
    zero_acc(acc);
    // tokens e1 - 1 downwards in tiles of 64; rows of a tile beyond its tokens are zero
    uint4 vr[2];
    auto fetch = [&](int a, int e1, int st) {
        const int n = e1 - a;
        for (int e = tid; e < CH * (KD / 8); e += 256) {
            const int i = e / (KD / 8), c8 = (e % (KD / 8)) * 8;
            bf16* dst = sK + st * CH * LDK + i * LDK + c8;
            if (i < n) cp_async16(dst, k + (((long)b * T + a + i) * G + grp) * KD + c8);
            else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
        }
        cp_async_commit();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = (tid + u * 256) / (VD / 8), c8 = ((tid + u * 256) % (VD / 8)) * 8;
            vr[u] = i < n ? *reinterpret_cast<const uint4*>(v + (((long)b * T + a + i) * H + h) * VD + c8) : make_uint4(0, 0, 0, 0);
        }
    };
    float part = 0.f;
    fetch(max(s1 - CH, w0), s1, 0);
    for (int r = s1 + tid; r <= m; r += 256) part += gb[(long)r * H];
    float after = block_sum(part);
    int st = 0;
    for (int e2 = s1; e2 > w0; e2 -= 256) {
        const int a2 = max(e2 - 256, w0), n2 = e2 - a2;
        // token a2 + i of the block: exp(after + sum_{r = a2+i+1 .. e2-1} g_r), by a scan from the end (thread j holds token n2 - 1 - j)
        const int i = n2 - 1 - tid;
        float x = (tid >= 1 && i >= 0) ? gb[(long)(a2 + i + 1) * H] : 0.f;
        const float first = gb[(long)a2 * H];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float t = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += t;
        }
        if (lane == 31) sRed[warp] = x;
        __syncthreads();
        float all = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            if (w < warp) x += sRed[w];
            all += sRed[w];
        }
        if (i >= 0) sDec[i] = fexp(after + x);
        after += all + first;
        __syncthreads();
        for (int e1 = e2; e1 > a2; e1 -= CH) {
            const int a = max(e1 - CH, w0), n = e1 - a;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int row = (tid + u * 256) / (VD / 8), c8 = ((tid + u * 256) % (VD / 8)) * 8;
                const float d = row < n ? sDec[a - a2 + row] : 0.f;
                uint32_t* xw = reinterpret_cast<uint32_t*>(&vr[u]);
#pragma unroll
                for (int q4 = 0; q4 < 4; ++q4) {
                    const __nv_bfloat162 t2 = *reinterpret_cast<const __nv_bfloat162*>(&xw[q4]);
                    xw[q4] = pack_bf16(__bfloat162float(t2.x) * d, __bfloat162float(t2.y) * d);
                }
                *reinterpret_cast<uint4*>(sV + st * CH * LDV + row * LDV + c8) = vr[u];
            }
            cp_async_wait<0>();
            __syncthreads();
            if (a > w0) fetch(max(a - CH, w0), a, st ^ 1);
            warp_gemm<MT, NPW, true, true>(acc, sK + st * CH * LDK, LDK, wr * 16 * MT, sV + st * CH * LDV, LDV, wc * 32, CH, lane);
            st ^= 1;
        }
    }
    const int lr = lane >> 2, lc2 = (lane & 3) * 2;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < 2 * NPW; ++nt)
#pragma unroll
            for (int e = 0; e < 4; e += 2)
                *reinterpret_cast<float2*>(out + (wr * 16 * MT + mt * 16 + lr + (e >> 1) * 8) * VD + wc * 32 + nt * 8 + lc2) =
                    make_float2(acc[mt][nt][e], acc[mt][nt][e + 1]);
    if (sums) {
        __syncthreads();
        add_segments(true);
    }
}

// The n < 64 tokens behind the last whole chunk of a prompt (its tail): their outputs, and the level states after the last of them.
// Everything that a decode step keeps in fp32 is fp32 here too: token i reads the states that stood before the first of these tokens,
// decayed, and the other tokens up to itself,
//     o_i = sum_l lambda_il exp(G_i) q_i S_l + sum_{j <= i} lambda_{i, level_of(i, j)} exp(G_i - G_j) (q_i k_j) v_j
// with G the cumulative log decay of these tokens.  q and k are bf16, so q k^T on the tensor cores has exact products and fp32 sums;
// q S_l takes S as three bf16 terms that hold its 24 bits; the rest is fp32 arithmetic.
//
// Two kernels, because the second sum and the levels that these tokens build need nothing of the whole chunks: mamba2_tail_intra_kernel can run
// while their segment summaries are made, and the kernel behind the states is short.  As one kernel behind the states it shared the
// SMs that the output's kernel left free and outlasted it: T = 1000, 48 heads, 38 us instead of 11 and 14, 74 us for the call instead of 58.
// A CTA owns TL of the 64 columns of one (batch, head); what bounds both is a chain of trips to L2 and of short products.
// Whole heads (TL = 64) do what the columns share once, sixteen columns a CTA shorten the chain of few heads: the call at 48 heads, T = 1500 74.5 us with 16 and
// 84.5 with 64, T = 3000 119 and 136; at 128 heads, T = 700 101.7 and 95.5; at 192, T = 100 75.9 and 64.4, T = 400 100 and 90.7.  Hence 96 heads.
constexpr int TL_WARPS = 8, TL_THREADS = 32 * TL_WARPS;

// a pair of fp32 values as three pairs of bf16 ones: the upper halves of the values, of what these leave, and the rest; an infinity stays one
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    auto cut = [](float v) { return __uint_as_float(__float_as_uint(v) & 0xffff0000u); };
    hi = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
    x = isinf(x) ? 0.f : x - cut(x);
    y = isinf(y) ? 0.f : y - cut(y);
    mid = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
    lo = pack_bf16(x - cut(x), y - cut(y));
}

// sums[i]: log decay of the tokens up to i; with `after`, of those behind token i.  resets[i]: how many of them decay to nothing (log decay -inf): these
// are counted and not summed, because a step forgets what was before it and goes on.  One warp.
__device__ __forceinline__ void tail_decays(const float* g, long stride, int n, bool after, float* sums, float* resets, int lane) {
    float x[2], c[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int i = after ? n - (2 * lane + u) : 2 * lane + u;
        x[u] = i >= 0 && i < n ? g[i * stride] : 0.f;
        c[u] = x[u] == -INFINITY ? 1.f : 0.f;
        if (c[u] != 0.f) x[u] = 0.f;
    }
    warp_cumsum64(x[0], x[1], lane);
    warp_cumsum64(c[0], c[1], lane);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int i = after ? n - 1 - (2 * lane + u) : 2 * lane + u;
        if (i >= 0) {
            sums[i] = x[u];
            resets[i] = c[u];
        }
    }
}
// rows of q or k of the tail into shared memory, zeros behind them
template <int KD>
__device__ __forceinline__ void tail_rows(bf16* dst, const bf16* src, long stride, int n, int tid) {
#pragma unroll
    for (int u = 0; u < CH * (KD / 8) / TL_THREADS; ++u) {
        const int e = tid + u * TL_THREADS, i = e / (KD / 8), c8 = (e % (KD / 8)) * 8;
        if (i < n) cp_async16(dst + i * (KD + PAD) + c8, src + i * stride + c8);
        else *reinterpret_cast<uint4*>(dst + i * (KD + PAD) + c8) = make_uint4(0, 0, 0, 0);
    }
}
// four outputs of a token, rounded to bf16, with the residual
__device__ __forceinline__ void tail_output(const Mamba2Tail& a, const float (&r)[4], long at, int h) {
    const float d = a.D ? load_param(a.D, h, a.d_f32) : 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float v = round_bf16(r[e]), xd = a.D ? __bfloat162float(a.x[at + e]) * d : 0.f;
        if (a.D && a.d_f32) reinterpret_cast<float*>(a.y)[at + e] = v + xd;
        else reinterpret_cast<bf16*>(a.y)[at + e] = __float2bfloat16(a.D ? v + round_bf16(xd) : v);
    }
}
// what a CTA works on
struct TailPlace {
    int c0, h, b, grp;
    long tok0, y0;             // first token of the tail in the split tensors; in y
    __device__ TailPlace(const Mamba2Tail& a, int B, int TL) {
        const int ncb = 64 / TL;
        c0 = blockIdx.x % ncb * TL;
        h = (blockIdx.x / ncb) % a.H;
        b = blockIdx.x / (ncb * a.H);
        grp = h / (a.H / a.G);
        tok0 = (long)B * a.T0 + (long)b * a.n;
        y0 = (long)b * (a.T0 + a.n) + a.T0;
    }
};

template <int KD, int TL>
struct TailIntraSmem {
    static constexpr int LDK = KD + PAD, LDP = CH + 4, LDD = TL + PAD;
    static constexpr size_t q_off = 0, k_off = q_off + 2ull * CH * LDK, p_off = k_off + 2ull * CH * LDK, v_off = p_off + 4ull * CH * LDP,
                            d_off = v_off + 4ull * CH * TL, g_off = d_off + 3ull * 2 * CH * LDD, lam_off = g_off + 16ull * CH,
                            total = lam_off + 4ull * CH * INTRA_LEVELS;
};

// the tokens among themselves: their part of the outputs (all of it without a whole chunk before them), the levels that they build
template <int KD, int TL>
__global__ void __launch_bounds__(TL_THREADS) mamba2_tail_intra_kernel(const __grid_constant__ Mamba2Tail a, int B) {
    chain_wait();
    using SM = TailIntraSmem<KD, TL>;
    constexpr int VD = 64, LDK = SM::LDK, LDP = SM::LDP, LDD = SM::LDD;
    extern __shared__ __align__(16) unsigned char smem[];
    bf16* sQ = reinterpret_cast<bf16*>(smem + SM::q_off);
    bf16* sK = reinterpret_cast<bf16*>(smem + SM::k_off);
    float* sP = reinterpret_cast<float*>(smem + SM::p_off);
    float* sV = reinterpret_cast<float*>(smem + SM::v_off);
    bf16* sD = reinterpret_cast<bf16*>(smem + SM::d_off);             // three terms of v decayed to the last token, [term][token][column]
    float *sG = reinterpret_cast<float*>(smem + SM::g_off), *sR = sG + CH, *sE = sR + CH, *sF = sE + CH;
    float* sLam = reinterpret_cast<float*>(smem + SM::lam_off);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane >> 2, lc2 = (lane & 3) * 2;
    const TailPlace w(a, B, TL);
    const int n = a.n, m = n - 1;
    tail_rows<KD>(sQ, a.q + (w.tok0 * a.G + w.grp) * KD, (long)a.G * KD, n, tid);
    tail_rows<KD>(sK, a.k + (w.tok0 * a.G + w.grp) * KD, (long)a.G * KD, n, tid);
    cp_async_commit();
    const int ti = tid / 4, tc4 = (tid & 3) * 4;           // token and first column of a thread
    {
        Packed<4> x[TL / 16];
#pragma unroll
        for (int u = 0; u < TL / 16; ++u) x[u].load_if(a.v + ((w.tok0 + ti) * a.H + w.h) * VD + w.c0 + tc4 + u * 16, true, ti < n);
        const bf16* lp = a.lam + ((w.tok0 + ti) * a.H + w.h) * a.lam_L;
        float lam[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) lam[u] = ti < n && (tid & 3) + 4 * u < min(a.L, INTRA_LEVELS) ? __bfloat162float(lp[(tid & 3) + 4 * u]) : 0.f;
#pragma unroll
        for (int u = 0; u < TL / 16; ++u) *reinterpret_cast<float4*>(sV + ti * TL + tc4 + u * 16) = make_float4(x[u][0], x[u][1], x[u][2], x[u][3]);
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if ((tid & 3) + 4 * u < INTRA_LEVELS) sLam[ti * INTRA_LEVELS + (tid & 3) + 4 * u] = lam[u];
    }
    if (warp == 0) tail_decays(a.g + w.tok0 * a.H + w.h, a.H, n, false, sG, sR, lane);
    if (warp == 1) {
        tail_decays(a.g + w.tok0 * a.H + w.h, a.H, n, true, sE, sF, lane);      // summed from the end, where the weights are large
        __syncwarp();
        for (int i = lane; i < n; i += 32) sE[i] = sF[i] == 0.f ? fexp(sE[i]) : 0.f;
    }
    cp_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (int c = tc4; c < TL; c += 16) {
        const float4 x = *reinterpret_cast<const float4*>(sV + ti * TL + c);
        const float e = ti < n ? sE[ti] : 0.f;
        uint32_t t0[3], t1[3];
        split3(x.x * e, x.y * e, t0[0], t0[1], t0[2]);
        split3(x.z * e, x.w * e, t1[0], t1[1], t1[2]);
#pragma unroll
        for (int u = 0; u < 3; ++u) *reinterpret_cast<uint2*>(sD + (u * CH + ti) * LDD + c) = make_uint2(t0[u], t1[u]);
    }
    // ---- weights: a tile of 16 tokens x half of the 64 a warp
    const int r0 = (warp & 3) * 16, k0 = (warp >> 2) * 32;
    if (r0 < n) {
        float acc[1][4][4];
        zero_acc(acc);
        if (k0 <= r0 + 15) warp_gemm<1, 2, false, false>(acc, sQ, LDK, r0, sK, LDK, k0, KD, lane);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = r0 + lr + (e >> 1) * 8, j = k0 + nt * 8 + lc2 + (e & 1);
                if (k0 + nt * 8 > r0 + 15) sP[i * LDP + j] = 0.f;              // above the diagonal
                else sP[i * LDP + j] = i < n && j <= i && sR[i] == sR[j] ? sLam[i * INTRA_LEVELS + level_of(i, j)] * fexp(sG[i] - sG[j]) * acc[0][nt][e] : 0.f;
            }
    }
    __syncthreads();
    // ---- outputs: a token and four columns of every sixteen a thread
    if (ti < n) {
        float r[TL / 16][4] = {};
        for (int j = 0; j <= ti; j += 4) {                 // weights beyond ti are zero
            const float4 p = *reinterpret_cast<const float4*>(sP + ti * LDP + j);
            const float pw[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int c = 0; c < TL / 16; ++c) {
                    const float4 x = *reinterpret_cast<const float4*>(sV + (j + u) * TL + tc4 + c * 16);
                    r[c][0] += pw[u] * x.x; r[c][1] += pw[u] * x.y; r[c][2] += pw[u] * x.z; r[c][3] += pw[u] * x.w;
                }
        }
#pragma unroll
        for (int c = 0; c < TL / 16; ++c) {
            const int col = w.c0 + tc4 + c * 16;
            if (a.T0 > 0) *reinterpret_cast<float4*>(a.part + (((long)w.b * n + ti) * a.H + w.h) * VD + col) = make_float4(r[c][0], r[c][1], r[c][2], r[c][3]);
            else tail_output(a, r[c], ((w.y0 + ti) * a.H + w.h) * VD + col, w.h);
        }
    }
    // ---- the levels inside the chunk, k^T times the decayed v of a level's tokens, sixteen state rows a warp; without a whole chunk before
    // them the others are empty
    for (int rt = warp; rt < KD / 16; rt += TL_WARPS)
        for (int l = 0; l < (a.T0 > 0 ? min(a.L, INTRA_LEVELS) : a.L); ++l) {
            int s0 = 0, s1 = 0;
            if (l == 0) {
                s0 = m;
                s1 = n;
            } else if (l < INTRA_LEVELS && ((m >> (l - 1)) & 1)) {
                s0 = (m >> l) << l;
                s1 = s0 + (1 << (l - 1));
            }
            float acc[TL / 8][4] = {};
            for (int kt = s0 & ~15; kt < s1; kt += 16) {
                uint32_t af[4];
                ldsm_x4_t(af, sK + (kt + (lane & 7) + (lane >> 4) * 8) * LDK + rt * 16 + ((lane >> 3) & 1) * 8);
                // tokens of the tile outside the level: kt + lc2 + {0, 1} in the first two registers, + 8 in the others
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int t = kt + lc2 + u * 8;
                    const uint32_t mask = (t >= s0 && t < s1 ? 0xffffu : 0u) | (t + 1 >= s0 && t + 1 < s1 ? 0xffff0000u : 0u);
                    af[2 * u] &= mask;
                    af[2 * u + 1] &= mask;
                }
#pragma unroll
                for (int u = 2; u >= 0; --u)
#pragma unroll
                    for (int c = 0; c < TL / 16; ++c) {
                        uint32_t bf[4];
                        ldsm_x4_t(bf, sD + (u * CH + kt + (lane & 15)) * LDD + c * 16 + (lane >> 4) * 8);
                        mma16816(acc[2 * c], af, bf[0], bf[1]);
                        mma16816(acc[2 * c + 1], af, bf[2], bf[3]);
                    }
            }
            float* P = a.states + ((((long)w.b * a.H + w.h) * a.L + l) * KD + rt * 16 + lr) * VD + w.c0 + lc2;
#pragma unroll
            for (int nt = 0; nt < TL / 8; ++nt)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) *reinterpret_cast<float2*>(P + (long)hh * 8 * VD + nt * 8) = make_float2(acc[nt][2 * hh], acc[nt][2 * hh + 1]);
        }
}

template <int KD, int TL>
struct TailLevelsSmem {
    static constexpr int LDK = KD + PAD, LDO = 8;
    static constexpr size_t q_off = 0, o_off = q_off + 2ull * CH * LDK, g_off = o_off + 4ull * CH * LDO * TL_WARPS, total = g_off + 8ull * CH;
};

// the states before the tail: left behind decayed, and their part of the outputs, which are complete then.  The levels go over the warps: warp w
// reads eight columns of a level once, and multiplies them with every token: the columns 8 (w % NT) .. of every (8 / NT)-th level, NT = TL / 8.
template <int KD, int TL>
__global__ void __launch_bounds__(TL_THREADS, 2) mamba2_tail_levels_kernel(const __grid_constant__ Mamba2Tail a, int B) {
    chain_wait();
    using SM = TailLevelsSmem<KD, TL>;
    constexpr int VD = 64, LDK = SM::LDK, LDO = SM::LDO, KS = KD / 16, NT = TL / 8, LW = TL_WARPS / NT;
    extern __shared__ __align__(16) unsigned char smem[];
    bf16* sQ = reinterpret_cast<bf16*>(smem + SM::q_off);
    float* sO = reinterpret_cast<float*>(smem + SM::o_off);           // [warp][token][column of its eight]
    float *sG = reinterpret_cast<float*>(smem + SM::g_off), *sR = sG + CH;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane >> 2, lc2 = (lane & 3) * 2;
    const TailPlace w(a, B, TL);
    const int n = a.n, tiles = (n + 15) / 16, nt = warp % NT;
    const unsigned high = (unsigned)a.T0 >> (INTRA_LEVELS - 1);
    float* S = a.states + ((long)w.b * a.H + w.h) * a.L * KD * VD + w.c0;
    int lev = -1;
    unsigned left = high;
    auto next_level = [&](int skip) {
        for (; skip > 0; --skip) left &= left - 1;
        lev = left ? INTRA_LEVELS + __ffs(left) - 1 : -1;
    };
    float s[KS][4];
    auto at = [&](int kk, int e) { return ((long)lev * KD + kk * 16 + lc2 + (e & 1) + (e >> 1) * 8) * VD + nt * 8 + lr; };
    auto load_level = [&]() {
#pragma unroll
        for (int kk = 0; kk < KS; ++kk)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[kk][e] = S[at(kk, e)];
    };
    next_level(warp / NT);
    if (lev >= 0) load_level();
    tail_rows<KD>(sQ, a.q + (w.tok0 * a.G + w.grp) * KD, (long)a.G * KD, n, tid);
    cp_async_commit();
    const int ti = tid / 4, tc4 = (tid & 3) * 4;
    if (warp == 0) {
        tail_decays(a.g + w.tok0 * a.H + w.h, a.H, n, false, sG, sR, lane);
        __syncwarp();
        for (int i = lane; i < n; i += 32) sG[i] = sR[i] == 0.f ? fexp(sG[i]) : 0.f;     // decay from before the first token
    }
    cp_async_wait<0>();
    __syncthreads();
    float* oW = sO + (long)warp * CH * LDO;
    const bf16* lam = a.lam + (w.tok0 * a.H + w.h) * a.lam_L;
    for (bool first = true; lev >= 0; first = false) {
        float wt[4][2];
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int i = t * 16 + lr + hh * 8;
                wt[t][hh] = i < n ? __bfloat162float(lam[(long)i * a.H * a.lam_L + lev]) * sG[i] : 0.f;
            }
        const float dn = sG[n - 1];
#pragma unroll
        for (int kk = 0; kk < KS; ++kk)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[at(kk, e)] = dn * s[kk][e];
        float acc[4][4] = {};
#pragma unroll
        for (int kk = 0; kk < KS; ++kk) {
            uint32_t hi[2], mid[2], lo[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) split3(s[kk][2 * u], s[kk][2 * u + 1], hi[u], mid[u], lo[u]);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                if (t >= tiles) continue;
                uint32_t af[4];
                ldsm_x4(af, sQ + (t * 16 + (lane & 15)) * LDK + kk * 16 + (lane >> 4) * 8);
                mma16816(acc[t], af, lo[0], lo[1]);
                mma16816(acc[t], af, mid[0], mid[1]);
                mma16816(acc[t], af, hi[0], hi[1]);
            }
        }
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int i = t * 16 + lr + hh * 8;
                if (i >= n) continue;
                float2* dst = reinterpret_cast<float2*>(oW + i * LDO + lc2);
                float2 r = first ? make_float2(0.f, 0.f) : *dst;
                r.x += wt[t][hh] * acc[t][2 * hh];
                r.y += wt[t][hh] * acc[t][2 * hh + 1];
                *dst = r;
            }
        next_level(LW);
        if (lev >= 0) load_level();
    }
    __syncthreads();
    if (ti < n)
#pragma unroll
        for (int c = tc4; c < TL; c += 16) {
            float r[4] = {};
            const int used = min(LW, __popc(high));        // of the warps of eight columns: those that had a level
            for (int u = 0; u < used; ++u) {
                const float4 x = *reinterpret_cast<const float4*>(sO + ((NT * u + (c >> 3)) * CH + ti) * LDO + (c & 7));
                r[0] += x.x; r[1] += x.y; r[2] += x.z; r[3] += x.w;
            }
            const float4 x = *reinterpret_cast<const float4*>(a.part + (((long)w.b * n + ti) * a.H + w.h) * VD + w.c0 + c);
            r[0] += x.x; r[1] += x.y; r[2] += x.z; r[3] += x.w;
            tail_output(a, r, ((w.y0 + ti) * a.H + w.h) * VD + w.c0 + c, w.h);
        }
}

// one decode step for one (batch, head) per CTA; thread t owns column t % VD and rows t / VD, + 256 / VD, ...
template <int MAXL>
__global__ void __launch_bounds__(256) mamba2_step_kernel(float* __restrict__ states, const bf16* __restrict__ q, const bf16* __restrict__ k,
                                                          const bf16* __restrict__ v, const float* __restrict__ g, const bf16* __restrict__ lam,
                                                          bf16* __restrict__ o, int H, int G, int K, int V, int L, int carry) {
    chain_wait();
    extern __shared__ float sh[];                        // q[K] | k[K] | partial outputs [256]
    float* sQ = sh;
    float* sKk = sh + K;
    float* sO = sh + 2 * K;
    const int tid = threadIdx.x;
    const int h = blockIdx.x % H, b = blockIdx.x / H;
    const int grp = h / (H / G);
    for (int i = tid; i < K; i += 256) {
        sQ[i] = __bfloat162float(q[((long)b * G + grp) * K + i]);
        sKk[i] = __bfloat162float(k[((long)b * G + grp) * K + i]);
    }
    float lm[MAXL];
#pragma unroll
    for (int l = 0; l < MAXL; ++l) lm[l] = (l < L) ? __bfloat162float(lam[((long)b * H + h) * L + l]) : 0.f;
    const float dec = __expf(g[(long)b * H + h]);
    __syncthreads();
    const int col = tid % V, rstep = 256 / V;
    const float vv = __bfloat162float(v[((long)b * H + h) * V + col]);
    float* S = states + (long)(b * H + h) * K * V * L;
    float osum = 0.f;
    for (int row = tid / V; row < K; row += rstep) {
        float* p = S + ((long)row * V + col) * L;
        float s[MAXL];
#pragma unroll
        for (int l = 0; l < MAXL; ++l) s[l] = (l < L) ? p[l] : 0.f;
        // cascade: levels 0 .. carry are summed into level carry
        float merged = 0.f;
#pragma unroll
        for (int l = 0; l < MAXL; ++l)
            if (l <= carry) {
                merged += s[l];
                s[l] = 0.f;
            }
#pragma unroll
        for (int l = 0; l < MAXL; ++l)
            if (l == carry) s[l] = merged;
        float acc = 0.f;
#pragma unroll
        for (int l = 0; l < MAXL; ++l) {
            s[l] *= dec;
            if (l == 0) s[l] = sKk[row] * vv;
            acc += lm[l] * s[l];
            if (l < L) p[l] = s[l];
        }
        osum += sQ[row] * acc;
    }
    sO[tid] = osum;
    __syncthreads();
    if (tid < V) {
        float t = 0.f;
        for (int r = 0; r < rstep; ++r) t += sO[r * V + tid];
        o[((long)b * H + h) * V + tid] = __float2bfloat16(t);
    }
}

int mamba2_prompt_states_launch(const bf16* k, const bf16* v, const float* g, float* states, const float* seg_F, const float* seg_D,
                                int B, int T0, int n, int H, int G, int K, int L, cudaStream_t stream) {
    dim3 grid(B * H, L);
    auto launch = [&](auto kern, size_t sm) -> cudaError_t {
        const cudaError_t e = allow_smem(kern, sm);
        if (e == cudaSuccess) launch_chained(kern, grid, 256, sm, stream, k, v, g, states, seg_F, seg_D, T0, n, H, G, L);
        return e;
    };
    const cudaError_t e = K == 128 ? launch(mamba2_prompt_state_kernel<128>, PromptStateSmem<128>::total)
                                   : launch(mamba2_prompt_state_kernel<64>, PromptStateSmem<64>::total);
    if (e != cudaSuccess) return (int)e;
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

template <typename KernT>
static int tail_launch(KernT kern, size_t sm, int TL, const Mamba2Tail& a, int B, cudaStream_t stream) {
    const cudaError_t e = allow_smem(kern, sm);
    if (e != cudaSuccess) return (int)e;
    launch_chained(kern, (unsigned)(B * a.H * (64 / TL)), TL_THREADS, sm, stream, a, B);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}
static bool tail_whole_heads(const Mamba2Tail& a, int B) { return (long)B * a.H >= 96; }      // see above
int mamba2_tail_intra_launch(const Mamba2Tail& a, int B, int K, cudaStream_t stream) {
    if (tail_whole_heads(a, B))
        return K == 128 ? tail_launch(mamba2_tail_intra_kernel<128, 64>, TailIntraSmem<128, 64>::total, 64, a, B, stream)
                        : tail_launch(mamba2_tail_intra_kernel<64, 64>, TailIntraSmem<64, 64>::total, 64, a, B, stream);
    return K == 128 ? tail_launch(mamba2_tail_intra_kernel<128, 16>, TailIntraSmem<128, 16>::total, 16, a, B, stream)
                    : tail_launch(mamba2_tail_intra_kernel<64, 16>, TailIntraSmem<64, 16>::total, 16, a, B, stream);
}
int mamba2_tail_levels_launch(const Mamba2Tail& a, int B, int K, cudaStream_t stream) {
    if (tail_whole_heads(a, B))
        return K == 128 ? tail_launch(mamba2_tail_levels_kernel<128, 64>, TailLevelsSmem<128, 64>::total, 64, a, B, stream)
                        : tail_launch(mamba2_tail_levels_kernel<64, 64>, TailLevelsSmem<64, 64>::total, 64, a, B, stream);
    return K == 128 ? tail_launch(mamba2_tail_levels_kernel<128, 16>, TailLevelsSmem<128, 16>::total, 16, a, B, stream)
                    : tail_launch(mamba2_tail_levels_kernel<64, 16>, TailLevelsSmem<64, 16>::total, 16, a, B, stream);
}

int mamba2_prompt_states_check(int B, int T, int H, int G, int K, int V, int L) {
    if (B <= 0 || T <= 0 || H <= 0 || G <= 0 || H % G != 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (!((K == 64 || K == 128) && V == 64) || L <= 0 || L > 32) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (L < 1 + (32 - __builtin_clz((unsigned)(T - 1) | 1u)) && T > 1) return LLATTN_ERR_TOO_FEW_LEVELS;
    return 0;
}

}  // namespace llattn

extern "C" {

int llattn_mamba2_final_state(const void* k, const void* v, const float* g, float* states,
                              int B, int T, int H, int G, int K, int V, int L, void* stream) {
    const int rc = llattn::mamba2_prompt_states_check(B, T, H, G, K, V, L);
    if (rc != 0) return rc;
    if (!k || !v || !g || !states) return LLATTN_ERR_NULL;
    using bf = __nv_bfloat16;
    dim3 grid(B * H, L);
    cudaStream_t st = (cudaStream_t)stream;
    if (K == 128) llattn::launch_chained(llattn::mamba2_final_state_kernel<128, 64>, grid, 256, 0, st, (const bf*)k, (const bf*)v, g, states, B,
            T, H, G, L);
    else llattn::launch_chained(llattn::mamba2_final_state_kernel<64, 64>, grid, 256, 0, st, (const bf*)k, (const bf*)v, g, states, B, T, H, G, L);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int llattn_mamba2_prompt_states(const void* k, const void* v, const float* g, float* states, const void* fwd_workspace,
                                size_t fwd_workspace_bytes, int B, int T, int tail, int H, int G, int K, int V, int L, void* stream) {
    if (T <= 0 || T % 64 != 0 || tail < 0 || tail >= 64) return LLATTN_ERR_BAD_LENGTH;
    const int rc = llattn::mamba2_prompt_states_check(B, T + tail, H, G, K, V, L);
    if (rc != 0) return rc;
    if (!k || !v || !g || !states) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {k, v, states})) return LLATTN_ERR_ALIGNMENT;
    const float *seg_F = nullptr, *seg_D = nullptr;
    if (fwd_workspace != nullptr) {
        const int e = llattn::mamba2_fwd_workspace_segments(fwd_workspace, fwd_workspace_bytes, B, T, H, G, K, V, &seg_F, &seg_D);
        if (e != 0) return e;
    }
    using bf = __nv_bfloat16;
    return llattn::mamba2_prompt_states_launch((const bf*)k, (const bf*)v, g, states, seg_F, seg_D, B, T, tail, H, G, K, L, (cudaStream_t)stream);
}

int llattn_mamba2_prompt_tail(const void* q, const void* k, const void* v, const float* g, const void* lambda, const void* x, const void* D,
                              int y_is_f32, void* y, float* states, int state_levels, float* tail_part, int B, int T, int tail, int H, int G, int K,
                              int V, int L, void* stream) {
    if (T < 0 || T % 64 != 0 || tail <= 0 || tail >= 64) return LLATTN_ERR_BAD_LENGTH;
    int rc = llattn::mamba2_prompt_states_check(B, T + tail, H, G, K, V, state_levels);
    if (rc != 0) return rc;
    if (L < state_levels) return LLATTN_ERR_TOO_FEW_LEVELS;
    if (!q || !k || !v || !g || !lambda || !y || !states || (D && !x) || (T > 0 && !tail_part)) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {q, k, v, states, tail_part})) return LLATTN_ERR_ALIGNMENT;
    using bf = __nv_bfloat16;
    const llattn::Mamba2Tail a{(const bf*)q, (const bf*)k, (const bf*)v, (const bf*)lambda, (const bf*)x, g, D, y, states, tail_part, T, tail, H, G,
                               state_levels, L, y_is_f32};
    rc = llattn::mamba2_tail_intra_launch(a, B, K, (cudaStream_t)stream);
    return rc != 0 || T == 0 ? rc : llattn::mamba2_tail_levels_launch(a, B, K, (cudaStream_t)stream);
}

int llattn_mamba2_step(float* states, const void* q, const void* k, const void* v, const float* g, const void* lambda, void* o,
                       int B, int H, int G, int K, int V, int L, int carry_level, void* stream) {
    if (B <= 0 || H <= 0 || G <= 0 || H % G != 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (K <= 0 || K > 1024 || V <= 0 || V > 256 || 256 % V != 0 || L <= 0 || L > 32) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (carry_level < 0 || carry_level >= L) return LLATTN_ERR_TOO_FEW_LEVELS;
    if (!states || !q || !k || !v || !g || !lambda || !o) return LLATTN_ERR_NULL;
    using bf = __nv_bfloat16;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t sm = (size_t)(2 * K + 256) * sizeof(float);
    if (L <= 16)
        llattn::launch_chained(llattn::mamba2_step_kernel<16>, B * H, 256, sm, st, states, (const bf*)q, (const bf*)k, (const bf*)v, g,
                (const bf*)lambda, (bf*)o, H, G, K, V, L, carry_level);
    else
        llattn::launch_chained(llattn::mamba2_step_kernel<32>, B * H, 256, sm, st, states, (const bf*)q, (const bf*)k, (const bf*)v, g,
                (const bf*)lambda, (bf*)o, H, G, K, V, L, carry_level);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

}  // extern "C"
