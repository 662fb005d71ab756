// One decode step on level-major states, with everything the layer does around the state update in the same kernel.
//
// Reference being replaced: hselective_state_update (hattention/mamba_apis.py:407-566), chunk_h_gated_delta_rule with an
// initial state (hattention/gated_delta_rule_apis.py:93-132) and the hattention_step both end in (hattention/kernel.py:
// 563-633; HState.cascade_weak / insert / step_output, hattention/recurrent.py:42-54, 79-98, 134-166).
//
// States are fp32, stored (B, H, L, K, V): a level of a head is one contiguous K x V block.  Only levels that hold tokens
// take part (`live`, from the token counts the host keeps): about half of the levels that have been reached, where the
// level-innermost layout of llattn_mamba2_step moves all L of them.  Per live level the state is read once and written
// once, so the step is bound by HBM (large batches) or by the latency of one pass through L2 (one sequence).
//
// What a step does: the levels 0 .. carry are summed into level `carry` (the others among them become zero), every live
// level is decayed (and, for the delta rule, multiplied by I - beta k k^T), level 0 becomes k v^T (beta k v^T), and
// o = q . sum_l lambda_l S_l.
//
// Measured on a B200, eight live levels of L = 15 (the bytes are those levels read and written once):
//   Mamba-2, K = 128, V = 64: B = 1, H = 48 7.5 us; B = 4, H = 32 13.7 us; B = 64, H = 32 188 us = 5.7 TB/s (the level-innermost
//   kernel behind the layer's torch operators: 110 us and 1200 us for a call at B = 1 and B = 64)
//   delta rule, K = V = 128: B = 1, H = 16 6.2 us; B = 16, H = 16 48.4 us = 5.5 TB/s (414 us for a call before)
#include "rowwise.cuh"
#include "../../include/llattn.h"

namespace llattn {

constexpr int ST_THREADS = 256;
constexpr int ST_MAXL = 32;

// 16 bytes if p, else zeros, without a branch: a branch around every load of a group keeps the compiler from having them all in
// flight (the delta-rule step took 177 us instead of 103 at B = 16, H = 16, K = V = 128)
__device__ __forceinline__ float4 ldg4_if(const float* ptr, bool p) {
    float4 r;
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %5, 0;\n mov.f32 %0, 0f00000000;\n mov.f32 %1, 0f00000000;\n mov.f32 %2, 0f00000000;\n"
                 " mov.f32 %3, 0f00000000;\n @p ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n}\n"
                 : "=&f"(r.x), "=&f"(r.y), "=&f"(r.z), "=&f"(r.w)
                 : "l"(ptr), "r"((int)p)
                 : "memory");
    return r;
}

struct M2StepArgs {
    float* states;          // (B,H,L,K,V)
    const bf16* q;          // (B,G,K)
    const bf16* k;          // (B,G,K)
    const bf16* x;          // (B,H,V): v itself when dt is null
    const bf16* dt;         // (B,H) or null
    const float* g;         // (B,H) log decay, used when dt is null
    const bf16* dl;         // (B,H,L): lambda itself when Lp is null
    const void* Lp;         // (H,L)
    const void* D;          // (H) or null
    const void* bias;       // (H) or null
    const float* A;         // (H)
    void* y;                // (B,H,V) bf16, or fp32 with an fp32 D
    int H, G, K, V, L;
    uint32_t live;
    int carry, lambda_mode, softplus;
    int lp_f32, d_f32, bias_f32;
};

// lambda of one level, with the rounding of torch's bf16 operators (each result rounded to bf16)
__device__ __forceinline__ float layer_lambda(const M2StepArgs& a, long bh, int h, int l) {
    const float d = __bfloat162float(a.dl[bh * a.L + l]);
    if (a.Lp == nullptr) return d;
    return lambda_torch(a.lambda_mode, load_param(a.Lp, h * a.L + l, a.lp_f32), d);
}

// A CTA owns COLS value columns of one (batch, head).  COLS = 64 (whole rows of a 64-wide head, 256 contiguous bytes) for
// batches that fill the chip; COLS = 16 splits a head over four CTAs, for the few heads of a single sequence, where the time
// is a handful of dependent memory round trips (8 columns, or every live level in one group, were slower: 10.2 / 9.9 us).
template <int COLS, int RPT, int NG, int CTAS>
__global__ void __launch_bounds__(ST_THREADS, CTAS) m2_layer_step_kernel(const __grid_constant__ M2StepArgs a) {
    chain_wait();
    constexpr int C4 = COLS / 4;                    // lanes per row, four columns each
    constexpr int R = ST_THREADS / C4;              // rows per pass
    extern __shared__ float sh[];                   // q[K] | k[K]
    __shared__ float sLam[ST_MAXL];
    __shared__ float sDec;
    __shared__ float sV[COLS];
    __shared__ float4 sO[8][C4];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ncb = a.V / COLS;
    const int cb = blockIdx.x % ncb;
    const int h = (blockIdx.x / ncb) % a.H;
    const int b = blockIdx.x / (ncb * a.H);
    const long bh = (long)b * a.H + h;
    const int grp = h / (a.H / a.G);
    float* sQ = sh;
    float* sK = sh + a.K;
    const int c4 = tid % C4, rg = tid / C4;
    const long kv = (long)a.K * a.V;
    float* S = a.states + bh * a.L * kv + cb * COLS + c4 * 4;
    // a group of levels is requested together, the first one before anything else
    int lev[NG];
    float4 s[NG][RPT];
    auto load_group = [&](uint32_t& m, int r0) {
#pragma unroll
        for (int u = 0; u < NG; ++u) {
            lev[u] = m ? __ffs(m) - 1 : -1;
            m &= m - 1;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int row = r0 + R * i;
                s[u][i] = ldg4_if(S + lev[u] * kv + (long)row * a.V, lev[u] >= 0 && row < a.K);
            }
        }
    };
    uint32_t m = a.live;
    load_group(m, rg);
    for (int i = tid; i < a.K; i += ST_THREADS) {
        sQ[i] = __bfloat162float(a.q[((long)b * a.G + grp) * a.K + i]);
        sK[i] = __bfloat162float(a.k[((long)b * a.G + grp) * a.K + i]);
    }
    if (tid < a.L) sLam[tid] = layer_lambda(a, bh, h, tid);
    if (tid >= 64 && tid < 64 + COLS) {
        float xv = __bfloat162float(a.x[bh * a.V + cb * COLS + tid - 64]);
        float g;
        if (a.dt != nullptr) {
            float t = __bfloat162float(a.dt[bh]);
            if (a.bias != nullptr) t += load_param(a.bias, h, a.bias_f32);
            const bool half = a.bias == nullptr || !a.bias_f32;      // dt stays bf16 between torch's operators
            if (half) t = round_bf16(t);
            if (a.softplus) {
                t = softplus_torch(t);
                if (half) t = round_bf16(t);
            }
            g = a.A[h] * t;
            xv = round_bf16(xv * t);
        } else {
            g = a.g[bh];
        }
        sV[tid - 64] = xv;
        if (tid == 64) sDec = fexp(g);
    }
    __syncthreads();
    const float dec = sDec;
    const float4 v4 = make_float4(sV[c4 * 4], sV[c4 * 4 + 1], sV[c4 * 4 + 2], sV[c4 * 4 + 3]);
    const float lam0 = sLam[0], lamc = sLam[a.carry];
    float4 o4 = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r0 = rg; r0 < a.K; r0 += R * RPT) {
        float4 acc[RPT], merged[RPT];
#pragma unroll
        for (int i = 0; i < RPT; ++i) acc[i] = merged[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (;;) {
#pragma unroll
            for (int u = 0; u < NG; ++u) {
                if (lev[u] < 0) continue;
                float* P = S + lev[u] * kv;
                const float lam = sLam[lev[u]];
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const int row = r0 + R * i;
                    if (row >= a.K) continue;
                    float4 t = s[u][i];
                    if (lev[u] <= a.carry) {
                        merged[i].x += t.x; merged[i].y += t.y; merged[i].z += t.z; merged[i].w += t.w;
                        if (lev[u] != a.carry && lev[u] != 0)
                            *reinterpret_cast<float4*>(P + (long)row * a.V) = make_float4(0.f, 0.f, 0.f, 0.f);
                    } else {
                        t.x *= dec; t.y *= dec; t.z *= dec; t.w *= dec;
                        *reinterpret_cast<float4*>(P + (long)row * a.V) = t;
                        acc[i].x += lam * t.x; acc[i].y += lam * t.y; acc[i].z += lam * t.z; acc[i].w += lam * t.w;
                    }
                }
            }
            if (m == 0) break;
            load_group(m, r0);
        }
        if (r0 + R * RPT < a.K) {
            // the next rows' first group, while these rows finish
            m = a.live;
            load_group(m, r0 + R * RPT);
        }
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int row = r0 + R * i;
            if (row >= a.K) continue;
            if (a.carry > 0) {
                float4 t = merged[i];
                t.x *= dec; t.y *= dec; t.z *= dec; t.w *= dec;
                *reinterpret_cast<float4*>(S + a.carry * kv + (long)row * a.V) = t;
                acc[i].x += lamc * t.x; acc[i].y += lamc * t.y; acc[i].z += lamc * t.z; acc[i].w += lamc * t.w;
            }
            const float kr = sK[row], qr = sQ[row];
            const float4 n = make_float4(kr * v4.x, kr * v4.y, kr * v4.z, kr * v4.w);
            *reinterpret_cast<float4*>(S + (long)row * a.V) = n;
            o4.x += qr * (acc[i].x + lam0 * n.x);
            o4.y += qr * (acc[i].y + lam0 * n.y);
            o4.z += qr * (acc[i].z + lam0 * n.z);
            o4.w += qr * (acc[i].w + lam0 * n.w);
        }
    }
#pragma unroll
    for (int d = C4; d < 32; d <<= 1) {
        o4.x += __shfl_xor_sync(0xffffffffu, o4.x, d);
        o4.y += __shfl_xor_sync(0xffffffffu, o4.y, d);
        o4.z += __shfl_xor_sync(0xffffffffu, o4.z, d);
        o4.w += __shfl_xor_sync(0xffffffffu, o4.w, d);
    }
    if (lane < C4) sO[warp][lane] = o4;
    __syncthreads();
    if (tid < COLS) {
        float o = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) o += reinterpret_cast<const float*>(sO[w])[tid];
        const long at = bh * a.V + cb * COLS + tid;
        o = round_bf16(o);
        if (a.D != nullptr) {
            const float xd = __bfloat162float(a.x[at]) * load_param(a.D, h, a.d_f32);
            if (a.d_f32) reinterpret_cast<float*>(a.y)[at] = o + xd;
            else reinterpret_cast<bf16*>(a.y)[at] = __float2bfloat16(o + round_bf16(xd));
        } else {
            reinterpret_cast<bf16*>(a.y)[at] = __float2bfloat16(o);
        }
    }
}

struct GdnStepArgs {
    float* states;          // (B,H,L,K,V)
    const bf16* q;          // (B,G,K)
    const bf16* k;          // (B,G,K)
    const bf16* v;          // (B,H,V)
    const bf16* beta;       // (B,H)
    const float* g;         // (B,H)
    const bf16* lam;        // (B,H,L)
    bf16* o;                // (B,H,V)
    int H, G, K, V, L;
    uint32_t live;
    int carry, l2norm;
    float scale;            // of the normalised q
    float lam_mul;          // lambda is rounded to bf16 after this factor; 0: taken as it is
};

// A CTA owns COLS value columns of one (batch, head).  The slice of NG levels is in registers between the two passes over it:
// k^T S_l of every level first (warp shuffles, then one exchange through shared memory for all of them), then the update, the
// store and the output; more live levels take another round.
template <int THREADS, int RPT, int NG, int CTAS, int COLS = 16>
__global__ void __launch_bounds__(THREADS, CTAS) gdn_layer_step_kernel(const __grid_constant__ GdnStepArgs a) {
    chain_wait();
    constexpr int C4 = COLS / 4, R = THREADS / C4, NW = THREADS / 32;
    __shared__ float sQ[256], sK[256];
    __shared__ float sLam[ST_MAXL];
    __shared__ float4 sRed[NW][NG + 1][C4];
    __shared__ float4 sKs[NG + 1][C4];
    __shared__ float4 sO[NW][C4];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ncb = a.V / COLS;
    const int cb = blockIdx.x % ncb;
    const int h = (blockIdx.x / ncb) % a.H;
    const int b = blockIdx.x / (ncb * a.H);
    const long bh = (long)b * a.H + h;
    const int grp = h / (a.H / a.G);
    // rounds of NG live levels; those up to the carry are summed, and their sum is one more slot of the round that has the last of them
    const int c4 = tid % C4, rg = tid / C4;
    const int col = cb * COLS + c4 * 4;
    const long kv = (long)a.K * a.V;
    float* S = a.states + bh * a.L * kv + col;
    uint32_t m = a.live;
    const uint32_t low = a.carry > 0 ? (2u << a.carry) - 1u : 0u;
    float4 s[NG + 1][RPT];
    int lev[NG + 1];
    auto load_group = [&]() {
#pragma unroll
        for (int u = 0; u < NG; ++u) {
            lev[u] = m ? __ffs(m) - 1 : -1;
            m &= m - 1;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int row = rg + R * i;
                s[u][i] = ldg4_if(S + lev[u] * kv + (long)row * a.V, lev[u] >= 0 && row < a.K);
            }
        }
    };
    load_group();                                   // before anything else
    if (warp < 2) {
        // q (warp 0) and k (warp 1), normalised with the two bf16 rounding points of the l2norm kernel
        const bf16* src = (warp == 0 ? a.q : a.k) + ((long)b * a.G + grp) * a.K;
        float* dst = warp == 0 ? sQ : sK;
        float f[8];
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            f[i] = lane + 32 * i < a.K ? __bfloat162float(src[lane + 32 * i]) : 0.f;
            ss += f[i] * f[i];
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
        const float rstd = rsqrtf(ss + 1e-6f);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (lane + 32 * i < a.K) {
                float y = f[i];
                if (a.l2norm) {
                    y = round_bf16(y * rstd);
                    if (warp == 0) y = round_bf16(y * a.scale);
                }
                dst[lane + 32 * i] = y;
            }
    } else if (warp == 2 && lane < a.L) {
        const float l = __bfloat162float(a.lam[bh * a.L + lane]);
        sLam[lane] = a.lam_mul != 0.f ? round_bf16(l * a.lam_mul) : l;
    }
    const float dec = fexp(a.g[bh]);
    const float be = __bfloat162float(a.beta[bh]);
    float4 v4;
    {
        const uint2 raw = *reinterpret_cast<const uint2*>(a.v + bh * a.V + col);
        const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
        v4 = make_float4(__bfloat162float(lo.x), __bfloat162float(lo.y), __bfloat162float(hi.x), __bfloat162float(hi.y));
    }
    float4 acc[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < RPT; ++i) s[NG][i] = make_float4(0.f, 0.f, 0.f, 0.f);
    bool carried = a.carry == 0;
    bool more = a.live != 0;
    while (more) {
        lev[NG] = -1;
        if (!carried) {
#pragma unroll
            for (int u = 0; u < NG; ++u) {
                if (lev[u] < 0 || !((low >> lev[u]) & 1u)) continue;
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const int row = rg + R * i;
                    s[NG][i].x += s[u][i].x; s[NG][i].y += s[u][i].y; s[NG][i].z += s[u][i].z; s[NG][i].w += s[u][i].w;
                    if (row < a.K && lev[u] != a.carry && lev[u] != 0)
                        *reinterpret_cast<float4*>(S + lev[u] * kv + (long)row * a.V) = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                lev[u] = -1;
            }
            if ((m & low) == 0) {
                lev[NG] = a.carry;
                carried = true;
            }
        }
        __syncthreads();                            // q, k, lambda staged; the exchange area is free again
        // k^T S_l
#pragma unroll
        for (int u = 0; u <= NG; ++u) {
            if (lev[u] < 0) continue;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int row = rg + R * i;
                const float kr = row < a.K ? sK[row] : 0.f;
                x.x += kr * s[u][i].x; x.y += kr * s[u][i].y; x.z += kr * s[u][i].z; x.w += kr * s[u][i].w;
            }
#pragma unroll
            for (int d = C4; d < 32; d <<= 1) {
                x.x += __shfl_xor_sync(0xffffffffu, x.x, d);
                x.y += __shfl_xor_sync(0xffffffffu, x.y, d);
                x.z += __shfl_xor_sync(0xffffffffu, x.z, d);
                x.w += __shfl_xor_sync(0xffffffffu, x.w, d);
            }
            if (lane < C4) sRed[warp][u][lane] = x;
        }
        __syncthreads();
        if (tid < (NG + 1) * COLS) {
            const int u = tid / COLS, c = tid % COLS;
            float x = 0.f;
#pragma unroll
            for (int w = 0; w < NW; ++w) x += reinterpret_cast<const float*>(&sRed[w][u][0])[c];
            reinterpret_cast<float*>(&sKs[u][0])[c] = x;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u <= NG; ++u) {
            if (lev[u] < 0) continue;
            const float lam = sLam[lev[u]];
            const float4 ks = sKs[u][c4];
            float* P = S + lev[u] * kv;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int row = rg + R * i;
                if (row >= a.K) continue;
                const float bk = be * sK[row];
                float4 t = s[u][i];
                t.x = dec * (t.x - bk * ks.x); t.y = dec * (t.y - bk * ks.y);
                t.z = dec * (t.z - bk * ks.z); t.w = dec * (t.w - bk * ks.w);
                *reinterpret_cast<float4*>(P + (long)row * a.V) = t;
                acc[i].x += lam * t.x; acc[i].y += lam * t.y; acc[i].z += lam * t.z; acc[i].w += lam * t.w;
            }
        }
        more = m != 0;
        if (more) load_group();
    }
    __syncthreads();
    const float lam0 = sLam[0];
    float4 o4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int row = rg + R * i;
        if (row >= a.K) continue;
        const float bk = be * sK[row], qr = sQ[row];
        const float4 n = make_float4(bk * v4.x, bk * v4.y, bk * v4.z, bk * v4.w);
        *reinterpret_cast<float4*>(S + (long)row * a.V) = n;
        o4.x += qr * (acc[i].x + lam0 * n.x);
        o4.y += qr * (acc[i].y + lam0 * n.y);
        o4.z += qr * (acc[i].z + lam0 * n.z);
        o4.w += qr * (acc[i].w + lam0 * n.w);
    }
#pragma unroll
    for (int d = C4; d < 32; d <<= 1) {
        o4.x += __shfl_xor_sync(0xffffffffu, o4.x, d);
        o4.y += __shfl_xor_sync(0xffffffffu, o4.y, d);
        o4.z += __shfl_xor_sync(0xffffffffu, o4.z, d);
        o4.w += __shfl_xor_sync(0xffffffffu, o4.w, d);
    }
    if (lane < C4) sO[warp][lane] = o4;
    __syncthreads();
    if (tid < COLS) {
        float o = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) o += reinterpret_cast<const float*>(&sO[w][0])[tid];
        a.o[bh * a.V + cb * COLS + tid] = __float2bfloat16(o);
    }
}

}  // namespace llattn

namespace {

// The launch goes to the stream's device; the caller's current device is left as it is.
struct OnDevice {
    int old = -1;
    cudaError_t err = cudaSuccess;
    explicit OnDevice(int dev) {
        int cur = dev;
        if ((err = cudaGetDevice(&cur)) == cudaSuccess && cur != dev) {
            err = cudaSetDevice(dev);
            if (err == cudaSuccess) old = cur;
        }
    }
    ~OnDevice() {
        if (old >= 0) cudaSetDevice(old);
    }
};

}  // namespace

extern "C" {

int llattn_mamba2_layer_step(float* states, const void* q, const void* k, const void* x, const void* dt, const float* g,
                             const void* dl, const void* Lp, int lp_is_f32, const void* D, int d_is_f32, const void* dt_bias,
                             int bias_is_f32, const float* A, void* y, int B, int H, int G, int K, int V, int L, unsigned live,
                             int carry_level, int lambda_mode, int dt_softplus, int device, void* stream) {
    if (B <= 0 || H <= 0 || G <= 0 || H % G != 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (K <= 0 || K > 1024 || V <= 0 || V > 256 || V % 16 != 0 || L <= 0 || L > 32) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (lambda_mode < 0 || lambda_mode > 2) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (carry_level < 0 || carry_level >= L || (L < 32 && (live >> L) != 0)) return LLATTN_ERR_TOO_FEW_LEVELS;
    if (!states || !q || !k || !x || !dl || !y || (!dt && !g) || (dt && !A)) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {states})) return LLATTN_ERR_ALIGNMENT;
    OnDevice on(device);
    if (on.err != cudaSuccess) return (int)on.err;
    using bf = __nv_bfloat16;
    llattn::M2StepArgs a{states, (const bf*)q, (const bf*)k, (const bf*)x, (const bf*)dt, g, (const bf*)dl, Lp, D, dt_bias, A, y,
                         H, G, K, V, L, live, carry_level, lambda_mode, dt_softplus, lp_is_f32, d_is_f32, bias_is_f32};
    const size_t sm = (size_t)2 * K * sizeof(float);
    cudaStream_t st = (cudaStream_t)stream;
    // whole rows per CTA once that gives two CTAs for every SM (K = 128, V = 64, whole rows / 16 columns: 192 heads 24.9 / 25.5 us, 240 28.4 / 32.4, 288 33.1 /
    // 35.9, 384 49.3 / 48.6: the line is on the safe side)
    if (V % 64 == 0 && (long)B * H * (V / 64) >= 296)
        llattn::launch_chained(llattn::m2_layer_step_kernel<64, 2, 4, 2>, B * H * (V / 64), llattn::ST_THREADS, sm, st, a);
    else
        llattn::launch_chained(llattn::m2_layer_step_kernel<16, 2, 6, 2>, B * H * (V / 16), llattn::ST_THREADS, sm, st, a);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int llattn_gdn_layer_step(float* states, const void* q, const void* k, const void* v, const void* beta, const float* g,
                          const void* lambda, void* o, int B, int H, int G, int K, int V, int L, unsigned live, int carry_level,
                          int l2norm, float scale, float lambda_mul, int device, void* stream) {
    if (B <= 0 || H <= 0 || G <= 0 || H % G != 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (K <= 0 || K > 256 || V <= 0 || V % 16 != 0 || L <= 0 || L > 32) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (carry_level < 0 || carry_level >= L || (L < 32 && (live >> L) != 0)) return LLATTN_ERR_TOO_FEW_LEVELS;
    if (!states || !q || !k || !v || !beta || !g || !lambda || !o) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {states}) || llattn::misaligned(8, {v})) return LLATTN_ERR_ALIGNMENT;
    OnDevice on(device);
    if (on.err != cudaSuccess) return (int)on.err;
    using bf = __nv_bfloat16;
    llattn::GdnStepArgs a{states, (const bf*)q, (const bf*)k, (const bf*)v, (const bf*)beta, g, (const bf*)lambda, (bf*)o,
                          H, G, K, V, L, live, carry_level, l2norm, scale, lambda_mul};
    const unsigned grid = (unsigned)(B * H * (V / 16));
    cudaStream_t st = (cudaStream_t)stream;
    // K = 128: with two CTAs for every SM and more, each thread takes four rows, so that more CTAs share an SM and one's reduction overlaps
    // another's loads: 13.2 against 15.2 us at B = 4, 54.6 against 60.3 us at B = 16 (H = 16, V = 128, eight live levels); below, two rows
    // each: 6.2 against 8.3 us at B = 1.  Where V allows, the CTA is 32 columns wide (whole 128-byte lines) and takes three levels a round:
    // 48.4 against 51.1 us at B = 16, 91.1 against 95.9 at B = 32, 20.8 against 23.5 at B = 8 (four levels a round 51.7, two 51.6)
    if (K <= 64) llattn::launch_chained(llattn::gdn_layer_step_kernel<256, 1, 8, 2>, grid, 256, 0, st, a);
    else if (K <= 128 && grid >= 296 && V % 32 == 0) llattn::launch_chained(llattn::gdn_layer_step_kernel<256, 4, 3, 2, 32>, grid / 2, 256, 0, st, a);
    else if (K <= 128 && grid >= 296) llattn::launch_chained(llattn::gdn_layer_step_kernel<128, 4, 4, 4>, grid, 128, 0, st, a);
    else if (K <= 128) llattn::launch_chained(llattn::gdn_layer_step_kernel<256, 2, 4, 2>, grid, 256, 0, st, a);
    else llattn::launch_chained(llattn::gdn_layer_step_kernel<512, 2, 4, 1>, grid, 512, 0, st, a);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

}  // extern "C"
