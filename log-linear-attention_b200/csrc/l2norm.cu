// Row-wise L2 normalisation of q / k and its backward for sm_100a (HBM-bound, one pass each).
//
// Reference being replaced: fla.modules.l2norm.l2norm_fwd / l2norm_bwd as called around the Gated
// DeltaNet drivers (hattention/kernel.py:20-29, 110-111, 224-225):
//     y  = bf16(bf16(x * rsqrt(sum x^2 + eps)) * scale)
//     dx = bf16(((dy * scale) - yhat (yhat . (dy * scale))) * rstd),   yhat = x * rstd in fp32
// A row (D <= 256 elements, D % 8 == 0) is handled by LPR lanes holding eight elements each.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/llattn.h"
#include "launch_count.h"

namespace llattn {

template <int LPR>
__global__ void __launch_bounds__(256) l2norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y,
                                                         long rows, int D, float scale, float eps) {
    chain_wait();
    const int lane = threadIdx.x % LPR;
    const long row = ((long)blockIdx.x * blockDim.x + threadIdx.x) / LPR;
    const bool active = row < rows && lane * 8 < D;
    float f[8];
    float ss = 0.f;
    if (active) {
        const uint4 raw = *reinterpret_cast<const uint4*>(x + row * D + lane * 8);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[2 * i] = __bfloat162float(h[i].x);
            f[2 * i + 1] = __bfloat162float(h[i].y);
            ss += f[2 * i] * f[2 * i] + f[2 * i + 1] * f[2 * i + 1];
        }
    }
#pragma unroll
    for (int d = LPR / 2; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
    if (active) {
        const float rstd = rsqrtf(ss + eps);
        uint4 out;
        __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat162 n = __floats2bfloat162_rn(f[2 * i] * rstd, f[2 * i + 1] * rstd);
            o[i] = __floats2bfloat162_rn(__bfloat162float(n.x) * scale, __bfloat162float(n.y) * scale);
        }
        *reinterpret_cast<uint4*>(y + row * D + lane * 8) = out;
    }
}

template <int LPR>
__global__ void __launch_bounds__(256) l2norm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ dy,
                                                         __nv_bfloat16* __restrict__ dx, long rows, int D, float scale, float eps) {
    chain_wait();
    const int lane = threadIdx.x % LPR;
    const long row = ((long)blockIdx.x * blockDim.x + threadIdx.x) / LPR;
    const bool active = row < rows && lane * 8 < D;
    float f[8], g[8];
    float ss = 0.f, dot = 0.f;
    if (active) {
        const uint4 raw = *reinterpret_cast<const uint4*>(x + row * D + lane * 8);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
        const float4 g0 = *reinterpret_cast<const float4*>(dy + row * D + lane * 8);
        const float4 g1 = *reinterpret_cast<const float4*>(dy + row * D + lane * 8 + 4);
        g[0] = g0.x * scale; g[1] = g0.y * scale; g[2] = g0.z * scale; g[3] = g0.w * scale;
        g[4] = g1.x * scale; g[5] = g1.y * scale; g[6] = g1.z * scale; g[7] = g1.w * scale;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[2 * i] = __bfloat162float(h[i].x);
            f[2 * i + 1] = __bfloat162float(h[i].y);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            ss += f[i] * f[i];
            dot += f[i] * g[i];
        }
    }
#pragma unroll
    for (int d = LPR / 2; d > 0; d >>= 1) {
        ss += __shfl_xor_sync(0xffffffffu, ss, d);
        dot += __shfl_xor_sync(0xffffffffu, dot, d);
    }
    if (active) {
        const float rstd = rsqrtf(ss + eps);
        const float yd = dot * rstd * rstd;          // (yhat . g) * rstd, with yhat = x rstd
        uint4 out;
        __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            o[i] = __floats2bfloat162_rn((g[2 * i] - f[2 * i] * yd) * rstd, (g[2 * i + 1] - f[2 * i + 1] * yd) * rstd);
        *reinterpret_cast<uint4*>(dx + row * D + lane * 8) = out;
    }
}

// The gradients that leave a Gated DeltaNet backward, in one pass over the rows: q and k through the l2norm (and scale), beta and
// lambda rounded to bf16 (lambda through its factor, rounded before and after it as two operators would).  16 lanes a row; K_in >= K columns of dq, dk are stored (padded keys).
struct GdnGradOut {
    const __nv_bfloat16 *q, *k;       // (rows,K)
    const float *dq, *dk;             // (rows,K_in)
    const float *db, *dl, *dg;        // (rows), (rows,L), (rows)
    __nv_bfloat16 *gq, *gk, *gb, *gl;
    float* gg;                        // (rows), with dg
    int rep;                          // the fp32 gradients have `rep` rows for each of these (parts of a wide value head), summed here
    long rows;
    int K, K_in, L;
    float scale, lam_mul;
};

__global__ void __launch_bounds__(256) gdn_grad_out_kernel(const __grid_constant__ GdnGradOut a) {
    chain_wait();
    const int lane = threadIdx.x & 15;
    const long row = (long)blockIdx.x * 16 + (threadIdx.x >> 4);
    const bool have = row < a.rows, act = have && lane * 8 < a.K;
    if (a.q) {
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const float scale = w == 0 ? a.scale : 1.f;
            float f[8] = {}, g[8] = {};
            float ss = 0.f, dot = 0.f;
            if (act) {
                const uint4 raw = *reinterpret_cast<const uint4*>((w == 0 ? a.q : a.k) + row * a.K + lane * 8);
                const float* d = (w == 0 ? a.dq : a.dk) + row * a.rep * a.K_in + lane * 8;
                float4 g0 = *reinterpret_cast<const float4*>(d), g1 = *reinterpret_cast<const float4*>(d + 4);
                for (int r = 1; r < a.rep; ++r) {
                    const float4 e0 = *reinterpret_cast<const float4*>(d + (long)r * a.K_in), e1 = *reinterpret_cast<const float4*>(d + (long)r * a.K_in + 4);
                    g0.x += e0.x; g0.y += e0.y; g0.z += e0.z; g0.w += e0.w;
                    g1.x += e1.x; g1.y += e1.y; g1.z += e1.z; g1.w += e1.w;
                }
                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
                g[0] = g0.x * scale; g[1] = g0.y * scale; g[2] = g0.z * scale; g[3] = g0.w * scale;
                g[4] = g1.x * scale; g[5] = g1.y * scale; g[6] = g1.z * scale; g[7] = g1.w * scale;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    f[2 * i] = __bfloat162float(h[i].x);
                    f[2 * i + 1] = __bfloat162float(h[i].y);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    ss += f[i] * f[i];
                    dot += f[i] * g[i];
                }
            }
#pragma unroll
            for (int d = 8; d > 0; d >>= 1) {
                ss += __shfl_xor_sync(0xffffffffu, ss, d);
                dot += __shfl_xor_sync(0xffffffffu, dot, d);
            }
            if (act) {
                const float rstd = rsqrtf(ss + 1e-6f), yd = dot * rstd * rstd;
                uint4 out;
                __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    o[i] = __floats2bfloat162_rn((g[2 * i] - f[2 * i] * yd) * rstd, (g[2 * i + 1] - f[2 * i + 1] * yd) * rstd);
                *reinterpret_cast<uint4*>((w == 0 ? a.gq : a.gk) + row * a.K + lane * 8) = out;
            }
        }
    }
    if (!have) return;
    if (lane >= 14) {
        const float* d = (lane == 15 ? a.db : a.dg);
        if (d != nullptr) {
            float x = d[row * a.rep];
            for (int r = 1; r < a.rep; ++r) x += d[row * a.rep + r];
            if (lane == 15) a.gb[row] = __float2bfloat16(x);
            else a.gg[row] = x;
        }
    }
    for (int j = lane; j < a.L; j += 16) {
        float s = a.dl[row * a.rep * a.L + j];
        for (int r = 1; r < a.rep; ++r) s += a.dl[(row * a.rep + r) * a.L + j];
        __nv_bfloat16 x = __float2bfloat16(s);
        if (a.lam_mul != 0.f) x = __float2bfloat16(__bfloat162float(x) * a.lam_mul);
        a.gl[row * a.L + j] = x;
    }
}

// dbeta and dlambda alone, of heads of one part: element by element, four a thread (with 16 lanes a row of 14 columns the pass took
// 73 us for 45 MB at 524,288 rows)
__device__ __forceinline__ void grad_cast(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long n, long i, float mul) {
    if (i >= n) return;
    float x[4];
    __nv_bfloat16 r[4];
    const int m = n - i < 4 ? (int)(n - i) : 4;
    const bool wide = m == 4 && (((uintptr_t)(src + i) & 15) | ((uintptr_t)(dst + i) & 7)) == 0;
    if (wide) *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(src + i);
    else for (int j = 0; j < m; ++j) x[j] = src[i + j];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j >= m) break;
        r[j] = __float2bfloat16(x[j]);
        if (mul != 0.f) r[j] = __float2bfloat16(__bfloat162float(r[j]) * mul);
    }
    if (wide) *reinterpret_cast<uint2*>(dst + i) = *reinterpret_cast<const uint2*>(r);
    else for (int j = 0; j < m; ++j) dst[i + j] = r[j];
}

__global__ void __launch_bounds__(256) gdn_grad_cast_kernel(const __grid_constant__ GdnGradOut a, unsigned blocks_l) {
    chain_wait();
    if (blockIdx.x < blocks_l) grad_cast(a.dl, a.gl, a.rows * a.L, ((long)blockIdx.x * 256 + threadIdx.x) * 4, a.lam_mul);
    else grad_cast(a.db, a.gb, a.rows, ((long)(blockIdx.x - blocks_l) * 256 + threadIdx.x) * 4, 0.f);
}

}  // namespace llattn

extern "C" {

int llattn_gdn_grad_out(const void* q, const void* k, const float* dq, const float* dk, const float* dbeta, const float* dlambda,
                        const float* dg, void* gq, void* gk, void* gbeta, void* glambda, float* gg, long rows, int rep, int K, int K_in, int L,
                        float scale, float lambda_mul, void* stream) {
    if (rows <= 0 || rep <= 0 || K <= 0 || K % 8 != 0 || K_in < K || K_in % 8 != 0 || K_in > 128 || L <= 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if ((q && (!k || !dq || !dk || !gq || !gk)) || !dbeta || !dlambda || !gbeta || !glambda || (dg && !gg)) return LLATTN_ERR_NULL;
    if (q && llattn::misaligned(16, {q, k, dq, dk, gq, gk})) return LLATTN_ERR_ALIGNMENT;
    using bf = __nv_bfloat16;
    llattn::GdnGradOut a{(const bf*)q, (const bf*)k, dq, dk, dbeta, dlambda, dg, (bf*)gq, (bf*)gk, (bf*)gbeta, (bf*)glambda, gg, rep, rows, K, K_in, L, scale,
                         lambda_mul};
    if (!q && rep == 1 && !dg) {
        const unsigned bl = (unsigned)((rows * L + 1023) / 1024), bb = (unsigned)((rows + 1023) / 1024);
        llattn::launch_chained(llattn::gdn_grad_cast_kernel, bl + bb, 256, 0, (cudaStream_t)stream, a, bl);
        LLATTN_LAUNCHED();
        return (int)cudaGetLastError();
    }
    llattn::launch_chained(llattn::gdn_grad_out_kernel, (unsigned)((rows + 15) / 16), 256, 0, (cudaStream_t)stream, a);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

static int l2norm_check(const void* a, const void* b, long rows, int D) {
    if (rows <= 0 || D <= 0 || D > 256 || D % 8 != 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (!a || !b) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {a, b})) return LLATTN_ERR_ALIGNMENT;
    return 0;
}

int llattn_l2norm_fwd(const void* x, void* y, long rows, int D, float scale, void* stream) {
    int rc = l2norm_check(x, y, rows, D);
    if (rc != 0) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const __nv_bfloat16* xi = (const __nv_bfloat16*)x;
    __nv_bfloat16* yo = (__nv_bfloat16*)y;
    const int lpr = D <= 64 ? 8 : (D <= 128 ? 16 : 32);
    const long blocks = (rows * lpr + 255) / 256;
    if (lpr == 8) { llattn::launch_chained(llattn::l2norm_fwd_kernel<8>, (unsigned)blocks, 256, 0, st, xi, yo, rows, D, scale, 1e-6f); LLATTN_LAUNCHED(); }
    else if (lpr == 16) { llattn::launch_chained(llattn::l2norm_fwd_kernel<16>, (unsigned)blocks, 256, 0, st, xi, yo, rows, D, scale, 1e-6f); LLATTN_LAUNCHED(); }
    else { llattn::launch_chained(llattn::l2norm_fwd_kernel<32>, (unsigned)blocks, 256, 0, st, xi, yo, rows, D, scale, 1e-6f); LLATTN_LAUNCHED(); }
    return (int)cudaGetLastError();
}

int llattn_l2norm_bwd(const void* x, const float* dy, void* dx, long rows, int D, float scale, void* stream) {
    int rc = l2norm_check(x, dx, rows, D);
    if (rc != 0) return rc;
    if (!dy) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {dy})) return LLATTN_ERR_ALIGNMENT;
    cudaStream_t st = (cudaStream_t)stream;
    const __nv_bfloat16* xi = (const __nv_bfloat16*)x;
    __nv_bfloat16* o = (__nv_bfloat16*)dx;
    const int lpr = D <= 64 ? 8 : (D <= 128 ? 16 : 32);
    const long blocks = (rows * lpr + 255) / 256;
    if (lpr == 8) { llattn::launch_chained(llattn::l2norm_bwd_kernel<8>, (unsigned)blocks, 256, 0, st, xi, dy, o, rows, D, scale, 1e-6f); LLATTN_LAUNCHED(); }
    else if (lpr == 16) { llattn::launch_chained(llattn::l2norm_bwd_kernel<16>, (unsigned)blocks, 256, 0, st, xi, dy, o, rows, D, scale, 1e-6f); LLATTN_LAUNCHED(); }
    else { llattn::launch_chained(llattn::l2norm_bwd_kernel<32>, (unsigned)blocks, 256, 0, st, xi, dy, o, rows, D, scale, 1e-6f); LLATTN_LAUNCHED(); }
    return (int)cudaGetLastError();
}

}  // extern "C"
