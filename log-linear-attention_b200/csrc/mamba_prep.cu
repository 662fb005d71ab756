// Element-wise preparation of the log-linear Mamba-2 layer call and its backward for sm_100a (HBM-bound;
// one pass over the (B,T,H,.) tensors per direction instead of about six).
//
// Reference being replaced: the torch ops around the kernel in hmamba_chunk_scan_combined
// (hattention/mamba_apis.py:346-366, 401-402) and compute_lambda (:70-85):
//     dt  = softplus(dt_raw + dt_bias)          v = x * dt           g = A * dt
//     lam = softplus(L * dl) | exp(-exp(L) softplus(dl)) | L * dl    y = o + D * x
// Rounding points follow torch's type promotion for bf16 activations with fp32 parameters (the
// products are fp32 there): dt and g stay fp32, v and lam are rounded once to bf16 (the cast at the
// kernel boundary, hattention/kernel.py), y = o + D x is fp32 or bf16 as the caller asks.
#include "rowwise.cuh"
#include "../../include/llattn.h"

namespace llattn {

struct PrepArgs {
    const __nv_bfloat16 *x, *dt_raw, *dl;      // (rows,P), (rows), (rows,L)
    const void *dt_bias, *Lp, *D;              // (H) or null, (H,L), (H) or null
    const float* A;                            // (H)
    int bias_f32, lp_f32, d_f32;
    __nv_bfloat16 *v, *lam;
    float* g;
    const __nv_bfloat16 *dv, *dy;
    const float *dg, *dlam;
    __nv_bfloat16 *dx, *ddt, *ddl;
    float *dA, *dbias, *dLp, *dD;
    int H, P, L, mode;
    int tokens, run;                           // B T, and how many of them a thread walks
    int lpr;                                   // lanes of a head, 8 columns each
    int row_blocks, lam_blocks;                // blocks of the x part and of the lambda part per run; the latter come first
    int lam8, lam_runs;                        // the lambda columns come in eights, at 16-byte boundaries; runs of that part
};

// Both passes: a group of LPR lanes owns one head and walks `run` tokens, eight columns a lane.  What depends on the (token, head)
// alone is evaluated once by the group, each lane for one of LPR tokens, and the parameter sums stay in registers over the run.  The
// loads of a token are not fetched ahead: few registers and many warps keep more bytes in flight (B = 2, T = 16384, 32 heads, L = 15:
// backward 321 us with a row per group, a shared-memory atomic per lambda column and a token per thread before; 130 us as it is; 136 us
// with the next token in flight, 212 us with two and a thread per lambda column).
template <int LPR>
__global__ void __launch_bounds__(256, 6) m2_prep_fwd_kernel(const __grid_constant__ PrepArgs a) {
    chain_wait();
    constexpr int U = 2;
    const int lam_grid = a.lam_blocks * a.lam_runs;
    if ((int)blockIdx.x < lam_grid) {
        const int per = (a.tokens + a.lam_runs - 1) / a.lam_runs, t0 = blockIdx.x / a.lam_blocks * per, t1 = min(a.tokens, t0 + per);
        const LambdaCols c{a.dl, (long)a.H * a.L, a.Lp, a.lp_f32, a.H * a.L, a.mode};
        const int block = blockIdx.x % a.lam_blocks;
        if (a.lam8) lambda_part_fwd<8, 1>(c, a.lam, t0, t1, block, a.lam_blocks);
        else lambda_part_fwd<1, 1>(c, a.lam, t0, t1, block, a.lam_blocks);
        return;
    }
    const int at = blockIdx.x - lam_grid;
    const int t0 = at / a.row_blocks * a.run, t1 = min(a.tokens, t0 + a.run);
    const int lane = threadIdx.x % LPR;
    const int h = at % a.row_blocks * ((int)blockDim.x / LPR) + threadIdx.x / LPR;
    if (h >= a.H) return;                      // whole groups
    const unsigned group = LPR == 32 ? 0xffffffffu : ((1u << LPR) - 1u) << (threadIdx.x & 31 & ~(LPR - 1));
    const bool act = lane * 8 < a.P;
    const float bias = a.dt_bias ? load_param(a.dt_bias, h, a.bias_f32) : 0.f, A = a.A[h];
    const long xs = (long)a.H * a.P, off = (long)h * a.P + lane * 8;
    float dtl = 0.f;
    for (int t = t0; t < t1; t += U) {
        Packed<8> c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) c[u].load_if(a.x + (t + u) * xs + off, true, act && t + u < t1);
        if ((t - t0) % LPR == 0 && t + lane < t1) {
            dtl = softplus_row(__bfloat162float(a.dt_raw[(long)(t + lane) * a.H + h]) + bias);
            a.g[(long)(t + lane) * a.H + h] = A * dtl;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (t + u >= t1) break;
            const float dt = __shfl_sync(group, dtl, (t - t0 + u) % LPR, LPR);
            float y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = c[u][i] * dt;
            if (act) store_row<8>(a.v + (t + u) * xs + off, y, true);
        }
    }
}

// gradients: dx = dv * dt (+ D * dy), d dt_raw = (sum_p dv x + A dg) sigmoid(dt_raw + bias), d dl, and the parameter sums dA,
// d dt_bias, dD (H) and dL (H,L): one global atomic per thread and entry at the end of the run.
template <int LPR>
__global__ void __launch_bounds__(256, 4) m2_prep_bwd_kernel(const __grid_constant__ PrepArgs a) {
    chain_wait();
    const int lam_grid = a.lam_blocks * a.lam_runs;
    if ((int)blockIdx.x < lam_grid) {
        const int per = (a.tokens + a.lam_runs - 1) / a.lam_runs, t0 = blockIdx.x / a.lam_blocks * per, t1 = min(a.tokens, t0 + per);
        const LambdaCols c{a.dl, (long)a.H * a.L, a.Lp, a.lp_f32, a.H * a.L, a.mode};
        __shared__ float sums[256 * 8];
        const int block = blockIdx.x % a.lam_blocks;
        if (a.lam8) lambda_part_bwd<8, 2>(c, a.dlam, a.ddl, c.dl_stride, a.dLp, t0, t1, block, a.lam_blocks, sums);
        else lambda_part_bwd<1, 4>(c, a.dlam, a.ddl, c.dl_stride, a.dLp, t0, t1, block, a.lam_blocks, sums);
        return;
    }
    const int at = blockIdx.x - lam_grid;
    const int t0 = at / a.row_blocks * a.run, t1 = min(a.tokens, t0 + a.run);
    const int lane = threadIdx.x % LPR;
    const int h = at % a.row_blocks * ((int)blockDim.x / LPR) + threadIdx.x / LPR;
    if (h >= a.H) return;
    const unsigned group = LPR == 32 ? 0xffffffffu : ((1u << LPR) - 1u) << (threadIdx.x & 31 & ~(LPR - 1));
    const bool act = lane * 8 < a.P;
    const float bias = a.dt_bias ? load_param(a.dt_bias, h, a.bias_f32) : 0.f, A = a.A[h], D = a.D ? load_param(a.D, h, a.d_f32) : 0.f;
    const long xs = (long)a.H * a.P, off = (long)h * a.P + lane * 8;
    float raw = 0.f, dtl = 0.f, dotl = 0.f, sA = 0.f, sB = 0.f, sD = 0.f;
    for (int t = t0; t < t1; ++t) {
        Packed<8> cx, cv, cy;
        cx.load_if(a.x + t * xs + off, true, act);
        cv.load_if(a.dv + t * xs + off, true, act);
        cy.load_if(a.dy + t * xs + off, true, act && a.D != nullptr);
        const int k = (t - t0) % LPR;
        if (k == 0 && t + lane < t1) {
            raw = __bfloat162float(a.dt_raw[(long)(t + lane) * a.H + h]) + bias;
            dtl = softplus_row(raw);
        }
        const float dt = __shfl_sync(group, dtl, k, LPR);
        float y[8], dot = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float dv = cv[i], dy = cy[i], xv = cx[i];
            dot += dv * xv;
            sD += dy * xv;
            y[i] = dv * dt + D * dy;
        }
        if (act) store_row<8>(a.dx + t * xs + off, y, true);
#pragma unroll
        for (int d = LPR / 2; d > 0; d >>= 1) dot += __shfl_xor_sync(group, dot, d);
        if (k == lane) dotl = dot;
        if (k == LPR - 1 || t + 1 == t1) {
            // a block of LPR tokens (or the rest of the run) is complete: one token a lane
            const int tt = t - k + lane;
            if (lane <= k) {
                const float dgv = a.dg[(long)tt * a.H + h];
                const float d_raw = (dotl + A * dgv) * (raw > 20.f ? 1.f : sigmoid_row(raw));
                a.ddt[(long)tt * a.H + h] = __float2bfloat16(d_raw);
                sA += dgv * dtl;
                sB += d_raw;
            }
        }
    }
#pragma unroll
    for (int d = LPR / 2; d > 0; d >>= 1) {
        sA += __shfl_xor_sync(group, sA, d);
        sB += __shfl_xor_sync(group, sB, d);
        sD += __shfl_xor_sync(group, sD, d);
    }
    if (lane == 0) {
        atomicAdd(&a.dA[h], sA);
        if (a.dbias) atomicAdd(&a.dbias[h], sB);
        if (a.D) atomicAdd(&a.dD[h], sD);
    }
}

template <int LPR, bool F32OUT>
__global__ void __launch_bounds__(256) m2_residual_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ x,
                                                          const float* __restrict__ D, void* __restrict__ y, long rows, int H, int P) {
    chain_wait();
    const int lane = threadIdx.x % LPR;
    const long row = ((long)blockIdx.x * blockDim.x + threadIdx.x) / LPR;
    if (row >= rows || lane * 8 >= P) return;
    const float d = D[row % H];
    const uint4 ro = *reinterpret_cast<const uint4*>(o + row * P + lane * 8);
    const uint4 rx = *reinterpret_cast<const uint4*>(x + row * P + lane * 8);
    const __nv_bfloat162* ho = reinterpret_cast<const __nv_bfloat162*>(&ro);
    const __nv_bfloat162* hx = reinterpret_cast<const __nv_bfloat162*>(&rx);
    float r[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        r[2 * i] = __bfloat162float(ho[i].x) + __bfloat162float(hx[i].x) * d;
        r[2 * i + 1] = __bfloat162float(ho[i].y) + __bfloat162float(hx[i].y) * d;
    }
    if (F32OUT) {
        float* yo = reinterpret_cast<float*>(y) + row * P + lane * 8;
        *reinterpret_cast<float4*>(yo) = make_float4(r[0], r[1], r[2], r[3]);
        *reinterpret_cast<float4*>(yo + 4) = make_float4(r[4], r[5], r[6], r[7]);
    } else {
        uint4 out;
        __nv_bfloat162* w = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = __floats2bfloat162_rn(r[2 * i], r[2 * i + 1]);
        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(y) + row * P + lane * 8) = out;
    }
}

static int lanes_per_row(int P) { return P <= 32 ? 4 : (P <= 64 ? 8 : (P <= 128 ? 16 : 32)); }

}  // namespace llattn

extern "C" {

static int prep_check(long rows, int H, int P, int L, int mode) {
    if (rows <= 0 || H <= 0 || rows % H != 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (P <= 0 || P > 256 || P % 8 != 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (L <= 0 || L > 64 || mode < 0 || mode > 2) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    return 0;
}

// Grid of a pass: runs long enough that the sums at their end are cheap, as many as fill the chip
static unsigned prep_grid(llattn::PrepArgs& a, long rows, int H, int P, int L, int mode, bool backward, int& threads) {
    a.H = H; a.P = P; a.L = L; a.mode = mode;
    a.tokens = (int)(rows / H);
    a.lpr = llattn::lanes_per_row(P);
    // few heads: smaller CTAs rather than idle threads
    const int want = (H * a.lpr + 31) / 32 * 32;
    threads = want < 64 ? 64 : want > 256 ? 256 : want;
    a.row_blocks = (H * a.lpr + threads - 1) / threads;
    a.lam8 = H * L % 8 == 0 && !llattn::misaligned(16, {a.dl, a.lam, a.dlam, a.ddl});
    a.lam_blocks = (H * L / (a.lam8 ? 8 : 1) + threads - 1) / threads;
    a.run = 64;
    while (a.run > (backward ? 8 : 4) && (long)a.row_blocks * ((a.tokens + a.run - 1) / a.run) * threads < 148 * 8 * 256) a.run /= 2;
    // forward: eight tokens a thread
    const int groups = H * L / (a.lam8 ? 8 : 1), per = groups < threads ? threads / groups : 1;
    a.lam_runs = backward ? llattn::lambda_runs(a.tokens, a.lam_blocks, a.lam8) : (a.tokens + 8 * per - 1) / (8 * per);
    return (unsigned)(a.row_blocks * ((a.tokens + a.run - 1) / a.run) + a.lam_blocks * a.lam_runs);
}

int llattn_mamba2_layer_prep_fwd(const void* x, const void* dt_raw, const void* dt_bias, int bias_is_f32, const float* A, const void* dl,
                                 const void* Lp, int lp_is_f32, void* v, float* g, void* lambda, long rows, int H, int P, int L,
                                 int lambda_mode, void* stream) {
    int rc = prep_check(rows, H, P, L, lambda_mode);
    if (rc != 0) return rc;
    if (!x || !dt_raw || !A || !dl || !Lp || !v || !g || !lambda) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {x, v})) return LLATTN_ERR_ALIGNMENT;
    using bf = __nv_bfloat16;
    cudaStream_t st = (cudaStream_t)stream;
    llattn::PrepArgs a = {};
    a.x = (const bf*)x; a.dt_raw = (const bf*)dt_raw; a.dl = (const bf*)dl; a.dt_bias = dt_bias; a.A = A; a.Lp = Lp;
    a.bias_f32 = bias_is_f32; a.lp_f32 = lp_is_f32;
    a.v = (bf*)v; a.lam = (bf*)lambda; a.g = g;
    int threads;
    const unsigned grid = prep_grid(a, rows, H, P, L, lambda_mode, false, threads);
    if (a.lpr == 4) llattn::launch_chained(llattn::m2_prep_fwd_kernel<4>, grid, threads, 0, st, a);
    else if (a.lpr == 8) llattn::launch_chained(llattn::m2_prep_fwd_kernel<8>, grid, threads, 0, st, a);
    else if (a.lpr == 16) llattn::launch_chained(llattn::m2_prep_fwd_kernel<16>, grid, threads, 0, st, a);
    else llattn::launch_chained(llattn::m2_prep_fwd_kernel<32>, grid, threads, 0, st, a);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int llattn_mamba2_prep_fwd(const void* x, const void* dt_raw, const float* dt_bias, const float* A, const void* dl, const float* Lp,
                           void* v, float* g, void* lambda, long rows, int H, int P, int L, int lambda_mode, void* stream) {
    return llattn_mamba2_layer_prep_fwd(x, dt_raw, dt_bias, 1, A, dl, Lp, 1, v, g, lambda, rows, H, P, L, lambda_mode, stream);
}

int llattn_mamba2_layer_prep_bwd(const void* x, const void* dt_raw, const void* dt_bias, int bias_is_f32, const float* A, const void* dl,
                                 const void* Lp, int lp_is_f32, const void* D, int d_is_f32, const void* dv, const float* dg,
                                 const float* dlambda, const void* dy, void* dx, void* ddt, void* ddl, float* dA, float* dbias,
                                 float* dLp, float* dD, long rows, int H, int P, int L, int lambda_mode, void* stream) {
    int rc = prep_check(rows, H, P, L, lambda_mode);
    if (rc != 0) return rc;
    if (!x || !dt_raw || !A || !dl || !Lp || !dv || !dg || !dlambda || !dx || !ddt || !ddl || !dA || !dLp) return LLATTN_ERR_NULL;
    if (D && (!dy || !dD)) return LLATTN_ERR_NULL;
    if (dt_bias && !dbias) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {x, dv, dx}) || (D && llattn::misaligned(16, {dy}))) return LLATTN_ERR_ALIGNMENT;
    using bf = __nv_bfloat16;
    cudaStream_t st = (cudaStream_t)stream;
    llattn::PrepArgs a = {};
    a.x = (const bf*)x; a.dt_raw = (const bf*)dt_raw; a.dl = (const bf*)dl; a.dt_bias = dt_bias; a.A = A; a.Lp = Lp; a.D = D;
    a.bias_f32 = bias_is_f32; a.lp_f32 = lp_is_f32; a.d_f32 = d_is_f32;
    a.dv = (const bf*)dv; a.dg = dg; a.dlam = dlambda; a.dy = (const bf*)dy;
    a.dx = (bf*)dx; a.ddt = (bf*)ddt; a.ddl = (bf*)ddl; a.dA = dA; a.dbias = dt_bias ? dbias : nullptr; a.dLp = dLp; a.dD = dD;
    int threads;
    const unsigned grid = prep_grid(a, rows, H, P, L, lambda_mode, true, threads);
    if (a.lpr == 4) llattn::launch_chained(llattn::m2_prep_bwd_kernel<4>, grid, threads, 0, st, a);
    else if (a.lpr == 8) llattn::launch_chained(llattn::m2_prep_bwd_kernel<8>, grid, threads, 0, st, a);
    else if (a.lpr == 16) llattn::launch_chained(llattn::m2_prep_bwd_kernel<16>, grid, threads, 0, st, a);
    else llattn::launch_chained(llattn::m2_prep_bwd_kernel<32>, grid, threads, 0, st, a);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int llattn_mamba2_prep_bwd(const void* x, const void* dt_raw, const float* dt_bias, const float* A, const void* dl, const float* Lp,
                           const float* D, const void* dv, const float* dg, const float* dlambda, const void* dy,
                           void* dx, void* ddt, void* ddl, float* dA, float* dbias, float* dLp, float* dD,
                           long rows, int H, int P, int L, int lambda_mode, void* stream) {
    return llattn_mamba2_layer_prep_bwd(x, dt_raw, dt_bias, 1, A, dl, Lp, 1, D, 1, dv, dg, dlambda, dy, dx, ddt, ddl, dA, dbias, dLp, dD, rows, H,
                                        P, L, lambda_mode, stream);
}

int llattn_mamba2_residual(const void* o, const void* x, const float* D, void* y, int y_is_f32, long rows, int H, int P, void* stream) {
    int rc = prep_check(rows, H, P, 1, 0);
    if (rc != 0) return rc;
    if (!o || !x || !D || !y) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {o, x, y})) return LLATTN_ERR_ALIGNMENT;
    using bf = __nv_bfloat16;
    cudaStream_t st = (cudaStream_t)stream;
    const int lpr = llattn::lanes_per_row(P);
    const unsigned blocks = (unsigned)((rows * lpr + 255) / 256);
#define RES(LPRV)                                                                                                          \
    do {                                                                                                                   \
        if (y_is_f32) llattn::launch_chained(llattn::m2_residual_kernel<LPRV, true>, blocks, 256, 0, st, (const bf*)o, (const bf*)x, D, y, rows, H, P);   \
        else llattn::launch_chained(llattn::m2_residual_kernel<LPRV, false>, blocks, 256, 0, st, (const bf*)o, (const bf*)x, D, y, rows, H, P);           \
    } while (0)
    if (lpr == 4) RES(4);
    else if (lpr == 8) RES(8);
    else if (lpr == 16) RES(16);
    else RES(32);
#undef RES
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

}  // extern "C"
