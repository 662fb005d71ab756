// What the log-linear Mamba-2 mixer does around the scan, for sm_100a: depthwise causal convolution + SiLU with the scan's
// preparation, the D residual with the gated RMSNorm, and the backward of both.
//
// Reference being replaced: hmamba_split_conv1d_scan_combined (hattention/mamba_apis.py:116-262), which calls causal_conv1d and
// mamba_ssm kernels for the convolution and the norm and torch operators for the rest.
//
// All four passes are bound by HBM.  They read the rows of the projection zxbcdtdl = [z | x B C | dt | dl] in place (no split
// copies), and the backward writes its slices of the gradient of that row in place (no concatenation).  At B = 1, T = 8192, 48
// heads of 64, N = 128 the torch operators took 3.2 ms of a 4.3 ms forward + backward step, most of it in transposes to and from
// the (B, D, T) layout of the library convolution, its three kernels (0.95 ms) and fp32 temporaries of the norm.
#include "rowwise.cuh"
#include "../../include/llattn.h"

namespace llattn {

constexpr int MX_P = 64;              // head width
constexpr int MX_W = 4;               // taps of the convolution

struct MixerArgs {
    const bf16* zx;            // (B,T,W) rows [z (dim) | x (dim) | B (GN) | C (GN) | dt (H) | dl (H L)]
    const void *conv_w, *conv_b;   // (dim + 2GN, 4), (dim + 2GN) or null
    const void *dt_bias, *Lp;  // (H), (H,L)
    const float* A;            // (H)
    int conv_w_f32, conv_b_f32, bias_f32, lp_f32;
    // forward results
    bf16 *x, *v, *k, *q;       // (B,T,H,P) twice, (B,T,G,N) twice: k is B, q is C
    float* g;                  // (B,T,H)
    bf16* lam;                 // (B,T,H,L)
    // backward inputs
    const bf16 *dv, *dy, *dq, *dk;
    const float *dg, *dlam;
    const void* D;             // (H) or null
    int d_f32;
    // backward results
    bf16* dzx;                 // (B,T,W); the z slice is written by the norm's backward
    float *dconv_w, *dconv_b;  // accumulated into cleared buffers, like the three below
    float *dA, *dbias, *dLp;
    int B, T, H, L, dim, gn, W, mode;
    int run;                   // tokens a thread walks
    int conv_blocks, lam_blocks;   // blocks of the convolution part and of the lambda part per run; the latter come first
    int lam8, lam_runs;        // the lambda columns come in eights, at 16-byte boundaries; runs of a sequence in that part
};

// ---- forward: a thread walks `run` tokens of four neighbouring channels, eight tokens at a time, with the last three inputs in
// registers.  The sixteen threads of a head share softplus(dt): each evaluates the one of a token in sixteen.
__global__ void __launch_bounds__(128, 6) mixer_prep_kernel(const __grid_constant__ MixerArgs a) {
    chain_wait();
    constexpr int N = 4, U = 8;
    const bool vec = (a.W & 3) == 0;
    const int lam_grid = a.lam_blocks * a.B * a.lam_runs;
    if ((int)blockIdx.x < lam_grid) {
        const int nr = a.lam_runs, q = blockIdx.x / a.lam_blocks;
        const int b = q / nr, per = (a.T + nr - 1) / nr, t0 = (q % nr) * per, t1 = min(a.T, t0 + per);
        const bf16* rows = a.zx + (long)b * a.T * a.W + 2 * a.dim + 2 * a.gn;
        const LambdaCols c{rows + a.H, a.W, a.Lp, a.lp_f32, a.H * a.L, a.mode};
        const int block = blockIdx.x % a.lam_blocks;
        bf16* lam = a.lam + (long)b * a.T * a.H * a.L;
        if (a.lam8) lambda_part_fwd<8, 2>(c, lam, t0, t1, block, a.lam_blocks);
        else lambda_part_fwd<1, 2>(c, lam, t0, t1, block, a.lam_blocks);
        return;
    }
    const int nrun = (a.T + a.run - 1) / a.run, at = (blockIdx.x - lam_grid) / a.conv_blocks;
    const int b = at / nrun, t0 = (at % nrun) * a.run, t1 = min(a.T, t0 + a.run);
    const int c0 = ((blockIdx.x - lam_grid) % a.conv_blocks * 128 + threadIdx.x) * N;
    if (c0 >= a.dim + 2 * a.gn) return;          // whole groups of sixteen threads (a head, or 64 of the B / C channels)
    float w[MX_W][N], bias[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        bias[i] = a.conv_b ? round_bf16(load_param(a.conv_b, c0 + i, a.conv_b_f32)) : 0.f;
#pragma unroll
        for (int j = 0; j < MX_W; ++j) w[j][i] = round_bf16(load_param(a.conv_w, (c0 + i) * MX_W + j, a.conv_w_f32));
    }
    const bf16* in = a.zx + (long)b * a.T * a.W + a.dim + c0;
    const bool is_x = c0 < a.dim;
    const int h = c0 / MX_P, lane16 = threadIdx.x & 15;
    const unsigned group = 0xffffu << (threadIdx.x & 16);
    const float A = is_x ? a.A[h] : 0.f;
    const float dtb = is_x && a.dt_bias ? load_param(a.dt_bias, h, a.bias_f32) : 0.f;
    const bf16* dts = a.zx + (long)b * a.T * a.W + 2 * a.dim + 2 * a.gn + h;
    bf16* out;
    int ostride;
    if (is_x) { out = a.x + (long)b * a.T * a.dim + c0; ostride = a.dim; }
    else if (c0 < a.dim + a.gn) { out = a.k + (long)b * a.T * a.gn + c0 - a.dim; ostride = a.gn; }
    else { out = a.q + (long)b * a.T * a.gn + c0 - a.dim - a.gn; ostride = a.gn; }
    // win[0..2]: tokens t - 3 .. t - 1; win[3 + u]: tokens of this group
    Packed<N> win[MX_W - 1 + U];
#pragma unroll
    for (int j = 0; j < MX_W - 1; ++j) {
        const int t = t0 - (MX_W - 1) + j;
        win[j].zero();
        if (t >= 0) win[j].load(in + (long)t * a.W, vec);
    }
    float dt16 = 0.f;
    for (int t = t0; t < t1; t += U) {
#pragma unroll
        for (int u = 0; u < U; ++u) win[MX_W - 1 + u].load_if(in + (long)(t + u) * a.W, vec, t + u < t1);
        if (is_x && ((t - t0) & 15) == 0 && t + lane16 < t1) {
            dt16 = softplus_row(__bfloat162float(dts[(long)(t + lane16) * a.W]) + dtb);
            a.g[((long)b * a.T + t + lane16) * a.H + h] = A * dt16;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (t + u >= t1) break;
            float y[N];
#pragma unroll
            for (int i = 0; i < N; ++i) {
                float s = bias[i];
#pragma unroll
                for (int j = 0; j < MX_W; ++j) s += w[j][i] * win[u + j][i];
                s = round_bf16(s);                   // the convolution's output, as a separate operator returns it
                y[i] = s * sigmoid_row(s);
            }
            store_row<N>(out + (long)(t + u) * ostride, y, true);
            if (is_x) {
                const float dt = __shfl_sync(group, dt16, (t - t0 + u) & 15, 16);
#pragma unroll
                for (int i = 0; i < N; ++i) y[i] = round_bf16(y[i]) * dt;
                store_row<N>(a.v + ((long)b * a.T + t + u) * a.dim + c0, y, true);
            }
        }
#pragma unroll
        for (int j = 0; j < MX_W - 1; ++j) win[j] = win[U + j];
    }
}

// ---- backward of the convolution and the preparation.  A thread walks the tokens of four channels; at token t it has the
// gradient before the activation of t, so the input gradient of t - 3 is complete.  The three tokens behind a run's end are
// evaluated by the next run too.  Sums over tokens (taps, bias, A, dt_bias) stay in registers until the end of the run, and the
// sixteen threads of a head share what depends on the token alone: each has one token of a block of sixteen.
__global__ void __launch_bounds__(128, 4) mixer_prep_bwd_kernel(const __grid_constant__ MixerArgs a) {
    chain_wait();
    constexpr int N = 4, U = 4;
    const bool vec = (a.W & 3) == 0;
    const int lam_grid = a.lam_blocks * a.B * a.lam_runs;
    if ((int)blockIdx.x < lam_grid) {
        __shared__ float sums[128 * 8];
        const int nr = a.lam_runs, q = blockIdx.x / a.lam_blocks;
        const int b = q / nr, per = (a.T + nr - 1) / nr, t0 = (q % nr) * per, t1 = min(a.T, t0 + per);
        const long row0 = (long)b * a.T;
        const long off = row0 * a.W + 2 * a.dim + 2 * a.gn + a.H;
        const LambdaCols c{a.zx + off, a.W, a.Lp, a.lp_f32, a.H * a.L, a.mode};
        const int block = blockIdx.x % a.lam_blocks;
        const float* dlam = a.dlam + row0 * a.H * a.L;
        if (a.lam8) lambda_part_bwd<8, 2>(c, dlam, a.dzx + off, a.W, a.dLp, t0, t1, block, a.lam_blocks, sums);
        else lambda_part_bwd<1, 4>(c, dlam, a.dzx + off, a.W, a.dLp, t0, t1, block, a.lam_blocks, sums);
        return;
    }
    const int nrun = (a.T + a.run - 1) / a.run, at = (blockIdx.x - lam_grid) / a.conv_blocks;
    const int b = at / nrun, t0 = (at % nrun) * a.run, t1 = min(a.T, t0 + a.run);
    const int c0 = ((blockIdx.x - lam_grid) % a.conv_blocks * 128 + threadIdx.x) * N;
    if (c0 >= a.dim + 2 * a.gn) return;             // whole groups of sixteen threads
    const long row0 = (long)b * a.T;
    const bool is_x = c0 < a.dim;
    const int h = is_x ? c0 / MX_P : 0, lane16 = threadIdx.x & 15;
    const unsigned group = 0xffffu << (threadIdx.x & 16);
    float w[MX_W][N], bias[N], dw[MX_W][N], db[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        bias[i] = a.conv_b ? round_bf16(load_param(a.conv_b, c0 + i, a.conv_b_f32)) : 0.f;
        db[i] = 0.f;
#pragma unroll
        for (int j = 0; j < MX_W; ++j) {
            w[j][i] = round_bf16(load_param(a.conv_w, (c0 + i) * MX_W + j, a.conv_w_f32));
            dw[j][i] = 0.f;
        }
    }
    const bf16* in = a.zx + row0 * a.W + a.dim + c0;
    const int dt_off = 2 * a.dim + 2 * a.gn + h;
    const float dtb = is_x && a.dt_bias ? load_param(a.dt_bias, h, a.bias_f32) : 0.f;
    const float Ah = is_x ? a.A[h] : 0.f, Dh = is_x && a.D ? load_param(a.D, h, a.d_f32) : 0.f;
    const bool use_dy = is_x && a.D != nullptr;
    const bf16 *up, *up2 = nullptr;
    int ustride = a.dim;
    if (is_x) {
        up = a.dv + row0 * a.dim + c0;
        if (use_dy) up2 = a.dy + row0 * a.dim + c0;
    } else {
        up = c0 < a.dim + a.gn ? a.dk + row0 * a.gn + c0 - a.dim : a.dq + row0 * a.gn + c0 - a.dim - a.gn;
        ustride = a.gn;
    }
    const int tend = min(t1 + MX_W - 1, a.T);       // tokens whose gradient before the activation is needed
    Packed<N> win[MX_W - 1 + U];
    float dp[MX_W - 1][N];
#pragma unroll
    for (int j = 0; j < MX_W - 1; ++j) {
        const int t = t0 - (MX_W - 1) + j;
        win[j].zero();
        if (t >= 0) win[j].load(in + (long)t * a.W, vec);
#pragma unroll
        for (int i = 0; i < N; ++i) dp[j][i] = 0.f;
    }
    float sA = 0.f, sB = 0.f, raw16 = 0.f, dt16 = 0.f, dot16 = 0.f;
    // tokens t1 .. t1 + 2 beyond the end of the sequence contribute zeros
    for (int t = t0; t < t1 + MX_W - 1; t += U) {
        Packed<N> cd[U], cy[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool p = t + u < tend;
            win[MX_W - 1 + u].load_if(in + (long)(t + u) * a.W, vec, p);
            cd[u].load_if(up + (long)(t + u) * ustride, true, p);
            cy[u].load_if(up2 + (long)(t + u) * ustride, true, p && use_dy);
        }
        if (is_x && ((t - t0) & 15) == 0) {
            raw16 = t + lane16 < tend ? __bfloat162float(a.zx[(row0 + t + lane16) * a.W + dt_off]) + dtb : 0.f;
            dt16 = softplus_row(raw16);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int tt = t + u;
            float dpt[N];
#pragma unroll
            for (int i = 0; i < N; ++i) dpt[i] = 0.f;
            if (tt < tend) {
                const float dt = is_x ? __shfl_sync(group, dt16, (tt - t0) & 15, 16) : 1.f;
                float dot = 0.f;
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    float s = bias[i];
#pragma unroll
                    for (int j = 0; j < MX_W; ++j) s += w[j][i] * win[u + j][i];
                    s = round_bf16(s);
                    const float sg = sigmoid_row(s), d = cd[u][i];
                    dot += d * round_bf16(s * sg);
                    dpt[i] = (d * dt + Dh * cy[u][i]) * sg * (1.f + s * (1.f - sg));
                }
                if (tt < t1) {
#pragma unroll
                    for (int i = 0; i < N; ++i) {
                        db[i] += dpt[i];
#pragma unroll
                        for (int j = 0; j < MX_W; ++j) dw[j][i] += dpt[i] * win[u + j][i];
                    }
                    if (is_x) {
#pragma unroll
                        for (int q = 8; q > 0; q >>= 1) dot += __shfl_xor_sync(group, dot, q);
                        if (((tt - t0) & 15) == lane16) dot16 = dot;
                    }
                }
            }
            const int to = tt - (MX_W - 1);
            if (to >= t0 && to < t1) {
                float di[N];
#pragma unroll
                for (int i = 0; i < N; ++i) di[i] = w[3][i] * dp[0][i] + w[2][i] * dp[1][i] + w[1][i] * dp[2][i] + w[0][i] * dpt[i];
                store_row<N>(a.dzx + (row0 + to) * a.W + a.dim + c0, di, vec);
            }
#pragma unroll
            for (int i = 0; i < N; ++i) {
                dp[0][i] = dp[1][i];
                dp[1][i] = dp[2][i];
                dp[2][i] = dpt[i];
            }
        }
        if (is_x && (((t - t0) & 15) == 16 - U || t + U >= t1 + MX_W - 1)) {
            // the block of sixteen tokens, or what the run has of it, is complete: one token a thread
            const int tt = t - ((t - t0) & 15) + lane16;
            if (tt < t1) {
                const float dgv = a.dg[(row0 + tt) * a.H + h];
                const float draw = (dot16 + Ah * dgv) * (raw16 > 20.f ? 1.f : sigmoid_row(raw16));
                a.dzx[(row0 + tt) * a.W + dt_off] = __float2bfloat16(draw);
                sA += dgv * dt16;
                sB += draw;
            }
        }
#pragma unroll
        for (int j = 0; j < MX_W - 1; ++j) win[j] = win[U + j];
    }
    if (a.conv_b) red_add_f32x4(a.dconv_b + c0, db[0], db[1], db[2], db[3]);
#pragma unroll
    for (int i = 0; i < N; ++i) red_add_f32x4(a.dconv_w + (c0 + i) * MX_W, dw[0][i], dw[1][i], dw[2][i], dw[3][i]);
    if (is_x) {
#pragma unroll
        for (int q = 8; q > 0; q >>= 1) {
            sA += __shfl_xor_sync(group, sA, q);
            sB += __shfl_xor_sync(group, sB, q);
        }
        if (lane16 == 0) {
            atomicAdd(&a.dA[h], sA);
            if (a.dt_bias) atomicAdd(&a.dbias[h], sB);
        }
    }
}

struct NormArgs {
    const bf16* o;             // (B T, dim)
    const bf16* x;             // (B T, dim), used with D
    const bf16* zx;            // z = first dim columns of rows of W
    const void *D, *w;         // (H) or null, (dim)
    int d_f32, w_f32;
    bf16* out;                 // (B T, dim)
    float* rstd;               // (B T)
    const bf16* dn;            // (B T, dim) gradient of out
    bf16* dy;                  // (B T, dim)
    bf16* dzx;
    float *dw, *dD;            // accumulated into cleared buffers
    int rows, dim, W;
    float eps;
};

// y = o + D x: fp32 with an fp32 D, else rounded once to bf16, as the residual pass of the layer call writes it
__device__ __forceinline__ float mixer_y(float o, float x, float d, bool have_d, bool d_f32) {
    const float y = o + x * d;
    return !have_d ? o : d_f32 ? y : round_bf16(y);
}

// sum over the CTA (at most 16 warps); s: two rows used in turn, so that one barrier a call is enough
__device__ __forceinline__ float block_sum(float v, float (&s)[2][16], int turn) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if (lane == 0) s[turn][warp] = v;
    __syncthreads();
    float r = lane < nw ? s[turn][lane] : 0.f;
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) r += __shfl_xor_sync(0xffffffffu, r, d);
    return __shfl_sync(0xffffffffu, r, 0);
}

// ---- out = RMSNorm((o + D x) silu(z)) w, one CTA a token, NV groups of eight columns a thread
template <int NV>
__global__ void __launch_bounds__(512) mixer_norm_kernel(const __grid_constant__ NormArgs a) {
    chain_wait();
    __shared__ float sred[2][16];
    const int tid = threadIdx.x;
    const bool vec = (a.W & 7) == 0;
    const long row = blockIdx.x;
    float s[NV][8];
    float ss = 0.f;
#pragma unroll
    for (int n = 0; n < NV; ++n) {
        const int c = (n * blockDim.x + tid) * 8;
        if (c >= a.dim) continue;
        Packed<8> o, x, z;
        o.load(a.o + row * a.dim + c, true);
        z.load(a.zx + row * a.W + c, vec);
        x.load_if(a.x + row * a.dim + c, true, a.D != nullptr);
        const float d = a.D ? load_param(a.D, c / MX_P, a.d_f32) : 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            s[n][i] = mixer_y(o[i], x[i], d, a.D != nullptr, a.d_f32) * z[i] * sigmoid_row(z[i]);
            ss += s[n][i] * s[n][i];
        }
    }
    const float rstd = rsqrtf(block_sum(ss, sred, 0) / (float)a.dim + a.eps);
    if (tid == 0) a.rstd[row] = rstd;
#pragma unroll
    for (int n = 0; n < NV; ++n) {
        const int c = (n * blockDim.x + tid) * 8;
        if (c >= a.dim) continue;
        float y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = s[n][i] * rstd * load_param(a.w, c + i, a.w_f32);
        store_row<8>(a.out + row * a.dim + c, y, true);
    }
}

// ---- its backward: persistent CTAs walk the tokens, so that the sums over tokens (w, D) stay in registers
template <int NV, int THREADS>
__global__ void __launch_bounds__(THREADS, NV == 1 ? 768 / THREADS : 1) mixer_norm_bwd_kernel(const __grid_constant__ NormArgs a) {
    chain_wait();
    __shared__ float sred[2][16];
    const int tid = threadIdx.x, lane = tid & 31;
    int turn = 0;
    const bool vec = (a.W & 7) == 0;
    float w[NV][8], dw[NV][8], d[NV], dD[NV];
#pragma unroll
    for (int n = 0; n < NV; ++n) {
        const int c = (n * THREADS + tid) * 8;
        const bool act = c < a.dim;
        d[n] = act && a.D ? load_param(a.D, c / MX_P, a.d_f32) : 0.f;
        dD[n] = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            w[n][i] = act ? load_param(a.w, c + i, a.w_f32) : 0.f;
            dw[n][i] = 0.f;
        }
    }
    for (long row = blockIdx.x; row < a.rows; row += gridDim.x) {
        Packed<8> o[NV], x[NV], z[NV], dn[NV];
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const int c = (n * THREADS + tid) * 8;
            const bool p = c < a.dim;
            o[n].load_if(a.o + row * a.dim + c, true, p);
            z[n].load_if(a.zx + row * a.W + c, vec, p);
            dn[n].load_if(a.dn + row * a.dim + c, true, p);
            x[n].load_if(a.x + row * a.dim + c, true, p && a.D != nullptr);
        }
        const float rstd = a.rstd[row];
        float y[NV][8], sg[NV][8], dot = 0.f;
#pragma unroll
        for (int n = 0; n < NV; ++n)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                y[n][i] = mixer_y(o[n][i], x[n][i], d[n], a.D != nullptr, a.d_f32);
                sg[n][i] = sigmoid_row(z[n][i]);
                const float s = y[n][i] * z[n][i] * sg[n][i], e = dn[n][i] * s;
                dw[n][i] += e * rstd;
                dot += e * w[n][i];
            }
        turn ^= 1;
        const float m = block_sum(dot, sred, turn) * rstd * rstd * rstd / (float)a.dim;
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const int c = (n * THREADS + tid) * 8;
            if (c >= a.dim) continue;
            float dy[8], dz[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float g = sg[n][i], si = z[n][i] * g, yy = y[n][i];
                const float ds = dn[n][i] * w[n][i] * rstd - yy * si * m;
                dy[i] = ds * si;
                dz[i] = ds * yy * (g + si * (1.f - g));
                dD[n] += round_bf16(dy[i]) * x[n][i];
            }
            store_row<8>(a.dy + row * a.dim + c, dy, true);
            store_row<8>(a.dzx + row * a.W + c, dz, vec);
        }
    }
#pragma unroll
    for (int n = 0; n < NV; ++n) {
        const int c = (n * THREADS + tid) * 8;
        // the eight lanes of a head
        float t = dD[n];
#pragma unroll
        for (int q = 4; q > 0; q >>= 1) t += __shfl_xor_sync(0xffffffffu, t, q);
        if (c >= a.dim) continue;
        if (a.D && (lane & 7) == 0) atomicAdd(&a.dD[c / MX_P], t);
        red_add_f32x4(a.dw + c, dw[n][0], dw[n][1], dw[n][2], dw[n][3]);
        red_add_f32x4(a.dw + c + 4, dw[n][4], dw[n][5], dw[n][6], dw[n][7]);
    }
}

}  // namespace llattn

extern "C" {

static int mixer_check(int B, int T, int H, int G, int N, int L, int mode) {
    if (B <= 0 || T <= 0 || H <= 0 || G <= 0 || H % G != 0 || N <= 0 || N % 64 != 0) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    if (L <= 0 || L > 64 || mode < 0 || mode > 2 || H * llattn::MX_P > 8192) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    return 0;
}

// tokens a thread walks: long enough that the halo and the final sums are cheap, short enough to give the chip `warps` of them
static int mixer_run(int B, int T, int warps_per_run, int lo, int hi, long warps) {
    int run = hi;
    while (run > lo && (long)B * ((T + run - 1) / run) * warps_per_run < warps) run /= 2;
    return run;
}

static void mixer_lambda_blocks(llattn::MixerArgs& a, bool backward) {
    a.lam8 = a.H * a.L % 8 == 0 && a.W % 8 == 0 && a.H % 8 == 0;
    a.lam_blocks = (a.H * a.L / (a.lam8 ? 8 : 1) + 127) / 128;
    // forward: eight tokens a thread
    const int groups = a.H * a.L / (a.lam8 ? 8 : 1), rows = groups < 128 ? 128 / groups : 1;
    a.lam_runs = backward ? llattn::lambda_runs(a.T, a.lam_blocks * a.B, a.lam8) : (a.T + 8 * rows - 1) / (8 * rows);
}

int llattn_mixer_prep_fwd(const void* zx, const void* conv_w, int conv_w_f32, const void* conv_b, int conv_b_f32, const void* dt_bias,
                          int bias_f32, const float* A, const void* Lp, int lp_f32, void* x, void* v, void* k, void* q, float* g,
                          void* lambda, int B, int T, int H, int G, int N, int L, int lambda_mode, void* stream) {
    const int rc = mixer_check(B, T, H, G, N, L, lambda_mode);
    if (rc != 0) return rc;
    if (!zx || !conv_w || !A || !Lp || !x || !v || !k || !q || !g || !lambda) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {zx, x, v, k, q, lambda})) return LLATTN_ERR_ALIGNMENT;
    using bf = __nv_bfloat16;
    llattn::MixerArgs a = {};
    a.zx = (const bf*)zx; a.conv_w = conv_w; a.conv_w_f32 = conv_w_f32; a.conv_b = conv_b; a.conv_b_f32 = conv_b_f32;
    a.dt_bias = dt_bias; a.bias_f32 = bias_f32; a.A = A; a.Lp = Lp; a.lp_f32 = lp_f32;
    a.x = (bf*)x; a.v = (bf*)v; a.k = (bf*)k; a.q = (bf*)q; a.g = g; a.lam = (bf*)lambda;
    a.B = B; a.T = T; a.H = H; a.L = L; a.dim = H * llattn::MX_P; a.gn = G * N; a.W = 2 * a.dim + 2 * a.gn + H + H * L; a.mode = lambda_mode;
    const int ch = a.dim + 2 * a.gn;
    a.conv_blocks = (ch / 4 + 127) / 128;
    a.run = mixer_run(B, T, ch / 128 + 1, 16, 64, 148 * 20);
    mixer_lambda_blocks(a, false);
    const unsigned grid = (unsigned)(a.conv_blocks * B * ((T + a.run - 1) / a.run) + a.lam_blocks * B * a.lam_runs);
    llattn::launch_chained(llattn::mixer_prep_kernel, grid, 128, 0, (cudaStream_t)stream, a);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int llattn_mixer_prep_bwd(const void* zx, const void* conv_w, int conv_w_f32, const void* conv_b, int conv_b_f32, const void* dt_bias,
                          int bias_f32, const float* A, const void* Lp, int lp_f32, const void* D, int d_f32, const void* dv, const void* dy,
                          const void* dq, const void* dk, const float* dg, const float* dlambda, void* dzx, float* dconv_w, float* dconv_b,
                          float* dA, float* dbias, float* dLp, int B, int T, int H, int G, int N, int L, int lambda_mode, void* stream) {
    const int rc = mixer_check(B, T, H, G, N, L, lambda_mode);
    if (rc != 0) return rc;
    if (!zx || !conv_w || !A || !Lp || !dv || !dq || !dk || !dg || !dlambda || !dzx || !dconv_w || !dA || !dLp) return LLATTN_ERR_NULL;
    if ((conv_b && !dconv_b) || (dt_bias && !dbias) || (D && !dy)) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {zx, dv, dq, dk, dlambda, dzx, dconv_w, dconv_b}) || (D && llattn::misaligned(16, {dy}))) return LLATTN_ERR_ALIGNMENT;
    using bf = __nv_bfloat16;
    llattn::MixerArgs a = {};
    a.zx = (const bf*)zx; a.conv_w = conv_w; a.conv_w_f32 = conv_w_f32; a.conv_b = conv_b; a.conv_b_f32 = conv_b_f32;
    a.dt_bias = dt_bias; a.bias_f32 = bias_f32; a.A = A; a.Lp = Lp; a.lp_f32 = lp_f32; a.D = D; a.d_f32 = d_f32;
    a.dv = (const bf*)dv; a.dy = (const bf*)dy; a.dq = (const bf*)dq; a.dk = (const bf*)dk; a.dg = dg; a.dlam = dlambda;
    a.dzx = (bf*)dzx; a.dconv_w = dconv_w; a.dconv_b = dconv_b; a.dA = dA; a.dbias = dbias; a.dLp = dLp;
    a.B = B; a.T = T; a.H = H; a.L = L; a.dim = H * llattn::MX_P; a.gn = G * N; a.W = 2 * a.dim + 2 * a.gn + H + H * L; a.mode = lambda_mode;
    const int ch = a.dim + 2 * a.gn;
    a.conv_blocks = (ch / 4 + 127) / 128;
    // short runs end in step with the lambda part: walks of up to 128 tokens for 20 warps an SM took (us, before / now) 149 / 131 at B = 1, T = 8192, 48 heads, 90 / 82 at B = 2,
    // T = 4096, 24 heads, 261 / 235 at B = 2, T = 8192, 48 heads, 48 / 44 at T = 2048 (with the lambda part's runs halved as well)
    a.run = mixer_run(B, T, ch / 128 + 1, 16, 32, 148 * 10);
    mixer_lambda_blocks(a, true);
    const unsigned grid = (unsigned)(a.conv_blocks * B * ((T + a.run - 1) / a.run) + a.lam_blocks * B * a.lam_runs);
    llattn::launch_chained(llattn::mixer_prep_bwd_kernel, grid, 128, 0, (cudaStream_t)stream, a);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

// eight columns a thread
static int norm_threads(int dim) { return (dim / 8 + 31) / 32 * 32; }

static int norm_check(long rows, int H) {
    return rows <= 0 || rows > 0x7fffffffl || H <= 0 || H * llattn::MX_P > 8192 ? LLATTN_ERR_UNSUPPORTED_SHAPE : 0;
}

int llattn_mixer_norm_fwd(const void* o, const void* x, const void* D, int d_f32, const void* zx, int zx_width, const void* w, int w_f32,
                          void* out, float* rstd, long rows, int H, float eps, void* stream) {
    const int rc = norm_check(rows, H);
    if (rc != 0) return rc;
    if (!o || !zx || !w || !out || !rstd || (D && !x)) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {o, zx, out}) || (D && llattn::misaligned(16, {x}))) return LLATTN_ERR_ALIGNMENT;
    using bf = __nv_bfloat16;
    llattn::NormArgs a = {};
    a.o = (const bf*)o; a.x = (const bf*)x; a.zx = (const bf*)zx; a.D = D; a.d_f32 = d_f32; a.w = w; a.w_f32 = w_f32;
    a.out = (bf*)out; a.rstd = rstd; a.rows = (int)rows; a.dim = H * llattn::MX_P; a.W = zx_width; a.eps = eps;
    cudaStream_t st = (cudaStream_t)stream;
    if (a.dim <= 4096) llattn::launch_chained(llattn::mixer_norm_kernel<1>, (unsigned)rows, norm_threads(a.dim), 0, st, a);
    else llattn::launch_chained(llattn::mixer_norm_kernel<2>, (unsigned)rows, 512, 0, st, a);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int llattn_mixer_norm_bwd(const void* o, const void* x, const void* D, int d_f32, const void* zx, int zx_width, const void* w, int w_f32,
                          const void* dn, const float* rstd, void* dy, void* dzx, float* dw, float* dD, long rows, int H, void* stream) {
    const int rc = norm_check(rows, H);
    if (rc != 0) return rc;
    if (!o || !zx || !w || !dn || !rstd || !dy || !dzx || !dw || (D && (!x || !dD))) return LLATTN_ERR_NULL;
    if (llattn::misaligned(16, {o, zx, dn, dy, dzx, dw}) || (D && llattn::misaligned(16, {x}))) return LLATTN_ERR_ALIGNMENT;
    using bf = __nv_bfloat16;
    llattn::NormArgs a = {};
    a.o = (const bf*)o; a.x = (const bf*)x; a.zx = (const bf*)zx; a.D = D; a.d_f32 = d_f32; a.w = w; a.w_f32 = w_f32;
    a.dn = (const bf*)dn; a.rstd = const_cast<float*>(rstd); a.dy = (bf*)dy; a.dzx = (bf*)dzx; a.dw = dw; a.dD = dD;
    a.rows = (int)rows; a.dim = H * llattn::MX_P; a.W = zx_width;
    cudaStream_t st = (cudaStream_t)stream;
    // as many CTAs as are resident (85 registers a thread; 128 for heads beyond 4096 columns)
    auto launch = [&](auto kern, int threads, int per_sm) {
        const long most = 148l * per_sm;
        llattn::launch_chained(kern, (unsigned)(rows < most ? rows : most), threads, 0, st, a);
    };
    if (a.dim <= 1024) launch(llattn::mixer_norm_bwd_kernel<1, 128>, 128, 6);
    else if (a.dim <= 2048) launch(llattn::mixer_norm_bwd_kernel<1, 256>, 256, 3);
    else if (a.dim <= 3072) launch(llattn::mixer_norm_bwd_kernel<1, 384>, 384, 2);
    else if (a.dim <= 4096) launch(llattn::mixer_norm_bwd_kernel<1, 512>, 512, 1);
    else launch(llattn::mixer_norm_bwd_kernel<2, 512>, 512, 1);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

}  // extern "C"
