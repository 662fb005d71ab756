// The tail of a Gated DeltaNet prompt: the n < 64 tokens behind its last whole chunk, and the level states after them.
//
// Reference being replaced: the steps of hattention_prefill (hattention/kernel.py:541-560) behind the chunkwise part, with step_state /
// step_output (hattention/recurrent.py:134-166): the tokens of the last whole chunk and the ones behind it, one launch a token there.
//
// Everything that a decode step keeps in fp32 is fp32 here too.  For a block of tokens with normalised keys k_i, write strengths beta_i
// and cumulative log decay G_i, that starts from the state S,
//     S_i = exp(G_i) S + sum_{j <= i} exp(G_i - G_j) k_j w_j^T,   (I + A) w = beta v - beta exp(G) k^T S,
//     A_ij = beta_i exp(G_i - G_j) (k_i k_j) for j < i,
// so that with X = (I + A)^-1, M = tril(q k^T exp(G_i - G_j)) X and n the last token of the block
//     S_n  = exp(G_n) S - Kd^T (W S) + R^T v        Kd_j = exp(G_n - G_j) k_j,  W = X (beta exp(G) k),  R = beta X^T Kd,
//     o_i  = lambda (Q~ S)_i + sum_j lambda_ij M_ij beta_j v_j                  Q~ = exp(G) q - M (beta exp(G) k);
// a write's share of an output is linear in it, so each takes the lambda of its own level.  The cascade only ever merges states at the first token of the tail:
// before it stands, for every set bit of T0 = 64 N, the state of a block of whole chunks.  Those of the higher bits come out of the scan and are advanced by the last
// whole chunk; the lowest one is the sum of the scan's lower ones, advanced by that chunk and its writes.
//   gdn_tail_prep_kernel   W, Kd, R of the last whole chunk and of the tail, Q~ and the weights of v, per head
//   gdn_tail_low_kernel    what the tail's tokens give one another, the levels inside their chunk; 64 value columns a CTA
//   gdn_tail_apply_kernel  a state of whole chunks and 64 value columns a CTA
//   gdn_tail_out_kernel    the sum of the outputs' parts
// The first two need nothing of the scan and run beside it, on SMs that it leaves idle.
// q k^T and k k^T are tensor-core products of bf16 operands (exact, fp32 sums); the rest is fp32 arithmetic, and the decays are differences of fp64 sums.
#include "llattn_common.cuh"
#include "llattn_gdn.h"
#include "side_stream.h"

namespace llattn {

constexpr int GT_K = 128, GT_THREADS = 256;
// fp32 scratch of a head: [k][token] or [token][k] tiles of the last whole chunk and of the tail
constexpr int GT_TILE = CH * GT_K;
constexpr int GT_W = 0, GT_KD = 2 * GT_TILE, GT_R = 4 * GT_TILE, GT_Q = 6 * GT_TILE, GT_P = 7 * GT_TILE, GT_E = GT_P + CH * CH, GT_HEAD = GT_E + 64;

// An M x 4 tile of a product, two columns in a register pair; add(): plus the outer product of M rows and four columns
template <int M>
struct Tile4 {
    f32x2 v[M][2];
    __device__ __forceinline__ Tile4() { clear(); }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int u = 0; u < M; ++u) v[u][0] = v[u][1] = 0ull;
    }
    __device__ __forceinline__ void add(const float (&x)[M], float4 y) {
        const f32x2 y0 = pack2(y.x, y.y), y1 = pack2(y.z, y.w);
#pragma unroll
        for (int u = 0; u < M; ++u) {
            const f32x2 d = pack2(x[u], x[u]);
            v[u][0] = fma2(d, y0, v[u][0]);
            v[u][1] = fma2(d, y1, v[u][1]);
        }
    }
    __device__ __forceinline__ float4 row(int u) const {
        const float2 a = unpack2(v[u][0]), b = unpack2(v[u][1]);
        return make_float4(a.x, a.y, b.x, b.y);
    }
};
__device__ __forceinline__ void outer(Tile4<4>& t, float4 x, float4 y) {
    const float f[4] = {x.x, x.y, x.z, x.w};
    t.add(f, y);
}
__device__ __forceinline__ void outer(Tile4<2>& t, float2 x, float4 y) {
    const float f[2] = {x.x, x.y};
    t.add(f, y);
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ld4(const bf16* p) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
}
__device__ __forceinline__ float4 operator*(float s, float4 v) { return make_float4(s * v.x, s * v.y, s * v.z, s * v.w); }
__device__ __forceinline__ float4 operator+(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 operator-(float4 a, float4 b) { return make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w); }

struct GdnTailPrepSmem {
    static constexpr int LDK = GT_K + PAD, LDT = CH + 4;
    static constexpr size_t q_off = 0, k_off = q_off + 2ull * CH * LDK, t_off = k_off + 2ull * CH * LDK, d_off = t_off + 5ull * 4 * CH * LDT,
                            f_off = d_off + 2ull * 8 * CH, total = f_off + 4ull * 4 * CH + 4ull * CH * INTRA_LEVELS;
};

// grid (B * heads, 4): a half of the key columns, of the last whole chunk (y < 2, where there is one) or of the tail.  A chain of latency: X is inverted from
// 16 x 16 blocks up (64 columns of one substitution each: 46 us for the kernel at 16 heads, 17 as it is).
__global__ void __launch_bounds__(GT_THREADS) gdn_tail_prep_kernel(const __grid_constant__ GdnTail a) {
    chain_wait();
    using SM = GdnTailPrepSmem;
    constexpr int LDK = SM::LDK, LDT = SM::LDT;
    extern __shared__ __align__(16) unsigned char smem[];
    bf16* sQ = reinterpret_cast<bf16*>(smem + SM::q_off);
    bf16* sK = reinterpret_cast<bf16*>(smem + SM::k_off);
    float* sA = reinterpret_cast<float*>(smem + SM::t_off);       // A [i][j]
    float* sX = sA + CH * LDT;                                    // X [i][j]
    float* sXt = sX + CH * LDT;                                   // X scaled by beta exp(G) of j, [j][i]
    float* sQK = sXt + CH * LDT;                                  // decayed q k^T, [j][i]
    float* sM = sQK + CH * LDT;                                   // M scaled by beta exp(G) of j, [j][i]
    double* sG = reinterpret_cast<double*>(smem + SM::d_off);     // cumulative log decay, and what is behind a token
    double* sH = sG + CH;
    float* sB = reinterpret_cast<float*>(smem + SM::f_off);       // beta
    float* sBG = sB + CH;                                         // beta exp(G)
    float* sR = sBG + CH;                                         // decays to nothing (log decay -inf) up to a token: counted, not summed
    float* sE = sR + CH;                                          // decay to the last token
    float* sLam = sE + CH;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane >> 2, lc2 = (lane & 3) * 2;
    const bool tail = blockIdx.y >= 2;
    const int half = (blockIdx.y & 1) * (GT_K / 2), blk = blockIdx.y >> 1;
    if (!tail && a.T0 == 0) return;
    const int h = blockIdx.x % a.H, b = blockIdx.x / a.H;
    const int n = tail ? a.n : CH, HR = a.H * a.rep;
    const long tok0 = tail ? (long)a.B * a.T0 + (long)b * a.n : (long)b * a.T0 + a.T0 - CH;
    const long row0 = tok0 * HR + h * a.rep;                      // of the head's first part: q, k, beta, g and lambda are the same for all
    float* out = a.scratch + (long)blockIdx.x * GT_HEAD;
    for (int e = tid; e < CH * (GT_K / 8); e += GT_THREADS) {
        const int i = e / (GT_K / 8), c8 = (e % (GT_K / 8)) * 8;
        if (i < n) {
            cp_async16(sK + i * LDK + c8, a.k + (row0 + (long)i * HR) * GT_K + c8);
            if (tail) cp_async16(sQ + i * LDK + c8, a.q + (row0 + (long)i * HR) * GT_K + c8);
        } else {
            *reinterpret_cast<uint4*>(sK + i * LDK + c8) = make_uint4(0, 0, 0, 0);
            if (tail) *reinterpret_cast<uint4*>(sQ + i * LDK + c8) = make_uint4(0, 0, 0, 0);
        }
    }
    cp_async_commit();
    if (tid < CH) sB[tid] = tid < n ? __bfloat162float(a.beta[row0 + (long)tid * HR]) : 0.f;
    if (tail)
        for (int e = tid; e < n * INTRA_LEVELS; e += GT_THREADS) {
            const int i = e / INTRA_LEVELS, l = e % INTRA_LEVELS;
            sLam[e] = l < a.L ? __bfloat162float(a.lam[(row0 + (long)i * HR) * a.L + l]) : 0.f;
        }
    if (warp == 0) {
        // sums from the front and from the back over the 64 places, two a lane
        double x[2], y[2];
        float c[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = 2 * lane + u;
            float v = i < n ? a.g[row0 + (long)i * HR] : 0.f;
            c[u] = v == -INFINITY ? 1.f : 0.f;
            if (c[u] != 0.f) v = 0.f;
            x[u] = v;
        }
        x[1] += x[0];
        double s = x[1];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const double t = __shfl_up_sync(0xffffffffu, s, d);
            if (lane >= d) s += t;
        }
        const double all = __shfl_sync(0xffffffffu, s, 31), prev = s - x[1];
        x[0] += prev;
        x[1] = s;
        y[0] = all - x[0];
        y[1] = all - x[1];
        warp_cumsum64(c[0], c[1], lane);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            sG[2 * lane + u] = x[u];
            sH[2 * lane + u] = y[u];
            sR[2 * lane + u] = c[u];
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    if (tid < CH) {
        sBG[tid] = sR[tid] == 0.f ? sB[tid] * fexp((float)sG[tid]) : 0.f;
        sE[tid] = sR[tid] == sR[CH - 1] ? fexp((float)sH[tid]) : 0.f;
        if (tid == 0) out[GT_E + blk] = sR[CH - 1] == 0.f ? fexp((float)sG[CH - 1]) : 0.f;
    }
    // ---- A and the decayed q k^T: a tile of 16 tokens x half of the 64 a warp
    {
        const int r0 = (warp & 3) * 16, k0 = (warp >> 2) * 32;
        float kk[1][4][4], qk[1][4][4];
        zero_acc(kk);
        zero_acc(qk);
        if (k0 <= r0 + 15) {
            warp_gemm<1, 2, false, false>(kk, sK, LDK, r0, sK, LDK, k0, GT_K, lane);
            if (tail) warp_gemm<1, 2, false, false>(qk, sQ, LDK, r0, sK, LDK, k0, GT_K, lane);
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = r0 + lr + (e >> 1) * 8, j = k0 + nt * 8 + lc2 + (e & 1);
                const float d = j <= i && sR[i] == sR[j] ? fexp((float)(sG[i] - sG[j])) : 0.f;
                sA[i * LDT + j] = j < i ? sB[i] * d * kk[0][nt][e] : 0.f;
                if (tail) sQK[j * LDT + i] = d * qk[0][nt][e];
            }
    }
    __syncthreads();
    // ---- X = (I + A)^-1: the 16 x 16 blocks of the diagonal by substitution, a column a thread; then [X 0; Y Z] with Y = -Z (A X) at 32 and at 64
    for (int e = tid; e < CH * (CH / 4); e += GT_THREADS) *reinterpret_cast<float4*>(sX + e / (CH / 4) * LDT + e % (CH / 4) * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    if (tid < CH) {
        const int d = tid & ~15, c = tid & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int j = 0; j < i; ++j) (j & 1 ? s1 : s0) += sA[(d + i) * LDT + d + j] * x[j];
            x[i] = i < c ? 0.f : (i == c ? 1.f : 0.f) - (s0 + s1);
            sX[(d + i) * LDT + tid] = x[i];
        }
    }
    __syncthreads();
#pragma unroll
    for (int w = 16; w < CH; w *= 2) {
        // the w x w blocks below the diagonal, one of every 2 w rows, a row and four columns a thread; sM holds A X
        const int each = w * w / 4, c0 = tid / each * 2 * w, i = tid % each / (w / 4), j = tid % (w / 4) * 4;
        const bool act = tid < CH / (2 * w) * each;
        if (act) {
            float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
            for (int l = 0; l < w; ++l) r = r + sA[(c0 + w + i) * LDT + c0 + l] * ld4(sX + (c0 + l) * LDT + c0 + j);
            *reinterpret_cast<float4*>(sM + (c0 + w + i) * LDT + c0 + j) = r;
        }
        __syncthreads();
        if (act) {
            float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
            for (int l = 0; l < w; ++l) r = r - sX[(c0 + w + i) * LDT + c0 + w + l] * ld4(sM + (c0 + w + l) * LDT + c0 + j);
            *reinterpret_cast<float4*>(sX + (c0 + w + i) * LDT + c0 + j) = r;
        }
        __syncthreads();
    }
    for (int e = tid; e < CH * CH; e += GT_THREADS) {
        const int i = e & 63, j = e >> 6;
        sXt[j * LDT + i] = sBG[j] * sX[i * LDT + j];
    }
    __syncthreads();
    // ---- the weights of v, [j][i], and M with its columns scaled
    if (tail) {
        Tile4<4> acc;
        const int i0 = (tid >> 4) * 4, j0 = (tid & 15) * 4;
#pragma unroll 4
        for (int l = j0; l < i0 + 4; ++l) outer(acc, ld4(sQK + l * LDT + i0), ld4(sX + l * LDT + j0));
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float4 r = acc.row(u);
            const float x[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const int i = i0 + u, j = j0 + w;
                const bool in = j <= i && i < n;
                if (half == 0) out[GT_P + j * CH + i] = in ? sLam[i * INTRA_LEVELS + level_of(i, j)] * x[w] * sB[j] : 0.f;
                sM[j * LDT + i] = in ? x[w] * sBG[j] : 0.f;
            }
        }
    }
    float* W = out + GT_W + blk * GT_TILE;
    float* Kd = out + GT_KD + blk * GT_TILE;
    float* R = out + GT_R + blk * GT_TILE;
    {
        // W^T [k][i] = sum_j k_j (scaled X)_ij
        const int k0 = half + (tid >> 4) * 4, i0 = (tid & 15) * 4;
        Tile4<4> acc;
#pragma unroll 4
        for (int j = 0; j < i0 + 4; ++j) outer(acc, ld4(sK + j * LDK + k0), ld4(sXt + j * LDT + i0));
#pragma unroll
        for (int u = 0; u < 4; ++u) *reinterpret_cast<float4*>(W + (k0 + u) * CH + i0) = acc.row(u);
    }
    {
        // R [j][k] = beta_j sum_{i >= j} X_ij Kd_i, and Kd [i][k]
        const int j0 = (tid >> 4) * 4, k0 = half + (tid & 15) * 4;
        Tile4<4> acc;
#pragma unroll 4
        for (int i = j0; i < n; ++i) outer(acc, ld4(sX + i * LDT + j0), sE[i] * ld4(sK + i * LDK + k0));
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            *reinterpret_cast<float4*>(R + (j0 + u) * GT_K + k0) = sB[j0 + u] * acc.row(u);
            *reinterpret_cast<float4*>(Kd + (j0 + u) * GT_K + k0) = sE[j0 + u] * ld4(sK + (j0 + u) * LDK + k0);
        }
    }
    if (!tail || a.T0 == 0) return;
    __syncthreads();
    {
        // Q~^T [k][i] = exp(G_i) q_i - sum_j k_j (scaled M)_ij
        const int k0 = half + (tid >> 4) * 4, i0 = (tid & 15) * 4;
        Tile4<4> acc;
#pragma unroll 4
        for (int j = 0; j < i0 + 4; ++j) outer(acc, ld4(sK + j * LDK + k0), ld4(sM + j * LDT + i0));
        float d[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) d[w] = sR[i0 + w] == 0.f ? fexp((float)sG[i0 + w]) : 0.f;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            auto q = [&](int w) { return d[w] * __bfloat162float(sQ[(i0 + w) * LDK + k0 + u]); };
            *reinterpret_cast<float4*>(out + GT_Q + (k0 + u) * CH + i0) = make_float4(q(0), q(1), q(2), q(3)) - acc.row(u);
        }
    }
}

// what a CTA of the kernels below works on: CB value columns of a head, by 8 CB threads in 32 groups of rows with four columns a thread
template <int CB>
struct GdnTailPlace {
    static constexpr int LDS = CB + 4, THREADS = 8 * CB;
    int c0, h, b, bh, n, tm, tn;
    long tail0;                // first token of the tail in the split tensors
    const float* head;
    float* S;                  // level l at S + l K V
    __device__ explicit GdnTailPlace(const GdnTail& a) {
        const int ncb = a.V / CB;
        c0 = blockIdx.x % ncb * CB;
        bh = blockIdx.x / ncb;
        h = bh % a.H;
        b = bh / a.H;
        n = a.n;
        tm = threadIdx.x / (CB / 4);
        tn = threadIdx.x % (CB / 4) * 4;
        tail0 = (long)a.B * a.T0 + (long)b * a.n;
        head = a.scratch + (long)bh * GT_HEAD;
        S = a.states + (long)bh * a.L * a.K * a.V + c0;
    }
    __device__ void stage(float* dst, const float* src, int floats) const {
        for (int e = threadIdx.x * 4; e < floats; e += THREADS * 4) cp_async16(dst + e, src + e);
        cp_async_commit();
    }
    // rows of v as fp32, zeros behind them
    __device__ void values(float* dst, const GdnTail& a, long tok0, int rows) const {
        const int i = threadIdx.x / (CB / 8), c = threadIdx.x % (CB / 8) * 8;
        uint4 r = make_uint4(0, 0, 0, 0);
        if (i < rows) r = *reinterpret_cast<const uint4*>(a.v + ((tok0 + i) * a.H + h) * a.V + c0 + c);
        const bf16* x = reinterpret_cast<const bf16*>(&r);
        *reinterpret_cast<float4*>(dst + i * LDS + c) = ld4(x);
        *reinterpret_cast<float4*>(dst + i * LDS + c + 4) = ld4(x + 4);
    }
    // a slot's part of the outputs of tokens 2 tm and 2 tm + 1, [slot][b][token][h][V]
    __device__ void part(const GdnTail& a, int slot, const Tile4<2>& r, float x0, float x1) const {
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (2 * tm + u < n)
                *reinterpret_cast<float4*>(a.part + ((((long)slot * a.B + b) * n + 2 * tm + u) * a.H + h) * a.V + c0 + tn) = (u ? x1 : x0) * r.row(u);
    }
    // rows 4 tm .. of a state
    __device__ void state(const GdnTail& a, int lev, const float4 (&r)[4]) const {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (4 * tm + u < a.K) *reinterpret_cast<float4*>(S + ((long)lev * a.K + 4 * tm + u) * a.V + tn) = r[u];
    }
};

struct GdnTailLowSmem {
    static constexpr size_t r_off = 0, p_off = 4ull * GT_TILE, v_off = p_off + 4ull * CH * CH, total = v_off + 4ull * CH * GdnTailPlace<64>::LDS;
};
// grid (B * heads * V / 64, 2 or 1): y = 0 the tail's tokens among themselves, y = 1 the writes of the last whole chunk, R^T v
__global__ void __launch_bounds__(512) gdn_tail_low_kernel(const __grid_constant__ GdnTail a, int slots) {
    chain_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    using W = GdnTailPlace<64>;
    constexpr int LDS = W::LDS;
    float* sR = reinterpret_cast<float*>(smem + GdnTailLowSmem::r_off);
    float* sP = reinterpret_cast<float*>(smem + GdnTailLowSmem::p_off);
    float* sV = reinterpret_cast<float*>(smem + GdnTailLowSmem::v_off);
    const W w(a);
    const int tm = w.tm, tn = w.tn, n = a.n, m = n - 1, N = a.T0 / CH, tz = N > 0 ? __ffs(N) - 1 : 0;
    if (blockIdx.y == 1) {
        w.stage(sR, w.head + GT_R, GT_TILE);
        w.values(sV, a, (long)w.b * a.T0 + a.T0 - CH, CH);
        cp_async_wait<0>();
        __syncthreads();
        Tile4<4> acc;
#pragma unroll 8
        for (int j = 0; j < CH; ++j) outer(acc, ld4(sR + j * GT_K + 4 * tm), ld4(sV + j * LDS + tn));
#pragma unroll
        for (int u = 0; u < 4; ++u) *reinterpret_cast<float4*>(a.writes + ((long)w.bh * GT_K + 4 * tm + u) * a.V + w.c0 + tn) = acc.row(u);
        return;
    }
    w.stage(sR, w.head + GT_R + GT_TILE, n * GT_K);
    w.stage(sP, w.head + GT_P, n * CH);
    w.values(sV, a, w.tail0, n);
    cp_async_wait<0>();
    __syncthreads();
    if (2 * tm < n) {
        Tile4<2> r;
#pragma unroll 4
        for (int j = 0; j < min(n, 2 * tm + 2); ++j) outer(r, *reinterpret_cast<const float2*>(sP + j * CH + 2 * tm), ld4(sV + j * LDS + tn));
        if (slots > 0) {
            w.part(a, slots, r, 1.f, 1.f);
        } else {
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (2 * tm + u < n) {
                    const float4 x = r.row(u);
                    *reinterpret_cast<uint2*>(a.o + (((long)w.b * n + 2 * tm + u) * a.H + w.h) * a.V + w.c0 + tn) =
                        make_uint2(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w));
                }
        }
    }
    // levels 0 .. 6 from their own writes; of the others, those that hold nothing are cleared (but for the ones that the first slot sums up)
    for (int lev = 0; lev < a.L; ++lev) {
        int s0 = 0, s1 = 0;
        if (lev == 0) {
            s0 = m;
            s1 = n;
        } else if (lev < INTRA_LEVELS && ((m >> (lev - 1)) & 1)) {
            s0 = (m >> lev) << lev;
            s1 = s0 + (1 << (lev - 1));
        } else if (lev >= INTRA_LEVELS && N > 0 && (lev - INTRA_LEVELS <= tz || ((N >> (lev - INTRA_LEVELS)) & 1))) {
            continue;
        }
        Tile4<4> acc;
#pragma unroll 4
        for (int j = s0; j < s1; ++j) outer(acc, ld4(sR + j * GT_K + 4 * tm), ld4(sV + j * LDS + tn));
        const float4 r[4] = {acc.row(0), acc.row(1), acc.row(2), acc.row(3)};
        w.state(a, lev, r);
    }
}

template <int CB>
struct GdnTailApplySmem {
    static constexpr size_t buf_off = 0, s_off = 4ull * 4 * GT_TILE, w_off = s_off + 4ull * GT_K * GdnTailPlace<CB>::LDS,
                            total = w_off + 4ull * CH * GdnTailPlace<CB>::LDS;
};
// grid (B * heads * V / CB, slots): slot z is the state of the z-th set bit of N = T0 / 64, carried over the last whole chunk and the tail
template <int CB>
__global__ void __launch_bounds__(GdnTailPlace<CB>::THREADS) gdn_tail_apply_kernel(const __grid_constant__ GdnTail a) {
    chain_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    using SM = GdnTailApplySmem<CB>;
    constexpr int LDS = GdnTailPlace<CB>::LDS;
    float* buf = reinterpret_cast<float*>(smem + SM::buf_off);
    float* sS = reinterpret_cast<float*>(smem + SM::s_off);
    float* sW = reinterpret_cast<float*>(smem + SM::w_off);
    const GdnTailPlace<CB> w(a);
    const int tm = w.tm, tn = w.tn, n = a.n;
    unsigned left = a.T0 / CH;
    for (int i = blockIdx.y; i > 0; --i) left &= left - 1;
    const int bit = __ffs(left) - 1;
    const bool merged = blockIdx.y == 0;
    auto tile = [&](int i) { return buf + i * GT_TILE; };
    w.stage(tile(0), w.head + GT_W, GT_TILE);
    w.stage(tile(1), w.head + GT_KD, GT_TILE);
    w.stage(tile(2), w.head + GT_W + GT_TILE, GT_TILE);
    w.stage(tile(3), w.head + GT_Q, GT_TILE);
    // what the scan left before the last whole chunk, under the bits of N - 1: the lower ones are this state's for the first slot
    float4 st[4], wr[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        st[u] = wr[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (merged) wr[u] = ld4(a.writes + ((long)w.bh * GT_K + 4 * tm + u) * a.V + w.c0 + tn);
    }
    const int lv0 = merged ? 0 : bit, lv1 = merged ? bit : bit + 1;
#pragma unroll 4
    for (int lv = lv0; lv < lv1; ++lv)
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (4 * tm + u < a.K) st[u] = st[u] + ld4(w.S + ((long)(INTRA_LEVELS + lv) * a.K + 4 * tm + u) * a.V + tn);
    auto put_state = [&]() {
#pragma unroll
        for (int u = 0; u < 4; ++u) *reinterpret_cast<float4*>(sS + (4 * tm + u) * LDS + tn) = st[u];
    };
    auto put_ws = [&](const Tile4<2>& r) {
#pragma unroll
        for (int u = 0; u < 2; ++u) *reinterpret_cast<float4*>(sW + (2 * tm + u) * LDS + tn) = r.row(u);
    };
    put_state();
    float lam[2];
#pragma unroll
    for (int u = 0; u < 2; ++u)
        lam[u] = 2 * tm + u < n ? __bfloat162float(a.lam[((w.tail0 + 2 * tm + u) * a.H + w.h) * a.rep * a.L + INTRA_LEVELS + bit]) : 0.f;
    const float e0 = w.head[GT_E], e1 = w.head[GT_E + 1];
    // ---- the last whole chunk: S = exp(G) S - Kd^T (W S) + R^T v
    cp_async_wait<3>();
    __syncthreads();
    {
        Tile4<2> r;
#pragma unroll 16
        for (int k = 0; k < GT_K; ++k) outer(r, *reinterpret_cast<const float2*>(tile(0) + k * CH + 2 * tm), ld4(sS + k * LDS + tn));
        put_ws(r);
    }
    cp_async_wait<2>();
    __syncthreads();
    w.stage(tile(0), w.head + GT_KD + GT_TILE, n * GT_K);
    {
        Tile4<4> acc;
#pragma unroll 16
        for (int j = 0; j < CH; ++j) outer(acc, ld4(tile(1) + j * GT_K + 4 * tm), ld4(sW + j * LDS + tn));
#pragma unroll
        for (int u = 0; u < 4; ++u) st[u] = (e0 * st[u] - acc.row(u)) + wr[u];
        put_state();
    }
    cp_async_wait<1>();
    __syncthreads();
    // ---- the tail: lambda Q~ S, then the state again
    if (2 * tm < n) {
        Tile4<2> r, q;
#pragma unroll 16
        for (int k = 0; k < GT_K; ++k) {
            const float4 y = ld4(sS + k * LDS + tn);
            outer(r, *reinterpret_cast<const float2*>(tile(2) + k * CH + 2 * tm), y);
            outer(q, *reinterpret_cast<const float2*>(tile(3) + k * CH + 2 * tm), y);
        }
        put_ws(r);
        w.part(a, blockIdx.y, q, lam[0], lam[1]);
    }
    cp_async_wait<0>();
    __syncthreads();
    Tile4<4> acc;
#pragma unroll 4
    for (int j = 0; j < n; ++j) outer(acc, ld4(tile(0) + j * GT_K + 4 * tm), ld4(sW + j * LDS + tn));
#pragma unroll
    for (int u = 0; u < 4; ++u) st[u] = e1 * st[u] - acc.row(u);
    w.state(a, INTRA_LEVELS + bit, st);
    if (merged) {
#pragma unroll
        for (int u = 0; u < 4; ++u) st[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int lv = 0; lv < bit; ++lv) w.state(a, INTRA_LEVELS + lv, st);
    }
}

__global__ void __launch_bounds__(256) gdn_tail_out_kernel(const __grid_constant__ GdnTail a, int slots) {
    chain_wait();
    const long per = (long)a.n * a.H * a.V, all = a.B * per, e = ((long)blockIdx.x * 256 + threadIdx.x) * 4;
    if (e >= all) return;
    float4 r = ld4(a.part + e);
    for (int z = 1; z < slots; ++z) r = r + ld4(a.part + z * all + e);
    const long b = e / per;
    bf16* o = a.o + (b * (a.T0 + a.n) + a.T0) * a.H * a.V + e % per;
    *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16(r.x, r.y), pack_bf16(r.z, r.w));
}

static int tail_slots(int T0) { return __builtin_popcount((unsigned)(T0 / CH)); }

void gdn_tail_scratch(GdnTail& a, float* base) {
    a.scratch = base;
    a.writes = base + (size_t)a.B * a.H * GT_HEAD;
    a.part = a.writes + (size_t)a.B * a.H * GT_K * a.V;
}
size_t gdn_tail_scratch_floats(int B, int T0, int n, int H, int V) {
    const size_t heads = (size_t)B * H * GT_HEAD;
    return T0 == 0 ? heads : heads + (size_t)B * H * GT_K * V + (size_t)(tail_slots(T0) + 1) * B * n * H * V;
}

// the kernels that need nothing of the scan
int gdn_tail_prep_launch(GdnTail& a, cudaStream_t stream) {
    cudaError_t e;
    if ((e = allow_smem(gdn_tail_prep_kernel, GdnTailPrepSmem::total)) != cudaSuccess || (e = allow_smem(gdn_tail_low_kernel, GdnTailLowSmem::total)) != cudaSuccess)
        return (int)e;
    a.side = a.T0 > 0 ? SideStream::get(stream) : nullptr;
    if (a.side && (e = a.side->fork(stream)) != cudaSuccess) return (int)e;
    cudaStream_t on = a.side ? a.side->stream() : stream;
    launch_chained(gdn_tail_prep_kernel, dim3(a.B * a.H, 4), GT_THREADS, GdnTailPrepSmem::total, on, a);
    LLATTN_LAUNCHED();
    launch_chained(gdn_tail_low_kernel, dim3(a.B * a.H * (a.V / 64), a.T0 > 0 ? 2 : 1), GdnTailPlace<64>::THREADS, GdnTailLowSmem::total, on, a, tail_slots(a.T0));
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int gdn_tail_join(const GdnTail& a, cudaStream_t stream) { return a.side ? (int)a.side->join(stream) : 0; }

// the states of whole chunks, behind the scan
template <int CB>
static cudaError_t launch_apply(const GdnTail& a, int slots, cudaStream_t stream) {
    const cudaError_t e = allow_smem(gdn_tail_apply_kernel<CB>, GdnTailApplySmem<CB>::total);
    if (e != cudaSuccess) return e;
    launch_chained(gdn_tail_apply_kernel<CB>, dim3(a.B * a.H * (a.V / CB), slots), GdnTailPlace<CB>::THREADS, GdnTailApplySmem<CB>::total, stream, a);
    LLATTN_LAUNCHED();
    return cudaSuccess;
}
int gdn_tail_apply_launch(const GdnTail& a, cudaStream_t stream) {
    int dev = 0, sms = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess || (e = sm_count(&sms, dev)) != cudaSuccess) return (int)e;
    const int slots = tail_slots(a.T0);
    // one CTA fits on an SM: 32 columns each while they all run at once, which halves the chain of one.  The call with 32 / 64: T = 777 at 8, 16, 24 heads
    // (64, 128, 192 CTAs of 32) 70.4 / 74.2, 85.0 / 91.8, 113.7 / 108.5 us; T = 1000 at 8 and 16 heads (128, 256) 78.5 / 84.5, 110.4 / 106.2
    e = (long)a.B * a.H * (a.V / 32) * slots <= sms ? launch_apply<32>(a, slots, stream) : launch_apply<64>(a, slots, stream);
    if (e != cudaSuccess) return (int)e;
    const long all = (long)a.B * a.n * a.H * a.V;
    launch_chained(gdn_tail_out_kernel, (unsigned)((all / 4 + 255) / 256), 256, 0, stream, a, slots + 1);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

}  // namespace llattn
