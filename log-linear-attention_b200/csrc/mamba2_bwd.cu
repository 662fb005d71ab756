// Log-linear Mamba-2 chunkwise backward for sm_100a.
//
// Reference being replaced: hattention/chunkwise.py:1286-1597 (driver) with kernels
// chunk_bwd_kernel_dh (:299-470), chunk_bwd_kernel_dqkwg (:663-958), chunk_bwd_kernel_dv
// (:973-1115).  Same segment / Fenwick organisation as the forward (see mamba2_fwd.cu):
//
//   m2_bwd_fwdorder_kernel : per (batch, head, segment), chunks in order.  Recomputes the low
//       level states; produces dq (intra + low levels), the intra part of dk, dlambda for the
//       intra and low levels.
//   m2_bwd_revorder_kernel : per (batch, head, segment), chunks in reverse.  Keeps the adjoint
//       low level states (readers insert (q*scale)^T do, contributors read the sum of the levels
//       whose bit is clear) plus the adjoint of the segment summary; produces dv and the level
//       part of dk.
//   m2_hi_bwd_q_kernel / m2_seg_dstate_kernel / m2_seg_dscan_kernel : the high levels at
//       segment granularity (dq, dlambda of readers; adjoint of the segment summaries).
//   m2_dg_kernel : dg = reverse in-chunk cumsum of (q_t.dq_t - k_t.dk_t) plus, per chunk, the
//       gradient carried across the chunk's end, assembled from per-chunk / per-level scalar
//       totals written by the kernels above (the reference's dG bookkeeping,
//       chunkwise.py:793-874, 938, 1596, without materialising h and dh).
// dq / dk are accumulated over the heads of a group in fp32 with red.global.add and converted to
// bf16 at the end (the reference writes per-head bf16 tensors and sums them on the host,
// chunkwise.py:1583-1591).
#include "llattn_common.cuh"
#include "llattn_mamba2.h"
#include "side_stream.h"

namespace llattn {

// store a 16 x (8*NT) per-warp fp32 fragment block into a fp32 group accumulator with red.add
template <int NT>
__device__ __forceinline__ void red_tile(float* base, long row_stride, int row0, int col0, const float (&acc)[1][NT][4], int lane) {
    const int lr = lane >> 2, lc2 = (lane & 3) * 2;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            float* dst = base + (long)(row0 + lr + hh * 8) * row_stride + col0 + nt * 8 + lc2;
            red_add_f32x2(dst, acc[0][nt][hh * 2], acc[0][nt][hh * 2 + 1]);
        }
}

// per-row dot product of a fragment block with a bf16 smem tile; result valid in every lane of a quad
template <int NT>
__device__ __forceinline__ void rowdot_tile(float (&out)[2], const float (&acc)[1][NT][4], const bf16* s, int ld, int row0, int col0, int lane) {
    const int lr = lane >> 2, lc2 = (lane & 3) * 2;
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        float sum = 0.f;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(s + (row0 + lr + hh * 8) * ld + col0 + nt * 8 + lc2);
            sum += acc[0][nt][hh * 2] * __bfloat162float(x.x) + acc[0][nt][hh * 2 + 1] * __bfloat162float(x.y);
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        out[hh] = sum;
    }
}

// ------------------------------------------------------------------------------------------
// forward-order pass
// ------------------------------------------------------------------------------------------
template <int KD, int VD, int MLOW>
struct Bwd1Smem {
    static constexpr int LDK = KD + PAD, LDV = VD + PAD, LDP = CH + PAD;
    static constexpr size_t q_off = 0;
    static constexpr size_t k_off = q_off + 2ull * CH * LDK * 2;
    static constexpr size_t v_off = k_off + 2ull * CH * LDK * 2;
    static constexpr size_t do_off = v_off + 2ull * CH * LDV * 2;
    static constexpr size_t ds_off = do_off + 2ull * CH * LDV * 2;
    static constexpr size_t vs_off = ds_off + 1ull * CH * LDP * 2;
    static constexpr size_t h_off = vs_off + 1ull * CH * LDV * 2;
    static constexpr size_t lam_off = h_off + (size_t)MLOW * KD * LDV * 2;    // float [2][64*MAX_L]
    static constexpr size_t g_off = lam_off + 2ull * CH * MAX_L * 4;
    static constexpr size_t gc_off = g_off + 2ull * CH * 4;
    static constexpr size_t dl_off = gc_off + CH * 4;                          // float [2][64][16]
    static constexpr size_t total = dl_off + 2ull * CH * 16 * 4;
};

template <int KD, int VD, int MLOW>
__global__ void __launch_bounds__(256, 1) m2_bwd_fwdorder_kernel(const Mamba2Params p) {
    chain_wait();
    using SM = Bwd1Smem<KD, VD, MLOW>;
    constexpr int LDK = SM::LDK, LDV = SM::LDV, LDP = SM::LDP;
    constexpr int SEG = 1 << MLOW, MT = KD / 64, NPS = VD / 32, NPK = KD / 32;
    static_assert(INTRA_LEVELS + MLOW <= 16, "dl staging too small");
    extern __shared__ __align__(16) unsigned char smem[];
    bf16* sQ = reinterpret_cast<bf16*>(smem + SM::q_off);
    bf16* sK = reinterpret_cast<bf16*>(smem + SM::k_off);
    bf16* sV = reinterpret_cast<bf16*>(smem + SM::v_off);
    bf16* sDO = reinterpret_cast<bf16*>(smem + SM::do_off);
    bf16* sDS = reinterpret_cast<bf16*>(smem + SM::ds_off);
    bf16* sVs = reinterpret_cast<bf16*>(smem + SM::vs_off);
    bf16* sH = reinterpret_cast<bf16*>(smem + SM::h_off);
    float* sLam = reinterpret_cast<float*>(smem + SM::lam_off);
    float* sG = reinterpret_cast<float*>(smem + SM::g_off);
    float* sGc = reinterpret_cast<float*>(smem + SM::gc_off);
    float* sDL = reinterpret_cast<float*>(smem + SM::dl_off);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.x % p.H;
    const int r = (blockIdx.x / p.H) % p.NS;
    const int b = blockIdx.x / (p.H * p.NS);
    const int grp = h / (p.H / p.G);
    const int L = p.L;
    const int nc = min(SEG, p.NT - r * SEG);
    const int wr = warp & 3, wc = warp >> 2;
    const int row0 = wr * 16;
    const int lr = lane >> 2, lc2 = (lane & 3) * 2;

    auto issue_tiles = [&](int cl, int st) {
        const long t0 = (long)(r * SEG + cl) * CH;
        load_tile_async<CH, KD, 256>(sQ + st * CH * LDK, p.q + (((long)b * p.T + t0) * p.G + grp) * KD, (long)p.G * KD, tid);
        load_tile_async<CH, KD, 256>(sK + st * CH * LDK, p.k + (((long)b * p.T + t0) * p.G + grp) * KD, (long)p.G * KD, tid);
        load_tile_async<CH, VD, 256>(sV + st * CH * LDV, p.v + (((long)b * p.T + t0) * p.H + h) * VD, (long)p.H * VD, tid);
        load_tile_async<CH, VD, 256>(sDO + st * CH * LDV, p.d_o + (((long)b * p.T + t0) * p.H + h) * VD, (long)p.H * VD, tid);
        cp_async_commit();
    };
    float lam_reg[(CH * MAX_L) / 256];
    float g_reg = 0.f;
    auto fetch_small = [&](int cl) {
        const long t0 = (long)(r * SEG + cl) * CH;
#pragma unroll
        for (int i = 0; i < (CH * MAX_L) / 256; ++i) {
            int e = tid + i * 256;
            int row = e / L, col = e % L;
            lam_reg[i] = (row < CH) ? __bfloat162float(p.l[(((long)b * p.T + t0 + row) * p.H + h) * L + col]) : 0.f;
        }
        if (tid < CH) g_reg = p.g[((long)b * p.T + t0 + tid) * p.H + h];
    };
    auto store_small = [&](int st) {
#pragma unroll
        for (int i = 0; i < (CH * MAX_L) / 256; ++i) {
            int e = tid + i * 256;
            if (e < CH * L) sLam[st * CH * MAX_L + e] = lam_reg[i];
        }
        if (tid < CH) sG[st * CH + tid] = g_reg;
    };

    float M[MLOW > 0 ? MLOW : 1][MT][2 * NPS][4];
    float dsum[MLOW > 0 ? MLOW : 1];
#pragma unroll
    for (int i = 0; i < (MLOW > 0 ? MLOW : 1); ++i) dsum[i] = 0.f;

    issue_tiles(0, 0);
    fetch_small(0);
    store_small(0);

    for (int cl = 0; cl < nc; ++cl) {
        const int st = cl & 1;
        const long t0 = (long)(r * SEG + cl) * CH;
        if (cl + 1 < nc) {
            issue_tiles(cl + 1, st ^ 1);
            fetch_small(cl + 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        if (warp == 0) {
            float x0 = sG[st * CH + 2 * lane], x1 = sG[st * CH + 2 * lane + 1];
            warp_cumsum64(x0, x1, lane);
            sGc[2 * lane] = x0;
            sGc[2 * lane + 1] = x1;
        }
        __syncthreads();
        const bf16* cQ = sQ + st * CH * LDK;
        const bf16* cK = sK + st * CH * LDK;
        const bf16* cV = sV + st * CH * LDV;
        const bf16* cDO = sDO + st * CH * LDV;
        const float* cLam = sLam + st * CH * MAX_L;
        const float glast = sGc[CH - 1];

        // ---- S = q k^T, dP = do v^T ; dS = dP * decay * lambda -> sDS ; dlambda (intra) bins
        {
            float accS[1][4][4], accP[1][4][4];
            zero_acc(accS);
            zero_acc(accP);
            warp_gemm<1, 2, false, false>(accS, cQ, LDK, row0, cK, LDK, wc * 32, KD, lane);
            warp_gemm<1, 2, false, false>(accP, cDO, LDV, row0, cV, LDV, wc * 32, VD, lane);
            float bins[2][INTRA_LEVELS];
#pragma unroll
            for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                for (int lv = 0; lv < INTRA_LEVELS; ++lv) bins[hh][lv] = 0.f;
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int i = row0 + lr + hh * 8;
                    const int j = wc * 32 + nt * 8 + lc2;
                    const float gi = sGc[i];
                    float dsv[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int jj = j + e;
                        float val = 0.f;
                        if (jj <= i) {
                            const int lev = level_of(i, jj);
                            const float ed = accP[0][nt][hh * 2 + e] * fexp(gi - sGc[jj]);
                            const float es = ed * accS[0][nt][hh * 2 + e];
#pragma unroll
                            for (int lv = 0; lv < INTRA_LEVELS; ++lv) bins[hh][lv] += (lev == lv) ? es : 0.f;
                            val = ed * cLam[i * L + lev];
                        }
                        dsv[e] = val;
                    }
                    *reinterpret_cast<uint32_t*>(sDS + i * LDP + j) = pack_bf16(dsv[0], dsv[1]);
                }
#pragma unroll
            for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                for (int lv = 0; lv < INTRA_LEVELS; ++lv) {
                    float x = bins[hh][lv];
                    x += __shfl_xor_sync(0xffffffffu, x, 1);
                    x += __shfl_xor_sync(0xffffffffu, x, 2);
                    if ((lane & 3) == 0) sDL[(wc * CH + row0 + lr + hh * 8) * 16 + lv] = x;
                }
        }
        for (int e = tid; e < CH * VD / 2; e += 256) {
            const int j = e / (VD / 2), c = (e % (VD / 2)) * 2;
            const float sc = fexp(glast - sGc[j]);
            __nv_bfloat162 vv = *reinterpret_cast<const __nv_bfloat162*>(cV + j * LDV + c);
            *reinterpret_cast<uint32_t*>(sVs + j * LDV + c) =
                pack_bf16(__bfloat162float(vv.x) * sc, __bfloat162float(vv.y) * sc);
        }
        __syncthreads();

        float wrow[2] = {0.f, 0.f};    // q.dq - k.dk (intra) for this warp's rows / column half
        // ---- dq = dS k + sum over set low bits lambda*scale * (do . H^T) ; dlambda of those levels
        {
            float acc[1][2 * NPK][4];
            zero_acc(acc);
            const int colk = wc * (KD / 2);
            warp_gemm<1, NPK, false, true>(acc, sDS, LDP, row0, cK, LDK, colk, CH, lane);
#pragma unroll
            for (int lv = 0; lv < MLOW; ++lv) {
                if ((cl >> lv) & 1) {
                    float tmp[1][2 * NPK][4];
                    zero_acc(tmp);
                    warp_gemm<1, NPK, false, false>(tmp, cDO, LDV, row0, sH + lv * KD * LDV, LDV, colk, VD, lane);
                    float rd[2];
                    rowdot_tile<2 * NPK>(rd, tmp, cQ, LDK, row0, colk, lane);
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        const int i = row0 + lr + hh * 8;
                        const float sc = fexp(sGc[i] + dsum[lv]);
                        const float rs = cLam[i * L + INTRA_LEVELS + lv] * sc;
                        if ((lane & 3) == 0) sDL[(wc * CH + i) * 16 + INTRA_LEVELS + lv] = sc * rd[hh];
#pragma unroll
                        for (int nt = 0; nt < 2 * NPK; ++nt) {
                            acc[0][nt][hh * 2] += rs * tmp[0][nt][hh * 2];
                            acc[0][nt][hh * 2 + 1] += rs * tmp[0][nt][hh * 2 + 1];
                        }
                    }
                } else {
                    if ((lane & 3) == 0) {
                        sDL[(wc * CH + row0 + lr) * 16 + INTRA_LEVELS + lv] = 0.f;
                        sDL[(wc * CH + row0 + lr + 8) * 16 + INTRA_LEVELS + lv] = 0.f;
                    }
                }
            }
            float rd[2];
            rowdot_tile<2 * NPK>(rd, acc, cQ, LDK, row0, colk, lane);
            wrow[0] += rd[0];
            wrow[1] += rd[1];
            red_tile<2 * NPK>(p.dq_acc + (((long)b * p.T + t0) * p.G + grp) * KD, (long)p.G * KD, row0, colk, acc, lane);
        }
        // ---- dk (intra) = dS^T q
        {
            float acc[1][2 * NPK][4];
            zero_acc(acc);
            const int colk = wc * (KD / 2);
            warp_gemm<1, NPK, true, true>(acc, sDS, LDP, row0, cQ, LDK, colk, CH, lane);
            float rd[2];
            rowdot_tile<2 * NPK>(rd, acc, cK, LDK, row0, colk, lane);
            wrow[0] -= rd[0];
            wrow[1] -= rd[1];
            red_tile<2 * NPK>(p.dk_acc + (((long)b * p.T + t0) * p.G + grp) * KD, (long)p.G * KD, row0, colk, acc, lane);
        }
        if ((lane & 3) == 0) {
            float* wp = p.wq + ((long)b * p.T + t0) * p.H + h;
            red_add_f32(wp + (long)(row0 + lr) * p.H, wrow[0]);
            red_add_f32(wp + (long)(row0 + lr + 8) * p.H, wrow[1]);
        }

        // ---- recompute KV_c and carry the low level states (same as the forward)
        if (MLOW > 0 && cl + 1 < nc) {
            const int j = __ffs(~cl) - 1;
            if (j < MLOW) {
                float kv[MT][2 * NPS][4];
                zero_acc(kv);
                warp_gemm<MT, NPS, true, true>(kv, cK, LDK, wr * 16 * MT, sVs, LDV, wc * (VD / 2), CH, lane);
#pragma unroll
                for (int lv = 0; lv < MLOW; ++lv) {
                    if (lv < j) {
                        const float dec = fexp(dsum[lv] + glast);
#pragma unroll
                        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                            for (int nt = 0; nt < 2 * NPS; ++nt)
#pragma unroll
                                for (int e = 0; e < 4; ++e) kv[mt][nt][e] += dec * M[lv][mt][nt][e];
                    }
                }
#pragma unroll
                for (int lv = 0; lv < MLOW; ++lv) {
                    if (lv == j) {
                        bf16* dst = sH + lv * KD * LDV;
#pragma unroll
                        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                            for (int nt = 0; nt < 2 * NPS; ++nt) {
#pragma unroll
                                for (int e = 0; e < 4; ++e) M[lv][mt][nt][e] = kv[mt][nt][e];
#pragma unroll
                                for (int hh = 0; hh < 2; ++hh) {
                                    const int rr = wr * 16 * MT + mt * 16 + lr + hh * 8;
                                    const int cc = wc * (VD / 2) + nt * 8 + lc2;
                                    *reinterpret_cast<uint32_t*>(dst + rr * LDV + cc) =
                                        pack_bf16(kv[mt][nt][hh * 2], kv[mt][nt][hh * 2 + 1]);
                                }
                            }
                        dsum[lv] = 0.f;
                    } else {
                        dsum[lv] += glast;
                    }
                }
            } else {
#pragma unroll
                for (int lv = 0; lv < MLOW; ++lv) dsum[lv] += glast;
            }
        }
        if (cl + 1 < nc) store_small(st ^ 1);
        __syncthreads();
        // ---- dlambda for the intra and low levels of this chunk (single writer per entry)
        for (int e = tid; e < CH * (INTRA_LEVELS + MLOW); e += 256) {
            const int i = e / (INTRA_LEVELS + MLOW), lv = e % (INTRA_LEVELS + MLOW);
            if (lv < L) p.dl[(((long)b * p.T + t0 + i) * p.H + h) * L + lv] = sDL[i * 16 + lv] + sDL[(CH + i) * 16 + lv];
        }
        // reader totals Z[c][lv] = sum_i lambda_i * dlambda_i for the low levels read by this chunk
        if (warp < MLOW && ((cl >> warp) & 1)) {
            const int col = INTRA_LEVELS + warp;
            float z = 0.f;
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
                const int i = lane + rr * 32;
                z += cLam[i * L + col] * (sDL[i * 16 + col] + sDL[(CH + i) * 16 + col]);
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) z += __shfl_xor_sync(0xffffffffu, z, d);
            if (lane == 0) p.Zc[(((long)b * p.H + h) * p.NT + r * SEG + cl) * p.LZ + warp] = z;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------
// reverse-order pass
// ------------------------------------------------------------------------------------------
template <int KD, int VD, int MLOW>
struct Bwd2Smem {
    static constexpr int LDK = KD + PAD, LDV = VD + PAD, LDP = CH + PAD;
    static constexpr size_t q_off = 0;
    static constexpr size_t k_off = q_off + 2ull * CH * LDK * 2;
    static constexpr size_t v_off = k_off + 2ull * CH * LDK * 2;
    static constexpr size_t do_off = v_off + 2ull * CH * LDV * 2;
    static constexpr size_t p_off = do_off + 2ull * CH * LDV * 2;
    static constexpr size_t vs_off = p_off + 1ull * CH * LDP * 2;
    static constexpr size_t dkv_off = vs_off + 1ull * CH * LDV * 2;            // bf16 [KD][LDV]
    static constexpr size_t qs_off = dkv_off + 1ull * KD * LDV * 2;            // bf16 [64][LDK]
    static constexpr size_t lam_off = qs_off + 1ull * CH * LDK * 2;            // float [2][64*MAX_L]
    static constexpr size_t g_off = lam_off + 2ull * CH * MAX_L * 4;
    static constexpr size_t gc_off = g_off + 2ull * CH * 4;
    static constexpr size_t y_off = gc_off + CH * 4;                           // float [8][MLOW+1]
    static constexpr size_t total = y_off + 8 * (MLOW + 1) * 4 + 16;
};

template <int KD, int VD, int MLOW>
__global__ void __launch_bounds__(256, 1) m2_bwd_revorder_kernel(const Mamba2Params p) {
    chain_wait();
    using SM = Bwd2Smem<KD, VD, MLOW>;
    constexpr int LDK = SM::LDK, LDV = SM::LDV, LDP = SM::LDP;
    constexpr int SEG = 1 << MLOW, MT = KD / 64, NPS = VD / 32, NPK = KD / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    bf16* sQ = reinterpret_cast<bf16*>(smem + SM::q_off);
    bf16* sK = reinterpret_cast<bf16*>(smem + SM::k_off);
    bf16* sV = reinterpret_cast<bf16*>(smem + SM::v_off);
    bf16* sDO = reinterpret_cast<bf16*>(smem + SM::do_off);
    bf16* sP = reinterpret_cast<bf16*>(smem + SM::p_off);
    bf16* sVs = reinterpret_cast<bf16*>(smem + SM::vs_off);
    bf16* sDKV = reinterpret_cast<bf16*>(smem + SM::dkv_off);
    bf16* sQs = reinterpret_cast<bf16*>(smem + SM::qs_off);
    float* sLam = reinterpret_cast<float*>(smem + SM::lam_off);
    float* sG = reinterpret_cast<float*>(smem + SM::g_off);
    float* sGc = reinterpret_cast<float*>(smem + SM::gc_off);
    float* sY = reinterpret_cast<float*>(smem + SM::y_off);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.x % p.H;
    const int r = (blockIdx.x / p.H) % p.NS;
    const int b = blockIdx.x / (p.H * p.NS);
    const int grp = h / (p.H / p.G);
    const int L = p.L;
    const int nc = min(SEG, p.NT - r * SEG);
    const int wr = warp & 3, wc = warp >> 2;
    const int row0 = wr * 16;
    const int lr = lane >> 2, lc2 = (lane & 3) * 2;

    auto issue_tiles = [&](int cl, int st) {
        const long t0 = (long)(r * SEG + cl) * CH;
        load_tile_async<CH, KD, 256>(sQ + st * CH * LDK, p.q + (((long)b * p.T + t0) * p.G + grp) * KD, (long)p.G * KD, tid);
        load_tile_async<CH, KD, 256>(sK + st * CH * LDK, p.k + (((long)b * p.T + t0) * p.G + grp) * KD, (long)p.G * KD, tid);
        load_tile_async<CH, VD, 256>(sV + st * CH * LDV, p.v + (((long)b * p.T + t0) * p.H + h) * VD, (long)p.H * VD, tid);
        load_tile_async<CH, VD, 256>(sDO + st * CH * LDV, p.d_o + (((long)b * p.T + t0) * p.H + h) * VD, (long)p.H * VD, tid);
        cp_async_commit();
    };
    float lam_reg[(CH * MAX_L) / 256];
    float g_reg = 0.f;
    auto fetch_small = [&](int cl) {
        const long t0 = (long)(r * SEG + cl) * CH;
#pragma unroll
        for (int i = 0; i < (CH * MAX_L) / 256; ++i) {
            int e = tid + i * 256;
            int row = e / L, col = e % L;
            lam_reg[i] = (row < CH) ? __bfloat162float(p.l[(((long)b * p.T + t0 + row) * p.H + h) * L + col]) : 0.f;
        }
        if (tid < CH) g_reg = p.g[((long)b * p.T + t0 + tid) * p.H + h];
    };
    auto store_small = [&](int st) {
#pragma unroll
        for (int i = 0; i < (CH * MAX_L) / 256; ++i) {
            int e = tid + i * 256;
            if (e < CH * L) sLam[st * CH * MAX_L + e] = lam_reg[i];
        }
        if (tid < CH) sG[st * CH + tid] = g_reg;
    };

    // adjoint low level states and the adjoint of this segment's summary (index MLOW)
    float RM[MLOW + 1][MT][2 * NPS][4];
#pragma unroll
    for (int lv = 0; lv <= MLOW; ++lv) zero_acc(RM[lv]);
    if (p.NS > 1 && r < p.NS - 1) {
        const float* dH = p.seg_dHf + (((long)b * p.H + h) * p.NS + r) * KD * VD;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < 2 * NPS; ++nt)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int rr = wr * 16 * MT + mt * 16 + lr + hh * 8;
                    const int cc = wc * (VD / 2) + nt * 8 + lc2;
                    float2 x = *reinterpret_cast<const float2*>(dH + rr * VD + cc);
                    RM[MLOW][mt][nt][hh * 2] = x.x;
                    RM[MLOW][mt][nt][hh * 2 + 1] = x.y;
                }
    }

    issue_tiles(nc - 1, 0);
    fetch_small(nc - 1);
    store_small(0);

    for (int it = 0; it < nc; ++it) {
        const int cl = nc - 1 - it;
        const int st = it & 1;
        const long t0 = (long)(r * SEG + cl) * CH;
        if (it + 1 < nc) {
            issue_tiles(cl - 1, st ^ 1);
            fetch_small(cl - 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        if (warp == 0) {
            float x0 = sG[st * CH + 2 * lane], x1 = sG[st * CH + 2 * lane + 1];
            warp_cumsum64(x0, x1, lane);
            sGc[2 * lane] = x0;
            sGc[2 * lane + 1] = x1;
        }
        __syncthreads();
        const bf16* cQ = sQ + st * CH * LDK;
        const bf16* cK = sK + st * CH * LDK;
        const bf16* cV = sV + st * CH * LDV;
        const bf16* cDO = sDO + st * CH * LDV;
        const float* cLam = sLam + st * CH * MAX_L;
        const float glast = sGc[CH - 1];

        // ---- P = (q k^T) * decay * lambda -> sP
        {
            float acc[1][4][4];
            zero_acc(acc);
            warp_gemm<1, 2, false, false>(acc, cQ, LDK, row0, cK, LDK, wc * 32, KD, lane);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int i = row0 + lr + hh * 8;
                    const int j = wc * 32 + nt * 8 + lc2;
                    const float gi = sGc[i];
                    float pv[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int jj = j + e;
                        float val = 0.f;
                        if (jj <= i) val = acc[0][nt][hh * 2 + e] * fexp(gi - sGc[jj]) * cLam[i * L + level_of(i, jj)];
                        pv[e] = val;
                    }
                    *reinterpret_cast<uint32_t*>(sP + i * LDP + j) = pack_bf16(pv[0], pv[1]);
                }
        }
        for (int e = tid; e < CH * VD / 2; e += 256) {
            const int j = e / (VD / 2), c = (e % (VD / 2)) * 2;
            const float sc = fexp(glast - sGc[j]);
            __nv_bfloat162 vv = *reinterpret_cast<const __nv_bfloat162*>(cV + j * LDV + c);
            *reinterpret_cast<uint32_t*>(sVs + j * LDV + c) =
                pack_bf16(__bfloat162float(vv.x) * sc, __bfloat162float(vv.y) * sc);
        }
        // ---- dKV_c = adjoint of the chunk summary: segment adjoint + levels whose bit is clear
        {
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int nt = 0; nt < 2 * NPS; ++nt)
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        float x0 = RM[MLOW][mt][nt][hh * 2], x1 = RM[MLOW][mt][nt][hh * 2 + 1];
#pragma unroll
                        for (int lv = 0; lv < MLOW; ++lv)
                            if (!((cl >> lv) & 1)) {
                                x0 += RM[lv][mt][nt][hh * 2];
                                x1 += RM[lv][mt][nt][hh * 2 + 1];
                            }
                        const int rr = wr * 16 * MT + mt * 16 + lr + hh * 8;
                        const int cc = wc * (VD / 2) + nt * 8 + lc2;
                        *reinterpret_cast<uint32_t*>(sDKV + rr * LDV + cc) = pack_bf16(x0, x1);
                    }
        }
        __syncthreads();

        // ---- Y[c][lv] = <KV_c, adjoint state lv> for the levels this chunk contributes to
        {
            float kv[MT][2 * NPS][4];
            zero_acc(kv);
            warp_gemm<MT, NPS, true, true>(kv, cK, LDK, wr * 16 * MT, sVs, LDV, wc * (VD / 2), CH, lane);
#pragma unroll
            for (int lv = 0; lv <= MLOW; ++lv) {
                float y = 0.f;
                if (lv == MLOW || !((cl >> lv) & 1)) {
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                        for (int nt = 0; nt < 2 * NPS; ++nt)
#pragma unroll
                            for (int e = 0; e < 4; ++e) y += kv[mt][nt][e] * RM[lv][mt][nt][e];
                }
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) y += __shfl_xor_sync(0xffffffffu, y, d);
                if (lane == 0) sY[warp * (MLOW + 1) + lv] = y;
            }
        }

        // ---- dv = P^T do + decay_j * (k . dKV)
        {
            float acc[1][2 * NPS][4], tmp[1][2 * NPS][4];
            zero_acc(acc);
            zero_acc(tmp);
            const int col0 = wc * (VD / 2);
            warp_gemm<1, NPS, true, true>(acc, sP, LDP, row0, cDO, LDV, col0, CH, lane);
            warp_gemm<1, NPS, false, true>(tmp, cK, LDK, row0, sDKV, LDV, col0, KD, lane);
            bf16* gdv = p.dv + (((long)b * p.T + t0) * p.H + h) * VD;
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int j = row0 + lr + hh * 8;
                const float sc = fexp(glast - sGc[j]);
#pragma unroll
                for (int nt = 0; nt < 2 * NPS; ++nt)
                    *reinterpret_cast<uint32_t*>(gdv + (long)j * p.H * VD + col0 + nt * 8 + lc2) =
                        pack_bf16(acc[0][nt][hh * 2] + sc * tmp[0][nt][hh * 2], acc[0][nt][hh * 2 + 1] + sc * tmp[0][nt][hh * 2 + 1]);
            }
        }
        // ---- dk (levels) = Vs . dKV^T
        {
            float acc[1][2 * NPK][4];
            zero_acc(acc);
            const int colk = wc * (KD / 2);
            warp_gemm<1, NPK, false, false>(acc, sVs, LDV, row0, sDKV, LDV, colk, VD, lane);
            float rd[2];
            rowdot_tile<2 * NPK>(rd, acc, cK, LDK, row0, colk, lane);
            if ((lane & 3) == 0) {
                float* wp = p.wq + ((long)b * p.T + t0) * p.H + h;
                red_add_f32(wp + (long)(row0 + lr) * p.H, -rd[0]);
                red_add_f32(wp + (long)(row0 + lr + 8) * p.H, -rd[1]);
            }
            red_tile<2 * NPK>(p.dk_acc + (((long)b * p.T + t0) * p.G + grp) * KD, (long)p.G * KD, row0, colk, acc, lane);
        }
        // ---- move the adjoint states back across chunk cl: decay, reset, reader insertions
        {
            const float dec = fexp(glast);
#pragma unroll
            for (int lv = 0; lv <= MLOW; ++lv) {
                const bool reset = (lv < MLOW) && ((cl & ((2 << lv) - 1)) == 0);
                const float f = reset ? 0.f : dec;
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int nt = 0; nt < 2 * NPS; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e) RM[lv][mt][nt][e] *= f;
            }
        }
#pragma unroll
        for (int lv = 0; lv < MLOW; ++lv) {
            if ((cl >> lv) & 1) {
                __syncthreads();     // previous users of sQs are done
                for (int e = tid; e < CH * KD / 2; e += 256) {
                    const int i = e / (KD / 2), c = (e % (KD / 2)) * 2;
                    const float rs = cLam[i * L + INTRA_LEVELS + lv] * fexp(sGc[i]);
                    __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(cQ + i * LDK + c);
                    *reinterpret_cast<uint32_t*>(sQs + i * LDK + c) = pack_bf16(__bfloat162float(x.x) * rs, __bfloat162float(x.y) * rs);
                }
                __syncthreads();
                warp_gemm<MT, NPS, true, true>(RM[lv], sQs, LDK, wr * 16 * MT, cDO, LDV, wc * (VD / 2), CH, lane);
            }
        }
        if (it + 1 < nc) store_small(st ^ 1);
        __syncthreads();
        if (tid <= MLOW) {
            float y = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) y += sY[w * (MLOW + 1) + tid];
            p.Yc[(((long)b * p.H + h) * p.NT + r * SEG + cl) * (MLOW + 1) + tid] = y;
        }
    }
}

// ------------------------------------------------------------------------------------------
// high levels, reader side: dq and dlambda of chunk c in segment r > 0
//   R = do . H0[r][j]^T ; dlambda[t, 7+MLOW+j] = s_i (R_i . q_i) ; dq_i += lambda s_i R_i,
//   s_i = exp(G_i + D_before_c)
// ------------------------------------------------------------------------------------------
template <int KD, int VD>
struct HiBwdSmem {
    static constexpr int LDK = KD + PAD, LDV = VD + PAD;
    static constexpr size_t q_off = 0;
    static constexpr size_t do_off = q_off + 1ull * CH * LDK * 2;
    static constexpr size_t h_off = do_off + 1ull * CH * LDV * 2;
    static constexpr size_t gc_off = h_off + 2ull * KD * LDV * 2;
    static constexpr size_t red_off = gc_off + CH * 4;
    static constexpr size_t dl_off = red_off + 16 * 4;             // float [2][64]
    static constexpr size_t total = dl_off + 2 * CH * 4;
};

template <int KD, int VD, int MLOW>
__global__ void __launch_bounds__(256, 1) m2_hi_bwd_q_kernel(const Mamba2Params p) {
    chain_wait();
    using SM = HiBwdSmem<KD, VD>;
    constexpr int LDK = SM::LDK, LDV = SM::LDV, SEG = 1 << MLOW, NPK = KD / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    bf16* sQ = reinterpret_cast<bf16*>(smem + SM::q_off);
    bf16* sDO = reinterpret_cast<bf16*>(smem + SM::do_off);
    bf16* sH = reinterpret_cast<bf16*>(smem + SM::h_off);
    float* sGc = reinterpret_cast<float*>(smem + SM::gc_off);
    float* sRed = reinterpret_cast<float*>(smem + SM::red_off);
    float* sDL = reinterpret_cast<float*>(smem + SM::dl_off);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.x % p.H;
    const int c = SEG + (blockIdx.x / p.H) % (p.NT - SEG);
    const int b = blockIdx.x / (p.H * (p.NT - SEG));
    const int r = c / SEG, cl = c % SEG;
    const int grp = h / (p.H / p.G);
    const long t0 = (long)c * CH;
    const int wr = warp & 3, wc = warp >> 2;
    const int row0 = wr * 16, colk = wc * (KD / 2);
    const int lr = lane >> 2;
    const bf16* H0 = p.seg_H0 + (((long)b * p.H + h) * p.NS + r) * p.LH * KD * VD;

    auto issue_state = [&](int j, int slot) {
        load_tile_async<KD, VD, 256>(sH + slot * KD * LDV, H0 + (long)j * KD * VD, VD, tid);
        cp_async_commit();
    };
    load_tile_async<CH, KD, 256>(sQ, p.q + (((long)b * p.T + t0) * p.G + grp) * KD, (long)p.G * KD, tid);
    load_tile_async<CH, VD, 256>(sDO, p.d_o + (((long)b * p.T + t0) * p.H + h) * VD, (long)p.H * VD, tid);
    cp_async_commit();
    int j = __ffs(r) - 1;
    issue_state(j, 0);

    float part = 0.f;
    {
        const float* gp = p.g + ((long)b * p.T + (long)r * SEG * CH) * p.H + h;
        for (int i = tid; i < cl * CH; i += 256) part += gp[(long)i * p.H];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) part += __shfl_xor_sync(0xffffffffu, part, d);
        if (lane == 0) sRed[warp] = part;
    }
    if (warp == 0) {
        const float* gp = p.g + ((long)b * p.T + t0) * p.H + h;
        float x0 = gp[(long)(2 * lane) * p.H], x1 = gp[(long)(2 * lane + 1) * p.H];
        warp_cumsum64(x0, x1, lane);
        sGc[2 * lane] = x0;
        sGc[2 * lane + 1] = x1;
    }
    __syncthreads();
    float dbefore = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) dbefore += sRed[w];

    float acc[1][2 * NPK][4];
    zero_acc(acc);
    int rem = r & (r - 1);
    int slot = 0;
    while (true) {
        const int jn = rem ? (__ffs(rem) - 1) : -1;
        if (jn >= 0) {
            issue_state(jn, slot ^ 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        float tmp[1][2 * NPK][4];
        zero_acc(tmp);
        warp_gemm<1, NPK, false, false>(tmp, sDO, LDV, row0, sH + slot * KD * LDV, LDV, colk, VD, lane);
        float rd[2];
        rowdot_tile<2 * NPK>(rd, tmp, sQ, LDK, row0, colk, lane);
        const int lcol = INTRA_LEVELS + MLOW + j;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int i = row0 + lr + hh * 8;
            const float sc = fexp(sGc[i] + dbefore);
            const float lam = __bfloat162float(p.l[(((long)b * p.T + t0 + i) * p.H + h) * p.L + lcol]);
            if ((lane & 3) == 0) sDL[wc * CH + i] = sc * rd[hh];
            const float rs = lam * sc;
#pragma unroll
            for (int nt = 0; nt < 2 * NPK; ++nt) {
                acc[0][nt][hh * 2] += rs * tmp[0][nt][hh * 2];
                acc[0][nt][hh * 2 + 1] += rs * tmp[0][nt][hh * 2 + 1];
            }
        }
        __syncthreads();
        if (tid < CH) p.dl[(((long)b * p.T + t0 + tid) * p.H + h) * p.L + lcol] = sDL[tid] + sDL[CH + tid];
        if (warp == 2) {
            float z = 0.f;
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
                const int i = lane + rr * 32;
                z += __bfloat162float(p.l[(((long)b * p.T + t0 + i) * p.H + h) * p.L + lcol]) * (sDL[i] + sDL[CH + i]);
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) z += __shfl_xor_sync(0xffffffffu, z, d);
            if (lane == 0) p.Zc[(((long)b * p.H + h) * p.NT + c) * p.LZ + MLOW + j] = z;
        }
        if (jn < 0) break;
        j = jn;
        rem &= rem - 1;
        slot ^= 1;
    }
    float rd[2];
    rowdot_tile<2 * NPK>(rd, acc, sQ, LDK, row0, colk, lane);
    if ((lane & 3) == 0) {
        float* wp = p.wq + ((long)b * p.T + t0) * p.H + h;
        red_add_f32(wp + (long)(row0 + lr) * p.H, rd[0]);
        red_add_f32(wp + (long)(row0 + lr + 8) * p.H, rd[1]);
    }
    red_tile<2 * NPK>(p.dq_acc + (((long)b * p.T + t0) * p.G + grp) * KD, (long)p.G * KD, row0, colk, acc, lane);
}

// ------------------------------------------------------------------------------------------
// high levels, reader summaries: for segment r >= 1 and high level j with bit j of r set
//   dF[r][j] = sum_{chunks c of r} (q_c * lambda[:, 7+MLOW+j] * exp(G + D_before_c))^T do_c
// (the adjoint of H0[r][j]; fp32 K x V)
// ------------------------------------------------------------------------------------------
template <int KD, int VD, int MLOW>
struct SegDSmem {
    static constexpr int LDK = KD + PAD, LDV = VD + PAD, SEG = 1 << MLOW;
    static constexpr size_t q_off = 0;
    static constexpr size_t do_off = q_off + 2ull * CH * LDK * 2;
    static constexpr size_t qs_off = do_off + 2ull * CH * LDV * 2;
    static constexpr size_t g_off = qs_off + 1ull * CH * LDK * 2;      // float [SEG*64]
    static constexpr size_t tot_off = g_off + (size_t)SEG * CH * 4;
    static constexpr size_t total = tot_off + SEG * 4 + 16;
};

template <int KD, int VD, int MLOW>
__global__ void __launch_bounds__(256, 1) m2_seg_dstate_kernel(const Mamba2Params p) {
    chain_wait();
    using SM = SegDSmem<KD, VD, MLOW>;
    constexpr int LDK = SM::LDK, LDV = SM::LDV, SEG = SM::SEG, MT = KD / 64, NPS = VD / 32;
    const int j = blockIdx.y;
    const int h = blockIdx.x % p.H;
    const int r = 1 + (blockIdx.x / p.H) % (p.NS - 1);
    const int b = blockIdx.x / (p.H * (p.NS - 1));
    if (!((r >> j) & 1)) return;
    extern __shared__ __align__(16) unsigned char smem[];
    bf16* sQ = reinterpret_cast<bf16*>(smem + SM::q_off);
    bf16* sDO = reinterpret_cast<bf16*>(smem + SM::do_off);
    bf16* sQs = reinterpret_cast<bf16*>(smem + SM::qs_off);
    float* sGs = reinterpret_cast<float*>(smem + SM::g_off);
    float* sTot = reinterpret_cast<float*>(smem + SM::tot_off);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int grp = h / (p.H / p.G);
    const int nc = min(SEG, p.NT - r * SEG);
    const int wr = warp & 3, wc = warp >> 2;
    const int lr = lane >> 2, lc2 = (lane & 3) * 2;
    const int lcol = INTRA_LEVELS + MLOW + j;

    auto issue_tiles = [&](int cl, int st) {
        const long t0 = (long)(r * SEG + cl) * CH;
        load_tile_async<CH, KD, 256>(sQ + st * CH * LDK, p.q + (((long)b * p.T + t0) * p.G + grp) * KD, (long)p.G * KD, tid);
        load_tile_async<CH, VD, 256>(sDO + st * CH * LDV, p.d_o + (((long)b * p.T + t0) * p.H + h) * VD, (long)p.H * VD, tid);
        cp_async_commit();
    };
    issue_tiles(0, 0);
    for (int c = warp; c < nc; c += 8) {
        const float* gp = p.g + ((long)b * p.T + (long)(r * SEG + c) * CH) * p.H + h;
        float x0 = gp[(long)(2 * lane) * p.H], x1 = gp[(long)(2 * lane + 1) * p.H];
        warp_cumsum64(x0, x1, lane);
        sGs[c * CH + 2 * lane] = x0;
        sGs[c * CH + 2 * lane + 1] = x1;
        if (lane == 31) sTot[c] = x1;
    }
    __syncthreads();
    if (tid == 0) {
        float run = 0.f;
        for (int c = 0; c < nc; ++c) {
            float t = sTot[c];
            sTot[c] = run;
            run += t;
        }
    }
    __syncthreads();

    float acc[MT][2 * NPS][4];
    zero_acc(acc);
    for (int cl = 0; cl < nc; ++cl) {
        const int st = cl & 1;
        const long t0 = (long)(r * SEG + cl) * CH;
        if (cl + 1 < nc) {
            issue_tiles(cl + 1, st ^ 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const bf16* cQ = sQ + st * CH * LDK;
        const float off = sTot[cl];
        for (int e = tid; e < CH * KD / 2; e += 256) {
            const int i = e / (KD / 2), c = (e % (KD / 2)) * 2;
            const float lam = __bfloat162float(p.l[(((long)b * p.T + t0 + i) * p.H + h) * p.L + lcol]);
            const float rs = lam * fexp(off + sGs[cl * CH + i]);
            __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(cQ + i * LDK + c);
            *reinterpret_cast<uint32_t*>(sQs + i * LDK + c) = pack_bf16(__bfloat162float(x.x) * rs, __bfloat162float(x.y) * rs);
        }
        __syncthreads();
        warp_gemm<MT, NPS, true, true>(acc, sQs, LDK, wr * 16 * MT, sDO + st * CH * LDV, LDV, wc * (VD / 2), CH, lane);
        __syncthreads();
    }
    float* dF = p.seg_dF + ((((long)b * p.H + h) * p.NS + r) * p.LH + j) * KD * VD;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < 2 * NPS; ++nt)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int rr = wr * 16 * MT + mt * 16 + lr + hh * 8;
                const int cc = wc * (VD / 2) + nt * 8 + lc2;
                *reinterpret_cast<float2*>(dF + rr * VD + cc) = make_float2(acc[mt][nt][hh * 2], acc[mt][nt][hh * 2 + 1]);
            }
}

// ------------------------------------------------------------------------------------------
// reverse per-level scan over segments (elementwise in K x V): adjoint of m2_seg_scan_kernel.
//   for r = NS-1 .. 0 : dHseg[r] = sum_{j: bit j of r clear} dH_j ; then dH_j is zeroed when
//   r % 2^(j+1) == 0, else decayed by exp(D_r) ; then dF[r][j] is added when bit j of r is set.
// ------------------------------------------------------------------------------------------
// Bound by HBM: it reads the reader summaries of the set bits and F once and writes dH once.  A thread owns two neighbouring elements of the
// K x V states and walks the segments with the loads of two in flight; the loads are predicated, not branched around, and the number of
// levels is a template parameter, so that 128-thread CTAs of a whole 65536-token problem (1024 of them) are resident at once.  (Four
// elements a thread, branches and one instantiation for up to ten levels: 411 us at B = 1, T = 65536, 32 heads.)
__device__ __forceinline__ float2 ldg2_if(const float* ptr, bool p) {
    float2 r;
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %3, 0;\n mov.f32 %0, 0f00000000;\n mov.f32 %1, 0f00000000;\n @p ld.global.nc.v2.f32 {%0, %1}, [%2];\n}\n"
                 : "=&f"(r.x), "=&f"(r.y)
                 : "l"(ptr), "r"((int)p));
    return r;
}

template <int LH, int KV>
__global__ void __launch_bounds__(128) m2_seg_dscan_kernel(const Mamba2Params p) {
    chain_wait();
    const long bh = blockIdx.y;
    const int e2 = (blockIdx.x * 128 + threadIdx.x) * 2;
    if (e2 >= KV) return;                       // whole warps: KV is a multiple of 64
    const float* dF = p.seg_dF + bh * p.NS * LH * KV + e2;
    const float* F = p.seg_F + bh * p.NS * KV + e2;
    const float* D = p.seg_D + bh * p.NS;
    float* dH = p.seg_dHf + bh * p.NS * KV + e2;
    float* Yseg = p.Yseg + bh * p.NS * LH;
    const int lane = threadIdx.x & 31;
    float2 st[LH];
#pragma unroll
    for (int j = 0; j < LH; ++j) st[j] = make_float2(0.f, 0.f);
    struct Loads {
        float2 f, dF[LH];
        float d;
    };
    auto fetch = [&](Loads& L, int r) {
        const bool in = r >= 0 && r < p.NS - 1;
        L.f = ldg2_if(F + (long)r * KV, in);
        L.d = in ? __ldg(D + r) : 0.f;
#pragma unroll
        for (int j = 0; j < LH; ++j) L.dF[j] = ldg2_if(dF + ((long)r * LH + j) * KV, r >= 0 && ((r >> j) & 1));
    };
    auto process = [&](const Loads& L, int r) {
        float2 out = make_float2(0.f, 0.f);
        const float d = (r < p.NS - 1) ? __expf(L.d) : 0.f;
        float y[LH];
#pragma unroll
        for (int j = 0; j < LH; ++j) {
            const bool bit = (r >> j) & 1;
            // <F_r, adjoint of level j after segment r>; zero where the level has no contributor here
            y[j] = bit ? 0.f : L.f.x * st[j].x + L.f.y * st[j].y;
            if (!bit) {
                out.x += st[j].x;
                out.y += st[j].y;
            }
            const float m = (r & ((2 << j) - 1)) == 0 ? 0.f : d;
            st[j].x = st[j].x * m + L.dF[j].x;
            st[j].y = st[j].y * m + L.dF[j].y;
        }
        if (r < p.NS - 1) {
#pragma unroll
            for (int j = 0; j < LH; ++j)
#pragma unroll
                for (int dd = 16; dd > 0; dd >>= 1) y[j] += __shfl_xor_sync(0xffffffffu, y[j], dd);
            // lane j adds the total of level j
            float mine = 0.f;
#pragma unroll
            for (int j = 0; j < LH; ++j) mine = lane == j ? y[j] : mine;
            if (lane < LH && !((r >> lane) & 1)) atomicAdd(Yseg + (long)r * LH + lane, mine);
            *reinterpret_cast<float2*>(dH + (long)r * KV) = out;
        }
    };
    Loads A, B;
    fetch(A, p.NS - 1);
    fetch(B, p.NS - 2);
    for (int r = p.NS - 1; r >= 0; r -= 2) {
        process(A, r);
        fetch(A, r - 2);
        if (r - 1 >= 0) {
            process(B, r - 1);
            fetch(B, r - 3);
        }
    }
}

template <int LH, int KV>
static void launch_dscan(const Mamba2Params& p, cudaStream_t stream) {
    if constexpr (LH > 0) {
        if (p.LH != LH) return launch_dscan<LH - 1, KV>(p, stream);
        llattn::launch_chained(m2_seg_dscan_kernel<LH, KV>, dim3((KV / 2 + 127) / 128, p.B * p.H), 128, 0, stream, p);
        LLATTN_LAUNCHED();
    }
}

// ------------------------------------------------------------------------------------------
// small elementwise kernels
// ------------------------------------------------------------------------------------------
// What the backward kernels expect before they start, in one launch (three clears and a small kernel before): the raw g from its in-chunk
// inclusive cumulative sum (what the forward returns and autograd saves), cleared accumulators and status word, cleared dlambda.
__global__ void __launch_bounds__(256) m2_bwd_init_kernel(const float* __restrict__ gc, float* __restrict__ g, unsigned n, unsigned H,
                                                          float4* __restrict__ acc, long acc4, float4* __restrict__ dl, long dl4,
                                                          float* __restrict__ dl_tail, int ntail) {
    chain_wait();
    const long i0 = (long)blockIdx.x * 256 + threadIdx.x, step = (long)gridDim.x * 256;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    for (long i = i0; i < acc4; i += step) acc[i] = z;
    for (long i = i0; i < dl4; i += step) dl[i] = z;
    if (i0 < ntail) dl_tail[i0] = 0.f;
    for (long i = i0; i < n; i += step) {
        const unsigned t = (unsigned)i / H;
        float x = gc[i];
        if ((t % CH) != 0) x -= gc[i - H];
        g[i] = x;
    }
}

// dg[r] = sum_{t >= r, t in chunk(r)} w[t]  +  X[chunk(r)]
// w[t] = q_t.dq_t - k_t.dk_t is the gradient w.r.t. the in-chunk cumulative sum G_t (the
// reference's dg before its reverse in-chunk cumsum, chunkwise.py:793-874, 1596); X[c] is the
// gradient that reaches the end of chunk c from every (target, source) pair that straddles it
// (the reference's dg_last: sum_j dk_j.k_j + exp(g_last) sum h*dh, chunkwise.py:865-874).  For
// level l and the block pair that contains c, X gets: the running sum of the contributor totals
// Y over the block's contributor chunks up to c (bit l of c clear), or the sum of the reader
// totals Z over the reader chunks after c (bit set).  Sums never extend beyond one block pair, so
// rounding differences between the two sides do not accumulate along the sequence.
//
// The table X is built by one CTA per (batch, head) and level, whose running sums are warp scans; then a thread per (chunk, head) walks
// the chunk's tokens, heads on neighbouring lanes.  (One kernel in which every slice of 64 chunks built the whole table, by chains of up
// to 2^l additions, took 162 us at T = 65536, 32 heads.)

// running sums over 32 chunks or segments, one a lane, inside half-blocks of `half` of them (a power of two)
__device__ __forceinline__ float half_suffix(float v, int half, int lane) {       // exclusive, from the end
    float s = v;
    const int n = half < 32 ? half : 32;
    for (int d = 1; d < n; d <<= 1) {
        const float t = __shfl_down_sync(0xffffffffu, s, d);
        if ((lane & (n - 1)) + d < n) s += t;
    }
    const float e = __shfl_down_sync(0xffffffffu, s, 1);
    return (lane & (n - 1)) == n - 1 ? 0.f : e;
}
__device__ __forceinline__ float half_prefix(float v, int half, int lane) {       // inclusive, from the start
    const int n = half < 32 ? half : 32;
    for (int d = 1; d < n; d <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, v, d);
        if ((lane & (n - 1)) >= d) v += t;
    }
    return v;
}

template <int MLOW>
__global__ void __launch_bounds__(256) m2_dg_table_kernel(const Mamba2Params p, int nlev) {
    chain_wait();
    constexpr int SEG = 1 << MLOW;
    const long bh = blockIdx.x;
    const int lv = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float* Zc = p.Zc + bh * p.NT * p.LZ;
    const float* Yc = p.Yc + bh * p.NT * (MLOW + 1);
    float* X = p.Xt + bh * p.NT;
    if (lv == nlev) {
        // contributor totals of all high levels together: running sum inside each segment
        for (int c0 = warp * 32; c0 < p.NT; c0 += 256) {
            const int c = c0 + lane;
            const float v = c < p.NT ? Yc[(long)c * (MLOW + 1) + MLOW] : 0.f;
            const float x = half_prefix(v, SEG, lane);
            if (c < p.NT) atomicAdd(&X[c], x);
        }
        return;
    }
    const int half = 1 << lv;
    // readers: after c, to the end of its half-block
    if (half <= 32) {
        for (int c0 = warp * 32; c0 < p.NT; c0 += 256) {
            const int c = c0 + lane;
            const bool reader = c < p.NT && ((c >> lv) & 1);
            const float x = half_suffix(reader ? Zc[(long)c * p.LZ + lv] : 0.f, half, lane);
            float add = reader ? x : 0.f;
            if (lv < MLOW) {
                // contributors: up to and with c
                const bool contributes = c < p.NT && !((c >> lv) & 1);
                const float y = half_prefix(contributes ? Yc[(long)c * (MLOW + 1) + lv] : 0.f, half, lane);
                if (contributes) add = y;
            }
            if (c < p.NT) atomicAdd(&X[c], add);
        }
    } else {
        const int nhalf = (p.NT + half - 1) / half;                    // half-blocks; the odd ones read
        for (int hb = 1 + 2 * warp; hb < nhalf; hb += 16) {
            float carry = 0.f;
            for (int c0 = (hb + 1) * half - 32; c0 >= hb * half; c0 -= 32) {
                const int c = c0 + lane;
                const float v = c < p.NT ? Zc[(long)c * p.LZ + lv] : 0.f;
                const float x = half_suffix(v, 32, lane);
                if (c < p.NT) atomicAdd(&X[c], carry + x);
                carry += __shfl_sync(0xffffffffu, x + v, 0);
            }
        }
    }
    if (lv >= MLOW) {
        // contributors of a high level, per segment: the segments before this one in its half-block
        const int j = lv - MLOW, hs = 1 << j;
        const float* Ys = p.Yseg + bh * p.NS * p.LH;
        for (int hb = 2 * warp; hb * hs < p.NS; hb += 16) {
            float carry = 0.f;
            for (int r0 = hb * hs; r0 < (hb + 1) * hs; r0 += 32) {
                const int r = r0 + lane;
                const bool in = lane < hs && r < p.NS - 1;
                const float v = in ? Ys[(long)r * p.LH + j] : 0.f;
                const float incl = half_prefix(v, 32, lane);
                const float before = __shfl_up_sync(0xffffffffu, incl, 1);
                const float excl = carry + (lane == 0 ? 0.f : before);
                carry += __shfl_sync(0xffffffffu, incl, 31);
                if (lane < hs && r < p.NS)
                    for (int c = r * SEG; c < (r + 1) * SEG && c < p.NT; ++c) atomicAdd(&X[c], excl);
            }
        }
    }
}

__global__ void __launch_bounds__(128) m2_dg_kernel(const Mamba2Params p, float* __restrict__ dg) {
    chain_wait();
    const long i = (long)blockIdx.x * 128 + threadIdx.x;               // (batch, chunk, head)
    if (i >= (long)p.B * p.NT * p.H) return;
    const int h = (int)(i % p.H);
    const long bc = i / p.H;
    const int c = (int)(bc % p.NT), b = (int)(bc / p.NT);
    const long base = bc * CH * p.H + h;
    float run = p.Xt[((long)b * p.H + h) * p.NT + c];
    for (int t = CH; t > 0; t -= 16) {
        float w[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) w[u] = __ldg(p.wq + base + (long)(t - 1 - u) * p.H);
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            run += w[u];
            dg[base + (long)(t - 1 - u) * p.H] = run;
        }
    }
}

__global__ void m2_cast_bf16_kernel(const float* __restrict__ src, bf16* __restrict__ dst, long n) {
    chain_wait();
    const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i + 3 < n) {
        float4 x = *reinterpret_cast<const float4*>(src + i);
        uint2 o;
        o.x = pack_bf16(x.x, x.y);
        o.y = pack_bf16(x.z, x.w);
        *reinterpret_cast<uint2*>(dst + i) = o;
    } else {
        for (long k = i; k < n; ++k) dst[k] = __float2bfloat16(src[k]);
    }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
template <int KD, int VD, int MLOW>
static int launch_fwdorder(const Mamba2Params& p, cudaStream_t stream) {
    cudaError_t e;
    auto kern = m2_bwd_fwdorder_kernel<KD, VD, MLOW>;
    if ((e = allow_smem(kern, Bwd1Smem<KD, VD, MLOW>::total)) != cudaSuccess) return (int)e;
    llattn::launch_chained(kern, p.B * p.H * p.NS, 256, Bwd1Smem<KD, VD, MLOW>::total, stream, p); LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

// dq, d lambda and the reader totals of the high levels
template <int KD, int VD, int MLOW>
static int launch_high_q(const Mamba2Params& p, cudaStream_t stream) {
    cudaError_t e;
    auto kern = m2_hi_bwd_q_kernel<KD, VD, MLOW>;
    if ((e = allow_smem(kern, HiBwdSmem<KD, VD>::total)) != cudaSuccess) return (int)e;
    llattn::launch_chained(kern, p.B * p.H * (p.NT - (1 << MLOW)), 256, HiBwdSmem<KD, VD>::total, stream, p); LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

template <int KD, int VD, int MLOW>
static int launch_high_and_revorder(const Mamba2Params& p, cudaStream_t stream, bool with_q) {
    cudaError_t e;
    if (p.NS > 1) {
        if (with_q) {
            const int rc = launch_high_q<KD, VD, MLOW>(p, stream);
            if (rc != 0) return rc;
        }
        auto kern = m2_seg_dstate_kernel<KD, VD, MLOW>;
        if ((e = allow_smem(kern, SegDSmem<KD, VD, MLOW>::total)) != cudaSuccess) return (int)e;
        dim3 grid(p.B * p.H * (p.NS - 1), p.LH);
        llattn::launch_chained(kern, grid, 256, SegDSmem<KD, VD, MLOW>::total, stream, p); LLATTN_LAUNCHED();
        launch_dscan<M2_MAX_LH, KD * VD>(p, stream);
    }
    auto kern = m2_bwd_revorder_kernel<KD, VD, MLOW>;
    if ((e = allow_smem(kern, Bwd2Smem<KD, VD, MLOW>::total)) != cudaSuccess) return (int)e;
    llattn::launch_chained(kern, p.B * p.H * p.NS, 256, Bwd2Smem<KD, VD, MLOW>::total, stream, p); LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

bool mamba2_bwd_uses_tc(const Mamba2Params& p) {
    // chunk_rounding keeps the digits that a layer's gradients had where only the warp-level kernels took these shapes.  It is not the more accurate
    // choice: the error of sum_t dg dt against fp64, in its absolute terms (mean of 4 heads and seeds, warp-level / tensor cores): T = 192 1.0e-3 / 1.0e-3,
    // T = 1088 1.5e-3 / 5.8e-4, T = 2112 7.3e-4 / 6.0e-4; K = 64, T = 576 2.2e-3 / 1.2e-3, T = 1088 7.9e-4 / 4.5e-4; even counts, which have no such
    // choice: T = 256 2.3e-3 / 1.6e-3, T = 2048 1.1e-3 / 7.8e-4.  Nor the faster one: see mamba2_uses_tc.
    return mamba2_uses_tc(p) && mamba2_bwd_shape_uses_tc(p);
}

template <int KD, int VD, int MLOW>
static int launch_bwd(Mamba2Params p, cudaStream_t stream) {
    int rc;
    const bool use_tc = mamba2_bwd_uses_tc(p);
    if (use_tc ? p.NT > 2 && !p.reuse_states : p.NS > 1 && !p.reuse_states) {
        // forward level states: recomputed unless the caller kept the forward call's workspace
        if (!use_tc) p.lo_H = nullptr;
        if ((rc = mamba2_fwd_states_dispatch(p, stream)) != 0) return rc;
    }
    if (use_tc) {
        if (p.NS > 1) {
            if ((rc = mamba2_readers_tc_launch(p, stream)) != 0) return rc;
            launch_dscan<M2_MAX_LH, KD * VD>(p, stream);
        }
        if (p.NT > 2 && (rc = mamba2_adjoint_tc_launch(p, stream)) != 0) return rc;
        return mamba2_gradients_tc_launch(p, stream);
    }
    // The forward-order pass and the chain high levels -> reverse-order pass only meet in the accumulators they add to.  A pass has one CTA
    // per (batch, head, segment): below three waves of them the two run side by side, beyond that each fills the chip by itself.
    if ((long)p.B * p.H * p.NS < 3 * 148) {
        if (SideStream* side = SideStream::get(stream)) {
            cudaError_t e;
            if ((e = side->fork(stream)) != cudaSuccess) return (int)e;
            rc = launch_fwdorder<KD, VD, MLOW>(p, side->stream());
            // (the kernel of the high levels' dq is not part of that chain: a layer's step at B = 2, T = 1984, 8 heads, K = 128
            //  224 -> 200 us, 24 heads with K = 64 341 -> 322, B = 2, T = 4032, 4 heads 178 -> 168)
            if (rc == 0 && p.NS > 1) rc = launch_high_q<KD, VD, MLOW>(p, side->stream());
            const int rc2 = launch_high_and_revorder<KD, VD, MLOW>(p, stream, false);
            if ((e = side->join(stream)) != cudaSuccess) return (int)e;
            return rc != 0 ? rc : rc2;
        }
    }
    if ((rc = launch_high_and_revorder<KD, VD, MLOW>(p, stream, true)) != 0) return rc;
    return launch_fwdorder<KD, VD, MLOW>(p, stream);
}

int mamba2_bwd_dispatch(Mamba2Params p, cudaStream_t stream) {
    if (p.K == 128 && p.V == 64) return launch_bwd<128, 64, M2_MLOW>(p, stream);
    if (p.K == 64 && p.V == 64) return launch_bwd<64, 64, M2_MLOW>(p, stream);
    return LLATTN_ERR_UNSUPPORTED_SHAPE;
}

int mamba2_bwd_init(const float* gc, float* g, long BT, int H, void* acc, size_t acc_bytes, float* dl, long ndl, cudaStream_t stream) {
    if (BT * H > 0xffffffffl) return LLATTN_ERR_UNSUPPORTED_SHAPE;
    long dl4 = ndl / 4, tail = ndl % 4;
    if ((uintptr_t)dl & 15) {
        const cudaError_t e = cudaMemsetAsync(dl, 0, (size_t)ndl * sizeof(float), stream);
        if (e != cudaSuccess) return (int)e;
        dl4 = tail = 0;
    }
    const long acc4 = (long)(acc_bytes / 16);
    long most = BT * H;
    if (acc4 > most) most = acc4;
    if (dl4 > most) most = dl4;
    const long blocks = (most + 255) / 256;
    llattn::launch_chained(m2_bwd_init_kernel, (unsigned)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, stream, 
        gc, g, (unsigned)(BT * H), (unsigned)H, (float4*)acc, acc4, (float4*)dl, dl4, dl + dl4 * 4, (int)tail);
    LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int mamba2_dg(const Mamba2Params& p, float* dg, cudaStream_t stream) {
    int nlev = 0;
    while ((1 << nlev) < p.NT) ++nlev;          // inter-chunk levels in use
    llattn::launch_chained(m2_dg_table_kernel<M2_MLOW>, dim3(p.B * p.H, nlev + 1), 256, 0, stream, p, nlev); LLATTN_LAUNCHED();
    llattn::launch_chained(m2_dg_kernel, (unsigned)(((long)p.B * p.NT * p.H + 127) / 128), 128, 0, stream, p, dg); LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

void cast_f32_to_bf16(const float* src, void* dst, long n, cudaStream_t stream) {
    const long thr = (n + 3) / 4;
    llattn::launch_chained(m2_cast_bf16_kernel, (unsigned)((thr + 255) / 256), 256, 0, stream, src, reinterpret_cast<bf16*>(dst), n); LLATTN_LAUNCHED();
}

}  // namespace llattn
