// Gradients of log-linear Mamba-2 on the 5th-generation tensor cores (tcgen05.mma, accumulators in tensor memory), K = 64 or 128, V = 64.
//
// Both kernels give a CTA a PAIR of chunks (128 tokens) of one q / k group and walk heads of that group, as the output kernel does: the heads share q, k
// and S = q k^T, and the gradients of q and k, sums over heads, stay in tensor memory until the CTA ends.  What a pair exchanges with the others are
// bf16 K x V tiles in global memory: the level states H_l that it reads, and the gradient A of its own summary, the sum of what its readers send back.
//   m2_dq_tc_kernel    dP = do v^T;  dS = dP decay lambda;  dq += dS k;  per level read: T = q H_l, dq += (do scale_l) H_l^T;  d lambda
//   m2_dkv_tc_kernel   dP again;  P = S decay lambda, dS;  dv = P^T do + scale (k A);  dk += dS^T q + (v scale) A^T
// Warps 0..7 turn S and dP into the operand tiles of a head, warps 8..15 do the per-row work of the levels and the outputs, two warps issue the products,
// one the loads, one the outputs, all ahead of one another as far as their rings allow.  A wait that gives up sets the CTA's abort flag, after which every other wait of
// the CTA ends at once; the warps that meet at barriers then go through the rest of their loops without waiting.
//
// The gradient w.r.t. the cumulative decay needs q_i.dq_i and k_j.dk_j per head, which the sums over heads no longer show: o is linear in lambda, so
// q_i.dq_i = sum_l lambda d lambda; inside a pair q_i.dq_i and k_j.dk_j are the row and column sums of one matrix, bf16(dS_ij) S_ij, so that they cancel
// as the exact sums do; and a state's share of k_j.dk_j is (v_j scale).(k_j A), from the operands of the products.
//
// What bounds them is the latency of instruction streams: the tile warps' phase between two products (about 2 k cycles a head) and the issue of products.
// The kernels before walked the segments of one head in order with one pair in flight per SM (15 k cycles a pair, twice) and added 64 KB of fp32 gradients
// of q or k per pair and head to global memory, three times.
// B = 2, T = 16384, 32 heads: 323 + 232 us, 871 with the readers' and the adjoints' kernels (140 + 176), where the two walks took 895 and the high levels' kernel 316.
#include "rowwise.cuh"
#include "tc_common.cuh"

namespace llattn {

namespace tcg {
constexpr int HC_MAX = 8;
constexpr int LAM_LD = 122;                  // row stride of the staged lambda values (as many as the output kernel takes): odd number of 32-bit words
constexpr int NTHREADS = 640, WORKERS = 512, MMA_WARP = 16, T_WARP = 17, TMA_WARP = 18, OUT_WARP = 19;
constexpr int NST = 3;                       // dq: stages of 16 KB for v and the level states
// launched with 96 registers a thread, 61440 in all: 256 x 112 + 256 x 104 + 128 x 48
__device__ __forceinline__ void regs_tiles() { asm volatile("setmaxnreg.inc.sync.aligned.u32 112;\n"); }
__device__ __forceinline__ void regs_rows() { asm volatile("setmaxnreg.inc.sync.aligned.u32 104;\n"); }
__device__ __forceinline__ void regs_issue() { asm volatile("setmaxnreg.dec.sync.aligned.u32 48;\n"); }
}  // namespace tcg

__device__ __forceinline__ void arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(umma::smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void bar_rows() { asm volatile("bar.sync 2, 256;\n" ::: "memory"); }
// fp32 staging box for a TMA reduce: 128 rows x 32 floats, 128-byte swizzled
__device__ __forceinline__ uint32_t grad_box_offset(int row, int col) {
    return (uint32_t)(row * 128 + (((col >> 2) ^ (row & 7)) << 4) + (col & 3) * 4);
}

// Which work a CTA has: heads [h0, h0 + nh) of group `grp`, tokens [t0, t0 + 128) of sequence b.  Pairs from the last one on: later pairs read more levels.
struct PairWork {
    int b, grp, pair, t0, h0, nh, NP;
    __device__ __forceinline__ PairWork(const Mamba2Params& p) {
        NP = (p.NT + 1) / 2;
        const int per_grp = p.H / p.G, nhc = (per_grp + p.hc - 1) / p.hc;
        int at = blockIdx.x;
        const int hchunk = at % nhc;
        at /= nhc;
        grp = at % p.G;
        at /= p.G;
        pair = NP - 1 - at % NP;
        b = at / NP;
        h0 = grp * per_grp + hchunk * p.hc;
        nh = min(p.hc, per_grp - hchunk * p.hc);
        t0 = pair * tc::PT;
    }
};

// columns 32 bx .. of an accumulator in tensor memory, as fp32 boxes for a TMA reduce-add; NW warps (two or more per lane quarter) share the KD / 32 boxes
template <int KD>
__device__ __forceinline__ void stage_gradient(unsigned char* stage, uint32_t taddr, int warp, int row, int part, int parts) {
    for (int bx = part; bx < KD / 32; bx += parts) {
        float t[32];
        umma::tmem_ld32(umma::tmem_addr(taddr, warp, bx * 32), t);
        unsigned char* box = stage + bx * 16384;
#pragma unroll
        for (int c = 0; c < 8; ++c)
            *reinterpret_cast<float4*>(box + grad_box_offset(row, c * 4)) = make_float4(t[c * 4], t[c * 4 + 1], t[c * 4 + 2], t[c * 4 + 3]);
    }
}

// The same in bf16 (tile layout of the operands), where no other CTA adds to them: the accumulators are neither cleared nor added to nor converted, passes over
// fp32 gradients that are as large as everything else where every head has its own q and k.  Walking one head a CTA shares nothing, and with the
// accumulators such calls took longer than on the kernels that walked segments (B = 16, T = 1024, 24 heads and groups: 921, 988 with accumulators, 779 us
// without; 12 groups of two 775, 683, 576).  The rounding is that of the conversion pass.
template <int KD>
__device__ __forceinline__ void stage_gradient_bf16(unsigned char* stage, uint32_t taddr, int warp, int row, int part, int parts) {
    for (int bx = part; bx < KD / 32; bx += parts) {
        float t[32];
        umma::tmem_ld32(umma::tmem_addr(taddr, warp, bx * 32), t);
#pragma unroll
        for (int c = 0; c < 32; c += 8)
            *reinterpret_cast<uint4*>(stage + umma::tile_offset(row, bx * 32 + c, tc::PT)) =
                make_uint4(pack_bf16(t[c], t[c + 1]), pack_bf16(t[c + 2], t[c + 3]), pack_bf16(t[c + 4], t[c + 5]), pack_bf16(t[c + 6], t[c + 7]));
    }
}
// by one thread: what the two above staged leaves
template <int KD>
__device__ __forceinline__ void store_gradient(const CUtensorMap* map, bool whole, int grp, int t0, int b, unsigned char* stage) {
    if (whole) {
#pragma unroll
        for (int c = 0; c < KD; c += 64) tma::store_seq_box(map, c, grp, t0, b, stage + c * tc::PT * 2);
    } else {
#pragma unroll
        for (int bx = 0; bx < KD / 32; ++bx) tma::reduce_add_seq_box(map, bx * 32, grp, t0, b, stage + bx * 16384);
    }
    tma::commit_group();
    tma::wait_group0();
}

// ------------------------------------------------------------------------------------------
// dq, d lambda, reader totals
// ------------------------------------------------------------------------------------------
namespace tcq {
constexpr int TM_S = 0, TM_DP = 128, TM_DQ = 256, TM_T = 384, TM_DOS = 448;     // DOS: two scaled copies of do, bf16, 32 columns each
// sums of a row: d lambda by level (6 and 7: of one half of the row), the other half's of levels 6 and 7, sum of bf16(dS) S by halves, of lambda d lambda over
// the levels read by sets of warps
constexpr int C_HALF = 14, C_TILE = 22, C_LEV = 24, NSUM = 27;
}  // namespace tcq

template <int KD>
struct DqTcSmem {
    static constexpr uint32_t q_off = 0;                                            // q and k: the fp32 staging of dq at the end
    static constexpr uint32_t k_off = q_off + tc::PT * KD * 2;
    static constexpr uint32_t ds_off = k_off + tc::PT * KD * 2;
    static constexpr uint32_t do_off = ds_off + tc::PT * tc::PT * 2;
    static constexpr uint32_t st_off = do_off + tc::V_BYTES;                        // [NST]
    static constexpr uint32_t g_off = st_off + tcg::NST * tc::V_BYTES;              // float [HC_MAX][2][128]
    static constexpr uint32_t c_off = g_off + tcg::HC_MAX * 256 * 4;                // float [HC_MAX][2]
    static constexpr uint32_t dl_off = c_off + tcg::HC_MAX * 2 * 4;                 // float [2][128][NSUM], of every other head
    static constexpr uint32_t lam_off = dl_off + 2 * 128 * tcq::NSUM * 4;           // bf16 [128][LAM_LD]
    static constexpr uint32_t bar_off = (lam_off + tc::PT * tcg::LAM_LD * 2 + 15) & ~15u;
    static constexpr uint32_t total = bar_off + 256 + 1024;
    static_assert(total <= 227 * 1024, "shared memory of an SM");
};

template <int KD>
__global__ void __launch_bounds__(tcg::NTHREADS, 1) m2_dq_tc_kernel(const __grid_constant__ Mamba2Params p) {
    chain_wait();
    using SM = DqTcSmem<KD>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = umma::align_1024(smem_raw);
    unsigned char* sQ = smem + SM::q_off;
    unsigned char* sK = smem + SM::k_off;
    unsigned char* sDS = smem + SM::ds_off;
    unsigned char* sDO = smem + SM::do_off;
    unsigned char* sSt = smem + SM::st_off;
    float* sG = reinterpret_cast<float*>(smem + SM::g_off);
    float* sC = reinterpret_cast<float*>(smem + SM::c_off);
    float* sDL = reinterpret_cast<float*>(smem + SM::dl_off);
    bf16* sLam = reinterpret_cast<bf16*>(smem + SM::lam_off);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::bar_off);
    uint64_t* full_qk = bars + 0;
    uint64_t* barS = bars + 1;
    uint64_t* dp_full = bars + 2;
    uint64_t* ds_full = bars + 3;          // 8: dS is written, dP has been read
    uint64_t* ds_empty = bars + 4;
    uint64_t* t_empty = bars + 6;          // 4: the warps whose turn the level was
    uint64_t* t_full = bars + 7;           // [2] one per set of warps, each of which sees every other level
    uint64_t* dos_full = bars + 9;         // [2] 4
    uint64_t* dos_empty = bars + 11;       // [2]
    uint64_t* done = bars + 13;
    uint64_t* do_full = bars + 14;
    uint64_t* do_empty = bars + 15;        // 257: the row threads, and dP
    uint64_t* t_done = bars + 16;
    uint64_t* dl_full = bars + 5;          // [2] 16: the sums of a head are written, of its tile and of its levels   (5, 17)
    uint64_t* dl_full1 = bars + 17;
    uint64_t* dl_empty = bars + 18;        // [2]
    uint64_t* st_full = bars + 20;         // [NST]
    uint64_t* st_empty = st_full + tcg::NST;   // [NST] 2: the two issuing warps
    constexpr int NBARS = 20 + 2 * tcg::NST;
    static_assert(NBARS * 8 <= 232, "barriers");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + SM::bar_off + 232);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SM::bar_off + 240);
    uint32_t* sink = reinterpret_cast<uint32_t*>(smem + SM::bar_off + 244);     // written only (tile release)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int L = p.L;
    const PairWork w(p);
    const int nlev = __popc(w.pair);

    if (warp == tcg::TMA_WARP && lane == 0) {
        for (int i = 0; i < NBARS; ++i) umma::mbar_init(&bars[i], i == 3 ? 8 : (i == 5 || i == 17) ? 16 : (i == 6 || i == 9 || i == 10) ? 4 : i == 15 ? 257 : i >= NBARS - tcg::NST ? 2 : 1);
        umma::fence_mbar_init();
        *abort_flag = *p.err;
    }
    __syncthreads();
    if (*abort_flag) return;

    if (warp >= tcg::MMA_WARP) {
        if (warp == tcg::TMA_WARP && lane == 0) {
            tma::expect_tx(full_qk, 2 * tc::PT * KD * 2);
#pragma unroll
            for (int c = 0; c < KD; c += 64) {
                tma::load_seq_panel(sQ + c * tc::PT * 2, &p.tm_q, c, w.grp, w.t0, w.b, full_qk);
                tma::load_seq_panel(sK + c * tc::PT * 2, &p.tm_k, c, w.grp, w.t0, w.b, full_qk);
            }
        }
        if (warp == tcg::MMA_WARP) umma::tmem_alloc(tmem_slot, tc::TM_COLS);
    } else {
        HeadsOfTokens<tcg::WORKERS> g;
        g.load(p.g, p, w.b, w.t0, w.h0, w.nh, tid);
        const int hd = tid >> 2;
        const float D = pair_decay(p, w.b, w.h0, w.nh, w.NP, w.pair, (1 << (w.pair & 3)) - 1, tid);
        stage_lambda<tcg::LAM_LD, tcg::WORKERS / 32>(p, w.b, w.t0, w.h0, w.nh, L, sLam, warp, lane);
        g.to_shared<256>(sG, w.nh, tid);
        if (warp == 0) {
            // decay between a state's formation and this pair: of pair level 1, of the high levels
            const float D0 = __shfl_sync(0xffffffffu, D, lane & ~3), D1 = __shfl_sync(0xffffffffu, D, (lane & ~3) + 1);
            const float D2 = __shfl_sync(0xffffffffu, D, (lane & ~3) + 2);
            if ((lane & 3) == 0 && hd < w.nh) {
                sC[hd * 2] = D2;
                sC[hd * 2 + 1] = D0 + D1 + D2;
            }
        }
        asm volatile("bar.sync 1, 512;\n" ::: "memory");
        if (warp < w.nh) pair_decay_tables<2>(sG + warp * 256, nullptr, lane);
        if (tid < 2 * tc::PT) {
            // d lambda of the levels that the pair does not read, for every head
            for (int i = 8; i < L; ++i)
                if (!((w.pair >> (i - 8)) & 1)) sDL[tid * tcq::NSUM + i] = 0.f;
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tbase = *tmem_slot;

    if (warp >= tcg::MMA_WARP) {
      tcg::regs_issue();
      if (warp == tcg::TMA_WARP) {
        if (lane == 0) {
            int st = 0, ndo = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int hh = 0; hh < w.nh && ok; ++hh) {
                const long bh = (long)w.b * p.H + w.h0 + hh;
                int bits = w.pair;
                if (hh > 0 && !(ok = umma::mbar_wait(do_empty, (hh - 1) & 1, abort_flag))) break;
                tma::expect_tx(do_full, tc::V_BYTES);
                tma::load_seq_panel(sDO, &p.tm_do, 0, w.h0 + hh, w.t0, w.b, do_full);
                ++ndo;
                for (int j = 0; j <= nlev; ++j) {
                    if (!(ok = umma::mbar_wait(&st_empty[st], ph, abort_flag))) break;
                    unsigned char* dst = sSt + st * tc::V_BYTES;
                    if (j == 0) {
                        tma::expect_tx(&st_full[st], tc::V_BYTES);
                        tma::load_seq_panel(dst, &p.tm_v, 0, w.h0 + hh, w.t0, w.b, &st_full[st]);
                    } else {
                        const int lv = __ffs(bits) - 1;
                        bits &= bits - 1;
                        tma::expect_tx(&st_full[st], KD * tc::VD * 2);
                        if (lv < 2) {
                            // a state of pair level 1 stays for two pairs
                            const long tile = bh * w.NP + (lv == 1 ? (w.pair & ~1) : w.pair);
                            tma::load_panel(dst, &p.tm_lo, 0, 0, (int)(tile * KD), &st_full[st]);
                        } else {
                            const long tile = (bh * p.NS + (w.pair >> 2)) * p.LH + (lv - 2);
                            tma::load_panel(dst, &p.tm_h0, 0, 0, (int)(tile * KD), &st_full[st]);
                        }
                    }
                    if (++st == tcg::NST) {
                        st = 0;
                        ph ^= 1;
                    }
                }
            }
            if (!ok) {
                // gave up: nothing may still be on its way into shared memory when the CTA ends
                const uint32_t limit = 1u << 16;
                umma::mbar_wait(full_qk, 0, limit);
                if (ndo > 0) umma::mbar_wait(do_full, (ndo - 1) & 1, limit);
                for (int i = 0; i < tcg::NST; ++i) umma::mbar_wait(&st_full[i], (i < st ? ph : ph ^ 1) ^ 1, limit);
            }
        }
        __syncwarp();
      } else if (warp == tcg::OUT_WARP) {
        // ---- d lambda rows, all levels of them (zeros where the pair reads none); q.dq; totals of level 7
        const int per = 32 / L, sub = lane / L, i = lane - sub * L, step_s = per * tcq::NSUM;
        const long step_d = (long)per * p.H * L;
        const bool halves = i == 6 || i == 7;
        for (int hh = 0; hh < w.nh; ++hh) {
            const int h = w.h0 + hh;
            umma::mbar_wait((hh & 1) ? dl_full1 : dl_full, (hh >> 1) & 1, abort_flag);
            const float* sums = sDL + (hh & 1) * 128 * tcq::NSUM;
            float z = 0.f;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int rr = u * 32 + lane;
                const float* d = sums + rr * tcq::NSUM;
                if (w.t0 + rr < p.T)
                    p.wq[((long)w.b * p.T + w.t0 + rr) * p.H + h] = (d[tcq::C_LEV] + d[tcq::C_LEV + 1]) + (d[tcq::C_TILE] + d[tcq::C_TILE + 1]);
                if (u >= 2 && L > 7) z += __bfloat162float(sLam[rr * tcg::LAM_LD + hh * L + 7]) * (d[7] + d[7 + tcq::C_HALF]);
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) z += __shfl_xor_sync(0xffffffffu, z, d);
            if (lane == 0) {
                // the second chunk reads the first; its contributor total is the same
                const long c = ((long)w.b * p.H + h) * p.NT + w.pair * 2;
                if (w.pair * 2 + 1 < p.NT) p.Zc[(c + 1) * p.LZ] = z;
                p.Yc[c * (M2_MLOW + 1)] = z;
            }
            // as many whole rows as fit on the lanes at once: a lane keeps its level, so that a step is two loads, a sum and a store.  (With 32 values of any
            // rows a step, or several tokens' rows of a wider index, the warp's 1500 instructions a head were the longest chain of the kernel.)
            const int left = min(tc::PT, p.T - w.t0);
            const float* src = sums + sub * tcq::NSUM + i;
            float* dst = p.dl + (((long)w.b * p.T + w.t0 + sub) * p.H + h) * L + i;
            int n = sub < per ? (left - sub + per - 1) / per : 0;
            for (; n >= 4; n -= 4) {
                float v[4], x[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = src[u * step_s];
                if (halves)
#pragma unroll
                    for (int u = 0; u < 4; ++u) x[u] = src[u * step_s + tcq::C_HALF];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    *dst = v[u] + x[u];
                    dst += step_d;
                }
                src += 4 * step_s;
            }
            for (; n > 0; --n, src += step_s, dst += step_d) *dst = halves ? src[0] + src[tcq::C_HALF] : src[0];
            __syncwarp();
            if (lane == 0) arrive(&dl_empty[hh & 1]);
        }
      } else if (warp == tcg::T_WARP) {
        // (whole warps issue, see umma::elect_one)
        constexpr uint32_t ID_KM64 = umma::idesc_bf16(128, 64, false, true);
        const uint32_t lead = umma::elect_one(), aQ = umma::smem_addr(sQ), aSt = umma::smem_addr(sSt);
        auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, umma::mbar_wait(bar, parity, abort_flag)); };
        bool ok = wait(full_qk, 0);
        int st = 0, turn = 0;
        uint32_t phst = 0;
        for (int hh = 0; hh < w.nh && ok; ++hh)
            for (int j = 0; j <= nlev; ++j) {
                if (!(ok = wait(&st_full[st], phst))) break;
                if (j > 0) {
                    if (!(ok = wait(t_empty, (turn & 1) ^ 1))) break;
                    umma::fence_after_sync();
                    umma::gemm_km_lead<tc::PT, KD, KD>(lead, tbase + tcq::TM_T, aQ, aSt + st * tc::V_BYTES, ID_KM64, false);
                    umma::commit_lead(lead, &t_full[turn & 1]);
                    umma::commit_lead(lead, &st_empty[st]);
                    ++turn;
                } else if (lead) {
                    arrive(&st_empty[st]);           // (the stage of v is the other issuing warp's)
                }
                __syncwarp();
                if (++st == tcg::NST) {
                    st = 0;
                    phst ^= 1;
                }
            }
        umma::commit_lead(lead, t_done);
        umma::mbar_wait(t_done, 0, 1u << 16);            // (short, unless a wait gave up: no product may read shared memory when the CTA ends)
        __syncwarp();
      } else if (warp == tcg::MMA_WARP) {
        constexpr uint32_t ID_KK = umma::idesc_bf16(128, 128, false, false);
        constexpr uint32_t ID_KM_KD = umma::idesc_bf16(128, KD, false, true), ID_KK_KD = umma::idesc_bf16(128, KD, false, false);
        const uint32_t lead = umma::elect_one();
        const uint32_t aK = umma::smem_addr(sK), aSt = umma::smem_addr(sSt), aDS = umma::smem_addr(sDS), aDO = umma::smem_addr(sDO);
        auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, umma::mbar_wait(bar, parity, abort_flag)); };
        bool ok = wait(full_qk, 0);
        umma::gemm_kk_lead<tc::PT, tc::PT, KD>(lead, tbase + tcq::TM_S, umma::smem_addr(sQ), aK, ID_KK, false);
        umma::commit_lead(lead, barS);
        int st = 0, dos = 0;
        uint32_t phst = 0, phdos = 0;
        bool started = false;                        // dq holds a product
        auto next_stage = [&]() {
            if (++st == tcg::NST) {
                st = 0;
                phst ^= 1;
            }
        };
        auto issue_dp = [&](int hh) -> bool {
            if (!(wait(do_full, hh & 1) && wait(&st_full[st], phst))) return false;
            umma::fence_after_sync();
            umma::gemm_kk_lead<tc::PT, tc::PT, tc::VD>(lead, tbase + tcq::TM_DP, aDO, aSt + st * tc::V_BYTES, ID_KK, false);
            umma::commit_lead(lead, dp_full);
            umma::commit_lead(lead, do_empty);
            umma::commit_lead(lead, &st_empty[st]);
            next_stage();
            return true;
        };
        ok = ok && issue_dp(0);
        for (int hh = 0; hh < w.nh && ok; ++hh) {
            for (int j = 0; j < nlev; ++j) {
                if (!(ok = wait(&st_full[st], phst) && wait(&dos_full[dos], phdos))) break;
                umma::fence_after_sync();
                umma::gemm_tk_lead<KD, tc::VD>(lead, tbase + tcq::TM_DQ, tbase + tcq::TM_DOS + dos * 32, aSt + st * tc::V_BYTES, ID_KK_KD, started);
                started = true;
                umma::commit_lead(lead, &dos_empty[dos]);
                umma::commit_lead(lead, &st_empty[st]);
                next_stage();
                dos ^= 1;
                if (dos == 0) phdos ^= 1;
            }
            if (!ok || !(ok = wait(ds_full, hh & 1))) break;
            // the next head's dP first: the warps that wait for it are the longer chain
            if (hh + 1 < w.nh && !(ok = issue_dp(hh + 1))) break;
            umma::fence_after_sync();
            umma::gemm_km_lead<tc::PT, tc::PT, tc::PT>(lead, tbase + tcq::TM_DQ, aDS, aK, ID_KM_KD, started);
            started = true;
            umma::commit_lead(lead, ds_empty);
        }
        umma::commit_lead(lead, done);
        if (!ok) umma::mbar_wait(done, 0, 1u << 16);     // gave up: no product may still read shared memory when the CTA ends
        __syncwarp();
      }
    } else if (warp < 8) {
        tcg::regs_tiles();
        // ---- S, dP -> dS (bf16 tile) and the d lambda sums of the 8 levels inside the pair.  This thread: row `row`, and in every 32-column block
        //      jb <= rb the 16 columns [jb*32 + ch*16, +16)
        const int rb = warp & 3, row = rb * 32 + lane, ch = warp >> 2;
        const bool B0 = lane & 1, B1 = lane & 2, B2 = lane & 4, B3 = lane & 8;
        const bool hi = (((lane >> 4) & 1) != ch);
        umma::mbar_wait(barS, 0, abort_flag);
        // blocks above the diagonal: zeros, which every head leaves as they are
#pragma unroll 1
        for (int jb = rb + 1; jb < 4; ++jb)
#pragma unroll
            for (int c = 0; c < 2; ++c)
                *reinterpret_cast<uint4*>(sDS + umma::tile_offset(row, jb * 32 + ch * 16 + c * 8, tc::PT)) = make_uint4(0u, 0u, 0u, 0u);
        for (int hh = 0; hh < w.nh; ++hh) {
            const float* tG = sG + hh * 256;
            const float* tCf = tG + 128;
            const float Gi = tG[row];
            float lam[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) lam[i] = (i < L) ? __bfloat162float(sLam[row * tcg::LAM_LD + hh * L + i]) : 0.f;
            umma::mbar_wait(dp_full, hh & 1, abort_flag);
            if (hh > 0) {
                umma::mbar_wait(ds_empty, (hh - 1) & 1, abort_flag);
            }
            if (hh >= 2) umma::mbar_wait(&dl_empty[hh & 1], ((hh >> 1) - 1) & 1, abort_flag);
            umma::fence_after_sync();
            float bins[8];
            f32x2 wq2 = 0;                           // sum_j bf16(dS_ij) S_ij: q_i.dq_i of the tile
#pragma unroll
            for (int i = 0; i < 8; ++i) bins[i] = 0.f;
            // blocks below the diagonal: one level per block, decay factorised through the block end
#pragma unroll 1
            for (int jb = 0; jb < rb; ++jb) {
                const int j0 = jb * 32 + ch * 16;
                uint32_t packed[8];
                float s[16], dp[16];
                umma::tmem_ld16x2(umma::tmem_addr(tbase + tcq::TM_S, warp, j0), s, umma::tmem_addr(tbase + tcq::TM_DP, warp, j0), dp);
                const bool lev6 = ((rb ^ jb) == 1);
                const float lm = lev6 ? lam[6] : lam[7];
                const float rf = fexp(Gi - tG[jb * 32 + 31]);
                const f32x2 rf2 = pack2(rf, rf), lm2 = pack2(lm, lm);
                f32x2 bsum2 = 0;
#pragma unroll
                for (int e = 0; e < 16; e += 4) {
                    const float4 cf = *reinterpret_cast<const float4*>(tCf + j0 + e);
#pragma unroll
                    for (int u = 0; u < 4; u += 2) {
                        const f32x2 s2 = pack2(s[e + u], s[e + u + 1]), dec = mul2(rf2, u ? pack2(cf.z, cf.w) : pack2(cf.x, cf.y));
                        const f32x2 ed = mul2(pack2(dp[e + u], dp[e + u + 1]), dec);
                        bsum2 = fma2(ed, s2, bsum2);
                        const uint32_t ds = pack_bf16(mul2(ed, lm2));
                        wq2 = fma2(bf16x2_f32x2(ds), s2, wq2);
                        packed[(e + u) >> 1] = ds;
                    }
                }
                const float bsum = sum2(bsum2);
                if (lev6) bins[6] += bsum; else bins[7] += bsum;
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    *reinterpret_cast<uint4*>(sDS + umma::tile_offset(row, j0 + c * 8, tc::PT)) =
                        make_uint4(packed[c * 4], packed[c * 4 + 1], packed[c * 4 + 2], packed[c * 4 + 3]);
            }
            // diagonal block, eight columns at a time (a run-time loop: short code, see below): levels 0..5, causal mask folded into the exponent.  The level of
            // (row, column) is the position of the highest bit in which they differ: lambda is picked by selects on the row's own bits, and the d lambda sum of
            // level k is the sum over the sibling block of size 2^(k-1) of the row's own position, taken from a binary tree of partial sums.  A thread whose
            // columns lie in the other half of the 32-block (bit 4 differs) has level 5 throughout.
            // Short code: four or five warps of a scheduler in as many roles do not fit its instruction cache with their loops unrolled (1.4 of 13.7 warps
            // waited for instructions).
#pragma unroll 1
            for (int hf = 0; hf < 2; ++hf) {
                const int j0 = rb * 32 + ch * 16 + hf * 8;
                const bool q3 = B3 != (hf != 0);                               // the columns are in the other half of the row's sixteen
                float s[8], dp[8], es[8];
                umma::tmem_ld8x2(umma::tmem_addr(tbase + tcq::TM_S, warp, j0), s, umma::tmem_addr(tbase + tcq::TM_DP, warp, j0), dp);
                const float lm45 = hi ? lam[5] : lam[4];
                const bool far = hi || q3;
                uint32_t packed[4];
#pragma unroll
                for (int e = 0; e < 8; e += 4) {
                    const float4 gj = *reinterpret_cast<const float4*>(tG + j0 + e);
                    const float gjv[4] = {gj.x, gj.y, gj.z, gj.w};
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int ee = e + u;                                  // low three bits of the column
                        const float d = (ch * 16 + hf * 8 + ee <= lane) ? (Gi - gjv[u]) : -INFINITY;
                        const float ed = dp[ee] * fexp(d);
                        es[ee] = ed * s[ee];
                        const bool q2 = (ee & 4) ? !B2 : B2, q1 = (ee & 2) ? !B1 : B1, q0 = (ee & 1) ? !B0 : B0;
                        float lm = q0 ? lam[1] : lam[0];
                        lm = q1 ? lam[2] : lm;
                        lm = q2 ? lam[3] : lm;
                        lm = far ? lm45 : lm;
                        dp[ee] = ed * lm;
                    }
#pragma unroll
                    for (int u = 0; u < 4; u += 2) {
                        const uint32_t ds = pack_bf16(dp[e + u], dp[e + u + 1]);
                        wq2 = fma2(bf16x2_f32x2(ds), pack2(s[e + u], s[e + u + 1]), wq2);
                        packed[(e + u) >> 1] = ds;
                    }
                }
                *reinterpret_cast<uint4*>(sDS + umma::tile_offset(row, j0, tc::PT)) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                // walk down the tree of partial sums along the row's own bits 2, 1, 0
                const float p0 = es[0] + es[1], p1 = es[2] + es[3], p2 = es[4] + es[5], p3 = es[6] + es[7];
                const float q0s = p0 + p1, q1s = p2 + p3, sum = q0s + q1s;
                const float e0 = B2 ? p2 : p0, e1 = B2 ? p3 : p1;
                float f4[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) f4[i] = B2 ? es[4 + i] : es[i];
                const float g0 = B1 ? f4[2] : f4[0], g1 = B1 ? f4[3] : f4[1];
                if (far) {
                    bins[4] += hi ? 0.f : sum;
                    bins[5] += hi ? sum : 0.f;
                } else {
                    bins[0] = B0 ? g1 : g0;
                    bins[1] = B0 ? g0 : g1;
                    bins[2] = B1 ? e0 : e1;
                    bins[3] = B2 ? q0s : q1s;
                }
            }
            // (a thread whose columns of the diagonal block lie in the row's own half has levels 0..4 of the row, the other one level 5)
            float* myDL = sDL + ((hh & 1) * 128 + row) * tcq::NSUM;
            if (hi) {
                myDL[5] = bins[5];
            } else {
#pragma unroll
                for (int i = 0; i < 5; ++i) myDL[i] = bins[i];
            }
            myDL[6 + ch * tcq::C_HALF] = bins[6];
            myDL[7 + ch * tcq::C_HALF] = bins[7];
            myDL[tcq::C_TILE + ch] = sum2(wq2);
            umma::fence_async_smem();
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                arrive(ds_full);
                arrive((hh & 1) ? dl_full1 : dl_full);
            }
        }
    } else {
        tcg::regs_rows();
        // ---- levels read: scaled copies of do (tensor memory, A operand of the dq product), d lambda = s_i (do_i . T_i).  A thread has a whole row;
        //      the two sets of four warps take the CTA's levels in turn
        const int rb = warp & 3, row = rb * 32 + lane, set = (warp - 8) >> 2;
        int turn = 0;                                // levels so far
        for (int hh = 0; hh < w.nh; ++hh) {
            const int h = w.h0 + hh;
            const float Gi = sG[hh * 256 + row];
            const float e0 = fexp(Gi), e1 = fexp(Gi + sC[hh * 2]), e2 = fexp(Gi + sC[hh * 2 + 1]);
            uint4 dox[8];
            umma::mbar_wait(do_full, hh & 1, abort_flag);
            {
                uint32_t digest = 0;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    dox[c] = *reinterpret_cast<const uint4*>(sDO + umma::tile_offset(row, c * 8, tc::PT));
                    digest ^= (dox[c].x ^ dox[c].y) ^ (dox[c].z ^ dox[c].w);
                }
                release_tile_after_loads(do_empty, sink, digest);
            }
            float wsum = 0.f;                        // this set's share of sum_l lambda d lambda
            float* myLev = sDL + ((hh & 1) * 128 + row) * tcq::NSUM;
            if (hh >= 2) umma::mbar_wait(&dl_empty[hh & 1], ((hh >> 1) - 1) & 1, abort_flag);
            int bits = w.pair;
            for (int j = 0; j < nlev; ++j, ++turn) {
                const int lv = __ffs(bits) - 1;
                bits &= bits - 1;
                if ((turn & 1) != set) continue;
                const float lm = __bfloat162float(sLam[row * tcg::LAM_LD + hh * L + 8 + lv]), sc = lv == 0 ? e0 : lv == 1 ? e1 : e2, rs = lm * sc;
                const uint32_t tdos = umma::tmem_addr(tbase + tcq::TM_DOS, warp, set * 32);
                if (turn >= 2) umma::mbar_wait(&dos_empty[set], ((turn >> 1) - 1) & 1, abort_flag);
                umma::fence_after_sync();
                const f32x2 rs2 = pack2(rs, rs);
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    uint32_t x[16];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t xw[4] = {dox[hf * 4 + c].x, dox[hf * 4 + c].y, dox[hf * 4 + c].z, dox[hf * 4 + c].w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) x[c * 4 + e] = pack_bf16(mul2(bf16x2_f32x2(xw[e]), rs2));
                    }
                    umma::tmem_st16u(tdos + hf * 16, x);
                }
                umma::tmem_wait_st();
                umma::fence_before_sync();
                __syncwarp();
                if (lane == 0) arrive(&dos_full[set]);
                umma::mbar_wait(&t_full[set], (turn >> 1) & 1, abort_flag);
                umma::fence_after_sync();
                f32x2 dot2[2] = {0, 0};
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    float x[32];
                    umma::tmem_ld32(umma::tmem_addr(tbase + tcq::TM_T, warp, hf * 32), x);
                    if (hf == 1) {
                        umma::fence_before_sync();
                        __syncwarp();
                        if (lane == 0) arrive(t_empty);
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t xw[4] = {dox[hf * 4 + c].x, dox[hf * 4 + c].y, dox[hf * 4 + c].z, dox[hf * 4 + c].w};
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            dot2[e & 1] = fma2(bf16x2_f32x2(xw[e]), pack2(x[c * 8 + 2 * e], x[c * 8 + 2 * e + 1]), dot2[e & 1]);
                    }
                }
                const float dot = sum2(dot2[0]) + sum2(dot2[1]);
                const float dlv = sc * dot;
                myLev[8 + lv] = dlv;
                float z = lm * dlv;
                wsum += z;
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) z += __shfl_xor_sync(0xffffffffu, z, d);
                // reader totals per chunk: two warps each, from zero
                const int c = w.pair * 2 + (rb >> 1);
                if (lane == 0 && c < p.NT) red_add_f32(p.Zc + (((long)w.b * p.H + h) * p.NT + c) * p.LZ + 1 + lv, z);
            }
            myLev[tcq::C_LEV + set] = wsum;
            __syncwarp();
            if (lane == 0) arrive((hh & 1) ? dl_full1 : dl_full);
        }
        // ---- dq of these heads, in the place of q and k (every level read is behind the barrier, every other product behind `done`)
        bar_rows();
        umma::mbar_wait(done, 0, abort_flag);
        umma::fence_after_sync();
        if (p.dq_out) stage_gradient_bf16<KD>(smem + SM::q_off, tbase + tcq::TM_DQ, warp, row, set, 2);
        else stage_gradient<KD>(smem + SM::q_off, tbase + tcq::TM_DQ, warp, row, set, 2);
        umma::fence_async_smem();
        bar_rows();
        if (tid == 256 && !*abort_flag) store_gradient<KD>(&p.tm_dq, p.dq_out != nullptr, w.grp, w.t0, w.b, smem + SM::q_off);
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (warp == tcg::MMA_WARP) {
        if (*abort_flag && lane == 0) atomicExch(p.err, 1);
        umma::tmem_dealloc(tbase, tc::TM_COLS);
    }
}

// ------------------------------------------------------------------------------------------
// dk, dv, contributor totals
// ------------------------------------------------------------------------------------------
namespace tck {
constexpr int TM_S = 0, TM_DP = 128, TM_DK = 256, TM_DV = 384, TM_U = 448;     // U: k A_l, then the scaled copy of v (bf16, 32 columns) in its place
constexpr int NINTRA = 8, LAM_LD = 72;       // lambda columns of a head staged here; row stride (16-byte rows of a head's eight)
}  // namespace tck

template <int KD>
struct DkvTcSmem {
    static constexpr uint32_t q_off = 0;                                            // q and k: the fp32 staging of dk at the end
    static constexpr uint32_t k_off = q_off + tc::PT * KD * 2;
    static constexpr uint32_t p_off = k_off + tc::PT * KD * 2;
    static constexpr uint32_t ds_off = p_off + tc::PT * tc::PT * 2;
    static constexpr uint32_t do_off = ds_off + tc::PT * tc::PT * 2;                // [2] do; then dv of the same head on its way out
    static constexpr uint32_t v_off = do_off + 2 * tc::V_BYTES;
    static constexpr uint32_t a_off = v_off + tc::V_BYTES;
    static constexpr uint32_t g_off = a_off + tc::V_BYTES;                          // float [HC_MAX][2][128]
    static constexpr uint32_t w_off = g_off + tcg::HC_MAX * 256 * 4;                // float [2][2][2][128] k.dk halves of a head's tile, and with its state, of every other head
    static constexpr uint32_t lam_off = w_off + 1024 * 4;                           // bf16 [128][LAM_LD]
    static constexpr uint32_t bar_off = (lam_off + tc::PT * tck::LAM_LD * 2 + 15) & ~15u;
    static_assert(lam_off % 16 == 0, "16-byte loads of lambda");
    static constexpr uint32_t total = bar_off + 256 + 1024;
};

template <int KD>
__global__ void __launch_bounds__(tcg::NTHREADS, 1) m2_dkv_tc_kernel(const __grid_constant__ Mamba2Params p) {
    chain_wait();
    using SM = DkvTcSmem<KD>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = umma::align_1024(smem_raw);
    unsigned char* sQ = smem + SM::q_off;
    unsigned char* sK = smem + SM::k_off;
    unsigned char* sP = smem + SM::p_off;
    unsigned char* sDS = smem + SM::ds_off;
    unsigned char* sDO = smem + SM::do_off;
    unsigned char* sV = smem + SM::v_off;
    unsigned char* sA = smem + SM::a_off;
    float* sG = reinterpret_cast<float*>(smem + SM::g_off);
    float* sW = reinterpret_cast<float*>(smem + SM::w_off);
    bf16* sLam = reinterpret_cast<bf16*>(smem + SM::lam_off);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::bar_off);
    uint64_t* full_qk = bars + 0;
    uint64_t* barS = bars + 1;
    uint64_t* dp_full = bars + 2;
    uint64_t* ps_full = bars + 3;          // 8: P and dS are written, dP has been read   (all four transposed)
    uint64_t* ps_empty = bars + 4;
    uint64_t* u_full = bars + 5;
    uint64_t* vs_full = bars + 6;          // 8: the scaled copy of v is in the place of U
    uint64_t* dv_full = bars + 7;
    uint64_t* dv_empty = bars + 8;         // 8
    uint64_t* done = bars + 9;
    uint64_t* do_full = bars + 10;         // [2]
    uint64_t* do_empty = bars + 12;        // [2]
    uint64_t* v_full = bars + 14;
    uint64_t* v_empty = bars + 15;         // 257: the row threads, and dP
    uint64_t* a_full = bars + 16;
    uint64_t* a_read = bars + 17;          // its products are complete
    uint64_t* out_full = bars + 18;        // [2] 8: dv and k.dk of a head are written
    constexpr int NBARS = 20;
    static_assert(NBARS * 8 <= 200, "barriers");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + SM::bar_off + 200);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SM::bar_off + 208);
    uint32_t* sink = reinterpret_cast<uint32_t*>(smem + SM::bar_off + 212);     // written only (tile release)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const PairWork w(p);
    // whether somebody reads a state that this pair contributes to: any pair but the last one has readers
    const bool read = w.pair + 1 < w.NP;

    if (warp == tcg::TMA_WARP && lane == 0) {
        for (int i = 0; i < NBARS; ++i) umma::mbar_init(&bars[i], (i == 3 || i == 6 || i == 8 || i >= 18) ? 8 : i == 15 ? 257 : 1);
        umma::fence_mbar_init();
        *abort_flag = *p.err;
    }
    __syncthreads();
    if (*abort_flag) return;

    if (warp >= tcg::MMA_WARP) {
        if (warp == tcg::TMA_WARP && lane == 0) {
            tma::expect_tx(full_qk, 2 * tc::PT * KD * 2);
#pragma unroll
            for (int c = 0; c < KD; c += 64) {
                tma::load_seq_panel(sQ + c * tc::PT * 2, &p.tm_q, c, w.grp, w.t0, w.b, full_qk);
                tma::load_seq_panel(sK + c * tc::PT * 2, &p.tm_k, c, w.grp, w.t0, w.b, full_qk);
            }
        }
        if (warp == tcg::MMA_WARP) umma::tmem_alloc(tmem_slot, tc::TM_COLS);
    } else {
        HeadsOfTokens<tcg::WORKERS> g;
        g.load(p.g, p, w.b, w.t0, w.h0, w.nh, tid);
        stage_lambda<tck::LAM_LD, tcg::WORKERS / 32>(p, w.b, w.t0, w.h0, w.nh, tck::NINTRA, sLam, warp, lane);
        g.to_shared<256>(sG, w.nh, tid);
        asm volatile("bar.sync 1, 512;\n" ::: "memory");
        if (warp < w.nh) pair_decay_tables<2>(sG + warp * 256, nullptr, lane);
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tbase = *tmem_slot;

    if (warp >= tcg::MMA_WARP) {
      tcg::regs_issue();
      if (warp == tcg::TMA_WARP) {
        if (lane == 0) {
            bool ok = true;
            int hh = 0, na = 0;
            for (; hh < w.nh && ok; ++hh) {
                const long bh = (long)w.b * p.H + w.h0 + hh;
                if (hh >= 2 && !(ok = umma::mbar_wait(&do_empty[hh & 1], ((hh >> 1) - 1) & 1, abort_flag))) break;
                tma::expect_tx(&do_full[hh & 1], tc::V_BYTES);
                tma::load_seq_panel(sDO + (hh & 1) * tc::V_BYTES, &p.tm_do, 0, w.h0 + hh, w.t0, w.b, &do_full[hh & 1]);
                if (hh >= 1 && !(ok = umma::mbar_wait(v_empty, (hh - 1) & 1, abort_flag))) break;
                tma::expect_tx(v_full, tc::V_BYTES);
                tma::load_seq_panel(sV, &p.tm_v, 0, w.h0 + hh, w.t0, w.b, v_full);
                if (read) {
                    if (hh >= 1 && !(ok = umma::mbar_wait(a_read, (hh - 1) & 1, abort_flag))) break;
                    tma::expect_tx(a_full, KD * tc::VD * 2);
                    tma::load_panel(sA, &p.tm_lo_a, 0, 0, (int)((bh * w.NP + w.pair) * KD), a_full);
                    ++na;
                }
            }
            if (!ok) {
                // gave up: nothing may still be on its way into shared memory when the CTA ends
                const uint32_t limit = 1u << 16;
                umma::mbar_wait(full_qk, 0, limit);
                for (int i = max(0, hh - 2); i <= hh && i < w.nh; ++i) umma::mbar_wait(&do_full[i & 1], (i >> 1) & 1, limit);
                for (int i = max(0, hh - 1); i <= hh && i < w.nh; ++i) umma::mbar_wait(v_full, i & 1, limit);
                if (na > 0) umma::mbar_wait(a_full, (na - 1) & 1, limit);
            }
        }
        __syncwarp();
      } else if (warp == tcg::OUT_WARP) {
        for (int hh = 0; hh < w.nh; ++hh) {
            umma::mbar_wait(&out_full[hh & 1], (hh >> 1) & 1, abort_flag);
            if (lane == 0) {
                if (!*abort_flag) tma::store_seq_box(&p.tm_dv, 0, w.h0 + hh, w.t0, w.b, sDO + (hh & 1) * tc::V_BYTES);
                tma::commit_group();
            }
            const float* W = sW + ((hh & 1) * 4 + 2) * 128;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int rr = u * 32 + lane;
                if (w.t0 + rr < p.T) red_add_f32(p.wq + ((long)w.b * p.T + w.t0 + rr) * p.H + w.h0 + hh, -(W[rr] + W[128 + rr]));
            }
            __syncwarp();
            if (lane == 0) {
                tma::wait_group_read0();
                arrive(&do_empty[hh & 1]);
            }
        }
        if (lane == 0) tma::wait_group0();
        __syncwarp();
      } else if (warp == tcg::T_WARP) {
        // states: U = k A, then dk += (v scale) A^T   (whole warps issue, see umma::elect_one)
        constexpr uint32_t ID_KM64 = umma::idesc_bf16(128, 64, false, true);
        const uint32_t lead = umma::elect_one(), aK = umma::smem_addr(sK), aA = umma::smem_addr(sA);
        auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, umma::mbar_wait(bar, parity, abort_flag)); };
        bool ok = wait(full_qk, 0);
        int n = 0;
        if (read)
            for (; n < w.nh && ok; ++n) {
                // (U's place holds the previous head's copy of v until a_read)
                if (!(ok = wait(a_full, n & 1))) break;
                if (n > 0 && !(ok = wait(a_read, (n - 1) & 1))) break;
                umma::fence_after_sync();
                umma::gemm_km_lead<tc::PT, KD, KD>(lead, tbase + tck::TM_U, aK, aA, ID_KM64, false);
                umma::commit_lead(lead, u_full);
            }
        if (!ok && n > 0) umma::mbar_wait(u_full, (n - 1) & 1, 1u << 16);     // gave up: no product may still read shared memory when the CTA ends
        __syncwarp();
      } else if (warp == tcg::MMA_WARP) {
        constexpr uint32_t ID_KK = umma::idesc_bf16(128, 128, false, false);
        constexpr uint32_t ID_KM64 = umma::idesc_bf16(128, 64, false, true);
        constexpr uint32_t ID_KM_KD = umma::idesc_bf16(128, KD, false, true), ID_KK_KD = umma::idesc_bf16(128, KD, false, false);
        const uint32_t lead = umma::elect_one();
        const uint32_t aQ = umma::smem_addr(sQ), aV = umma::smem_addr(sV), aA = umma::smem_addr(sA), aDO = umma::smem_addr(sDO);
        const uint32_t aP = umma::smem_addr(sP), aDS = umma::smem_addr(sDS);
        auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, umma::mbar_wait(bar, parity, abort_flag)); };
        bool ok = wait(full_qk, 0);
        umma::gemm_kk_lead<tc::PT, tc::PT, KD>(lead, tbase + tck::TM_S, umma::smem_addr(sK), aQ, ID_KK, false);
        umma::commit_lead(lead, barS);
        bool started = false;                        // dk holds a product
        auto issue_dp = [&](int hh) -> bool {
            if (!(wait(&do_full[hh & 1], (hh >> 1) & 1) && wait(v_full, hh & 1))) return false;
            umma::fence_after_sync();
            umma::gemm_kk_lead<tc::PT, tc::PT, tc::VD>(lead, tbase + tck::TM_DP, aV, aDO + (hh & 1) * tc::V_BYTES, ID_KK, false);
            umma::commit_lead(lead, dp_full);
            umma::commit_lead(lead, v_empty);
            return true;
        };
        ok = ok && issue_dp(0);
        for (int hh = 0; hh < w.nh && ok; ++hh) {
            if (read) {
                if (!(ok = wait(vs_full, hh & 1))) break;
                umma::fence_after_sync();
                umma::gemm_tk_lead<KD, tc::VD>(lead, tbase + tck::TM_DK, tbase + tck::TM_U, aA, ID_KK_KD, started);
                started = true;
                umma::commit_lead(lead, a_read);
            }
            if (!(ok = wait(ps_full, hh & 1))) break;
            // the next head's dP first: the warps that wait for it are the longer chain
            if (hh + 1 < w.nh && !(ok = issue_dp(hh + 1))) break;
            if (hh > 0 && !(ok = wait(dv_empty, (hh - 1) & 1))) break;
            umma::fence_after_sync();
            umma::gemm_km_lead<tc::PT, tc::PT, tc::PT>(lead, tbase + tck::TM_DV, aP, aDO + (hh & 1) * tc::V_BYTES, ID_KM64, false);
            umma::commit_lead(lead, dv_full);
            umma::gemm_km_lead<tc::PT, tc::PT, tc::PT>(lead, tbase + tck::TM_DK, aDS, aQ, ID_KM_KD, started);
            started = true;
            umma::commit_lead(lead, ps_empty);
        }
        umma::commit_lead(lead, done);
        if (!ok) umma::mbar_wait(done, 0, 1u << 16);     // gave up: no product may still read shared memory when the CTA ends
        __syncwarp();
      }
    } else if (warp < 8) {
        tcg::regs_tiles();
        // ---- S, dP -> P, dS, transposed: this thread has row j = `row` (a source) and, in every 32-column block ib >= rb of targets, the 16 columns
        //      [ib*32 + ch*16, +16), so that the sums over targets that k_j.dk_j takes stay in a thread
        const int rb = warp & 3, row = rb * 32 + lane, ch = warp >> 2;
        const bool B0 = lane & 1, B1 = lane & 2, B2 = lane & 4, B3 = lane & 8;
        const bool hi = (((lane >> 4) & 1) != ch);
        umma::mbar_wait(barS, 0, abort_flag);
        // blocks of targets before the source: zeros, which every head leaves as they are
#pragma unroll 1
        for (int ib = 0; ib < rb; ++ib)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const uint32_t off = umma::tile_offset(row, ib * 32 + ch * 16 + c * 8, tc::PT);
                *reinterpret_cast<uint4*>(sP + off) = make_uint4(0u, 0u, 0u, 0u);
                *reinterpret_cast<uint4*>(sDS + off) = make_uint4(0u, 0u, 0u, 0u);
            }
        for (int hh = 0; hh < w.nh; ++hh) {
            const float* tG = sG + hh * 256;
            const float Gj = tG[row], cfj = tG[128 + row], gend = tG[rb * 32 + 31];      // cfj = exp(gend - Gj)
            umma::mbar_wait(dp_full, hh & 1, abort_flag);
            if (hh > 0) umma::mbar_wait(ps_empty, (hh - 1) & 1, abort_flag);
            umma::fence_after_sync();
            f32x2 wk2 = 0;
            uint32_t pp[8], pd[8];
            auto store = [&](int i0) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const uint32_t off = umma::tile_offset(row, i0 + c * 8, tc::PT);
                    *reinterpret_cast<uint4*>(sP + off) = make_uint4(pp[c * 4], pp[c * 4 + 1], pp[c * 4 + 2], pp[c * 4 + 3]);
                    *reinterpret_cast<uint4*>(sDS + off) = make_uint4(pd[c * 4], pd[c * 4 + 1], pd[c * 4 + 2], pd[c * 4 + 3]);
                }
            };
            // blocks behind the diagonal one: one level per block, decay factorised through the end of the source's block
            const f32x2 cf2 = pack2(cfj, cfj);
#pragma unroll 1
            for (int ib = rb + 1; ib < 4; ++ib) {
                const int i0 = ib * 32 + ch * 16;
                // lane i of a half warp makes the factor of target i0 + i: exp(G_i - gend), lambda_i
                const int lev = ((rb ^ ib) == 1) ? 6 : 7, it = i0 + (lane & 15);
                const float fe = fexp(tG[it] - gend);
                const float fl = __bfloat162float(sLam[it * tck::LAM_LD + hh * tck::NINTRA + lev]);
                float s[16], dp[16];
                umma::tmem_ld16x2(umma::tmem_addr(tbase + tck::TM_S, warp, i0), s, umma::tmem_addr(tbase + tck::TM_DP, warp, i0), dp);
#pragma unroll
                for (int e = 0; e < 16; e += 2) {
                    const f32x2 dec = mul2(pack2(__shfl_sync(0xffffffffu, fe, e), __shfl_sync(0xffffffffu, fe, e + 1)), cf2);
                    const f32x2 lm2 = pack2(__shfl_sync(0xffffffffu, fl, e), __shfl_sync(0xffffffffu, fl, e + 1));
                    const f32x2 s2 = pack2(s[e], s[e + 1]);
                    pp[e >> 1] = pack_bf16(mul2(mul2(s2, dec), lm2));
                    pd[e >> 1] = pack_bf16(mul2(mul2(pack2(dp[e], dp[e + 1]), dec), lm2));
                    wk2 = fma2(bf16x2_f32x2(pd[e >> 1]), s2, wk2);
                }
                store(i0);
            }
            // diagonal block, eight columns at a time: the level of (target, source) is the position of the highest bit in which they differ; a target's six
            // lambdas are one load for all lanes, the selects are on the source's own bits
#pragma unroll 1
            for (int hf = 0; hf < 2; ++hf) {
                const int i0 = rb * 32 + ch * 16 + hf * 8;
                const bool q3 = B3 != (hf != 0);
                float s[8], dp[8];
                umma::tmem_ld8x2(umma::tmem_addr(tbase + tck::TM_S, warp, i0), s, umma::tmem_addr(tbase + tck::TM_DP, warp, i0), dp);
                const bf16* lrow = sLam + i0 * tck::LAM_LD + hh * tck::NINTRA;
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    const float2 gi = *reinterpret_cast<const float2*>(tG + i0 + e);
                    const bool q1 = (e & 2) ? !B1 : B1, q2 = (e & 4) ? !B2 : B2;
                    float lmv[2], dcv[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const uint4 lw = *reinterpret_cast<const uint4*>(lrow + (e + u) * tck::LAM_LD);
                        const bool q0 = u ? !B0 : B0;
                        uint32_t lm = q0 ? (lw.x & 0xffff0000u) : (lw.x << 16);
                        lm = q1 ? (lw.y << 16) : lm;
                        lm = q2 ? (lw.y & 0xffff0000u) : lm;
                        lm = q3 ? (lw.z << 16) : lm;
                        lm = hi ? (lw.z & 0xffff0000u) : lm;
                        lmv[u] = __uint_as_float(lm);
                        dcv[u] = fexp((ch * 16 + hf * 8 + e + u >= lane) ? ((u ? gi.y : gi.x) - Gj) : -INFINITY);
                    }
                    const f32x2 dec = pack2(dcv[0], dcv[1]), lm2 = pack2(lmv[0], lmv[1]), s2 = pack2(s[e], s[e + 1]);
                    pp[e >> 1] = pack_bf16(mul2(mul2(s2, dec), lm2));
                    pd[e >> 1] = pack_bf16(mul2(mul2(pack2(dp[e], dp[e + 1]), dec), lm2));
                    wk2 = fma2(bf16x2_f32x2(pd[e >> 1]), s2, wk2);
                }
                const uint32_t off = umma::tile_offset(row, i0, tc::PT);
                *reinterpret_cast<uint4*>(sP + off) = make_uint4(pp[0], pp[1], pp[2], pp[3]);
                *reinterpret_cast<uint4*>(sDS + off) = make_uint4(pd[0], pd[1], pd[2], pd[3]);
            }
            sW[((hh & 1) * 4 + ch) * 128 + row] = sum2(wk2);
            umma::fence_async_smem();
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) arrive(ps_full);
        }
    } else {
        tcg::regs_rows();
        // ---- the state contributed to, dv rows.  This thread: row `row`, columns ch*32 .. +31
        const int rb = warp & 3, row = rb * 32 + lane, ch = (warp - 8) >> 2;
        for (int hh = 0; hh < w.nh; ++hh) {
            uint32_t vx[16];
            umma::mbar_wait(v_full, hh & 1, abort_flag);
            {
                uint32_t digest = 0;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint4 x = *reinterpret_cast<const uint4*>(sV + umma::tile_offset(row, ch * 32 + c * 8, tc::PT));
                    vx[c * 4] = x.x; vx[c * 4 + 1] = x.y; vx[c * 4 + 2] = x.z; vx[c * 4 + 3] = x.w;
                    digest ^= (x.x ^ x.y) ^ (x.z ^ x.w);
                }
                release_tile_after_loads(v_empty, sink, digest);
            }
            f32x2 o[16];
            float wk = 0.f;
            if (read) {
                // what its readers send back, through k: the same roundings as those of the copy of v that the product for dk takes
                const float sc = fexp(sG[hh * 256 + 127] - sG[hh * 256 + row]);
                const f32x2 sc2 = pack2(sc, sc);
                f32x2 wk2 = 0;
                const uint32_t tu = umma::tmem_addr(tbase + tck::TM_U, warp, 0);
                uint32_t x[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) x[e] = pack_bf16(mul2(bf16x2_f32x2(vx[e]), sc2));
                umma::mbar_wait(u_full, hh & 1, abort_flag);
                umma::fence_after_sync();
                float uu[32];
                umma::tmem_ld32(tu + ch * 32, uu);
                // both warps of the lane quarter have read U: the copy of v takes its place
                umma::fence_before_sync();
                asm volatile("bar.sync %0, 64;\n" ::"r"(3 + rb) : "memory");
                umma::fence_after_sync();
                umma::tmem_st16u(tu + ch * 16, x);
                umma::tmem_wait_st();
                umma::fence_before_sync();
                __syncwarp();
                if (lane == 0) arrive(vs_full);
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const f32x2 u2 = pack2(uu[2 * e], uu[2 * e + 1]);
                    wk2 = fma2(bf16x2_f32x2(x[e]), u2, wk2);
                    o[e] = mul2(sc2, u2);
                }
                wk = sum2(wk2);
            } else {
#pragma unroll
                for (int e = 0; e < 16; ++e) o[e] = 0;
            }
            umma::mbar_wait(dv_full, hh & 1, abort_flag);
            umma::fence_after_sync();
            {
                float x[32];
                umma::tmem_ld32(umma::tmem_addr(tbase + tck::TM_DV, warp, ch * 32), x);
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float2 a = unpack2(o[e]);
                    vx[e] = pack_bf16(a.x + x[2 * e], a.y + x[2 * e + 1]);
                }
            }
            sW[((hh & 1) * 4 + 2 + ch) * 128 + row] = wk + sW[((hh & 1) * 4 + ch) * 128 + row];     // (the tile's sums are there with dS)
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) arrive(dv_empty);
            // dv leaves by way of the place of do, which its product was the last to read
            unsigned char* sOut = sDO + (hh & 1) * tc::V_BYTES;
#pragma unroll
            for (int c = 0; c < 4; ++c)
                *reinterpret_cast<uint4*>(sOut + umma::tile_offset(row, ch * 32 + c * 8, tc::PT)) =
                    make_uint4(vx[c * 4], vx[c * 4 + 1], vx[c * 4 + 2], vx[c * 4 + 3]);
            umma::fence_async_smem();
            __syncwarp();
            if (lane == 0) arrive(&out_full[hh & 1]);
        }
        // ---- dk of these heads
        umma::mbar_wait(done, 0, abort_flag);
        umma::fence_after_sync();
        if (p.dk_out) stage_gradient_bf16<KD>(smem + SM::q_off, tbase + tck::TM_DK, warp, row, ch, 2);
        else stage_gradient<KD>(smem + SM::q_off, tbase + tck::TM_DK, warp, row, ch, 2);
        umma::fence_async_smem();
        bar_rows();
        if (tid == 256 && !*abort_flag) store_gradient<KD>(&p.tm_dk, p.dk_out != nullptr, w.grp, w.t0, w.b, smem + SM::q_off);
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (warp == tcg::MMA_WARP) {
        if (*abort_flag && lane == 0) atomicExch(p.err, 1);
        umma::tmem_dealloc(tbase, tc::TM_COLS);
    }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
static int gradient_maps(Mamba2Params& p) {
    const long NP = (p.NT + 1) / 2, BH = (long)p.B * p.H;
    int rc, dev = -1, sms = 0;
    if ((rc = tma::make_seq_map(&p.tm_q, p.q, p.B, p.T, p.G, p.K, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_k, p.k, p.B, p.T, p.G, p.K, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_v, p.v, p.B, p.T, p.H, p.V, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_do, p.d_o, p.B, p.T, p.H, p.V, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_dv, p.dv, p.B, p.T, p.H, p.V, tc::PT, 2)) != 0) return rc;
    if (p.dq_out) {
        if ((rc = tma::make_seq_map(&p.tm_dq, p.dq_out, p.B, p.T, p.G, p.K, tc::PT, 2)) != 0) return rc;
        if ((rc = tma::make_seq_map(&p.tm_dk, p.dk_out, p.B, p.T, p.G, p.K, tc::PT, 2)) != 0) return rc;
    } else {
        if ((rc = tma::make_seq_map(&p.tm_dq, p.dq_acc, p.B, p.T, p.G, p.K, tc::PT, 4)) != 0) return rc;
        if ((rc = tma::make_seq_map(&p.tm_dk, p.dk_acc, p.B, p.T, p.G, p.K, tc::PT, 4)) != 0) return rc;
    }
    if (NP > 1) {
        if ((rc = tma::make_panel_map(&p.tm_lo, p.lo_H, BH * NP * p.K, 1, p.V, p.K)) != 0) return rc;
        if ((rc = tma::make_panel_map(&p.tm_lo_a, p.lo_A, BH * NP * p.K, 1, p.V, p.K)) != 0) return rc;
    }
    if (p.NS > 1) {
        if ((rc = tma::make_panel_map(&p.tm_h0, p.seg_H0, BH * p.NS * p.LH * p.K, 1, p.V, p.K)) != 0) return rc;
    }
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = sm_count(&sms, dev);
    if (e != cudaSuccess) return (int)e;
    p.hc = mamba2_heads_per_cta(p, sms);
    return 0;
}

template <int KD>
static int launch_gradients(const Mamba2Params& p, cudaStream_t stream) {
    const int per_grp = p.H / p.G, grid = p.B * ((p.NT + 1) / 2) * p.G * ((per_grp + p.hc - 1) / p.hc);
    auto kq = m2_dq_tc_kernel<KD>;
    auto kk = m2_dkv_tc_kernel<KD>;
    cudaError_t e;
    if ((e = allow_smem(kq, DqTcSmem<KD>::total)) != cudaSuccess || (e = allow_smem(kk, DkvTcSmem<KD>::total)) != cudaSuccess) return (int)e;
    llattn::launch_chained(kq, grid, tcg::NTHREADS, DqTcSmem<KD>::total, stream, p); LLATTN_LAUNCHED();
    llattn::launch_chained(kk, grid, tcg::NTHREADS, DkvTcSmem<KD>::total, stream, p); LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int mamba2_gradients_tc_launch(const Mamba2Params& p_in, cudaStream_t stream) {
    Mamba2Params p = p_in;
    const int rc = gradient_maps(p);
    if (rc != 0) return rc;
    return p.K == 128 ? launch_gradients<128>(p, stream) : launch_gradients<64>(p, stream);
}

}  // namespace llattn
