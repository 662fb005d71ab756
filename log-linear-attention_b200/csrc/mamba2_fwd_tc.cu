// Log-linear Mamba-2 outputs on the 5th-generation tensor cores (tcgen05.mma, accumulators in tensor memory), K = 64 or 128, V = 64.
//
// One CTA takes a PAIR of chunks (128 tokens) of one q / k group and walks heads of that group:
//     S   = q k^T                     128 x 128 x K    once: the heads of a group share q and k
//     T_l = q H_l                     128 x  64 x K    per head and level whose bit is set in the pair's number
//     O   = P v                       128 x  64 x 128  per head; P is S under the head's decays, causal mask and lambda (levels 0..7)
//     o_i = sum_l lambda_l exp(G_i + c_l) T_l,i + O_i
// Every level state a pair reads is in global memory as a bf16 K x V tile (the low levels from m2_state_tc_kernel, the high ones from the scan over
// segments), so pairs and heads do not depend on one another.  Two teams take the heads in turn, each with rings of its own; the products of a head are a
// stream of JOBS of one shape, A (q or P) times a 16 KB tile that TMA brings into the team's ring of stages, result in one of its two 64-column slots:
//     warp 18 + team       (one lane) tiles ahead into the ring, and the rows of x where y = o + D x
//     warp 16 + team       one chain of K / 16 (or 8) tensor-core instructions per job
//     warps 4 team ..      S -> P of its next head, into tensor memory; a thread has a whole row
//     warps 8 + 4 team ..  slots -> running sum in registers, output rows
// (warps of two teams; a CTA of one head is one team: warps 0, 4, 8 and 9 on.)  None of them waits for another but through the rings.  A wait that gives up sets the CTA's abort flag, after which every other wait of the CTA ends at
// once; warps that work in step go through the rest of their loops without waiting.
//
// What bounds it is the latency of instruction streams, not a unit (the tensor core is busy 29 % of the time, DRAM 35 %): one stream of jobs took
// 1.2 k cycles a job for the waits and the issue of eight instructions, hence two; the row warps' sums overlap the other team's outputs.
// B = 2, T = 16384, 32 heads: 180 us (half of the issue slots), where a kernel that walked a segment's pairs with one in flight per SM and one for the high levels
// took 303 + 127; B = 8, T = 4096, 24 heads: the whole forward 465 -> 261 us.
#include "rowwise.cuh"
#include "tc_common.cuh"

namespace llattn {

namespace tco {
constexpr int HC_MAX = 8;                 // heads per CTA
constexpr int LAM_MAX = 120, LAM_LD = 122;   // lambda values of a token staged per CTA; the row stride is an odd number of 32-bit words
constexpr int INTRA = 8;                  // of them the levels inside the pair
constexpr int COEF_MAX = 56;              // (head, level read) combinations of a CTA
constexpr int NSLOT = 2;                  // per team: tensor-memory slots of 64 columns
// Two teams, one CTA per SM.  A CTA of one head (one head a group, or a call too small to fill the chip with more) has work for one team only: with half of the
// threads, of tensor memory (P in the place of S) and of shared memory two of them share an SM, which a chain of loads, S, P and two products leaves idle
// for the most part.  B = 16, T = 1024, 24 heads and groups: 161 -> 92 us (with the kernels that walked segments 131 and 26 for the high levels); calls
// of fewer CTAs than SMs, us of the whole forward: T = 128, 24 heads 20.5 -> 19.6, T = 640, 4 heads 25.6 -> 24.9, T = 2048, 8 heads 33.0 -> 33.0.
template <int TEAMS>
struct Teams {
    static constexpr int NST = TEAMS == 2 ? 3 : 2;                            // per team: stages of 16 KB
    static constexpr int HC = TEAMS == 2 ? HC_MAX : 1;                        // heads
    static constexpr int LD = TEAMS == 2 ? LAM_LD : 22, LDI = HC * INTRA + 2; // (odd numbers of 32-bit words)
    static constexpr int COEF = TEAMS == 2 ? COEF_MAX : 12;                   // (a pair reads at most 12 levels)
    static constexpr int WORKERS = 256 * TEAMS, MMA_WARP = WORKERS / 32, TMA_WARP = MMA_WARP + TEAMS;
    static constexpr int NTHREADS = TEAMS == 2 ? 640 : 320;                   // (20 warps: registers move between warpgroups of four)
    static constexpr int TM_S = 0, TM_P = TEAMS == 2 ? 128 : 0, TM_SLOT = 128 * TEAMS, TM_COLS = 256 * TEAMS;
};
// two teams: launched with 96 registers a thread, 61440 in all: 256 x 88 + 256 x 128 + 128 x 48
__device__ __forceinline__ void regs_tiles() { asm volatile("setmaxnreg.dec.sync.aligned.u32 88;\n"); }
__device__ __forceinline__ void regs_rows() { asm volatile("setmaxnreg.inc.sync.aligned.u32 128;\n"); }
__device__ __forceinline__ void regs_issue() { asm volatile("setmaxnreg.dec.sync.aligned.u32 48;\n"); }
}  // namespace tco

// the four row warps of a team
__device__ __forceinline__ void team_barrier(int team) { asm volatile("bar.sync %0, 128;\n" ::"r"(2 + team) : "memory"); }

template <int KD, int TEAMS>
struct OutTcSmem {
    using TM = tco::Teams<TEAMS>;
    static constexpr uint32_t st_off = 0;                                           // [TEAMS][NST]
    static constexpr uint32_t q_off = TEAMS * TM::NST * tc::V_BYTES;
    static constexpr uint32_t k_off = q_off + tc::PT * KD * 2;                      // k, until S is complete; then per team
    static constexpr uint32_t x_off = k_off;                                        // [TEAMS] rows of x, then of the output
    static constexpr uint32_t g_off = x_off + 2 * tc::V_BYTES;                      // float [HC][2][128]: G | Cf
    static constexpr uint32_t c_off = g_off + TM::HC * 256 * 4;                     // float [HC][4]: decay since a state was formed (2), D
    static constexpr uint32_t coef_off = c_off + TM::HC * 4 * 4;                    // float [COEF][128]: lambda exp(G + c) of the levels read
    static constexpr uint32_t lami_off = coef_off + TM::COEF * 128 * 4;             // bf16 [128][LDI]
    static constexpr uint32_t lam_off = st_off;                                     // during the preparation: bf16 [128][LD] ...
    static constexpr uint32_t cum_off = st_off + 2 * tc::V_BYTES - (TEAMS == 2 ? 0 : 512);      // ... float [HC][128]
    static constexpr uint32_t bar_off = (lami_off + tc::PT * TM::LDI * 2 + 15) & ~15u;
    static constexpr uint32_t total = bar_off + 320 + 1024;                         // + slack for 1024-byte alignment
    static_assert(tc::PT * TM::LD * 2 <= cum_off && cum_off + TM::HC * 512 <= q_off, "lambda and the sums in the places of the stages");
    static_assert(TEAMS == 2 || 2 * (total + 1024) <= 228 * 1024, "two CTAs per SM");
};

// RES: 0 writes o; 1, 2 write y = o + D x of a layer (bf16 / fp32), o rounded to bf16 first as if it were stored; 3 is 1 with D x rounded to
// bf16 too (prompts, whose sum is two operators' with a bf16 D).
template <int KD, int RES, int TEAMS>
__global__ void __launch_bounds__(tco::Teams<TEAMS>::NTHREADS, TEAMS == 2 ? 1 : 2) m2_out_tc_kernel(const __grid_constant__ Mamba2Params p) {
    chain_wait();
    using SM = OutTcSmem<KD, TEAMS>;
    using TM = tco::Teams<TEAMS>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = umma::align_1024(smem_raw);
    constexpr int NST = TM::NST, NSLOT = tco::NSLOT;
    unsigned char* sQ = smem + SM::q_off;
    unsigned char* sK = smem + SM::k_off;
    float* sG = reinterpret_cast<float*>(smem + SM::g_off);
    float* sC = reinterpret_cast<float*>(smem + SM::c_off);
    float* sCoef = reinterpret_cast<float*>(smem + SM::coef_off);
    bf16* sLam = reinterpret_cast<bf16*>(smem + SM::lam_off);
    bf16* sLami = reinterpret_cast<bf16*>(smem + SM::lami_off);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::bar_off);
    uint64_t* full_qk = bars + 0;
    uint64_t* barS = bars + 1;
    constexpr int TEAM_BARS = 5 + 2 * NSLOT + 2 * NST, NBARS = 2 + TEAMS * TEAM_BARS;
    static_assert(NBARS * 8 <= 296, "barriers");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + SM::bar_off + 296);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SM::bar_off + 304);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int L = p.L, NP = (p.NT + 1) / 2;
    // (pairs from the last one on: later pairs read more levels)
    const int per_grp = p.H / p.G, nhc = (per_grp + p.hc - 1) / p.hc;
    int at = blockIdx.x;
    const int hchunk = at % nhc;
    at /= nhc;
    const int grp = at % p.G;
    at /= p.G;
    const int pair = NP - 1 - at % NP, b = at / NP;
    const int h0 = grp * per_grp + hchunk * p.hc;
    const int nh = min(p.hc, per_grp - hchunk * p.hc);
    const int t0 = pair * tc::PT;
    const int njobs = __popc(pair) + 1;

    if (warp == TM::TMA_WARP && lane == 0) {
        for (int i = 0; i < NBARS; ++i)
            umma::mbar_init(&bars[i], i >= 2 && ((i - 2) % TEAM_BARS == 0 || (i - 2) % TEAM_BARS >= TEAM_BARS - NSLOT) ? 4 : 1);
        umma::fence_mbar_init();
        *abort_flag = *p.err;                        // an earlier CTA gave up: do not pile on
    }
    __syncthreads();
    if (*abort_flag) return;                         // uniform: every thread reads the same shared word

    if (warp >= TM::MMA_WARP) {
        if (warp == TM::TMA_WARP && lane == 0) {
            tma::expect_tx(full_qk, 2 * tc::PT * KD * 2);
#pragma unroll
            for (int c = 0; c < KD; c += 64) {
                tma::load_seq_panel(sQ + c * tc::PT * 2, &p.tm_q, c, grp, t0, b, full_qk);
                tma::load_seq_panel(sK + c * tc::PT * 2, &p.tm_k, c, grp, t0, b, full_qk);
            }
        }
        if (warp == TM::MMA_WARP) umma::tmem_alloc(tmem_slot, TM::TM_COLS);
    } else {
        // (loads from global memory together: a latency each, of 1 to 2 k cycles, is what the preparation consists of)
        HeadsOfTokens<TM::WORKERS> g;
        g.load(p.g, p, b, t0, h0, nh, tid);
        const int pl = pair & 3, hd = tid >> 2;
        float D = pair_decay(p, b, h0, nh, NP, pair, (1 << pl) - 1, tid);
        if (RES && (tid & 3) == 3 && hd < nh) D = load_param(p.res_D, h0 + hd, RES == 2);
        stage_lambda<TM::LD, TM::WORKERS / 32>(p, b, t0, h0, nh, L, sLam, warp, lane);
        g.template to_shared<256>(sG, nh, tid);
        if (warp == 0) {
            // decay between a state's formation and this pair: of pair level 1, of the high levels; and D
            const float D0 = __shfl_sync(0xffffffffu, D, lane & ~3), D1 = __shfl_sync(0xffffffffu, D, (lane & ~3) + 1);
            const float D2 = __shfl_sync(0xffffffffu, D, (lane & ~3) + 2), D3 = __shfl_sync(0xffffffffu, D, (lane & ~3) + 3);
            if ((lane & 3) == 0 && hd < nh) {
                sC[hd * 4] = D2;
                sC[hd * 4 + 1] = D0 + D1 + D2;
                sC[hd * 4 + 2] = D3;
            }
        }
        asm volatile("bar.sync 1, %0;\n" ::"n"(TM::WORKERS) : "memory");
        // (the in-chunk cumulative sums go to global memory by way of the first stage)
        float* sCum = reinterpret_cast<float*>(smem + SM::cum_off);
        if (warp < nh) pair_decay_tables<2>(sG + warp * 256, sCum + warp * 128, lane);
        asm volatile("bar.sync 1, %0;\n" ::"n"(TM::WORKERS) : "memory");
        heads_to_global<128, TM::WORKERS>(p.g_cum, p, b, t0, h0, nh, sCum, tid);
        // what the heads' loops take from lambda: the levels inside the pair, and a factor per level read; a head per 128 threads
        for (int hh = tid >> 7; hh < nh; hh += 2 * TEAMS) {
            const int row = tid & 127;
            const unsigned short* l = reinterpret_cast<const unsigned short*>(sLam + row * TM::LD + hh * L);
            uint32_t li[tco::INTRA];
#pragma unroll
            for (int i = 0; i < tco::INTRA; ++i) li[i] = i < L ? l[i] : 0;
#pragma unroll
            for (int i = 0; i < tco::INTRA; i += 2)
                *reinterpret_cast<uint32_t*>(sLami + row * TM::LDI + hh * tco::INTRA + i) = li[i] | li[i + 1] << 16;
            const float G = sG[hh * 256 + row], c1 = sC[hh * 4], c2 = sC[hh * 4 + 1];
            const float e0 = fexp(G), e1 = fexp(G + c1), e2 = fexp(G + c2);
            float* coef = sCoef + hh * (njobs - 1) * 128 + row;
            int bits = pair;
#pragma unroll 4
            for (int j = 0; j < njobs - 1; ++j) {
                const int lv = __ffs(bits) - 1;
                bits &= bits - 1;
                coef[j * 128] = __uint_as_float((uint32_t)l[8 + lv] << 16) * (lv == 0 ? e0 : lv == 1 ? e1 : e2);
            }
        }
        umma::fence_async_smem();                    // tiles take the places of lambda and of the sums
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tbase = *tmem_slot;
    // the team's barriers, tensor-memory columns and stages
    const int team = TEAMS == 1 ? 0 : warp >= TM::MMA_WARP ? (warp & 1) : ((warp >> 2) & 1);
    uint64_t* p_full = bars + 2 + team * TEAM_BARS;      // 4: one arrival per warp
    uint64_t* p_empty = p_full + 1;
    uint64_t* x_full = p_full + 2;
    uint64_t* x_empty = p_full + 3;
    uint64_t* done = p_full + 4;
    uint64_t* st_full = p_full + 5;                      // [NST]
    uint64_t* st_empty = st_full + NST;
    uint64_t* slot_full = st_empty + NST;                // [NSLOT]
    uint64_t* slot_empty = slot_full + NSLOT;            // [NSLOT] 4
    const uint32_t tP = tbase + TM::TM_P + team * 64, tSlot = tbase + TM::TM_SLOT + team * NSLOT * 64;
    unsigned char* sSt = smem + SM::st_off + team * NST * tc::V_BYTES;
    unsigned char* sX = smem + SM::x_off + team * tc::V_BYTES;

    if (warp >= TM::MMA_WARP) {
      if (TEAMS == 2) tco::regs_issue();
      if (warp >= TM::TMA_WARP) {
        if (lane == 0) {
            int st = 0, nx = 0;                      // stage, tiles of x requested
            uint32_t ph = 1;                         // parity of the "empty" wait: passes at once on the first round
            bool ok = true;
            for (int hh = team; hh < nh && ok; hh += TEAMS) {
                const long bh = (long)b * p.H + h0 + hh;
                int bits = pair;
                for (int j = 0; j < njobs; ++j) {
                    if (!(ok = umma::mbar_wait(&st_empty[st], ph, abort_flag))) break;
                    unsigned char* dst = sSt + st * tc::V_BYTES;
                    if (bits) {
                        const int lv = __ffs(bits) - 1;
                        bits &= bits - 1;
                        tma::expect_tx(&st_full[st], KD * tc::VD * 2);
                        if (lv < 2) {
                            // a state of pair level 1 stays for two pairs
                            const long tile = bh * NP + (lv == 1 ? (pair & ~1) : pair);
                            tma::load_panel(dst, &p.tm_lo, 0, 0, (int)(tile * KD), &st_full[st]);
                        } else {
                            const long tile = (bh * p.NS + (pair >> 2)) * p.LH + (lv - 2);
                            tma::load_panel(dst, &p.tm_h0, 0, 0, (int)(tile * KD), &st_full[st]);
                        }
                    } else {
                        tma::expect_tx(&st_full[st], tc::V_BYTES);
                        tma::load_seq_panel(dst, &p.tm_v, 0, h0 + hh, t0, b, &st_full[st]);
                    }
                    if (++st == NST) {
                        st = 0;
                        ph ^= 1;
                    }
                }
                if (RES && ok) {
                    // (the first one: the place of k, when S is complete)
                    if (!(ok = nx == 0 ? umma::mbar_wait(barS, 0, abort_flag) : umma::mbar_wait(x_empty, (nx - 1) & 1, abort_flag))) break;
                    tma::expect_tx(x_full, tc::V_BYTES);
                    tma::load_seq_panel(sX, &p.tm_x, 0, h0 + hh, t0, b, x_full);
                    ++nx;
                }
            }
            if (!ok) {
                // gave up: nothing may still be on its way into shared memory when the CTA ends (each stage's last load has completed or is the
                // one of this parity)
                const uint32_t limit = 1u << 16;
                umma::mbar_wait(full_qk, 0, limit);
                for (int i = 0; i < NST; ++i) umma::mbar_wait(&st_full[i], (i < st ? ph : ph ^ 1) ^ 1, limit);
                if (nx > 0) umma::mbar_wait(x_full, (nx - 1) & 1, limit);
            }
        }
        __syncwarp();
      } else {
        // (the whole warp, see umma::elect_one)
        constexpr uint32_t ID_S = umma::idesc_bf16(128, 128, false, false);
        constexpr uint32_t ID_KM = umma::idesc_bf16(128, 64, false, true);
        const uint32_t lead = umma::elect_one();
        const uint32_t aSt = umma::smem_addr(sSt), aQ = umma::smem_addr(sQ);
        auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, umma::mbar_wait(bar, parity, abort_flag)); };
        bool ok = wait(full_qk, 0);
        if (team == 0) {
            umma::gemm_kk_lead<tc::PT, tc::PT, KD>(lead, tbase + TM::TM_S, aQ, umma::smem_addr(sK), ID_S, false);
            umma::commit_lead(lead, barS);
        }
        int st = 0, slot = 0;
        uint32_t phst = 0, phslot = 1, php = 0;
        for (int hh = team; hh < nh && ok; hh += TEAMS) {
            for (int j = 0; j < njobs; ++j) {
                if (!(ok = wait(&st_full[st], phst) && wait(&slot_empty[slot], phslot))) break;
                const uint32_t d = tSlot + slot * 64, tile = aSt + st * tc::V_BYTES;
                if (j + 1 < njobs) {
                    umma::fence_after_sync();
                    umma::gemm_km_lead<tc::PT, KD, KD>(lead, d, aQ, tile, ID_KM, false);
                } else {
                    if (!(ok = wait(p_full, php))) break;
                    php ^= 1;
                    umma::fence_after_sync();
                    umma::gemm_tm_lead<tc::PT, tc::PT>(lead, d, tP, tile, ID_KM, false);
                    umma::commit_lead(lead, p_empty);
                }
                umma::commit_lead(lead, &slot_full[slot]);
                umma::commit_lead(lead, &st_empty[st]);
                if (++st == NST) {
                    st = 0;
                    phst ^= 1;
                }
                if (++slot == NSLOT) {
                    slot = 0;
                    phslot ^= 1;
                }
            }
        }
        if (!ok) {
            // gave up: no product may still read shared memory when the CTA ends
            umma::commit_lead(lead, done);
            umma::mbar_wait(done, 0, 1u << 16);
        }
        __syncwarp();
      }
    } else if (warp < 4 * TEAMS) {
        if (TEAMS == 2) tco::regs_tiles();
        // ---- S -> P of every other head (bf16 pairs, A operand of P v).  This thread: row `row`, the 32-column blocks jb <= rb
        const int rb = warp & 3, row = rb * 32 + lane;
        const bool B0 = lane & 1, B1 = lane & 2, B2 = lane & 4, B3 = lane & 8, B4 = lane & 16;
        const uint32_t dst = umma::tmem_addr(tP, warp, 0);
        umma::mbar_wait(barS, 0, abort_flag);
        umma::fence_after_sync();
        auto zeros = [&]() {
            const uint32_t z[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll 1
            for (int c = (rb + 1) * 16; c < 64; c += 8) umma::tmem_st8u(dst + c, z);
        };
        // blocks above the diagonal: zeros, which every head leaves as they are
        if (TEAMS == 2) zeros();
        for (int hh = team; hh < nh; hh += TEAMS) {
            const float* tG = sG + hh * 256;
            const float* tCf = tG + 128;
            const float Gi = tG[row];
            float lam[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t w = *reinterpret_cast<const uint32_t*>(sLami + row * TM::LDI + hh * tco::INTRA + 2 * i);
                lam[2 * i] = __uint_as_float(w << 16);
                lam[2 * i + 1] = __uint_as_float(w & 0xffff0000u);
            }
            if (hh >= TEAMS) {
                umma::mbar_wait(p_empty, (hh / TEAMS - 1) & 1, abort_flag);
                umma::fence_after_sync();
            }
            // blocks below the diagonal: one level per block, decay factorised through the block end
#pragma unroll 1
            for (int jb = 0; jb < rb; ++jb) {
                float s[32];
                umma::tmem_ld32(umma::tmem_addr(tbase + TM::TM_S, warp, jb * 32), s);
                const float lm = ((rb ^ jb) == 1) ? lam[6] : lam[7];
                const float rf = lm * fexp(Gi - tG[jb * 32 + 31]);
                const f32x2 rf2 = pack2(rf, rf);
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    uint32_t x[8];
#pragma unroll
                    for (int e = 0; e < 16; e += 4) {
                        const float4 cf = *reinterpret_cast<const float4*>(tCf + jb * 32 + hf * 16 + e);
                        const float* y = s + hf * 16 + e;
                        const float2 a = unpack2(mul2(mul2(pack2(y[0], y[1]), rf2), pack2(cf.x, cf.y)));
                        const float2 c = unpack2(mul2(mul2(pack2(y[2], y[3]), rf2), pack2(cf.z, cf.w)));
                        x[e / 2] = pack_bf16(a.x, a.y);
                        x[e / 2 + 1] = pack_bf16(c.x, c.y);
                    }
                    umma::tmem_st8u(dst + jb * 16 + hf * 8, x);
                }
            }
            // diagonal block: levels 0..5, causal mask folded into the exponent.  The level of (row, column) is the position of the highest bit in
            // which they differ: per bit, "differs" is the row's own bit or its complement, so lambda is picked by selects on predicates.
            // Eight columns at a time in a run-time loop: four or five warps of a scheduler in as many roles do not fit its instruction cache unrolled.
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                const int j0 = rb * 32 + c * 8;
                const bool q3 = B3 != ((c & 1) != 0), q4 = B4 != ((c & 2) != 0);
                const float lm45 = q4 ? lam[5] : lam[4];
                const bool far = q3 || q4;
                float s[8];
                umma::tmem_ld8(umma::tmem_addr(tbase + TM::TM_S, warp, j0), s);
                uint32_t x[4];
#pragma unroll
                for (int e = 0; e < 8; e += 4) {
                    const float4 gj = *reinterpret_cast<const float4*>(tG + j0 + e);
                    const float gjv[4] = {gj.x, gj.y, gj.z, gj.w};
                    const bool q2 = (e & 4) ? !B2 : B2;
                    float y[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const bool q1 = (u & 2) ? !B1 : B1, q0 = (u & 1) ? !B0 : B0;
                        float lm = q0 ? lam[1] : lam[0];
                        lm = q1 ? lam[2] : lm;
                        lm = q2 ? lam[3] : lm;
                        lm = far ? lm45 : lm;
                        const float d = (c * 8 + e + u <= lane) ? (Gi - gjv[u]) : -INFINITY;
                        y[u] = s[e + u] * fexp(d) * lm;
                    }
                    x[e / 2] = pack_bf16(y[0], y[1]);
                    x[e / 2 + 1] = pack_bf16(y[2], y[3]);
                }
                umma::tmem_st4u(dst + rb * 16 + c * 4, x);
            }
            if (TEAMS == 1) zeros();                 // (P grows in the place of S behind the columns that are still to be read)
            umma::tmem_wait_st();
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(umma::smem_addr(p_full)) : "memory");
        }
    } else {
        if (TEAMS == 2) tco::regs_rows();
        // ---- slots -> output rows of every other head.  This thread: row `row`
        const int rb = warp & 3, row = rb * 32 + lane;
        int slot = 0;
        uint32_t ph = 0;
        for (int hh = team; hh < nh; hh += TEAMS) {
            const int h = h0 + hh;
            f32x2 o[32];
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = 0;
            for (int j = 0; j < njobs; ++j) {
                const float rs = j + 1 < njobs ? sCoef[(hh * (njobs - 1) + j) * 128 + row] : 1.f;
                const f32x2 rs2 = pack2(rs, rs);
                umma::mbar_wait(&slot_full[slot], ph, abort_flag);
                umma::fence_after_sync();
                constexpr int CW = TEAMS == 2 ? 32 : 16;         // columns at a time: as many as the registers hold
#pragma unroll
                for (int c = 0; c < 64; c += CW) {
                    float x[CW];
                    umma::tmem_ld(umma::tmem_addr(tSlot + slot * 64, warp, c), x);
                    if (c == 64 - CW) {
                        umma::fence_before_sync();
                        __syncwarp();
                        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(umma::smem_addr(&slot_empty[slot])) : "memory");
                    }
#pragma unroll
                    for (int e = 0; e < CW / 2; ++e) o[c / 2 + e] = fma2(rs2, pack2(x[2 * e], x[2 * e + 1]), o[c / 2 + e]);
                }
                if (++slot == NSLOT) {
                    slot = 0;
                    ph ^= 1;
                }
            }
            // The rows leave by way of shared memory in one bulk store: 32-byte stores of threads that own rows (a line per lane) kept the load / store
            // pipe, and with it every wait of the CTA, busy for 1 to 2 k cycles a head.
            const bool issuer = (tid & 127) == 0;
            if (RES) {
                umma::mbar_wait(x_full, (hh / TEAMS) & 1, abort_flag);
                const float dh = sC[hh * 4 + 2];
                const f32x2 dh2 = pack2(dh, dh);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 xr = *reinterpret_cast<const uint4*>(sX + umma::tile_offset(row, c * 8, tc::PT));
                    const uint32_t xw[4] = {xr.x, xr.y, xr.z, xr.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 of = unpack2(o[c * 4 + e]);
                        const uint32_t ob = pack_bf16(of.x, of.y);       // o rounded to bf16
                        const f32x2 ob2 = pack2(__uint_as_float(ob << 16), __uint_as_float(ob & 0xffff0000u));
                        const f32x2 xf2 = pack2(__uint_as_float(xw[e] << 16), __uint_as_float(xw[e] & 0xffff0000u));
                        if (RES == 3) {
                            const float2 m = unpack2(mul2(xf2, dh2));
                            const uint32_t mb = pack_bf16(m.x, m.y);
                            const float2 y = unpack2(ob2);
                            o[c * 4 + e] = pack2(y.x + __uint_as_float(mb << 16), y.y + __uint_as_float(mb & 0xffff0000u));
                        } else {
                            o[c * 4 + e] = fma2(xf2, dh2, ob2);
                        }
                    }
                }
            } else if (issuer) {
                tma::wait_group_read0();             // the rows of this team's previous head have left
            }
            if (RES == 0) {
                if (hh < TEAMS) umma::mbar_wait(barS, 0, abort_flag);      // (the place of k)
                team_barrier(team);
            }
            if (RES == 2) {
                // fp32 rows in two boxes of 32 columns, one behind the other in x's place (its words are all in use above)
#pragma unroll
                for (int bx = 0; bx < 2; ++bx) {
                    team_barrier(team);
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const float2 y0 = unpack2(o[bx * 16 + 2 * c]), y1 = unpack2(o[bx * 16 + 2 * c + 1]);
                        *reinterpret_cast<float4*>(sX + row * 128 + ((c ^ (row & 7)) << 4)) = make_float4(y0.x, y0.y, y1.x, y1.y);
                    }
                    umma::fence_async_smem();
                    team_barrier(team);
                    if (issuer) {
                        if (!*abort_flag) tma::store_seq_box(&p.tm_y, bx * 32, h, t0, b, sX);
                        tma::commit_group();
                        tma::wait_group_read0();
                    }
                }
            } else {
                // (every thread rewrites its own row)
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 y = unpack2(o[c * 4 + e]);
                        w[e] = pack_bf16(y.x, y.y);
                    }
                    *reinterpret_cast<uint4*>(sX + umma::tile_offset(row, c * 8, tc::PT)) = make_uint4(w[0], w[1], w[2], w[3]);
                }
                umma::fence_async_smem();
                team_barrier(team);
                if (issuer) {
                    if (!*abort_flag) tma::store_seq_box(&p.tm_y, 0, h, t0, b, sX);
                    tma::commit_group();
                    if (RES) tma::wait_group_read0();
                }
            }
            if (RES && issuer) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(umma::smem_addr(x_empty)) : "memory");
        }
        if ((tid & 127) == 0) tma::wait_group0();
    }
    umma::fence_before_sync();
    __syncthreads();                                 // everybody is done with tensor memory
    umma::fence_after_sync();
    if (warp == TM::MMA_WARP) {
        if (*abort_flag && lane == 0) atomicExch(p.err, 1);
        umma::tmem_dealloc(tbase, TM::TM_COLS);
    }
}

// ------------------------------------------------------------------------------------------
// Sequences of two to four pairs (T <= 512), whose calls lend no scratch for level states (256 bytes of workspace): one CTA per (batch, head) walks its pairs in
// order and keeps the states on chip, masters in registers in the tensor-memory readout layout (one state row per thread), bf16 copies as MN-major operands.
//   S = q k^T, T = q H_level, O = P v, KV = k^T (v * decay) per pair
// It stays for those calls: with scratch, states and outputs apart would be the faster way for most of them.  The forward call on this kernel / on those two, us
// (sequences x tokens x heads): 1 x 192 x 8 26.7 / 29.0, 4 x 256 x 32 29.8 / 33.0, 1 x 256 x 48 29.8 / 29.9; 1 x 384 x 48 34.8 / 32.2, 1 x 512 x 48 41.0 / 35.2,
// 8 x 512 x 24 62 / 45, 32 x 192 x 24 88 / 64, 32 x 512 x 24 158 / 114; with one head a group 16 x 512 x 24 94 / 94.
// ------------------------------------------------------------------------------------------
template <int MLOW>
struct FwdTcSmem {
    static constexpr int MP = MLOW - 1;              // pair levels kept on chip
    static constexpr uint32_t q_off = 0;
    static constexpr uint32_t v_off = q_off + tc::Q_BYTES;             // [2]
    static constexpr uint32_t k_off = v_off + 2 * tc::V_BYTES;         // [2]
    static constexpr uint32_t p_off = k_off + 2 * tc::Q_BYTES;
    static constexpr uint32_t vs_off = p_off + tc::PT * tc::PT * 2;
    static constexpr uint32_t h_off = vs_off + tc::V_BYTES;
    static constexpr uint32_t gp_off = h_off + (MP > 0 ? MP : 1) * tc::H_BYTES;   // float [2][3][128]: decay tables of this pair and the next
    static constexpr uint32_t lam_off = gp_off + 2 * 3 * 128 * 4;      // bf16 [128][L <= 32]
    static constexpr uint32_t bar_off = lam_off + 128 * (MAX_L + 2) * 2;   // 10 mbarriers + tmem slot + abort flag     // 4 mbarriers + tmem slot + abort flag
    static constexpr uint32_t total = bar_off + 128 + 1024;             // + slack for 1024-byte alignment
};

template <int MLOW, bool WHOLE, int RES>
__global__ void __launch_bounds__(tc::NTHREADS, 1) m2_one_segment_tc_kernel(const __grid_constant__ Mamba2Params p) {
    chain_wait();
    using SM = FwdTcSmem<MLOW>;
    constexpr int MP = SM::MP;
    constexpr int NLAM = 8 + (MP > 0 ? MP : 1);
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* sQ = smem + SM::q_off;            // single buffer, refilled as soon as S and T are done
    unsigned char* sV = smem + SM::v_off;            // [2]
    unsigned char* sK = smem + SM::k_off;            // [2]
    unsigned char* sP = smem + SM::p_off;
    unsigned char* sVs = smem + SM::vs_off;
    unsigned char* sH = smem + SM::h_off;
    float* sTab = reinterpret_cast<float*>(smem + SM::gp_off);     // [2][3][128]: per pair, G | Cf | Vf (see decay_tables)
    bf16* sLam = reinterpret_cast<bf16*>(smem + SM::lam_off);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::bar_off);     // MMA completion: S, T, O, KV
    uint64_t* full_q = bars + 4;                     // TMA completion: q tile
    uint64_t* full_kv = bars + 5;                    // [2] k and v tiles of a stage
    uint64_t* empty_q = bars + 7;                    // tensor core is done reading the q tile
    uint64_t* empty_kv = bars + 8;                   // [2] ... the k and v tiles of a stage
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + SM::bar_off + 80);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SM::bar_off + 88);
    static_assert(MP <= 2, "two tensor-memory slots for level reads");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.x % p.H, b = blockIdx.x / p.H;
    const int grp = h / (p.H / p.G);
    const int L = p.L;
    const int npairs = (p.NT + 1) / 2;
    const int res_n = RES == 1 ? p.res_T : p.res_n;  // (a layer's y has the tokens of x)

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < 10; ++i) umma::mbar_init(&bars[i], 1);
        umma::fence_mbar_init();
        *abort_flag = *p.err;                        // an earlier CTA gave up: do not pile on
    }
    __syncthreads();
    if (*abort_flag) return;                         // uniform: every thread reads the same shared word

    constexpr uint32_t ID_S = umma::idesc_bf16(128, 128, false, false);
    constexpr uint32_t ID_KM = umma::idesc_bf16(128, 64, false, true);
    constexpr uint32_t ID_MM = umma::idesc_bf16(128, 64, true, true);

    if (warp >= tc::MMA_WARP) {
        // ================= third warpgroup: one warp issues the tensor-core work =================
        RegisterSplit<56, 224>::release();
        if (warp == tc::MMA_WARP + 1) {
            // ---- TMA producer: one lane streams the tiles of the segment through the stages
            if (lane == 0) {
                for (int pl = 0; pl < npairs; ++pl) {
                    const int st = pl & 1, row0 = pl * tc::PT;
                    if (pl >= 2 && !umma::mbar_wait(&empty_kv[st], ((pl - 2) >> 1) & 1, abort_flag)) break;
                    tma::expect_tx(&full_kv[st], tc::Q_BYTES + tc::V_BYTES);
                    tma::load_seq_panel(sK + st * tc::Q_BYTES, &p.tm_k, 0, grp, row0, b, &full_kv[st]);
                    tma::load_seq_panel(sK + st * tc::Q_BYTES + tc::Q_BYTES / 2, &p.tm_k, 64, grp, row0, b, &full_kv[st]);
                    tma::load_seq_panel(sV + st * tc::V_BYTES, &p.tm_v, 0, h, row0, b, &full_kv[st]);
                    if (pl >= 1 && !umma::mbar_wait(empty_q, (pl - 1) & 1, abort_flag)) break;
                    tma::expect_tx(full_q, tc::Q_BYTES);
                    tma::load_seq_panel(sQ, &p.tm_q, 0, grp, row0, b, full_q);
                    tma::load_seq_panel(sQ + tc::Q_BYTES / 2, &p.tm_q, 64, grp, row0, b, full_q);
                }
            }
            return;
        }
        if (warp > tc::MMA_WARP) return;
        umma::tmem_alloc(tmem_slot, tc::TM_COLS);
        umma::fence_before_sync();
        bar_work();                                  // publishes the tensor-memory base address
        umma::fence_after_sync();
        const uint32_t tbase = *tmem_slot;
        for (int pl = 0; pl < npairs; ++pl) {
            const int st = pl & 1;
            const uint32_t aQ = umma::smem_addr(sQ), aK = umma::smem_addr(sK + st * tc::Q_BYTES);
            const uint32_t aV = umma::smem_addr(sV + st * tc::V_BYTES);
            // (no barrier here: the end-of-pair barrier of the previous pair is all the tensor core needs; the decay
            //  tables of this pair were written one pair ahead)
            if (lane == 0) {
                umma::mbar_wait(full_q, pl & 1, abort_flag);
                umma::mbar_wait(&full_kv[st], (pl >> 1) & 1, abort_flag);
                umma::gemm_kk<tc::PT, tc::PT, tc::KD>(tbase + tc::TM_S, aQ, aK, ID_S, false);
                umma::commit(&bars[0]);
                int slot = 0;
#pragma unroll
                for (int lv = 0; lv < MP; ++lv)
                    if ((pl >> lv) & 1) {
                        umma::gemm_km<tc::PT, tc::KD, tc::KD>(tbase + (slot == 0 ? tc::TM_T0 : tc::TM_T1), aQ,
                                                              umma::smem_addr(sH + lv * tc::H_BYTES), ID_KM, false);
                        ++slot;
                    }
                if (slot > 0) umma::commit(&bars[1]);
                umma::commit(empty_q);               // q tile may be overwritten once S and the level reads are done
            }
            __syncwarp();
            umma::fence_before_sync();
            bar_work();                              // barrier 2: P and Vs are written
            umma::fence_after_sync();
            if (lane == 0) {
                umma::gemm_km<tc::PT, tc::PT, tc::PT>(tbase + tc::TM_O, umma::smem_addr(sP), aV, ID_KM, false);
                umma::commit(&bars[2]);
                umma::gemm_mm<tc::PT, tc::PT, tc::PT>(tbase + tc::TM_KV, aK, umma::smem_addr(sVs), ID_MM, false);
                umma::commit(&bars[3]);
                umma::commit(&empty_kv[st]);         // k / v stage may be refilled
            }
            __syncwarp();
            umma::fence_before_sync();
            bar_work();                              // barrier 3: end of the pair
            umma::fence_after_sync();
            if (*abort_flag) break;
        }
        if (*abort_flag && lane == 0) atomicExch(p.err, 1);
        umma::fence_before_sync();
        bar_work();                                  // everybody is done with tensor memory
        umma::tmem_dealloc(tbase, tc::TM_COLS);
        return;
    }

    // ================= warps 0..7: loads, decay / mask / lambda, outputs, level states =================
    RegisterSplit<56, 224>::acquire();
    const int rb = warp & 3;                         // 32-row block of this thread's tensor-memory lane
    const int row = rb * 32 + lane;
    const int ch = warp >> 2;                        // column half handled by this thread

    // lambda rows of the pair (two threads per row, staged through shared memory) and raw g of the
    // pair (warps 0 and 1), fetched one pair ahead
    float g_n[4];
    constexpr int LAMR = (tc::PT * NLAM + 255) / 256;   // only the NLAM columns these kernels read are fetched
    uint32_t lam_r[LAMR];                            // one 32-bit register per 16-bit element
    uint32_t lam_rc[LAMR];                           // (row << 8) | column of each element, 0xffffffff = none
    const int NC = L < NLAM ? L : NLAM;             // columns of a lambda row that are fetched
#pragma unroll
    for (int i = 0; i < LAMR; ++i) {
        const int e = tid + i * 256;
        const int rr = e / NC, cc = e - rr * NC;
        lam_rc[i] = (rr < tc::PT) ? (uint32_t)((rr << 8) | cc) : 0xffffffffu;
    }
    auto fetch_small = [&](int pl) {
        const long t0 = (long)pl * tc::PT;
        const unsigned short* lp = reinterpret_cast<const unsigned short*>(p.l) + (((long)b * p.T + t0) * p.H + h) * L;
#pragma unroll
        for (int i = 0; i < LAMR; ++i)
            if (lam_rc[i] != 0xffffffffu)
                lam_r[i] = (WHOLE || t0 + (lam_rc[i] >> 8) < p.T) ? lp[(long)(lam_rc[i] >> 8) * p.H * L + (lam_rc[i] & 255)] : (unsigned short)0;
    };
    // raw g of a pair: one warp (the one that builds the decay tables), four consecutive tokens per lane
    auto fetch_g = [&](int pl) {
        const long t0 = (long)pl * tc::PT;
        const float* gp = p.g + ((long)b * p.T + t0 + 4 * lane) * p.H + h;
#pragma unroll
        for (int i = 0; i < 4; ++i) g_n[i] = (WHOLE || t0 + 4 * lane < p.T) ? gp[(long)i * p.H] : 0.f;
    };
    // Decay tables of pair `pl` from the g values in g_n, by one full warp: G (pair-wide inclusive cumulative sum),
    // Cf = exp(G[end of 32-block] - G[j]), Vf = exp(G[127] - G[j]); also the in-chunk cumulative sum to global memory.
    // Built one pair ahead into the other half of sTab, so that a pair starts without a barrier of its own.
    auto decay_tables = [&](int pl) {
        float* tG = sTab + (pl & 1) * 384;
        const long t0 = (long)pl * tc::PT;
        float gq[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) gq[i] = g_n[i];
        gq[1] += gq[0];
        gq[2] += gq[1];
        gq[3] += gq[2];
        float tot = gq[3];                           // inclusive scan of lane totals inside each chunk (16 lanes)
#pragma unroll
        for (int d = 1; d < 16; d <<= 1) {
            const float t = __shfl_up_sync(0xffffffffu, tot, d);
            if ((lane & 15) >= d) tot += t;
        }
        const float gla = __shfl_sync(0xffffffffu, tot, 15);        // end of the first chunk
        const float glb = __shfl_sync(0xffffffffu, tot, 31);        // end of the second chunk (in-chunk)
        const float glp = gla + glb;
        const float cbase = tot - gq[3];                            // in-chunk exclusive prefix of this lane
        const float pbase = cbase + (lane >= 16 ? gla : 0.f);       // pair-wide
        const float gend = __shfl_sync(0xffffffffu, tot, (lane & ~7) + 7) + (lane >= 16 ? gla : 0.f);
        float* gc = p.g_cum + ((long)b * p.T + t0 + 4 * lane) * p.H + h;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float G = pbase + gq[i];
            tG[4 * lane + i] = G;
            tG[128 + 4 * lane + i] = fexp(gend - G);
            tG[256 + 4 * lane + i] = fexp(glp - G);
            if (WHOLE || t0 + 4 * lane < p.T) gc[(long)i * p.H] = cbase + gq[i];
        }
    };
    constexpr int TABLE_WARP = 4;                    // lane quarter 0 (one 32 x 32 block of the S tile): the warp with slack
    auto store_lam = [&]() {
#pragma unroll
        for (int i = 0; i < LAMR; ++i)
            if (lam_rc[i] != 0xffffffffu)
                sLam[(lam_rc[i] >> 8) * tc::LAM_LD + (lam_rc[i] & 255)] = __ushort_as_bfloat16((unsigned short)lam_r[i]);
    };
    fetch_small(0);
    store_lam();
    if (warp == TABLE_WARP) {
        fetch_g(0);
        decay_tables(0);
        if (npairs > 1) fetch_g(1);
    }
    umma::fence_before_sync();
    bar_work();
    umma::fence_after_sync();
    const uint32_t tbase = *tmem_slot;

    float M[MP > 0 ? MP : 1][32];     // masters: row `row` of each low pair-level state, 32 columns
    float dsum[MP > 0 ? MP : 1];
#pragma unroll
    for (int i = 0; i < (MP > 0 ? MP : 1); ++i) dsum[i] = 0.f;
    uint32_t phS = 0, phT = 0, phO = 0, phKV = 0;

    for (int pl = 0; pl < npairs; ++pl) {
        const int st = pl & 1;
        const long t0 = (long)pl * tc::PT;
        const float* sGp = sTab + (pl & 1) * 384;    // tables of this pair (written while the previous pair ran)
        const float* sCf = sGp + 128;
        const float* sVf = sGp + 256;
        if (pl + 1 < npairs) fetch_small(pl + 1);
        // x rows of the pair into L2 (held in registers from here on they cost the products below more than they save)
        if (RES && ch == 0 && t0 + row < res_n)
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p.res_x + (((long)b * p.res_T + t0 + row) * p.H + h) * tc::VD));
        umma::mbar_wait(&full_kv[st], (pl >> 1) & 1, abort_flag);      // the v tile (read below with generic loads)
        int nread = 0;
#pragma unroll
        for (int lv = 0; lv < MP; ++lv) nread += (pl >> lv) & 1;
        const float Gi = sGp[row];
        const float glp = sGp[tc::PT - 1];
        // this row's lambda: levels 0..7 inside the pair, then the low pair levels
        float lam[NLAM];
#pragma unroll
        for (int i = 0; i < NLAM; ++i) lam[i] = (i < L) ? __bfloat162float(sLam[row * tc::LAM_LD + i]) : 0.f;

        // ---- Vs = v * exp(glp - G_j)   (same swizzled offsets as v)
        {
            const unsigned char* cV = sV + st * tc::V_BYTES;
#pragma unroll
            for (int i = tid; i < tc::PT * (tc::VD / 8); i += 256) {
                const int j = i / (tc::VD / 8), c = (i % (tc::VD / 8)) * 8;
                const float sc = sVf[j];
                const uint32_t off = umma::tile_offset(j, c, tc::PT);
                uint4 x = *reinterpret_cast<const uint4*>(cV + off);
                uint32_t* xw = reinterpret_cast<uint32_t*>(&x);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    __nv_bfloat162 v2 = *reinterpret_cast<__nv_bfloat162*>(&xw[e]);
                    xw[e] = pack_bf16(__bfloat162float(v2.x) * sc, __bfloat162float(v2.y) * sc);
                }
                *reinterpret_cast<uint4*>(sVs + off) = x;
            }
        }
        // ---- wait for S (and the level reads); the q tile is then free for the next pair
        umma::mbar_wait(&bars[0], phS, abort_flag);
        phS ^= 1;
        if (nread > 0) {
            umma::mbar_wait(&bars[1], phT, abort_flag);
            phT ^= 1;
        }
        umma::fence_after_sync();
        // ---- S -> P (bf16, K-major A operand of P v).  This thread: row `row`, and in every 32-column
        //      block jb <= rb the 16 columns [jb*32 + ch*16, +16)
        // blocks above the diagonal: zeros
#pragma unroll 1
        for (int jb = rb + 1; jb < 4; ++jb) {
            const int j0 = jb * 32 + ch * 16;
#pragma unroll
            for (int c = 0; c < 2; ++c)
                *reinterpret_cast<uint4*>(sP + umma::tile_offset(row, j0 + c * 8, tc::PT)) = make_uint4(0u, 0u, 0u, 0u);
        }
        // Blocks below the diagonal, four columns at a time in run-time loops (one short copy of the body instead of
        // four unrolled 16-column copies: measured faster in this kernel, where the phase has a single accumulator).
#pragma unroll 1
        for (int jb = 0; jb < rb; ++jb) {
            // one level per block, decay factorised through the block end
            const float lm = ((rb ^ jb) == 1) ? lam[6] : lam[7];
            const float rf = lm * fexp(Gi - sGp[jb * 32 + 31]);
#pragma unroll 1
            for (int cc = 0; cc < 4; ++cc) {
                const int j0 = jb * 32 + ch * 16 + cc * 4;
                float s[4];
                umma::tmem_ld4(umma::tmem_addr(tbase + tc::TM_S, warp, j0), s);
                const float4 cf = *reinterpret_cast<const float4*>(sCf + j0);
                *reinterpret_cast<uint2*>(sP + umma::tile_offset(row, j0, tc::PT)) =
                    make_uint2(pack_bf16(s[0] * rf * cf.x, s[1] * rf * cf.y), pack_bf16(s[2] * rf * cf.z, s[3] * rf * cf.w));
            }
        }
        // diagonal block: levels 0..5, causal mask folded into the exponent.  The level of (row, column) is the position of the
        // highest bit in which they differ: per bit, "differs" is the row's own bit or its complement, so lambda is picked by
        // selects on predicates instead of comparisons per element.
        const bool B0 = lane & 1, B1 = lane & 2, B2 = lane & 4, B3 = lane & 8;
        const bool hi = (((lane >> 4) & 1) != ch);
#pragma unroll 1
        for (int cc = 0; cc < 4; ++cc) {
            const int jc = ch * 16 + cc * 4;             // first of the four columns, inside the block
            const int j0 = rb * 32 + jc;
            float s[4];
            umma::tmem_ld4(umma::tmem_addr(tbase + tc::TM_S, warp, j0), s);
            const float4 gj = *reinterpret_cast<const float4*>(sGp + j0);
            const float gjv[4] = {gj.x, gj.y, gj.z, gj.w};
            const bool q2 = B2 != bool(cc & 1), q3 = B3 != bool(cc & 2);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int jj = jc + u;
                const bool q1 = (u & 2) ? !B1 : B1, q0 = (u & 1) ? !B0 : B0;
                float lm = q0 ? lam[1] : lam[0];
                lm = q1 ? lam[2] : lm;
                lm = q2 ? lam[3] : lm;
                lm = q3 ? lam[4] : lm;
                lm = hi ? lam[5] : lm;
                const float d = (jj <= lane) ? (Gi - gjv[u]) : -INFINITY;
                s[u] = s[u] * fexp(d) * lm;
            }
            *reinterpret_cast<uint2*>(sP + umma::tile_offset(row, j0, tc::PT)) = make_uint2(pack_bf16(s[0], s[1]), pack_bf16(s[2], s[3]));
        }
        if (warp == TABLE_WARP && pl + 1 < npairs) {
            decay_tables(pl + 1);
            if (pl + 2 < npairs) fetch_g(pl + 2);
        }
        umma::fence_async_smem();
        umma::fence_before_sync();
        bar_work();                                  // barrier 2
        umma::fence_after_sync();

        // ---- output row of this thread: columns ch*32 .. +31
        float o[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] = 0.f;
        uint4 xr[RES ? 4 : 1];
        if (RES) {
            const bf16* gx = p.res_x + (((long)b * p.res_T + t0) * p.H + h) * tc::VD + (tid & 7) * 8;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int rr = (tid >> 3) + u * 32;
                xr[u] = t0 + rr < res_n ? __ldg(reinterpret_cast<const uint4*>(gx + (long)rr * p.H * tc::VD)) : make_uint4(0, 0, 0, 0);
            }
        }
        if (nread > 0) {
            int slot = 0;
#pragma unroll
            for (int lv = 0; lv < MP; ++lv)
                if ((pl >> lv) & 1) {
                    float t[32];
                    umma::tmem_ld32(umma::tmem_addr(tbase + (slot == 0 ? tc::TM_T0 : tc::TM_T1), warp, ch * 32), t);
                    const float rs = lam[8 + lv] * fexp(Gi + dsum[lv]);
#pragma unroll
                    for (int e = 0; e < 32; ++e) o[e] += rs * t[e];
                    ++slot;
                }
        }
        {
            umma::mbar_wait(&bars[2], phO, abort_flag);
            phO ^= 1;
            umma::fence_after_sync();
            float t[32];
            umma::tmem_ld32(umma::tmem_addr(tbase + tc::TM_O, warp, ch * 32), t);
            // P v has completed, so the P tile is free: stage the bf16 output rows there and copy
            // them out with 8 lanes per 128-byte row (coalesced) instead of one row per lane
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint4 x;
                uint32_t* xw = reinterpret_cast<uint32_t*>(&x);
#pragma unroll
                for (int e = 0; e < 4; ++e) xw[e] = pack_bf16(o[c * 8 + e * 2] + t[c * 8 + e * 2], o[c * 8 + e * 2 + 1] + t[c * 8 + e * 2 + 1]);
                *reinterpret_cast<uint4*>(sP + umma::tile_offset(row, ch * 32 + c * 8, tc::PT)) = x;
            }
            asm volatile("bar.sync 2, 256;\n" ::: "memory");
            if (RES) {
                const float dh = load_param(p.res_D, h, RES == 2);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int rr = (tid >> 3) + u * 32, c = (tid & 7) * 8;
                    if (t0 + rr >= res_n) continue;
                    const uint4 ov = *reinterpret_cast<const uint4*>(sP + umma::tile_offset(rr, c, tc::PT));
                    const uint32_t ow[4] = {ov.x, ov.y, ov.z, ov.w}, xw[4] = {xr[u].x, xr[u].y, xr[u].z, xr[u].w};
                    float y[8];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 of = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ow[e]));
                        const float2 xf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xw[e]));
                        y[2 * e] = of.x + (RES == 3 ? round_bf16(xf.x * dh) : xf.x * dh);
                        y[2 * e + 1] = of.y + (RES == 3 ? round_bf16(xf.y * dh) : xf.y * dh);
                    }
                    const long at = (((long)b * p.res_T + t0 + rr) * p.H + h) * tc::VD + c;
                    if (RES == 2) {
                        uint32_t w[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(y[e]);
                        st_global_32B(reinterpret_cast<float*>(p.res_y) + at, w);
                    } else {
                        *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(p.res_y) + at) =
                            make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
                    }
                }
            }
            bf16* go = p.o + (((long)b * p.oT + t0) * p.H + h) * tc::VD;
#pragma unroll
            for (int i = RES ? tc::PT * 8 : tid; i < tc::PT * 8; i += 256) {
                const int rr = i >> 3, c = (i & 7) * 8;
                if (WHOLE || t0 + rr < p.T)
                    *reinterpret_cast<uint4*>(go + (long)rr * p.H * tc::VD + c) = *reinterpret_cast<const uint4*>(sP + umma::tile_offset(rr, c, tc::PT));
            }
        }
        // ---- pair summary and the Fenwick carry over pair levels (thread = state row `row`)
        umma::mbar_wait(&bars[3], phKV, abort_flag);
        phKV ^= 1;
        umma::fence_after_sync();
        if (MP > 0 && pl + 1 < npairs) {
            const int j = __ffs(~pl) - 1;
            if (j < MP) {
                float kv[32];
                umma::tmem_ld32(umma::tmem_addr(tbase + tc::TM_KV, warp, ch * 32), kv);
#pragma unroll
                for (int lv = 0; lv < MP; ++lv)
                    if (lv < j) {
                        const float dec = fexp(dsum[lv] + glp);
#pragma unroll
                        for (int e = 0; e < 32; ++e) kv[e] += dec * M[lv][e];
                    }
#pragma unroll
                for (int lv = 0; lv < MP; ++lv) {
                    if (lv == j) {
#pragma unroll
                        for (int e = 0; e < 32; ++e) M[lv][e] = kv[e];
                        unsigned char* dst = sH + lv * tc::H_BYTES;
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            *reinterpret_cast<uint4*>(dst + umma::tile_offset(row, ch * 32 + c * 8, tc::KD)) =
                                make_uint4(pack_bf16(kv[c * 8], kv[c * 8 + 1]), pack_bf16(kv[c * 8 + 2], kv[c * 8 + 3]),
                                           pack_bf16(kv[c * 8 + 4], kv[c * 8 + 5]), pack_bf16(kv[c * 8 + 6], kv[c * 8 + 7]));
                        dsum[lv] = 0.f;
                    } else {
                        dsum[lv] += glp;
                    }
                }
            } else {
#pragma unroll
                for (int lv = 0; lv < MP; ++lv) dsum[lv] += glp;
            }
        }
        if (pl + 1 < npairs) store_lam();            // every read of this pair's lambda is done (barrier 2)
        umma::fence_async_smem();
        umma::fence_before_sync();
        bar_work();                                  // barrier 3
        umma::fence_after_sync();
        if (*abort_flag) break;                      // uniform: read after the barrier
    }
    umma::fence_before_sync();
    bar_work();
}

template <int RES>
static int launch_one_segment(const Mamba2Params& p, cudaStream_t stream) {
    auto kern = mamba2_whole_pairs(p) ? m2_one_segment_tc_kernel<M2_MLOW, true, RES> : m2_one_segment_tc_kernel<M2_MLOW, false, RES>;
    const size_t sm = FwdTcSmem<M2_MLOW>::total;
    cudaError_t e = allow_smem(kern, sm);
    if (e != cudaSuccess) return (int)e;
    llattn::launch_chained(kern, p.B * p.H, tc::NTHREADS, sm, stream, p); LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int mamba2_fwd_one_segment_tc_launch(const Mamba2Params& p_in, cudaStream_t stream) {
    Mamba2Params p = p_in;
    int rc;
    if ((rc = tma::make_seq_map(&p.tm_q, p.q, p.B, p.T, p.G, p.K, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_k, p.k, p.B, p.T, p.G, p.K, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_v, p.v, p.B, p.T, p.H, p.V, tc::PT, 2)) != 0) return rc;
    if (!p.res_D) return launch_one_segment<0>(p, stream);
    if (p.res_f32) return launch_one_segment<2>(p, stream);
    return p.res_round ? launch_one_segment<3>(p, stream) : launch_one_segment<1>(p, stream);
}

// Heads per CTA of the output and gradient kernels: the fewest rounds of CTAs over the SMs, a CTA counted as its heads and two more (q, k, S, tables).  Many heads
// share S and the loads of q and k; few fill the chip when a call is small.  Two lies between what the kernels show: at B = 2, T = 16384, 32 heads a CTA of
// n heads takes 2.0 (n + 2.7) us of outputs (two teams), 5.0 (n + 1.3) of dq, 3.3 (n + 2.1) of dk and dv.  The rule against the best n of one to eight (outputs /
// dq / dkv, us): 1 x 1024 x 48 (sequences, tokens, heads) 12/22/17, none better; 1 x 4096 x 32 23/51/34, none; 2 x 4096 x 24 32/72/56, none;
// 4 x 2048 x 32, K = 64 36/83/63, none; 8 x 4096 x 24 six heads 109/244/188, eight 102/245/194; 1 x 65536 x 32, where L = 17 leaves six, 344/890/517.
int mamba2_heads_per_cta(const Mamba2Params& p, int sms) {
    int reads = 1;                                   // levels that a pair reads at most
    while ((p.NT + 1) / 2 > 1 << reads) ++reads;
    const int per_grp = p.H / p.G, most = min(min(min(tco::HC_MAX, tco::LAM_MAX / p.L), tco::COEF_MAX / reads), per_grp);
    const long pairs = (long)p.B * ((p.NT + 1) / 2) * p.G;
    int best = 1;
    long cost = 0;
    for (int hc = 1; hc <= most; ++hc) {
        const long ctas = pairs * ((per_grp + hc - 1) / hc), c = ((ctas + sms - 1) / sms) * (hc + 2);
        if (hc == 1 || c <= cost) {
            best = hc;
            cost = c;
        }
    }
    return best;
}

bool mamba2_cta_has_group(const Mamba2Params& p) {
    int dev = -1, sms = 0;
    return cudaGetDevice(&dev) == cudaSuccess && sm_count(&sms, dev) == cudaSuccess && mamba2_heads_per_cta(p, sms) >= p.H / p.G;
}

template <int KD, int RES, int TEAMS>
static int launch_out_teams(const Mamba2Params& p, cudaStream_t stream) {
    auto kern = m2_out_tc_kernel<KD, RES, TEAMS>;
    const size_t sm = OutTcSmem<KD, TEAMS>::total;
    cudaError_t e = allow_smem(kern, sm);
    if (e != cudaSuccess) return (int)e;
    const int per_grp = p.H / p.G;
    llattn::launch_chained(kern, p.B * ((p.NT + 1) / 2) * p.G * ((per_grp + p.hc - 1) / p.hc), tco::Teams<TEAMS>::NTHREADS, sm, stream, p); LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}
template <int KD, int RES>
static int launch_out(const Mamba2Params& p, cudaStream_t stream) {
    return p.hc == 1 ? launch_out_teams<KD, RES, 1>(p, stream) : launch_out_teams<KD, RES, 2>(p, stream);
}

template <int KD>
static int launch_out_for(const Mamba2Params& p, cudaStream_t stream) {
    if (!p.res_D) return launch_out<KD, 0>(p, stream);
    if (p.res_f32) return launch_out<KD, 2>(p, stream);
    return p.res_round ? launch_out<KD, 3>(p, stream) : launch_out<KD, 1>(p, stream);
}

int mamba2_out_tc_launch(const Mamba2Params& p_in, cudaStream_t stream) {
    Mamba2Params p = p_in;
    const long NP = (p.NT + 1) / 2, BH = (long)p.B * p.H;
    int rc, dev = -1, sms = 0;
    if ((rc = tma::make_seq_map(&p.tm_q, p.q, p.B, p.T, p.G, p.K, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_k, p.k, p.B, p.T, p.G, p.K, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_v, p.v, p.B, p.T, p.H, p.V, tc::PT, 2)) != 0) return rc;
    // y of a prompt has the tail's tokens as well; rows behind the whole chunks are not written here
    if (p.res_D) rc = tma::make_seq_map(&p.tm_y, p.res_y, p.B, p.res_n, p.H, p.V, tc::PT, p.res_f32 ? 4 : 2, p.res_T);
    else rc = tma::make_seq_map(&p.tm_y, p.o, p.B, p.T, p.H, p.V, tc::PT, 2, p.oT);
    if (rc != 0) return rc;
    if (p.res_D && (rc = tma::make_seq_map(&p.tm_x, p.res_x, p.B, p.res_T, p.H, p.V, tc::PT, 2)) != 0) return rc;
    if (NP > 1 && (rc = tma::make_panel_map(&p.tm_lo, p.lo_H, BH * NP * p.K, 1, p.V, p.K)) != 0) return rc;
    if (p.NS > 1 && (rc = tma::make_panel_map(&p.tm_h0, p.seg_H0, BH * p.NS * p.LH * p.K, 1, p.V, p.K)) != 0) return rc;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = sm_count(&sms, dev);
    if (e != cudaSuccess) return (int)e;
    p.hc = mamba2_heads_per_cta(p, sms);
    return p.K == 128 ? launch_out_for<128>(p, stream) : launch_out_for<64>(p, stream);
}

}  // namespace llattn
