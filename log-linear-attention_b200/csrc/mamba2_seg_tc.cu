// Level states of the log-linear Mamba-2 path and their gradients on tcgen05 / TMA (K = 64 or 128, V = 64, segments of 2^MLOW chunks = 2^(MLOW-1) pairs of
// 128 tokens): one CTA per (batch, head, segment) makes the states inside its segment and the segment's summary (forward), or what the readers in its
// segment send back to the states they read (backward).  Same mathematics as m2_seg_state_kernel (mamba2_fwd.cu) and m2_seg_dstate_kernel (mamba2_bwd.cu),
// which make the part of the segments' summaries.
#include "tc_common.cuh"

namespace llattn {

// cumulative decay from each pair's start, inclusive, of the chunks [0, 8) of segment r, a chunk per warp (zeros behind the sequence): sG[512]; sTot[8] the chunks'
__device__ __forceinline__ void segment_pair_sums(const Mamba2Params& p, int b, int h, int r, float* sG, float* sTot, int warp, int lane) {
    const int c = r * 8 + warp;
    float x0 = 0.f, x1 = 0.f;
    if (c < p.NT) {
        const float* gp = p.g + ((long)b * p.T + (long)c * CH) * p.H + h;
        x0 = gp[(long)(2 * lane) * p.H];
        x1 = gp[(long)(2 * lane + 1) * p.H];
    }
    warp_cumsum64(x0, x1, lane);
    const float tot = __shfl_sync(0xffffffffu, x1, 31);
    if (lane == 0) sTot[warp] = tot;
    bar_compute();
    const float before = (warp & 1) ? sTot[warp - 1] : 0.f;
    sG[warp * CH + 2 * lane] = x0 + before;
    sG[warp * CH + 2 * lane + 1] = x1 + before;
}
__device__ __forceinline__ void arrive_on(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(umma::smem_addr(bar)) : "memory");
}
// a half row of do (32 columns), times rs, into the same place of a tile
__device__ __forceinline__ void scaled_half_row(unsigned char* dst, const uint4 (&dox)[4], float rs, int row, int ch) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const uint32_t xw[4] = {dox[c].x, dox[c].y, dox[c].z, dox[c].w};
        uint32_t out[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) out[e] = pack_bf16(__uint_as_float(xw[e] << 16) * rs, __uint_as_float(xw[e] & 0xffff0000u) * rs);
        *reinterpret_cast<uint4*>(dst + umma::tile_offset(row, ch * 32 + c * 8, tc::PT)) = make_uint4(out[0], out[1], out[2], out[3]);
    }
}

// ------------------------------------------------------------------------------------------
// backward: what the readers of the high level states send back, dF[r][j] = sum over the pairs of segment r of q^T (do lambda_j exp(G)), G from the segment's
// start, for every set bit j of r: fp32 K x V summaries for the scan over segments.  One CTA per (batch, head, segment) and four set levels; a job is a level
// of a pair: a scaled copy of do in a ring of stages times q^T, accumulated in the level's tensor-memory slot.
// The kernel is latency throughout (16 % of the issue slots busy with one CTA per SM), so what a CTA holds is cut to let two share an SM: one tile of q, two
// copies, four slots: at B = 2, T = 16384, 32 heads 232 us with one CTA per SM, 140 with two.
// ------------------------------------------------------------------------------------------
namespace tcr {
constexpr int MAXLH = 4;                 // high levels of a CTA
constexpr int NST = 2, NTHREADS = 320, TMA_WARP = 9, TM_COLS = 256;
}
template <int MLOW>
struct ReadersTcSmem {
    static constexpr int SEG = 1 << MLOW;
    static constexpr uint32_t q_off = 0;                                   // 32 KB
    static constexpr uint32_t do_off = q_off + tc::Q_BYTES;                // [2] 16 KB
    static constexpr uint32_t st_off = do_off + 2 * tc::V_BYTES;           // [NST] 16 KB
    static constexpr uint32_t gs_off = st_off + tcr::NST * tc::V_BYTES;    // float [SEG * 64], [SEG]
    static constexpr uint32_t lam_off = gs_off + (SEG * 64 + SEG) * 4;     // bf16 [MAXLH][SEG * 64]
    static constexpr uint32_t bar_off = lam_off + tcr::MAXLH * SEG * 64 * 2;
    static constexpr uint32_t total = bar_off + 256 + 1024;
};

template <int MLOW>
__global__ void __launch_bounds__(tcr::NTHREADS, 2) m2_readers_tc_kernel(const __grid_constant__ Mamba2Params p) {
    chain_wait();
    using SM = ReadersTcSmem<MLOW>;
    constexpr int SEG = SM::SEG, SEGP = SEG / 2;
    static_assert(SEG == 8, "a chunk per warp");
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = umma::align_1024(smem_raw);
    unsigned char* sQ = smem + SM::q_off;
    unsigned char* sDO = smem + SM::do_off;
    unsigned char* sSt = smem + SM::st_off;
    float* sGs = reinterpret_cast<float*>(smem + SM::gs_off);
    float* sTot = sGs + SEG * 64;
    bf16* sLam = reinterpret_cast<bf16*>(smem + SM::lam_off);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::bar_off);
    uint64_t* full = bars + 0;       // [2] do of a pair
    uint64_t* full_q = bars + 2;
    uint64_t* empty = bars + 3;      // q and do of a pair (its products wait for every thread's copies of its do)
    uint64_t* done = bars + 4;
    uint64_t* st_full = bars + 5;    // [NST] 8: a scaled copy is written
    uint64_t* st_empty = bars + 5 + tcr::NST;
    constexpr int NBARS = 5 + 2 * tcr::NST;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + SM::bar_off + 200);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SM::bar_off + 208);
    static_assert(NBARS * 8 <= 200, "barriers");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int NP = (p.NT + 1) / 2;
    const int h = blockIdx.x % p.H;
    const int r = 1 + (blockIdx.x / p.H) % (p.NS - 1);
    const int b = (blockIdx.x / (p.H * (p.NS - 1))) % p.B, part = blockIdx.x / (p.H * (p.NS - 1) * p.B);
    const int grp = h / (p.H / p.G);
    const long bh = (long)b * p.H + h;
    const int npairs = min(SEGP, NP - r * SEGP);
    // this CTA's four of the segment's set high levels
    int himask = r;
    for (int i = 0; i < part * tcr::MAXLH; ++i) himask &= himask - 1;
    const int nl = min(__popc(himask), tcr::MAXLH);
    if (nl == 0) return;                     // (uniform)

    if (tid == tcr::TMA_WARP * 32) {
        for (int i = 0; i < NBARS; ++i) umma::mbar_init(&bars[i], i >= 5 && i < 5 + tcr::NST ? 8 : 1);
        umma::fence_mbar_init();
        *abort_flag = *p.err;
    }
    __syncthreads();
    if (*abort_flag) return;
    if (warp == tc::MMA_WARP) umma::tmem_alloc(tmem_slot, tcr::TM_COLS);
    if (warp < 8) {
        // lambda of the levels read
        unsigned short x[SEG * 64 * tcr::MAXLH / 256];
        int lev = himask;
        for (int i = 0; i < (tid & 3) && lev; ++i) lev &= lev - 1;
        const unsigned short* gl = reinterpret_cast<const unsigned short*>(p.l) + ((long)b * p.T * p.H + h) * p.L + INTRA_LEVELS + MLOW + __ffs(lev) - 1;
#pragma unroll
        for (int i = 0; i < SEG * 64 * tcr::MAXLH / 256; ++i) {
            const int t = r * SEG * 64 + (tid >> 2) + i * 64;
            x[i] = t < p.T && (tid & 3) < nl ? __ldg(gl + (long)t * p.H * p.L) : (unsigned short)0;
        }
#pragma unroll
        for (int i = 0; i < SEG * 64 * tcr::MAXLH / 256; ++i) sLam[(tid & 3) * SEG * 64 + (tid >> 2) + i * 64] = __ushort_as_bfloat16(x[i]);
        segment_pair_sums(p, b, h, r, sGs, sTot, warp, lane);
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tbase = *tmem_slot;

    if (warp == tcr::TMA_WARP) {
        if (lane == 0) {
            int pl = 0, nq = 0;
            for (; pl < npairs; ++pl) {
                const int st = pl & 1, row0 = (r * SEGP + pl) * tc::PT;
                // (its place: free since the q of the pair before was asked for)
                tma::expect_tx(&full[st], tc::V_BYTES);
                tma::load_seq_panel(sDO + st * tc::V_BYTES, &p.tm_do, 0, h, row0, b, &full[st]);
                if (pl >= 1 && !umma::mbar_wait(empty, (pl - 1) & 1, abort_flag)) {
                    ++pl;
                    break;
                }
                tma::expect_tx(full_q, tc::Q_BYTES);
                tma::load_seq_panel(sQ, &p.tm_q, 0, grp, row0, b, full_q);
                tma::load_seq_panel(sQ + tc::Q_BYTES / 2, &p.tm_q, 64, grp, row0, b, full_q);
                nq = pl + 1;
            }
            // every load is waited for by other warps, unless a wait gave up: nothing may still be on its way into shared memory when the CTA ends
            for (int i = max(0, pl - 2); i < pl; ++i) umma::mbar_wait(&full[i & 1], (i >> 1) & 1, 1u << 16);
            if (nq > 0) umma::mbar_wait(full_q, (nq - 1) & 1, 1u << 16);
        }
        __syncwarp();
    } else if (warp == tc::MMA_WARP) {
        // (the whole warp, see umma::elect_one)
        constexpr uint32_t ID_MM64 = umma::idesc_bf16(128, 64, true, true);
        const uint32_t lead = umma::elect_one();
        auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, umma::mbar_wait(bar, parity, abort_flag)); };
        int st = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int pl = 0; pl < npairs && ok; ++pl) {
            if (!(ok = wait(full_q, pl & 1))) break;
            const uint32_t aQ = umma::smem_addr(sQ);
            for (int i = 0; i < nl; ++i) {
                if (!(ok = wait(&st_full[st], ph))) break;
                umma::fence_after_sync();
                umma::gemm_mm_lead<tc::PT, tc::PT, tc::PT>(lead, tbase + i * 64, aQ, umma::smem_addr(sSt + st * tc::V_BYTES), ID_MM64, pl > 0);
                umma::commit_lead(lead, &st_empty[st]);
                if (++st == tcr::NST) {
                    st = 0;
                    ph ^= 1;
                }
            }
            umma::commit_lead(lead, empty);
        }
        umma::commit_lead(lead, done);
        if (!ok) umma::mbar_wait(done, 0, 1u << 16);     // gave up: no product may still read shared memory when the CTA ends
        __syncwarp();
    } else {
        const int rb = warp & 3, row = rb * 32 + lane, ch = warp >> 2;
        int st = 0;
        uint32_t ph = 1;
        float before = 0.f;                          // decay of the segment's pairs before this one
        for (int pl = 0; pl < npairs; ++pl) {
            const float ehi = fexp(sGs[pl * tc::PT + row] + before);
            before += sGs[pl * tc::PT + tc::PT - 1];
            umma::mbar_wait(&full[pl & 1], (pl >> 1) & 1, abort_flag);
            uint4 dox[4];
#pragma unroll
            for (int c = 0; c < 4; ++c)
                dox[c] = *reinterpret_cast<const uint4*>(sDO + (pl & 1) * tc::V_BYTES + umma::tile_offset(row, ch * 32 + c * 8, tc::PT));
            for (int i = 0; i < nl; ++i) {
                const float rs = __bfloat162float(sLam[i * SEG * 64 + pl * tc::PT + row]) * ehi;
                umma::mbar_wait(&st_empty[st], ph, abort_flag);
                scaled_half_row(sSt + st * tc::V_BYTES, dox, rs, row, ch);
                umma::fence_async_smem();
                __syncwarp();
                if (lane == 0) arrive_on(&st_full[st]);
                if (++st == tcr::NST) {
                    st = 0;
                    ph ^= 1;
                }
            }
        }
        umma::mbar_wait(done, 0, abort_flag);
        umma::fence_after_sync();
        // the summaries leave in boxes of 32 columns by way of the places of q and do in turn
        int bits = himask;
        for (int i = 0; i < nl; ++i) {
            const int j = __ffs(bits) - 1;
            bits &= bits - 1;
            float t[32];
            umma::tmem_ld32(umma::tmem_addr(tbase + i * 64, warp, ch * 32), t);
            unsigned char* place = (i & 1) ? sDO : sQ;
            unsigned char* box = place + ch * tc::V_BYTES;
            if (i >= 2) {
                if (tid == 0) tma::wait_group_read1();
                bar_compute();
            }
#pragma unroll
            for (int c = 0; c < 8; ++c)
                *reinterpret_cast<float4*>(box + row * 128 + ((c ^ (row & 7)) << 4)) = make_float4(t[c * 4], t[c * 4 + 1], t[c * 4 + 2], t[c * 4 + 3]);
            umma::fence_async_smem();
            bar_compute();
            if (tid == 0) {
                const int at = (int)(((bh * p.NS + r) * p.LH + j) * p.K);
                if (!*abort_flag)
                    for (int bx = 0; bx < 2; ++bx) tma::store_box(&p.tm_df, bx * 32, 0, at, place + bx * tc::V_BYTES);
                tma::commit_group();
            }
        }
        if (tid == 0) tma::wait_group0();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (warp == tc::MMA_WARP) {
        if (*abort_flag && lane == 0) atomicExch(p.err, 1);
        umma::tmem_dealloc(tbase, tcr::TM_COLS);
    }
}

// ------------------------------------------------------------------------------------------
// backward: the gradient of every pair's summary.  One CTA per (batch, head, segment) walks the segment's pairs from the last one on:
//   R_l  += q^T (do lambda_l exp(G))     what pair pl sends back to the pair levels that it reads (tensor memory, fp32)
//   A_pl  = what comes back to pair pl: from later segments, from the pairs of its segment that read a state with it    (one bf16 tile, fp32 until then)
//   Y     = <k^T (v exp(G_end - G)) of each chunk, A's parts>     contributor totals per level, from the fp32 parts
// Two CTAs per SM (238 -> 175 us at B = 2, T = 16384, 32 heads), with one tile of each operand and four 64-column slots each, as the steps of a CTA are a chain: R of pair level 1, of pair level 0, the
// summaries of a pair's two chunks.
// ------------------------------------------------------------------------------------------
namespace tca {
constexpr int NTHREADS = 320, TMA_WARP = 9, TM_COLS = 256;
constexpr int SLOT_R1 = 0, SLOT_R0 = 1, SLOT_KV = 2;
}
template <int MLOW>
struct AdjointTcSmem {
    static constexpr int SEG = 1 << MLOW;
    static constexpr uint32_t x_off = 0;                                   // 32 KB: q or k
    static constexpr uint32_t y_off = x_off + tc::Q_BYTES;                 // 16 KB: do or v (scaled in place)
    static constexpr uint32_t d_off = y_off + tc::V_BYTES;                 // 16 KB: a scaled copy of do, or A on its way out
    static constexpr uint32_t hi_off = d_off + tc::V_BYTES;                // 32 KB: fp32 gradient of the segment's summary, two boxes of 32 columns
    static constexpr uint32_t gs_off = hi_off + 2 * tc::V_BYTES;           // float [SEG * 64], [SEG]
    static constexpr uint32_t y_sum_off = gs_off + (SEG * 64 + SEG) * 4;   // float [8][8]
    static constexpr uint32_t lam_off = y_sum_off + 64 * 4;                // bf16 [2][SEG * 64]
    static constexpr uint32_t bar_off = lam_off + 2 * SEG * 64 * 2;
    static constexpr uint32_t total = bar_off + 128 + 1024;
};

template <int MLOW>
__global__ void __launch_bounds__(tca::NTHREADS, 2) m2_adjoint_tc_kernel(const __grid_constant__ Mamba2Params p) {
    chain_wait();
    using SM = AdjointTcSmem<MLOW>;
    constexpr int SEG = SM::SEG, SEGP = SEG / 2;
    static_assert(SEG == 8, "a chunk per warp, four pairs");
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = umma::align_1024(smem_raw);
    unsigned char* sX = smem + SM::x_off;
    unsigned char* sY = smem + SM::y_off;
    unsigned char* sD = smem + SM::d_off;
    unsigned char* sHi = smem + SM::hi_off;
    float* sGs = reinterpret_cast<float*>(smem + SM::gs_off);
    float* sTot = sGs + SEG * 64;
    float* sYs = reinterpret_cast<float*>(smem + SM::y_sum_off);
    bf16* sLam = reinterpret_cast<bf16*>(smem + SM::lam_off);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::bar_off);
    uint64_t* full = bars + 0;       // the step's tiles
    uint64_t* empty = bars + 1;
    uint64_t* hi_full = bars + 2;
    uint64_t* r_full = bars + 3;     // a reading step's products are complete
    uint64_t* scaled = bars + 4;     // 8: v is scaled
    uint64_t* kv_full = bars + 5;
    uint64_t* d_full = bars + 6;     // 8: a copy of do is written
    uint64_t* d_empty = bars + 7;
    constexpr int NBARS = 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + SM::bar_off + 96);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SM::bar_off + 104);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int NP = (p.NT + 1) / 2;
    const int h = blockIdx.x % p.H;
    const int r = (blockIdx.x / p.H) % p.NS;
    const int b = blockIdx.x / (p.H * p.NS);
    const int grp = h / (p.H / p.G);
    const long bh = (long)b * p.H + h;
    const int npairs = min(SEGP, NP - r * SEGP);
    const bool later = r < p.NS - 1;                 // later segments read this one's summary
    const int nc = later ? SEGP : npairs - 1;        // pairs that are read

    if (tid == tca::TMA_WARP * 32) {
        for (int i = 0; i < NBARS; ++i) umma::mbar_init(&bars[i], i == 4 || i == 6 ? 8 : 1);
        umma::fence_mbar_init();
        *abort_flag = *p.err;
    }
    __syncthreads();
    if (*abort_flag) return;
    if (warp == tc::MMA_WARP) umma::tmem_alloc(tmem_slot, tca::TM_COLS);
    if (warp < 8) {
        const unsigned short* gl = reinterpret_cast<const unsigned short*>(p.l) + ((long)b * p.T * p.H + h) * p.L + 8 + (tid & 1);
        unsigned short x[SEG * 64 * 2 / 256];
#pragma unroll
        for (int i = 0; i < SEG * 64 * 2 / 256; ++i) {
            const int t = r * SEG * 64 + (tid >> 1) + i * 128;
            x[i] = t < p.T && 8 + (tid & 1) < p.L ? __ldg(gl + (long)t * p.H * p.L) : (unsigned short)0;
        }
#pragma unroll
        for (int i = 0; i < SEG * 64 * 2 / 256; ++i) sLam[(tid & 1) * SEG * 64 + (tid >> 1) + i * 128] = __ushort_as_bfloat16(x[i]);
        segment_pair_sums(p, b, h, r, sGs, sTot, warp, lane);
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tbase = *tmem_slot;

    // steps, for every pair from the last one on: q, do if it reads (any but the segment's first), k, v if it is read
    if (warp == tca::TMA_WARP) {
        if (lane == 0) {
            if (later) {
                tma::expect_tx(hi_full, p.K * tc::VD * 4);
                for (int bx = 0; bx < 2; ++bx) tma::load_panel(sHi + bx * tc::V_BYTES, &p.tm_dh, bx * 32, 0, (int)((bh * p.NS + r) * p.K), hi_full);
            }
            int s = 0;
            bool ok = true;
            for (int pl = npairs - 1; pl >= 0 && ok; --pl)
                for (int own = 0; own < 2; ++own) {
                    if (own ? pl >= nc : pl == 0) continue;
                    if (s > 0 && !(ok = umma::mbar_wait(empty, (s - 1) & 1, abort_flag))) break;
                    const int row0 = (r * SEGP + pl) * tc::PT;
                    const CUtensorMap* x = own ? &p.tm_k : &p.tm_q;
                    tma::expect_tx(full, tc::Q_BYTES + tc::V_BYTES);
                    tma::load_seq_panel(sY, own ? &p.tm_v : &p.tm_do, 0, h, row0, b, full);
                    tma::load_seq_panel(sX, x, 0, grp, row0, b, full);
                    tma::load_seq_panel(sX + tc::Q_BYTES / 2, x, 64, grp, row0, b, full);
                    ++s;
                }
            // (see m2_readers_tc_kernel)
            if (s > 0) umma::mbar_wait(full, (s - 1) & 1, 1u << 16);
            if (later) umma::mbar_wait(hi_full, 0, 1u << 16);
        }
        __syncwarp();
    } else if (warp == tc::MMA_WARP) {
        constexpr uint32_t ID_MM64 = umma::idesc_bf16(128, 64, true, true);
        const uint32_t lead = umma::elect_one();
        const uint32_t aX = umma::smem_addr(sX), aY = umma::smem_addr(sY), aD = umma::smem_addr(sD);
        auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, umma::mbar_wait(bar, parity, abort_flag)); };
        int s = 0, nd = 0, ns = 0, nr = 0;
        bool ok = true;
        auto job = [&](int slot, bool accumulate) -> bool {
            if (!wait(d_full, nd & 1)) return false;
            ++nd;
            umma::fence_after_sync();
            umma::gemm_mm_lead<tc::PT, tc::PT, tc::PT>(lead, tbase + slot * 64, aX, aD, ID_MM64, accumulate);
            umma::commit_lead(lead, d_empty);
            return true;
        };
        for (int pl = npairs - 1; pl >= 0 && ok; --pl) {
            if (pl > 0) {
                if (!(ok = wait(full, s & 1))) break;
                if (pl >= 2) ok = job(tca::SLOT_R1, pl == 2 && npairs == 4);
                if (ok && (pl & 1)) ok = job(tca::SLOT_R0, false);
                umma::commit_lead(lead, empty);
                umma::commit_lead(lead, r_full);
                ++nr;
                ++s;
                if (!ok) break;
            }
            if (pl < nc) {
                if (!(ok = wait(scaled, ns & 1))) break;
                ++ns;
                umma::fence_after_sync();
                umma::gemm_mm_lead<tc::PT, tc::PT, 64>(lead, tbase + tca::SLOT_KV * 64, aX, aY, ID_MM64, false);                   // first chunk of the pair
                umma::gemm_mm_lead<tc::PT, tc::PT, 64>(lead, tbase + (tca::SLOT_KV + 1) * 64, aX + 64 * umma::ROW_BYTES, aY + 64 * umma::ROW_BYTES, ID_MM64, false);
                umma::commit_lead(lead, empty);
                umma::commit_lead(lead, kv_full);
                ++s;
            }
        }
        if (!ok) {
            // gave up: no product may still read shared memory when the CTA ends
            umma::commit_lead(lead, hi_full);
            umma::mbar_wait(hi_full, later ? 1 : 0, 1u << 16);
        }
        __syncwarp();
    } else {
        const int rb = warp & 3, row = rb * 32 + lane, ch = warp >> 2;
        const uint32_t tcol = umma::tmem_addr(tbase, warp, ch * 32);
        int s = 0, nd = 0, nkv = 0, nr = 0, seen = 0;        // steps, copies, summaries, reading steps so far; those whose products are known to be complete
        bool stored = false;
        float since = 0.f;                           // decay over the pairs behind this one
        if (later) umma::mbar_wait(hi_full, 0, abort_flag);
        for (int pl = npairs - 1; pl >= 0; --pl) {
            const float glp = sGs[pl * tc::PT + tc::PT - 1];
            if (pl > 0) {
                const float e = fexp(sGs[pl * tc::PT + row]);
                // (a pair that nobody reads has not waited for its own products: two completions later their parity would say that they never were)
                for (; seen < nr; ++seen) umma::mbar_wait(r_full, seen & 1, abort_flag);
                umma::mbar_wait(full, s & 1, abort_flag);
                ++s;
                uint4 dox[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) dox[c] = *reinterpret_cast<const uint4*>(sY + umma::tile_offset(row, ch * 32 + c * 8, tc::PT));
                auto copy = [&](float rs) {
                    if (nd > 0) umma::mbar_wait(d_empty, (nd - 1) & 1, abort_flag);
                    if (stored) {
                        if (tid == 0) tma::wait_group_read0();
                        bar_compute();
                        stored = false;
                    }
                    ++nd;
                    scaled_half_row(sD, dox, rs, row, ch);
                    umma::fence_async_smem();
                    umma::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) arrive_on(d_full);
                };
                if (pl >= 2) {
                    if (pl == 2 && npairs == 4) {
                        // what pair 3 sent back has decayed over pair 2, which adds to it
                        umma::fence_after_sync();
                        const float dec = fexp(glp);
#pragma unroll
                        for (int c = 0; c < 32; c += 16) {
                            float t[16];
                            umma::tmem_ld16(tcol + tca::SLOT_R1 * 64 + c, t);
#pragma unroll
                            for (int i = 0; i < 16; ++i) t[i] *= dec;
                            umma::tmem_st16(tcol + tca::SLOT_R1 * 64 + c, t);
                        }
                        umma::tmem_wait_st();
                    }
                    copy(__bfloat162float(sLam[SEG * 64 + pl * tc::PT + row]) * e);
                }
                if (pl & 1) copy(__bfloat162float(sLam[pl * tc::PT + row]) * e);
                ++nr;
            }
            if (pl < nc) {
                umma::mbar_wait(full, s & 1, abort_flag);
                ++s;
#pragma unroll
                for (int x = tid; x < tc::PT * (tc::VD / 8); x += 256) {
                    const int j = x / (tc::VD / 8), c = (x % (tc::VD / 8)) * 8;
                    const float sc = fexp(glp - sGs[pl * tc::PT + j]);
                    const f32x2 sc2 = pack2(sc, sc);
                    const uint32_t off = umma::tile_offset(j, c, tc::PT);
                    uint4 y = *reinterpret_cast<const uint4*>(sY + off);
                    uint32_t* yw = reinterpret_cast<uint32_t*>(&y);
#pragma unroll
                    for (int e = 0; e < 4; ++e) yw[e] = pack_bf16(mul2(bf16x2_f32x2(yw[e]), sc2));
                    *reinterpret_cast<uint4*>(sY + off) = y;
                }
                umma::fence_async_smem();
                umma::fence_before_sync();           // (the summaries that these products overwrite have been read)
                __syncwarp();
                if (lane == 0) arrive_on(scaled);
                const bool l0 = (pl & 1) == 0 && pl + 1 < npairs, l1 = pl < 2 && npairs > 2;
                // factors of the parts: later segments', pair level 0's, pair level 1's (decayed over pair 1 for pair 0)
                const float fh = later && row < p.K ? fexp(since) : 0.f, f1 = pl == 0 ? fexp(sGs[2 * tc::PT - 1]) : 1.f;
                for (; seen < nr; ++seen) umma::mbar_wait(r_full, seen & 1, abort_flag);
                if (nd > 0) umma::mbar_wait(d_empty, (nd - 1) & 1, abort_flag);
                if (stored) {
                    if (tid == 0) tma::wait_group_read0();
                    bar_compute();
                }
                umma::mbar_wait(kv_full, nkv & 1, abort_flag);
                ++nkv;
                umma::fence_after_sync();
                f32x2 y2[6];
#pragma unroll
                for (int u = 0; u < 6; ++u) y2[u] = 0;
                const f32x2 fh2 = pack2(fh, fh), f12 = pack2(f1, f1);
#pragma unroll 1
                for (int c = 0; c < 32; c += 8) {
                    // eight columns at a time: the state parts, then the two chunks' summaries against them
                    f32x2 hi2[4], r0[4], r1[4], sum[4];
                    const float4 ha = *reinterpret_cast<const float4*>(sHi + ch * tc::V_BYTES + row * 128 + (((c >> 2) ^ (row & 7)) << 4));
                    const float4 hb = *reinterpret_cast<const float4*>(sHi + ch * tc::V_BYTES + row * 128 + ((((c >> 2) + 1) ^ (row & 7)) << 4));
                    float ka[8], kb[8], ta[8], tb[8];
                    umma::tmem_ld8x4(tcol + tca::SLOT_KV * 64 + c, ka, tcol + (tca::SLOT_KV + 1) * 64 + c, kb, tcol + tca::SLOT_R0 * 64 + c, ta,
                                     tcol + tca::SLOT_R1 * 64 + c, tb);
                    hi2[0] = pack2(ha.x, ha.y); hi2[1] = pack2(ha.z, ha.w); hi2[2] = pack2(hb.x, hb.y); hi2[3] = pack2(hb.z, hb.w);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        // (what a slot holds before it was ever written, or a row of the summary that does not exist, is no number: selected away)
                        hi2[e] = fh != 0.f ? mul2(hi2[e], fh2) : 0;
                        r0[e] = l0 ? pack2(ta[2 * e], ta[2 * e + 1]) : 0;
                        r1[e] = l1 ? mul2(pack2(tb[2 * e], tb[2 * e + 1]), f12) : 0;
                        const f32x2 one = pack2(1.f, 1.f);
                        sum[e] = fma2(r1[e], one, fma2(r0[e], one, hi2[e]));
                        const f32x2 a2 = pack2(ka[2 * e], ka[2 * e + 1]), b2 = pack2(kb[2 * e], kb[2 * e + 1]);
                        y2[0] = fma2(a2, r0[e], y2[0]);
                        y2[1] = fma2(b2, r0[e], y2[1]);
                        y2[2] = fma2(a2, r1[e], y2[2]);
                        y2[3] = fma2(b2, r1[e], y2[3]);
                        y2[4] = fma2(a2, hi2[e], y2[4]);
                        y2[5] = fma2(b2, hi2[e], y2[5]);
                    }
                    *reinterpret_cast<uint4*>(sD + umma::tile_offset(row, ch * 32 + c, tc::PT)) =
                        make_uint4(pack_bf16(sum[0]), pack_bf16(sum[1]), pack_bf16(sum[2]), pack_bf16(sum[3]));
                }
#pragma unroll
                for (int u = 0; u < 6; ++u) {
                    float y = sum2(y2[u]);
#pragma unroll
                    for (int d = 16; d > 0; d >>= 1) y += __shfl_xor_sync(0xffffffffu, y, d);
                    if (lane == 0) sYs[warp * 8 + u] = y;
                }
                umma::fence_async_smem();
                umma::fence_before_sync();
                bar_compute();
                if (tid == 0) {
                    if (!*abort_flag) tma::store_box(&p.tm_lo_a, 0, 0, (int)((bh * NP + r * SEGP + pl) * p.K), sD);
                    tma::commit_group();
                }
                stored = true;
                if (tid >= 32 && tid < 38) {
                    // contributor totals per chunk: pair levels 0, 1, then the high ones together
                    const int u = tid - 32;
                    float t = 0.f;
#pragma unroll
                    for (int w = 0; w < 8; ++w) t += sYs[w * 8 + u];
                    const int c = (r * SEGP + pl) * 2 + (u & 1);
                    if (c < p.NT) p.Yc[(bh * p.NT + c) * (MLOW + 1) + 1 + (u >> 1)] = t;
                }
                bar_compute();                       // the totals have been read
            } else if (warp == 0 && lane < 6) {
                // the sequence's last pair: nobody reads it
                const int c = (NP - 1) * 2 + (lane & 1);
                if (c < p.NT) p.Yc[(bh * p.NT + c) * (MLOW + 1) + 1 + (lane >> 1)] = 0.f;
            }
            since += glp;
        }
        if (tid == 0) tma::wait_group0();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (warp == tc::MMA_WARP) {
        if (*abort_flag && lane == 0) atomicExch(p.err, 1);
        umma::tmem_dealloc(tbase, tca::TM_COLS);
    }
}

// ------------------------------------------------------------------------------------------
// forward: level states inside a segment and the segment's summary.  One CTA per (batch, head, segment) walks its pairs of 128 tokens:
//   KV_p = k^T (v exp(G_end of the pair - G))                  tensor core, one 64-column slot per pair
//   F    = KV_0; then KV_p + exp(glp_p) F                      fp32 in registers
// What later pairs of the segment read leaves as bf16 K x V tiles, in the place of the first pair that reads it: F after pair 0 (read by pair 1), F after
// pair 1 (pairs 2 and 3), KV_2 (pair 3); the first pair's place takes the decays glp; F after the last pair is the segment's summary, with its total decay, for the scan over segments.
// The last segment of a sequence has no summary and its last pair no reader.
// Two CTAs per SM: the products are short, a CTA mostly waits for its tiles (87 us at B = 2, T = 16384, 32 heads; the summaries alone took 100).
// ------------------------------------------------------------------------------------------
namespace tcst {
constexpr int NTHREADS = 320, TMA_WARP = 9, TM_COLS = 256;
}
template <int MLOW>
struct StateTcSmem {
    static constexpr int SEG = 1 << MLOW;
    static constexpr uint32_t k_off = 0;                                   // [2] 32 KB
    static constexpr uint32_t v_off = k_off + 2 * tc::Q_BYTES;             // [2] 16 KB, scaled in place
    static constexpr uint32_t gs_off = v_off + 2 * tc::V_BYTES;            // float [SEG * 64]: exp(G_end of the pair - G)
    static constexpr uint32_t tot_off = gs_off + SEG * 64 * 4;             // float [SEG]: chunk totals
    static constexpr uint32_t bar_off = tot_off + SEG * 4;
    static constexpr uint32_t total = bar_off + 160 + 1024;
};

template <int MLOW>
__global__ void __launch_bounds__(tcst::NTHREADS, 2) m2_state_tc_kernel(const __grid_constant__ Mamba2Params p) {
    chain_wait();
    using SM = StateTcSmem<MLOW>;
    constexpr int SEG = SM::SEG, SEGP = SEG / 2;
    static_assert(SEGP * 64 <= tcst::TM_COLS && SEG == 8, "a slot per pair, a chunk per warp");
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = umma::align_1024(smem_raw);
    unsigned char* sK = smem + SM::k_off;
    unsigned char* sV = smem + SM::v_off;
    float* sE = reinterpret_cast<float*>(smem + SM::gs_off);
    float* sTot = reinterpret_cast<float*>(smem + SM::tot_off);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::bar_off);
    uint64_t* full_kv = bars + 0;    // [2]
    uint64_t* empty_kv = bars + 2;   // [2] tensor core is done with the k / v stage
    uint64_t* scaled = bars + 4;     // [2] v is scaled (one arrival per element-wise warp)
    uint64_t* barKV = bars + 6;      // [SEGP] the pair's product is complete
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + SM::bar_off + 128);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SM::bar_off + 136);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int NP = (p.NT + 1) / 2, nseg = p.lo_H ? p.NS : p.NS - 1;
    const int h = blockIdx.x % p.H;
    const int r = (blockIdx.x / p.H) % nseg;
    const int b = blockIdx.x / (p.H * nseg);
    const int grp = h / (p.H / p.G);
    const long bh = (long)b * p.H + h;
    const bool last = r == p.NS - 1;
    const int np = last ? NP - r * SEGP - 1 : SEGP;          // pairs that this CTA sums
    if (np == 0) return;                                     // (uniform)

    if (tid == tcst::TMA_WARP * 32) {
        for (int i = 0; i < 6 + SEGP; ++i) umma::mbar_init(&bars[i], i == 4 || i == 5 ? 8 : 1);
        umma::fence_mbar_init();
        *abort_flag = *p.err;
    }
    __syncthreads();
    if (*abort_flag) return;
    if (warp == tc::MMA_WARP) umma::tmem_alloc(tmem_slot, tcst::TM_COLS);
    if (warp < 8) {
        // One chunk per warp, four consecutive tokens per lane (both half warps the same): its cumulative decay, summed in the order of the output kernel,
        // so that the sums of a forward call are the ones that a backward call finds in g_cum; then exp(G_end of the pair - G)
        float x[4] = {0.f, 0.f, 0.f, 0.f};
        if (warp < 2 * np) {
            const float* gp = (p.cum_in ? p.cum_in : p.g) + ((long)b * p.T + (long)(r * SEG + warp) * CH + 4 * (lane & 15)) * p.H + h;
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = __ldg(gp + (long)i * p.H);
        }
        if (!p.cum_in) {
            x[1] += x[0];
            x[2] += x[1];
            x[3] += x[2];
            float t = x[3];
#pragma unroll
            for (int d = 1; d < 16; d <<= 1) {
                const float u = __shfl_up_sync(0xffffffffu, t, d);
                if ((lane & 15) >= d) t += u;
            }
            const float base = t - x[3];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] += base;
        }
        const float tot = __shfl_sync(0xffffffffu, x[3], 15);
        if (lane == 0) sTot[warp] = tot;
        bar_compute();
        const float behind = tot + ((warp & 1) ? 0.f : sTot[warp + 1]);     // from the chunk's start to the pair's end
        if (lane < 16)
            *reinterpret_cast<float4*>(sE + warp * CH + 4 * lane) = make_float4(fexp(behind - x[0]), fexp(behind - x[1]), fexp(behind - x[2]), fexp(behind - x[3]));
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tbase = *tmem_slot;

    if (warp == tcst::TMA_WARP) {
        if (lane == 0) {
            const int brow = r * SEG * CH;
            int pl = 0;
            for (; pl < np; ++pl) {
                const int st = pl & 1, row0 = brow + pl * tc::PT;
                if (pl >= 2 && !umma::mbar_wait(&empty_kv[st], ((pl - 2) >> 1) & 1, abort_flag)) break;
                tma::expect_tx(&full_kv[st], tc::Q_BYTES + tc::V_BYTES);
                tma::load_seq_panel(sK + st * tc::Q_BYTES, &p.tm_k, 0, grp, row0, b, &full_kv[st]);
                tma::load_seq_panel(sK + st * tc::Q_BYTES + tc::Q_BYTES / 2, &p.tm_k, 64, grp, row0, b, &full_kv[st]);
                tma::load_seq_panel(sV + st * tc::V_BYTES, &p.tm_v, 0, h, row0, b, &full_kv[st]);
            }
            // gave up: nothing may still be on its way into shared memory when the CTA ends
            if (pl < np)
                for (int i = pl - 2; i < pl; ++i) umma::mbar_wait(&full_kv[i & 1], (i >> 1) & 1, 1u << 16);
        }
        __syncwarp();
    } else if (warp == tc::MMA_WARP) {
        if (lane == 0) {
            constexpr uint32_t ID_MM64 = umma::idesc_bf16(128, 64, true, true);
            int pl = 0;
            for (; pl < np; ++pl) {
                const int st = pl & 1;
                if (!umma::mbar_wait(&scaled[st], (pl >> 1) & 1, abort_flag)) break;
                umma::fence_after_sync();
                umma::gemm_mm<tc::PT, tc::PT, tc::PT>(tbase + pl * 64, umma::smem_addr(sK + st * tc::Q_BYTES), umma::smem_addr(sV + st * tc::V_BYTES),
                                                      ID_MM64, false);
                umma::commit(&empty_kv[st]);
                umma::commit(&barKV[pl]);
            }
            if (pl < np && pl > 0) umma::mbar_wait(&barKV[pl - 1], 0, 1u << 16);     // gave up: no product may still read shared memory
        }
        __syncwarp();
    } else {
        const int rb = warp & 3, row = rb * 32 + lane, ch = warp >> 2;
        auto scale_v = [&](int pl) {
            const int st = pl & 1;
            umma::mbar_wait(&full_kv[st], (pl >> 1) & 1, abort_flag);
            unsigned char* cV = sV + st * tc::V_BYTES;
#pragma unroll
            for (int i = tid; i < tc::PT * (tc::VD / 8); i += 256) {
                const int j = i / (tc::VD / 8), c = (i % (tc::VD / 8)) * 8;
                const float sc = sE[pl * tc::PT + j];
                const uint32_t off = umma::tile_offset(j, c, tc::PT);
                uint4 x = *reinterpret_cast<const uint4*>(cV + off);
                uint32_t* xw = reinterpret_cast<uint32_t*>(&x);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    __nv_bfloat162 v2 = *reinterpret_cast<__nv_bfloat162*>(&xw[e]);
                    xw[e] = pack_bf16(__bfloat162float(v2.x) * sc, __bfloat162float(v2.y) * sc);
                }
                *reinterpret_cast<uint4*>(cV + off) = x;
            }
            umma::fence_async_smem();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(umma::smem_addr(&scaled[st])) : "memory");
        };
        float f[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) f[e] = 0.f;
        float gend = 0.f;
        scale_v(0);
        for (int pl = 0; pl < np; ++pl) {
            if (pl + 1 < np) scale_v(pl + 1);
            umma::mbar_wait(&barKV[pl], 0, abort_flag);
            umma::fence_after_sync();
            float kv[32];
            umma::tmem_ld32(umma::tmem_addr(tbase + pl * 64, warp, ch * 32), kv);
            const float glp = sTot[2 * pl] + sTot[2 * pl + 1], dec = fexp(glp);
            gend += glp;
            if (tid == 0 && p.lo_H) reinterpret_cast<float*>(p.lo_H + (bh * NP + r * SEGP) * p.K * tc::VD)[pl] = glp;
#pragma unroll
            for (int e = 0; e < 32; ++e) f[e] = kv[e] + dec * f[e];
            if (p.lo_H && pl + 1 < SEGP && row < p.K) {
                bf16* dst = p.lo_H + ((bh * NP + r * SEGP + pl + 1) * p.K + row) * tc::VD + ch * 32;
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t w[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const int i = c * 16 + 2 * e;
                        w[e] = pl == 2 ? pack_bf16(kv[i], kv[i + 1]) : pack_bf16(f[i], f[i + 1]);
                    }
                    st_global_32B(dst + c * 16, w);
                }
            }
        }
        if (!last) {
            float* F = p.seg_F + (bh * p.NS + r) * p.K * tc::VD + row * tc::VD + ch * 32;
            if (row < p.K)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t w[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(f[c * 8 + e]);
                st_global_32B(F + c * 8, w);
            }
            if (tid == 0) p.seg_D[bh * p.NS + r] = gend;
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (warp == tc::MMA_WARP) {
        if (*abort_flag && lane == 0) atomicExch(p.err, 1);
        umma::tmem_dealloc(tbase, tcst::TM_COLS);
    }
}

int mamba2_state_tc_launch(const Mamba2Params& p_in, cudaStream_t stream) {
    Mamba2Params p = p_in;
    int rc;
    if ((rc = tma::make_seq_map(&p.tm_k, p.k, p.B, p.T, p.G, p.K, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_v, p.v, p.B, p.T, p.H, p.V, tc::PT, 2)) != 0) return rc;
    auto kern = m2_state_tc_kernel<M2_MLOW>;
    const size_t sm = StateTcSmem<M2_MLOW>::total;
    cudaError_t e = allow_smem(kern, sm);
    if (e != cudaSuccess) return (int)e;
    llattn::launch_chained(kern, p.B * p.H * (p.lo_H ? p.NS : p.NS - 1), tcst::NTHREADS, sm, stream, p); LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int mamba2_readers_tc_launch(const Mamba2Params& p_in, cudaStream_t stream) {
    Mamba2Params p = p_in;
    int rc;
    if ((rc = tma::make_seq_map(&p.tm_q, p.q, p.B, p.T, p.G, p.K, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_do, p.d_o, p.B, p.T, p.H, p.V, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_f32_box_map(&p.tm_df, p.seg_dF, (long)p.B * p.H * p.NS * p.LH * p.K, 1, p.V, p.K)) != 0) return rc;
    auto kern = m2_readers_tc_kernel<M2_MLOW>;
    const size_t sm = ReadersTcSmem<M2_MLOW>::total;
    cudaError_t e = allow_smem(kern, sm);
    if (e != cudaSuccess) return (int)e;
    // (CTAs for levels that a segment does not have end at once: 1 segment in 32 has five up to T = 16384)
    llattn::launch_chained(kern, p.B * p.H * (p.NS - 1) * ((p.LH + tcr::MAXLH - 1) / tcr::MAXLH), tcr::NTHREADS, sm, stream, p); LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

int mamba2_adjoint_tc_launch(const Mamba2Params& p_in, cudaStream_t stream) {
    Mamba2Params p = p_in;
    const long BH = (long)p.B * p.H;
    int rc;
    if ((rc = tma::make_seq_map(&p.tm_q, p.q, p.B, p.T, p.G, p.K, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_k, p.k, p.B, p.T, p.G, p.K, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_v, p.v, p.B, p.T, p.H, p.V, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_seq_map(&p.tm_do, p.d_o, p.B, p.T, p.H, p.V, tc::PT, 2)) != 0) return rc;
    if ((rc = tma::make_panel_map(&p.tm_lo_a, p.lo_A, BH * ((p.NT + 1) / 2) * p.K, 1, p.V, p.K)) != 0) return rc;
    if (p.NS > 1 && (rc = tma::make_f32_box_map(&p.tm_dh, p.seg_dHf, BH * p.NS * p.K, 1, p.V, p.K)) != 0) return rc;
    auto kern = m2_adjoint_tc_kernel<M2_MLOW>;
    const size_t sm = AdjointTcSmem<M2_MLOW>::total;
    cudaError_t e = allow_smem(kern, sm);
    if (e != cudaSuccess) return (int)e;
    llattn::launch_chained(kern, p.B * p.H * p.NS, tca::NTHREADS, sm, stream, p); LLATTN_LAUNCHED();
    return (int)cudaGetLastError();
}

}  // namespace llattn
