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
// start, for every set bit j of r: fp32 K x V summaries for the scan over segments.  One CTA per (batch, head, segment); a job is a level of a pair: a
// scaled copy of do in a ring of stages times q^T, accumulated in the level's tensor-memory slot.
// ------------------------------------------------------------------------------------------
namespace tcr {
constexpr int MAXLH = 5;                 // high levels of one launch
constexpr int NST = 6, NTHREADS = 320, TMA_WARP = 9;
}
template <int MLOW>
struct ReadersTcSmem {
    static constexpr int SEG = 1 << MLOW;
    static constexpr uint32_t q_off = 0;                                   // [2] 32 KB
    static constexpr uint32_t do_off = q_off + 2 * tc::Q_BYTES;            // [2] 16 KB
    static constexpr uint32_t st_off = do_off + 2 * tc::V_BYTES;           // [NST] 16 KB
    static constexpr uint32_t gs_off = st_off + tcr::NST * tc::V_BYTES;    // float [SEG * 64], [SEG]
    static constexpr uint32_t lam_off = gs_off + (SEG * 64 + SEG) * 4;     // bf16 [MAXLH][SEG * 64]
    static constexpr uint32_t bar_off = lam_off + tcr::MAXLH * SEG * 64 * 2;
    static constexpr uint32_t total = bar_off + 256 + 1024;
};

template <int MLOW>
__global__ void __launch_bounds__(tcr::NTHREADS, 1) m2_readers_tc_kernel(const __grid_constant__ Mamba2Params p) {
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
    uint64_t* full = bars + 0;       // [2] q and do of a pair
    uint64_t* empty = bars + 2;      // [2] (the products of a pair wait for every thread's copies of its do)
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
    const int b = blockIdx.x / (p.H * (p.NS - 1));
    const int grp = h / (p.H / p.G);
    const long bh = (long)b * p.H + h;
    const int npairs = min(SEGP, NP - r * SEGP);
    // set high levels of this segment inside this launch's window of five levels
    const int himask = (r >> p.lev_lo) & ((1 << tcr::MAXLH) - 1), nl = __popc(himask);
    if (nl == 0) return;                     // (uniform)

    if (tid == tcr::TMA_WARP * 32) {
        for (int i = 0; i < NBARS; ++i) umma::mbar_init(&bars[i], i >= 5 && i < 5 + tcr::NST ? 8 : 1);
        umma::fence_mbar_init();
        *abort_flag = *p.err;
    }
    __syncthreads();
    if (*abort_flag) return;
    if (warp == tc::MMA_WARP) umma::tmem_alloc(tmem_slot, tc::TM_COLS);
    if (warp < 8) {
        // lambda of the levels read
        const int base = INTRA_LEVELS + MLOW + p.lev_lo;
        for (int e = tid; e < SEG * 64 * tcr::MAXLH; e += 256) {
            const int i = e / tcr::MAXLH, j = e - i * tcr::MAXLH, t = r * SEG * 64 + i;
            if ((himask >> j) & 1) sLam[j * SEG * 64 + i] = t < p.T ? p.l[(((long)b * p.T + t) * p.H + h) * p.L + base + j] : __float2bfloat16(0.f);
        }
        segment_pair_sums(p, b, h, r, sGs, sTot, warp, lane);
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tbase = *tmem_slot;

    if (warp == tcr::TMA_WARP) {
        if (lane == 0) {
            int pl = 0;
            for (; pl < npairs; ++pl) {
                const int st = pl & 1, row0 = (r * SEGP + pl) * tc::PT;
                if (pl >= 2 && !umma::mbar_wait(&empty[st], ((pl - 2) >> 1) & 1, abort_flag)) break;
                tma::expect_tx(&full[st], tc::Q_BYTES + tc::V_BYTES);
                tma::load_seq_panel(sDO + st * tc::V_BYTES, &p.tm_do, 0, h, row0, b, &full[st]);
                tma::load_seq_panel(sQ + st * tc::Q_BYTES, &p.tm_q, 0, grp, row0, b, &full[st]);
                tma::load_seq_panel(sQ + st * tc::Q_BYTES + tc::Q_BYTES / 2, &p.tm_q, 64, grp, row0, b, &full[st]);
            }
            // every load is waited for by the MMA warp, unless a wait gave up: nothing may still be on its way into shared memory when the CTA ends
            for (int i = max(0, pl - 2); i < pl; ++i) umma::mbar_wait(&full[i & 1], (i >> 1) & 1, 1u << 16);
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
            if (!(ok = wait(&full[pl & 1], (pl >> 1) & 1))) break;
            const uint32_t aQ = umma::smem_addr(sQ + (pl & 1) * tc::Q_BYTES);
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
            umma::commit_lead(lead, &empty[pl & 1]);
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
            int bits = himask;
            for (int i = 0; i < nl; ++i) {
                const int j = __ffs(bits) - 1;
                bits &= bits - 1;
                const float rs = __bfloat162float(sLam[j * SEG * 64 + pl * tc::PT + row]) * ehi;
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
        // the summaries leave in boxes of 32 columns by way of the ring, two levels at a time
        int bits = himask;
        for (int i = 0; i < nl; ++i) {
            const int j = p.lev_lo + __ffs(bits) - 1;
            bits &= bits - 1;
            float t[32];
            umma::tmem_ld32(umma::tmem_addr(tbase + i * 64, warp, ch * 32), t);
            unsigned char* box = sSt + ((i & 1) * 2 + ch) * tc::V_BYTES;
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
                    for (int bx = 0; bx < 2; ++bx) tma::store_box(&p.tm_df, bx * 32, 0, at, sSt + ((i & 1) * 2 + bx) * tc::V_BYTES);
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
        umma::tmem_dealloc(tbase, tc::TM_COLS);
    }
}

// ------------------------------------------------------------------------------------------
// backward: the gradient of every pair's summary.  One CTA per (batch, head, segment):
//   R_pl,l = q^T (do lambda_l exp(G))        pairs 1.. of the segment, the pair levels that they read (tensor memory, fp32)
//   A_pl   = what comes back to pair pl: from later segments, from the pairs of its segment that read a state with it    (one bf16 tile, fp32 until then)
//   Y      = <k^T (v exp(G_end - G)) of each chunk, A's parts>     contributor totals per level, from the fp32 parts
// The segment's pairs are walked in order for R, then in reverse for A and Y.
// ------------------------------------------------------------------------------------------
namespace tca {
constexpr int NST = 3, NTHREADS = 320, TMA_WARP = 9;
constexpr int SLOT_KV = 4;               // slots 0..3: R of (pair 1, level 0), (2, 1), (3, 1), (3, 0); 4..7: two pairs of chunk summaries
}
template <int MLOW>
struct AdjointTcSmem {
    static constexpr int SEG = 1 << MLOW;
    static constexpr uint32_t x_off = 0;                                   // [2] 32 KB: q, then k
    static constexpr uint32_t y_off = x_off + 2 * tc::Q_BYTES;             // [2] 16 KB: do, then v (scaled in place)
    static constexpr uint32_t st_off = y_off + 2 * tc::V_BYTES;            // [NST] 16 KB: scaled copies of do, then A on its way out
    static constexpr uint32_t hi_off = st_off + tca::NST * tc::V_BYTES;    // 32 KB: fp32 gradient of the segment's summary, two boxes of 32 columns
    static constexpr uint32_t gs_off = hi_off + 2 * tc::V_BYTES;           // float [SEG * 64], [SEG]
    static constexpr uint32_t y_sum_off = gs_off + (SEG * 64 + SEG) * 4;   // float [8][8]
    static constexpr uint32_t lam_off = y_sum_off + 64 * 4;                // bf16 [2][SEG * 64]
    static constexpr uint32_t bar_off = lam_off + 2 * SEG * 64 * 2;
    static constexpr uint32_t total = bar_off + 256 + 1024;
};

template <int MLOW>
__global__ void __launch_bounds__(tca::NTHREADS, 1) m2_adjoint_tc_kernel(const __grid_constant__ Mamba2Params p) {
    chain_wait();
    using SM = AdjointTcSmem<MLOW>;
    constexpr int SEG = SM::SEG, SEGP = SEG / 2;
    static_assert(SEG == 8, "a chunk per warp, four pairs");
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = umma::align_1024(smem_raw);
    unsigned char* sX = smem + SM::x_off;
    unsigned char* sY = smem + SM::y_off;
    unsigned char* sSt = smem + SM::st_off;
    unsigned char* sHi = smem + SM::hi_off;
    float* sGs = reinterpret_cast<float*>(smem + SM::gs_off);
    float* sTot = sGs + SEG * 64;
    float* sYs = reinterpret_cast<float*>(smem + SM::y_sum_off);
    bf16* sLam = reinterpret_cast<bf16*>(smem + SM::lam_off);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::bar_off);
    uint64_t* full = bars + 0;       // [2]
    uint64_t* empty = bars + 2;      // [2]
    uint64_t* hi_full = bars + 4;
    uint64_t* r_full = bars + 5;     // every R is complete
    uint64_t* scaled = bars + 6;     // [2] 8: v is scaled
    uint64_t* kv_full = bars + 8;    // [2]
    uint64_t* st_full = bars + 10;   // [NST] 8
    uint64_t* st_empty = bars + 10 + tca::NST;
    constexpr int NBARS = 10 + 2 * tca::NST;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + SM::bar_off + 200);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SM::bar_off + 208);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int NP = (p.NT + 1) / 2;
    const int h = blockIdx.x % p.H;
    const int r = (blockIdx.x / p.H) % p.NS;
    const int b = blockIdx.x / (p.H * p.NS);
    const int grp = h / (p.H / p.G);
    const long bh = (long)b * p.H + h;
    const int npairs = min(SEGP, NP - r * SEGP);
    const bool later = r < p.NS - 1;                 // later segments read this one's summary
    const int nr = npairs - 1, nc = later ? SEGP : npairs - 1;      // pairs that read, pairs that are read

    if (tid == tca::TMA_WARP * 32) {
        for (int i = 0; i < NBARS; ++i) umma::mbar_init(&bars[i], i == 6 || i == 7 || (i >= 10 && i < 10 + tca::NST) ? 8 : 1);
        umma::fence_mbar_init();
        *abort_flag = *p.err;
    }
    __syncthreads();
    if (*abort_flag) return;
    if (warp == tc::MMA_WARP) umma::tmem_alloc(tmem_slot, tc::TM_COLS);
    if (warp < 8) {
        for (int e = tid; e < SEG * 64 * 2; e += 256) {
            const int i = e >> 1, j = e & 1, t = r * SEG * 64 + i;
            sLam[j * SEG * 64 + i] = t < p.T && 8 + j < p.L ? p.l[(((long)b * p.T + t) * p.H + h) * p.L + 8 + j] : __float2bfloat16(0.f);
        }
        segment_pair_sums(p, b, h, r, sGs, sTot, warp, lane);
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tbase = *tmem_slot;

    // steps: q, do of the pairs 1..nr, then k, v of the pairs nc - 1..0
    if (warp == tca::TMA_WARP) {
        if (lane == 0) {
            if (later) {
                tma::expect_tx(hi_full, p.K * tc::VD * 4);
                for (int bx = 0; bx < 2; ++bx) tma::load_panel(sHi + bx * tc::V_BYTES, &p.tm_dh, bx * 32, 0, (int)((bh * p.NS + r) * p.K), hi_full);
            }
            int s = 0;
            for (; s < nr + nc; ++s) {
                const int st = s & 1, pl = s < nr ? s + 1 : nc - 1 - (s - nr), row0 = (r * SEGP + pl) * tc::PT;
                if (s >= 2 && !umma::mbar_wait(&empty[st], ((s - 2) >> 1) & 1, abort_flag)) break;
                tma::expect_tx(&full[st], tc::Q_BYTES + tc::V_BYTES);
                tma::load_seq_panel(sY + st * tc::V_BYTES, s < nr ? &p.tm_do : &p.tm_v, 0, h, row0, b, &full[st]);
                tma::load_seq_panel(sX + st * tc::Q_BYTES, s < nr ? &p.tm_q : &p.tm_k, 0, grp, row0, b, &full[st]);
                tma::load_seq_panel(sX + st * tc::Q_BYTES + tc::Q_BYTES / 2, s < nr ? &p.tm_q : &p.tm_k, 64, grp, row0, b, &full[st]);
            }
            // (see m2_readers_tc_kernel)
            for (int i = max(0, s - 2); i < s; ++i) umma::mbar_wait(&full[i & 1], (i >> 1) & 1, 1u << 16);
            if (later) umma::mbar_wait(hi_full, 0, 1u << 16);
        }
        __syncwarp();
    } else if (warp == tc::MMA_WARP) {
        constexpr uint32_t ID_MM64 = umma::idesc_bf16(128, 64, true, true);
        const uint32_t lead = umma::elect_one();
        auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, umma::mbar_wait(bar, parity, abort_flag)); };
        int st = 0, s = 0;
        uint32_t ph = 0;
        bool ok = true;
        auto job = [&](uint32_t aQ, int slot) -> bool {
            if (!wait(&st_full[st], ph)) return false;
            umma::fence_after_sync();
            umma::gemm_mm_lead<tc::PT, tc::PT, tc::PT>(lead, tbase + slot * 64, aQ, umma::smem_addr(sSt + st * tc::V_BYTES), ID_MM64, false);
            umma::commit_lead(lead, &st_empty[st]);
            if (++st == tca::NST) {
                st = 0;
                ph ^= 1;
            }
            return true;
        };
        for (; s < nr && ok; ++s) {
            const int pl = s + 1;
            if (!(ok = wait(&full[s & 1], (s >> 1) & 1))) break;
            const uint32_t aQ = umma::smem_addr(sX + (s & 1) * tc::Q_BYTES);
            if (pl & 1) ok = job(aQ, pl == 1 ? 0 : 3);
            if (ok && pl >= 2) ok = job(aQ, pl - 1);
            umma::commit_lead(lead, &empty[s & 1]);
        }
        umma::commit_lead(lead, r_full);
        for (; s < nr + nc && ok; ++s) {
            const int i = s - nr;
            if (!(ok = wait(&scaled[i & 1], (i >> 1) & 1))) break;
            umma::fence_after_sync();
            const uint32_t aK = umma::smem_addr(sX + (s & 1) * tc::Q_BYTES), aV = umma::smem_addr(sY + (s & 1) * tc::V_BYTES);
            const uint32_t d = tbase + (tca::SLOT_KV + (i & 1) * 2) * 64;
            umma::gemm_mm_lead<tc::PT, tc::PT, 64>(lead, d, aK, aV, ID_MM64, false);                                           // first chunk of the pair
            umma::gemm_mm_lead<tc::PT, tc::PT, 64>(lead, d + 64, aK + 64 * umma::ROW_BYTES, aV + 64 * umma::ROW_BYTES, ID_MM64, false);
            umma::commit_lead(lead, &empty[s & 1]);
            umma::commit_lead(lead, &kv_full[i & 1]);
        }
        if (!ok) umma::mbar_wait(r_full, 0, 1u << 16);   // gave up: no product may still read shared memory when the CTA ends (the later ones are short)
        __syncwarp();
    } else {
        const int rb = warp & 3, row = rb * 32 + lane, ch = warp >> 2;
        {
            int st = 0;
            uint32_t ph = 1;
            auto copy = [&](const uint4 (&dox)[4], float rs) {
                umma::mbar_wait(&st_empty[st], ph, abort_flag);
                scaled_half_row(sSt + st * tc::V_BYTES, dox, rs, row, ch);
                umma::fence_async_smem();
                __syncwarp();
                if (lane == 0) arrive_on(&st_full[st]);
                if (++st == tca::NST) {
                    st = 0;
                    ph ^= 1;
                }
            };
            for (int s = 0; s < nr; ++s) {
                const int pl = s + 1;
                const float e = fexp(sGs[pl * tc::PT + row]);
                umma::mbar_wait(&full[s & 1], (s >> 1) & 1, abort_flag);
                uint4 dox[4];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    dox[c] = *reinterpret_cast<const uint4*>(sY + (s & 1) * tc::V_BYTES + umma::tile_offset(row, ch * 32 + c * 8, tc::PT));
                if (pl & 1) copy(dox, __bfloat162float(sLam[pl * tc::PT + row]) * e);
                if (pl >= 2) copy(dox, __bfloat162float(sLam[SEG * 64 + pl * tc::PT + row]) * e);
            }
        }
        auto scale_v = [&](int i) {
            const int s = nr + i, pl = nc - 1 - i;
            umma::mbar_wait(&full[s & 1], (s >> 1) & 1, abort_flag);
            unsigned char* cV = sY + (s & 1) * tc::V_BYTES;
            const float glp = sGs[pl * tc::PT + tc::PT - 1];
#pragma unroll
            for (int x = tid; x < tc::PT * (tc::VD / 8); x += 256) {
                const int j = x / (tc::VD / 8), c = (x % (tc::VD / 8)) * 8;
                const float sc = fexp(glp - sGs[pl * tc::PT + j]);
                const uint32_t off = umma::tile_offset(j, c, tc::PT);
                uint4 y = *reinterpret_cast<const uint4*>(cV + off);
                uint32_t* yw = reinterpret_cast<uint32_t*>(&y);
#pragma unroll
                for (int e = 0; e < 4; ++e) yw[e] = pack_bf16(__uint_as_float(yw[e] << 16) * sc, __uint_as_float(yw[e] & 0xffff0000u) * sc);
                *reinterpret_cast<uint4*>(cV + off) = y;
            }
            umma::fence_async_smem();
            umma::fence_before_sync();               // (the chunk summaries that these products overwrite have been read)
            __syncwarp();
            if (lane == 0) arrive_on(&scaled[i & 1]);
        };
        // R0 (level 0, for even pairs), R1 (level 1), the segment's: this thread's 32 columns of state row `row`
        float R0[32], R1[32], Hi[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) R0[e] = R1[e] = Hi[e] = 0.f;
        if (nc > 0) scale_v(0);
        if (later) {
            umma::mbar_wait(hi_full, 0, abort_flag);
            if (row < p.K)
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float4 x = *reinterpret_cast<const float4*>(sHi + ch * tc::V_BYTES + row * 128 + ((c ^ (row & 7)) << 4));
                Hi[c * 4] = x.x; Hi[c * 4 + 1] = x.y; Hi[c * 4 + 2] = x.z; Hi[c * 4 + 3] = x.w;
            }
        }
        umma::mbar_wait(r_full, 0, abort_flag);
        umma::fence_after_sync();
        // (what pair 2 or pair 1 finds where the walk starts there, at the end of a sequence)
        if (nc == 3 || nc == 2) umma::tmem_ld32(umma::tmem_addr(tbase + (nc - 1) * 64, warp, ch * 32), R1);
        for (int i = 0; i < nc; ++i) {
            const int pl = nc - 1 - i;
            if (i + 1 < nc) scale_v(i + 1);
            const bool l0 = (pl & 1) == 0 && pl + 1 < npairs, l1 = pl < 2 && npairs > 2;
            if (l0) umma::tmem_ld32(umma::tmem_addr(tbase + (pl == 0 ? 0 : 3) * 64, warp, ch * 32), R0);
            float ka[32], kb[32];
            umma::mbar_wait(&kv_full[i & 1], (i >> 1) & 1, abort_flag);
            umma::fence_after_sync();
            umma::tmem_ld32(umma::tmem_addr(tbase + (tca::SLOT_KV + (i & 1) * 2) * 64, warp, ch * 32), ka);
            umma::tmem_ld32(umma::tmem_addr(tbase + (tca::SLOT_KV + (i & 1) * 2 + 1) * 64, warp, ch * 32), kb);
            uint32_t pk[16];
            float y[6];
#pragma unroll
            for (int u = 0; u < 6; ++u) y[u] = 0.f;
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
                float x0 = Hi[e], x1 = Hi[e + 1];
                y[4] += ka[e] * x0 + ka[e + 1] * x1;
                y[5] += kb[e] * x0 + kb[e + 1] * x1;
                if (l0) {
                    y[0] += ka[e] * R0[e] + ka[e + 1] * R0[e + 1];
                    y[1] += kb[e] * R0[e] + kb[e + 1] * R0[e + 1];
                    x0 += R0[e];
                    x1 += R0[e + 1];
                }
                if (l1) {
                    y[2] += ka[e] * R1[e] + ka[e + 1] * R1[e + 1];
                    y[3] += kb[e] * R1[e] + kb[e + 1] * R1[e + 1];
                    x0 += R1[e];
                    x1 += R1[e + 1];
                }
                pk[e >> 1] = pack_bf16(x0, x1);
            }
#pragma unroll
            for (int u = 0; u < 6; ++u) {
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) y[u] += __shfl_xor_sync(0xffffffffu, y[u], d);
                if (lane == 0) sYs[warp * 8 + u] = y[u];
            }
            unsigned char* out = sSt + (i % tca::NST) * tc::V_BYTES;
            if (i >= tca::NST) {
                if (tid == 0) tma::wait_group_read<tca::NST - 1>();
                bar_compute();
            }
#pragma unroll
            for (int c = 0; c < 4; ++c)
                *reinterpret_cast<uint4*>(out + umma::tile_offset(row, ch * 32 + c * 8, p.K)) = make_uint4(pk[c * 4], pk[c * 4 + 1], pk[c * 4 + 2], pk[c * 4 + 3]);
            umma::fence_async_smem();
            bar_compute();
            if (tid == 0) {
                if (!*abort_flag) tma::store_box(&p.tm_lo_a, 0, 0, (int)((bh * NP + r * SEGP + pl) * p.K), out);
                tma::commit_group();
            }
            if (tid >= 32 && tid < 38) {
                // contributor totals per chunk: pair levels 0, 1, then the high ones together
                const int u = tid - 32;
                float t = 0.f;
#pragma unroll
                for (int w = 0; w < 8; ++w) t += sYs[w * 8 + u];
                const int c = (r * SEGP + pl) * 2 + (u & 1);
                if (c < p.NT) p.Yc[(bh * p.NT + c) * (MLOW + 1) + 1 + (u >> 1)] = t;
            }
            // one pair further back: what the later ones send has decayed over this one, which adds what it reads itself
            const float dec = fexp(sGs[pl * tc::PT + tc::PT - 1]);
#pragma unroll
            for (int e = 0; e < 32; ++e) {
                Hi[e] *= dec;
                R1[e] *= dec;
            }
            if (pl >= 2) {
                float t[32];
                umma::tmem_ld32(umma::tmem_addr(tbase + (pl - 1) * 64, warp, ch * 32), t);
#pragma unroll
                for (int e = 0; e < 32; ++e) R1[e] += t[e];
            }
            bar_compute();                           // the totals have been read
        }
        if (nc < npairs && warp == 0 && lane < 6) {
            // the sequence's last pair: nobody reads it
            const int c = (NP - 1) * 2 + (lane & 1);
            if (c < p.NT) p.Yc[(bh * p.NT + c) * (MLOW + 1) + 1 + (lane >> 1)] = 0.f;
        }
        if (tid == 0) tma::wait_group0();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (warp == tc::MMA_WARP) {
        if (*abort_flag && lane == 0) atomicExch(p.err, 1);
        umma::tmem_dealloc(tbase, tc::TM_COLS);
    }
}

// ------------------------------------------------------------------------------------------
// forward: level states inside a segment and the segment's summary.  One CTA per (batch, head, segment) walks its pairs of 128 tokens:
//   KV_p = k^T (v exp(G_end of the pair - G))                  tensor core, one 64-column slot per pair
//   F    = KV_0; then KV_p + exp(glp_p) F                      fp32 in registers
// What later pairs of the segment read leaves as bf16 K x V tiles, in the place of the first pair that reads it: F after pair 0 (read by pair 1), F after
// pair 1 (pairs 2 and 3), KV_2 (pair 3); the first pair's place takes the decays glp; F after the last pair is the segment's summary, with its total decay, for the scan over segments.
// The last segment of a sequence has no summary and its last pair no reader.
// Two CTAs per SM: the products are short, a CTA mostly waits for its tiles.
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
    // one launch per window of five segment levels (a single one up to T = 16384); their outputs are disjoint
    for (p.lev_lo = 0; p.lev_lo < p.LH; p.lev_lo += tcr::MAXLH) {
        llattn::launch_chained(kern, p.B * p.H * (p.NS - 1), tcr::NTHREADS, sm, stream, p); LLATTN_LAUNCHED();
    }
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
