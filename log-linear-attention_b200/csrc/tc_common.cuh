// Pieces shared by the tcgen05 kernels of the log-linear Mamba-2 path: tile geometry, warp roles,
// CTA barriers, optional phase timing.
#pragma once
#include "llattn_common.cuh"
#include "llattn_mamba2.h"
#include "tma.cuh"
#include "umma.cuh"

namespace llattn {

// Optional phase timing for tuning (build with -DLLATTN_STAMPS): three threads of one CTA record
// clock64() at fixed points of one pair; a function beside the kernels copies the table to the host.
#ifdef LLATTN_STAMPS
static __device__ long long g_stamps[3][32];
#define STAMP()                                                             \
    do {                                                                    \
        if (stamp_slot >= 0 && nstamp < 32) g_stamps[stamp_slot][nstamp++] = clock64(); \
    } while (0)
#define STAMPR()                                                            \
    do {                                                                    \
        if (stamp_slot >= 0 && nstamp < 16) g_stamps[stamp_slot][16 + nstamp++] = clock64(); \
    } while (0)
#else
#define STAMP() do { } while (0)
#define STAMPR() do { } while (0)
#endif

namespace tc {
constexpr int KD = 128, VD = 64, PT = 128;          // pair of chunks = 128 tokens
constexpr uint32_t Q_BYTES = PT * KD * 2;            // 32 KB
constexpr uint32_t V_BYTES = PT * VD * 2;            // 16 KB
constexpr uint32_t H_BYTES = KD * VD * 2;            // 16 KB
// tensor memory columns
constexpr int TM_S = 0, TM_O = 128, TM_T0 = 192, TM_T1 = 256, TM_KV = 320, TM_COLS = 512;
// warps 0..7 do the element-wise work (two per tensor-memory lane quarter), warp 8 issues the MMAs;
// the CTA is launched with three warpgroups so that registers can be moved from the third to the
// first two (setmaxnreg); warps 9..11 exit at once
constexpr int NTHREADS = 384, MMA_WARP = 8;
constexpr int LAM_LD = MAX_L + 2;   // row stride of the staged lambda tile: odd number of 32-bit words, no bank conflicts
}  // namespace tc


// CTA-wide barrier over the 8 element-wise warps and the MMA warp (the spare warps of the third
// warpgroup exit at once and never take part)
// Register hand-over between the third warpgroup (TMA producer, MMA issuer, two idle warps) and the two
// element-wise warpgroups.  The kernel is launched with 168 registers per thread (384 threads); what the third
// group gives up must cover what the other two take, otherwise setmaxnreg.inc waits for registers that never
// become free.  The check is on the values themselves, so an unbalanced pair does not compile.
template <int DEC, int INC>
struct RegisterSplit {
    static_assert(DEC % 8 == 0 && INC % 8 == 0 && DEC >= 24 && INC <= 256, "setmaxnreg takes multiples of 8 in [24, 256]");
    static_assert(128 * (168 - DEC) >= 256 * (INC - 168), "the register pool does not cover this split");
    __device__ static __forceinline__ void release() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(DEC)); }
    __device__ static __forceinline__ void acquire() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(INC)); }
};

// Hands a TMA-filled tile back to the producer from a thread that has read it with ld.shared.  The arrive must
// not be performed before those loads have returned (the producer would refill the tile under them), and
// nothing orders a plain arrive after earlier loads whose results are not used yet.  So the release is preceded,
// in program order and in the same asm block, by a shared-memory store whose VALUE is computed from every loaded
// word: the store cannot issue before the loads have delivered their data, and the arrive issues after it.
// `sink` is any 4-byte shared-memory word that nothing reads (one per thread or shared by all).
__device__ __forceinline__ void release_tile_after_loads(uint64_t* bar, uint32_t* sink, uint32_t digest_of_loaded_words) {
    asm volatile(
        "st.shared.u32 [%0], %1;\n\tmbarrier.arrive.shared::cta.b64 _, [%2];\n"
        ::"r"(umma::smem_addr(sink)), "r"(digest_of_loaded_words), "r"(umma::smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ void bar_work() { asm volatile("bar.sync 1, 288;\n" ::: "memory"); }

// one 32-byte global store (a full sector per lane; two 16-byte stores of a thread that owns a row would touch every sector twice)
__device__ __forceinline__ void st_global_32B(void* dst, const uint32_t (&w)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n"
                 ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}

// barrier over the 8 element-wise warps only
__device__ __forceinline__ void bar_compute() { asm volatile("bar.sync 2, 256;\n" ::: "memory"); }

// ---- what the kernels that walk the heads of a pair (128 tokens from t0 on) need per head, prepared by WARPS warps.  A warp-wide access to values a head
// apart touches a line per lane and costs the load / store pipe about two cycles a line, during which nothing else of the CTA gets through it: hence
// all heads of a token at a time, through shared memory.

// raw log decay of heads [h0, h0 + nh) of every token (zeros behind the sequence): loads here, into sG[head][LD] by heads_to_shared.  nh <= 8.
template <int THREADS>
struct HeadsOfTokens {
    static constexpr int N = tc::PT * 8 / THREADS;
    float v[N];
    __device__ __forceinline__ void load(const float* src, const Mamba2Params& p, int b, int t0, int h0, int nh, int tid) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int e = tid + i * THREADS, t = e / nh, hh = e - t * nh;
            v[i] = t < tc::PT && t0 + t < p.T ? __ldg(src + ((long)b * p.T + t0 + t) * p.H + h0 + hh) : 0.f;
        }
    }
    template <int LD>
    __device__ __forceinline__ void to_shared(float* sG, int nh, int tid) const {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int e = tid + i * THREADS, t = e / nh, hh = e - t * nh;
            if (t < tc::PT) sG[hh * LD + t] = v[i];
        }
    }
};
// sG[head][LD] to global memory
template <int LD, int THREADS>
__device__ __forceinline__ void heads_to_global(float* dst, const Mamba2Params& p, int b, int t0, int h0, int nh, const float* sG, int tid) {
#pragma unroll
    for (int i = 0; i < tc::PT * 8 / THREADS; ++i) {
        const int e = tid + i * THREADS, t = e / nh, hh = e - t * nh;
        if (t < tc::PT && t0 + t < p.T) dst[((long)b * p.T + t0 + t) * p.H + h0 + hh] = sG[hh * LD + t];
    }
}
// decays over the pairs of the segment before and behind pair `pair` (D[i] of its four pairs where `need` has bit i): thread 4 hh + i of the CTA loads D[i]
__device__ __forceinline__ float pair_decay(const Mamba2Params& p, int b, int h0, int nh, int NP, int pair, int need, int tid) {
    const int hh = tid >> 2, i = tid & 3;
    if (hh >= nh || !((need >> i) & 1)) return 0.f;
    return __ldg(reinterpret_cast<const float*>(p.lo_H + (((long)b * p.H + h0 + hh) * NP + (pair & ~3)) * p.K * p.V) + i);
}
// One head per warp, four consecutive tokens per lane, from the raw decay in tG[0, 128): G (cumulative over the pair) in its place, Cf = exp(G[end of
// 32-block] - G) behind it, with TABLES = 3 also Vf = exp(G[127] - G); the in-chunk cumulative sum into `cum` where there is one.
template <int TABLES>
__device__ __forceinline__ void pair_decay_tables(float* tG, float* cum, int lane) {
    const float4 g = *reinterpret_cast<const float4*>(tG + 4 * lane);
    float gq[4] = {g.x, g.y, g.z, g.w};
    gq[1] += gq[0];
    gq[2] += gq[1];
    gq[3] += gq[2];
    float tot = gq[3];                               // inclusive scan of lane totals inside each chunk (16 lanes)
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, tot, d);
        if ((lane & 15) >= d) tot += t;
    }
    const float gla = __shfl_sync(0xffffffffu, tot, 15), glp = gla + __shfl_sync(0xffffffffu, tot, 31);   // end of the first chunk, of the pair
    const float cbase = tot - gq[3];                                // in-chunk exclusive prefix of this lane
    const float pbase = cbase + (lane >= 16 ? gla : 0.f);           // pair-wide
    const float gend = __shfl_sync(0xffffffffu, tot, (lane & ~7) + 7) + (lane >= 16 ? gla : 0.f);
    float G[4], cf[4], vf[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        G[i] = pbase + gq[i];
        cf[i] = fexp(gend - G[i]);
        vf[i] = fexp(glp - G[i]);
    }
    if (cum) *reinterpret_cast<float4*>(cum + 4 * lane) = make_float4(gq[0] + cbase, gq[1] + cbase, gq[2] + cbase, gq[3] + cbase);
    *reinterpret_cast<float4*>(tG + 4 * lane) = make_float4(G[0], G[1], G[2], G[3]);
    *reinterpret_cast<float4*>(tG + 128 + 4 * lane) = make_float4(cf[0], cf[1], cf[2], cf[3]);
    if (TABLES == 3) *reinterpret_cast<float4*>(tG + 256 + 4 * lane) = make_float4(vf[0], vf[1], vf[2], vf[3]);
}
// lambda columns [0, ncol) of heads [h0, h0 + nh) for the 128 tokens from t0 on, ncol a head, as rows of LD values (zeros behind the sequence and the levels).  A warp takes
// a token at a time, eight or more in flight: with one index over all values (a division each, few loads in flight) this took 12 k cycles a CTA.
template <int LD, int WARPS>
__device__ __forceinline__ void stage_lambda(const Mamba2Params& p, int b, int t0, int h0, int nh, int ncol, bf16* sLam, int warp, int lane) {
    const int L = p.L, left = p.T - t0, n = nh * ncol;
    const bf16* gl = p.l + (((long)b * p.T + t0) * p.H + h0) * L;
    const long ldg = (long)p.H * L;
    constexpr int ROWS = tc::PT / WARPS;
    static_assert(LD <= 128 && LD % 2 == 0, "two words a lane");
    if (ncol == L && ((reinterpret_cast<uintptr_t>(gl) | (uintptr_t)(ldg * 2) | (uintptr_t)(n * 2)) & 3) == 0) {
        uint32_t x[ROWS][2];
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int rr = warp + i * WARPS, cc = lane + u * 32;
                x[i][u] = rr < left && 2 * cc < n ? __ldg(reinterpret_cast<const uint32_t*>(gl + rr * ldg) + cc) : 0u;
            }
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (2 * (lane + u * 32) < n) reinterpret_cast<uint32_t*>(sLam + (warp + i * WARPS) * LD)[lane + u * 32] = x[i][u];
    } else {
        const unsigned short* g16 = reinterpret_cast<const unsigned short*>(gl);
        for (int c0 = 0; c0 < n; c0 += 32) {
            const int cc = c0 + lane, hh = cc / ncol, at = hh * L + cc - hh * ncol;
            const bool there = cc < n && cc - hh * ncol < L;
            unsigned short x[ROWS];
#pragma unroll
            for (int i = 0; i < ROWS; ++i) x[i] = warp + i * WARPS < left && there ? __ldg(g16 + (warp + i * WARPS) * ldg + at) : (unsigned short)0;
#pragma unroll
            for (int i = 0; i < ROWS; ++i)
                if (cc < n) sLam[(warp + i * WARPS) * LD + cc] = __ushort_as_bfloat16(x[i]);
        }
    }
}

// g_stamps lives in one translation unit only
}  // namespace llattn
