// Helpers of the element-wise passes around the scans (preparation, convolution, norms).  These passes are bound by HBM: what counts
// is bytes in flight and as few special-function instructions per byte as possible.
#pragma once
#include "llattn_common.cuh"

namespace llattn {

__device__ __forceinline__ float softplus_row(float x) { return x > 20.f ? x : log1pf(__expf(x)); }
// within the 2 ulp of __fdividef and, for negative x, the 2 + 1.2 |x| ulp of __expf(-x): far below the rounding to bf16 behind it.  A correctly
// rounded division would be a third of the instructions of the passes that use it
__device__ __forceinline__ float sigmoid_row(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16(x)); }

// What torch's operators on bf16 tensors give, each result rounded to bf16: the inference calls (prompts, decode steps) keep these rounding
// points of the operator sequence around the recurrence.
__device__ __forceinline__ float softplus_torch(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float lambda_torch(int mode, float lp, float d) {
    lp = round_bf16(lp);
    if (mode == 0) return round_bf16(softplus_torch(round_bf16(lp * d)));
    if (mode == 1) return round_bf16(expf(round_bf16(-round_bf16(expf(lp)) * round_bf16(softplus_torch(d)))));
    return round_bf16(lp * d);
}

// N consecutive bf16 values as packed words; `vec`: the address is a multiple of the words' size
template <int N>
struct Packed {
    uint32_t w[N / 2];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < N / 2; ++i) w[i] = 0u;
    }
    __device__ __forceinline__ void load(const bf16* p, bool vec) {
        static_assert(N == 4 || N == 8, "8 or 16 bytes");
        if (vec) {
            if (N == 8) {
                const uint4 r = *reinterpret_cast<const uint4*>(p);
                w[0] = r.x; w[1] = r.y; w[N / 2 - 2] = r.z; w[N / 2 - 1] = r.w;
            } else {
                const uint2 r = *reinterpret_cast<const uint2*>(p);
                w[0] = r.x; w[1] = r.y;
            }
        } else {
            const unsigned short* s = reinterpret_cast<const unsigned short*>(p);
#pragma unroll
            for (int i = 0; i < N / 2; ++i) w[i] = (uint32_t)s[2 * i] | ((uint32_t)s[2 * i + 1] << 16);
        }
    }
    // zeros unless `p`.  The aligned load is predicated, not branched around: a branch per load keeps the compiler from having the
    // loads of a group in flight together
    __device__ __forceinline__ void load_if(const bf16* ptr, bool vec, bool p) {
        if (!vec) {
            zero();
            if (p) load(ptr, false);
        } else if (N == 8) {
            asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %5, 0;\n mov.b32 %0, 0;\n mov.b32 %1, 0;\n mov.b32 %2, 0;\n mov.b32 %3, 0;\n"
                         " @p ld.global.v4.b32 {%0, %1, %2, %3}, [%4];\n}\n"
                         : "=&r"(w[0]), "=&r"(w[1]), "=&r"(w[N / 2 - 2]), "=&r"(w[N / 2 - 1])
                         : "l"(ptr), "r"((int)p));
        } else {
            asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %3, 0;\n mov.b32 %0, 0;\n mov.b32 %1, 0;\n @p ld.global.v2.b32 {%0, %1}, [%2];\n}\n"
                         : "=&r"(w[0]), "=&r"(w[1])
                         : "l"(ptr), "r"((int)p));
        }
    }
    // a bf16 is the upper half of an fp32
    __device__ __forceinline__ float operator[](int i) const { return __uint_as_float((i & 1) ? (w[i >> 1] & 0xffff0000u) : (w[i >> 1] << 16)); }
};

template <int N>
__device__ __forceinline__ void store_row(bf16* p, const float (&f)[N], bool vec) {
    if (vec) {
        uint32_t w[N / 2];
#pragma unroll
        for (int i = 0; i < N / 2; ++i) w[i] = pack_bf16(f[2 * i], f[2 * i + 1]);
        if (N == 8) *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[N / 2 - 2], w[N / 2 - 1]);
        else *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) p[i] = __float2bfloat16(f[i]);
    }
}

// Gradients of lambda = f(lp, d): of d, and of lp
__device__ __forceinline__ void lambda_grad(int mode, float lp, float elp, float d, float gl, float& gd, float& gp) {
    if (mode == 0) {
        const float u = lp * d, s = u > 20.f ? 1.f : sigmoid_row(u);
        gd = gl * s * lp;
        gp = gl * s * d;
    } else if (mode == 1) {
        const float sp = softplus_row(d), r = __expf(-elp * sp);
        gd = -gl * r * elp * (d > 20.f ? 1.f : sigmoid_row(d));
        gp = -gl * r * elp * sp;
    } else {
        gd = gl * lp;
        gp = gl * d;
    }
}
__device__ __forceinline__ float lambda_value(int mode, float lp, float elp, float d) {
    if (mode == 0) return softplus_row(lp * d);
    if (mode == 1) return __expf(-elp * softplus_row(d));
    return lp * d;
}

__device__ __forceinline__ void red_add_f32x4(float* addr, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// The lambda part of a pass: lambda (or the gradients of dl and Lp) of the (head, level) columns of tokens t0 .. t1 - 1 by one CTA.  A
// thread owns VL neighbouring columns (VL = 8: 16 bytes of dl a load; VL = 1 where the columns do not come in eights) and every
// (blockDim / columns)-th token, UT of them at a time: their loads are issued before the first of their stores.  Row strides are in elements; the pointers are those of the tensors' first token.
struct LambdaCols {
    const bf16* dl;
    long dl_stride;
    const void* Lp;
    int lp_f32, n, mode;       // n = H L
};

// Runs of tokens of the lambda part in a backward pass: its sums go to the few addresses of L, so there are only as many runs as fill the chip (at B = 2,
// T = 16384, 32 heads the backward pass took 214 us with the 2048 runs of its other part, 104 us without its lambda part).  One CTA per SM: they come
// first and hold back the other part (that pass with 296 / 148 / 100 / 74 CTAs 128 / 119 / 120 / 124 us, T = 4096 alone 39 / 29 / 25 / 21, B = 4, T = 8192,
// 16 heads 81 / 79 / 91 / 110); two where a thread has one column (B = 8, T = 2048, 10 heads, L = 15: 75 us, with one 91).
inline int lambda_runs(int tokens, int blocks, bool eights) {
    const int ctas = eights ? 148 : 296, most = blocks >= ctas ? 1 : ctas / blocks, runs = (tokens + 15) / 16;
    return runs < most ? runs : most;
}

// the columns of a token, as they are in memory
template <int VL>
struct LambdaRow {
    Packed<8> w;
    bf16 one;
    __device__ __forceinline__ void load(const bf16* p) {
        if (VL == 8) w.load(p, true);
        else one = p[0];
    }
    __device__ __forceinline__ float operator[](int i) const { return VL == 8 ? w[i] : __bfloat162float(one); }
};
template <int VL>
__device__ __forceinline__ void load_cols(float (&f)[VL], const float* p) {
    if (VL == 8) {
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        f[0] = a.x; f[VL / 8] = a.y; f[VL / 4] = a.z; f[VL * 3 / 8] = a.w;
        f[VL / 2] = b.x; f[VL * 5 / 8] = b.y; f[VL * 3 / 4] = b.z; f[VL * 7 / 8] = b.w;
    } else {
        f[0] = p[0];
    }
}
template <int VL>
__device__ __forceinline__ void store_cols(bf16* p, const float (&f)[VL]) {
    if (VL == 8) store_row<8>(p, reinterpret_cast<const float(&)[8]>(f), true);
    else p[0] = __float2bfloat16(f[0]);
}

template <int VL, int UT>
__device__ __forceinline__ void lambda_part_fwd(const LambdaCols& c, bf16* lam, int t0, int t1, int block, int nblocks) {
    const int groups = c.n / VL;                               // threads of a token
    const int per = min(groups, (int)blockDim.x), rows = blockDim.x / per;
    const int r = threadIdx.x / per;
    for (int gidx = block * per + threadIdx.x % per; gidx < groups && r < rows; gidx += nblocks * per) {
        const int e = gidx * VL;
        float lp[VL], elp[VL];
#pragma unroll
        for (int i = 0; i < VL; ++i) {
            lp[i] = load_param(c.Lp, e + i, c.lp_f32);
            elp[i] = __expf(lp[i]);
        }
        for (int t = t0 + r; t < t1; t += UT * rows) {
            LambdaRow<VL> in[UT];
#pragma unroll
            for (int u = 0; u < UT; ++u) in[u].load(c.dl + min(t + u * rows, t1 - 1) * c.dl_stride + e);
#pragma unroll
            for (int u = 0; u < UT; ++u) {
                if (t + u * rows >= t1) break;
                float d[VL];
#pragma unroll
                for (int i = 0; i < VL; ++i) d[i] = lambda_value(c.mode, lp[i], elp[i], in[u][i]);
                store_cols<VL>(lam + (long)(t + u * rows) * c.n + e, d);
            }
        }
    }
}

template <int VL, int UT>
__device__ __forceinline__ void lambda_part_bwd(const LambdaCols& c, const float* dlam, bf16* ddl, long ddl_stride, float* dLp, int t0, int t1,
                                                int block, int nblocks, float* sums) {
    // sums: blockDim * VL floats of shared memory.  The threads that share columns add up there, so that a column costs one global
    // atomic per CTA (one per thread, on the few addresses of L, took longer than the whole pass)
    const int groups = c.n / VL;
    const int per = min(groups, (int)blockDim.x), rows = blockDim.x / per;
    const int r = threadIdx.x / per;
    for (int g0 = block * per; g0 < groups; g0 += nblocks * per) {
        const int gidx = g0 + threadIdx.x % per;
        const bool act = gidx < groups && r < rows;
        const int e = act ? gidx * VL : 0;
        float lp[VL], elp[VL], sum[VL];
#pragma unroll
        for (int i = 0; i < VL; ++i) {
            lp[i] = load_param(c.Lp, e + i, c.lp_f32);
            elp[i] = __expf(lp[i]);
            sum[i] = 0.f;
        }
        for (int t = act ? t0 + r : t1; t < t1; t += UT * rows) {
            LambdaRow<VL> in[UT];
            float gl[UT][VL];
#pragma unroll
            for (int u = 0; u < UT; ++u) {
                const long tt = min(t + u * rows, t1 - 1);
                in[u].load(c.dl + tt * c.dl_stride + e);
                load_cols<VL>(gl[u], dlam + tt * c.n + e);
            }
#pragma unroll
            for (int u = 0; u < UT; ++u) {
                if (t + u * rows >= t1) break;
                float d[VL];
#pragma unroll
                for (int i = 0; i < VL; ++i) {
                    float gp;
                    lambda_grad(c.mode, lp[i], elp[i], in[u][i], gl[u][i], d[i], gp);
                    sum[i] += gp;
                }
                store_cols<VL>(ddl + (t + u * rows) * ddl_stride + e, d);
            }
        }
        if (rows > 1) {
            __syncthreads();
#pragma unroll
            for (int i = 0; i < VL; ++i) sums[i * blockDim.x + threadIdx.x] = sum[i];
            __syncthreads();
            if (r == 0)
                for (int q = 1; q < rows; ++q)
#pragma unroll
                    for (int i = 0; i < VL; ++i) sum[i] += sums[i * blockDim.x + q * per + threadIdx.x];
        }
        if (act && r == 0) {
#pragma unroll
            for (int i = 0; i < VL; ++i) atomicAdd(&dLp[e + i], sum[i]);
        }
    }
}

}  // namespace llattn
