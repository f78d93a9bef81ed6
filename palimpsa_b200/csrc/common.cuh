// Shared device helpers for the Palimpsa sm_100a kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/palimpsa_b200.h"

namespace palimpsa {

// Tokens per staged block.  Equal to the checkpoint interval, so that every staged block of a
// sequence starts on a checkpoint.
constexpr int TB = PALIMPSA_CKPT_INTERVAL;

// ---------------------------------------------------------------------------------------------
// Packed FP32 arithmetic: sm_100 executes two FP32 lanes per instruction on 64-bit register
// pairs (fma.rn.f32x2 and friends), halving the issue slots of the element-wise recurrence.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 dup2(float x) { return make_float2(x, x); }

// One MUFU op, relative error <= 2^-23.
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float2 rcp2(float2 x) { return make_float2(rcp_approx(x.x), rcp_approx(x.y)); }

// ---------------------------------------------------------------------------------------------
// Asynchronous global->shared copies (LDGSTS).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------------------------------------
// io dtype handling.  DT is PALIMPSA_F32 / BF16 / F16.
// ---------------------------------------------------------------------------------------------
__host__ __device__ __forceinline__ int dtype_size(int dt) { return dt == PALIMPSA_F32 ? 4 : 2; }

// Four consecutive values, group index idx4, from a 16-byte aligned buffer (shared or global).
template <int DT>
__device__ __forceinline__ float4 ld4(const void* base, int idx4) {
    if (DT == PALIMPSA_F32) {
        return reinterpret_cast<const float4*>(base)[idx4];
    } else {
        uint2 u = reinterpret_cast<const uint2*>(base)[idx4];
        float2 a, b;
        if (DT == PALIMPSA_BF16) {
            a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
            b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
        } else {
            a = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
            b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
        }
        return make_float4(a.x, a.y, b.x, b.y);
    }
}

// N (2 or 4) consecutive floats in one access, as pairs.
template <int N>
__device__ __forceinline__ void ld_cols(const float* p, float2 (&x)[N / 2]) {
    if constexpr (N == 4) {
        const float4 y = *reinterpret_cast<const float4*>(p);
        x[0] = make_float2(y.x, y.y), x[1] = make_float2(y.z, y.w);
    } else {
        x[0] = *reinterpret_cast<const float2*>(p);
    }
}
template <int N>
__device__ __forceinline__ void st_cols(float* p, const float2 (&x)[N / 2]) {
    if constexpr (N == 4) *reinterpret_cast<float4*>(p) = make_float4(x[0].x, x[0].y, x[1].x, x[1].y);
    else *reinterpret_cast<float2*>(p) = x[0];
}

// One value from global memory, any alignment.
template <int DT>
__device__ __forceinline__ float ld1(const void* base, long long idx) {
    if (DT == PALIMPSA_F32) return reinterpret_cast<const float*>(base)[idx];
    if (DT == PALIMPSA_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(base)[idx]);
    return __half2float(reinterpret_cast<const __half*>(base)[idx]);
}

// Four values starting at element idx, each read only if its index is below limit (else 0).
template <int DT>
__device__ __forceinline__ float4 ld4_guarded(const void* base, long long idx, long long limit) {
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    if (idx + 0 < limit) r.x = ld1<DT>(base, idx + 0);
    if (idx + 1 < limit) r.y = ld1<DT>(base, idx + 1);
    if (idx + 2 < limit) r.z = ld1<DT>(base, idx + 2);
    if (idx + 3 < limit) r.w = ld1<DT>(base, idx + 3);
    return r;
}

__device__ __forceinline__ void st1(void* base, long long idx, float x, int dt) {
    if (dt == PALIMPSA_F32)
        reinterpret_cast<float*>(base)[idx] = x;
    else if (dt == PALIMPSA_BF16)
        reinterpret_cast<__nv_bfloat16*>(base)[idx] = __float2bfloat16_rn(x);
    else
        reinterpret_cast<__half*>(base)[idx] = __float2half_rn(x);
}

__host__ __device__ __forceinline__ int round_up(int x, int m) { return (x + m - 1) / m * m; }

// Token range of sequence n.
__device__ __forceinline__ void seq_range(const palimpsa_problem& p, int n, int& bos, int& len) {
    if (p.cu_seqlens) {
        bos = p.cu_seqlens[n];
        len = p.cu_seqlens[n + 1] - bos;
    } else {
        bos = n * p.seq_len;
        len = p.seq_len;
    }
    if (len < 0) len = 0;
}

// First checkpoint slot of sequence n.
__device__ __forceinline__ long long seq_first_slot(const palimpsa_problem& p, int n) {
    if (p.chunk_offsets) return p.chunk_offsets[n];
    return (long long)n * ((p.seq_len + TB - 1) / TB);
}

// Store four values as duplicated pairs {x,x,y,y},{z,z,w,w} (operands of packed FP32 instructions).
__device__ __forceinline__ void st_dup4(float4* dst, int i, float4 x) {
    dst[2 * i] = make_float4(x.x, x.x, x.y, x.y);
    dst[2 * i + 1] = make_float4(x.z, x.z, x.w, x.w);
}


// How the threads of a CTA split the 16-byte chunks of a [tokens][chunks] tile among themselves: thread ->
// (first token, chunk), then every `step` tokens.  Computed once per kernel, so that the per-block copy loops
// carry no integer division.  `step` = 0: the thread count is not a multiple of the chunk count (generic loop).
struct ChunkSplit {
    int t0, c, step;
};
__device__ __forceinline__ ChunkSplit chunk_split(int chunks, int nthr, int tid) {
    ChunkSplit s{0, 0, 0};
    if (chunks > 0 && chunks <= nthr && nthr % chunks == 0) {
        s.t0 = tid / chunks;
        s.c = tid - s.t0 * chunks;
        s.step = nthr / chunks;
    }
    return s;
}

// ---------------------------------------------------------------------------------------------
// The recurrence without its decay.  A block of 16 tokens is cut into windows; over the tokens of one, F_t is the product of the
// decays f up to t, u_t = 1 - F_t, and w_t the product of those behind t.  The state is held as
//     forward   M' = w_t M,   B' = w_t (I - u_t Ip)     M' += (w_t v_t) k_t^T    B' += (w_t b_t) (k_t^2)^T    Z_t = w_t u_t Ip
//     backward  M' = M / F_t, B' = (I - u_t Ip) / F_t   M' += (v_t / F_t) k_t^T  B' += (b_t / F_t) (k_t^2)^T  Z_t = u_t Ip / F_t
//     and in both  mu_t = M' / (B' + Z_t)
// -- one packed FMA per pair of state elements instead of a multiply and an FMA for M and two FMAs for I.  B' starts from the
// true I of the window's start and only positive terms join it, so a small I beside a large Ip keeps its bits.  In front of the
// tokens named by `special` the state is scaled, M' <- s M', B' <- s B' + c: in the forward at each window's first (s is the
// product of that window, c what the last one left: u Ip s), so that the window ends with M itself and the newest terms, which
// weigh most, are not rounded by a scale; in the backward at the first token of every window after the block's first (s is the
// product of the last one), which costs a block nothing at its start, where its checkpoint is read twice.
// F, u and w are worked out in 64 bits and rounded once: they have to agree, since where b is small I = F I + u Ip must stay
// where it is, and u must not be taken from a rounded product where Ip is large beside I.  (In 32 bits the error of the final mu
// was 1.04 to 1.29 times that of a walk with the decay in every step, of o and the gradients 1.02 to 1.09 times; now 0.4 to 0.9 and
// 0.45 to 1.0.  With I0 = 0.01, Ip = 1000 and decays near 0.99, 48x48, o was off by 7.5e-5, now by 5e-7.)  What that costs is the
// helper warps' time between two hand-overs: backward 0.99 -> 1.02 ms at B=8 T=2048 H=16 48x48, whose two helpers have none to
// spare, 2.16 -> 2.18 at H=6 d=128; the forward, two blocks at a time, 0.57 -> 0.574 (0.595 one at a time).
// Scales reach 2^-48 (SCALE_LO): the float range that is left holds states and gradients from 1e-20 to 1e20 in all their bits (at
// 2^-64 v of 1e20 gave NaN, d_o of 1e-20 lost 10 bits), and g * gt may be 2 a token for a block to be one window.  Where the
// decays are faster, a new one begins in front of a group of 4 tokens, and in a group that is too fast by itself (or has an f
// above 1) every token is alone: in the backward without any scale (F = 1), its s and c those of the plain recurrence.
// ---------------------------------------------------------------------------------------------
constexpr double SCALE_LO = 0x1p-48;

struct BlockScale {
    float f;           // decay of this lane's token (1 past the end)
    float w, z;        // w_t or 1 / F_t, and Z_t
    float s, c;        // what is done to the state in front of the token: 1, 0 where it is left alone
    float end;         // of the block's last window: forward, what is missing from its last I, u Ip; backward, F
    unsigned special;  // bit t: token t has s and c; the forward's bit 0 is always set (the same for the whole block)
};
// By a whole warp: lanes 0 to 15 hold the tokens of one block, lanes 16 to 31 those of another, or the same again.
template <bool BACKWARD>
__device__ __forceinline__ BlockScale block_scale(float gt, bool live, float gh, float iph, int lane) {
    static_assert(TB == 16, "two blocks in a warp");
    constexpr unsigned ALL = 0xffffffffu;
    BlockScale b;
    const int t = lane & 15, half = lane & 16;
    // f with the bits that 1 - f needs, and with what gt * gh was rounded by
    const float x = live ? gt * gh : 0.f, xl = live ? fmaf(gt, gh, -x) : 0.f, u1 = -expm1f(-x), f1 = expf(-x);
    double f = fabsf(u1) < 0.5f ? 1. - (double)u1 : (double)f1;
    if (fabsf(xl) < 1.f) f = fma(f, -(double)xl, f);
    b.f = (float)f;
    int first = 0, last = 15;  // this token's window
    bool alone = false;
    auto up_to = [&]() __attribute__((always_inline)) {  // product over the window up to this token
        double y = f;
#pragma unroll
        for (int d = 1; d < 16; d *= 2) {
            const double o = __shfl_up_sync(ALL, y, d, 16);
            if (t - d >= first) y *= o;
        }
        return y;
    };
    double F = up_to();
    b.special = BACKWARD ? 0 : 1;
    const unsigned many = __ballot_sync(ALL, !(F >= SCALE_LO && b.f <= 1.f));
    if (many) {  // more than one window, in one of the two blocks at least
        double g4 = f;  // of the group of 4
        g4 *= __shfl_xor_sync(ALL, g4, 1);
        g4 *= __shfl_xor_sync(ALL, g4, 2);
        const unsigned out = __ballot_sync(ALL, !(g4 >= SCALE_LO && b.f <= 1.f)) >> half;
        double cum = 1.;
        unsigned starts = 0, single = 0;
#pragma unroll
        for (int q = 0; q < TB / 4; ++q) {
            const double g = __shfl_sync(ALL, g4, 4 * q, 16);
            const bool slow = (out >> (4 * q)) & 15u, fresh = q == 0 || !(cum * g >= SCALE_LO);
            starts |= (slow ? 15u : fresh ? 1u : 0u) << (4 * q);
            single |= (slow ? 15u : 0u) << (4 * q);
            cum = slow ? 0. : fresh ? g : cum * g;  // the group after one of single tokens begins a window
        }
        // tokens past the end begin none in the forward, which does not always walk them
        if (!BACKWARD) starts = (starts & (__ballot_sync(ALL, live) >> half)) | 1u;
        if ((many >> half) & 0xffffu) {  // a block's scalars depend on nothing but the block
            b.special = starts;
            alone = BACKWARD && ((single >> t) & 1u);
            first = 31 - __clz(starts & ((2u << t) - 1u));
            last = __ffs((starts >> t >> 1) | (1u << (15 - t))) - 1 + t;
        }
        F = up_to();
        if (alone) F = 1.;
    }
    const double u = 1. - F;
    b.s = 1.f, b.c = 0.f;
    if (BACKWARD) {
        b.w = __frcp_rn((float)F);
        b.z = (float)(u * b.w) * iph;
        b.end = (float)__shfl_sync(ALL, F, 15, 16);
        if (many) {
            double s = __shfl_up_sync(ALL, F, 1, 16);
            if (t != first || t == 0) s = 1.;
            if (alone) s *= f;
            b.s = (float)s;
            b.c = (float)(1. - s) * iph;
            b.special = (__ballot_sync(ALL, !(s == 1.)) >> half) & 0xffffu;
        }
    } else {
        double P = f;  // product from this token to the window's end
#pragma unroll
        for (int d = 1; d < 16; d *= 2) {
            const double o = __shfl_down_sync(ALL, P, d, 16);
            if (t + d <= last) P *= o;
        }
        const double behind = __shfl_down_sync(ALL, P, 1, 16), w = t == last ? 1. : behind;
        b.w = (float)w;
        b.z = (float)(u * w) * iph;
        b.end = (float)__shfl_sync(ALL, u, 15, 16) * iph;
        if (t == first) b.s = (float)P;
        if (many) {
            const double before = __shfl_up_sync(ALL, u, 1, 16);
            if (t == first && t > 0) b.c = (float)(P * before) * iph;
        }
    }
    return b;
}

// Sum N per-lane values over the L lanes that differ from this one in the low log2(L) bits
// (L = 2^s <= 32).  "Transposed" butterfly: each step exchanges half of the remaining values, so it
// costs N-1 (+ a few) shuffles instead of N*log2(L).  An odd remainder above one is padded with a zero (N itself is
// even or one).  On return x[i], i < xreduce_count<N, L>(lane), holds the sum of value xreduce_index<N, L>(lane) + i.
template <int N, int L>
__device__ __forceinline__ void xreduce(float (&x)[N], int lane) {
    static_assert(N == 1 || N % 2 == 0, "no room for the padding");
    int n = N;
#pragma unroll
    for (int off = L / 2; off >= 1; off >>= 1) {
        if (n > 1) {
            if (n & 1) x[n++] = 0.f;
            const int half = n / 2;
            const bool up = (lane & off) != 0;
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                if (i < half) {
                    const float keep = up ? x[i + half] : x[i];
                    const float send = up ? x[i] : x[i + half];
                    x[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
            }
            n = half;
        } else {
            x[0] += __shfl_xor_sync(0xffffffffu, x[0], off);
        }
    }
}
// First value of this lane's share, how many of N values a lane is left with at most, and how many of them are this
// lane's to write: none where another lane holds the same one or only padding is left.
template <int N, int L>
__device__ __forceinline__ int xreduce_index(int lane) {
    int idx = 0, n = N;
#pragma unroll
    for (int off = L / 2; off >= 1; off >>= 1) {
        if (n > 1) {
            n = (n + 1) / 2;
            if (lane & off) idx += n;
        }
    }
    return idx;
}
template <int N, int L>
__host__ __device__ constexpr int xreduce_most() {
    int n = N;
    for (int off = L / 2; off >= 1; off >>= 1)
        if (n > 1) n = (n + 1) / 2;
    return n;
}
template <int N, int L>
__device__ __forceinline__ int xreduce_count(int lane) {
    int n = N, count = N;
#pragma unroll
    for (int off = L / 2; off >= 1; off >>= 1) {
        if (n > 1) {
            n = (n + 1) / 2;
            count = (lane & off) ? (count > n ? count - n : 0) : (count < n ? count : n);
        } else if (lane & off) {
            count = 0;
        }
    }
    return count;
}

}  // namespace palimpsa
