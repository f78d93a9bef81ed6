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
// The recurrence without its decay.  Inside a window of tokens over which F_t is the product of the decays f, the scaled
// state M' = M / F, B' = (I - (1 - F) Ip) / F obeys
//     M'_t = M'_{t-1} + (v_t / F_t) k_t^T        B'_t = B'_{t-1} + (b_t / F_t) (k_t^2)^T
//     I_t / F_t = B'_t + Z_t,  Z_t = (1 - F_t) Ip / F_t          mu_t = M'_t / (B'_t + Z_t)
// -- one packed FMA per pair of state elements instead of a multiply and an FMA for M and two FMAs for I.  B' starts from the
// true I of the window's start and only positive terms join it, so a small I beside a large Ip keeps its bits.  Every
// rounding is relative to the value it rounds, as before; F only has to stay in the range of a float, for which a window ends
// when F would fall below SCALE_LO (gradients of that window's end are held multiplied by F).  A block of 16 tokens is one window unless its decays are faster than that: then a new one
// begins in front of a group of 4 tokens, and a group that leaves the range by itself (or has an f above 1) is walked token by
// token in unscaled form (F = 1).  A token that begins a window or is walked by itself first scales the state it finds, by s:
//     M' <- s M'        B' <- s B' + (1 - s) Ip
// (s = F at the window's end, times f_t for a token by itself; s = 1 elsewhere: the state is left alone.)
// ---------------------------------------------------------------------------------------------
constexpr float SCALE_LO = 0x1p-64f;

struct BlockScale {
    float f;           // decay of this lane's token (1 past the end)
    float inv;         // 1 / F_t
    float z;           // Z_t
    float s, c;        // scale of the state in front of the token, and (1 - s) Ip
    float end;         // F at the end of the block, by which its last window ends (the same for the whole block)
    unsigned special;  // bit t: token t has s != 1 (the same for the whole block)
};
// By a whole warp: lanes 0 to 15 hold the tokens of one block, lanes 16 to 31 those of another, or the same again.
__device__ __forceinline__ BlockScale block_scale(float gt, bool live, float gh, float iph, int lane) {
    static_assert(TB == 16, "two blocks in a warp");
    BlockScale b;
    const int t = lane & 15, j = t & 3, half = lane & 16;
    b.f = live ? expf(-gt * gh) : 1.f;
    float x = b.f;  // product over the group up to this token
    const float y1 = __shfl_up_sync(0xffffffffu, x, 1, 4);
    if (j >= 1) x *= y1;
    const float y2 = __shfl_up_sync(0xffffffffu, x, 2, 4);
    if (j >= 2) x *= y2;
    float grp[TB / 4], F = x;
#pragma unroll
    for (int q = 0; q < TB / 4; ++q) grp[q] = __shfl_sync(0xffffffffu, x, 4 * q + 3, 16);
    if (t >= 4) F = x * (t < 8 ? grp[0] : t < 12 ? grp[0] * grp[1] : grp[0] * grp[1] * grp[2]);
    b.s = 1.f;
    b.special = 0;
    const unsigned many = __ballot_sync(0xffffffffu, !(F >= SCALE_LO && b.f <= 1.f));
    if (many) {  // more than one window, in one of the two blocks at least
        const unsigned out = __ballot_sync(0xffffffffu, !(x >= SCALE_LO && b.f <= 1.f)) >> half;
        float cum = 1.f, base = 1.f, s = 1.f;
        bool alone = false;
#pragma unroll
        for (int q = 0; q < TB / 4; ++q) {
            const float next = cum * grp[q];
            const bool slow = (out >> (4 * q)) & 15u, fresh = slow || !(next >= SCALE_LO);
            if ((t >> 2) == q) {
                alone = slow;
                base = fresh ? 1.f : cum;
                s = fresh && j == 0 ? cum : 1.f;
            }
            cum = slow ? 1.f : fresh ? grp[q] : next;
        }
        if ((many >> half) & 0xffffu) {  // a block's scalars depend on nothing but the block
            b.s = alone ? s * b.f : s;
            F = alone ? 1.f : base * x;
        }
        b.special = (__ballot_sync(0xffffffffu, b.s != 1.f) >> half) & 0xffffu;
    }
    b.inv = __frcp_rn(F);
    b.z = (1.f - F) * iph * b.inv;
    b.c = (1.f - b.s) * iph;
    b.end = __shfl_sync(0xffffffffu, F, 15, 16);
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
