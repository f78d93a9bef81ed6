// Single-token decode step of the Palimpsa operator (sm_100a): HBM-bound.
//
// Every sequence-head owns a (mu, I) state of V x K float32 pairs that must be read and written once
// per generated token (2 x 2 x V x K x 4 bytes; 262 144 B at V = K = 128), against ~1 KB of token
// inputs.  The kernel is therefore laid out for memory throughput only: KL lanes share a state row and own
// J float4 column groups of it each (J = 3 where d_k / 4 is three times a power of two: 48, 96, 192), so that
// every padded d_k uses all lanes; each warp issues the loads of RB row sets (2 x RB x J 16-byte loads per
// lane) before it touches any of them, to keep enough bytes in flight; the update runs in place.  Outputs are
// reduced over the lanes of a row with one batched (transposed) butterfly per RB row sets.
// Measured (state bytes over time, of a 6 550 GB/s copy): 256 sequences x 12 heads of 128x128 6 640 GB/s, 61 x 16 of
// 96x192 45 us = 6 390 GB/s, 64 x 16 of 48x48 6.0 us; before, d_k = 48, 96, 192 and 256 and odd sizes ran on the general
// forward kernel at 1 600 - 1 800 GB/s (170 and 22 us for those two).
//
// Replaces the reference's use of fused_palimpsa_recurrent_fwd_kernel with T = 1 and a cached state
// (fused_recurrent_palimpsa.py:24-154 called from palimpsa/layers/palimpsa.py:317-331), including the
// seven separate float32 casts it makes per step (fused_recurrent_palimpsa.py:226-236).
#include "common.cuh"
#include "host.h"

namespace palimpsa {

struct DecArgs {
    palimpsa_problem p;
    void* o;
    void* o_var;
    float* final_mu;
    float* final_I;
    int tiles;  // row tiles per sequence-head
};

constexpr long long DEC_SMALL_WARPS = B200_SMS * 16;  // warps that cover the device once at 4 CTAs per SM

template <int DT>
__device__ __forceinline__ float4 ldg4(const void* base, long long idx) {  // idx: element index, multiple of 4
    if (DT == PALIMPSA_F32) return *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + idx);
    const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const unsigned short*>(base) + idx);
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

// Element c of chunk j of lane kl.  VEC: 16-byte groups, column 4 (j KL + kl) + c.  Otherwise (d_k not a multiple of 4, or
// a buffer that is not 16-byte aligned) single elements, column (4 j + c) KL + kl, so that neighbouring lanes still read
// neighbouring addresses.
template <int KL, bool VEC>
__device__ __forceinline__ int dec_col(int j, int c, int kl) {
    return VEC ? 4 * (j * KL + kl) + c : (4 * j + c) * KL + kl;
}
template <int KL, bool VEC, int DT>
__device__ __forceinline__ float4 dec_ld(const void* base, long long row, int j, int kl, int K, float pad) {
    if (VEC) {
        const int c0 = 4 * (j * KL + kl);
        return c0 < K ? ldg4<DT>(base, row + c0) : make_float4(pad, pad, pad, pad);
    }
    float e[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int col = dec_col<KL, VEC>(j, c, kl);
        e[c] = col < K ? ld1<DT>(base, row + col) : pad;
    }
    return make_float4(e[0], e[1], e[2], e[3]);
}
template <int KL, bool VEC>
__device__ __forceinline__ float4 dec_ld_state(const float* base, long long row, int j, int kl, int K, float pad) {
    if (VEC) {
        const int c0 = 4 * (j * KL + kl);
        return c0 < K ? __ldcs(reinterpret_cast<const float4*>(base + row + c0)) : make_float4(pad, pad, pad, pad);
    }
    return dec_ld<KL, VEC, PALIMPSA_F32>(base, row, j, kl, K, pad);
}
template <int KL, bool VEC>
__device__ __forceinline__ void dec_st_state(float* base, long long row, int j, int kl, int K, float4 x) {
    if (VEC) {
        const int c0 = 4 * (j * KL + kl);
        if (c0 < K) __stcs(reinterpret_cast<float4*>(base + row + c0), x);
        return;
    }
    const float e[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int col = dec_col<KL, VEC>(j, c, kl);
        if (col < K) base[row + col] = e[c];
    }
}

// One CTA = 4 warps x (32 / KL) rows x RB row sets of one sequence-head; blockIdx.x runs over (sequence-head, row tile).
template <int KL, int J, int RB, bool UNC, bool VEC, int DT>
__global__ void __launch_bounds__(128) decode_kernel(const DecArgs a) {
    constexpr int RG = 32 / KL, ROWS_PER_WARP = RG * RB, NRED = RB * (UNC ? 2 : 1);
    const palimpsa_problem& p = a.p;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int kl = lane % KL, rg = lane / KL;
    const int nh = blockIdx.x / a.tiles, tile = blockIdx.x - nh * a.tiles, h = nh % p.H;
    const int K = p.K, V = p.V;
    const int rbase = (tile * 4 + w) * ROWS_PER_WARP + rg;  // rows rbase + i*RG, i < RB

    // ---- state rows first: everything else hides behind these loads ----------------------------------
    const long long sbase = (long long)nh * V * K;
    float4 mu[RB][J], pr[RB][J];
#pragma unroll
    for (int i = 0; i < RB; ++i) {
        const int row = rbase + i * RG;
#pragma unroll
        for (int j = 0; j < J; ++j) {
            if (row < V) {
                mu[i][j] = dec_ld_state<KL, VEC>(p.init_mu, sbase + (long long)row * K, j, kl, K, 0.f);
                pr[i][j] = dec_ld_state<KL, VEC>(p.init_I, sbase + (long long)row * K, j, kl, K, 1.f);
            } else {
                mu[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
                pr[i][j] = make_float4(1.f, 1.f, 1.f, 1.f);
            }
        }
    }
    // ---- token inputs ------------------------------------------------------------------------------------
    float vv[RB], bb[RB];
#pragma unroll
    for (int i = 0; i < RB; ++i) {
        const int row = rbase + i * RG;
        vv[i] = row < V ? ld1<DT>(p.v, (long long)nh * V + row) : 0.f;
        bb[i] = row < V ? ld1<DT>(p.b, (long long)nh * V + row) : 0.f;
    }
    float4 k4[J], q4[J];
    const float sc = p.scale;
#pragma unroll
    for (int j = 0; j < J; ++j) {
        k4[j] = dec_ld<KL, VEC, DT>(p.k, (long long)nh * K, j, kl, K, 0.f);
        q4[j] = dec_ld<KL, VEC, DT>(p.q, (long long)nh * K, j, kl, K, 0.f);
        q4[j] = make_float4(q4[j].x * sc, q4[j].y * sc, q4[j].z * sc, q4[j].w * sc);
    }
    const float f = expf(-p.gt[nh] * p.g[h]);
    const float c = (1.f - f) * p.Ip[h];
    float red[NRED];
#pragma unroll
    for (int i = 0; i < RB; ++i) {
        const int row = rbase + i * RG;
        float y = 0.f, yv = 0.f;
        auto upd = [&](float& m, float& pi, float kx, float qx) {
            const float fi = f * pi;
            const float mm = fmaf(m, fi, vv[i] * kx);       // f * (mu*I) + v k
            const float in = fi + fmaf(bb[i], kx * kx, c);  // f * I + (1-f) Ip + b k^2
            float r = rcp_approx(in);
            r = fmaf(r, fmaf(-in, r, 1.f), r);              // one Newton step: the stored mean keeps full precision
            m = mm * r;
            pi = in;
            y = fmaf(m, qx, y);
            if (UNC) yv = fmaf(r, qx * qx, yv);
        };
#pragma unroll
        for (int j = 0; j < J; ++j) {
            upd(mu[i][j].x, pr[i][j].x, k4[j].x, q4[j].x);
            upd(mu[i][j].y, pr[i][j].y, k4[j].y, q4[j].y);
            upd(mu[i][j].z, pr[i][j].z, k4[j].z, q4[j].z);
            upd(mu[i][j].w, pr[i][j].w, k4[j].w, q4[j].w);
            if (row < V) {
                dec_st_state<KL, VEC>(a.final_mu, sbase + (long long)row * K, j, kl, K, mu[i][j]);
                dec_st_state<KL, VEC>(a.final_I, sbase + (long long)row * K, j, kl, K, pr[i][j]);
            }
        }
        red[i * (UNC ? 2 : 1)] = y;
        // o_var = scale * sum q^2 / I with q already scaled once: divide one scale back out
        if (UNC) red[i * 2 + 1] = (sc != 0.f) ? yv / sc : 0.f;
    }
    xreduce<NRED, KL>(red, lane);
    constexpr int REM = NRED >= KL ? NRED / KL : 1;
    const int base = xreduce_index<NRED, KL>(lane);
    const bool owner = NRED >= KL ? true : (kl & (KL / (NRED < KL ? NRED : KL) - 1)) == 0;
    if (owner) {
#pragma unroll
        for (int j = 0; j < REM; ++j) {
            const int id = base + j;
            const int which = UNC ? (id & 1) : 0;
            const int i = UNC ? (id >> 1) : id;
            const int row = rbase + i * RG;
            if (row < V) st1(which ? a.o_var : a.o, (long long)nh * V + row, red[j], p.io_dtype);
        }
    }
}

template <int KL, int J, int RB, bool VEC>
static int launch_decode_t(DecArgs a, cudaStream_t stream) {
    const palimpsa_problem& p = a.p;
    constexpr int ROWS_PER_CTA = 4 * (32 / KL) * RB;
    a.tiles = (p.V + ROWS_PER_CTA - 1) / ROWS_PER_CTA;
    const long long ctas = (long long)a.tiles * p.num_seqs * p.H;
    if (ctas > 0x7fffffffLL) return PALIMPSA_E_SHAPE;
    const bool unc = (p.flags & PALIMPSA_FLAG_UNCERTAINTY) != 0;
#define PALIMPSA_DEC_LAUNCH(U, D) decode_kernel<KL, J, RB, U, VEC, D><<<(unsigned)ctas, 128, 0, stream>>>(a)
    if (p.io_dtype == PALIMPSA_BF16) {
        if (unc) PALIMPSA_DEC_LAUNCH(true, PALIMPSA_BF16); else PALIMPSA_DEC_LAUNCH(false, PALIMPSA_BF16);
    } else if (p.io_dtype == PALIMPSA_F32) {
        if (unc) PALIMPSA_DEC_LAUNCH(true, PALIMPSA_F32); else PALIMPSA_DEC_LAUNCH(false, PALIMPSA_F32);
    } else {
        if (unc) PALIMPSA_DEC_LAUNCH(true, PALIMPSA_F16); else PALIMPSA_DEC_LAUNCH(false, PALIMPSA_F16);
    }
#undef PALIMPSA_DEC_LAUNCH
    return cudaGetLastError() == cudaSuccess ? PALIMPSA_OK : PALIMPSA_E_LAUNCH;
}

// True if this call is one token per sequence on a state that is read and written: any d_k, any alignment.
bool decode_supported(const palimpsa_fwd_params* prm) {
    const palimpsa_problem& p = prm->p;
    return !p.cu_seqlens && p.seq_len == 1 && p.init_mu && prm->final_mu && !prm->ckpt_M;
}

// RB row sets per warp: enough bytes in flight per warp once the grid fills the device.  One set while it does not (the
// shortest chain from load to store: 48x48, 1 sequence x 16 heads 1.7 us), and where d_v would leave half of the taller
// CTA's warps without rows (16x32 heads: 128-row CTAs 3.7 TB/s).
template <int KL, int J, int RB>
static int launch_decode_k(const DecArgs& a, bool vec, cudaStream_t stream) {
    if (!vec) return launch_decode_t<KL, J, 1, false>(a, stream);
    const long long warps = (long long)a.p.num_seqs * a.p.H * ((a.p.V + 32 / KL - 1) / (32 / KL));  // with one set each
    if (RB > 1 && (warps < DEC_SMALL_WARPS || 2 * a.p.V <= 4 * (32 / KL) * RB)) return launch_decode_t<KL, J, 1, true>(a, stream);
    return launch_decode_t<KL, J, RB, true>(a, stream);
}

int launch_decode(const palimpsa_fwd_params* prm, cudaStream_t stream) {
    DecArgs a{};
    a.p = prm->p;
    a.o = prm->o;
    a.o_var = prm->o_var;
    a.final_mu = prm->final_mu;
    a.final_I = prm->final_I;
    const palimpsa_problem& p = a.p;
    auto al = [](const void* x, int m) { return (reinterpret_cast<uintptr_t>(x) & (m - 1)) == 0; };
    const int io_al = p.io_dtype == PALIMPSA_F32 ? 16 : 8;
    const bool vec = p.K % 4 == 0 && al(p.q, io_al) && al(p.k, io_al) && al(p.init_mu, 16) && al(p.init_I, 16) &&
                     al(a.final_mu, 16) && al(a.final_I, 16);
    switch (palimpsa_padded_k(p.K)) {
        case 16: return launch_decode_k<4, 1, 4>(a, vec, stream);
        case 32: return launch_decode_k<8, 1, 4>(a, vec, stream);
        case 48: return launch_decode_k<4, 3, 2>(a, vec, stream);
        case 64: return launch_decode_k<16, 1, 4>(a, vec, stream);
        case 96: return launch_decode_k<8, 3, 2>(a, vec, stream);
        case 128: return launch_decode_k<32, 1, 8>(a, vec, stream);
        case 192: return launch_decode_k<16, 3, 2>(a, vec, stream);
        case 256: return launch_decode_k<32, 2, 4>(a, vec, stream);
        default: return PALIMPSA_E_DIM;
    }
}

// ---- the token inputs of a replayed step: up to 8 small buffers copied in one launch -------------------------------
struct CopyArgs {
    const char* src[8];
    char* dst[8];
    unsigned long long bytes[8];
};
__global__ void __launch_bounds__(256) copy_buffers_kernel(const CopyArgs a) {
    const char* src = a.src[blockIdx.y];
    char* dst = a.dst[blockIdx.y];
    const unsigned long long n = a.bytes[blockIdx.y], step = (unsigned long long)gridDim.x * blockDim.x;
    unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x, done = 0;
    if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0) {
        for (unsigned long long c = i; c < n / 16; c += step) reinterpret_cast<int4*>(dst)[c] = reinterpret_cast<const int4*>(src)[c];
        done = n / 16 * 16;
    }
    for (unsigned long long c = done + i; c < n; c += step) dst[c] = src[c];
}

int launch_copy_buffers(const void* const* src, void* const* dst, const size_t* bytes, int n, cudaStream_t stream) {
    CopyArgs a{};
    size_t most = 0;
    for (int i = 0; i < n; ++i) {
        a.src[i] = static_cast<const char*>(src[i]);
        a.dst[i] = static_cast<char*>(dst[i]);
        a.bytes[i] = bytes[i];
        most = bytes[i] > most ? bytes[i] : most;
    }
    if (most == 0) return PALIMPSA_OK;
    const size_t blocks = (most + 4095) / 4096;  // 16 bytes per thread, at most two CTAs per SM
    copy_buffers_kernel<<<dim3((unsigned)(blocks > 296 ? 296 : blocks), n), 256, 0, stream>>>(a);
    return cudaGetLastError() == cudaSuccess ? PALIMPSA_OK : PALIMPSA_E_LAUNCH;
}

}  // namespace palimpsa
