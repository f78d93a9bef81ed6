// Backward kernels of the Palimpsa operator (sm_100a).
//
// Main kernel: one CTA owns TV state rows x all KP columns of one (sequence, head) and walks the
// sequence's 16-token blocks from the last to the first.  Per block it
//   1. takes the block's start state (M, I) from the checkpoint the forward saved, which lies in
//      shared memory beside the block's operands (the helper warps brought both one block ahead),
//   2. sweeps forward once, parking the state at the start of each 4-token group (thread-private
//      slots in shared memory),
//   3. per group, last first: recomputes the 4 per-token states into registers, then walks the
//      tokens in reverse, carrying the state gradients (GM, -GI) in registers:
//          r    = 1 / (B + Z)           mu = M*r                    h = dy*q_s * r
//          GM  += h                     -GI += h*mu (+ dy_var/F * (q*r)^2)
//          dq  += dy*mu   dk += GM*v/F + 2k*GI*b/F   dv/F += GM*k   db/F += GI*k^2
//          f*df = <GM, M_prev> + <GI, B_prev - Ip>
//      all in the scaled form in which neither the state nor its gradient decays from token to token (block_scale in
//      common.cuh; GM, GI are the gradients of the scaled M and B): the algebra of chunk_palimpsa_bwd_kernel,
//      chunk_palimpsa_forgetting_scalar.py:343-434, divided by F, with the previous state carried forward instead of rebuilt
//      by a division, :409-410.  Blocks in which the state is scaled on the way take other copies of the walk, one for scales in
//      front of groups, one for scales in front of any token, which also scale the gradients there (B=8 T=2048 H=6 d=128, ms with
//      one window, windows in front of groups, tokens by themselves: 2.18, 2.40, 2.49; the plain recurrence 2.38).
// Reductions: over d_k (dv, db) by xor-shuffles inside the lanes of a row; over d_v (dq, dk) first
// in registers across a thread's rows, then across the CTA's row groups through shared memory, and
// across the CTAs of different row tiles through fp32 partial buffers in the workspace, which the
// finishing kernel sums in a fixed order (bitwise reproducible; no atomics).
// Helper warps stage the next block (checkpoint by cp.async; inputs through registers, where they wait while a group is summed,
// into fp32 operands of a second operand stage) and do all that follows a group's partials in shared memory (sums over the row
// groups, casts, global stores).  All hand-overs are mbarriers with bounded waits: the compute warps meet no CTA barrier and
// drift apart.
// What bounds the walk is the issue rate: a packed FP32 instruction takes two issue cycles, a pair of state elements 28 per
// token in the reverse walk and 7 in the two forward steps (14 before the scaled form), and operand loads, shuffle sums and moves
// come on top.  The scaled form, with the first term of every sum as a product instead of an FMA on a zero, took the backward at
// B=8 T=4096 H=6 d=128 from 4.75 to 4.31 ms, at H=16 48x48 from 2.15 to 1.98 and at B=4 T=2048 H=16 96x192 from 4.06 to 3.84; as a
// branch per group instead of per block it was 4.63 and 2.11 (moves of the gradients where the two copies meet).  So it
// pays to have 12 elements a thread (two warps per scheduler) rather than 8 (three), and to take staging off those warps.
// Through registers, because a copy in shared memory to convert from costs 10 to 37 KB, for want of which some shapes had one
// operand stage or one group buffer, and because rows that start at any offset can only be loaded one by one, which four warps
// do not get done between two groups.  One wave of 148 CTAs, T = 512, converted from shared memory -> through registers, us:
// 128x88 bf16 296 -> 291, 48x48 268 -> 269, 48x48 float32 with the uncertainty output 379 -> 305, 96x32 436 -> 375, 192x12 407 ->
// 269, 256x8 426 -> 363; rows at any offset: 127x87 363 -> 296, 95x23 411 -> 269, 47x47 415 -> 277, 15x63 238 -> 165.
// One CTA per SM, beside the smallest tilings; bwd_config has the choice of the tile.
//
// Finishing kernels: (1) per (token, head) row: sum the row tiles, cast dq/dk, form
// dgt = -g f df and the per-row terms of dg and dIp; (2) per head: ordered sum over rows.
#include <atomic>
#include <cmath>
#include <initializer_list>
#include <mutex>
#include <type_traits>
#include <utility>

#include "host.h"
#include "tc_common.cuh"

namespace palimpsa {

constexpr int GR = 4;  // tokens per register-resident group

// 0 ok; 5 / 6: a bounded wait on the split-phase barriers of the backward's group reduction gave up
__device__ int g_bwd_status = 0;

__device__ __forceinline__ void st2(void* base, long long idx, float2 x, int dt) {  // idx even, base aligned for it
    if (dt == PALIMPSA_F32)
        *reinterpret_cast<float2*>(reinterpret_cast<float*>(base) + idx) = x;
    else if (dt == PALIMPSA_BF16)
        *reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<__nv_bfloat16*>(base) + idx) = __floats2bfloat162_rn(x.x, x.y);
    else
        *reinterpret_cast<__half2*>(reinterpret_cast<__half*>(base) + idx) = __floats2half2_rn(x.x, x.y);
}

struct BwdArgs {
    palimpsa_problem p;
    const void* d_o;
    const void* d_o_var;
    const float* ckpt_M;
    const float* ckpt_I;
    float *dq_part, *dk_part, *df_part, *dip_part;
    void *dv, *db;
    int vec_k, vec_v;  // four columns of q and k, two rows of v, b and the output gradients come in one load: else one by one
    int rows;        // state rows of a tile: as many as the CTA's warps hold, or fewer
    int kbuf;        // shared-memory buffers for the per-group d_k-indexed partials: 2 where they fit, else 1
    int rows_total;  // tokens * H
    // segments (gridDim.z of them per sequence; seg_len tokens each, a multiple of 16; 0 = whole sequence)
    int seg_len;
    const float* carry_M;  // [N,G,H,V,KP] dL/d(end state of the segment), (M, I) form, or NULL (zero)
    const float* carry_I;
    float* rloc_M;         // [N,G,H,V,KP] dL/d(start state of the segment), or NULL
    float* rloc_I;
};

struct BwdSmem {
    int ks, qs, vb, dys2, dyvs2, fc2, zz2, fi2, blk;  // offsets inside an operand stage; the two stages come first
    int op_stage, slots, ckb;
    int kred, dvs, dbs, wred, fgr;  // per-group partials handed to the helper warps, kbuf buffers of each
    int bars;                       // mbarriers: full[2], empty[2], staged[2], done[2]; then the failure flag
    int ck_stage;  // bytes of one (M, I) checkpoint stage
    int total;
};

// Shared-memory plan of one backward CTA (KP padded d_k, NE state elements per thread, W compute warps that hold TV state rows
// in WV row groups).  Operands v, b, dy are stored with every value duplicated ({x, x}), v and b of a row side by side, so
// that one 128-bit load yields the two register pairs the packed FP32 instructions want.
__host__ __device__ inline BwdSmem bwd_smem_layout(int KP, int TV, int NE, int W, int WV, bool unc, int kbuf) {
    BwdSmem s;
    int off = 0;
    auto take = [&](int bytes) {
        int o = off;
        off += round_up(bytes, 16);
        return o;
    };
    s.ks = take(TB * KP * 4);
    s.qs = take(TB * KP * 4);
    s.vb = take(TB * TV * 16);
    s.dys2 = take(TB * TV * 8);
    s.dyvs2 = unc ? take(TB * TV * 8) : 0;
    s.fc2 = take(TB * 16);  // {s, s, c, c}
    s.zz2 = take(TB * 8);   // {Z, Z}
    s.fi2 = take(TB * 8);   // {f, 1 / F}
    s.blk = take(16);       // F at the block's end, BlockScale::special
    s.op_stage = off;
    off *= 2;
    s.slots = take(2 * 2 * NE * 32 * W * 4);
    s.ck_stage = 2 * TV * KP * 4;
    s.ckb = take(2 * s.ck_stage);
    s.kred = take(kbuf * GR * WV * 2 * KP * 4);  // kbuf = 2 group buffers where they fit (host's choice), else 1
    s.dvs = take(kbuf * GR * TV * 4);
    s.dbs = take(kbuf * GR * TV * 4);
    s.wred = take(kbuf * W * GR * 2 * 4);
    s.fgr = take(kbuf * GR * 8);
    s.bars = take(80);
    s.total = off;
    return s;
}

// Asynchronous copy of one block's checkpoint rows (M, I) into checkpoint stage `stage_idx`, by `nthr` threads.
__device__ __forceinline__ void bwd_issue_ckpt(const BwdArgs& a, int nthr, int tid, unsigned char* sm, const BwdSmem& L,
                                               int stage_idx, int KP, int TV, long long slot, int h, int v0, int tvw) {
    const palimpsa_problem& p = a.p;
    unsigned char* ck = sm + L.ckb + stage_idx * L.ck_stage;
    const int cr = KP / 4;
    const long long base = ((slot * p.H + h) * (long long)p.V + v0) * KP;
    for (int i = tid; i < tvw * cr; i += nthr) {
        cp_async16(ck + i * 16, a.ckpt_M + base + (long long)i * 4);
        cp_async16(ck + TV * KP * 4 + i * 16, a.ckpt_I + base + (long long)i * 4);
    }
}

// A thread's share of TS tokens of a block on its way from global memory to the operand stage: loaded as it lies there, and
// converted when it is stored.  Between the two the helper warps wait for a group and sum it, so that neither the loads'
// latency nor, where rows start at any offset, the many single loads are in anybody's way.
template <int KP, int TV, int TS, int NTH, bool UNC>
struct BwdStaging {
    static constexpr int F0 = NTH > 64 ? NTH - 64 : 0;  // the threads that write a block's scalars: neither the first nor the last warp's
    static constexpr int K4 = KP / 4, V2 = TV / 2, NQ = (TS * K4 + NTH - 1) / NTH, NV = (TS * V2 + NTH - 1) / NTH;
    unsigned q[NQ][4], k[NQ][4];                // 4 columns: packed 16-bit pairs in [0], [1] where they came in one load
    unsigned v[NV][2], b[NV][2], o[NV][2], ov[NV][2];  // 2 rows: a packed 16-bit pair in [0]
    float gt;                                   // step size of token lane & 15 of the block
    BlockScale sc;                              // and what bwd_scale has made of the block's
};

// N consecutive elements of ES bytes at element e, the first n of them (the others 0).
template <int ES, int N>
__device__ __forceinline__ void ld_words(unsigned (&w)[N], const void* base, long long e, int n, bool vec) {
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = 0;
    if (vec) {
        if (n > 0) {
            const char* p = reinterpret_cast<const char*>(base) + e * ES;
            if constexpr (ES * N == 16) {
                const uint4 x = *reinterpret_cast<const uint4*>(p);
                w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w;
            } else if constexpr (ES * N == 8) {
                const uint2 x = *reinterpret_cast<const uint2*>(p);
                w[0] = x.x, w[1] = x.y;
            } else {
                w[0] = *reinterpret_cast<const unsigned*>(p);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i < n)
                w[i] = ES == 4 ? reinterpret_cast<const unsigned*>(base)[e + i] : reinterpret_cast<const unsigned short*>(base)[e + i];
    }
}
template <int DT>
__device__ __forceinline__ float word_value(unsigned w) {  // of a single element
    if (DT == PALIMPSA_F32) return __uint_as_float(w);
    if (DT == PALIMPSA_BF16) return __uint_as_float(w << 16);
    return __half2float(__ushort_as_half((unsigned short)w));
}
template <int DT, int N>
__device__ __forceinline__ void word_values(const unsigned (&w)[N], float (&x)[N], bool vec) {
    if (DT != PALIMPSA_F32 && vec) {
#pragma unroll
        for (int i = 0; i < N; i += 2) {
            x[i] = word_value<DT>(w[i / 2] & 0xffffu);
            x[i + 1] = word_value<DT>(w[i / 2] >> 16);
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] = word_value<DT>(w[i]);
    }
}

// Tokens [ts, ts + TS) of the block of nt tokens that starts at token tok0, by NTH threads.
template <int ES, int KP, int TV, int TS, int NTH, bool UNC>
__device__ __forceinline__ void bwd_load(BwdStaging<KP, TV, TS, NTH, UNC>& s, const BwdArgs& a, int tid, long long tok0, int ts,
                                         int nt, int h, int v0, int tvw) {
    using S = BwdStaging<KP, TV, TS, NTH, UNC>;
    const palimpsa_problem& p = a.p;
#pragma unroll
    for (int x = 0; x < S::NQ; ++x) {
        const int i = tid + x * NTH, t = ts + i / S::K4, c = 4 * (i % S::K4);
        const long long row = ((tok0 + t) * p.H + h) * (long long)p.K + c;
        const int n = t < nt && i < TS * S::K4 ? p.K - c : 0;
        ld_words<ES>(s.q[x], p.q, row, n, a.vec_k);
        ld_words<ES>(s.k[x], p.k, row, n, a.vec_k);
    }
#pragma unroll
    for (int x = 0; x < S::NV; ++x) {
        const int i = tid + x * NTH, t = ts + i / S::V2, r = 2 * (i % S::V2);
        const long long row = ((tok0 + t) * p.H + h) * (long long)p.V + v0 + r;
        const int n = t < nt && i < TS * S::V2 ? tvw - r : 0;
        ld_words<ES>(s.v[x], p.v, row, n, a.vec_v);
        ld_words<ES>(s.b[x], p.b, row, n, a.vec_v);
        ld_words<ES>(s.o[x], a.d_o, row, n, a.vec_v);
        if (UNC) ld_words<ES>(s.ov[x], a.d_o_var, row, n, a.vec_v);
    }
    if (ts == 0) {
        const int t = tid & (TB - 1);
        s.gt = t < nt ? p.gt[(tok0 + t) * p.H + h] : 0.f;
    }
}

// The scalars of a block of nt tokens.  By whole warps, each for itself; between the block's first load and its first store.
template <int KP, int TV, int TS, int NTH, bool UNC>
__device__ __forceinline__ void bwd_scale(BwdStaging<KP, TV, TS, NTH, UNC>& s, int tid, int nt, float gh, float iph) {
    s.sc = block_scale<true>(s.gt, (tid & (TB - 1)) < nt, gh, iph, tid & 31);
}

// What bwd_load brought, as fp32 operands into the operand stage `op`: v, b and the uncertainty's gradient divided by F
// (block_scale).  By whole warps.
template <int DT, int KP, int TV, int TS, int NTH, bool UNC>
__device__ __forceinline__ void bwd_store(BwdStaging<KP, TV, TS, NTH, UNC>& s, const BwdArgs& a, int tid, unsigned char* op,
                                          const BwdSmem& L, int ts) {
    using S = BwdStaging<KP, TV, TS, NTH, UNC>;
    if (ts == 0 && tid >= S::F0 && tid < S::F0 + TB) {
        const int t = tid & (TB - 1);
        reinterpret_cast<float4*>(op + L.fc2)[t] = make_float4(s.sc.s, s.sc.s, s.sc.c, s.sc.c);
        reinterpret_cast<float2*>(op + L.zz2)[t] = make_float2(s.sc.z, s.sc.z);
        reinterpret_cast<float2*>(op + L.fi2)[t] = make_float2(s.sc.f, s.sc.w);
        if (t == 0) *reinterpret_cast<float2*>(op + L.blk) = make_float2(s.sc.end, __uint_as_float(s.sc.special));
    }
    float4* qs = reinterpret_cast<float4*>(op + L.qs) + ts * S::K4;
    float4* ks = reinterpret_cast<float4*>(op + L.ks) + ts * S::K4;
    // The scale goes with q; with the uncertainty output, which wants q and q squared, with the output gradients instead.
    const float sq = UNC ? 1.f : a.p.scale, so = UNC ? a.p.scale : 1.f;
#pragma unroll
    for (int x = 0; x < S::NQ; ++x) {
        const int i = tid + x * NTH;
        if (i >= TS * S::K4) break;
        float q[4], k[4];
        word_values<DT>(s.q[x], q, a.vec_k);
        word_values<DT>(s.k[x], k, a.vec_k);
        qs[i] = make_float4(q[0] * sq, q[1] * sq, q[2] * sq, q[3] * sq);
        ks[i] = make_float4(k[0], k[1], k[2], k[3]);
    }
    float4* vb = reinterpret_cast<float4*>(op + L.vb) + ts * TV;
    float4* dys = reinterpret_cast<float4*>(op + L.dys2) + ts * S::V2;
    float4* dyvs = reinterpret_cast<float4*>(op + L.dyvs2) + ts * S::V2;
#pragma unroll
    for (int x = 0; x < S::NV; ++x) {
        const int i = tid + x * NTH;
        const float inv = __shfl_sync(0xffffffffu, s.sc.w, (ts + i / S::V2) & (TB - 1));
        if (i >= TS * S::V2) break;
        float v[2], b[2], o[2];
        word_values<DT>(s.v[x], v, a.vec_v);
        word_values<DT>(s.b[x], b, a.vec_v);
        word_values<DT>(s.o[x], o, a.vec_v);
        v[0] *= inv, v[1] *= inv, b[0] *= inv, b[1] *= inv;
        vb[2 * i] = make_float4(v[0], v[0], b[0], b[0]);
        vb[2 * i + 1] = make_float4(v[1], v[1], b[1], b[1]);
        dys[i] = make_float4(o[0] * so, o[0] * so, o[1] * so, o[1] * so);
        if (UNC) {
            word_values<DT>(s.ov[x], o, a.vec_v);
            o[0] *= so * inv, o[1] *= so * inv;
            dyvs[i] = make_float4(o[0], o[0], o[1], o[1]);
        }
    }
}

// Threads of a CTA: W compute warps, and helper warps: as many as fit beside the compute warps without costing those
// registers, which are handed out per scheduler (8 warps of an SM may have 255 per thread, 12 may have 168).
__host__ __device__ constexpr int bwd_helpers(int W) { return W == 6 ? 2 : 4; }
__host__ __device__ constexpr int bwd_threads(int W) { return 32 * (W + bwd_helpers(W)); }

// Where an even share is too little for the walk (8 warps of 12 state elements spill 200 bytes at 168 registers), the
// warpgroup of helpers gives up registers that the compute warpgroups take: {entry, compute, helper} registers per thread,
// {0, 0, 0} = no split.  The compute warps wait for the helpers' registers, so the block must have been launched with enough
// for all: bwd_split_fits asks the compiled kernel before the first launch.
// (With the uncertainty output 224 and 56 registers: 2.67 ms at B=8 T=2048 H=6 d=128, with 208 and 88 2.46.)
struct RegSplit {
    int entry, compute, helper;
};
__host__ __device__ constexpr RegSplit bwd_split(int W, int RV, int RK) {
    return W == 8 && RV * RK == 12 ? RegSplit{168, 208, 88} : RegSplit{0, 0, 0};
}

// CTAs of an SM that the registers have to do for: two of the smallest tilings.  At d_k = 32 that spilled 36 bytes (72 now): 148 / 296 / 740
// CTAs of 32x32, T = 512, take 175 / 268 / 658 us, with one 148 / 289 / 715; with the uncertainty output it would spill 192:
// 205 / 340 / 831 us against 164 / 320 / 792.
__host__ __device__ constexpr int bwd_min_ctas(int RK, int KG, int W, bool unc) {
    return KG == 8 && W == 4 && (RK == 2 || (RK == 4 && !unc)) ? 2 : 1;
}

// Tokens of a block that the helper warps carry through registers at a time (BwdStaging): the whole block where they have the
// registers, since every step costs a helper its address and type branches again (48x48 on 6 warps, B=8 T=4096 H=16: 1.98 ms, half
// a block at a time 2.05).  With the uncertainty output smaller steps are (float32, T=2048, 1.18 and 1.12 ms): what 40 registers hold, a
// whole block on 4 warps of d_k = 48 and 96, half of one on 6 and on 8 of d_k = 256, a quarter on 6 of d_k = 192.
__host__ __device__ constexpr int bwd_step_tokens(int KP, int TV, int HT, bool unc, RegSplit split) {
    const int room = split.entry > 0 ? split.helper - 54 : unc ? 40 : 72;
    for (int ts = TB; ts > 4; ts /= 2)
        if ((ts * KP / 4 + HT - 1) / HT * 8 + (ts * TV / 2 + HT - 1) / HT * (unc ? 8 : 6) <= room) return ts;
    return 4;
}

template <int RV, int NP>
struct State {
    float2 M[RV][NP], I[RV][NP];
};

template <int RK, int KG, int RV, int W, bool UNC, bool CO>
__global__ void __launch_bounds__(bwd_threads(W), bwd_min_ctas(RK, KG, W, UNC))
bwd_kernel(const BwdArgs a) {
    constexpr int KP = RK * KG, VG = 32 / KG, NP = RK / 2, NE = RV * RK, KP2 = KP / 2;
    constexpr int TV = W * VG * RV, WV = W * VG, NTHR = 32 * W, HW = bwd_helpers(W), HT = 32 * HW;
    static_assert(TV % 2 == 0, "the operand tiles are converted two rows at a time");
    constexpr RegSplit SPLIT = bwd_split(W, RV, RK);
    static_assert(SPLIT.entry == 0 || (W % 4 == 0 && HW == 4 &&
                                       W * SPLIT.compute + 4 * SPLIT.helper <= (W + 4) * SPLIT.entry),
                  "whole warpgroups on both sides, and no more registers than the block has at launch");
    constexpr int NG = TB / GR;       // groups per block
    constexpr int NR1 = GR * RV * 2;  // per-group d_v-indexed partials of a thread: (token, row, dv|db)
    constexpr int NR2 = GR * 2;       // per-group per-token scalars: (token, df|sum GI)
    extern __shared__ __align__(16) unsigned char sm[];
    const palimpsa_problem& p = a.p;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int kg = lane % KG, vg = lane / KG, wv = w * VG + vg;
    const int row0 = wv * RV;
    const int ny = blockIdx.y / p.H, h = blockIdx.y - ny * p.H;
    const int n = p.seq_order ? p.seq_order[ny] : ny;  // blocks start in grid order: a packed batch lists its longest sequences first
    const int tile = blockIdx.x;
    const int v0 = tile * a.rows;
    const int tvw = min(a.rows, p.V - v0);
    const int es = dtype_size(p.io_dtype);
    const int KBUF = a.kbuf;  // shared-memory buffers for the d_k-indexed partials of a token group (1 or 2)
    const BwdSmem L = bwd_smem_layout(KP, TV, NE, W, WV, UNC, KBUF);
    int bos, len;
    seq_range(p, n, bos, len);
    // this CTA's segment of the sequence: tokens [s0, s1), blocks [blk0, blk1)
    const int g = blockIdx.z, G = gridDim.z;
    const int s0 = a.seg_len > 0 ? min(len, g * a.seg_len) : 0;
    const int s1 = a.seg_len > 0 ? min(len, s0 + a.seg_len) : len;
    const long long seg_base = (((long long)n * G + g) * p.H + h) * p.V;  // row index into [N,G,H,V,KP] buffers
    if (s1 <= s0) {  // empty segment: the end-state gradient is the start-state gradient
        if (a.rloc_M) {
            for (int i = tid; i < tvw * (KP / 4); i += bwd_threads(W)) {
                const long long e = (seg_base + v0) * KP + (long long)i * 4;
                float4 cm = make_float4(0.f, 0.f, 0.f, 0.f), ci = cm;
                if (!CO && a.carry_M) {
                    cm = *reinterpret_cast<const float4*>(a.carry_M + e);
                    ci = *reinterpret_cast<const float4*>(a.carry_I + e);
                }
                *reinterpret_cast<float4*>(a.rloc_M + e) = cm;
                *reinterpret_cast<float4*>(a.rloc_I + e) = ci;
            }
        }
        return;
    }
    const float gh = p.g[h], iph = p.Ip[h];
    const int V = p.V;
    const long long slot0 = seq_first_slot(p, n);
    const int blk0 = s0 / TB, blk1 = (s1 + TB - 1) / TB;
    const int nblk = blk1 - blk0;
    const bool has_carry = !CO && a.carry_M != nullptr;
    const bool has_init = p.init_mu != nullptr || (p.flags & PALIMPSA_FLAG_EXPLICIT_INIT);

    // Hand-overs, all waits bounded (a wait that gives up is recorded below):
    //   full[b] / empty[b]   a group's partials, buffer b = gi & (KBUF - 1): one arrival per compute / helper warp
    //   staged[s] / done[s]  block it, s = it & 1: its operands and checkpoint lie in shared memory (one arrival per helper
    //                        warp); the compute warps are through with it (one per compute warp)
    unsigned long long* full = reinterpret_cast<unsigned long long*>(sm + L.bars);
    unsigned long long* empty = full + 2;
    unsigned long long* staged = full + 4;
    unsigned long long* done = full + 6;
    int* fail_flag = reinterpret_cast<int*>(full + 8);
    unsigned use = 0;  // how often this thread has been through buffer KBUF - 1, the first one of a block
    int wait_fail = 0;
    float* dvs = reinterpret_cast<float*>(sm + L.dvs);
    float* dbs = reinterpret_cast<float*>(sm + L.dbs);
    float* wred = reinterpret_cast<float*>(sm + L.wred);
    float2* fgr = reinterpret_cast<float2*>(sm + L.fgr);  // {f, 1 / F}
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            mbar_init_n(&full[b], W);
            mbar_init_n(&empty[b], HW);
            mbar_init_n(&staged[b], HW);
            mbar_init_n(&done[b], W);
        }
        *fail_flag = 0;
        tc::mbar_init_fence();
    }
    // the block that is walked first, by all threads
    auto tok0_of = [&](int it) __attribute__((always_inline)) { return (long long)bos + (blk1 - 1 - it) * TB; };
    auto load = [&](auto& s, int id, int it, int ts) __attribute__((always_inline)) {
        const int nt = min(TB, len - (blk1 - 1 - it) * TB);
        if (es == 4) bwd_load<4>(s, a, id, tok0_of(it), ts, nt, h, v0, tvw);
        else bwd_load<2>(s, a, id, tok0_of(it), ts, nt, h, v0, tvw);
    };
    auto scale = [&](auto& s, int id, int it) __attribute__((always_inline)) {
        bwd_scale(s, id, min(TB, len - (blk1 - 1 - it) * TB), gh, iph);
    };
    auto store = [&](auto& s, int id, int it, int ts) __attribute__((always_inline)) {
        unsigned char* op = sm + (it & 1) * L.op_stage;
        if (p.io_dtype == PALIMPSA_BF16) bwd_store<PALIMPSA_BF16>(s, a, id, op, L, ts);
        else if (p.io_dtype == PALIMPSA_F32) bwd_store<PALIMPSA_F32>(s, a, id, op, L, ts);
        else bwd_store<PALIMPSA_F16>(s, a, id, op, L, ts);
    };
    bwd_issue_ckpt(a, bwd_threads(W), tid, sm, L, 0, KP, TV, slot0 + blk1 - 1, h, v0, tvw);
    cp_async_commit();
    {
        BwdStaging<KP, TV, TB, bwd_threads(W), UNC> s;
        load(s, tid, 0, 0);
        scale(s, tid, 0);
        store(s, tid, 0, 0);
    }
    cp_async_wait<0>();
    __syncthreads();

    // (inlined, as every lambda in it: a call would need registers that a split warp does not have)
    auto help = [&](const int ht) __attribute__((always_inline)) {
        // ---- helper warps ---------------------------------------------------------------------------------------
        // In front of the walk: the next block's checkpoint by cp.async, its inputs TS tokens at a time through registers into
        // the other operand stage.  Behind it, everything a group leaves once its partials lie in shared memory: dq / dk
        // summed over the CTA's row groups and written to this row tile's partials, dv / db cast and written, the per-token
        // scalars summed over the warps.
        constexpr int KP4 = KP / 4, TS = bwd_step_tokens(KP, TV, HT, UNC, SPLIT);
        BwdStaging<KP, TV, TS, HT, UNC> next;
        auto arrive_staged = [&](int it) __attribute__((always_inline)) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&staged[it & 1]);
        };
        arrive_staged(0);
        if (nblk > 1) {
            load(next, ht, 1, 0);
            scale(next, ht, 1);
        }

        // Two rows of dv / db in one store: d_v even (then a tile's rows are too), both buffers aligned for a pair.
        const bool pairs = V % 2 == 0 && ((reinterpret_cast<uintptr_t>(a.dv) | reinterpret_cast<uintptr_t>(a.db)) & (2 * es - 1)) == 0;
        const float4* kred4 = reinterpret_cast<const float4*>(sm + L.kred);
        for (int it = 0; it < nblk; ++it) {
            const int t0 = (blk1 - 1 - it) * TB, nt = min(TB, len - t0);
            const long long tok0 = (long long)bos + t0;
            const bool more = it + 1 < nblk;
            int ts = 0;
#pragma unroll 1
            for (int gi = NG - 1; gi >= 0; --gi) {
                // While a group is walked: a step of the next block, and the loads of the step after it.
                if (more && ts < TB) {
                    if (ts == 0) {  // the stages were block it - 1's
                        if (it > 0 && !wait_fail && !mbar_wait_idle(&done[(it - 1) & 1], ((it - 1) >> 1) & 1)) wait_fail = 5;
                        bwd_issue_ckpt(a, HT, ht, sm, L, (it + 1) & 1, KP, TV, slot0 + blk1 - 2 - it, h, v0, tvw);
                        cp_async_commit();
                    }
                    store(next, ht, it + 1, ts);
                    ts += TS;
                    if (ts < TB || it + 2 < nblk) load(next, ht, it + (ts < TB ? 1 : 2), ts < TB ? ts : 0);
                }
                if (more && gi == (TS < 8 ? 0 : 1)) {  // as early as can be: warps that are ahead wait for it
                    cp_async_wait<0>();
                    arrive_staged(it + 1);
                }
                if (!CO) {
                    const int b = gi & (KBUF - 1);
                    if (!wait_fail && !mbar_wait_idle(&full[b], use & 1)) wait_fail = 5;
                    if (b == 0) ++use;
                    const int ng = min(GR, nt - gi * GR);  // tokens of the group that exist (<= 0 past the sequence end)
                    const long long trow = (tok0 + gi * GR) * p.H + h;  // (token, head) row of the group's first token
                    const size_t prow = (size_t)tile * a.rows_total + trow;
                    for (int i = ht; i < ng * 2 * KP4; i += HT) {
                        const int j = i / (2 * KP4), which = i / KP4 - 2 * j, c4 = i % KP4;
                        const float4* src = kred4 + ((b * GR + j) * WV * 2 + which) * KP4 + c4;
                        float2 s0 = make_float2(0.f, 0.f), s1 = s0;
#pragma unroll
                        for (int x = 0; x < WV; ++x) {
                            const float4 y = src[x * 2 * KP4];
                            s0 = fadd2(s0, make_float2(y.x, y.y));
                            s1 = fadd2(s1, make_float2(y.z, y.w));
                        }
                        if (!UNC) {
                            const float2 m = dup2(which ? 1.f : p.scale);
                            s0 = fmul2(m, s0);
                            s1 = fmul2(m, s1);
                        }
                        reinterpret_cast<float4*>(which ? a.dk_part : a.dq_part)[(prow + (size_t)j * p.H) * KP4 + c4] =
                            make_float4(s0.x, s0.y, s1.x, s1.y);
                    }
                    for (int i = ht; i < ng * (TV / 2); i += HT) {
                        const int j = i / (TV / 2), r = 2 * (i - j * (TV / 2));
                        const float2 inv = dup2(fgr[b * GR + j].y);
                        const float2 x = fmul2(inv, *reinterpret_cast<const float2*>(dvs + b * GR * TV + 2 * i));
                        const float2 y = fmul2(make_float2(-inv.x, -inv.y), *reinterpret_cast<const float2*>(dbs + b * GR * TV + 2 * i));
                        const long long e = (trow + (long long)j * p.H) * V + v0 + r;
                        if (pairs && r < tvw) {
                            st2(a.dv, e, x, p.io_dtype);
                            st2(a.db, e, y, p.io_dtype);
                        } else if (r < tvw) {
                            st1(a.dv, e, x.x, p.io_dtype);
                            st1(a.db, e, y.x, p.io_dtype);
                            if (r + 1 < tvw) {
                                st1(a.dv, e + 1, x.y, p.io_dtype);
                                st1(a.db, e + 1, y.y, p.io_dtype);
                            }
                        }
                    }
                    if (ht >= HT - 32 && lane < ng) {
                        float df = 0.f, s2 = 0.f;
#pragma unroll
                        for (int x = 0; x < W; ++x) {
                            const float2 y = reinterpret_cast<const float2*>(wred)[(b * W + x) * GR + lane];
                            df += y.x;
                            s2 += y.y;
                        }
                        const float2 fi = fgr[b * GR + lane];
                        s2 *= -fi.y;
                        float dip = (1.f - fi.x) * s2;
                        if (t0 + gi * GR + lane == 0 && !has_init) dip += fi.x * s2;  // I_0 = Ip: the start-state gradient reaches Ip
                        a.df_part[prow + (size_t)lane * p.H] = df;
                        a.dip_part[prow + (size_t)lane * p.H] = dip;
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[b]);
                }
            }
            if (it + 2 < nblk) scale(next, ht, it + 2);  // while nothing waits for it
        }
        cp_async_wait<0>();
        if (wait_fail) *fail_flag = wait_fail;
        __syncthreads();
    };
    // ---- compute warps -------------------------------------------------------------------------------------------------
    auto walk = [&]() __attribute__((always_inline)) {
        if (w * VG * RV >= tvw) {
            // A warp without rows (a tile lower than the CTA, or the last one): its share of every sum is zero, written once;
            // after that it only keeps the hand-overs going, each no earlier than the others can use it.
            if (!CO) {
                for (int i = lane; i < KBUF * GR * VG * 2 * KP2; i += 32) {
                    const int bj = i / (VG * 2 * KP2);
                    reinterpret_cast<float2*>(sm + L.kred)[(bj * WV + w * VG) * 2 * KP2 + i - bj * (VG * 2 * KP2)] = make_float2(0.f, 0.f);
                }
                for (int i = lane; i < KBUF * GR; i += 32)
                    reinterpret_cast<float2*>(wred)[((i / GR) * W + w) * GR + i % GR] = make_float2(0.f, 0.f);
            }
            for (int it = 0; it < nblk; ++it) {
                if (!wait_fail && !mbar_wait_idle(&staged[it & 1], (it >> 1) & 1)) wait_fail = 6;
                for (int gi = NG - 1; !CO && gi >= 0; --gi) {
                    const int b = gi & (KBUF - 1);
                    if (!wait_fail && !mbar_wait_idle(&empty[b], (use & 1) ^ 1)) wait_fail = 6;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full[b]);
                    if (b == 0) ++use;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&done[it & 1]);
            }
            if (wait_fail) *fail_flag = wait_fail;
            __syncthreads();
            return;
        }

        float4* slots4 = reinterpret_cast<float4*>(sm + L.slots) + tid;
        float2* kred2 = reinterpret_cast<float2*>(sm + L.kred);

        // running state gradients: GM = dL/dM_t, nGI = -dL/dI_t of the earliest token processed so far
        float2 GM[RV][NP], nGI[RV][NP];
#pragma unroll
        for (int r = 0; r < RV; ++r)
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                GM[r][q] = nGI[r][q] = make_float2(0.f, 0.f);
                if (has_carry && row0 + r < tvw) {
                    const long long e = (seg_base + v0 + row0 + r) * KP + RK * kg + 2 * q;
                    const float2 cm = *reinterpret_cast<const float2*>(a.carry_M + e);
                    const float2 ci = *reinterpret_cast<const float2*>(a.carry_I + e);
                    GM[r][q] = cm;
                    nGI[r][q] = make_float2(-ci.x, -ci.y);
                }
            }

        // pairs of adjacent columns or rows: two 8-byte pairs go as one 16-byte access where the tiling allows it
        auto ld_pairs = [&](const float2* base, float2 (&dst)[NP]) __attribute__((always_inline)) {
            if constexpr (NP % 2 == 0) {
#pragma unroll
                for (int q = 0; q < NP; q += 2) {
                    const float4 x = *reinterpret_cast<const float4*>(base + q);
                    dst[q] = make_float2(x.x, x.y);
                    dst[q + 1] = make_float2(x.z, x.w);
                }
            } else {
#pragma unroll
                for (int q = 0; q < NP; ++q) dst[q] = base[q];
            }
        };
        // no memory operand: the next token's operands may be loaded above it (they lie elsewhere)
        auto st_pairs = [&](float2* base, const float2 (&src)[NP]) __attribute__((always_inline)) {
            if constexpr (NP % 2 == 0) {
#pragma unroll
                for (int q = 0; q < NP; q += 2)
                    asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(tc::smem_u32(base + q)), "f"(src[q].x), "f"(src[q].y),
                                 "f"(src[q + 1].x), "f"(src[q + 1].y));
            } else {
#pragma unroll
                for (int q = 0; q < NP; ++q)
                    asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(tc::smem_u32(base + q)), "f"(src[q].x), "f"(src[q].y));
            }
        };
        auto ld_rows = [&](const float2* base, float2 (&dst)[RV]) __attribute__((always_inline)) {
            if constexpr (RV % 2 == 0) {
#pragma unroll
                for (int r = 0; r < RV; r += 2) {
                    const float4 x = *reinterpret_cast<const float4*>(base + r);
                    dst[r] = make_float2(x.x, x.y);
                    dst[r + 1] = make_float2(x.z, x.w);
                }
            } else {
#pragma unroll
                for (int r = 0; r < RV; ++r) dst[r] = base[r];
            }
        };
        auto load_ck = [&](State<RV, NP>& s, int stage_idx) __attribute__((always_inline)) {
            const float2* ckM = reinterpret_cast<const float2*>(sm + L.ckb + stage_idx * L.ck_stage) + row0 * KP2 + NP * kg;
#pragma unroll
            for (int r = 0; r < RV; ++r) {
                ld_pairs(ckM + r * KP2, s.M[r]);
                ld_pairs(ckM + (TV + r) * KP2, s.I[r]);
                if (row0 + r >= tvw) {
#pragma unroll
                    for (int q = 0; q < NP; ++q) {
                        s.M[r][q] = make_float2(0.f, 0.f);
                        s.I[r][q] = make_float2(1.f, 1.f);
                    }
                }
            }
        };
        auto load_slot = [&](State<RV, NP>& s, int slot) {
            const float4* sl = slots4 + slot * (NE / 2) * NTHR;
#pragma unroll
            for (int r = 0; r < RV; ++r)
#pragma unroll
                for (int q = 0; q < NP; ++q) {
                    const float4 x = sl[(r * NP + q) * NTHR];
                    s.M[r][q] = make_float2(x.x, x.y);
                    s.I[r][q] = make_float2(x.z, x.w);
                }
        };
        auto store_slot = [&](const State<RV, NP>& s, int slot) {
            float4* sl = slots4 + slot * (NE / 2) * NTHR;
#pragma unroll
            for (int r = 0; r < RV; ++r)
#pragma unroll
                for (int q = 0; q < NP; ++q)
                    sl[(r * NP + q) * NTHR] = make_float4(s.M[r][q].x, s.M[r][q].y, s.I[r][q].x, s.I[r][q].y);
        };
        for (int it = 0; it < nblk; ++it) {
            const int st = it & 1;
            // this block's operand stage; this thread's d_k columns are RK*kg .. RK*kg+RK-1: pair q covers columns RK*kg + 2q, +1
            const unsigned char* op = sm + st * L.op_stage;
            const float2* ks2 = reinterpret_cast<const float2*>(op + L.ks) + NP * kg;
            const float2* qs2 = reinterpret_cast<const float2*>(op + L.qs) + NP * kg;
            const float4* vb4 = reinterpret_cast<const float4*>(op + L.vb) + row0;
            const float2* dys2 = reinterpret_cast<const float2*>(op + L.dys2) + row0;
            const float2* dyvs2 = reinterpret_cast<const float2*>(op + L.dyvs2) + row0;
            const float4* fc2 = reinterpret_cast<const float4*>(op + L.fc2);
            const float2* zz2 = reinterpret_cast<const float2*>(op + L.zz2);
            // one forward step of the recurrence on token tl of the staged block: P to s; `scaled`: its s may differ from 1
            auto fstep = [&](auto scaled, const State<RV, NP>& from, State<RV, NP>& s, int tl) __attribute__((always_inline)) {
                constexpr bool SCALED = decltype(scaled)::value == 2;
                const float4 fv = SCALED ? fc2[tl] : make_float4(1.f, 1.f, 0.f, 0.f);
                const float2 ff = make_float2(fv.x, fv.y), cc = make_float2(fv.z, fv.w);
                float2 kpv[NP], kk[NP];
                ld_pairs(ks2 + tl * KP2, kpv);
#pragma unroll
                for (int q = 0; q < NP; ++q) kk[q] = fmul2(kpv[q], kpv[q]);
#pragma unroll
                for (int r = 0; r < RV; ++r) {
                    const float4 x = vb4[tl * TV + r];
                    const float2 vr = make_float2(x.x, x.y), br = make_float2(x.z, x.w);
#pragma unroll
                    for (int q = 0; q < NP; ++q) {
                        s.M[r][q] = SCALED ? ffma2(ff, from.M[r][q], fmul2(vr, kpv[q])) : ffma2(vr, kpv[q], from.M[r][q]);
                        s.I[r][q] = SCALED ? ffma2(ff, from.I[r][q], ffma2(br, kk[q], cc)) : ffma2(br, kk[q], from.I[r][q]);
                    }
                }
            };
            if (!wait_fail && !tc::mbar_wait(&staged[st], (it >> 1) & 1)) wait_fail = 6;

            // Tokens past the end of the sequence (last block only) were staged as identity steps (f = 1,
            // all other operands 0): they leave the state and every gradient untouched, so the block is
            // always processed as NG full groups with no per-token conditionals.
            const float2 blk = *reinterpret_cast<const float2*>(op + L.blk);
            const unsigned special = __float_as_uint(blk.y);
            // Three copies of the walk: over a block of one window; of windows that begin in front of groups, whose scale is applied to
            // the state that the group finds; of any windows.
            static_assert(GR == 4, "the groups that block_scale begins windows in front of");
            auto edge = [&](State<RV, NP>& s, int g) __attribute__((always_inline)) {
                const float4 fv = fc2[g * GR];
                const float2 ff = make_float2(fv.x, fv.y), cc = make_float2(fv.z, fv.w);
#pragma unroll
                for (int r = 0; r < RV; ++r)
#pragma unroll
                    for (int q = 0; q < NP; ++q) {
                        s.M[r][q] = fmul2(ff, s.M[r][q]);
                        s.I[r][q] = ffma2(ff, s.I[r][q], cc);
                    }
            };
            auto block = [&](auto scaled) __attribute__((always_inline)) {
                constexpr bool EDGES = decltype(scaled)::value == 1, SCALED = decltype(scaled)::value == 2;
                // ---- forward sweep: park the start states of groups 1 .. NG-2, keep the last group's in registers
                State<RV, NP> P[GR + 1];
                load_ck(P[0], st);
#pragma unroll 1
                for (int g = 0; g < NG - 1; ++g) {
                    if (EDGES) edge(P[0], g);
#pragma unroll
                    for (int j = 0; j < GR; ++j) fstep(scaled, P[0], P[0], g * GR + j);
                    if (g < NG - 2) store_slot(P[0], g);
                }
                // the gradients of the block's end state become those of the last window's scaled state
#pragma unroll
                for (int r = 0; r < RV; ++r)
#pragma unroll
                    for (int q = 0; q < NP; ++q) {
                        GM[r][q] = fmul2(dup2(blk.x), GM[r][q]);
                        nGI[r][q] = fmul2(dup2(blk.x), nGI[r][q]);
                    }

                // Per group: the states of its four tokens from P[0] on, then the reverse walk over them.  A token that has
                // scaled the state it found, by s, scales the gradient on its way back.
#pragma unroll 1
                for (int gi = NG - 1; gi >= 0; --gi) {
                    if (gi == 0)
                        load_ck(P[0], st);
                    else if (gi < NG - 1)
                        load_slot(P[0], gi - 1);
                    if (EDGES) edge(P[0], gi);
                    const int b = gi & (KBUF - 1);
                    float red1[NR1], red2[NR2];
#pragma unroll
                    for (int j = 0; j < GR; ++j) fstep(scaled, P[j], P[j + 1], gi * GR + j);
#pragma unroll
                    for (int j = GR - 1; j >= 0; --j) {
                        const int tl = gi * GR + j;
                        const float2 z = zz2[tl];
                        const float s = SCALED ? fc2[tl].x : 1.f;
                        float2 dqs[NP], Ak[NP], Bk[NP], Uk[NP];
                        constexpr int RS = RV == 2 ? 2 : 1;  // accumulators: two shorten the dependent chains, three cost registers
                        float2 Sa[RS], Sb[RS], Sc[RS];
#pragma unroll
                        for (int r = 0; r < RS; ++r) Sa[r] = Sb[r] = Sc[r] = make_float2(0.f, 0.f);
                        auto add = [](bool first, float2& sum, float2 x, float2 y) __attribute__((always_inline)) { sum = first ? fmul2(x, y) : ffma2(x, y, sum); };
                        float2 kp[NP], kk[NP], qp[NP];
                        ld_pairs(ks2 + tl * KP2, kp);
                        ld_pairs(qs2 + tl * KP2, qp);
#pragma unroll
                        for (int q = 0; q < NP; ++q) kk[q] = fmul2(kp[q], kp[q]);
                        float2 dyr[RV], dyvr[RV];
                        ld_rows(dys2 + tl * TV, dyr);
#pragma unroll
                        for (int r = 0; r < RV; ++r) dyvr[r] = make_float2(0.f, 0.f);
                        if (UNC) ld_rows(dyvs2 + tl * TV, dyvr);
#pragma unroll
                        for (int r = 0; r < RV; ++r) {
                            const float4 x = vb4[tl * TV + r];
                            const float2 vv = make_float2(x.x, x.y), bv = make_float2(x.z, x.w);
                            const float2 dy = dyr[r];
                            const float2 dyv = dyvr[r];
                            float2 dva, dba;
#pragma unroll
                            for (int q = 0; q < NP; ++q) {
                                const float2 rr = rcp2(fadd2(P[j + 1].I[r][q], z));
                                const float2 mu = fmul2(P[j + 1].M[r][q], rr);
                                const float2 qr = UNC ? fmul2(qp[q], rr) : make_float2(0.f, 0.f);
                                const float2 hh = UNC ? fmul2(dy, qr) : fmul2(fmul2(dy, qp[q]), rr);
                                GM[r][q] = fadd2(GM[r][q], hh);
                                nGI[r][q] = ffma2(hh, mu, nGI[r][q]);
                                if (UNC) nGI[r][q] = ffma2(fmul2(dyv, qr), qr, nGI[r][q]);
                                if (!CO) {
                                    add(r == 0, dqs[q], dy, mu);
                                    if (UNC) add(r == 0, Uk[q], dyv, rr);
                                    add(r == 0, Ak[q], GM[r][q], vv);
                                    add(r == 0, Bk[q], nGI[r][q], bv);
                                    add(q == 0, dva, GM[r][q], kp[q]);
                                    add(q == 0, dba, nGI[r][q], kk[q]);
                                    add(r < RS && q == 0, Sa[r % RS], GM[r][q], P[j].M[r][q]);
                                    add(r < RS && q == 0, Sb[r % RS], nGI[r][q], P[j].I[r][q]);
                                    Sc[r % RS] = r < RS && q == 0 ? nGI[r][q] : fadd2(Sc[r % RS], nGI[r][q]);
                                }
                                if (SCALED) {
                                    GM[r][q] = fmul2(dup2(s), GM[r][q]);
                                    nGI[r][q] = fmul2(dup2(s), nGI[r][q]);
                                }
                            }
                            red1[(j * RV + r) * 2 + 0] = dva.x + dva.y;
                            red1[(j * RV + r) * 2 + 1] = dba.x + dba.y;  // of -GI, as the sum below: the helpers turn the sign
                        }
                        // this row group's share of dq (the helpers multiply it by the scale) and dk for the token -> shared memory
                        if (!CO) {
                            if (j == GR - 1)  // first write of the group: the helpers must be done with the buffer's last contents
                                if (!wait_fail && !tc::mbar_wait(&empty[b], (use & 1) ^ 1)) wait_fail = 6;  // after one failure: no more waiting
                            float2* dst = kred2 + b * (GR * WV * 2 * KP2) + ((j * WV + wv) * 2) * KP2 + NP * kg;
                            const float2 m2 = dup2(-2.f);
#pragma unroll
                            for (int q = 0; q < NP; ++q) {
                                if (UNC) dqs[q] = ffma2(fmul2(dup2(2.f), qp[q]), Uk[q], dqs[q]);
                                Ak[q] = ffma2(fmul2(m2, kp[q]), Bk[q], Ak[q]);
                            }
                            st_pairs(dst, dqs);
                            st_pairs(dst + KP2, Ak);
                        }
                        float2 sa = Sa[0], sb = Sb[0], scv = Sc[0];
#pragma unroll
                        for (int r = 1; r < RS; ++r) {
                            sa = fadd2(sa, Sa[r]);
                            sb = fadd2(sb, Sb[r]);
                            scv = fadd2(scv, Sc[r]);
                        }
                        const float sc_ = scv.x + scv.y;
                        const float fdf = (sa.x + sa.y) - (sb.x + sb.y) + iph * sc_;
                        red2[j * 2 + 0] = SCALED ? s * fdf : fdf;
                        red2[j * 2 + 1] = sc_;
                    }
                    if (EDGES) {
                        const float2 ff = dup2(fc2[gi * GR].x);
#pragma unroll
                        for (int r = 0; r < RV; ++r)
#pragma unroll
                            for (int q = 0; q < NP; ++q) {
                                GM[r][q] = fmul2(ff, GM[r][q]);
                                nGI[r][q] = fmul2(ff, nGI[r][q]);
                            }
                    }
                    if (!CO) {  // a carry-only pass wants nothing but the state gradients
                        // d_v-indexed sums over the KG lanes of a row; per-token scalars over the whole warp
                        xreduce<NR1, KG>(red1, lane);
                        {
                            const int base = xreduce_index<NR1, KG>(lane), count = xreduce_count<NR1, KG>(lane);
#pragma unroll
                            for (int i = 0; i < xreduce_most<NR1, KG>(); ++i)
                                if (i < count) {
                                    const int id = base + i;
                                    const int j = id / (RV * 2), r = (id / 2) % RV, which = id & 1;
                                    (which ? dbs : dvs)[(b * GR + j) * TV + row0 + r] = red1[i];
                                }
                        }
                        xreduce<NR2, 32>(red2, lane);
                        if ((lane & (32 / NR2 - 1)) == 0) {
                            const int id = xreduce_index<NR2, 32>(lane);
                            wred[((b * W + w) * GR + (id >> 1)) * 2 + (id & 1)] = red2[0];
                        }
                        if (tid < GR) fgr[b * GR + tid] = reinterpret_cast<const float2*>(op + L.fi2)[gi * GR + tid];
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&full[b]);  // this warp's partials of the group are written
                        if (b == 0) ++use;
                    }
                }
            };
            if (special == 0) block(std::integral_constant<int, 0>{});
            else if ((special & ~0x1111u) == 0) block(std::integral_constant<int, 1>{});
            else block(std::integral_constant<int, 2>{});
            __syncwarp();
            if (lane == 0) mbar_arrive(&done[st]);
        }

        if (wait_fail) *fail_flag = wait_fail;
        __syncthreads();
        const bool failed = *fail_flag != 0;
        if (tid == 0 && failed) {
            // a barrier wait ran out: record it and mark this CTA's results as invalid (NaN in the decay-gradient
            // partial of its first token, which the finishing kernels carry into dgt and dg; or in the state gradients below)
            atomicCAS(&g_bwd_status, 0, *fail_flag);
            if (!CO) a.df_part[(size_t)tile * a.rows_total + (size_t)((long long)bos + s0) * p.H + h] = __int_as_float(0x7fc00000);
        }

        // ---- gradient w.r.t. the segment's start state: that of the first window's ------------------------------
        if (a.rloc_M) {
            const float bad = failed ? __int_as_float(0x7fc00000) : 1.f;
#pragma unroll
            for (int r = 0; r < RV; ++r) {
                if (row0 + r < tvw) {
#pragma unroll
                    for (int q = 0; q < NP; ++q) {
                        const long long e = (seg_base + v0 + row0 + r) * KP + RK * kg + 2 * q;
                        *reinterpret_cast<float2*>(a.rloc_M + e) = make_float2(bad * GM[r][q].x, bad * GM[r][q].y);
                        *reinterpret_cast<float2*>(a.rloc_I + e) = make_float2(-bad * nGI[r][q].x, -bad * nGI[r][q].y);
                    }
                }
            }
        }
    };
    // The roles in two orders, for the register allocation that comes of it: with the uncertainty output and 6 or 4 warps of 12
    // elements the walk takes 302 us a wave (48x48, T = 512) with its code first and 319 with the helpers' first.
    if (UNC && w < W) {
        if constexpr (SPLIT.entry > 0) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SPLIT.compute));
        walk();
    } else if (UNC || w >= W) {
        if constexpr (SPLIT.entry > 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SPLIT.helper));
        help(tid - NTHR);
    } else {
        if constexpr (SPLIT.entry > 0) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SPLIT.compute));
        walk();
    }
}

// ---- finishing kernel 1 ----------------------------------------------------------------------------------
// CTAs from nb on: dq, dk = the row tiles' partials summed in tile order and cast.  A thread owns four consecutive
// columns of a row (16-byte loads, all tiles' loads independent); as many whole rows as fit share a CTA, so that no
// lane idles whatever d_k is.  The first nb CTAs: the per-token scalars of a strided share of the tokens, thread = (token
// lane, head): df and dIp terms summed over the tiles, dgt written, dg and dIp terms accumulated per head and reduced over
// the CTA's token lanes in a fixed order, in 64 bits: dg sums terms of both signs that may cancel to a few thousandths of what
// they add up to, and float sums left it off by 1.1e-5 where 64-bit ones leave 0.4e-5.  HBM-bound: 8 (KP tiles + 1) bytes read per (token, head), and K io values written
// twice.  With one warp per row, 48-column rows kept 12 of 32 lanes busy: 336 us at B=8 T=4096 H=16 d_k=d_v=48.
constexpr int FIN_THREADS = 256, FIN_SCALAR_CTAS = 148;

__device__ __forceinline__ void st4(void* base, long long idx, float4 x, int dt) {  // idx a multiple of 4, base aligned for it
    if (dt == PALIMPSA_F32) {
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(base) + idx) = x;
        return;
    }
    uint2 u;
    if (dt == PALIMPSA_BF16) {
        const __nv_bfloat162 a = __floats2bfloat162_rn(x.x, x.y), b = __floats2bfloat162_rn(x.z, x.w);
        u = make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
    } else {
        const __half2 a = __floats2half2_rn(x.x, x.y), b = __floats2half2_rn(x.z, x.w);
        u = make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
    }
    *reinterpret_cast<uint2*>(reinterpret_cast<unsigned short*>(base) + idx) = u;
}

__global__ void __launch_bounds__(FIN_THREADS)
bwd_finish_rows(const palimpsa_problem p, const float* __restrict__ dq_part, const float* __restrict__ dk_part,
                const float* __restrict__ df_part, const float* __restrict__ dip_part, void* dq, void* dk, float* dgt,
                double* w_dg, double* w_dip, int tiles, int tiles_k, int KP, long long rows, int vec, int nb) {
    const int tid = threadIdx.x;
    if ((int)blockIdx.x >= nb) {
        const int col_ctas = gridDim.x - nb;
        const int KP4 = KP / 4, rpc = FIN_THREADS / KP4, r = tid / KP4, c4 = tid - r * KP4, kc = 4 * c4;
        if (r >= rpc || kc >= p.K) return;
        const size_t step = (size_t)rows * KP4;
        for (long long row = (long long)(blockIdx.x - nb) * rpc + r; row < rows; row += (long long)col_ctas * rpc) {
            const float4* pq = reinterpret_cast<const float4*>(dq_part) + (size_t)row * KP4 + c4;
            const float4* pk = reinterpret_cast<const float4*>(dk_part) + (size_t)row * KP4 + c4;
            float4 sq = make_float4(0.f, 0.f, 0.f, 0.f), sk = sq;
#pragma unroll 6
            for (int t = 0; t < tiles; ++t) {
                const float4 x = __ldcs(pq + t * step), y = __ldcs(pk + t * step);
                sq.x += x.x, sq.y += x.y, sq.z += x.z, sq.w += x.w;
                sk.x += y.x, sk.y += y.y, sk.z += y.z, sk.w += y.w;
            }
            if (tiles_k > tiles) {  // dk has one slot more than dq: the carried-gradient terms
                const float4 y = pk[tiles * step];
                sk.x += y.x, sk.y += y.y, sk.z += y.z, sk.w += y.w;
            }
            if (vec) {  // K a multiple of 4, dq and dk aligned for four values
                st4(dq, row * p.K + kc, sq, p.io_dtype);
                st4(dk, row * p.K + kc, sk, p.io_dtype);
            } else {
                const float q4[4] = {sq.x, sq.y, sq.z, sq.w}, k4[4] = {sk.x, sk.y, sk.z, sk.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (kc + i < p.K) {
                        st1(dq, row * p.K + kc + i, q4[i], p.io_dtype);
                        st1(dk, row * p.K + kc + i, k4[i], p.io_dtype);
                    }
            }
        }
        return;
    }
    __shared__ double red[2][FIN_THREADS];
    const int b = blockIdx.x, H = p.H;
    const long long tokens = rows / H;
    const int lanes = H <= FIN_THREADS ? FIN_THREADS / H : 1;  // token lanes
    for (int h0 = 0; h0 < H; h0 += FIN_THREADS) {              // one turn unless there are more heads than threads
        const int lane = H <= FIN_THREADS ? tid / H : 0, h = h0 + (H <= FIN_THREADS ? tid - lane * H : tid);
        double a0 = 0., a1 = 0.;
        if (lane < lanes && h < H) {
            const float gh = p.g[h];
            for (long long tok = (long long)b * lanes + lane; tok < tokens; tok += (long long)nb * lanes) {
                const long long row = tok * H + h;
                double df = 0., dip = 0.;
#pragma unroll 4
                for (int t = 0; t < tiles_k; ++t) {
                    df += df_part[(size_t)t * rows + row];
                    dip += dip_part[(size_t)t * rows + row];
                }
                dgt[row] = -gh * (float)df;
                a0 -= p.gt[row] * df;
                a1 += dip;
            }
        }
        red[0][tid] = a0;
        red[1][tid] = a1;
        for (int n = lanes; n > 1; n = (n + 1) / 2) {  // lanes of the upper half join those of the lower
            const int upper = lane + (n + 1) / 2;
            __syncthreads();
            if (upper < n && h < H) {
                red[0][tid] = a0 += red[0][upper * H + h];
                red[1][tid] = a1 += red[1][upper * H + h];
            }
        }
        if (lane == 0 && h < H) {
            w_dg[(size_t)b * H + h] = a0;
            w_dip[(size_t)b * H + h] = a1;
        }
        __syncthreads();
    }
}

// ---- finishing kernel 2: one warp per head, ordered sum over the scalar CTAs' partials -------------------------
__global__ void __launch_bounds__(32) bwd_finish_heads(const double* __restrict__ w_dg, const double* __restrict__ w_dip,
                                                       float* dg, float* dIp, int nb, int H) {
    const int h = blockIdx.x, lane = threadIdx.x;
    double a0 = 0., a1 = 0.;
    for (int b = lane; b < nb; b += 32) {
        a0 += w_dg[(size_t)b * H + h];
        a1 += w_dip[(size_t)b * H + h];
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        a0 += __shfl_xor_sync(0xffffffffu, a0, off);
        a1 += __shfl_xor_sync(0xffffffffu, a1, off);
    }
    if (lane == 0) {
        dg[h] = (float)a0;
        dIp[h] = (float)a1;
    }
}

// -------------------------------------------------------------------------------------------------
// Host side
// -------------------------------------------------------------------------------------------------
// Thread tilings: RK columns x KG lanes of a row, by padded d_k.
struct BwdShape {
    int RK, KG;
};
static BwdShape bwd_shape(int KP) {
    switch (KP) {
        case 16: return {2, 8};
        case 32: return {4, 8};
        case 48: return {6, 8};
        case 64: return {4, 16};
        case 96: return {6, 16};
        case 128: return {4, 32};
        case 192: return {6, 32};
        case 256: return {8, 32};
        default: return {0, 0};
    }
}
// Tile heights a CTA may have at each tiling, as W compute warps of RV rows a thread (launch_bwd_t instantiates these); a
// tile lower than its warps hold leaves the last ones idle.  8 warps of 3 rows hold 24 (48 at d_k = 64): 22 (44) rows cost them
// the same and come first, for the tiles of a d_v that both cut into as many.
struct BwdTile {
    int rows, RV, W;
};
static const BwdTile* bwd_tile_choices(int KP) {
    static const BwdTile k16[] = {{64, 2, 8}, {32, 2, 4}, {}}, k48[] = {{64, 2, 8}, {48, 2, 6}, {32, 2, 4}, {}},
                         k64[] = {{44, 3, 8}, {32, 2, 8}, {16, 2, 4}, {}}, k96[] = {{32, 2, 8}, {24, 2, 6}, {16, 2, 4}, {}},
                         k128[] = {{22, 3, 8}, {24, 3, 8}, {16, 2, 8}, {8, 2, 4}, {}},
                         k192[] = {{16, 2, 8}, {12, 2, 6}, {8, 2, 4}, {}}, k256[] = {{8, 1, 8}, {}};
    switch (KP) {
        case 48: return k48;
        case 64: return k64;
        case 96: return k96;
        case 128: return k128;
        case 192: return k192;
        case 256: return k256;
        default: return k16;
    }
}
// What a token costs a CTA (the walk, and what does not grow with the rows), in units of which 4 warps take 8.  One wave, T =
// 512, bf16, us at 4 / 6 / 8 warps (8 of 3 rows): d_k = 48 190 / 254 / 330, 96 181 / 247 / 328, 192 189 / 263 / 349, 64 146 / - / 216
// (286), 128 149 / - / 229 (272), 32 170 / - / 220, 16 117 / - / 165, 256 - / - / 374.  With the uncertainty output 204 / 300 / 362,
// 211 / 273 / 363, 211 / 284 / 388, 161 / - / 233 (322), 167 / - / 249 (302), 163 / - / 244, 129 / - / 187, - / - / 363.  The
// state-gradient pass of exact segments takes 0.45 to 0.55 of that at every height.  The costs are those before the scaled form
// (d_k = 64: 151, 230, 285), with which the planner's cuts were fitted; where they are off most, 44 rows of d_k = 64, the choice is even:
// three waves of 286 at d_v = 128, four of 216 with 32 rows (B=8 T=4096 H=16: 6.75 ms, 6.83 before the scaled form, 7.2 while 44 rows took 314).
static double bwd_tile_cost(const BwdTile& t, int KP, int NE, bool unc) {
    if (t.RV == 3) return KP == 64 ? (unc ? 17.2 : 15.1) : unc ? 16.4 : 15.7;
    return t.W == 4 ? 8 : t.W == 6 ? 11 : NE == 12 ? 14.2 : 12;
}
struct BwdConfig {
    BwdShape s;
    BwdTile t;
    int smem, kbuf;
    double cost;
};
// The choice that costs least: waves of CTAs (one per SM) times the cost of a token.  CTAs of equal sequences, or of their
// equal segments, finish together, so their waves are whole ones.
static BwdConfig bwd_config(const palimpsa_problem& p) {
    BwdConfig best{};
    best.s = bwd_shape(palimpsa_padded_k(p.K));
    if (!best.s.RK) return best;
    const BwdShape s = best.s;
    const int VG = 32 / s.KG, KP = s.RK * s.KG;
    const bool unc = (p.flags & PALIMPSA_FLAG_UNCERTAINTY) != 0;
    const double units = (double)p.num_seqs * p.H;
    for (const BwdTile* t = bwd_tile_choices(KP); t->W; ++t) {
        BwdConfig c{s, *t, 0, 0, 0};
        for (c.kbuf = 2;; c.kbuf = 1) {
            c.smem = bwd_smem_layout(KP, t->W * VG * t->RV, t->RV * s.RK, t->W, t->W * VG, unc, c.kbuf).total;
            if (c.kbuf == 1 || c.smem <= 227 * 1024) break;
        }
        if (c.smem > 227 * 1024) continue;
        const int tiles = (p.V + t->rows - 1) / t->rows;
        const bool cut = p.segments > 1;
        const double cost = bwd_tile_cost(*t, KP, t->RV * s.RK, unc);
        const double share = (units > 0 ? units : 1) * tiles / B200_SMS;  // of a wave, per segment
        if (p.segments == BWD_FEWEST_TILES) {
            c.cost = 1000.0 * tiles + cost;
        } else if (p.cu_seqlens || units == 0 || p.segments == 2) {
            // documents fill the waves up, beyond the first few; no grid given, or two segments: a share of many waves
            c.cost = (units > 0 && !cut && share <= 3 ? ceil(share) : share) * cost;
        } else {
            const int G = cut ? p.segments : 1, per = ((p.seq_len + G - 1) / G + TB - 1) / TB * TB;
            const double full = cut && per > 0 ? (double)p.seq_len / per : G;  // segments, the last one by its share
            c.cost = (ceil(share * full) + 1e-3 * share * full) * cost / G;       // of equal waves the fuller ones
        }
        if (!best.t.W || c.cost < best.cost) best = c;
    }
    return best;
}

double bwd_token_cost(const palimpsa_problem& p) { return bwd_config(p).cost; }

int bwd_tile_rows(const palimpsa_problem& p) {
    return bwd_config(p).t.rows;  // 0: nothing fits
}

void bwd_plan(const palimpsa_problem& p, int32_t* plan) {
    const BwdConfig c = bwd_config(p);
    plan[0] = c.t.rows, plan[1] = c.t.W, plan[2] = c.kbuf;
}

BwdWorkspace bwd_workspace_layout(const palimpsa_problem& p) {
    BwdWorkspace ws{};
    ws.KP = palimpsa_padded_k(p.K);
    const int TV = bwd_tile_rows(p);
    if (!TV) return ws;
    ws.tiles = (p.V + TV - 1) / TV;
    const size_t rows = (size_t)p.total_tokens * p.H;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        size_t o = off;
        off += (bytes + 255) / 256 * 256;
        return o;
    };
    ws.dq_part = take((size_t)ws.tiles * rows * ws.KP * 4);
    // one slot more than there are row tiles: the carried-gradient terms of a segmented backward go there
    ws.dk_part = take((size_t)(ws.tiles + 1) * rows * ws.KP * 4);
    ws.df_part = take((size_t)(ws.tiles + 1) * rows * 4);
    ws.dip_part = take((size_t)(ws.tiles + 1) * rows * 4);
    ws.w_dg = take((size_t)FIN_SCALAR_CTAS * p.H * 8);
    ws.w_dip = take((size_t)FIN_SCALAR_CTAS * p.H * 8);
    ws.total = off;
    return ws;
}

// Does the compiled kernel start with the registers its split was made for?  (Fewer, and the wait for the compute warps'
// share would not end.)  Asked once: a property of the binary.
template <auto Kern>
static bool bwd_split_fits(RegSplit split) {
    if (!split.entry) return true;
    static std::atomic<int> regs{0};
    int r = regs.load(std::memory_order_relaxed);
    if (!r) {
        cudaFuncAttributes attr;
        if (cudaFuncGetAttributes(&attr, Kern) != cudaSuccess) return false;
        regs.store(r = attr.numRegs, std::memory_order_relaxed);
    }
    return r == split.entry;
}

template <int RK, int KG, int RV, int W>
static int launch_bwd_w(const BwdArgs& a, int tiles, int num_seg, bool carry_only, cudaStream_t stream) {
    constexpr int VG = 32 / KG, TV = W * VG * RV;
    const palimpsa_problem& p = a.p;
    const bool unc = (p.flags & PALIMPSA_FLAG_UNCERTAINTY) != 0;
    const BwdSmem L = bwd_smem_layout(RK * KG, TV, RV * RK, W, W * VG, unc, a.kbuf);
    if (L.total > 227 * 1024) return PALIMPSA_E_DIM;
    dim3 grid(tiles, p.num_seqs * p.H, num_seg);
    dim3 block(bwd_threads(W), 1, 1);
#define PALIMPSA_BWD_LAUNCH(U, C)                                                                                 \
    do {                                                                                                          \
        if (!allow_smem<bwd_kernel<RK, KG, RV, W, U, C>>(L.total)) return PALIMPSA_E_LAUNCH;                        \
        if (!bwd_split_fits<bwd_kernel<RK, KG, RV, W, U, C>>(bwd_split(W, RV, RK))) return PALIMPSA_E_LAUNCH;    \
        bwd_kernel<RK, KG, RV, W, U, C><<<grid, block, L.total, stream>>>(a);                                     \
    } while (0)
    if (carry_only) {
        if (unc) PALIMPSA_BWD_LAUNCH(true, true); else PALIMPSA_BWD_LAUNCH(false, true);
    } else {
        if (unc) PALIMPSA_BWD_LAUNCH(true, false); else PALIMPSA_BWD_LAUNCH(false, false);
    }
#undef PALIMPSA_BWD_LAUNCH
    return cudaGetLastError() == cudaSuccess ? PALIMPSA_OK : PALIMPSA_E_LAUNCH;
}

template <int RK, int KG>
static int launch_bwd_t(const BwdArgs& args, int tiles, int num_seg, bool carry_only, cudaStream_t stream) {
    const BwdConfig cfg = bwd_config(args.p);
    BwdArgs a = args;
    a.rows = cfg.t.rows;
    a.kbuf = cfg.kbuf;
#define PALIMPSA_W(rv, n)                                                                                \
    if (cfg.t.W == n && cfg.t.RV == rv) return launch_bwd_w<RK, KG, rv, n>(a, tiles, num_seg, carry_only, stream)
    constexpr int KP = RK * KG;
    if constexpr (KP == 256) {
        PALIMPSA_W(1, 8);
    } else {
        PALIMPSA_W(2, 8);
        PALIMPSA_W(2, 4);
    }
    if constexpr (RK == 6) PALIMPSA_W(2, 6);
    if constexpr (KP == 64 || KP == 128) PALIMPSA_W(3, 8);
#undef PALIMPSA_W
    return PALIMPSA_E_DIM;
}

int bwd_wait_status() {
    int s = 0;
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    if (cudaMemcpyFromSymbol(&s, g_bwd_status, sizeof(int)) != cudaSuccess) return -1;
    if (s) {
        const int zero = 0;
        if (cudaMemcpyToSymbol(g_bwd_status, &zero, sizeof(int)) != cudaSuccess) return -1;
    }
    return s;
}

int launch_bwd(const palimpsa_bwd_params* prm, const palimpsa_segments* segs, bool carry_only, cudaStream_t stream,
               int stages) {
    const palimpsa_problem& p = prm->p;
    const BwdWorkspace ws = bwd_workspace_layout(p);
    if (!ws.tiles) return PALIMPSA_E_DIM;
    char* base = reinterpret_cast<char*>(prm->workspace);
    BwdArgs a{};
    a.p = p;
    int num_seg = 1;
    if (segs) {
        num_seg = segs->num_segments;
        a.seg_len = segs->seg_len;
        a.carry_M = carry_only ? nullptr : segs->carry_M;
        a.carry_I = carry_only ? nullptr : segs->carry_I;
        a.rloc_M = segs->rloc_M;
        a.rloc_I = segs->rloc_I;
    }
    if (carry_only) stages = 1;
    a.d_o = prm->d_o;
    a.d_o_var = (p.flags & PALIMPSA_FLAG_UNCERTAINTY) ? prm->d_o_var : nullptr;
    a.ckpt_M = prm->ckpt_M;
    a.ckpt_I = prm->ckpt_I;
    a.dq_part = reinterpret_cast<float*>(base + ws.dq_part);
    a.dk_part = reinterpret_cast<float*>(base + ws.dk_part);
    a.df_part = reinterpret_cast<float*>(base + ws.df_part);
    a.dip_part = reinterpret_cast<float*>(base + ws.dip_part);
    a.dv = prm->dv;
    a.db = prm->db;
    a.rows_total = p.total_tokens * p.H;
    const int es = dtype_size(p.io_dtype);
    const auto starts_on = [](std::initializer_list<const void*> ptrs, int bytes) {
        for (const void* x : ptrs)
            if (reinterpret_cast<uintptr_t>(x) & (bytes - 1)) return false;
        return true;
    };
    a.vec_k = p.K % 4 == 0 && starts_on({p.q, p.k}, 4 * es);
    a.vec_v = p.V % 2 == 0 && starts_on({p.v, p.b, a.d_o, a.d_o_var}, 2 * es);  // tiles start on even rows
    int rc = PALIMPSA_OK;
    if (stages & 1) switch (ws.KP) {
        case 16: rc = launch_bwd_t<2, 8>(a, ws.tiles, num_seg, carry_only, stream); break;
        case 32: rc = launch_bwd_t<4, 8>(a, ws.tiles, num_seg, carry_only, stream); break;
        case 48: rc = launch_bwd_t<6, 8>(a, ws.tiles, num_seg, carry_only, stream); break;
        case 64: rc = launch_bwd_t<4, 16>(a, ws.tiles, num_seg, carry_only, stream); break;
        case 96: rc = launch_bwd_t<6, 16>(a, ws.tiles, num_seg, carry_only, stream); break;
        case 128: rc = launch_bwd_t<4, 32>(a, ws.tiles, num_seg, carry_only, stream); break;
        case 192: rc = launch_bwd_t<6, 32>(a, ws.tiles, num_seg, carry_only, stream); break;
        case 256: rc = launch_bwd_t<8, 32>(a, ws.tiles, num_seg, carry_only, stream); break;
        default: return PALIMPSA_E_DIM;
    }
    if (rc != PALIMPSA_OK) return rc;
    if (!(stages & 2)) return PALIMPSA_OK;
    const long long rows = a.rows_total;
    int nb = 0;
    if (rows > 0) {
        const int rpc = FIN_THREADS / (ws.KP / 4), lanes = p.H <= FIN_THREADS ? FIN_THREADS / p.H : 1;
        const long long groups = (rows + rpc - 1) / rpc, tgroups = (p.total_tokens + lanes - 1) / lanes;
        const int col_ctas = (int)(groups < B200_SMS * 32 ? groups : B200_SMS * 32);
        nb = (int)(tgroups < FIN_SCALAR_CTAS ? tgroups : FIN_SCALAR_CTAS);
        const uintptr_t both = reinterpret_cast<uintptr_t>(prm->dq) | reinterpret_cast<uintptr_t>(prm->dk);
        bwd_finish_rows<<<col_ctas + nb, FIN_THREADS, 0, stream>>>(
            p, a.dq_part, a.dk_part, a.df_part, a.dip_part, prm->dq, prm->dk, prm->dgt,
            reinterpret_cast<double*>(base + ws.w_dg), reinterpret_cast<double*>(base + ws.w_dip), ws.tiles,
            ws.tiles + ((stages & 4) ? 1 : 0), ws.KP, rows, p.K % 4 == 0 && (both & (4 * es - 1)) == 0, nb);
        if (cudaGetLastError() != cudaSuccess) return PALIMPSA_E_LAUNCH;
    }
    bwd_finish_heads<<<p.H, 32, 0, stream>>>(reinterpret_cast<double*>(base + ws.w_dg),
                                             reinterpret_cast<double*>(base + ws.w_dip), prm->dg, prm->dIp, nb, p.H);
    return cudaGetLastError() == cudaSuccess ? PALIMPSA_OK : PALIMPSA_E_LAUNCH;
}

// ---- backward with library-owned scratch -----------------------------------------------------------
// For callers that cannot allocate device memory themselves: the partial-sum scratch of the backward
// lives in this fixed array instead of a caller-provided workspace.  Every device on which the library's
// backward code gets loaded (primary context) carries the array from then until the process exits.  Host code may not use the array's name as an address; the
// device address is looked up once per device below.
static __device__ __align__(256) unsigned char g_static_scratch[PALIMPSA_STATIC_SCRATCH_BYTES];

int launch_bwd_static(const palimpsa_bwd_params* prm, cudaStream_t stream) {
    constexpr int MAX_DEV = 64;
    static void* addr[MAX_DEV] = {};
    static std::mutex mu;
    palimpsa_bwd_params local = *prm;
    BwdWorkspace ws = bwd_workspace_layout(local.p);
    if (ws.total > (size_t)PALIMPSA_STATIC_SCRATCH_BYTES) {  // short tiles for a small grid, too many of them: take tall ones
        local.p.segments = BWD_FEWEST_TILES;
        ws = bwd_workspace_layout(local.p);
    }
    if (!ws.tiles) return PALIMPSA_E_DIM;
    if (ws.total > (size_t)PALIMPSA_STATIC_SCRATCH_BYTES) return PALIMPSA_E_LIMIT;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEV) return PALIMPSA_E_LAUNCH;
    void* ptr = nullptr;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!addr[dev]) {
            void* sym = nullptr;
            // may be the call that loads this module on the device (lazy loading): the array is reserved now,
            // and a device without 96 MiB to spare fails here
            if (cudaGetSymbolAddress(&sym, g_static_scratch) != cudaSuccess || !sym) {
                (void)cudaGetLastError();
                return PALIMPSA_E_SYMBOL;
            }
            addr[dev] = sym;
        }
        ptr = addr[dev];
    }
    local.workspace = ptr;
    local.workspace_bytes = PALIMPSA_STATIC_SCRATCH_BYTES;
    return launch_bwd(&local, nullptr, false, stream, 3);
}

}  // namespace palimpsa
