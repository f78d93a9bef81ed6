// Forward kernel of the Palimpsa operator for tall row tiles (sm_100a): one CTA per SM.
//
// fwd.cu's kernel runs CTAs of at most 4 warps, several per SM, each of which converts the q and k rows of its head for
// itself, between two CTA barriers per 16 tokens.  Here up to 12 compute warps share one tile: a block's operands are
// converted once per SM, by helper warps, one block ahead of the walk, and the compute warps meet no barrier: they wait for
// the staged block (an mbarrier), walk its 16 tokens with the state in registers, and hand the reduced outputs back the same
// way.  The floor is the MUFU pipe: a pair of state elements takes two reciprocals, 16 cycles of it, per token.  What keeps the
// kernel from that floor is the issue rate: the pair's packed FP32 instructions take 11 issue cycles (2.05 measured for FMUL2, 2.3 for
// FFMA2 with a shared operand), and the rest of a token (operand loads, the sums over a row's lanes) and the helper warps come on top.
// Forward with checkpoints, ms, fwd.cu's kernel -> this one with the decay in every step -> in the scaled form (block_scale in
// common.cuh; 5 packed operations a pair instead of 6) -> with 2 rows of 6 or 8 columns a thread where it had one row of 12 or 16
// (d_k other than 128: half the operand loads and squares of k per element, for one more value to sum over the lanes): B=8 T=4096
// H=6 d=128 1.49 -> 1.26 -> 1.16, H=16 d=48 1.11 -> 0.84 -> 0.81 -> 0.71 (1 row of 6 there: launch_tall_t), B=4 T=2048 H=16 96x192
// 1.31 -> 1.03 -> 0.97 -> 0.95, with the uncertainty output 1.31 -> 1.31 -> 1.15; without checkpoints: B=2 T=3001 H=16 96x192
// 1.07 -> 0.73 -> 0.68 -> 0.66, B=4 T=2048 H=6 256x128 0.64 -> 0.59 -> 0.57.
//
//   thread layout   lane = vg*KG + kg, as in fwd.cu: RV rows x RK columns, interleaved float4 column groups, or halves of them
//                   where a lane has 6 columns.
//   blocks          16 tokens; tokens past the end are staged as identity steps (f = 1, all else 0), so that the walk has
//                   no conditionals.  Groups in which a token scales the state take a second copy of the walk.
//   warps without rows (a tile lower than 12 warps hold) only keep the hand-overs going.
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "fwd.h"
#include "tc_common.cuh"

namespace palimpsa {

// 0 ok; 8: a bounded wait of the tall-tile forward gave up
__device__ int g_fwd_status = 0;

constexpr int FT_W = 12, FT_HW = 4, FT_NTHR = 32 * FT_W, FT_HT = 32 * FT_HW;

struct TallSmem {
    int qs, ks, qqs, vb, fc, zz, blk, op_stage;  // offsets inside an operand stage; two stages from 0
    int ys, yvs, y_stage;               // reduced outputs, two stages
    int bars;                           // staged[2], done[2]; failure flag
    int raw, rq, rk, rv, rb;
    int total;
};

// v and b of a row lie side by side, each value twice: one 128-bit load yields both packed operands.
__host__ __device__ inline TallSmem tall_smem_layout(int KP, int TV, int es, bool unc) {
    TallSmem s;
    int off = 0;
    auto take = [&](int bytes) {
        int o = off;
        off += round_up(bytes, 16);
        return o;
    };
    s.qs = take(TB * KP * 4);
    s.ks = take(TB * KP * 4);
    s.qqs = unc ? take(TB * KP * 4) : 0;
    s.vb = take(TB * TV * 16);
    s.fc = take(TB * 16);  // {s, s, c, c}
    s.zz = take(TB * 8);   // {Z, Z}
    s.blk = take(16);      // BlockScale::end, special
    s.op_stage = off;
    off *= 2;
    s.ys = off;
    s.yvs = s.ys + TB * TV * 4;
    s.y_stage = TB * TV * 4 * (unc ? 2 : 1);
    off += 2 * s.y_stage;
    s.bars = take(48);
    s.raw = off;
    int r = 0;
    auto rtake = [&](int bytes) {
        int o = r;
        r += round_up(bytes, 16);
        return o;
    };
    s.rq = rtake(TB * KP * es);
    s.rk = rtake(TB * KP * es);
    s.rv = rtake(TB * TV * es);
    s.rb = rtake(TB * TV * es);
    s.total = off + r;
    return s;
}

// Asynchronous copies of one block of nt tokens by the helper warps (aligned rows only).
__device__ __forceinline__ void tall_issue(const FwdArgs& a, int ht, unsigned char* stage, const TallSmem& L, int es, int KP,
                                           int TV, long long tok0, int nt, int h, int v0, int tvw) {
    const palimpsa_problem& p = a.p;
    const int cq = p.K * es / 16, cv = tvw * es / 16;
    const char* gq = reinterpret_cast<const char*>(p.q);
    const char* gk = reinterpret_cast<const char*>(p.k);
    const char* gv = reinterpret_cast<const char*>(p.v);
    const char* gb = reinterpret_cast<const char*>(p.b);
    for (int i = ht; i < nt * cq; i += FT_HT) {
        const int t = i / cq, c = i - t * cq;
        const long long src = ((tok0 + t) * p.H + h) * (long long)p.K * es + c * 16;
        const int dst = t * KP * es + c * 16;
        cp_async16(stage + L.rq + dst, gq + src);
        cp_async16(stage + L.rk + dst, gk + src);
    }
    for (int i = ht; i < nt * cv; i += FT_HT) {
        const int t = i / cv, c = i - t * cv;
        const long long src = (((tok0 + t) * p.H + h) * (long long)p.V + v0) * es + c * 16;
        const int dst = t * TV * es + c * 16;
        cp_async16(stage + L.rv + dst, gv + src);
        cp_async16(stage + L.rb + dst, gb + src);
    }
}

// One block of fp32 operands (v and b times w: block_scale), by the helper warps.  ALIGNED: from the raw stage;
// otherwise element by element from global memory (any K, V, alignment).
template <int DT, bool ALIGNED, bool UNC, int KP, int TV>
__device__ __forceinline__ void tall_convert(const FwdArgs& a, int ht, const unsigned char* raw, unsigned char* op,
                                             const TallSmem& L, long long tok0, int nt, int h, int v0, int tvw,
                                             const BlockScale& bs, int half) {  // half: the block's first lane in bs
    const palimpsa_problem& p = a.p;
    constexpr int K4 = KP / 4, V4 = TV / 4;
    float4* qs = reinterpret_cast<float4*>(op + L.qs);
    float4* ks = reinterpret_cast<float4*>(op + L.ks);
    float4* qqs = reinterpret_cast<float4*>(op + L.qqs);
    if ((ht ^ half) < TB) {
        const int t = ht ^ half;
        reinterpret_cast<float4*>(op + L.fc)[t] = make_float4(bs.s, bs.s, bs.c, bs.c);
        reinterpret_cast<float2*>(op + L.zz)[t] = make_float2(bs.z, bs.z);
        if (t == 0) *reinterpret_cast<float2*>(op + L.blk) = make_float2(bs.end, __uint_as_float(bs.special));
    }
    const float sc = p.scale;
#pragma unroll 2
    for (int i0 = 0; i0 < TB * K4; i0 += FT_HT) {
        const int i = i0 + ht, t = i / K4, c4 = i - t * K4;
        const float scv = UNC ? sc * __shfl_sync(0xffffffffu, bs.w, half | (t & 15)) : 0.f;
        if (i >= TB * K4) break;
        float4 qv = make_float4(0.f, 0.f, 0.f, 0.f), kv = qv;
        if (t < nt && c4 * 4 < p.K) {
            if (ALIGNED) {
                qv = ld4<DT>(raw + L.rq, i);
                kv = ld4<DT>(raw + L.rk, i);
            } else {
                const long long row = ((tok0 + t) * p.H + h) * (long long)p.K;
                qv = ld4_guarded<DT>(p.q, row + c4 * 4, row + p.K);
                kv = ld4_guarded<DT>(p.k, row + c4 * 4, row + p.K);
            }
        }
        qs[i] = make_float4(qv.x * sc, qv.y * sc, qv.z * sc, qv.w * sc);
        ks[i] = kv;
        if (UNC) qqs[i] = make_float4(scv * qv.x * qv.x, scv * qv.y * qv.y, scv * qv.z * qv.z, scv * qv.w * qv.w);
    }
    float4* vb = reinterpret_cast<float4*>(op + L.vb);
#pragma unroll 2
    for (int i0 = 0; i0 < TB * V4; i0 += FT_HT) {
        const int i = i0 + ht, t = i / V4, r = 4 * (i - t * V4);
        const float wt = __shfl_sync(0xffffffffu, bs.w, half | (t & 15));
        if (i >= TB * V4 || r >= tvw) continue;  // rows past the tile belong to idle warps, or are never written out
        float4 vv = make_float4(0.f, 0.f, 0.f, 0.f), bv = vv;
        if (t < nt) {
            if (ALIGNED) {
                vv = ld4<DT>(raw + L.rv, i);
                bv = ld4<DT>(raw + L.rb, i);
            } else {
                const long long row = ((tok0 + t) * p.H + h) * (long long)p.V + v0;
                vv = ld4_guarded<DT>(p.v, row + r, row + tvw);
                bv = ld4_guarded<DT>(p.b, row + r, row + tvw);
            }
        }
        vv = make_float4(vv.x * wt, vv.y * wt, vv.z * wt, vv.w * wt);
        bv = make_float4(bv.x * wt, bv.y * wt, bv.z * wt, bv.w * wt);
        vb[4 * i] = make_float4(vv.x, vv.x, bv.x, bv.x);
        vb[4 * i + 1] = make_float4(vv.y, vv.y, bv.y, bv.y);
        vb[4 * i + 2] = make_float4(vv.z, vv.z, bv.z, bv.z);
        vb[4 * i + 3] = make_float4(vv.w, vv.w, bv.w, bv.w);
    }
}

// Tokens whose outputs are summed together over a row's lanes: as many as give each of the KG lanes one sum, 4 to 8.
template <int KG, int RV, bool UNC>
__host__ __device__ constexpr int tall_group() {
    constexpr int g = KG / (RV * (UNC ? 2 : 1));
    return g < 8 ? 4 : 8;
}

template <int RK, int KG, int RV, bool UNC, unsigned POLLS = tc::SPIN_LIMIT>
__global__ void __launch_bounds__(FT_NTHR + FT_HT, 1) fwd_tall_kernel(const FwdArgs a, const int rows) {
    constexpr int KP = RK * KG, VG = 32 / KG, CW = RK % 4 ? 2 : 4, J = RK / CW, E = CW / 2, TV = FT_W * VG * RV, GF = tall_group<KG, RV, UNC>();
    constexpr int NRED = GF * RV * (UNC ? 2 : 1);
    static_assert(TV % 8 == 0 && TB % GF == 0, "raw rows of 16-bit values start on 16 bytes, blocks are whole groups");
    extern __shared__ __align__(16) unsigned char sm[];
    const palimpsa_problem& p = a.p;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int kg = lane % KG, vg = lane / KG;
    // Columns of a lane: groups of four, every KG-th; with two columns a group the lanes of the upper half have the second half of
    // the groups of those of the lower.
    constexpr int GS = CW == 4 ? 4 * KG : 2 * KG;  // from one group of a lane to its next
    const int col0 = CW == 4 ? 4 * kg : 4 * (kg % (KG / 2)) + 2 * (kg / (KG / 2));
    const int row0 = (w * VG + vg) * RV;
    const int ny = blockIdx.y / p.H, h = blockIdx.y - ny * p.H;
    const int n = p.seq_order ? p.seq_order[ny] : ny;  // blocks start in grid order: a packed batch lists its longest sequences first
    const int v0 = blockIdx.x * rows;
    const int tvw = min(rows, p.V - v0);
    const int es = dtype_size(p.io_dtype);
    const TallSmem L = tall_smem_layout(KP, TV, es, UNC);
    int bos, len;
    seq_range(p, n, bos, len);
    const float gh = p.g[h], iph = p.Ip[h];
    const int K = p.K, V = p.V;
    const bool vecK = (K % 4) == 0;
    // this CTA's segment of the sequence: tokens [s0, s1)
    const int g = blockIdx.z, G = gridDim.z;
    const int s0 = a.seg_len > 0 ? min(len, g * a.seg_len) : 0;
    const int s1 = a.seg_len > 0 ? min(len, s0 + a.seg_len) : len;
    const int blk0 = s0 / TB, nblk = s1 > s0 ? (s1 + TB - 1) / TB - blk0 : 0;

    // staged[s] / done[s], s = block & 1: its operands lie in shared memory (one arrival per helper warp); the compute warps
    // are through with it and its outputs lie in shared memory (one per compute warp).  All waits are bounded (POLLS).  A
    // warp that gives up goes on arriving, so that no other waits for it; what is computed from then on, by any warp, is not
    // valid, and in the end all outputs and states of the tile are made NaN.
    unsigned long long* staged = reinterpret_cast<unsigned long long*>(sm + L.bars);
    unsigned long long* done = staged + 2;
    int* fail_flag = reinterpret_cast<int*>(staged + 4);
    int wait_fail = 0;
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init_n(&staged[s], FT_HW);
            mbar_init_n(&done[s], FT_W);
        }
        *fail_flag = 0;
        tc::mbar_init_fence();
    }
    __syncthreads();

    if (w >= FT_W) {
        // ---- helper warps: operands one block ahead of the walk, outputs one block behind it ----------------------
        const int ht = tid - FT_NTHR;
        unsigned char* raw = sm + L.raw;
        auto tokens = [&](int it) __attribute__((always_inline)) { return min(TB, s1 - (blk0 + it) * TB); };
        auto token0 = [&](int it) __attribute__((always_inline)) { return (long long)bos + (blk0 + it) * TB; };
        auto issue = [&](int it) __attribute__((always_inline)) {
            if (a.aligned && it < nblk) tall_issue(a, ht, raw, L, es, KP, TV, token0(it), tokens(it), h, v0, tvw);
            cp_async_commit();
        };
        auto bar_helpers = [&]() __attribute__((always_inline)) { asm volatile("bar.sync 1, %0;" ::"n"(FT_HT) : "memory"); };
        // Scalars are worked out for two blocks at a time, by every warp for itself: lanes 0 to 15 have the tokens of block it, an even
        // one, 16 to 31 those of the next.
        float gt = 0.f;
        bool live = false;
        auto load_gt = [&](int it) __attribute__((always_inline)) {
            const int b = it + (lane >> 4);
            live = b < nblk && (lane & 15) < tokens(b);
            if (live) gt = p.gt[(token0(b) + (lane & 15)) * p.H + h];
        };
        // and that block's scalars: before the wait for the walk, or after it where 16 elements a thread leave no registers to keep
        // them (B=8 T=4096 H=6 d=128: 1.13 after, 1.16 before; B=2 T=3001 H=16 96x192 0.70 after, 0.68 before)
        constexpr bool EARLY = RK * RV < 16;
        BlockScale bs;
        auto scale = [&](int it) __attribute__((always_inline)) {  // while the rows arrive, or the walk goes on
            if (it & 1) return;
            bs = block_scale<false>(gt, live, gh, iph, lane);
            load_gt(it + 2);
        };
        auto convert = [&](int it) __attribute__((always_inline)) {
            cp_async_wait<0>();
            bar_helpers();  // every lane's copies have landed
            unsigned char* op = sm + (it & 1) * L.op_stage;
#define PALIMPSA_CONVERT(DT, AL) \
    tall_convert<DT, AL, UNC, KP, TV>(a, ht, raw, op, L, token0(it), tokens(it), h, v0, tvw, bs, 16 * (it & 1))
            if (a.aligned) {
                if (p.io_dtype == PALIMPSA_BF16) PALIMPSA_CONVERT(PALIMPSA_BF16, true);
                else if (p.io_dtype == PALIMPSA_F32) PALIMPSA_CONVERT(PALIMPSA_F32, true);
                else PALIMPSA_CONVERT(PALIMPSA_F16, true);
            } else {
                if (p.io_dtype == PALIMPSA_BF16) PALIMPSA_CONVERT(PALIMPSA_BF16, false);
                else if (p.io_dtype == PALIMPSA_F32) PALIMPSA_CONVERT(PALIMPSA_F32, false);
                else PALIMPSA_CONVERT(PALIMPSA_F16, false);
            }
#undef PALIMPSA_CONVERT
            bar_helpers();  // the raw stage has been read
            issue(it + 1);
        };
        auto arrive = [&](int it) __attribute__((always_inline)) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&staged[it & 1]);
        };
        auto wait_done = [&](int it) __attribute__((always_inline)) {
            if (!wait_fail && !mbar_wait_idle(&done[it & 1], (it >> 1) & 1, POLLS)) wait_fail = 8;
        };
        auto write_outputs = [&](int it) __attribute__((always_inline)) {
            const float* ys = reinterpret_cast<const float*>(sm + L.ys + (it & 1) * L.y_stage);
            const float* yvs = reinterpret_cast<const float*>(sm + L.yvs + (it & 1) * L.y_stage);
            const long long tok0 = token0(it);
            const int nt = tokens(it);
            for (int i = ht; i < nt * TV; i += FT_HT) {
                const int t = i / TV, r = i - t * TV;
                if (r < tvw) {
                    const long long e = ((tok0 + t) * p.H + h) * (long long)V + v0 + r;
                    st1(a.o, e, ys[i], p.io_dtype);
                    if (UNC) st1(a.o_var, e, yvs[i], p.io_dtype);
                }
            }
        };
        issue(0);
        load_gt(0);
        if (nblk > 0) {
            scale(0);
            convert(0);
            arrive(0);
            if (EARLY) scale(1);
        }
        for (int it = 0; it < nblk; ++it) {
            if (it > 0) wait_done(it - 1);  // frees the operand stage of block it + 1
            if (!EARLY && it + 1 < nblk) scale(it + 1);
            if (it + 1 < nblk) convert(it + 1);
            if (it > 0) write_outputs(it - 1);  // before the block that reuses their stage is released
            if (it + 1 < nblk) {
                arrive(it + 1);
                if (EARLY) scale(it + 2);
            }
        }
        if (nblk > 0) {
            wait_done(nblk - 1);
            write_outputs(nblk - 1);
        }
        cp_async_wait<0>();
        if (wait_fail) *fail_flag = wait_fail;
        __syncthreads();
        if (*fail_flag) {
            // somebody gave up: NaN over the tile's outputs, the final states that the compute warps have written, and the
            // checkpoint that the backward begins with
            if (ht == 0) atomicCAS(&g_fwd_status, 0, *fail_flag);
            const float bad = __int_as_float(0x7fc00000);
            for (int t = s0; t < s1; ++t)
                for (int i = ht; i < tvw; i += FT_HT) {
                    const long long e = (((long long)bos + t) * p.H + h) * (long long)V + v0 + i;
                    st1(a.o, e, bad, p.io_dtype);
                    if (UNC) st1(a.o_var, e, bad, p.io_dtype);
                }
            const long long state = ((long long)n * p.H + h) * V + v0;
            const long long last = ((seq_first_slot(p, n) + blk0 + nblk - 1) * p.H + h) * V + v0;
            for (int i = ht; i < tvw * KP; i += FT_HT) {
                const int row = i / KP, c = i - row * KP;
                if (a.final_mu && s1 == len && (s0 < len || g == 0) && c < K) {
                    a.final_mu[(state + row) * K + c] = bad;
                    a.final_I[(state + row) * K + c] = bad;
                }
                if (a.ckpt_M && nblk > 0) {
                    a.ckpt_M[(last + row) * KP + c] = bad;
                    a.ckpt_I[(last + row) * KP + c] = bad;
                }
            }
        }
        return;
    }

    // ---- compute warps ---------------------------------------------------------------------------------------------
    const bool idle = w * VG * RV >= tvw;
    const long long seg_base = (((long long)n * G + g) * p.H + h) * V;  // row index into [N,G,H,V,KP] buffers
    const long long st_base = ((long long)n * p.H + h) * V;
    const long long slot0 = seq_first_slot(p, n);
    float2 M[RV][J][E], I[RV][J][E];  // columns col0 + j*GS + 2e, + 1
#pragma unroll
    for (int r = 0; r < RV; ++r) {
        const int row = row0 + r;
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int kc = col0 + j * GS;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                M[r][j][e] = make_float2(0.f, 0.f);
                I[r][j][e] = make_float2(1.f, 1.f);
            }
            if (row < tvw) {
                if (a.start_M) {
                    const long long e = (seg_base + v0 + row) * KP + kc;
                    ld_cols<CW>(a.start_M + e, M[r][j]);
                    ld_cols<CW>(a.start_I + e, I[r][j]);
                } else if (kc < K) {
                    if (p.init_mu) {
                        const long long e = (st_base + v0 + row) * K + kc;
                        if (vecK) {
                            ld_cols<CW>(p.init_mu + e, M[r][j]);
                            ld_cols<CW>(p.init_I + e, I[r][j]);
                        } else {
#pragma unroll
                            for (int c = 0; c < CW; ++c)
                                if (kc + c < K) {
                                    (c & 1 ? M[r][j][c / 2].y : M[r][j][c / 2].x) = p.init_mu[e + c];
                                    (c & 1 ? I[r][j][c / 2].y : I[r][j][c / 2].x) = p.init_I[e + c];
                                }
                        }
#pragma unroll
                        for (int c = 0; c < E; ++c) M[r][j][c] = fmul2(M[r][j][c], I[r][j][c]);
                    } else {
#pragma unroll
                        for (int c = 0; c < E; ++c) I[r][j][c] = dup2(iph);
                    }
                }
            }
        }
    }
    float missing = 0.f;  // from I since the last block: u Ip (block_scale)
    for (int it = 0; it < nblk; ++it) {
        if (idle) {
            if (!wait_fail && !mbar_wait_idle(&staged[it & 1], (it >> 1) & 1, POLLS)) wait_fail = 8;
            __syncwarp();
            if (lane == 0) mbar_arrive(&done[it & 1]);
            continue;
        }
        // ---- checkpoint: state before the first token of this block ---------------------------------------------
        if (a.ckpt_M) {
            const long long cbase = ((slot0 + blk0 + it) * p.H + h) * V + v0;
#pragma unroll
            for (int r = 0; r < RV; ++r) {
                if (row0 + r < tvw) {
#pragma unroll
                    for (int j = 0; j < J; ++j) {
                        const long long e = (cbase + row0 + r) * KP + col0 + j * GS;
                        st_cols<CW>(a.ckpt_M + e, M[r][j]);
                        float2 i[E];
#pragma unroll
                        for (int c = 0; c < E; ++c) i[c] = fadd2(I[r][j][c], dup2(missing));
                        st_cols<CW>(a.ckpt_I + e, i);
                    }
                }
            }
        }
        const unsigned char* op = sm + (it & 1) * L.op_stage;
        const float* qs = reinterpret_cast<const float*>(op + L.qs) + col0;
        const float* ks = reinterpret_cast<const float*>(op + L.ks) + col0;
        const float* qqs = reinterpret_cast<const float*>(op + L.qqs) + col0;
        const float4* vb4 = reinterpret_cast<const float4*>(op + L.vb) + row0;
        const float4* fc = reinterpret_cast<const float4*>(op + L.fc);
        const float2* zz = reinterpret_cast<const float2*>(op + L.zz);
        float* ys = reinterpret_cast<float*>(sm + L.ys + (it & 1) * L.y_stage);
        float* yvs = reinterpret_cast<float*>(sm + L.yvs + (it & 1) * L.y_stage);
        if (!wait_fail && !tc::mbar_wait(&staged[it & 1], (it >> 1) & 1, POLLS)) wait_fail = 8;
        const int end = min(TB, s1 - (blk0 + it) * TB);
        const float2 blk = *reinterpret_cast<const float2*>(op + L.blk);
        const unsigned special = __float_as_uint(blk.y);
        // GF tokens from tg on; `scaled`: some of them scale the state first
        auto group = [&](auto scaled, int tg, auto& red) __attribute__((always_inline)) {
            constexpr bool SCALED = decltype(scaled)::value;
#pragma unroll
            for (int jt = 0; jt < GF; ++jt) {
                const int t = tg + jt;
                float4 fcv = SCALED ? fc[t] : make_float4(1.f, 1.f, 0.f, 0.f);
                if (SCALED && t == 0) fcv.z = fcv.w = fcv.x * missing;
                const float2 ff = make_float2(fcv.x, fcv.y), cc = make_float2(fcv.z, fcv.w), z = zz[t];
                float2 vr[RV], br[RV], acc[RV], accv[RV];
#pragma unroll
                for (int r = 0; r < RV; ++r) {
                    const float4 x = vb4[t * TV + r];
                    vr[r] = make_float2(x.x, x.y);
                    br[r] = make_float2(x.z, x.w);
                    acc[r] = accv[r] = make_float2(0.f, 0.f);
                }
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    const int idx = t * KP + j * GS;
                    float2 kp[E], kkp[E], qp[E], qqp[E];
                    ld_cols<CW>(ks + idx, kp);
                    ld_cols<CW>(qs + idx, qp);
                    if (UNC) ld_cols<CW>(qqs + idx, qqp);
#pragma unroll
                    for (int e = 0; e < E; ++e) kkp[e] = fmul2(kp[e], kp[e]);
#pragma unroll
                    for (int r = 0; r < RV; ++r) {
#pragma unroll
                        for (int e = 0; e < E; ++e) {
                            M[r][j][e] = ffma2(vr[r], kp[e], SCALED ? fmul2(ff, M[r][j][e]) : M[r][j][e]);
                            I[r][j][e] = ffma2(br[r], kkp[e], SCALED ? ffma2(ff, I[r][j][e], cc) : I[r][j][e]);
                            const float2 rr = rcp2(fadd2(I[r][j][e], z));
                            acc[r] = ffma2(fmul2(M[r][j][e], rr), qp[e], acc[r]);
                            if (UNC) accv[r] = ffma2(rr, qqp[e], accv[r]);
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < RV; ++r) {
                    red[(jt * RV + r) * (UNC ? 2 : 1)] = acc[r].x + acc[r].y;
                    if (UNC) red[(jt * RV + r) * 2 + 1] = accv[r].x + accv[r].y;
                }
            }
        };
#pragma unroll 1
        for (int tg = 0; tg < end; tg += GF) {
            float red[NRED];
            const unsigned bits = (special >> tg) & ((1u << GF) - 1u);
            if (bits & ~1u) {
                group(std::true_type{}, tg, red);
            } else {
                if (bits) {  // a window begins with the group: the state is scaled here, and the group has nothing more to scale
                    float4 fcv = fc[tg];
                    if (tg == 0) fcv.z = fcv.w = fcv.x * missing;
#pragma unroll
                    for (int r = 0; r < RV; ++r)
#pragma unroll
                        for (int j = 0; j < J; ++j)
#pragma unroll
                            for (int e = 0; e < E; ++e) {
                                M[r][j][e] = fmul2(make_float2(fcv.x, fcv.y), M[r][j][e]);
                                I[r][j][e] = ffma2(make_float2(fcv.x, fcv.y), I[r][j][e], make_float2(fcv.z, fcv.w));
                            }
                }
                group(std::false_type{}, tg, red);
            }
            xreduce<NRED, KG>(red, lane);
            const int base = xreduce_index<NRED, KG>(lane), count = xreduce_count<NRED, KG>(lane);
#pragma unroll
            for (int i = 0; i < xreduce_most<NRED, KG>(); ++i)
                if (i < count) {
                    const int id = base + i, which = UNC ? (id & 1) : 0, jr = UNC ? (id >> 1) : id;
                    const int jt = jr / RV, r = jr % RV;
                    (which ? yvs : ys)[(tg + jt) * TV + row0 + r] = red[i];
                }
        }
        missing = blk.x;
        __syncwarp();
        if (lane == 0) mbar_arrive(&done[it & 1]);
    }
    // ---- final state in the API's (mu, I) form: written by the segment that holds the last token -----
    if (a.final_mu && !idle && s1 == len && (s0 < len || g == 0)) {
#pragma unroll
        for (int r = 0; r < RV; ++r) {
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const int kc = col0 + j * GS;
                if (row0 + r < tvw && kc < K) {
#pragma unroll
                    for (int e = 0; e < E; ++e) I[r][j][e] = fadd2(I[r][j][e], dup2(missing));
                    float2 mu[E];
#pragma unroll
                    for (int e = 0; e < E; ++e) mu[e] = make_float2(M[r][j][e].x / I[r][j][e].x, M[r][j][e].y / I[r][j][e].y);
                    const long long e = (st_base + v0 + row0 + r) * K + kc;
                    if (vecK) {
                        st_cols<CW>(a.final_mu + e, mu);
                        st_cols<CW>(a.final_I + e, I[r][j]);
                    } else {
#pragma unroll
                        for (int c = 0; c < CW; ++c)
                            if (kc + c < K) {
                                a.final_mu[e + c] = c & 1 ? mu[c / 2].y : mu[c / 2].x;
                                a.final_I[e + c] = c & 1 ? I[r][j][c / 2].y : I[r][j][c / 2].x;
                            }
                    }
                }
            }
        }
    }
    if (wait_fail) *fail_flag = wait_fail;
    __syncthreads();
}

#ifndef PALIMPSA_TALL_KERNEL_ONLY  // a test compiles the kernel alone
// -------------------------------------------------------------------------------------------------
// Host side
// -------------------------------------------------------------------------------------------------
// The thread tilings, one per padded d_k: X(RK, KG, RV), 12 or 16 state elements a thread.  The sums of a row add up in
// the same order as with fwd.cu's tiling at that d_k.
#define PALIMPSA_TALL_TILINGS(X)       \
    switch (KP) {                      \
        case 48: X(6, 8, 2); break;    \
        case 64: X(8, 8, 2);  break;   \
        case 96: X(6, 16, 2); break;   \
        case 128: X(8, 16, 2); break;  \
        case 192: X(6, 32, 2);  break; \
        case 256: X(8, 32, 2);  break; \
        default: break;                \
    }

struct TallPlan {
    int rows, tiles;
    double cost;  // per token of the longest-running SM, cycles
};
// Tile height: of all counts of tiles the one that costs least, waves of CTAs (one per SM) times what a token costs a CTA.
// That is 190 cycles and 8.3 per state element on a scheduler's lanes: measured, with the decay in every step and one row of
// twice the columns a thread where there are two rows now, 588 with 12 warps of 16 elements (48 a
// lane and scheduler: 48 rows of d_k = 128), 490 with 12 of 12, 455 with 8 of 16, 411 with 6 of 12.
template <int RK, int KG, int RV>
static TallPlan tall_plan(const palimpsa_problem& p, int num_seg) {
    constexpr int RPW = 32 / KG * RV;
    TallPlan best{0, 0, 0.};
    const double units = (double)p.num_seqs * p.H * num_seg;
    for (int n = (p.V + FT_W * RPW - 1) / (FT_W * RPW); n <= (p.V + 7) / 8; ++n) {
        const int rows = ((p.V + n - 1) / n + 7) / 8 * 8;  // 16-byte rows of 16-bit elements
        const int tiles = (p.V + rows - 1) / rows, warps = (rows + RPW - 1) / RPW;
        const double share = units * tiles / B200_SMS;
        // CTAs of equal sequences finish together; documents fill the waves up, beyond the first few
        const double waves = p.cu_seqlens && share > 3 ? share : ceil(share);
        const double cost = waves * (190 + 8.3 * RK * RV * ((warps + 3) / 4));
        if (!best.rows || cost < best.cost) best = {rows, tiles, cost};
    }
    return best;
}

// fwd.cu's kernel by the same measure: `rows` a tile, `elements` of state a thread, n of its CTAs on an SM.  Measured, 4 warps:
// 367, 497, 666 and 859 with 1 to 4 CTAs of 16 elements; 494, 701, 1158 and 1350 of 24; 597, 886 and 932 with 2, 3 and 4 of 2
// warps of 32; more run through at 13.6 per element.  The uncertainty output costs 16 elements 1.17, 1.2 and, from three CTAs on,
// 1.4 times that, more elements 1.05, 1.17 and 1.2 times, the tall tiles 1.25 times.
static double short_cost(const palimpsa_problem& p, int num_seg, int rows, int elements) {
    const int KP = palimpsa_padded_k(p.K), tiles = (p.V + rows - 1) / rows;
    const double share = (double)p.num_seqs * p.H * num_seg * tiles / B200_SMS, n = ceil(share);
    const int warps = rows * KP / (32 * elements);
    const bool few = elements <= 16;
    const double unc = !(p.flags & PALIMPSA_FLAG_UNCERTAINTY) ? 1
                       : n <= 1                               ? (few ? 1.17 : 1.05)
                       : n <= 2                               ? (few ? 1.2 : 1.17)
                                                              : (few ? 1.4 : 1.2);
    if (share > 4) return unc * 13.6 * warps / 4. * elements * share;
    const double load = ceil(n * warps / 4) * elements;  // elements on the lanes of the busiest scheduler
    if (elements >= 32) return unc * (260 + 10.4 * load);
    if (load > 48) return unc * (n < 4 ? 16 : 13.8) * load;
    return unc * (elements > 16 ? 300 + 8.1 * load : 235 + 8.4 * load);
}

// Taken where a CTA's tokens make up for what it costs to start: 1300 cycles beside fwd.cu's kernel at 4 warps of 16 elements
// (its other tilings start no sooner), and 9500 for every wave after the first, since CTAs that fill an SM do not overlap.
// Device time, us, fwd.cu's kernel against this one, 128x128 bf16: 2 heads, T = 16 / 48 / 64 / 256 5.9 / 12.1 / 15.1 / 51.5
// against 6.4 / 11.9 / 14.6 / 44.7; 64 heads (two waves) 11.2 / 25.0 / 32.7 / 118 against 15.0 / 30.7 / 38.1 / 125; 12 heads with the
// uncertainty output, T = 64 / 256 20.6 / 62.7 against 21.7 / 59.4.  The estimates are good for about 4 %: below that it stays
// with the kernel that shares an SM.
bool fwd_tall_pays(const palimpsa_problem& p, int num_seg, int short_rows, int short_elements) {
    const int KP = palimpsa_padded_k(p.K);
    TallPlan t{0, 0, 0.};
#define PALIMPSA_X(RK, KG, RV) t = tall_plan<RK, KG, RV>(p, num_seg)
    PALIMPSA_TALL_TILINGS(PALIMPSA_X)
#undef PALIMPSA_X
    if (!t.rows) return false;
    const double units = (double)p.num_seqs * p.H * num_seg, waves = ceil(units * t.tiles / B200_SMS);
    const double tokens = units > 0 ? (double)p.total_tokens * p.H / units : 0;
    const double start = (short_elements <= 16 ? 1300 : 0) + (waves > 1 ? 9500 * (waves - 1) : 0);
    const double cost = t.cost * (p.flags & PALIMPSA_FLAG_UNCERTAINTY ? 1.25 : 1);
    return start + cost * tokens < 0.96 * short_cost(p, num_seg, short_rows, short_elements) * tokens;
}

template <int RK, int KG, int RV>
static int launch_tall_k(const FwdArgs& a, const TallPlan& t, int num_seg, cudaStream_t stream) {
    const palimpsa_problem& p = a.p;
    const bool unc = (p.flags & PALIMPSA_FLAG_UNCERTAINTY) != 0;
    const TallSmem L = tall_smem_layout(RK * KG, FT_W * (32 / KG) * RV, dtype_size(p.io_dtype), unc);
    const dim3 grid(t.tiles, p.num_seqs * p.H, num_seg), block(FT_NTHR + FT_HT, 1, 1);
    if (unc) {
        if (!allow_smem<fwd_tall_kernel<RK, KG, RV, true>>(L.total)) return PALIMPSA_E_LAUNCH;
        fwd_tall_kernel<RK, KG, RV, true><<<grid, block, L.total, stream>>>(a, t.rows);
    } else {
        if (!allow_smem<fwd_tall_kernel<RK, KG, RV, false>>(L.total)) return PALIMPSA_E_LAUNCH;
        fwd_tall_kernel<RK, KG, RV, false><<<grid, block, L.total, stream>>>(a, t.rows);
    }
    return cudaGetLastError() == cudaSuccess ? PALIMPSA_OK : PALIMPSA_E_LAUNCH;
}

// Tiles of up to 12 warps of one row a thread (48 rows at d_k = 48) fill half of the warps or less with two: with one all have rows,
// and each scheduler has as many.  B=8 T=4096 H=16 48x48 (48 rows: 6 warps or 12): 0.81 -> 0.71 ms; T=37 of 4 sequences 12.0 -> 10.2 us.
template <int RK, int KG, int RV>
static int launch_tall_t(const FwdArgs& a, int num_seg, cudaStream_t stream) {
    const TallPlan t = tall_plan<RK, KG, RV>(a.p, num_seg);
    if constexpr (RK == 6 && FT_W * (32 / KG) % 8 == 0)  // whole 16-byte chunks of 16-bit rows
        if (t.rows <= FT_W * (32 / KG)) return launch_tall_k<RK, KG, 1>(a, t, num_seg, stream);
    return launch_tall_k<RK, KG, RV>(a, t, num_seg, stream);
}

int fwd_tall_rows(const palimpsa_problem& p, int num_seg) {
    const int KP = palimpsa_padded_k(p.K);
#define PALIMPSA_X(RK, KG, RV) return tall_plan<RK, KG, RV>(p, num_seg).rows
    PALIMPSA_TALL_TILINGS(PALIMPSA_X)
#undef PALIMPSA_X
    return 0;
}

int launch_fwd_tall(const FwdArgs& a, int num_seg, cudaStream_t stream) {
    const int KP = palimpsa_padded_k(a.p.K);
#define PALIMPSA_X(RK, KG, RV) return launch_tall_t<RK, KG, RV>(a, num_seg, stream)
    PALIMPSA_TALL_TILINGS(PALIMPSA_X)
#undef PALIMPSA_X
    return PALIMPSA_E_DIM;
}

#endif

int fwd_wait_status() {
    int s = 0;
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    if (cudaMemcpyFromSymbol(&s, g_fwd_status, sizeof(int)) != cudaSuccess) return -1;
    if (s) {
        const int zero = 0;
        if (cudaMemcpyToSymbol(g_fwd_status, &zero, sizeof(int)) != cudaSuccess) return -1;
    }
    return s;
}

}  // namespace palimpsa
