// Host-side declarations shared by the translation units of libpalimpsa_b200.so.
#pragma once

#include <cuda_runtime.h>

#include <mutex>

#include "../../include/palimpsa_b200.h"

namespace palimpsa {

// SMs of the one GPU this library is built for.  Tile heights are chosen by it, on the host and without a device, so that a
// workspace query and the launch that follows agree everywhere.
constexpr int B200_SMS = 148;

// Lets a kernel use the `bytes` of dynamic shared memory it is about to be launched with.  The attribute belongs to the
// kernel in one context (cudaDeviceReset, or another context on the device, starts from the default again), so it is set on
// every launch; and never lower than before, so that a thread that launches with less does not take it from another that is
// about to launch with more.  (Not simply to the maximum: the attribute also moves the split between shared memory and L1.)
template <auto Kern>
bool allow_smem(int bytes) {
    static std::mutex setting;
    static int most = 0;
    std::lock_guard<std::mutex> lock(setting);
    const int limit = bytes > most ? bytes : most;
    if (cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess) return false;
    most = limit;
    return true;
}

// Enqueue the forward kernel (fwd.cu).  Parameters are assumed validated.  With `segs` every sequence is
// cut into segs->num_segments segments that run as separate CTAs: `summary` = false starts each from
// segs->start_M/start_I; `summary` = true computes the zero-start end state and decay of every segment.
int launch_fwd(const palimpsa_fwd_params* prm, const palimpsa_segments* segs, bool summary, cudaStream_t stream);

// Single-token decode step (decode.cu): dedicated HBM-bound kernel, when it covers the call.
bool decode_supported(const palimpsa_fwd_params* prm);
int launch_decode(const palimpsa_fwd_params* prm, cudaStream_t stream);
int launch_copy_buffers(const void* const* src, void* const* dst, const size_t* bytes, int n, cudaStream_t stream);

// palimpsa_problem::segments, internal: as few row tiles as possible, the least scratch a backward of this size runs with.
constexpr int BWD_FEWEST_TILES = -1;

// Backward (bwd.cu): main kernel (stages bit 0) + the two finishing kernels (bit 1); bit 2: the finishing
// kernels also sum the extra partial slot that carry_tc.cu fills.
int launch_bwd(const palimpsa_bwd_params* prm, const palimpsa_segments* segs, bool carry_only, cudaStream_t stream,
               int stages);

// Segment summaries on the tensor cores (summary_tc.cu): bf16 inputs, d_v <= 128, padded d_k in {32,48,64,96,128}.
bool summary_tc_supported(const palimpsa_problem& p);
int launch_summary_tc(const palimpsa_problem& p, const palimpsa_segments& segs, cudaStream_t stream);
int summary_tc_status();

// Carried-gradient terms of a segmented backward on the tensor cores (carry_tc.cu).
bool carry_tc_shape(const palimpsa_problem& p);      // by sizes, type and flags alone
bool carry_tc_supported(const palimpsa_problem& p);  // and by the alignment of its tensors
int launch_carry_tc(const palimpsa_bwd_params* prm, const palimpsa_segments& segs, cudaStream_t stream);
int carry_tc_status();
int fwd_wait_status();  // 0, or the code of a bounded wait of the tall-tile forward that gave up
int bwd_wait_status();  // 0, or the code of a bounded barrier wait of the backward main kernel that gave up

// What a launch of these sizes takes: {1 for the tall-tile kernel, rows of a tile}; {rows, compute warps, group buffers}.
void fwd_plan(const palimpsa_problem& p, int32_t* plan);
void bwd_plan(const palimpsa_problem& p, int32_t* plan);

// Boundary scans over segments (segments.cu).
int launch_combine_fwd(const palimpsa_problem& p, const palimpsa_segments& segs, const float* in_M, const float* in_J,
                       float* out_M, float* out_J, cudaStream_t stream);
int launch_combine_bwd(const palimpsa_problem& p, const palimpsa_segments& segs, const float* in_M, const float* in_I,
                       float* out_M, float* out_I, cudaStream_t stream);

// Checkpoint slots and start order of a packed batch's sequences (segments.cu).
int launch_varlen_plan(const int32_t* cu_seqlens, int n, int32_t* chunk_offsets, int32_t* order, cudaStream_t stream);

// Stream-ordered flags in peer-mapped memory (peer.cu): a bounded wait until *flag >= value, and a release store.
int launch_peer_wait(const void* flag, unsigned long long value, unsigned timeout_ms, float* poison, cudaStream_t stream);
int launch_peer_signal(void* flag, unsigned long long value, cudaStream_t stream);
int peer_status();   // 0, or 7 when a wait ran out

// A context-parallel hop split in two (segments.cu): what this rank adds to a state passing through, computed
// before the state arrives, and out = decay_product * in + total when it does.
int launch_relay_total(const palimpsa_problem& p, const palimpsa_segments& segs, int backward, float* tot_A,
                       float* tot_B, cudaStream_t stream);
int launch_relay(const palimpsa_problem& p, const palimpsa_segments& segs, const float* in_A, const float* in_B,
                 const float* tot_A, const float* tot_B, float* out_A, float* out_B, cudaStream_t stream);

// Backward whose scratch is the library's own fixed device array (bwd.cu).
int launch_bwd_static(const palimpsa_bwd_params* prm, cudaStream_t stream);

// State rows (d_v) one forward CTA owns at these head dimensions (0: d_k unsupported).
int fwd_tile_rows(int K, int V);

// State rows (d_v) one backward CTA owns for this problem; the number of row tiles follows.
int bwd_tile_rows(const palimpsa_problem& p);
double bwd_token_cost(const palimpsa_problem& p);  // estimated time per token of the backward, 0 if unsupported

// Layout of the backward scratch memory (byte offsets from a 256-byte aligned base).
struct BwdWorkspace {
    size_t dq_part, dk_part;    // float [tiles][tokens*H][KP]   (dk, df, dip: tiles + 1 slots)
    size_t df_part, dip_part;   // float [tiles][tokens*H]
    size_t w_dg, w_dip;         // double [scalar CTAs of the finishing kernel][H]
    size_t total;
    int tiles, KP;
};
BwdWorkspace bwd_workspace_layout(const palimpsa_problem& p);

}  // namespace palimpsa
