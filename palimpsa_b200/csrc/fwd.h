// What the two forward kernels share on the host side (fwd.cu, fwd_tall.cu).
#pragma once

#include "host.h"

namespace palimpsa {

struct FwdArgs {
    palimpsa_problem p;
    void* o;
    void* o_var;
    float* final_mu;
    float* final_I;
    float* ckpt_M;
    float* ckpt_I;
    int aligned;  // 1: every io row is 16-byte aligned and a multiple of 16 bytes
    // segments (gridDim.z of them per sequence; seg_len tokens each, a multiple of 16)
    int seg_len;
    const float* start_M;  // [N,G,H,V,KP] (M, I) at the start of every segment, or NULL
    const float* start_I;
    float* sum_M;          // summary mode: [N,G,H,V,KP] end state of the segment started from zero, (M, J) form
    float* sum_J;
    float* decay;          // summary mode: [N,G,H] product of f over the segment
};

// Is the tall-tile kernel the faster one for this call (fwd_tall.cu)?  `short_rows`, `short_elements`: the other kernel's tile
// height and state elements per thread.
bool fwd_tall_pays(const palimpsa_problem& p, int num_seg, int short_rows, int short_elements);
int fwd_tall_rows(const palimpsa_problem& p, int num_seg);
int launch_fwd_tall(const FwdArgs& a, int num_seg, cudaStream_t stream);

}  // namespace palimpsa
