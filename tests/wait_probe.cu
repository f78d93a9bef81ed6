// Test-only library (NOT part of libpalimpsa_b200.so): runs the bounded mbarrier wait of the product kernels
// (tc::mbar_wait, palimpsa_b200/csrc/tc_common.cuh) to its give-up path on purpose, the way the tensor-core
// kernels would meet it: one small CTA allocates TMEM, waits on an mbarrier with a poll limit given by the
// caller, records a status code, frees its TMEM and returns.  With `arrive` = 0 nobody ever arrives at the
// barrier, so the wait runs out by construction after `limit` polls (nothing hangs and nothing faults); with
// `arrive` = 1 one thread arrives first and the wait succeeds.
#include "../palimpsa_b200/csrc/host.h"
#include "../palimpsa_b200/csrc/tc_common.cuh"

namespace {

__global__ void __launch_bounds__(32) wait_probe_kernel(int arrive, unsigned limit, int* status) {
    __shared__ __align__(8) unsigned long long bar;
    __shared__ unsigned tmem_slot;
    using namespace palimpsa;
    if (threadIdx.x == 0) {
        tc::mbar_init(&bar);
        tc::mbar_init_fence();
    }
    tc::tmem_alloc(&tmem_slot, 32);
    tc::fence_before_sync();
    __syncwarp();
    tc::fence_after_sync();
    const unsigned tmem = tmem_slot;
    if (arrive && threadIdx.x == 0)
        asm volatile("{\n.reg .b64 st;\nmbarrier.arrive.shared::cta.b64 st, [%0];\n}" ::"r"(tc::smem_u32(&bar)) : "memory");
    __syncwarp();
    const bool ok = tc::mbar_wait(&bar, 0, limit);
    if (threadIdx.x == 0) *status = ok ? 0 : 7;     // 7: the probe's own code for "the wait gave up"
    __syncwarp();
    tc::fence_before_sync();
    tc::tmem_free(tmem, 32);
}

}  // namespace

// status_dev: one int in device memory.  Returns 0, or -1 if the launch was refused.
extern "C" int palimpsa_test_wait_probe(int arrive, unsigned limit, int* status_dev, void* cuda_stream) {
    wait_probe_kernel<<<1, 32, 0, static_cast<cudaStream_t>(cuda_stream)>>>(arrive, limit, status_dev);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// A launch with `bytes` of dynamic shared memory by way of the library's allow_smem; with `reset` the process first drops
// its context on the device (for a process of its own).  0, or the step that failed.
namespace {
__global__ void smem_probe_kernel(int bytes) {
    extern __shared__ unsigned char sm[];
    for (int i = threadIdx.x; i < bytes; i += blockDim.x) sm[i] = (unsigned char)i;
}
}  // namespace
extern "C" int palimpsa_test_smem_grant(int bytes, int reset) {
    if (reset && cudaDeviceReset() != cudaSuccess) return -1;
    if (!palimpsa::allow_smem<smem_probe_kernel>(bytes)) return -2;
    smem_probe_kernel<<<1, 32, bytes>>>(bytes);
    if (cudaGetLastError() != cudaSuccess) return -3;
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : -4;
}

// The tall-tile forward's kernel, one tiling (97 <= d_k <= 128, tiles of `rows` rows), with the product's poll limit or one of 0.
// With 0 every wait gives up at once, by construction; all accesses stay inside the buffers of an ordinary launch, and nothing
// waits for anything but the CTA barriers that all threads reach.
#define PALIMPSA_TALL_KERNEL_ONLY
#include "../palimpsa_b200/csrc/fwd_tall.cu"

namespace {
template <unsigned POLLS>
int launch_tall(const palimpsa::FwdArgs& a, int rows, cudaStream_t stream) {
    using namespace palimpsa;
    const TallSmem L = tall_smem_layout(128, FT_W * 2 * 2, dtype_size(a.p.io_dtype), true);
    const dim3 grid((a.p.V + rows - 1) / rows, a.p.num_seqs * a.p.H, 1);
    if (!allow_smem<fwd_tall_kernel<8, 16, 2, true, POLLS>>(L.total)) return -2;
    fwd_tall_kernel<8, 16, 2, true, POLLS><<<grid, FT_NTHR + FT_HT, L.total, stream>>>(a, rows);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
}  // namespace
extern "C" int palimpsa_test_tall_forward(const palimpsa_fwd_params* prm, int rows, int give_up, int aligned, void* cuda_stream) {
    palimpsa::FwdArgs a{};
    a.p = prm->p;
    a.o = prm->o, a.o_var = prm->o_var, a.final_mu = prm->final_mu, a.final_I = prm->final_I;
    a.ckpt_M = prm->ckpt_M, a.ckpt_I = prm->ckpt_I;
    a.aligned = aligned;
    if (a.p.K <= 96 || a.p.K > 128 || rows > palimpsa::FT_W * 2 * 2 || rows % 8 || !a.o_var) return -4;
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    return give_up ? launch_tall<0>(a, rows, stream) : launch_tall<palimpsa::tc::SPIN_LIMIT>(a, rows, stream);
}
extern "C" int palimpsa_test_tall_status(void) { return palimpsa::fwd_wait_status(); }
