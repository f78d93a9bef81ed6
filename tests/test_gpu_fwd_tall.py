"""The tall-tile forward kernel and the rule that takes it, against the float64 oracle: every tiling, one block and several, a
ragged last block, tiles lower than 12 warps hold, idle warps, padded d_k, element loads, initial states,
packed rows, exact segments."""
import pytest
import torch

from oracle import palimpsa_oracle as orc
from tests.gpu_util import DEV, compare, run_cuda, run_oracle, tol_for
from tests.helpers import fwd_plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plan,N,H,T,K,V,dtype,unc,init", [
    ((0, 16), 1, 2, 1, 128, 128, torch.bfloat16, False, False),   # too short to make up for its start
    ((0, 16), 1, 2, 16, 128, 40, torch.float32, True, True),
    ((1, 16), 2, 3, 83, 128, 128, torch.float16, False, True),
    ((0, 16), 48, 3, 35, 128, 128, torch.bfloat16, False, False), # several waves
    ((1, 48), 8, 6, 70, 128, 128, torch.bfloat16, False, False),  # tiles of 48 rows: all 12 warps
    ((1, 48), 8, 6, 49, 128, 128, torch.float16, True, True),
    ((1, 32), 7, 3, 49, 127, 129, torch.bfloat16, False, False),  # element loads
    ((1, 16), 2, 2, 66, 96, 196, torch.bfloat16, True, False),
    ((1, 48), 2, 16, 20, 96, 192, torch.bfloat16, False, False),  # 12 warps
    ((1, 48), 2, 16, 20, 96, 192, torch.float32, True, False),
    ((0, 32), 64, 2, 17, 96, 192, torch.bfloat16, False, False),
    ((1, 16), 2, 2, 97, 90, 50, torch.float32, False, True),      # element loads
    ((1, 24), 2, 2, 33, 50, 66, torch.bfloat16, False, False),    # element loads of 16-bit values
    ((0, 64), 2, 2, 40, 22, 70, torch.float16, True, False),      # d_k <= 32: always the kernel for short tiles
    ((1, 48), 128, 1, 18, 48, 48, torch.bfloat16, False, False),
    ((1, 96), 64, 2, 37, 48, 96, torch.float32, True, False),     # 12 warps
    ((1, 64), 96, 1, 31, 64, 64, torch.float16, False, False),
    ((1, 96), 100, 1, 33, 64, 96, torch.float16, False, False),   # 12 warps
    ((1, 24), 2, 2, 65, 63, 65, torch.float32, True, True),
    ((1, 8), 2, 2, 34, 180, 30, torch.bfloat16, False, False),
    ((1, 24), 32, 1, 33, 192, 96, torch.bfloat16, False, False),  # 12 warps
    ((1, 24), 12, 3, 40, 192, 96, torch.float32, True, False),
    ((1, 8), 2, 2, 34, 256, 24, torch.float32, True, False),
    ((1, 24), 37, 1, 33, 256, 96, torch.float32, False, False),   # 12 warps
    ((1, 24), 40, 1, 40, 256, 72, torch.bfloat16, True, False),
])
def test_forward_and_backward_match_oracle(plan, N, H, T, K, V, dtype, unc, init):
    assert fwd_plan(N, T, H, K, V, dtype, unc) == plan
    inp = orc.make_inputs(T + K, B=N, T=T, H=H, K=K, V=V, dtype=dtype)
    mu0 = I0 = None
    if init:
        g = torch.Generator().manual_seed(1)
        mu0 = 0.3 * torch.randn(N, H, V, K, generator=g)
        I0 = 0.5 + torch.rand(N, H, V, K, generator=g)
    got = run_cuda(inp, "chunk", unc=unc, mu0=mu0, I0=I0)
    compare(got, run_oracle(inp, unc=unc, mu0=mu0, I0=I0), tol_for(dtype), what=f"{N}x{H} T={T} {K}x{V}")


def test_packed_rows_with_empty_documents():
    inp = orc.make_inputs(5, B=1, T=150, H=2, K=128, V=72)
    cu = [0, 0, 70, 71, 71, 150]
    compare(run_cuda(inp, "chunk", cu=cu), run_oracle(inp, cu=cu), tol_for(torch.float32), what="packed")


@pytest.mark.parametrize("K,V", [(128, 64), (96, 40), (47, 33)])
def test_exact_segments(K, V):
    from palimpsa_b200.ops import chunk_palimpsa
    inp = orc.make_inputs(K, B=1, T=200, H=2, K=K, V=V)
    a = [inp[n].to(DEV) for n in ("q", "k", "v", "b", "gt", "g", "Ip")]
    o, mu, I = chunk_palimpsa(*a, output_final_state=True, num_segments=4)
    got = {"o": o.cpu(), "final_mu": mu.cpu(), "final_I": I.cpu()}
    compare(got, run_oracle(inp), tol_for(torch.float32), names=[*got], what=f"4 segments, {K}x{V}")


@pytest.mark.parametrize("B,plan", [(8, (1, 48)), (24, (0, 16))])
def test_neither_tile_nor_kernel_changes_the_result(B, plan):
    """A batch that takes 12-warp tiles, one that takes the kernel for short tiles, and the same sequences one by one (lower
    tiles of the kernel for tall ones) agree to the bit: every row is walked by the same arithmetic."""
    from palimpsa_b200.ops import chunk_palimpsa
    T, H, K, V = 70, 6, 128, 128
    assert fwd_plan(B, T, H, K, V, torch.bfloat16) == plan and fwd_plan(1, T, H, K, V, torch.bfloat16) == (1, 16)
    inp = orc.make_inputs(9, B=B, T=T, H=H, K=K, V=V, dtype=torch.bfloat16)
    a = [inp[n].to(DEV) for n in ("q", "k", "v", "b", "gt", "g", "Ip")]
    with torch.no_grad():
        o = chunk_palimpsa(*a)
        one = torch.cat([chunk_palimpsa(*[x[i:i + 1] for x in a[:5]], *a[5:]) for i in range(B)])
    assert torch.equal(o, one)
