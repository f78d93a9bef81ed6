"""The backward's staged blocks: sequences of several blocks (both operand stages and both barrier phases in use), a ragged
last block, warps without rows in the last tile, steps of 4, 8 and 16 tokens, and the state-gradient
pass of exact segments, against the float64 oracle."""
import pytest
import torch

from oracle import palimpsa_oracle as orc
from tests.gpu_util import DEV, compare, run_cuda, run_oracle, tol_for
from tests.helpers import GRADS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,H,T,K,V,dtype,unc", [
    (1, 2, 83, 128, 128, torch.bfloat16, False),   # 3 rows a thread, tiles of 22 rows starting at every even offset
    (25, 4, 67, 128, 24, torch.bfloat16, False),   # tiles of 24
    (2, 2, 81, 128, 67, torch.float32, True),      # odd rows
    (2, 2, 66, 64, 90, torch.float16, False),      # tiles of 44 rows and one of 2
    (2, 2, 97, 48, 57, torch.bfloat16, False),     # a second tile of one row: all but one warp without rows
    (2, 2, 70, 96, 97, torch.bfloat16, True),
    (2, 2, 65, 31, 65, torch.float32, True),       # element loads
    (2, 2, 79, 16, 33, torch.float16, True),
    (1, 2, 50, 192, 30, torch.float32, False),
    (1, 2, 50, 256, 20, torch.bfloat16, False),
])
def test_blocks_in_flight(N, H, T, K, V, dtype, unc):
    inp = orc.make_inputs(T + K, B=N, T=T, H=H, K=K, V=V, dtype=dtype)
    compare(run_cuda(inp, "chunk", unc=unc), run_oracle(inp, unc=unc), tol_for(dtype), what=f"{N}x{H} T={T} {K}x{V}")


@pytest.mark.parametrize("K,V,unc", [(128, 40, False), (64, 48, True), (48, 50, False), (31, 9, False)])
def test_state_gradient_pass(K, V, unc):
    """Exact float32 segments: a carry-only pass (whose waits are the staged blocks alone), then each segment's backward."""
    from palimpsa_b200.ops import chunk_palimpsa
    inp = orc.make_inputs(K, B=1, T=150, H=2, K=K, V=V)
    a = {n: inp[n].to(DEV).requires_grad_() for n in ("q", "k", "v", "b", "gt", "g", "Ip")}
    out = chunk_palimpsa(*a.values(), output_uncertainty=unc, num_segments=3)
    got = dict(zip(("o", "o_var"), out)) if unc else {"o": out}
    sum((got[n] * inp["d" + n].to(DEV)).sum() for n in got).backward()
    got.update({"d" + n: x.grad for n, x in a.items()})
    compare({n: x.detach().cpu() for n, x in got.items()}, run_oracle(inp, unc=unc), tol_for(torch.float32),
            names=[*got], what=f"3 segments, {K}x{V}")
    assert set(GRADS) <= set(got)
