"""The forward's tilings of 1 or 2 rows of 6 or 8 columns a thread beside those of 2 rows of 12 or 16 in the kernel for short tiles.
All add up a row's sums in the same order, whatever the batch size."""
import pytest
import torch

from oracle import palimpsa_oracle as orc
from tests.gpu_util import DEV, compare, run_cuda, run_oracle, tol_for
from tests.helpers import fwd_plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plan,alone,N,H,K,V", [
    ((1, 96), (1, 32), 64, 2, 48, 96),   # 12 warps of 2 rows a thread; 1 row a thread
    ((0, 48), (1, 24), 24, 16, 48, 48),  # the kernel for short tiles; 1 row a thread
    ((1, 48), (1, 24), 8, 16, 46, 48),   # rows that are no whole vectors
    ((0, 32), (1, 16), 64, 2, 96, 192),
    ((0, 32), (1, 32), 96, 4, 64, 64),
    ((0, 16), (1, 8), 48, 4, 192, 48),
    ((0, 16), (1, 8), 64, 4, 256, 32),
])
def test_neither_tile_nor_kernel_changes_the_result(plan, alone, N, H, K, V):
    from palimpsa_b200.ops import chunk_palimpsa
    T = 70
    assert fwd_plan(N, T, H, K, V, torch.bfloat16) == plan and fwd_plan(1, T, H, K, V, torch.bfloat16) == alone
    inp = orc.make_inputs(9, B=N, T=T, H=H, K=K, V=V, dtype=torch.bfloat16)
    a = [inp[n].to(DEV) for n in ("q", "k", "v", "b", "gt", "g", "Ip")]
    with torch.no_grad():
        o = chunk_palimpsa(*a)
        one = torch.cat([chunk_palimpsa(*[x[i:i + 1] for x in a[:5]], *a[5:]) for i in range(N)])
    assert torch.equal(o, one)


@pytest.mark.parametrize("N,H,T,K,V,dtype,unc,init", [
    (2, 2, 35, 48, 48, torch.float32, False, True),
    (2, 2, 35, 46, 20, torch.float32, True, True),
    (64, 2, 19, 48, 90, torch.float32, True, True),
    (40, 16, 17, 47, 48, torch.bfloat16, False, False),
    (24, 16, 20, 48, 48, torch.float32, True, True),
    (2, 2, 35, 96, 24, torch.bfloat16, False, True),     # 1 row a thread, 24 rows
    (2, 2, 35, 192, 8, torch.bfloat16, True, False),     # 12 rows would not be whole chunks: 2 rows a thread
    (2, 2, 35, 192, 32, torch.float16, False, True),
    (3, 2, 35, 256, 16, torch.bfloat16, False, True),
    (2, 2, 35, 64, 8, torch.float16, True, True),
])
def test_matches_oracle(N, H, T, K, V, dtype, unc, init):
    inp = orc.make_inputs(T + K, B=N, T=T, H=H, K=K, V=V, dtype=dtype)
    mu0 = I0 = None
    if init:
        g = torch.Generator().manual_seed(1)
        mu0 = 0.3 * torch.randn(N, H, V, K, generator=g)
        I0 = 0.5 + torch.rand(N, H, V, K, generator=g)
    got, ref = run_cuda(inp, "chunk", unc=unc, mu0=mu0, I0=I0), run_oracle(inp, unc=unc, mu0=mu0, I0=I0)
    compare(got, ref, tol_for(dtype), names=["o", "final_mu", "final_I", "dq", "dk", "dv", "db", "dgt"], what=f"{N}x{H} {K}x{V}")


@pytest.mark.parametrize("N,H,K,V", [(64, 2, 48, 96), (24, 16, 48, 48), (64, 2, 96, 192), (48, 4, 192, 48)])
@pytest.mark.parametrize("decay", [1.0, 6.0, 40.0])
def test_nor_the_uncertainty_and_the_states(N, H, K, V, decay):
    """Also where blocks have several windows, or none: the kernels' groups of tokens differ."""
    from palimpsa_b200.ops import chunk_palimpsa
    inp = orc.make_inputs(9, B=N, T=45, H=H, K=K, V=V, dtype=torch.bfloat16)
    a = [inp[n].to(DEV) for n in ("q", "k", "v", "b", "gt", "g", "Ip")]
    a[4] = decay * a[4]
    flat = lambda out: [*out[0], *out[1:]]
    with torch.no_grad():
        every = flat(chunk_palimpsa(*a, output_final_state=True, output_uncertainty=True))
        one = [flat(chunk_palimpsa(*[x[i:i + 1] for x in a[:5]], *a[5:], output_final_state=True, output_uncertainty=True)) for i in range(N)]
    for x, *parts in zip(every, *one):
        assert torch.equal(x, torch.cat(parts))
