"""Decays from slow to instant, against the float64 oracle: the kernels walk a block's tokens without decay, on a state divided by
the product F of the decays, and begin a new window where F would fall below 2^-64 -- in front of a group of four tokens, or token
by token.  Forward, backward, segments."""
import pytest
import torch

from oracle import palimpsa_oracle as orc
from tests.gpu_util import DEV, compare, run_cuda, run_oracle, tol_for

pytestmark = pytest.mark.gpu


def _with_decay(inp, kind):
    gt, gen = inp["gt"], torch.Generator().manual_seed(3)
    some = torch.rand(gt.shape, generator=gen)
    inp["gt"] = {
        "slow": lambda: 0.05 * gt,   # (1 - f) Ip has 24 bits of f behind it: much slower, and dIp has no five digits left
        "windows": lambda: 8 * gt,                                           # several windows in a block
        "alone": lambda: 60 * gt,                                            # most tokens by themselves
        "resets": lambda: torch.where(some < 0.1, 300 + 0 * gt, 0.2 * gt),   # f = 0 now and then
        "mixed": lambda: gt * torch.exp(3 * torch.randn(gt.shape, generator=gen)),
    }[kind]()
    return inp


@pytest.mark.parametrize("kind", ["slow", "windows", "alone", "resets", "mixed"])
@pytest.mark.parametrize("N,H,T,K,V,unc,init", [
    (2, 2, 37, 128, 40, False, False),   # tall forward tiles; a ragged last block
    (1, 2, 70, 48, 33, True, True),
    (1, 2, 35, 128, 72, True, False),    # short forward tiles
    (1, 3, 50, 31, 65, False, True),
    (1, 2, 21, 16, 9, True, False),
    (10, 4, 33, 96, 49, False, False),   # 6 warps in the backward
    (1, 1, 34, 192, 20, False, False),
])
def test_matches_oracle(kind, N, H, T, K, V, unc, init):
    inp = _with_decay(orc.make_inputs(T + K, B=N, T=T, H=H, K=K, V=V), kind)
    mu0 = I0 = None
    if init:
        g = torch.Generator().manual_seed(1)
        mu0 = 0.3 * torch.randn(N, H, V, K, generator=g)
        I0 = 0.5 + torch.rand(N, H, V, K, generator=g)
    got, ref = run_cuda(inp, "chunk", unc=unc, mu0=mu0, I0=I0), run_oracle(inp, unc=unc, mu0=mu0, I0=I0)
    compare(got, ref, tol_for(torch.float32), names=[n for n in got if n != "dg"], what=f"{kind} {K}x{V}")
    # dg = sum of gt dgt / g, whose terms may cancel: each is good to the same tolerance of its own size
    terms = (inp["gt"].double() * ref["dgt"].double()).abs().sum((0, 1)) / inp["g"].double()
    assert bool(((got["dg"].double() - ref["dg"].double()).abs() <= tol_for(torch.float32) * terms).all())


@pytest.mark.parametrize("kind", ["windows", "alone", "mixed"])
def test_segments(kind):
    from palimpsa_b200.ops import chunk_palimpsa
    inp = _with_decay(orc.make_inputs(7, B=1, T=150, H=2, K=64, V=48), kind)
    a = {n: inp[n].to(DEV).requires_grad_() for n in ("q", "k", "v", "b", "gt", "g", "Ip")}
    o, mu, I = chunk_palimpsa(*a.values(), output_final_state=True, num_segments=4)
    (o * inp["do"].to(DEV)).sum().backward()
    got = {"o": o, "final_mu": mu, "final_I": I, **{"d" + n: x.grad for n, x in a.items()}}
    compare({n: x.detach().cpu() for n, x in got.items()}, run_oracle(inp), tol_for(torch.float32), names=[n for n in got if n != "dg"], what=kind)


def test_small_precision_beside_a_large_prior():
    """I far below Ip and no decay: the scaled state starts from I itself, not from its distance to Ip."""
    inp = orc.make_inputs(9, B=1, T=40, H=2, K=48, V=16)
    inp["gt"], inp["Ip"], inp["b"] = 0 * inp["gt"], torch.full((2,), 1e4), 1e-3 * inp["b"]
    mu0, I0 = torch.randn(1, 2, 16, 48, generator=torch.Generator().manual_seed(1)), torch.full((1, 2, 16, 48), 1e-3)
    compare(run_cuda(inp, "chunk", mu0=mu0, I0=I0), run_oracle(inp, mu0=mu0, I0=I0), tol_for(torch.float32),
            names=["o", "final_mu", "final_I", "dq", "dk", "dv", "db"], what="small I")
