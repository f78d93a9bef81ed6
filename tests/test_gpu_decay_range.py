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


def _norm_err(x, ref):
    return float((x.double() - ref.double()).norm() / ref.double().norm())


def _plain_walk(inp, mu0, I0):
    """The recurrence with its decay in every step, every operation rounded to float32 (FMAs once), the final state's errors: what a
    kernel without windows has."""
    r = lambda x: x.float().double()
    k, v, b = (inp[n].double() for n in ("k", "v", "b"))
    x, Ip = r(inp["gt"].double() * inp["g"].double()), inp["Ip"].double()[None, :, None, None]
    f = torch.exp(-x.float()).double()
    N, T, H, K = k.shape
    I = (torch.ones(N, H, v.shape[-1], K).double() * Ip) if I0 is None else I0.double()
    M = torch.zeros_like(I) if mu0 is None else r(mu0.double() * I)
    for t in range(T):
        ft, kt = f[:, t, :, None, None], k[:, t, :, None, :]
        M = r(ft * M + r(v[:, t, :, :, None] * kt))
        I = r(ft * I + r(b[:, t, :, :, None] * r(kt * kt) + r(r(1 - ft) * Ip)))
    return r(M / I), I


@pytest.mark.parametrize("K,V", [(48, 48), (128, 40)])
@pytest.mark.parametrize("kind", ["slow", "usual", "windows"])
def test_final_state_no_further_off_than_with_a_decay_in_every_step(kind, K, V):
    inp = orc.make_inputs(11, B=2, T=256, H=4, K=K, V=V)
    inp["gt"] = {"slow": 0.1, "usual": 1.0, "windows": 8.0}[kind] * inp["gt"]
    got, ref = run_cuda(inp, "chunk", grads=False), run_oracle(inp)
    mu, I = _plain_walk(inp, None, None)
    # 5 %: how far two such runs of other seeds differ (the product of rounded decays had 10 to 30 % more in mu)
    assert _norm_err(got["final_mu"], ref["final_mu"]) < 1.05 * _norm_err(mu, ref["final_mu"])
    assert _norm_err(got["final_I"], ref["final_I"]) < 1.05 * _norm_err(I, ref["final_I"])


@pytest.mark.parametrize("K,V,unc", [(48, 16, False), (128, 40, True), (64, 48, False)])
def test_slow_decay_towards_a_large_prior(K, V, unc):
    """1 - F times Ip is most of what I gains: with 1 - F from rounded decays 2^-25 / (1 - f) of it was wrong, 1e-5 to 1e-4 here."""
    inp = orc.make_inputs(12, B=2, T=96, H=4, K=K, V=V)
    inp["gt"], inp["Ip"] = 0.01 * inp["gt"], torch.full((4,), 1e3)
    mu0 = 0.3 * torch.randn(2, 4, V, K, generator=torch.Generator().manual_seed(1))
    I0 = torch.full((2, 4, V, K), 1e-2)
    got, ref = run_cuda(inp, "chunk", unc=unc, mu0=mu0, I0=I0), run_oracle(inp, unc=unc, mu0=mu0, I0=I0)
    errs = {n: _norm_err(got[n], ref[n]) for n in ("o", "final_mu", "final_I", "dq", "dk", "dv", "db")}
    assert max(errs.values()) < 3e-6, errs  # some fifty roundings of 2^-24


@pytest.mark.parametrize("K,V", [(48, 40), (128, 24)])
@pytest.mark.parametrize("vs,dos", [(1e20, 1.0), (1e-20, 1.0), (1.0, 1e20), (1.0, 1e-20)])
def test_large_and_small_values_keep_their_bits(vs, dos, K, V):
    """At decays just too slow for a second window, and faster ones: the scales reach 2^48."""
    inp = orc.make_inputs(13, B=1, T=70, H=3, K=K, V=V)
    inp["gt"], inp["g"] = torch.ones(1, 70, 3), torch.tensor([2.05, 2.7, 9.0])
    inp["v"], inp["do"] = vs * inp["v"], dos * inp["do"]
    got, ref = run_cuda(inp, "chunk"), run_oracle(inp)
    errs = {n: _norm_err(got[n], ref[n]) for n in ("o", "final_mu", "final_I", "dq", "dk", "dv", "db", "dgt")}
    assert max(errs.values()) < 2e-6, errs


@pytest.mark.parametrize("K,V", [(16, 9), (48, 33), (128, 24)])
def test_growing_states(K, V):
    """f above 1 (a negative step) now and then: those groups go token by token, the last ones before a sequence's ragged end too."""
    inp = orc.make_inputs(14, B=2, T=41, H=2, K=K, V=V)
    some = torch.rand(inp["gt"].shape, generator=torch.Generator().manual_seed(2))
    inp["gt"] = torch.where(some < 0.1, -0.05 * inp["gt"], 0.5 * inp["gt"])
    inp["gt"][:, -1] = -0.05
    got, ref = run_cuda(inp, "chunk"), run_oracle(inp)
    compare(got, ref, tol_for(torch.float32), names=[n for n in got if n != "dg"], what=f"f > 1 {K}x{V}")


@pytest.mark.parametrize("kind", ["windows", "alone", "resets"])
@pytest.mark.parametrize("K,V", [(48, 48), (128, 40)])
def test_packed(kind, K, V):
    cu = [0, 1, 38, 53, 54, 121]
    inp = _with_decay(orc.make_inputs(15, B=1, T=cu[-1], H=2, K=K, V=V), kind)
    got, ref = run_cuda(inp, "chunk", cu=cu), run_oracle(inp, cu=cu)
    compare(got, ref, tol_for(torch.float32), names=[n for n in got if n != "dg"], what=f"packed {kind}")


@pytest.mark.parametrize("kind", ["windows", "resets"])
def test_segments_with_tensor_core_carry(kind):
    """bf16 heads of 128x128: the carried gradients' decay terms come from the tensor-core pass."""
    from palimpsa_b200.ops import chunk_palimpsa
    inp = _with_decay(orc.make_inputs(16, B=1, T=300, H=2, K=128, V=128, dtype=torch.bfloat16), kind)
    a = {n: inp[n].to(DEV).requires_grad_() for n in ("q", "k", "v", "b", "gt", "g", "Ip")}
    o = chunk_palimpsa(*a.values(), num_segments=3)
    (o.float() * inp["do"].to(DEV).float()).sum().backward()
    got, ref = {"o": o, **{"d" + n: x.grad for n, x in a.items()}}, run_oracle(inp)
    compare({n: x.detach().cpu() for n, x in got.items()}, ref, tol_for(torch.bfloat16), names=[n for n in got if n != "dg"], what=kind)
    terms = (inp["gt"].double() * ref["dgt"].double()).abs().sum((0, 1)) / inp["g"].double()
    assert bool(((a["g"].grad.cpu().double() - ref["dg"].double()).abs() <= tol_for(torch.bfloat16) * terms).all())
