"""Every tiling of the decode kernel (padded d_k, element-wise loads, one or several row sets per warp) against the
float64 oracle, and the one-launch copy of a replayed step's inputs."""
import pytest
import torch

from oracle import palimpsa_oracle as orc
from tests.gpu_util import DEV, tol_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,H,K,V,dtype,unc", [
    (2, 3, 15, 5, torch.float32, True),       # scalar loads, fewer rows than a warp covers
    (3, 2, 16, 33, torch.bfloat16, False),    # one row past a 32-row CTA
    (2, 2, 47, 84, torch.float32, True),      # scalar loads, three chunks per lane
    (2, 2, 52, 31, torch.float32, False),     # d_k inside the padding of 64
    (64, 8, 48, 65, torch.float32, True),     # several row sets per warp, ragged last tile
    (80, 8, 96, 63, torch.float32, False),
    (40, 8, 128, 129, torch.float32, True),
    (2, 2, 192, 17, torch.float16, True),
    (24, 8, 256, 40, torch.float32, False),
    (70000, 1, 16, 2, torch.float32, False),  # more sequence-heads than a grid's second dimension takes
])
def test_tiling_matches_oracle(N, H, K, V, dtype, unc):
    from palimpsa_b200.ops import decode_step
    inp = orc.make_inputs(K + V, B=N, T=1, H=H, K=K, V=V, dtype=dtype)
    mu, I = orc.make_states(9, N, H, V, K, inp["Ip"])
    ref_o, ref_ov, ref_mu, ref_I = orc.oracle_forward(*[inp[n] for n in ("q", "k", "v", "b", "gt", "g", "Ip")], mu, I,
                                                      output_uncertainty=True)
    mu, I = mu.to(DEV), I.to(DEV)
    out = decode_step(*[inp[n].to(DEV) for n in ("q", "k", "v", "b", "gt", "g", "Ip")], mu, I, output_uncertainty=unc)
    got = dict(mu=(mu, ref_mu), I=(I, ref_I), o=(out[0] if unc else out, ref_o))
    if unc:
        got["o_var"] = (out[1], ref_ov)
    for n, (x, ref) in got.items():
        # the state is float32 whatever the io dtype, from inputs that io holds exactly
        assert orc.rel_err(x, ref) <= (1e-5 if n in ("mu", "I") else tol_for(dtype)), n


def test_replayed_step_takes_any_input_layout():
    """Contiguous inputs go through one copy launch, others through tensor copies: same static buffers either way."""
    from palimpsa_b200.ops import DecodeGraph
    N, H, K, V = 3, 2, 24, 20
    inp = {n: x.to(DEV) for n, x in orc.make_inputs(5, B=N, T=1, H=H, K=K, V=V, dtype=torch.bfloat16).items()}
    dec = DecodeGraph(inp["g"], inp["Ip"], torch.zeros(N, H, V, K, device=DEV), torch.ones(N, H, V, K, device=DEV))
    strided = inp["q"].transpose(1, 2).contiguous().transpose(1, 2)
    dec.step(strided, inp["k"].float(), inp["v"][:, 0], inp["b"], inp["gt"])
    for n in ("q", "k", "v", "b", "gt"):
        assert torch.equal(getattr(dec, n), inp[n]), n
    kept = dec.v.clone()
    dec.step(q=inp["q"])
    assert torch.equal(dec.v, kept)
    with pytest.raises(ValueError):
        dec.step(q=inp["q"][:1])
