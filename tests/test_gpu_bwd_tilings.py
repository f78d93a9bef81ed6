"""The backward's tile heights (rows and warps of a CTA by head size, element type and grid), with one and two group buffers,
ragged last tiles, tokens past the last whole block and rows that start at any offset, against the float64 oracle."""
import ctypes as C

import pytest
import torch

from oracle import palimpsa_oracle as orc
from tests.gpu_util import DEV, compare, run_cuda, run_oracle, tol_for
from tests.helpers import bwd_plan

pytestmark = pytest.mark.gpu


def _tiles(N, T, H, K, V, io, unc, G):
    """Row tiles of the backward, from what its workspace holds per (token, head): 2 tiles + 1 rows of d_k and 2 (tiles + 1)
    scalars, beside the per-head partials and six roundings to 256 bytes."""
    from palimpsa_b200 import _lib as L
    p = L.Problem()
    p.num_seqs, p.seq_len, p.total_tokens, p.H, p.K, p.V = N, T, N * T, H, K, V
    p.io_dtype, p.segments, p.flags = io, G, L.FLAG_UNCERTAINTY if unc else 0
    rest = L.lib().palimpsa_bwd_workspace_bytes(C.byref(p)) - 2 * 296 * H * 4
    fits = [t for t in range(1, 80)
            if 0 <= rest - 4 * N * T * H * (L.lib().palimpsa_padded_k(K) * (2 * t + 1) + 2 * (t + 1)) <= 6 * 256]
    assert len(fits) == 1
    return fits[0]


@pytest.mark.parametrize("rows,warps,buffers,N,H,T,K,V,dtype,unc,G", [
    (64, 8, 2, 15, 2, 17, 16, 129, torch.bfloat16, False, 1),
    (32, 4, 2, 2, 1, 33, 16, 33, torch.float32, True, 1),
    (64, 8, 2, 15, 2, 17, 32, 129, torch.float16, True, 1),
    (32, 4, 2, 1, 2, 35, 31, 33, torch.bfloat16, False, 1),
    (64, 8, 1, 24, 4, 17, 48, 63, torch.float32, True, 1),       # registers split between the warpgroups, as at every d_k
    (64, 8, 1, 24, 4, 18, 48, 62, torch.bfloat16, False, 1),     # with 8 warps of 12 elements
    (64, 8, 1, 5, 1, 80, 48, 241, torch.float32, False, 5),      # the state-gradient pass of exact segments too
    (48, 6, 2, 10, 4, 17, 48, 97, torch.bfloat16, False, 1),
    (48, 6, 2, 10, 4, 17, 48, 97, torch.bfloat16, True, 1),
    (32, 4, 2, 1, 2, 17, 47, 33, torch.float32, True, 1),
    (44, 8, 1, 15, 4, 17, 64, 65, torch.float32, True, 1),
    (44, 8, 2, 15, 2, 17, 64, 129, torch.bfloat16, False, 1),
    (32, 8, 2, 15, 2, 17, 60, 65, torch.float32, False, 1),
    (16, 4, 2, 1, 2, 19, 64, 17, torch.float16, False, 1),
    (32, 8, 1, 24, 4, 17, 96, 31, torch.bfloat16, False, 1),
    (32, 8, 1, 48, 2, 5, 90, 30, torch.float32, True, 1),
    (32, 8, 1, 5, 1, 80, 96, 121, torch.float32, True, 5),
    (24, 6, 2, 10, 4, 17, 96, 49, torch.float32, False, 1),
    (16, 4, 2, 2, 1, 17, 96, 17, torch.bfloat16, True, 1),
    (24, 8, 2, 25, 4, 17, 128, 23, torch.bfloat16, False, 1),    # registers split
    (24, 8, 2, 50, 2, 18, 120, 23, torch.float32, True, 1),
    (22, 8, 2, 24, 2, 17, 128, 110, torch.float32, True, 1),
    (24, 8, 2, 15, 2, 17, 128, 67, torch.bfloat16, False, 1),
    (16, 8, 2, 15, 2, 17, 128, 33, torch.float32, True, 1),
    (8, 4, 2, 1, 2, 17, 128, 9, torch.bfloat16, True, 1),
    (16, 8, 1, 24, 4, 17, 192, 15, torch.float32, False, 1),
    (16, 8, 1, 48, 2, 5, 180, 15, torch.bfloat16, True, 1),
    (12, 6, 2, 5, 1, 64, 192, 61, torch.bfloat16, False, 4),
    (12, 6, 2, 10, 4, 17, 192, 25, torch.float32, True, 1),
    (8, 4, 2, 2, 1, 17, 180, 9, torch.float32, True, 1),
    (8, 8, 1, 2, 1, 17, 256, 7, torch.float32, True, 1),
])
def test_every_tile_matches_oracle(rows, warps, buffers, N, H, T, K, V, dtype, unc, G):
    """Every tile a CTA may have, with the group buffers that fit beside it, as the library says that it takes them."""
    from palimpsa_b200 import _lib as L
    from palimpsa_b200.ops import chunk_palimpsa
    io = {torch.float32: L.F32, torch.bfloat16: L.BF16, torch.float16: L.F16}[dtype]
    assert bwd_plan(N, T, H, K, V, dtype, unc, G) == (rows, warps, buffers)
    assert _tiles(N, T, H, K, V, io, unc, G) == -(-V // rows)
    inp = orc.make_inputs(K + V, B=N, T=T, H=H, K=K, V=V, dtype=dtype)
    a = {n: inp[n].to(DEV).requires_grad_() for n in ("q", "k", "v", "b", "gt", "g", "Ip")}
    out = chunk_palimpsa(*a.values(), output_uncertainty=unc, num_segments=G)
    got = dict(zip(("o", "o_var"), out)) if unc else {"o": out}
    sum((got[n].float() * inp["d" + n].to(DEV).float()).sum() for n in got).backward()
    got.update({"d" + n: x.grad for n, x in a.items()})
    ref = run_oracle(inp, unc=unc)
    compare({n: x.detach().cpu() for n, x in got.items()}, ref, tol_for(dtype), names=list(got), what=f"{rows} rows, {K}x{V}")


@pytest.mark.parametrize("K,V,dtype,unc,off", [
    (47, 65, torch.bfloat16, False, 0),   # odd rows of 16-bit values: every second one starts between two words
    (95, 23, torch.float16, True, 1),
    (127, 45, torch.float32, False, 0),
    (64, 66, torch.bfloat16, False, 1),   # whole rows of vectors, on buffers that do not start on one
    (48, 48, torch.bfloat16, True, 2),
    (128, 24, torch.float32, False, 1),
    (60, 50, torch.bfloat16, False, 4),   # rows of words, but not of 16 bytes
    (20, 34, torch.float32, True, 3),
    (189, 13, torch.bfloat16, True, 3),
    (255, 9, torch.float16, False, 7),
])
def test_rows_at_any_offset(K, V, dtype, unc, off):
    """Inputs that start `off` elements into their buffers give what the same values give at the front of theirs, to the bit."""
    from palimpsa_b200.ops import chunk_palimpsa
    N, T, H = 2, 37, 2
    inp = orc.make_inputs(K * V, B=N, T=T, H=H, K=K, V=V, dtype=dtype)
    res = []
    for shift in (0, off):
        def place(x):
            buf = torch.empty(x.numel() + shift, dtype=x.dtype, device=DEV)
            buf[shift:] = x.flatten().to(DEV)
            return buf[shift:].view(x.shape)
        a = {n: (place(inp[n]) if n in "qkvb" else inp[n].to(DEV)).requires_grad_() for n in ("q", "k", "v", "b", "gt", "g", "Ip")}
        out = chunk_palimpsa(*a.values(), output_uncertainty=unc, num_segments=1)
        out = list(out) if unc else [out]
        grads = torch.autograd.grad(out, list(a.values()), [place(inp[n]) for n in ("do", "do_var")[:len(out)]])
        res.append([x.detach().cpu() for x in (*out, *grads)])
    assert all(torch.equal(x, y) for x, y in zip(*res))
    names = ["o", "o_var"][:len(out)] + ["d" + n for n in a]
    compare(dict(zip(names, res[1])), run_oracle(inp, unc=unc), tol_for(dtype), names=names, what=f"{K}x{V} +{off}")


@pytest.mark.parametrize("N,H,T,K,V,dtype,unc", [
    (2, 1, 33, 16, 9, torch.float32, True),       # one row past a lane group
    (38, 4, 17, 31, 65, torch.float32, False),    # unaligned rows
    (2, 2, 35, 32, 100, torch.bfloat16, True),
    (16, 8, 17, 48, 64, torch.bfloat16, False),
    (16, 8, 17, 48, 56, torch.float32, True),
    (2, 2, 47, 47, 49, torch.float32, False),     # second tile of one row
    (8, 6, 17, 64, 128, torch.bfloat16, False),
    (5, 1, 31, 64, 66, torch.float32, True),
    (12, 2, 17, 96, 192, torch.bfloat16, False),
    (16, 2, 17, 90, 192, torch.float32, False),   # element loads
    (32, 4, 5, 96, 196, torch.bfloat16, True),    # ragged last tile
    (8, 8, 17, 128, 64, torch.float32, True), 
    (8, 6, 17, 128, 90, torch.bfloat16, False),
    (1, 2, 49, 128, 24, torch.bfloat16, True),
    (4, 4, 17, 192, 126, torch.bfloat16, False),  # 126 rows
    (2, 1, 19, 180, 30, torch.float32, True),
    (2, 2, 18, 256, 20, torch.float32, True),
])
def test_backward_tiling_matches_oracle(N, H, T, K, V, dtype, unc):
    inp = orc.make_inputs(K + V, B=N, T=T, H=H, K=K, V=V, dtype=dtype)
    compare(run_cuda(inp, "chunk", unc=unc), run_oracle(inp, unc=unc), tol_for(dtype), what=f"{N}x{H} {K}x{V}")


@pytest.mark.parametrize("segments", [0, 2])
def test_tile_height_follows_the_grid_and_the_workspace_query_with_it(segments):
    """A small grid takes shorter tiles (more row tiles, more scratch) than one of many waves or of segments."""
    from palimpsa_b200 import _lib as L
    p = L.Problem()
    p.num_seqs, p.seq_len, p.total_tokens, p.H, p.K, p.V, p.io_dtype, p.segments = 1, 64, 64, 2, 128, 128, L.BF16, segments
    tiles = 16 if segments == 0 else 6
    row = 4 * (128 * (2 * tiles + 1) + 2 * (tiles + 1))
    need = L.lib().palimpsa_bwd_workspace_bytes(C.byref(p))
    assert 0 <= need - 128 * row - 2 * 296 * 2 * 4 <= 6 * 256
    assert L.lib().palimpsa_bwd_token_cost(C.byref(p)) > 0


@pytest.mark.parametrize("B,T,H,K,V,dtype,unc", [
    (2, 256, 2, 64, 64, torch.float32, False),    # the shortest sequence that is cut
    (1, 257, 3, 31, 65, torch.float32, True),     # ragged last segment, unaligned rows
    (1, 1000, 2, 128, 128, torch.float16, False),
    (3, 511, 1, 48, 96, torch.float32, False),
])
def test_short_sequences_in_segments_match_oracle(B, T, H, K, V, dtype, unc):
    """Float32 and float16 sequences under 2048 tokens run in segments (exact float32 boundary states)."""
    from palimpsa_b200 import _lib as L
    from palimpsa_b200.ops.palimpsa._core import plan_segments
    io = L.F32 if dtype == torch.float32 else L.F16
    assert plan_segments(B, T, H, K, V, backward=True, io_dtype=io, uncertainty=unc) > 1
    inp = orc.make_inputs(T, B=B, T=T, H=H, K=K, V=V, dtype=dtype)
    mu0, I0 = orc.make_states(5, B, H, V, K, inp["Ip"])
    for state in ({}, dict(mu0=mu0, I0=I0)):
        got = run_cuda(inp, "chunk", unc=unc, **state)
        compare(got, run_oracle(inp, unc=unc, **state), tol_for(dtype), what=f"{B}x{H} T={T}")


def test_a_workspace_sized_for_more_sequences_serves_fewer():
    """A grid takes shorter tiles, and with them more scratch, than one of a sequence more: a workspace that was asked for
    with the larger batch still runs the smaller one (with taller tiles); one too small for any tiling is refused."""
    from palimpsa_b200 import _lib as L
    from palimpsa_b200.ops.palimpsa import _core
    lib, T, K = L.lib(), 40, 128

    def need(N):
        p = L.Problem()
        p.num_seqs, p.seq_len, p.total_tokens, p.H, p.K, p.V, p.io_dtype = N, T, N * T, 1, K, K, L.F32
        return lib.palimpsa_bwd_workspace_bytes(C.byref(p))

    N = next(n for n in range(8, 80) if need(n) > need(n + 1))
    own, large = need(N), need(N + 1)
    inp = {n: x.to(DEV) for n, x in orc.make_inputs(7, B=N, T=T, H=1, K=K, V=K).items()}
    a = [inp[n] for n in ("q", "k", "v", "b", "gt", "g", "Ip")]
    p = _core._problem(*a, None, None, None, None, K ** -0.5, 0)
    _, _, _, _, ckM, ckI, _, _ = _core.fwd_op(*a, None, None, None, K ** -0.5, False, True, False, False, 1)
    got = []
    for size in (own, large, 1 << 16):
        out = [torch.full_like(x, float("nan")) for x in a]
        ws = torch.empty(size, dtype=torch.uint8, device=DEV)
        prm = L.BwdParams()
        prm.struct_size, prm.p, prm.d_o = C.sizeof(L.BwdParams), p, inp["do"].data_ptr()
        prm.ckpt_M, prm.ckpt_I = ckM.data_ptr(), ckI.data_ptr()
        prm.dq, prm.dk, prm.dv, prm.db, prm.dgt, prm.dg, prm.dIp = [x.data_ptr() for x in out]
        prm.workspace, prm.workspace_bytes = ws.data_ptr(), size
        rc = lib.palimpsa_chunk_bwd(C.byref(prm), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == (-5 if size == 1 << 16 else 0)
        torch.cuda.synchronize()
        got.append(out)
    for x, y in zip(got[0], got[1]):
        assert orc.rel_err(y, x) <= 1e-5           # float32, sums in another order
