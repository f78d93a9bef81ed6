"""The torch custom-op registrations (schema, fake/meta kernels, autograd wiring) as torch.compile and
activation checkpointing need them (the reference's blocks are GradientCheckpointingLayers,
palimpsa/models/palimpsa/modeling_palimpsa.py:34)."""
import pytest
import torch

from oracle import palimpsa_oracle as orc
from tests.gpu_util import DEV

pytestmark = pytest.mark.gpu


def _args(T=40, dtype=torch.float32, grad=True):
    inp = orc.make_inputs(1, B=2, T=T, H=2, K=32, V=16, dtype=dtype)
    return [inp[n].to(DEV).requires_grad_(grad) for n in ("q", "k", "v", "b", "gt", "g", "Ip")]


def test_opcheck_forward_op():
    from palimpsa_b200.ops.palimpsa import _core
    q, k, v, b, gt, g, Ip = _args()
    args = (q, k, v, b, gt, g, Ip, None, None, None, 0.25, False, True, True, False, 1)
    torch.library.opcheck(_core.fwd_op, args, test_utils=("test_schema", "test_faketensor", "test_autograd_registration"))


def test_activation_checkpointing_recomputes_consistently():
    from torch.utils.checkpoint import checkpoint
    from palimpsa_b200.ops import chunk_palimpsa
    a1, a2 = _args(), _args()
    o1 = chunk_palimpsa(*a1)
    o2 = checkpoint(lambda *xs: chunk_palimpsa(*xs), *a2, use_reentrant=False)
    w = torch.randn_like(o1)
    (o1 * w).sum().backward()
    (o2 * w).sum().backward()
    assert torch.equal(o1, o2)
    for x, y in zip(a1, a2):
        assert torch.equal(x.grad, y.grad)


def test_torch_compile_traces_through_the_op():
    from palimpsa_b200.ops import chunk_palimpsa
    args = _args(grad=False)

    def f(q, k, v, b, gt, g, Ip):
        return chunk_palimpsa(q * 1.0, k, v, b, gt, g, Ip) + 1.0

    ref = f(*args)
    out = torch.compile(f, backend="aot_eager", fullgraph=True)(*args)
    assert torch.allclose(ref, out)


def _decode_args(dtype=torch.bfloat16):
    N, H, K, V = 3, 2, 32, 16
    inp = orc.make_inputs(3, B=N, T=1, H=H, K=K, V=V, dtype=dtype)
    mu, I = orc.make_states(4, N, H, V, K, inp["Ip"])
    return [inp[n].to(DEV) for n in ("q", "k", "v", "b", "gt", "g", "Ip")] + [mu.to(DEV), I.to(DEV)]


def test_opcheck_decode_step_op():
    """``palimpsa_b200::decode_step`` declares that it mutates the two cache tensors; schema and fake kernel agree."""
    from palimpsa_b200.ops.palimpsa import decode as D
    args = (*_decode_args(), 0.25, True)
    torch.library.opcheck(D.decode_step_op, args, test_utils=("test_schema", "test_faketensor"))


def test_torch_compile_decode_loop_updates_the_cache_in_place():
    from palimpsa_b200.ops import decode_step
    args = _decode_args()
    ref_args = [x.clone() for x in args]

    def loop(q, k, v, b, gt, g, Ip, mu, I):
        o = None
        for _ in range(3):
            o = decode_step(q, k, v, b, gt, g, Ip, mu, I)
        return o + 0.0

    ref = loop(*ref_args)
    out = torch.compile(loop, backend="aot_eager", fullgraph=True)(*args)
    assert torch.equal(ref, out)
    assert torch.equal(args[7], ref_args[7]) and torch.equal(args[8], ref_args[8])      # caches advanced identically
    assert not torch.equal(args[7], _decode_args()[7])


def _raises_before_launch(op, args, i, bad, exc):
    args = list(args)
    args[i] = bad
    with pytest.raises(exc):
        op(*args)
    torch.cuda.synchronize()


def test_registered_operators_check_every_tensor():
    """Called directly, the operators refuse host tensors, another dtype and a wrong length (each would be a bad address or
    garbage in the kernel), and take rows of any stride."""
    from palimpsa_b200.ops.palimpsa import _core, decode as D
    a = _args(grad=False)
    fwd = (*a, None, None, None, 0.25, False, True, True, False, 1)
    for i in range(7):
        _raises_before_launch(_core.fwd_op, fwd, i, a[i].cpu(), (RuntimeError, ValueError))
    _raises_before_launch(_core.fwd_op, fwd, 4, a[4].bfloat16(), TypeError)
    _raises_before_launch(_core.fwd_op, fwd, 5, a[5][:1], ValueError)
    _raises_before_launch(_core.fwd_op, fwd, 2, a[2].bfloat16(), TypeError)
    o, _, _, _, ckM, ckI, _, _ = _core.fwd_op(*fwd)
    strided = [x.transpose(1, 2).contiguous().transpose(1, 2) if x.dim() == 4 else x for x in a]
    assert torch.equal(_core.fwd_op(*strided, *fwd[7:])[0], o)
    bwd = (torch.ones_like(o), None, *a, None, None, ckM, ckI, 0.25, False, False, None)
    for i in (0, 2, 7, 8, 11):
        _raises_before_launch(_core.bwd_op, bwd, i, bwd[i].cpu(), (RuntimeError, ValueError))
    _raises_before_launch(_core.bwd_op, bwd, 11, ckM[:2], ValueError)
    ref = _core.bwd_op(*bwd)
    got = _core.bwd_op(torch.ones_like(o)[..., :1].expand_as(o), *bwd[1:])
    assert all(torch.equal(x, y) for x, y in zip(ref, got))
    dec = (*_decode_args(), 0.25, False)
    for i in (0, 5, 7):
        _raises_before_launch(D.decode_step_op, dec, i, dec[i].cpu(), (RuntimeError, ValueError))
    _raises_before_launch(D.decode_step_op, dec, 7, dec[7].bfloat16(), TypeError)


def _state():
    return torch.zeros(2, 2, 16, 32, device=DEV), torch.ones(2, 2, 16, 32, device=DEV)


@pytest.mark.parametrize("pre_dispatch", [False, True])
def test_traced_calls_depend_on_their_inputs(pre_dispatch):
    """Both fx tracers see the operator; a graph with the traced call's result as a constant would pass on one input."""
    from torch.fx.experimental.proxy_tensor import make_fx
    from palimpsa_b200.ops import chunk_palimpsa, decode_step
    graph = make_fx(lambda *x: chunk_palimpsa(*x), pre_dispatch=pre_dispatch)(*_args(grad=False))
    other = [x * 0.5 for x in _args(grad=False)]
    assert torch.equal(graph(*other), chunk_palimpsa(*other))
    step = make_fx(lambda *x: decode_step(*x), pre_dispatch=pre_dispatch)(*_args(T=1, grad=False), *_state())
    other = [x * 0.5 for x in _args(T=1, grad=False)]
    s1, s2 = _state(), _state()
    assert torch.equal(step(*other, *s1), decode_step(*other, *s2)) and torch.equal(s1[0], s2[0])


def test_jit_trace_records_the_operator():
    from palimpsa_b200.ops import chunk_palimpsa, decode_step
    f = torch.jit.trace(lambda *x: chunk_palimpsa(*x), tuple(_args(grad=False)), check_trace=False)
    other = [x * 0.5 for x in _args(grad=False)]
    assert "palimpsa_b200::fwd" in str(f.graph) and torch.equal(f(*other), chunk_palimpsa(*other))
    f = torch.jit.trace(lambda *x: decode_step(*x), (*_args(T=1, grad=False), *_state()), check_trace=False)
    other = [x * 0.5 for x in _args(T=1, grad=False)]
    assert torch.equal(f(*other, *_state()), decode_step(*other, *_state()))


def test_negated_views_are_read_with_their_sign():
    from palimpsa_b200.ops import DecodeGraph, chunk_palimpsa, decode_step
    a = _args(grad=False)
    neg = [torch._neg_view(a[0]), *a[1:]]
    assert torch.equal(chunk_palimpsa(*neg), chunk_palimpsa(-a[0], *a[1:]))
    t = _args(T=1, grad=False)
    assert torch.equal(decode_step(torch._neg_view(t[0]), *t[1:], *_state()), decode_step(-t[0], *t[1:], *_state()))
    g1, g2 = DecodeGraph(t[5], t[6], *_state(), dtype=torch.float32), DecodeGraph(t[5], t[6], *_state(), dtype=torch.float32)
    assert torch.equal(g1.step(torch._neg_view(t[0]), *t[1:5]), g2.step(-t[0], *t[1:5]))


def test_subclasses_and_function_modes_see_the_operator():
    from torch.overrides import TorchFunctionMode
    from palimpsa_b200.ops import chunk_palimpsa, decode_step

    class Sub(torch.Tensor):
        pass

    a, t = _args(grad=False), _args(T=1, grad=False)
    assert type(chunk_palimpsa(a[0].as_subclass(Sub), *a[1:])) is Sub
    assert type(decode_step(t[0].as_subclass(Sub), *t[1:], *_state())) is Sub
    seen = []

    class Mode(TorchFunctionMode):
        def __torch_function__(self, f, types, args=(), kwargs=None):
            seen.append(str(f))
            return f(*args, **(kwargs or {}))

    with Mode():
        chunk_palimpsa(*a)
    assert any("palimpsa_b200" in s or "fwd" in s for s in seen)


def test_a_call_below_autograd_makes_no_graph():
    """Inside another operator's kernel autograd is off by dispatch key although gradients are enabled."""
    from palimpsa_b200.ops import chunk_palimpsa
    a = _args()
    with torch._C._AutoDispatchBelowAutograd():
        o = chunk_palimpsa(*a)
    assert not o.requires_grad
    with torch.inference_mode():
        assert torch.equal(chunk_palimpsa(*a), o)


def test_ordinary_calls_take_the_direct_route():
    """Plain tensors go straight to the kernels, with gradients or without, under autocast, in inference mode, with hooks on
    saved tensors; the native entry hands everything else back."""
    from torch.utils._python_dispatch import TorchDispatchMode
    from palimpsa_b200.ops.palimpsa import _core
    ext = _core.native()

    def direct(a):
        run = ext.run(*a, None, None, None, False, False, None, False, None, True) is not NotImplemented
        t = [x.detach()[:, :1] if x.dim() > 1 else x.detach() for x in a]
        step = ext.decode_step(*t, *_state(), None, False) is not NotImplemented
        assert run == step
        return run

    a = _args()
    assert direct(a) and direct(_args(grad=False)) and direct([torch.nn.Parameter(x) for x in a])
    with torch.no_grad():
        assert direct(a)
    with torch.inference_mode():
        assert direct(a) and direct([x + 0 for x in a])
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert direct(a)
    with torch.autograd.graph.save_on_cpu():
        assert direct(a)
    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, f, types, args=(), kwargs=None):
            return f(*args, **(kwargs or {}))

    with Mode():
        assert not direct(a)
    with torch._C._AutoDispatchBelowAutograd():
        assert not direct(a)
    assert not direct([torch._neg_view(a[0].detach()), *a[1:]])
    assert not direct([x.detach().cpu() for x in a])


def test_an_exported_program_loads_after_a_bare_import(tmp_path):
    import os
    import subprocess
    import sys
    from palimpsa_b200.ops import chunk_palimpsa

    class Mod(torch.nn.Module):
        def forward(self, *x):
            return chunk_palimpsa(*x)

    path = str(tmp_path / "p.pt2")
    torch.export.save(torch.export.export(Mod(), tuple(_args(grad=False))), path)
    prog = f"import palimpsa_b200, torch\nprint('loaded', torch.export.load({path!r}).graph)"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", prog], capture_output=True, text=True, cwd=root)
    assert r.returncode == 0 and "palimpsa_b200.fwd" in r.stdout, r.stderr[-1500:]


def test_compiled_autograd_takes_the_nodes():
    """Compiled autograd hashes a node's state; the operator's and the layer passes' hold plain numbers."""
    import torch._dynamo.compiled_autograd as ca
    from palimpsa_b200.layers import layer_epilogue, layer_prologue
    from palimpsa_b200.ops import chunk_palimpsa

    def step():
        gen = torch.Generator(DEV).manual_seed(3)
        r = lambda *s: torch.randn(*s, generator=gen, device=DEV).requires_grad_()
        a = [r(2, 9, 2, 32), r(2, 9, 2, 32), r(2, 9, 4, 16), r(2, 9, 4, 16), r(2, 9, 4), r(2, 9, 4), r(4), r(4)]
        w, D, g, Ip = r(16), r(4), torch.ones(4, device=DEV, requires_grad=True), torch.ones(4, device=DEV, requires_grad=True)
        q, k, v, b, dt = layer_prologue(*a)
        y = layer_epilogue(chunk_palimpsa(q, k, v, b, dt, g, Ip), a[2], D, w, a[3], eps=1e-4)
        return (y ** 2).sum(), [*a, w, D, g, Ip]

    loss, ref = step()
    loss.backward()
    loss, got = step()
    with ca._enable(torch.compile(backend="eager")):
        loss.backward()
    assert all(torch.equal(x.grad, y.grad) for x, y in zip(ref, got))


def test_a_profile_names_the_operators():
    from palimpsa_b200.ops import chunk_palimpsa, decode_step
    a = _args()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        chunk_palimpsa(*a).sum().backward()
        decode_step(*_args(T=1, grad=False), *_state())
    names = {e.key for e in prof.key_averages()}
    assert {"palimpsa_b200::fwd", "palimpsa_b200::bwd", "palimpsa_b200::decode_step"} <= names


def test_the_carry_switch_holds_on_the_operator_route(monkeypatch):
    """carry_on_tensor_cores = False: the exact carried terms, whichever way the call reaches the kernels."""
    from palimpsa_b200.ops import chunk_palimpsa
    from palimpsa_b200.ops.palimpsa import _core
    inp = orc.make_inputs(17, B=1, T=300, H=2, K=64, V=128, dtype=torch.bfloat16)
    inp["gt"] = inp["gt"] * 0.05

    def grads(call):
        a = [inp[n].to(DEV).requires_grad_() for n in ("q", "k", "v", "b", "gt", "g", "Ip")]
        return torch.autograd.grad(call(a), a, inp["do"].to(DEV))

    direct = lambda a: chunk_palimpsa(*a, num_segments=3)
    op = lambda a: _core.fwd_op(*a, None, None, None, 64 ** -0.5, False, True, False, False, 3)[0]
    rounded = grads(direct)
    assert all(torch.equal(x, y) for x, y in zip(rounded, grads(op)))
    monkeypatch.setattr(_core, "carry_on_tensor_cores", False)
    exact = grads(direct)
    assert not torch.equal(exact[4], rounded[4])
    assert all(torch.equal(x, y) for x, y in zip(exact, grads(op)))
    traced = grads(lambda a: torch.compile(direct, backend="aot_eager")(a))
    assert all(torch.equal(x, y) for x, y in zip(exact, traced))
