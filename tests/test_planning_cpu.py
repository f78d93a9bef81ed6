"""Host-side planning logic that needs no GPU: segment planning, slice widths, shard bounds."""
import pytest


def test_plan_segments():
    from palimpsa_b200.ops.palimpsa._core import plan_segments, segment_len
    assert plan_segments(8, 4096, 6, 128, 128) == 1        # 384 (sequence, head, tile) CTAs fill the GPU
    assert plan_segments(4, 4096, 6, 128, 128) == 1        # 192 CTAs: still above the SM count
    assert plan_segments(3, 4096, 6, 128, 128) == 16       # 144 CTAs: 256-token segments
    assert plan_segments(1, 131072, 12, 128, 128) == 32    # long sequence: capped at 32 pieces
    assert plan_segments(1, 1024, 2, 64, 64) == 1          # short sequences never
    assert plan_segments(1, 2048, 1, 64, 64) == 8
    # with a backward to follow, the backward grid decides (one CTA of up to 12 warps per SM, 148 SMs assumed here)
    kw = dict(backward=True)
    assert plan_segments(8, 4096, 6, 128, 128, **kw) == 1     # 288 CTAs of 22 rows = 1.95 waves
    assert plan_segments(4, 4096, 6, 128, 128, **kw) == 1     # 144 CTAs = 0.97 of a wave
    assert plan_segments(5, 4096, 6, 128, 128, **kw) == 16    # 180 CTAs = 1.2 waves: the second one mostly idle
    assert plan_segments(2, 4096, 6, 128, 128, **kw) == 16    # 72 CTAs: half the SMs idle
    assert plan_segments(8, 4096, 16, 48, 48, **kw) == 1      # the 170M model's heads: 128 CTAs = 0.86 of a wave
    assert plan_segments(8, 4096, 12, 64, 64, **kw) == 16     # 192 CTAs = 1.3 waves
    assert plan_segments(8, 1024, 12, 64, 64, **kw) == 1      # short sequences never
    # packed rows: only the document count is known; segments when the documents alone cannot fill one wave
    assert plan_segments(7, 16384, 16, 48, 48, packed=True, **kw) == 32     # 112 CTAs: the longest document binds
    assert plan_segments(14, 32768, 16, 48, 48, packed=True, **kw) == 1     # 224 CTAs, started longest first
    assert plan_segments(14, 32768, 6, 128, 128, packed=True, **kw) == 1
    assert plan_segments(3, 32768, 6, 128, 128, packed=True) == 32          # forward only: 144 forward CTAs
    for T, G in ((4096, 16), (333, 3), (17, 4), (1, 1)):
        L = segment_len(T, G)
        assert L % 16 == 0 and L * G >= T and L >= 16


def test_bf16_boundaries_are_rounded_only_where_the_grid_is_starved():
    """bf16 shapes whose carried terms or summaries go through the tensor cores (rounded there) stay uncut where the grid of
    the nominal tiles fills 80 % of its waves, however the tile heights are tuned; the same shapes in float32 and float16,
    and those only the exact passes serve, are cut by cost alone."""
    from palimpsa_b200 import _lib as L
    from palimpsa_b200.ops.palimpsa._core import plan_segments
    kw = dict(backward=True)
    for N, K, V in ((30, 64, 128), (60, 64, 128), (40, 96, 96), (40, 80, 96), (128, 48, 48), (24, 128, 128)):
        assert plan_segments(N, 4096, 1, K, V, **kw) == 1, (N, K, V)
    assert all(plan_segments(n, 4096, 1, 64, 128, packed=True, **kw) == 1 for n in range(37, 50))
    assert plan_segments(30, 4096, 1, 64, 128, io_dtype=L.F16, **kw) == 16       # exact: 3.39 ms uncut, 3.28 cut
    # starved grids: rounded, and faster cut
    assert plan_segments(16, 4096, 1, 128, 128, **kw) == 16                      # 3.02 ms uncut, 2.51 cut
    assert plan_segments(32, 4096, 1, 96, 96, **kw) == 16                        # 3.56 / 3.04
    # exact passes cost more: 16 heads of 96x192 3.54 ms uncut, 3.79 cut; 64 of 128x64 in float16 5.61 / 6.66
    assert plan_segments(16, 4096, 1, 96, 192, **kw) == 1
    assert plan_segments(64, 4096, 1, 128, 64, io_dtype=L.F16, **kw) == 1
    assert plan_segments(8, 4096, 1, 96, 192, **kw) == 16                        # 2.94 / 2.17


def test_ramped_widths():
    from palimpsa_b200.host_pipeline import ramped_widths
    assert ramped_widths(8) == [1, 2, 2, 2, 1]
    assert ramped_widths(9, middle=3) == [1, 3, 3, 1, 1]
    assert ramped_widths(1) == [1] and ramped_widths(2) == [1, 1]
    for b in range(1, 40):
        w = ramped_widths(b)
        assert sum(w) == b and min(w) >= 1 and w[0] == 1 and w[-1] == 1


def test_shard_bounds_cover_without_overlap():
    from palimpsa_b200.parallel import shard_bounds
    for n in (0, 1, 7, 8, 131072):
        for world in (1, 2, 3, 8):
            spans = [shard_bounds(n, r, world) for r in range(world)]
            assert spans[0][0] == 0 and spans[-1][1] == n
            assert all(a[1] == b[0] for a, b in zip(spans, spans[1:]))
            sizes = [hi - lo for lo, hi in spans]
            assert max(sizes) - min(sizes) <= 1


def test_layer_wrappers_reject_cpu_tensors():
    import torch
    from palimpsa_b200.layers import layer_epilogue, layer_prologue
    x = torch.zeros(1, 2, 2, 8)
    with pytest.raises(RuntimeError):
        layer_epilogue(x, None, None, torch.ones(8))
    with pytest.raises(RuntimeError):
        layer_prologue(x, x, x, x, torch.zeros(1, 2, 2), torch.zeros(1, 2, 2), torch.zeros(2), torch.zeros(2))


def test_layer_prologue_without_heads_is_an_error():
    """No query heads at all: an exception (the head ratio is not divided by zero).  Fake tensors stand in for the GPU's;
    a child process, since an integer division by zero would end it."""
    import os
    import subprocess
    import sys
    prog = ("import torch\n"
            "from torch._subclasses.fake_tensor import FakeTensorMode\n"
            "from palimpsa_b200.layers import layer_prologue\n"
            "with FakeTensorMode(allow_non_fake_inputs=True):\n"
            "    e = lambda *s: torch.empty(*s, device='cuda')\n"
            "    try:\n"
            "        layer_prologue(e(1, 2, 0, 8), e(1, 2, 0, 8), e(1, 2, 4, 8), e(1, 2, 4, 8), e(1, 2, 4), e(1, 2, 4), e(4), e(4))\n"
            "    except ValueError as x:\n"
            "        print('ValueError', x)\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", prog], capture_output=True, text=True, cwd=root)
    assert r.returncode == 0 and "ValueError layer_prologue" in r.stdout, (r.returncode, r.stderr[-500:])


def test_another_torch_version_rebuilds_the_front_end(monkeypatch, tmp_path):
    from palimpsa_b200 import build as b
    monkeypatch.setattr(b, "_older", lambda target, sources: False)      # by their times the files are up to date
    monkeypatch.setattr(b, "EXT_STAMP", str(tmp_path / "stamp"))
    assert b.needs_build()                                               # built for an unknown version
    (tmp_path / "stamp").write_text(b._torch_version() + "\n")
    assert not b.needs_build()
    monkeypatch.setattr(b, "_torch_version", lambda: "0.0.1")
    assert b.needs_build()


def _in_fresh_process(prog):
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", prog], capture_output=True, text=True, cwd=root)
    assert r.returncode == 0, r.stderr[-1500:]
    return r.stdout


def test_threads_may_make_the_first_call_together():
    out = _in_fresh_process("""
import sys, threading
from palimpsa_b200.ops.palimpsa import _core
sys.setswitchinterval(1e-6)
gate, errors = threading.Barrier(8), []
def first():
    gate.wait()
    try:
        _core.native()
    except Exception as e:
        errors.append(e)
threads = [threading.Thread(target=first) for _ in range(8)]
[t.start() for t in threads]
[t.join() for t in threads]
print("errors", errors)
""")
    assert "errors []" in out


def test_importing_the_package_registers_the_operators():
    """A program saved with an operator call in it has to load in a process that has only imported the package."""
    out = _in_fresh_process("""
import palimpsa_b200, torch
print([str(getattr(torch.ops.palimpsa_b200, n).default._schema).split("(")[0] for n in ("fwd", "bwd", "decode_step")])
""")
    assert "palimpsa_b200::fwd" in out and "palimpsa_b200::bwd" in out and "palimpsa_b200::decode_step" in out


def test_the_module_can_be_reloaded():
    """A reload registers the fake kernels over those that are there."""
    assert "again" in _in_fresh_process("""
import importlib
from palimpsa_b200.ops.palimpsa import _core
importlib.reload(_core)
print("again", _core.native())
""")


def test_an_unbuilt_package_imports_and_says_so_at_the_first_call():
    out = _in_fresh_process("""
import ctypes, torch
real = ctypes.CDLL
def refuse(path, *a, **k):
    raise OSError(path)
ctypes.CDLL = refuse
import palimpsa_b200
from palimpsa_b200 import _lib
try:
    palimpsa_b200.chunk_palimpsa(*[torch.zeros(1, 1, 1, 16)] * 4, torch.zeros(1, 1, 1), torch.ones(1), torch.ones(1))
except _lib.PalimpsaLibraryError as e:
    print("loud", e)
""")
    assert "loud" in out


def _fake(T, decode=False):
    import torch
    e = lambda *s, **kw: torch.empty(*s, device="cuda", **kw)
    a = [e(2, T, 2, 32), e(2, T, 2, 32), e(2, T, 2, 16), e(2, T, 2, 16), e(2, T, 2), e(2), e(2)]
    return a + [e(2, 2, 16, 32), e(2, 2, 16, 32)] if decode else a


def test_fake_tensors_go_through_the_registered_operators():
    """Shape propagation without a GPU, outside of any compiler: forward (and backward where there is a GPU), and decode."""
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode
    from palimpsa_b200.ops import chunk_palimpsa, decode_step, fused_recurrent_palimpsa
    with FakeTensorMode():
        for fn in (chunk_palimpsa, fused_recurrent_palimpsa):
            a = [x.requires_grad_() for x in _fake(2100)]
            o, mu, I = fn(*a, output_final_state=True)
            assert o.shape == (2, 2100, 2, 16) and mu.shape == I.shape == (2, 2, 16, 32) and o.device.type == "cuda"
            assert o.requires_grad
            if torch.cuda.is_available():      # torch's own backward needs a device for fake CUDA tensors too
                o.sum().backward()
                assert a[0].grad.shape == a[0].shape and a[5].grad.shape == (2,)
        assert decode_step(*_fake(1, decode=True)).shape == (2, 1, 2, 16)


def test_options_are_taken_by_their_truth_and_value():
    """Flags of any type, a float as a segment count and numbers of other types as a scale, as from Python code before the
    native entries: conversions happen in front of them (fake tensors are handed back, so nothing runs here)."""
    import numpy as np
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode
    from palimpsa_b200.ops import chunk_palimpsa, decode_step, fused_recurrent_palimpsa
    with FakeTensorMode():
        a = _fake(64)
        for fn in (chunk_palimpsa, fused_recurrent_palimpsa):
            out, mu, I = fn(*a, output_final_state=object(), output_uncertainty=[1], scale=np.float32(0.5))
            assert len(out) == 2 and mu.shape == I.shape
        assert chunk_palimpsa(*a, num_segments=4.0, scale="0.5", output_final_state="").shape == (2, 64, 2, 16)
        assert len(decode_step(*_fake(1, decode=True), scale="0.5", output_uncertainty="yes")) == 2


@pytest.mark.parametrize("T", [64, 600, 3000])
def test_a_symbolic_length_stays_symbolic(T):
    """The plan is made for the traced length without fixing it."""
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.fx.experimental.symbolic_shapes import DimDynamic, ShapeEnv, StatelessSymbolicContext
    from palimpsa_b200.ops import chunk_palimpsa
    env = ShapeEnv()
    mode = FakeTensorMode(shape_env=env)
    like = [torch.empty(s, device="meta") for s in ((2, T, 2, 32), (2, T, 2, 16), (2, T, 2), (2,))]
    free = lambda t: StatelessSymbolicContext([DimDynamic.DYNAMIC if i == 1 else DimDynamic.STATIC for i in range(t.dim())])
    with mode:
        q, v, gt, g = [mode.from_tensor(t, symbolic_context=free(t)) for t in like]
        s = q.shape[1]
        cuda = lambda *shape: torch.empty(*shape, device="cuda")
        o = chunk_palimpsa(cuda(2, s, 2, 32), cuda(2, s, 2, 32), cuda(2, s, 2, 16), cuda(2, s, 2, 16), cuda(2, s, 2), cuda(2),
                           cuda(2))
        assert isinstance(o.shape[1], torch.SymInt) and str(o.shape[1]) == str(s) and not str(s).isdigit()


def test_missing_library_is_a_loud_error(monkeypatch, tmp_path):
    """No CPU or PyTorch fallback: without the built CUDA library every entry fails with a clear message."""
    from palimpsa_b200 import _lib
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", str(tmp_path / "libpalimpsa_b200.so"))
    with pytest.raises(_lib.PalimpsaLibraryError, match="no CPU or PyTorch fallback"):
        _lib.lib()


def test_forward_tile_rows_from_the_library():
    """Pure host function of the C ABI: nominal rows of one forward CTA per head shape (what plan_segments counts CTAs with)."""
    from palimpsa_b200 import _lib
    lib = _lib.lib()
    assert lib.palimpsa_fwd_tile_rows(128, 128) == 16
    assert lib.palimpsa_fwd_tile_rows(64, 64) == 32
    assert lib.palimpsa_fwd_tile_rows(64, 8) == 16         # short d_v: one warp instead of two, half the tile
    assert lib.palimpsa_fwd_tile_rows(300, 64) == 0        # d_k above the supported maximum
    assert lib.palimpsa_fwd_tile_rows(48, 48) == 48        # three warps: no idle rows at the 170M model's heads
    assert lib.palimpsa_bwd_tile_rows(128, 128, _lib.BF16, 0) == 22   # 22 of the 24 rows of 8 warps x 3: 6 tiles = 132 rows
    assert lib.palimpsa_bwd_tile_rows(48, 48, _lib.BF16, 0) == 48     # 6 warps x 8 rows
    assert lib.palimpsa_bwd_tile_rows(48, 96, _lib.BF16, 0) == 48
    assert lib.palimpsa_bwd_tile_rows(64, 64, _lib.BF16, 0) == 32
    assert lib.palimpsa_bwd_tile_rows(300, 64, _lib.BF16, 0) == 0
    assert lib.palimpsa_bwd_tile_rows(64, 64, 99, 0) == 0             # unknown element type
    assert lib.palimpsa_last_error_string(_lib.E_SYMBOL).startswith(b"the library's own scratch array")


def test_the_forward_takes_tall_tiles_where_they_pay():
    """Not for the few tokens that do not make up for filling an SM with one CTA, nor where a second wave has to start."""
    import torch
    from tests.helpers import fwd_plan
    bf = torch.bfloat16
    assert [fwd_plan(1, T, 12, 128, 128, bf)[0] for T in (1, 16, 32, 64, 512)] == [0, 0, 0, 1, 1]
    assert [fwd_plan(1, T, 12, 128, 128, bf, unc=True)[0] for T in (64, 256)] == [0, 1]
    assert [fwd_plan(4, T, 16, 128, 128, bf)[0] for T in (16, 64, 256, 4096)] == [0, 0, 0, 0]    # 64 heads: two waves
    assert [fwd_plan(4, T, 16, 48, 96, bf)[0] for T in (2, 37, 4096)] == [1, 1, 1]
    assert fwd_plan(8, 4096, 6, 128, 128, bf) == (1, 48) and fwd_plan(2, 3001, 16, 96, 192, bf) == (1, 48)
    assert fwd_plan(8, 0, 6, 128, 128, bf)[0] == 0
    assert fwd_plan(40, 40 * 20, 6, 128, 128, bf, packed=True)[0] == 0


def test_backward_tiles_by_what_they_cost():
    import torch
    from tests.helpers import bwd_plan
    bf = torch.bfloat16
    assert bwd_plan(8, 4096, 6, 128, 128, bf) == (22, 8, 2)
    assert bwd_plan(8, 4096, 16, 48, 48, bf) == (48, 6, 2)
    assert bwd_plan(17, 699, 12, 96, 192, bf) == (32, 8, 1)           # 9 waves of 6 tiles
    assert bwd_plan(14, 27244, 16, 96, 192, bf, packed=True)[0] == 32
    assert bwd_plan(50, 32768, 6, 128, 72, bf, packed=True)[0] == 24   # 3 tiles for packed rows too
    # as many rows in shared memory whatever the element type; the tallest tile of every d_k serves as the least scratch
    for K in (16, 32, 48, 64, 96, 128, 192, 256):
        for unc in (False, True):
            plans = {bwd_plan(64, 2048, 8, K, 192, dt, unc) for dt in (torch.float32, bf, torch.float16)}
            assert len(plans) == 1


def test_plans_are_refused_for_what_no_launch_takes():
    import ctypes as C
    from palimpsa_b200 import _lib as L
    lib, plan, p = L.lib(), (C.c_int32 * 3)(), L.Problem()
    for fn in (lib.palimpsa_fwd_plan, lib.palimpsa_bwd_plan):
        p.num_seqs, p.seq_len, p.total_tokens, p.H, p.K, p.V, p.io_dtype = 1, 64, 64, 2, 300, 64, L.F32
        assert fn(C.byref(p), plan) != 0
        p.K = 64
        assert fn(C.byref(p), plan) == 0 and fn(C.byref(p), None) == L.E_NULL and fn(None, plan) != 0
        p.num_seqs = 0
        assert fn(C.byref(p), plan) != 0
