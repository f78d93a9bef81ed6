"""The give-up path of the library's bounded in-kernel waits, executed once, safely.

A test-only library (``tests/wait_probe.cu``, not linked into ``libpalimpsa_b200.so``) launches one 32-thread CTA
that waits with the product kernels' ``tc::mbar_wait`` on an mbarrier nobody arrives at, with a poll limit of a
few thousand: the wait runs out by construction, the kernel records its code, frees the TMEM it allocated and
returns.  The test checks the code, that the same kernel succeeds when somebody does arrive, and that the
device keeps working (a normal forward/backward right after)."""
import ctypes as C
import os

import pytest
import torch

from oracle import palimpsa_oracle as orc
from tests import wait_probe
from tests.gpu_util import compare, run_cuda, run_oracle
from tests.helpers import TOL_FP32

pytestmark = pytest.mark.gpu


def test_bounded_wait_runs_out_and_the_device_stays_usable():
    if not os.path.exists(wait_probe.LIB):
        wait_probe.build()
    lib = C.CDLL(wait_probe.LIB)
    lib.palimpsa_test_wait_probe.argtypes = [C.c_int, C.c_uint, C.c_void_p, C.c_void_p]
    status = torch.full((1,), -5, dtype=torch.int32, device="cuda:0")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.palimpsa_test_wait_probe(0, 4000, status.data_ptr(), stream) == 0
    torch.cuda.synchronize()
    assert status.item() == 7                      # nobody arrived: the wait gave up after 4000 polls and said so
    assert lib.palimpsa_test_wait_probe(1, 4000, status.data_ptr(), stream) == 0
    torch.cuda.synchronize()
    assert status.item() == 0                      # with an arrival the same wait completes
    assert lib.palimpsa_test_wait_probe(0, 100, status.data_ptr(), stream) == 0   # TMEM was freed: allocate again
    torch.cuda.synchronize()
    assert status.item() == 7
    inp = orc.make_inputs(3, B=1, T=40, H=2, K=32, V=16)
    compare(run_cuda(inp, "chunk"), run_oracle(inp), TOL_FP32, what="after the probe")
    from palimpsa_b200 import _lib
    assert _lib.lib().palimpsa_tensor_core_status() == 0     # the probe's own status word is not the library's


def test_peer_wait_runs_out_records_its_code_and_poisons_the_buffer():
    """The stream-ordered wait on a peer's flag (used by the context-parallel hops) on ONE GPU: a flag nobody sets
    makes it run out after its wall-clock limit (5 ms here); it records code 7, writes a NaN into the buffer it
    guards and lets the stream go on.  After a signal the same wait passes."""
    from palimpsa_b200 import _lib
    lib = _lib.lib()
    lib.palimpsa_tensor_core_status()                                   # clear whatever earlier tests left
    flag = torch.zeros(1, dtype=torch.int64, device="cuda:0")
    guarded = torch.ones(4, dtype=torch.float32, device="cuda:0")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.palimpsa_peer_wait(flag.data_ptr(), 1, 5, guarded.data_ptr(), stream) == 0
    torch.cuda.synchronize()
    assert lib.palimpsa_tensor_core_status() == 7
    assert torch.isnan(guarded[0]) and bool((guarded[1:] == 1).all())
    assert lib.palimpsa_tensor_core_status() == 0                       # reading cleared it
    guarded.fill_(1.0)
    assert lib.palimpsa_peer_signal(flag.data_ptr(), 3, stream) == 0    # sequence numbers only grow: 3 >= 1 and >= 2
    assert lib.palimpsa_peer_wait(flag.data_ptr(), 1, 5, guarded.data_ptr(), stream) == 0
    assert lib.palimpsa_peer_wait(flag.data_ptr(), 2, 5, guarded.data_ptr(), stream) == 0
    torch.cuda.synchronize()
    assert flag.item() == 3 and lib.palimpsa_tensor_core_status() == 0 and bool((guarded == 1).all())
    assert lib.palimpsa_peer_wait(None, 1, 5, None, stream) == _lib.E_NULL
    assert lib.palimpsa_peer_signal(flag.data_ptr() + 4, 1, stream) == _lib.E_ALIGN   # flags are 8-byte aligned


@pytest.mark.parametrize("T,V,rows,aligned", [(45, 40, 48, 1), (16, 40, 16, 1), (45, 33, 24, 0)])
def test_tall_forward_that_gives_up_marks_its_outputs_states_and_checkpoint(T, V, rows, aligned):
    """The tall-tile forward's kernel from the test-only library.  With a poll limit of 0 every wait gives up: the code is
    recorded, and all outputs, the final states and the checkpoint that a backward begins with are NaN in every row, idle warps
    and ragged tiles included.  With the product's limit the same launch matches the oracle."""
    from palimpsa_b200 import _lib as L
    from palimpsa_b200.ops.palimpsa import _core
    if not os.path.exists(wait_probe.LIB):
        wait_probe.build()
    lib = C.CDLL(wait_probe.LIB)
    run = lib.palimpsa_test_tall_forward
    run.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_void_p]
    N, H, K = 2, 2, 128
    inp = orc.make_inputs(T, B=N, T=T, H=H, K=K, V=V)
    a = [inp[n].to("cuda:0") for n in ("q", "k", "v", "b", "gt", "g", "Ip")]
    prm = L.FwdParams()
    prm.struct_size, prm.p = C.sizeof(L.FwdParams), _core._problem(*a, None, None, None, None, K ** -0.5, L.FLAG_UNCERTAINTY)
    slots = N * -(-T // 16)
    out = {"o": torch.empty_like(a[2]), "o_var": torch.empty_like(a[2])}
    out.update({n: torch.empty(N, H, V, K, device="cuda:0") for n in ("final_mu", "final_I")})
    out.update({n: torch.empty(slots, H, V, K, device="cuda:0") for n in ("ckpt_M", "ckpt_I")})
    for n, x in out.items():
        setattr(prm, n, x.data_ptr())
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for give_up in (1, 0):
        for x in out.values():
            x.zero_()
        assert run(C.addressof(prm), rows, give_up, aligned, stream) == 0
        assert lib.palimpsa_test_tall_status() == (8 if give_up else 0)
        assert lib.palimpsa_test_tall_status() == 0                         # reading cleared it
        last = [n * (slots // N) + slots // N - 1 for n in range(N)]
        marked = [out[n] for n in ("o", "o_var", "final_mu", "final_I")] + [out[n][last] for n in ("ckpt_M", "ckpt_I")]
        assert all(bool((x.isnan() if give_up else x.isfinite()).all()) for x in marked)
    ref = run_oracle(inp, unc=True)
    got = {n: out[n].cpu() for n in ("o", "o_var", "final_mu", "final_I")}
    compare(got, ref, TOL_FP32, names=[*got], what="product's poll limit")


def test_large_shared_memory_is_granted_again_in_a_new_context():
    """A kernel's shared-memory limit lives in one context: after cudaDeviceReset the next launch has to raise it again.  In
    a process of its own, which ends its own context only."""
    import subprocess
    import sys
    if not os.path.exists(wait_probe.LIB):
        wait_probe.build()
    prog = ("import ctypes\n"
            f"f = ctypes.CDLL({wait_probe.LIB!r}).palimpsa_test_smem_grant\n"
            "print([f(100 * 1024, 0), f(200 * 1024, 0), f(100 * 1024, 1), f(100 * 1024, 0), f(228 * 1024, 0), f(8192, 0)])\n")
    r = subprocess.run([sys.executable, "-c", prog], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "[0, 0, 0, 0, -2, 0]", (r.stdout, r.stderr[-500:])
