"""Several Python threads in front of one GPU."""
import threading
import time

import pytest
import torch

from oracle import palimpsa_oracle as orc
from tests.gpu_util import DEV

pytestmark = pytest.mark.gpu


def _args(T):
    inp = orc.make_inputs(1, B=2, T=T, H=2, K=32, V=16)
    return [inp[n].to(DEV) for n in ("q", "k", "v", "b", "gt", "g", "Ip")]


@pytest.mark.parametrize("what", ["chunk", "decode", "layer"])
def test_a_call_that_waits_for_the_device_lets_other_threads_run(what):
    """A stream busy for about a second and more launches than its queue holds: the call that then waits for a free place
    must not keep the interpreter from the other threads."""
    from palimpsa_b200.layers import layer_epilogue
    from palimpsa_b200.ops import chunk_palimpsa, decode_step
    a = _args(1 if what == "decode" else 16)
    mu, I = torch.zeros(2, 2, 16, 32, device=DEV), torch.ones(2, 2, 16, 32, device=DEV)
    w = torch.ones(16, device=DEV)
    call = {"chunk": lambda: chunk_palimpsa(*a), "decode": lambda: decode_step(*a, mu, I),
            "layer": lambda: layer_epilogue(a[2], None, None, w)}[what]
    call()
    torch.cuda.synchronize()
    took = []

    def worker():
        t0 = time.perf_counter()
        with torch.no_grad():
            for _ in range(4000):
                call()
        took.append(time.perf_counter() - t0)

    torch.cuda._sleep(2_000_000_000)                  # about one second
    th = threading.Thread(target=worker)
    worst, last = 0.0, time.perf_counter()
    th.start()
    while th.is_alive():
        time.sleep(0.001)
        now = time.perf_counter()
        worst, last = max(worst, now - last), now
    th.join()
    torch.cuda.synchronize()
    assert took[0] > 0.5                               # it did wait
    assert worst < 0.25, f"the other thread stood still for {worst:.2f} s"
