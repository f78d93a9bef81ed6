"""The packed-batch plan kernel: checkpoint slots and start order of the documents, against torch (whole numbers: equal)."""
import ctypes as C

import pytest
import torch

from tests.gpu_util import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 1025, 2048, 2049])     # one warp, padding to 4, CTA edges, sorted / unsorted
def test_plan_matches_torch(n):
    from palimpsa_b200 import _lib as L
    gen = torch.Generator().manual_seed(n)
    lens = torch.randint(0, 50, (n,), generator=gen)                   # ties and empty documents included
    cu = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)]).to(torch.int32).to(DEV)
    coff, order = (torch.full((n,), -1, dtype=torch.int32, device=DEV) for _ in range(2))
    L.check(L.lib().palimpsa_varlen_plan(cu.data_ptr(), n, coff.data_ptr(), order.data_ptr(),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream)), "plan")
    blocks = (lens + L.CKPT_INTERVAL - 1) // L.CKPT_INTERVAL
    assert torch.equal(coff.cpu().long(), blocks.cumsum(0) - blocks)
    want = torch.argsort(lens, descending=True, stable=True) if n <= 2048 else torch.arange(n)
    assert torch.equal(order.cpu().long(), want)
