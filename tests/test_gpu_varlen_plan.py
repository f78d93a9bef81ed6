"""The packed-batch plan kernel: checkpoint slots and start order of the documents, against torch (whole numbers: equal)."""
import ctypes as C

import pytest
import torch

from tests.gpu_util import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 1025, 2048, 2049, 2080, 5000, 40000])     # one warp, padding to 4, CTA edges, ranked / counted
def test_plan_matches_torch(n):
    from palimpsa_b200 import _lib as L
    gen = torch.Generator().manual_seed(n)
    lens = torch.randint(0, 50, (n,), generator=gen)                   # ties and empty documents included
    lens[-1] = 30_000                                                  # a long one last
    cu = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)]).to(torch.int32).to(DEV)
    coff, order = (torch.full((n,), -1, dtype=torch.int32, device=DEV) for _ in range(2))
    L.check(L.lib().palimpsa_varlen_plan(cu.data_ptr(), n, coff.data_ptr(), order.data_ptr(),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream)), "plan")
    blocks = (lens + L.CKPT_INTERVAL - 1) // L.CKPT_INTERVAL
    assert torch.equal(coff.cpu().long(), blocks.cumsum(0) - blocks)
    if n > 2048:                               # by class, four to a power of two, in order of index inside one
        e = lens.clamp(min=1).log2().floor().long()
        lens = torch.where(lens < 4, lens, 4 * e + lens // (1 << (e - 2).clamp(min=0)) % 4)
    want = torch.argsort(lens, descending=True, stable=True)
    assert torch.equal(order.cpu().long(), want)
