"""Layer kernels for 16-bit rows of at most 128 elements (8 or 16 lanes a row) against the torch restatement: both lane counts,
rows that leave lanes idle, odd row counts, head groups, and rows just outside of them that the other kernels take."""
import pytest
import torch

from oracle import layer_oracle as lo
from tests.gpu_util import tol_for
from tests.test_gpu_layer import _check, _epilogue_pair, _prologue_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 8, 8), (1, 33, 3, 1, 64, 64), (3, 7, 5, 5, 72, 16), (2, 19, 4, 2, 120, 128),
                                   (1, 301, 6, 3, 48, 96), (1, 9, 2, 2, 128, 136), (1, 9, 2, 2, 60, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_prologue(shape, dtype):
    B, T, H, Hq, K, V = shape
    got, ref = _prologue_pair(lo.make_layer_inputs(5, B, T, H, Hq, K, V, dtype), dtype)
    _check(got, ref, tol_for(dtype), f"prologue {shape} {dtype}")


@pytest.mark.parametrize("shape", [(1, 1, 1, 8), (1, 33, 3, 64), (3, 7, 5, 72), (1, 2111, 7, 128), (2, 19, 4, 104), (1, 9, 2, 132)])
@pytest.mark.parametrize("dtype,residual,gated", [(torch.bfloat16, True, True), (torch.float16, False, True),
                                                  (torch.bfloat16, False, False)])
def test_epilogue(shape, dtype, residual, gated):
    B, T, H, V = shape
    got, ref = _epilogue_pair(lo.make_layer_inputs(6, B, T, H, H, 16, V, dtype), dtype, residual, gated)
    _check(got, ref, tol_for(dtype), f"epilogue {shape} {dtype} residual={residual} gated={gated}")


def test_rows_off_a_16_byte_boundary_take_the_other_kernels():
    from palimpsa_b200.layers import layer_epilogue
    dev = "cuda:0"
    g = torch.Generator(device=dev).manual_seed(0)
    base = torch.randn(5 * 2 * 128 + 4, generator=g, device=dev).to(torch.bfloat16)
    o = base[4:].view(1, 5, 2, 128)
    w = torch.ones(128, device=dev)
    assert o.data_ptr() % 16 == 8
    assert torch.allclose(layer_epilogue(o, None, None, w).float(), layer_epilogue(o.clone(), None, None, w).float(), atol=2e-2)
