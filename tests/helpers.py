"""Shared helpers for the test-suite (fixtures loading, tolerances)."""
import os

import numpy as np
import torch

GOLDEN_DIR = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
GOLDEN_CASES = ("check_style_unc", "bench_style", "initial_state", "varlen")
GRADS = ("dq", "dk", "dv", "db", "dgt", "dg", "dIp")

# max|x-ref| / max|ref| bounds.  fp32 and bf16 are the operator's stated tolerances against a
# float64 recurrence; GOLDEN_TOL bounds float64-oracle vs the reference's float32 run.
TOL_FP32 = 1e-5
TOL_BF16 = 2e-2
GOLDEN_TOL = 2e-5


def load_golden(name):
    z = np.load(os.path.join(GOLDEN_DIR, name + ".npz"))
    inp = {k[3:]: torch.from_numpy(z[k]) for k in z.files if k.startswith("in_")}
    out = {k[4:]: torch.from_numpy(z[k]) for k in z.files if k.startswith("out_")}
    meta = {k[5:]: z[k].item() for k in z.files if k.startswith("meta_")}
    return inp, out, meta


def _plan(which, N, T, H, K, V, dtype, unc, segments, packed, n):
    """What the library would launch for these sizes (a host query; no GPU needed)."""
    import ctypes as C

    from palimpsa_b200 import _lib as L
    p = L.Problem()
    p.num_seqs, p.seq_len, p.total_tokens, p.H, p.K, p.V = N, 0 if packed else T, T if packed else N * T, H, K, V
    p.io_dtype = {torch.float32: L.F32, torch.bfloat16: L.BF16, torch.float16: L.F16}[dtype]
    p.flags, p.segments, p.cu_seqlens = (L.FLAG_UNCERTAINTY if unc else 0), segments, (16 if packed else None)
    plan = (C.c_int32 * 3)()
    assert getattr(L.lib(), which)(C.byref(p), plan) == 0
    return tuple(plan[:n])


def fwd_plan(N, T, H, K, V, dtype=torch.float32, unc=False, segments=0, packed=False):
    """(1 for the forward kernel for tall tiles, rows of a tile); T of a packed batch is that of all its documents."""
    return _plan("palimpsa_fwd_plan", N, T, H, K, V, dtype, unc, segments, packed, 2)


def bwd_plan(N, T, H, K, V, dtype=torch.float32, unc=False, segments=0, packed=False):
    """(rows of a tile, compute warps, group buffers) of the backward."""
    return _plan("palimpsa_bwd_plan", N, T, H, K, V, dtype, unc, segments, packed, 3)
