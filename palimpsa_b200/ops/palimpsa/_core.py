"""What the operator's Python functions share: the native front end and its registered torch operators, the general
form of the call, and the planning and parameter helpers for code that drives the C ABI itself.

Eager calls go to the native front end (csrc/torch_ops.cpp), which checks, allocates and launches without Python in
between.  ``torch.ops.palimpsa_b200.{fwd, bwd, decode_step}`` are registered there too; their fake kernels are here.
There is no fallback: CPU tensors are rejected and a missing library raises.
"""
from __future__ import annotations

import ctypes as C
import threading
from typing import Optional

import torch
from torch import Tensor
from torch.overrides import has_torch_function_variadic

from ... import _lib as L

_DT = {torch.float32: L.F32, torch.bfloat16: L.BF16, torch.float16: L.F16}

# Segmented backward: take the tensor-core route for the carried-gradient terms wherever the library supports
# the problem (bf16, d_v <= 128, padded d_k in {32,48,64,96,128}).  Tests set this to False to exercise the
# two-pass CUDA-core route on the same problems.
carry_on_tensor_cores = True


def _ptr(t: Optional[Tensor]):
    return None if t is None or t.numel() == 0 else t.data_ptr()


def _problem(q, k, v, b, gt, g, Ip, cu_seqlens, chunk_offsets, init_mu, init_I, scale, flags, seq_order=None) -> L.Problem:
    B, T, H, K = q.shape
    V = v.shape[-1]
    p = L.Problem()
    p.num_seqs = B if cu_seqlens is None else cu_seqlens.numel() - 1
    p.seq_len = T if cu_seqlens is None else 0
    p.total_tokens = B * T
    p.H, p.K, p.V = H, K, V
    p.io_dtype = _DT[q.dtype]
    p.flags = flags
    p.scale = float(scale)
    p.q, p.k, p.v, p.b = _ptr(q), _ptr(k), _ptr(v), _ptr(b)
    p.gt, p.g, p.Ip = _ptr(gt), _ptr(g), _ptr(Ip)
    p.cu_seqlens = _ptr(cu_seqlens)
    p.chunk_offsets = _ptr(chunk_offsets)
    p.init_mu, p.init_I = _ptr(init_mu), _ptr(init_I)
    p.seq_order = _ptr(seq_order)
    return p


def _stream(t: Tensor):
    return C.c_void_p(torch.cuda.current_stream(t.device).cuda_stream)


def _require_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise RuntimeError(
                "palimpsa_b200 runs on CUDA (sm_100a) only and has no CPU path; "
                "for CPU tensors use palimpsa_b200.ops.palimpsa_ref (naive recurrence).")


def padded_k(K: int) -> int:
    for s in (16, 32, 48, 64, 96, 128, 192, 256):
        if K <= s:
            return s
    raise ValueError(f"d_k = {K} is above the supported maximum of 256")


def _ckpt_slots(total_tokens: int, num_seqs: int) -> int:
    return (total_tokens + L.CKPT_INTERVAL - 1) // L.CKPT_INTERVAL + num_seqs


B200_SM_COUNT = 148     # used only when no CUDA device is visible (planning on a build machine)
_sm_count_cache = {}


def sm_count(device=None) -> int:
    """Streaming multiprocessors of ``device`` (default: the current CUDA device)."""
    if not torch.cuda.is_available():
        return B200_SM_COUNT
    idx = torch.cuda.current_device() if device is None else torch.device(device).index
    if idx is None:
        idx = torch.cuda.current_device()
    if idx not in _sm_count_cache:
        _sm_count_cache[idx] = torch.cuda.get_device_properties(idx).multi_processor_count
    return _sm_count_cache[idx]


@torch.compiler.assume_constant_result        # ints in, int out: evaluated once when a caller is traced by torch.compile
def plan_segments(N: int, T: int, H: int, K: int, V: int, device=None, backward: bool = False,
                  io_dtype: int = L.BF16, uncertainty: bool = False, packed: bool = False) -> int:
    """How many segments to cut every sequence into on one GPU.  Segments cost an extra summary pass
    (and the carried-gradient terms in backward: about a fifth of a step), so they are only used when the grid of
    (sequence, head, row-tile) CTAs would leave SMs idle, e.g. one very long sequence or a narrow batch slice.

    Forward only: the forward grid has fewer CTAs than the device has SMs.  With a backward to follow
    (``backward=True``) the backward kernel decides, since it is 3/4 of the step and keeps one CTA per SM: segments
    when its estimated time per token (``palimpsa_bwd_token_cost``: waves of CTAs times what their warps cost, at the
    tile height it would take) is by enough above that of the cut grid.  How much is enough, from 270 timed steps
    (T = 4096, 16x32 to 256x256, three types): 1.05 where the uncut grid is one wave and the boundary terms go through
    the tensor cores (16 heads of 128x128 bf16: 3.02 ms uncut, 2.51 cut), 1.15 where it is more (54: 5.60 / 4.34; 72 of
    64x128, ratio 1.14: 5.40 / 5.78; of the present kernels 32 of 128x128, T = 18793, 1.19: 20.5 / 19.5; 36, T = 4931,
    1.06: 5.54 / 6.09); with the exact float32 passes, which walk twice, 1.25 and 1.55 (16 heads of 96x192,
    1.19: 3.61 / 3.99; 64 of 128x64 float16, 1.31: 5.61 / 6.66; 54 of 64x128 float16, 1.52: 5.79 / 5.78).

    bfloat16 shapes that the tensor-core passes serve round their boundary terms, so accuracy is in play there: they are
    cut only where the grid at fixed nominal tile heights leaves a fifth of its waves idle, whatever the estimate says
    (30 heads of 64x128 stay exact and uncut at 3.24 ms, 2.49 in segments).

    Below 2048 tokens only float32 and float16 are cut, down to segments of 64 tokens and to one wave of CTAs: their
    boundary states and carried gradients are exact float32, so the results keep their accuracy.  A walk costs a serial
    chain per token and an idle GPU whatever else it does: 2 sequences x 4 heads of 64x64, T = 512, forward and backward:
    441 us uncut (16 CTAs), 123 in 8 segments; 4 x 4 heads of 31x65, T = 511, with the uncertainty output: 375 / 217 us
    in 4.  Forward only, from 3 segments up (24 heads of 31x65, T = 256: 70 / 53 us in 3); with a backward where
    the uncut walk is 1.6 times that of one wave of segments, whose gradients take two passes, plus 400 units (18 us) of
    launches.  280 float32 calls of 256 to 1900 tokens, 5 head sizes, 1 to 64 sequence-heads: the 166 that are cut take
    0.11 to 0.88 of their uncut time.  bfloat16 stays uncut there: its usual route would round; through the exact passes 8
    heads of 64x64, T = 512 take 130 us in 8 segments instead of 364.

    ``packed``: N documents of unequal length in one row of T tokens (``cu_seqlens``).  Only N and T are known
    without a host synchronisation.  With more CTAs than SMs the documents, started longest first, fill the waves by
    themselves (14 or 19 documents in 32 768 tokens: 4.3 ms unsegmented, 5.0-6.0 ms segmented); with fewer, the
    longest document is the critical path and segments of T / G tokens shorten it (7 documents x 16 heads in
    16 384 tokens: 4.16 -> 2.79 ms)."""
    sizes = [_known(x) for x in (N, T, H, K, V)]
    if None in sizes:
        return 1
    return L.torch_ops().plan_segments(*sizes, sm_count(device), bool(backward), int(io_dtype), bool(uncertainty),
                                       bool(packed))


def _known(x):
    """The size a plan is made for: a symbolic one counts with the value it is traced at.  Any number of segments is right
    for any size, so no guard is put on it and the traced graph holds for the other sizes too."""
    return x.node.hint if isinstance(x, torch.SymInt) else int(x)


def segment_len(T: int, G: int) -> int:
    per = (T + G - 1) // G
    return max(L.CKPT_INTERVAL, (per + L.CKPT_INTERVAL - 1) // L.CKPT_INTERVAL * L.CKPT_INTERVAL)


def make_segments(N, G, seg_len, H, V, K, dev, fwd: bool, with_rloc=True):
    """Allocates the [N,G,H,V,KP] boundary buffers and returns (ctypes struct, dict of tensors)."""
    KP = padded_k(K)
    f32 = dict(dtype=torch.float32, device=dev)
    sg = L.Segments()
    sg.num_segments, sg.seg_len = G, seg_len
    t = {}
    names = ("sum_M", "sum_J", "start_M", "start_I") if fwd else ("carry_M", "carry_I", "rloc_M", "rloc_I")
    for n in names:
        t[n] = torch.empty(N, G, H, V, KP, **f32)
        setattr(sg, n, t[n].data_ptr())
    if fwd:
        t["decay"] = torch.empty(N, G, H, **f32)
        sg.decay = t["decay"].data_ptr()
    return sg, t


_native = None
_loading = threading.Lock()


def native():
    """The native front end; the first call, of whichever thread, loads it and registers the operators' fake kernels.
    Importing this module makes that call where the package is built: a saved program (torch.export, TorchScript) or code
    that names ``torch.ops.palimpsa_b200`` needs the operators to exist, not a call of this package first."""
    global _native
    with _loading:
        if _native is None:
            ext = L.torch_ops()
            torch.library.register_fake("palimpsa_b200::fwd", _fwd_fake, allow_override=True)
            torch.library.register_fake("palimpsa_b200::bwd", _bwd_fake, allow_override=True)
            torch.library.register_fake("palimpsa_b200::decode_step", _decode_fake, allow_override=True)
            _native = ext
    return _native


def __getattr__(name):       # fwd_op, bwd_op: the registered operators, loaded on first use
    if name in ("fwd_op", "bwd_op"):
        native()
        return getattr(torch.ops.palimpsa_b200, name[:-3]).default
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


@torch.compiler.assume_constant_result        # runs when a caller is traced: the operators exist before they are named
def ensure_ops_registered() -> bool:
    native()
    return True


def _fwd_fake(q, k, v, b, gt, g, Ip, init_mu, init_I, cu_seqlens, scale, uncertainty, save_ckpt, want_final, recurrent,
              num_segments):
    B, T, H, K = q.shape
    V = v.shape[-1]
    N = B if cu_seqlens is None else cu_seqlens.numel() - 1
    f32 = dict(dtype=torch.float32, device=q.device)
    o = q.new_empty(B, T, H, V)
    o_var = q.new_empty(B, T, H, V) if uncertainty else q.new_empty(0)
    fmu = q.new_empty((N, H, V, K) if want_final else (0,), **f32)
    fI = q.new_empty((N, H, V, K) if want_final else (0,), **f32)
    cs = (_ckpt_slots(B * T, N), H, V, padded_k(K)) if save_ckpt else (0,)
    coff = q.new_empty((N,) if cu_seqlens is not None else (0,), dtype=torch.int32)
    seg = num_segments > 1 and T > 0
    decay = q.new_empty((N, num_segments, H) if seg else (0,), **f32)
    return o, o_var, fmu, fI, q.new_empty(cs, **f32), q.new_empty(cs, **f32), coff, decay


def _bwd_fake(do, do_var, q, k, v, b, gt, g, Ip, cu_seqlens, chunk_offsets, ckpt_M, ckpt_I, scale, explicit_init,
              recurrent, seg_decay):
    B, T, H, K = q.shape
    f32 = dict(dtype=torch.float32, device=q.device)
    return (torch.empty_like(q), torch.empty_like(k), torch.empty_like(v), torch.empty_like(b),
            q.new_empty(B, T, H, **f32), q.new_empty(H, **f32), q.new_empty(H, **f32))


def _decode_fake(q, k, v, b, gt, g, Ip, mu_state, I_state, scale, uncertainty):
    N, _, H, _ = q.shape
    V = v.shape[-1]
    return q.new_empty(N, 1, H, V), (q.new_empty(N, 1, H, V) if uncertainty else q.new_empty(0))


def takes_general_route(*args) -> bool:
    """A compiler traces the caller, or an argument's class or an active mode overrides torch functions: the call has to
    appear as the registered operator.  What else may stand between it and the kernels, the native entries see themselves."""
    return torch.compiler.is_compiling() or has_torch_function_variadic(*args)


def run_general(q, k, v, b, gt, g, Ip, initial_mu_state, initial_I_state, scale, output_final_state, output_uncertainty,
               cu_seqlens, recurrent: bool, out_dtype, num_segments: Optional[int] = None, var_dtype=None):
    """chunk_palimpsa / fused_recurrent_palimpsa around the registered operator, with the checks and the dtype policy of the
    native front end in Python that can be traced: what compilers, tracers, transforms, fake and wrapped tensors take."""
    ensure_ops_registered()
    if q.dim() != 4 or k.shape != q.shape or v.dim() != 4 or b.shape != v.shape or v.shape[:3] != q.shape[:3]:
        raise ValueError("expected q,k [B,T,H,K] and v,b [B,T,H,V]")
    B, T, H, K = q.shape
    V = v.shape[-1]
    if tuple(gt.shape) != (B, T, H) or tuple(g.shape) != (H,) or tuple(Ip.shape) != (H,):
        raise ValueError("expected gt [B,T,H] and g, Ip [H]")
    _require_cuda(q, k, v, b, gt, g, Ip, initial_mu_state, initial_I_state, cu_seqlens)
    if q.dtype not in _DT:
        raise TypeError(f"unsupported dtype {q.dtype}; use float32, bfloat16 or float16")
    if cu_seqlens is not None:
        cu_seqlens = cu_seqlens.to(torch.int32).contiguous()
        N = cu_seqlens.numel() - 1
    else:
        N = B
    if (initial_mu_state is None) != (initial_I_state is None):
        raise ValueError("initial_mu_state and initial_I_state must be given together")
    if initial_mu_state is not None:
        if tuple(initial_mu_state.shape) != (N, H, V, K) or tuple(initial_I_state.shape) != (N, H, V, K):
            raise ValueError(f"initial states must have shape {(N, H, V, K)}")
        initial_mu_state = initial_mu_state.detach().float().contiguous()
        initial_I_state = initial_I_state.detach().float().contiguous()
    # One io dtype per call: the widest of the four token tensors (the reference's kernels read each tensor in its
    # own dtype and compute in fp32, so a narrower choice would round an input the reference does not round;
    # under autocast its layers do pass fp32 q/k next to bf16 v).
    io = q.dtype
    for x in (k, v, b):
        io = torch.promote_types(io, x.dtype)
    if io not in _DT:
        raise TypeError(f"unsupported dtype combination {[x.dtype for x in (q, k, v, b)]}")
    q, k, v, b = [x.to(io).contiguous() for x in (q, k, v, b)]
    gt, g, Ip = [x.float().contiguous() for x in (gt, g, Ip)]
    save_ckpt = torch.is_grad_enabled() and any(x.requires_grad for x in (q, k, v, b, gt, g, Ip))
    if num_segments is None:
        num_segments = plan_segments(N, T, H, K, V, q.device, backward=bool(save_ckpt), io_dtype=_DT[io],
                                     uncertainty=bool(output_uncertainty), packed=cu_seqlens is not None)
    o, o_var, fmu, fI, _, _, _, _ = torch.ops.palimpsa_b200.fwd(q, k, v, b, gt, g, Ip, initial_mu_state, initial_I_state,
                                                                cu_seqlens, float(scale), bool(output_uncertainty),
                                                                save_ckpt, bool(output_final_state), recurrent,
                                                                int(num_segments))
    if out_dtype is not None and out_dtype != o.dtype:
        o = o.to(out_dtype)
    if output_uncertainty and var_dtype is not None and var_dtype != o_var.dtype:
        o_var = o_var.to(var_dtype)
    out = (o, o_var) if output_uncertainty else o
    if output_final_state:
        return out, fmu, fI
    return out


try:
    native()
except L.PalimpsaLibraryError:      # not built, or for another torch: the first call says so
    pass
