"""The work that a program built on palimpsa_b200 gives it, as cases that can be timed one by one.

Every case goes through the package's public entry points only.  ``kind`` picks the call:

    decode     one token for each of N running sequences: ``decode_step`` on the in-place (mu, I) cache
               (``entry="step"``), the same step replayed from a CUDA graph (``entry="graph"``), or the layer's own
               form, ``fused_recurrent_palimpsa`` with the cached states passed in and new ones handed back
               (``entry="layer"``)
    recurrent  ``fused_recurrent_palimpsa`` without gradients on a short prompt (the layers take it up to 64 tokens)
    prefill    ``chunk_palimpsa`` without gradients, final states handed to the decode cache
    train      ``chunk_palimpsa`` forward and backward
    packed     the same on one packed row of documents of different lengths (``cu_seqlens``)
    layer      ``layer_prologue`` and ``layer_epilogue`` forward and backward: the layer around the operator

Head shapes are those of the shipped configurations and of the benchmark: 48x48 and 48x96 with 16 heads (170M models),
96x192 with 16 heads (760M), 128x128 with 6 or 12 heads (benchmark), 64x64 with 4 heads in float32 (parity
configuration), 31x65 (the check script's odd shape), 16x32 (associative recall).
"""
import math

import torch
import torch.nn.functional as F

from palimpsa_b200 import chunk_palimpsa, decode_step, fused_recurrent_palimpsa
from palimpsa_b200.layers import layer_epilogue, layer_prologue
from palimpsa_b200.ops import DecodeGraph

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
DEV = "cuda"


def listed():
    return [
        # one user, one token, the 170M model: nothing but latency
        dict(name="decode_single", kind="decode", entry="step", N=1, H=16, K=48, V=48, dtype="bf16", unc=False),
        # a few dozen users on the 760M model, called as the reference's layer calls its cached fused op
        dict(name="decode_760m", kind="decode", entry="layer", N=61, H=16, K=96, V=192, dtype="bf16", unc=False),
        # a full server: 256 sequences, 805 MB of state read and written per token
        dict(name="decode_serving", kind="decode", entry="step", N=256, H=12, K=128, V=128, dtype="bf16", unc=False),
        # short prompts before decoding, 170M model with the wider value heads; the length is no multiple of anything
        dict(name="recurrent_short", kind="recurrent", B=4, T=37, H=16, K=48, V=96, dtype="bf16", unc=False),
        # long prompts of the 760M model, ragged length
        dict(name="prefill_760m", kind="prefill", B=2, T=3001, H=16, K=96, V=192, dtype="bf16", unc=False),
        # the parity configuration, float32: a small training step
        dict(name="train_fp32_small", kind="train", B=2, T=512, H=4, K=64, V=64, dtype="fp32", unc=False),
        # the check script's shape: odd sizes, uncertainty output, float32
        dict(name="train_odd_uncertainty", kind="train", B=4, T=511, H=4, K=31, V=65, dtype="fp32", unc=True),
        # the 170M model's training step
        dict(name="train_170m", kind="train", B=8, T=4096, H=16, K=48, V=48, dtype="bf16", unc=False),
        # one packed row of documents, as the training recipe feeds it
        dict(name="train_packed", kind="packed", T=32768, doc_min=128, doc_max=4096, H=6, K=128, V=128, dtype="bf16"),
        # the benchmark's training step
        dict(name="train_d128", kind="train", B=8, T=4096, H=6, K=128, V=128, dtype="bf16", unc=False),
        # one very long sequence
        dict(name="train_long", kind="train", B=1, T=131072, H=12, K=128, V=128, dtype="bf16", unc=False),
        # the element-wise work of the layer around the benchmark's operator
        dict(name="layer_d128", kind="layer", B=8, T=4096, H=6, Hq=6, K=128, V=128, dtype="bf16"),
    ]


# (d_k, d_v) a user's configuration may name, with the head counts that go with it
HEADS = [(16, 32), (48, 48), (48, 96), (64, 64), (96, 192), (128, 128), (32, 128), (31, 65)]
MAX_TRAIN = 4.0e11       # flops of a drawn training or prefill case: well below the largest listed one
MAX_STATE = 200 * 2**20  # bytes of a drawn decode case's (mu, I) cache


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "recurrent", "prefill", "train", "train", "packed", "layer"])
    if rng.random() < 0.75:
        K, V = rng.choice(HEADS)
    else:  # a size nobody tuned for
        K, V = rng.randint(8, 128), rng.randint(8, 200)
    c = dict(kind=kind, H=rng.choice([2, 4, 6, 8, 12, 16]), K=K, V=V,
             dtype=rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"]))
    unc = rng.random() < 0.15
    E = K * V
    if kind == "decode":
        top = max(2, min(512, MAX_STATE // (8 * E * c["H"])))
        c.update(entry=rng.choice(["step", "step", "layer", "graph"]), N=_log(rng, 1, top), unc=unc)
    elif kind == "recurrent":
        c.update(B=_log(rng, 1, 32), T=rng.randint(2, 64), unc=unc)
    elif kind == "layer":
        c.update(B=_log(rng, 1, 8), T=_log(rng, 32, 4096), Hq=c["H"] if rng.random() < 0.6 else c["H"] // 2)
    else:
        T = _log(rng, 65, 16384) if kind == "prefill" else _log(rng, 64, 8192)
        if kind == "packed":
            c.update(T=max(1024, T * 4), doc_min=rng.choice([1, 64, 128]), doc_max=rng.choice([512, 2048, 4096]))
            tokens = c["T"]
        else:
            top = max(1, int(MAX_TRAIN / (42.0 * E * c["H"] * T)))
            c.update(B=_log(rng, 1, min(64, top)), T=T, unc=unc)
            tokens = c["B"] * T
        while c["H"] > 1 and 42.0 * E * c["H"] * tokens > MAX_TRAIN:
            c["H"] //= 2
    return c


def _dims(case):
    B = case.get("N", case.get("B", 1))
    T = 1 if case["kind"] == "decode" else case["T"]
    return B, T, case["H"], case["K"], case["V"], DTYPES[case["dtype"]]


def _doc_offsets(case, gen):
    """Documents of uniformly drawn length until the row is full; the last one is cut."""
    ends, tot = [0], 0
    while tot < case["T"]:
        n = int(torch.randint(case["doc_min"], case["doc_max"] + 1, (1,), generator=gen))
        tot = min(case["T"], tot + n)
        ends.append(tot)
    return torch.tensor(ends, dtype=torch.int32, device=DEV)


def prepare(case, seed):
    B, T, H, K, V, io = _dims(case)
    gen = torch.Generator(device=DEV).manual_seed(seed)

    def rn(*shape):
        return torch.randn(*shape, generator=gen, device=DEV)

    s = {"case": case}
    if case["kind"] == "layer":
        Hq = case["Hq"]
        ins = [F.silu(rn(B, T, Hq, K)).to(io), F.silu(rn(B, T, Hq, K)).to(io), F.silu(rn(B, T, H, V)).to(io),
               rn(B, T, H, V).to(io), rn(B, T, H).to(io), rn(B, T, H).to(io), rn(H) - 2.0, 0.1 * rn(H)]
        s["pro"] = [x.requires_grad_(True) for x in ins]
        s["pro_cot"] = [(0.1 * rn(B, T, H, n)).to(io) for n in (K, K, V, V)] + [0.1 * rn(B, T, H)]
        s["epi"] = [x.requires_grad_(True) for x in ((0.2 * rn(B, T, H, V)).to(io), ins[2].detach().clone(),
                                                     1.0 + 0.1 * rn(H), 1.0 + 0.1 * rn(V), rn(B, T, H, V).to(io))]
        s["epi_cot"] = (0.1 * rn(B, T, H, V)).to(io)
        return s
    # the operator's inputs as the layer produces them: normalised q and k, gates in (0, 1), positive step sizes
    s["q"] = F.normalize(rn(B, T, H, K), dim=-1).to(io)
    s["k"] = F.normalize(rn(B, T, H, K), dim=-1).to(io)
    s["v"] = rn(B, T, H, V).to(io)
    s["b"] = torch.sigmoid(rn(B, T, H, V)).to(io)
    s["gt"] = F.softplus(rn(B, T, H))
    s["g"] = F.softplus(rn(H))
    s["Ip"] = torch.ones(H, device=DEV)
    if case["kind"] == "decode":
        s["mu"] = 0.2 * rn(B, H, V, K)
        s["I"] = 1.0 + F.softplus(rn(B, H, V, K))
        if case["entry"] == "graph":
            s["graph"] = DecodeGraph(s["g"], s["Ip"], s["mu"], s["I"], dtype=io, output_uncertainty=case["unc"])
    if case["kind"] in ("train", "packed"):
        s["do"] = rn(B, T, H, V).to(io)
        if case.get("unc"):
            s["do_var"] = rn(B, T, H, V).to(io)
        if case["kind"] == "packed":
            s["cu_seqlens"] = _doc_offsets(case, torch.Generator().manual_seed(seed))
        s["leaves"] = [s[n].requires_grad_(True) for n in ("q", "k", "v", "b", "gt", "g", "Ip")]
    return s


def _flat(out):
    return list(out) if isinstance(out, tuple) else [out]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "layer":
        outs = layer_prologue(*s["pro"])
        y = layer_epilogue(*s["epi"])
        grads = torch.autograd.grad(outs, s["pro"], s["pro_cot"]) + torch.autograd.grad(y, s["epi"], s["epi_cot"])
        return [*outs, y, *grads]
    args = [s[n] for n in ("q", "k", "v", "b", "gt", "g", "Ip")]
    if kind == "decode":
        if case["entry"] == "graph":
            return [*_flat(s["graph"].step(*args[:5])), s["mu"], s["I"]]
        if case["entry"] == "step":
            out = decode_step(*args, s["mu"], s["I"], output_uncertainty=case["unc"])
        else:
            with torch.no_grad():
                out, s["mu"], s["I"] = fused_recurrent_palimpsa(
                    *args, initial_mu_state=s["mu"], initial_I_state=s["I"], output_final_state=True,
                    output_uncertainty=case["unc"])
        return [*_flat(out), s["mu"], s["I"]]
    if kind in ("recurrent", "prefill"):
        op = fused_recurrent_palimpsa if kind == "recurrent" else chunk_palimpsa
        with torch.no_grad():
            out, mu, I = op(*args, output_final_state=True, output_uncertainty=case["unc"])
        return [*_flat(out), mu, I]
    out = _flat(chunk_palimpsa(*s["leaves"], output_uncertainty=case.get("unc", False), cu_seqlens=s.get("cu_seqlens")))
    cot = [s["do"], s["do_var"]] if case.get("unc") else [s["do"]]
    return [*(x.detach() for x in out), *torch.autograd.grad(out, s["leaves"], cot)]


def work(case):
    """Bytes: every input read once and every output written once.  Flops per state element and token: 11 forward
    (recurrence, one reciprocal, output), 31 more backward; the uncertainty output adds 2 and 6."""
    B, T, H, K, V, io = _dims(case)
    es = torch.empty(0, dtype=io).element_size()
    rows, E, kind = B * T * H, K * V, case["kind"]
    if kind == "layer":
        qrows = B * T * case["Hq"]
        pro = es * (2 * qrows * K + 2 * rows * V + 2 * rows) + es * rows * (2 * K + 2 * V) + 4 * rows
        pro_bwd = pro + es * (2 * qrows * K + 2 * rows * V + 2 * rows)
        epi, epi_bwd = 4 * es * rows * V, 7 * es * rows * V
        return {"bytes": pro + pro_bwd + epi + epi_bwd, "flops": rows * (20 * K + 60 * V)}
    unc = 1 if case.get("unc") else 0
    fwd = rows * (es * (2 * K + (3 + unc) * V) + 4)
    flops = rows * E * (11 + 2 * unc)
    if kind == "decode":
        return {"bytes": fwd + 16 * B * H * E, "flops": flops}
    if kind in ("recurrent", "prefill"):
        return {"bytes": fwd + 8 * B * H * E, "flops": flops}
    bwd = rows * (es * (2 * K + (3 + unc) * V) + 4)          # d_o (and d_o_var) in, dq dk dv db dgt out
    return {"bytes": fwd + bwd, "flops": flops + rows * E * (31 + 6 * unc)}


def tolerance(case):
    return {"bf16": {"rel": 1e-2}, "fp16": {"rel": 2e-3}, "fp32": {"rel": 1e-5}}[case["dtype"]]
