"""The calls whose speed counts: what a model built on this package asks of it, through the public ops and the layer.

Every case is one pass of one kind of work:

  decode      one token per sequence with the fp32 state updated in place (GLA and KDA)
  gla         `chunk_gla`: a prompt (forward only) or a training step (forward + gradients); dense or packed
              sequences of any length; bf16 with heads of 128 or 64 channels, fp32 with 64
  simple_gla  `chunk_simple_gla`: long sequences with one scalar gate per head and token, or a constant decay per head
  kda         `chunk_kda` training step
  layer       `GatedLinearAttention` with its default head split (keys half as wide as values): training step, prompt,
              or one generated token
  neighbours  the steps around an attention block: L2 norm of q and k, gate activation, gated RMS norm

Inputs are drawn on the GPU from the seed with the distributions of the benchmark (`tops_b200.synth`): q, k, v and the
cotangents N(0, 1), log-gates log_sigmoid(N(0, 1)) / 16, states 0.1 N(0, 1), beta sigmoid(N(0, 1)).
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "pallas-kernel_b200")
if _PKG not in sys.path:
    sys.path.insert(1, _PKG)

from tops_b200.layers import Cache, GatedLinearAttention  # noqa: E402
from tops_b200.ops.gate import kda_gate_fwd  # noqa: E402
from tops_b200.ops.gla import chunk_gla, fused_recurrent_gla_decode_  # noqa: E402
from tops_b200.ops.kda import chunk_kda, fused_recurrent_kda_decode_  # noqa: E402
from tops_b200.ops.norm import FusedRMSNormGated, l2norm  # noqa: E402
from tops_b200.ops.simple_gla import chunk_simple_gla  # noqa: E402

_DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}


def listed():
    return [
        # one user's next token: the smallest call there is, all latency
        {"name": "gla_decode_one", "kind": "decode", "op": "gla", "B": 1, "H": 16, "K": 128, "V": 128},
        # a serving batch of 128 sequences: the whole state crosses HBM once in and once out
        {"name": "gla_decode_batch", "kind": "decode", "op": "gla", "B": 128, "H": 32, "K": 128, "V": 128},
        {"name": "kda_decode_batch", "kind": "decode", "op": "kda", "B": 16, "H": 32, "K": 128, "V": 128},
        # the reference's own CPU-sized call in fp32: parity checks and small experiments
        {"name": "gla_fwd_fp32", "kind": "gla", "dtype": "fp32", "B": 2, "T": 512, "H": 4, "D": 64, "docs": 0, "state": False,
         "train": False},
        # a prompt of arbitrary length before generation: no gradients, the final state is kept
        {"name": "gla_prefill", "kind": "gla", "dtype": "bf16", "B": 1, "T": 3001, "H": 16, "D": 128, "docs": 0,
         "state": False, "train": False},
        # the headline training step
        {"name": "gla_train", "kind": "gla", "dtype": "bf16", "B": 8, "T": 4096, "H": 16, "D": 128, "docs": 0, "state": True,
         "train": True},
        # documents packed into one row, as training data usually is
        {"name": "gla_train_packed", "kind": "gla", "dtype": "bf16", "B": 1, "T": 16384, "H": 16, "D": 128, "docs": 13,
         "state": False, "train": True},
        # one very long sequence
        {"name": "simple_gla_long", "kind": "simple_gla", "B": 1, "T": 65536, "H": 32, "gate": "g"},
        {"name": "kda_train", "kind": "kda", "B": 4, "T": 8192, "H": 32},
        # the layer as its constructor's defaults make it (hidden 1024, 4 heads: K = 128, V = 256)
        {"name": "layer_train", "kind": "layer", "mode": "train", "B": 4, "T": 2048, "hidden": 1024, "heads": 4},
        {"name": "layer_decode", "kind": "layer", "mode": "decode", "B": 8, "T": 1, "hidden": 1024, "heads": 4},
        # gate, norms and their gradients at the tensor size of the headline step
        {"name": "neighbours", "kind": "neighbours", "B": 8, "T": 4096, "H": 16, "D": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """Token counts: half of them whole chunks of 64, half as they come."""
    n = _log(rng, lo, hi)
    return max(64, n // 64 * 64) if rng.random() < 0.5 else n


def draw(rng):
    kind = rng.choice(["decode", "gla", "gla", "gla", "simple_gla", "kda", "layer", "layer", "neighbours"])
    if kind == "decode":
        H = rng.choice([4, 8, 16, 32])
        return {"kind": kind, "op": rng.choice(["gla", "kda"]), "B": _log(rng, 1, 128), "H": H, "K": 128,
                "V": rng.choice([64, 128, 128, 256])}
    if kind == "gla":
        dtype, D = rng.choice([("bf16", 128), ("bf16", 128), ("bf16", 64), ("fp32", 64)])
        H = rng.choice([2, 4, 8, 16])
        most = (1 << 19) if dtype == "bf16" else (1 << 16)   # tokens x heads
        if rng.random() < 1 / 3:
            T = _length(rng, 512, most // H // 2)
            return {"kind": kind, "dtype": dtype, "B": 1, "T": T, "H": H, "D": D, "docs": rng.randint(2, max(2, min(32, T // 64))),
                    "state": rng.random() < 0.5, "train": rng.random() < 0.75}
        B = _log(rng, 1, 8)
        return {"kind": kind, "dtype": dtype, "B": B, "T": _length(rng, 65, min(8192, most // H // B)), "H": H, "D": D, "docs": 0,
                "state": rng.random() < 0.5, "train": rng.random() < 0.5}
    if kind == "simple_gla":
        H = rng.choice([8, 16, 32])
        return {"kind": kind, "B": 1, "T": _length(rng, 1024, 65536), "H": H, "gate": rng.choice(["g", "gamma"])}
    if kind == "kda":
        B, H = _log(rng, 1, 4), rng.choice([4, 8, 16, 32])
        return {"kind": kind, "B": B, "T": _log(rng, 256, 8192) // 64 * 64, "H": H}
    if kind == "layer":
        hidden, heads = rng.choice([(512, 4), (1024, 4), (2048, 8)])
        mode = rng.choice(["train", "prefill", "decode"])
        B = _log(rng, 1, 64 if mode == "decode" else 8)
        T = 1 if mode == "decode" else _length(rng, 65, min(4096, 16384 // B))
        return {"kind": kind, "mode": mode, "B": B, "T": T, "hidden": hidden, "heads": heads}
    B = _log(rng, 1, 8)
    return {"kind": kind, "B": B, "T": _log(rng, 64, 4096), "H": rng.choice([4, 8, 16]), "D": rng.choice([64, 128])}


class _Draws:
    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, dtype=torch.bfloat16, scale=1.0):
        x = torch.randn(*shape, generator=self.gen, device="cuda", dtype=torch.float32)
        return (x * scale if scale != 1.0 else x).to(dtype)

    def gate(self, *shape, dtype=torch.bfloat16):
        return (torch.nn.functional.logsigmoid(self.normal(*shape, dtype=torch.float32)) / 16).to(dtype)

    def unit(self, *shape, dtype=torch.bfloat16):
        return torch.nn.functional.normalize(self.normal(*shape, dtype=torch.float32), dim=-1).to(dtype)


def _documents(T, docs, seed):
    """Boundaries of `docs` documents of uneven lengths in a row of T tokens."""
    cuts = torch.randperm(T - 1, generator=torch.Generator().manual_seed(seed))[: docs - 1] + 1
    return [0, *sorted(cuts.tolist()), T]


def prepare(case, seed):
    d = _Draws(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "decode":
        B, H, K, V = (case[n] for n in "BHKV")
        unit = case["op"] == "kda"
        s["q"] = d.unit(B, 1, H, K) if unit else d.normal(B, 1, H, K)
        s["k"] = d.unit(B, 1, H, K) if unit else d.normal(B, 1, H, K)
        s["v"], s["g"] = d.normal(B, 1, H, V), d.gate(B, 1, H, K)
        if unit:
            s["beta"] = torch.sigmoid(d.normal(B, 1, H, dtype=torch.float32)).to(torch.bfloat16)
        s["state"] = d.normal(B, H, K, V, dtype=torch.float32, scale=0.1)
        return s
    if kind == "neighbours":
        B, T, H, D = (case[n] for n in "BTHD")
        for n in ("q", "k", "raw", "x", "gate"):
            s[n] = d.normal(B, T, H, D).requires_grad_()
        s["A_log"] = torch.log(1 + 15 * torch.rand(H, generator=d.gen, device="cuda")).requires_grad_()
        s["dt_bias"] = d.normal(H * D, dtype=torch.float32).requires_grad_()
        s["norm"] = FusedRMSNormGated(D, device="cuda")
        s["cotangents"] = [d.normal(B, T, H, D) for _ in range(4)]
        return s
    if kind == "layer":
        with torch.random.fork_rng(devices=["cuda"]):
            torch.manual_seed(seed)
            layer = GatedLinearAttention(hidden_size=case["hidden"], num_heads=case["heads"], layer_idx=0)
        s["layer"] = layer.to("cuda", torch.bfloat16)
        s["x"] = d.normal(case["B"], case["T"], case["hidden"])
        if case["mode"] == "train":
            s["x"].requires_grad_()
            s["do"] = d.normal(case["B"], case["T"], case["hidden"])
            s["inputs"] = [s["x"], *layer.parameters()]
        elif case["mode"] == "decode":
            s["cache"] = Cache()
            state = d.normal(case["B"], case["heads"], layer.head_k_dim, layer.head_v_dim, dtype=torch.float32, scale=0.1)
            s["cache"].update(recurrent_state=state, layer_idx=0)
        return s
    B, T, H = (case[n] for n in "BTH")
    D = case.get("D", 128)
    dtype = _DTYPES[case.get("dtype", "bf16")]
    train = case.get("train", True)
    unit = kind == "kda"
    s["q"] = d.unit(B, T, H, D) if unit else d.normal(B, T, H, D, dtype=dtype)
    s["k"] = d.unit(B, T, H, D) if unit else d.normal(B, T, H, D, dtype=dtype)
    s["v"] = d.normal(B, T, H, D, dtype=dtype)
    names = ["q", "k", "v"]
    if kind == "simple_gla" and case["gate"] == "gamma":
        s["gamma"] = -torch.exp2(-5 - 3 * torch.rand(H, generator=d.gen, device="cuda"))
    else:
        s["g"] = d.gate(B, T, H, dtype=dtype) if kind == "simple_gla" else d.gate(B, T, H, D, dtype=dtype)
        names.append("g")
    if unit:
        s["beta"] = torch.sigmoid(d.normal(B, T, H, dtype=torch.float32)).to(dtype)
        names.append("beta")
    docs = case.get("docs", 0)
    s["cu"] = _documents(T, docs, seed) if docs else None
    N = docs or B
    if case.get("state", kind == "kda"):
        s["h0"] = d.normal(N, H, D, D, dtype=torch.float32, scale=0.1)
        names.append("h0")
    if train:
        s["do"] = d.normal(B, T, H, D, dtype=dtype)
        s["dht"] = d.normal(N, H, D, D, dtype=torch.float32, scale=0.1)
        s["inputs"] = [s[n].requires_grad_() for n in names]
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "decode":
        if case["op"] == "kda":
            o = fused_recurrent_kda_decode_(s["q"], s["k"], s["v"], s["g"], s["beta"], s["state"])
        else:
            o = fused_recurrent_gla_decode_(s["q"], s["k"], s["v"], s["g"], s["state"])
        return o, s["state"]
    if kind == "neighbours":
        outs = [l2norm(s["q"]), l2norm(s["k"]),
                kda_gate_fwd(s["raw"], s["A_log"], s["dt_bias"], output_dtype=torch.bfloat16), s["norm"](s["x"], s["gate"])]
        grads = torch.autograd.grad(outs, [s["q"], s["k"], s["raw"], s["A_log"], s["dt_bias"], s["x"], s["gate"],
                                           s["norm"].weight], s["cotangents"])
        return *outs, *grads
    if kind == "layer":
        if case["mode"] == "train":
            o = s["layer"](s["x"])[0]
            return o, *torch.autograd.grad(o, s["inputs"], s["do"])
        with torch.no_grad():
            if case["mode"] == "decode":
                o, _, cache = s["layer"](s["x"], past_key_values=s["cache"], use_cache=True)
            else:
                o, _, cache = s["layer"](s["x"], past_key_values=Cache(), use_cache=True)
            return o, cache[0]["recurrent_state"]
    if kind == "gla":
        o, ht = chunk_gla(s["q"], s["k"], s["v"], s["g"], initial_state=s.get("h0"), output_final_state=True,
                          cu_seqlens=s["cu"])
    elif kind == "simple_gla":
        o, ht = chunk_simple_gla(s["q"], s["k"], s["v"], g=s.get("g"), g_gamma=s.get("gamma"), output_final_state=True)
    else:
        o, ht = chunk_kda(s["q"], s["k"], s["v"], s["g"], s["beta"], initial_state=s["h0"], output_final_state=True)
    if "do" not in s:
        return o, ht
    return o, ht, *torch.autograd.grad([o, ht], s["inputs"], [s["do"], s["dht"]])


def work(case):
    """Bytes: every input read once, every output written once.  Operations: the multiply-adds of the recurrence
    itself (state update and read-out per token, and the four products of its gradient), which no chunking saves."""
    kind = case["kind"]
    if kind == "decode":
        B, H, K, V = (case[n] for n in "BHKV")
        bytes_ = B * H * (8 * K * V + 2 * (3 * K + 2 * V)) + (2 * B * H if case["op"] == "kda" else 0)
        return {"bytes": bytes_, "flops": B * H * K * V * (6 if case["op"] == "kda" else 4)}
    if kind == "neighbours":
        n = case["B"] * case["T"] * case["H"] * case["D"]
        return {"bytes": 18 * 2 * n, "flops": 60 * n}
    if kind == "layer":
        n, hid = case["B"] * case["T"], case["hidden"]
        K, V, heads = hid // 2, hid, case["heads"]
        weights = hid * (2 * K + 3 * V + 16) + 16 * K
        proj, rec, state = 2 * n * weights, 4 * n * (K // heads) * V, 4 * case["B"] * K * (V // heads)
        if case["mode"] == "train":
            return {"bytes": 2 * (4 * n * hid + 2 * weights), "flops": 3 * (proj + rec)}
        return {"bytes": 2 * (2 * n * hid + weights) + state * (2 if case["mode"] == "decode" else 1), "flops": proj + rec}
    B, T, H = (case[n] for n in "BTH")
    D = case.get("D", 128)
    es = 4 if case.get("dtype") == "fp32" else 2
    n = B * T * H
    states = (case.get("docs", 0) or B) * H * D * D * 4
    gate = {"g": 1, "gamma": 0}.get(case.get("gate"), D)
    beta = 1 if kind == "kda" else 0
    has_h0 = case.get("state", kind == "kda")
    products = 6 if kind == "kda" else 4
    fwd_in, fwd_out = n * (3 * D + gate + beta) * es, n * D * es
    if not case.get("train", True):
        return {"bytes": fwd_in + fwd_out + states * (2 if has_h0 else 1), "flops": products * n * D * D}
    return {"bytes": 2 * (fwd_in + fwd_out) + states * (4 if has_h0 else 2), "flops": 3 * products * n * D * D}


def tolerance(case):
    """bf16 operands and results with fp32 accumulation: two correct implementations round gated operands and chunk
    states at other places, a few 1e-3 per tensor in the 2-norm.  fp32: sums in another order.  A decode step rounds
    only its bf16 output; its fp32 state follows the same recurrence."""
    if case["kind"] == "decode":
        return {"rel": 2e-3, "max": 0.02}
    if case.get("dtype") == "fp32":
        return {"rel": 2e-5, "max": 1e-3}
    if case["kind"] == "neighbours":
        return {"rel": 4e-3, "max": 0.02}
    return {"rel": 1e-2, "max": 0.25}
